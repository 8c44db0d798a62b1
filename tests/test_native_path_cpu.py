"""When the package's operators go through the compiled module, without a GPU."""
import pytest
import torch

from cutlass_flash_atten_fp8_b200 import api, build

F8 = torch.float8_e4m3fn


def test_module_is_taken_when_built_and_left_alone_when_stale(monkeypatch):
    build.build_binding()
    assert not build.binding_is_stale()
    monkeypatch.setattr(api, "_native_module", None)
    assert api._native() and hasattr(api._native(), "_forward")
    monkeypatch.setattr(build, "_binding_digest", lambda: "0" * 64)
    assert build.binding_is_stale()
    monkeypatch.setattr(api, "_native_module", None)
    assert api._native() is False


def test_an_installed_copy_without_sources_is_not_stale(monkeypatch):
    build.build_binding()

    def gone():
        raise FileNotFoundError
    monkeypatch.setattr(build, "_binding_digest", gone)
    assert not build.binding_is_stale()


@pytest.mark.parametrize("native", [True, False])
def test_the_same_complaints_either_way(monkeypatch, native):
    build.build_binding()
    monkeypatch.setattr(api, "_native_module", None if native else False)
    q = torch.zeros(1, 1, 128, 64).to(F8)
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        api.flash_attention_v2_cutlass(q, q, q, False, 0.125, v_layout="natural")
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        api.flash_attention_v2_cutlass(q, q, q, False, 0.125, v_layout="upside down")
    with pytest.raises(RuntimeError, match="x must be a CUDA tensor"):
        api.quantize_e4m3(torch.zeros(4, 4, dtype=torch.float16))


def test_a_module_built_for_another_torch_is_stale(monkeypatch):
    build.build_binding()
    monkeypatch.setattr(torch, "__version__", "1.0")
    assert build.binding_is_stale()

    def gone():
        raise FileNotFoundError
    monkeypatch.setattr(build, "_binding_digest", gone)          # an installed copy notices as well
    assert build.binding_is_stale()


@pytest.mark.parametrize("error", [ImportError("undefined symbol"), OSError("cannot open shared object file")])
def test_a_module_that_does_not_load_leaves_ctypes(monkeypatch, error):
    build.build_binding()

    def broken(spec):
        raise error
    monkeypatch.setattr(api, "_native_module", None)
    monkeypatch.setattr(api.importlib.util, "module_from_spec", broken)
    with pytest.warns(UserWarning, match="through ctypes"):
        assert api._native() is False
    q = torch.zeros(1, 1, 128, 64).to(F8)
    with pytest.raises(RuntimeError, match="q must be a CUDA tensor"):
        api.flash_attention_v2_cutlass(q, q, q, False, 0.125, v_layout="natural")
