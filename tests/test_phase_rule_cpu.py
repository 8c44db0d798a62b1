"""The waits on the score buffers' barriers (csrc/phase_rule.h, compiled here for the host as the kernel uses
it) against a model of one query tile: in every state that the order of issue allows, a wait for PV(sb-1) before
O is rescaled passes exactly when that product is complete, and the waits for scores and P likewise."""
import os
import shutil
import subprocess

import pytest

from cutlass_flash_atten_fp8_b200.build import CSRC

# A tile's issuer: the first kNB scores, then PV(sb) and the scores that go where it has read; wide: one product for
# the scores of an even sub-block and the next one.  The tensor core completes what was issued in order.
MODEL = r"""
#include <cstdio>
#include <vector>
#include "phase_rule.h"
struct Op { bool pv; int sb; };
static std::vector<Op> issue_order(int kNB, bool wide, int n) {
  std::vector<Op> ops;
  auto qk = [&](int s) { if (s < n) { ops.push_back({false, s}); if (wide && s + 1 < n) ops.push_back({false, s + 1}); } };
  for (int s = 0; s < kNB; s += wide ? 2 : 1) qk(s);
  for (int sb = 0; sb < n; ++sb) {
    ops.push_back({true, sb});
    if (!wide) qk(sb + kNB); else if (sb & 1) qk(sb + 3);
  }
  return ops;
}
static bool passes(uint32_t completed, uint32_t parity) { return ((completed & 1u) ^ 1u) == parity; }
template <int kNB>
int run(bool wide, int kW) {
  int wrong = 0, old_rule_wrong = 0;
  for (int first = 0; first <= 2 * kNB + 1; ++first)          // sub-blocks of the item before
    for (int n = 1; n <= 4 * kNB + 3; ++n) {
      uint32_t base[kNB] = {}, bits = 0, pvs = first;
      for (int sb = 0; sb < first; ++sb) ++base[sb % kNB];
      for (int b = 0; b < kNB; ++b) bits ^= fa8::phases_used<kNB>(b, first) << b;
      const auto ops = issue_order(kNB, wide, n);
      auto at = [&](bool pv, int sb) { int i = 0; while (ops[i].pv != pv || ops[i].sb != sb) ++i; return i; };
      for (int sb = 0; sb < n; ++sb) {
        // done = operations complete: PV(sb) cannot be (its P comes from the waiting warp)
        const int most = at(true, sb);
        const int seen = sb >= kW ? at(false, sb - kW) + 1 : 0;
        for (int done = seen; done <= most; ++done) {
          uint32_t s[kNB], o[kNB], total = pvs;
          for (int b = 0; b < kNB; ++b) s[b] = o[b] = base[b];
          for (int i = 0; i < done; ++i) { ops[i].pv ? (++o[ops[i].sb % kNB], ++total) : ++s[ops[i].sb % kNB]; }
          const bool have_s = at(false, sb) < done;
          wrong += passes(s[sb % kNB], fa8::phase_parity<kNB>(bits, sb)) != have_s;
          if (!have_s || sb == 0) continue;
          const bool quiet = at(true, sb - 1) < done;
          wrong += passes(o[(sb - 1) % kNB], fa8::phase_parity<kNB>(bits, sb - 1)) != quiet;
          old_rule_wrong += passes(total, (pvs + sb - 1) & 1u) != quiet;
          // P handed over: those of the products complete, and any further ones before this warp's
          int last = -1;
          for (int i = 0; i < done; ++i) if (ops[i].pv) last = ops[i].sb;
          for (int i = 0; i < done; ++i) if (!ops[i].pv && ops[i].sb - kNB > last) last = ops[i].sb - kNB;
          for (int handed = last + 1; handed <= sb; ++handed) {
            uint32_t p = base[(sb - 1) % kNB];
            for (int x = 0; x < handed; ++x) p += x % kNB == (sb - 1) % kNB;
            wrong += passes(p, fa8::phase_parity<kNB>(bits, sb - 1)) != (handed > sb - 1);
          }
        }
      }
    }
  std::printf("%d %d\n", wrong, old_rule_wrong);
  return 0;
}
int main() { return run<2>(false, 2) + run<3>(false, 2) + run<4>(true, 4); }
"""


def test_waits_pass_exactly_when_the_product_is_complete(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "model.cpp", str(tmp_path / "model")
    src.write_text(MODEL)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I" + CSRC, str(src), "-o", exe], check=True)
    two, three, four = (tuple(map(int, line.split())) for line in subprocess.run([exe], check=True, capture_output=True,
                                                                                 text=True).stdout.splitlines())
    assert two[0] == three[0] == four[0] == 0
    # one barrier for all products of the tile is enough with two buffers only
    assert two[1] == 0 and three[1] > 0 and four[1] > 0


def test_the_kernel_uses_these_rules():
    with open(os.path.join(CSRC, "fa8_fwd_sm100.cu")) as f:
        text = f.read()
    for wait in ("bar_s_full(i, b), phase_parity<kNB>(ph_bits, sb)", "bar_p_full(i, (sb - 1) % kNB), phase_parity<kNB>(ph_bits, sb - 1)",
                 "bar_o_done(i, (sb - 1) % kNB), phase_parity<kNB>(ph_bits, sb - 1)"):
        assert wait in text
