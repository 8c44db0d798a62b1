// Attention for few query rows against a long key/value sequence (decoding), sm_100a.
//
// What bounds it: memory.  One key and one value row (2 * head_dim bytes) serve `rows` query
// rows (the query heads that share a key/value head, times their query positions), at most a
// few dozen, so a pass cannot be faster than K and V can be read.  The prefill kernel
// (fa8_fwd_sm100.cu) pads the query rows to 128, computes 128 rows of exponentials per key and
// gives a slice to one SM however long its sequence is; here
//   * query heads sharing a key/value head are rows of one tile (without a causal mask the rows
//     of a group are contiguous in Q, O and the log-sum-exp and attend to the same keys), so
//     K and V are read once per group instead of once per head;
//   * a slice's keys are split over a thread-block cluster and over the warps of each of its
//     CTAs; the partial sums are put together through distributed shared memory, so the split
//     needs no workspace and no second launch;
//   * a warp streams 32 keys at a time from global memory straight into registers, in the order
//     in which mma.m16n8k16 wants its operands (all loads are 8 or 16 bytes a thread, whole
//     32-byte sectors), the next keys' loads in flight while the current ones are worked on.  There is no
//     shared-memory staging, hence no barrier and no wait in the loop.  tcgen05 would want 128
//     rows (or 128 lanes of keys and a transposed P through shared memory) for what is 48 small
//     products per 8 KB read (head dim 128, up to eight rows).
//
// Operand layouts.  S = Q K^T with the query rows as M (16, eight of them padding when RB = 1)
// and eight keys as N; the k index of the instruction may be permuted as long as both operands
// agree, so thread (g, t) = (lane / 4, lane % 4) takes bytes 16 t .. 16 t + 15 of every 64 of a
// row: each of the four words of a 16-byte load, widened to fp16, is its part of one k-step.
// O^T = V^T P^T with 16 output columns as M, the rows as N and 16 keys as k: a thread's P values of
// two score tiles are its part of the B operand as they stand, and its part of the A operand is
// two columns of four keys, paired up by byte permutations of rows of V.
//
// Numerics are those of the prefill kernel: P = 2^(c s - c m) in fp32, rounded to fp8 after the
// fp32 row sum, with m the exact row maximum over the first 64 keys of the slice (every warp of
// the cluster starts from it), raised by a warp, for itself, when the eight P of a thread in one step add
// up to more than 448 (no single one is larger then).  How many CTAs and warps share the keys depends on the
// number of slices and SMs, so the order of the fp32 sums, and which warps have raised their maximum, do
// too: the last bits of a slice's output change with the other slices of the launch.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "fa8_kernel.h"
#include "ptx_sm100.cuh"

namespace fa8 {

namespace {

namespace cg = cooperative_groups;

constexpr int kStepKeys = 32;          // keys of one warp step = k of one PV instruction
constexpr int kFirstKeys = 64;         // keys the starting maximum is taken over
constexpr float kRaiseAbove = 448.f;   // largest e4m3 value

// Every fp8 value is an fp16 value too, so a product of widened operands with an fp32 sum is the fp8
// product.  The instruction's own fp8 form is carried out in fp16 as well on this architecture, but
// widens both operands again for every product; widening each K and V word once by hand takes 421
// instructions per warp step instead of 652 (ncu), 51 us instead of 57 at batch 16, 8 key/value heads,
// 8192 keys, head dim 128.
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Four fp8 -> two pairs of fp16, ascending.
template <bool kE5M2>
__device__ __forceinline__ void widen4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  if (kE5M2) {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
        "cvt.rn.f16x2.e5m2x2 %0, l;\n\tcvt.rn.f16x2.e5m2x2 %1, h;\n\t}" : "=r"(lo), "=r"(hi) : "r"(w));
  } else {
    asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
        "cvt.rn.f16x2.e4m3x2 %0, l;\n\tcvt.rn.f16x2.e4m3x2 %1, h;\n\t}" : "=r"(lo), "=r"(hi) : "r"(w));
  }
}

// Two fp32 rounded to fp8, as a pair of fp16.
template <bool kE5M2>
__device__ __forceinline__ uint32_t round2(float a, float b) {
  uint32_t r;
  if (kE5M2) {
    asm("{\n\t.reg .b16 x;\n\tcvt.rn.satfinite.e5m2x2.f32 x, %2, %1;\n\tcvt.rn.f16x2.e5m2x2 %0, x;\n\t}" : "=r"(r) : "f"(a), "f"(b));
  } else {
    asm("{\n\t.reg .b16 x;\n\tcvt.rn.satfinite.e4m3x2.f32 x, %2, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, x;\n\t}" : "=r"(r) : "f"(a), "f"(b));
  }
  return r;
}

// Head dims up to W run in the instance built for W; bytes past head_dim are zeros in registers.
// RB: blocks of eight query rows a CTA works on (16 rows need a second PV product per column
// block; at W = 256 their accumulators do not fit the registers).
template <int W, int RB>
struct DCfg {
  static constexpr int kChunks = W / 64;                 // 64-byte pieces of a K row
  static constexpr int kSteps = W / 16;                  // k-steps of Q K^T
  static constexpr int kVWords = W == 64 ? 2 : 4;        // V words of a thread per key and column block
  static constexpr int kVBlocks = W == 256 ? 2 : 1;      // column blocks of 128
  static constexpr int kTilesPerBlock = 2 * kVWords;     // PV products (16 columns each) per column block
  static constexpr int kMTiles = W / 16;
  static constexpr int kRows = 8 * RB;
  static constexpr int kORow = W + 4;                    // floats per row of a partial sum in shared memory
  // Most warps of a CTA, and of an SM: what the register file holds at this instance's registers
  // per thread.
  static constexpr int kMaxWarps = W == 64 ? 16 : (W == 128 && RB == 1 ? 12 : 8);
  static constexpr int smem_bytes(int warps) {
    return warps * kRows * kORow * 4 + 2 * (warps + 1) * kRows * 4;
  }
};

// kExact: head_dim is W.
template <int W, int RB, bool kE5M2, bool kExact>
__global__ void __launch_bounds__(32 * DCfg<W, RB>::kMaxWarps, 1) fa8_decode_kernel(const DecodeArgs a) {
  using C = DCfg<W, RB>;
  extern __shared__ __align__(16) float smem[];
  const int warps = blockDim.x >> 5;
  // [warp][row][column] partial sums, then [warp + 1][row] maxima (times c) and row sums, the
  // last entry of each being the CTA's own
  float* s_o = smem;
  float* s_m = smem + warps * C::kRows * C::kORow;
  float* s_l = s_m + (warps + 1) * C::kRows;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n_split = a.n_split;
  const int rank = blockIdx.x % n_split;
  const int work = blockIdx.x / n_split;
  const int slice = work / a.row_blocks;
  const int row0 = (work - slice * a.row_blocks) * C::kRows;
  const int D = kExact ? W : a.head_dim, Sk = a.seqlen_k;
  start_after_predecessor();
  let_successor_start();
  // An earlier launch's expired wait is still in the status word: leave O alone, tell the host
  // (as the prefill kernel does).  The barriers below are passed all the same.
  const bool stale = __any_sync(0xffffffffu, a.status != nullptr && *reinterpret_cast<volatile int*>(a.status) != 0);
  if (stale && a.host_status != nullptr && threadIdx.x == 0 && *reinterpret_cast<volatile int*>(a.host_status) == 0)
    *reinterpret_cast<volatile int*>(a.host_status) = 0x5717;

  const uint8_t* kp = a.k + static_cast<size_t>(slice) * Sk * D;
  const uint8_t* vp = a.v + static_cast<size_t>(slice) * Sk * D;

  // Key steps of this CTA: a contiguous range, its warps taking them in turn.
  const int n_steps = (Sk + kStepKeys - 1) / kStepKeys;
  const int step_lo = static_cast<int>(static_cast<int64_t>(n_steps) * rank / n_split);
  const int step_hi = static_cast<int>(static_cast<int64_t>(n_steps) * (rank + 1) / n_split);

  // Rows past the last key are read as the last key again (its memory is there): no branch around a
  // load.  The scores of such keys are masked and their values cleared before use, for the last
  // key's may be an infinity.  Columns past head_dim are zeros.
  const int k_col = 16 * t, v_col = (C::kVWords * 4) * g;
  auto load_k = [&](uint4 (&r)[C::kChunks], int key) {
    const uint8_t* p = kp + static_cast<size_t>(min(key, Sk - 1)) * D + k_col;
#pragma unroll
    for (int c = 0; c < C::kChunks; ++c) {
      r[c] = make_uint4(0u, 0u, 0u, 0u);
      if (kExact || 64 * c + k_col < D) r[c] = ld_stream16(p + 64 * c);
    }
  };
  auto v_key = [&](int key0, int i) { return key0 + 16 * (i >> 2) + 8 * ((i >> 1) & 1) + 2 * t + (i & 1); };
  auto load_v = [&](uint32_t (&r)[8][C::kVWords], int key0, int blk) {
    const int col = 128 * blk + v_col;
#pragma unroll
    for (int i = 0; i < 8; ++i) {                       // k word i / 4, byte i % 4
      const int key = v_key(key0, i);
      const uint8_t* p = vp + static_cast<size_t>(min(key, Sk - 1)) * D + col;
#pragma unroll
      for (int w = 0; w < C::kVWords; ++w) r[i][w] = 0u;
      if (kExact || col < D) {
        if constexpr (C::kVWords == 2) {
          const uint2 x = ld_stream8(p);
          r[i][0] = x.x; r[i][1] = x.y;
        } else {
          const uint4 x = ld_stream16(p);
          r[i][0] = x.x; r[i][1] = x.y; r[i][2] = x.z; r[i][3] = x.w;
        }
      }
    }
  };

  // Q rows as A operands; rows past the last one are zeros.
  uint32_t qa[C::kSteps][RB][2];
#pragma unroll
  for (int h = 0; h < RB; ++h) {
    const int row = row0 + g + 8 * h;
    const uint8_t* p = a.q + (static_cast<size_t>(slice) * a.rows + row) * D + k_col;
#pragma unroll
    for (int c = 0; c < C::kChunks; ++c) {
      uint4 x = make_uint4(0u, 0u, 0u, 0u);
      if (row < a.rows && 64 * c + k_col < D) x = ld_global(reinterpret_cast<const uint4*>(p + 64 * c));
      widen4<kE5M2>(x.x, qa[4 * c][h][0], qa[4 * c][h][1]);
      widen4<kE5M2>(x.y, qa[4 * c + 1][h][0], qa[4 * c + 1][h][1]);
      widen4<kE5M2>(x.z, qa[4 * c + 2][h][0], qa[4 * c + 2][h][1]);
      widen4<kE5M2>(x.w, qa[4 * c + 3][h][0], qa[4 * c + 3][h][1]);
    }
  }
  auto scores = [&](const uint4 (&kr)[C::kChunks], float (&s)[4]) {
    s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll
    for (int c = 0; c < C::kChunks; ++c) {
      const uint32_t w[4] = {kr[c].x, kr[c].y, kr[c].z, kr[c].w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        uint32_t b0, b1;
        widen4<kE5M2>(w[u], b0, b1);
        const auto& qw = qa[4 * c + u];
        mma_f16(s, qw[0][0], RB == 2 ? qw[RB - 1][0] : 0u, qw[0][1], RB == 2 ? qw[RB - 1][1] : 0u, b0, b1);
      }
    }
  };

  // Loads are kept ahead of their use: those of the first step go out now, before the starting
  // maximum.  At W = 256 half of a step's K and of its V is held at a time (registers).
  constexpr int kHeld = W == 256 ? 2 : 4;                // score tiles whose K is in registers
  uint4 kr[kHeld][C::kChunks];
  uint32_t vr[8][C::kVWords];
  int step = step_lo + warp;
  const bool any = step < step_hi && !stale;
  if (any) {
#pragma unroll
    for (int j = 0; j < kHeld; ++j) load_k(kr[j], step * kStepKeys + 8 * j + g);
    load_v(vr, step * kStepKeys, 0);
  }

  // Scale of each of this thread's rows, and the starting maximum: each warp takes every
  // warps-th tile of the first 64 keys.
  float c_row[RB], m_row[RB], o_mul = a.o_scale;
  auto row_scale = [&](int row) {
    float x = 1.f;
    if (a.descale_q != nullptr)
      x *= ld_global(a.descale_q + (a.descale_per_head ? static_cast<size_t>(slice) * a.group + min(row, a.rows - 1) / a.seqlen_q : 0));
    if (a.descale_k != nullptr) x *= ld_global(a.descale_k + (a.descale_per_head ? slice : 0));
    return x;
  };
  if (a.descale_v != nullptr) o_mul *= ld_global(a.descale_v + (a.descale_per_head ? slice : 0));
#pragma unroll
  for (int h = 0; h < RB; ++h) {
    c_row[h] = a.scale_log2 * row_scale(row0 + g + 8 * h);
    m_row[h] = -INFINITY;
  }
  for (int tile = warp; tile < kFirstKeys / 8; tile += warps) {
    uint4 k0[C::kChunks];
    float s[4];
    load_k(k0, 8 * tile + g);                            // keys past the end repeat the last one
    scores(k0, s);
#pragma unroll
    for (int h = 0; h < RB; ++h) m_row[h] = fmaxf(m_row[h], fmaxf(s[2 * h], s[2 * h + 1]));
  }
  auto quad_max = [&](float x) {
    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
    return fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
  };
#pragma unroll
  for (int h = 0; h < RB; ++h) {
    m_row[h] = quad_max(m_row[h]);
    if (t == 0) s_m[warp * C::kRows + 8 * h + g] = m_row[h];
  }
  __syncthreads();
  float nm[RB], l_row[RB];
#pragma unroll
  for (int h = 0; h < RB; ++h) {
    for (int w = 0; w < warps; ++w) m_row[h] = fmaxf(m_row[h], s_m[w * C::kRows + 8 * h + g]);
    nm[h] = m_row[h] == -INFINITY ? 0.f : -m_row[h] * c_row[h];
    l_row[h] = 0.f;
  }
  __syncthreads();                                       // s_m is written again below

  float o[C::kMTiles][RB][4];
#pragma unroll
  for (int j = 0; j < C::kMTiles; ++j)
#pragma unroll
    for (int h = 0; h < RB; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][h][e] = 0.f;

  if (any) {
    for (; step < step_hi; step += warps) {
      const int key0 = step * kStepKeys;
      const int next = key0 + warps * kStepKeys;
      const bool more = step + warps < step_hi;
      float s[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        scores(kr[j % kHeld], s[j]);
        if (j + kHeld < 4) load_k(kr[j], key0 + 8 * (j + kHeld) + g);
      }
      if (more) {
#pragma unroll
        for (int j = 0; j < kHeld; ++j) load_k(kr[j], next + 8 * j + g);
      }
      if (key0 + kStepKeys > Sk) {                        // the sequence's last step
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (key0 + 8 * j + 2 * t + (e & 1) >= Sk) s[j][e] = -INFINITY;
      }
      float p[RB][8], sum[RB];
      auto exponentials = [&] {
#pragma unroll
        for (int h = 0; h < RB; ++h) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) p[h][2 * j + e] = ex2_approx(fmaf(s[j][2 * h + e], c_row[h], nm[h]));
          sum[h] = ((p[h][0] + p[h][1]) + (p[h][2] + p[h][3])) + ((p[h][4] + p[h][5]) + (p[h][6] + p[h][7]));
        }
      };
      exponentials();
      bool calm = true;
#pragma unroll
      for (int h = 0; h < RB; ++h) calm = calm && sum[h] <= kRaiseAbove;
      if (!__all_sync(0xffffffffu, calm)) {
        // Some row has outgrown the fp8 range (or holds a NaN): take this step's maximum in.
#pragma unroll
        for (int h = 0; h < RB; ++h) {
          float mx = m_row[h];
#pragma unroll
          for (int j = 0; j < 4; ++j) mx = fmaxf(mx, fmaxf(s[j][2 * h], s[j][2 * h + 1]));
          mx = quad_max(mx);
          const float nm_new = mx == -INFINITY ? 0.f : -mx * c_row[h];
          const float alpha = ex2_approx(nm_new - nm[h]);
          l_row[h] *= alpha;
          // rows 2t and 2t + 1 of the row block are the columns of O^T this thread holds
          const float a0 = __shfl_sync(0xffffffffu, alpha, 8 * t), a1 = __shfl_sync(0xffffffffu, alpha, 8 * t + 4);
#pragma unroll
          for (int j = 0; j < C::kMTiles; ++j) {
            o[j][h][0] *= a0; o[j][h][2] *= a0;
            o[j][h][1] *= a1; o[j][h][3] *= a1;
          }
          m_row[h] = mx;
          nm[h] = nm_new;
        }
        exponentials();
      }
      uint32_t pb[RB][4];                                 // one word per score tile
#pragma unroll
      for (int h = 0; h < RB; ++h) {
        l_row[h] += sum[h];
#pragma unroll
        for (int j = 0; j < 4; ++j) pb[h][j] = round2<kE5M2>(p[h][2 * j], p[h][2 * j + 1]);
      }
#pragma unroll
      for (int blk = 0; blk < C::kVBlocks; ++blk) {
        if (key0 + kStepKeys > Sk) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int w = 0; w < C::kVWords; ++w)
              if (v_key(key0, i) >= Sk) vr[i][w] = 0u;
        }
#pragma unroll
        for (int w = 0; w < C::kVWords; ++w) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {                   // 16 keys each
            // bytes of two keys side by side, two columns a word
            const uint32_t* x = &vr[4 * u][w];
            constexpr int kKey = C::kVWords;              // words from one key to the next
            uint32_t a[4][2];
            widen4<kE5M2>(__byte_perm(x[0], x[kKey], 0x5140), a[0][0], a[1][0]);
            widen4<kE5M2>(__byte_perm(x[2 * kKey], x[3 * kKey], 0x5140), a[0][1], a[1][1]);
            widen4<kE5M2>(__byte_perm(x[0], x[kKey], 0x7362), a[2][0], a[3][0]);
            widen4<kE5M2>(__byte_perm(x[2 * kKey], x[3 * kKey], 0x7362), a[2][1], a[3][1]);
#pragma unroll
            for (int h = 0; h < RB; ++h) {
              mma_f16(o[blk * C::kTilesPerBlock + 2 * w][h], a[0][0], a[1][0], a[0][1], a[1][1], pb[h][2 * u], pb[h][2 * u + 1]);
              mma_f16(o[blk * C::kTilesPerBlock + 2 * w + 1][h], a[2][0], a[3][0], a[2][1], a[3][1], pb[h][2 * u], pb[h][2 * u + 1]);
            }
          }
        }
        if (blk + 1 < C::kVBlocks) load_v(vr, key0, blk + 1);
        else if (more) load_v(vr, next, 0);
      }
    }
  }

  // Partial sums of this warp -> shared memory.  Product j of a column block holds columns
  // v_col + 2j (rows g) and v_col + 2j + 1 (rows g + 8 of the instruction).
#pragma unroll
  for (int h = 0; h < RB; ++h) {
    l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 1);
    l_row[h] += __shfl_xor_sync(0xffffffffu, l_row[h], 2);
    if (t == 0) {
      s_m[warp * C::kRows + 8 * h + g] = -nm[h];
      s_l[warp * C::kRows + 8 * h + g] = l_row[h];
    }
    float* r0 = s_o + (warp * C::kRows + 8 * h + 2 * t) * C::kORow;
#pragma unroll
    for (int j = 0; j < C::kMTiles; ++j) {
      const int col = 128 * (j / C::kTilesPerBlock) + v_col + 2 * (j % C::kTilesPerBlock);
      *reinterpret_cast<float2*>(r0 + col) = make_float2(o[j][h][0], o[j][h][2]);
      *reinterpret_cast<float2*>(r0 + C::kORow + col) = make_float2(o[j][h][1], o[j][h][3]);
    }
  }
  __syncthreads();

  // The CTA's sum, in the place of warp 0's: every thread takes four columns of a row at a time.
  const int n_rows = min(C::kRows, a.rows - row0), quads = D / 4;
  for (int i = threadIdx.x; i < n_rows * quads; i += blockDim.x) {
    const int r = i / quads, col = 4 * (i - r * quads);
    float m = s_m[r];
    for (int w = 1; w < warps; ++w) m = fmaxf(m, s_m[w * C::kRows + r]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (int w = 0; w < warps; ++w) {
      const float f = ex2_approx(s_m[w * C::kRows + r] - m);
      const float4 x = *reinterpret_cast<const float4*>(s_o + (w * C::kRows + r) * C::kORow + col);
      acc.x += x.x * f; acc.y += x.y * f; acc.z += x.z * f; acc.w += x.w * f;
      l += s_l[w * C::kRows + r] * f;
    }
    *reinterpret_cast<float4*>(s_o + r * C::kORow + col) = acc;
    if (col == 0) {
      s_m[warps * C::kRows + r] = m;
      s_l[warps * C::kRows + r] = l;
    }
  }
  // The cluster's sum: each CTA writes its share of the output.
  cg::cluster_group cluster = cg::this_cluster();
  if (n_split > 1) cluster.sync();
  else __syncthreads();
  for (int i = rank * blockDim.x + threadIdx.x; i < n_rows * quads && !stale; i += n_split * blockDim.x) {
    const int r = i / quads, col = 4 * (i - r * quads);
    float m = -INFINITY;
    for (int p = 0; p < n_split; ++p)
      m = fmaxf(m, n_split > 1 ? *cluster.map_shared_rank(s_m + warps * C::kRows + r, p) : s_m[warps * C::kRows + r]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (int p = 0; p < n_split; ++p) {
      const float* po = s_o + r * C::kORow + col;
      const float* pm = s_m + warps * C::kRows + r;
      const float* pl = s_l + warps * C::kRows + r;
      if (n_split > 1) {
        po = cluster.map_shared_rank(po, p);
        pm = cluster.map_shared_rank(pm, p);
        pl = cluster.map_shared_rank(pl, p);
      }
      const float f = ex2_approx(*pm - m);
      const float4 x = *reinterpret_cast<const float4*>(po);
      acc.x += x.x * f; acc.y += x.y * f; acc.z += x.z * f; acc.w += x.w * f;
      l += *pl * f;
    }
    const float inv = ((l == 0.f || l != l) ? 1.f : 1.f / l) * o_mul;
    const size_t row = static_cast<size_t>(slice) * a.rows + row0 + r;
    const uint2 out = make_uint2(pack_half2(acc.x * inv, acc.y * inv), pack_half2(acc.z * inv, acc.w * inv));
    *reinterpret_cast<uint2*>(a.o + row * D + col) = out;
    // log(sum exp(scale s)): m is in units of log2
    if (a.lse != nullptr && col == 0) a.lse[row] = m * 0.6931471805599453f + __logf(l);
  }
  if (n_split > 1) cluster.sync();                         // no CTA leaves while its shared memory is read
}

template <int W, int RB, bool kE5M2, bool kExact>
cudaError_t launch_decode_inst(DecodeArgs a, int sms, cudaStream_t stream) {
  using C = DCfg<W, RB>;
  auto kernel = &fa8_decode_kernel<W, RB, kE5M2, kExact>;
  // Per device, set up by the first launch: kernel attributes, and 1 + the clusters of sixteen of the
  // largest CTAs that the device runs at once (0 = not yet).
  static std::atomic<int> big_clusters[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool cached = dev >= 0 && dev < 64;
  int big = cached ? big_clusters[dev].load(std::memory_order_acquire) : 0;
  if (big == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes(C::kMaxWarps));
    if (e != cudaSuccess) return e;
    int n = 0;
    cudaLaunchConfig_t probe{};
    probe.gridDim = dim3(16, 1, 1);
    probe.blockDim = dim3(32 * C::kMaxWarps, 1, 1);
    probe.dynamicSmemBytes = C::smem_bytes(C::kMaxWarps);
    cudaLaunchAttribute size[1];
    size[0].id = cudaLaunchAttributeClusterDimension;
    size[0].val.clusterDim.x = 16;
    size[0].val.clusterDim.y = 1;
    size[0].val.clusterDim.z = 1;
    probe.attrs = size;
    probe.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &probe) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    big = 1 + n;
    if (cached) big_clusters[dev].store(big, std::memory_order_release);
  }
  a.row_blocks = (a.rows + C::kRows - 1) / C::kRows;
  const int64_t items = static_cast<int64_t>(a.n_slices) * a.row_blocks;
  int warps = 4;
  a.n_split = decode_split(items, a.seqlen_k, C::kMaxWarps, sms, items < big ? 16 : 8, &warps);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(items * a.n_split), 1, 1);
  cfg.blockDim = dim3(32 * warps, 1, 1);
  cfg.dynamicSmemBytes = C::smem_bytes(warps);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {overlap_attribute()};
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(a.n_split);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.n_split > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <int W, int RB, bool kE5M2>
cudaError_t launch_decode_one(const DecodeArgs& a, int sms, cudaStream_t stream) {
  return a.head_dim == W ? launch_decode_inst<W, RB, kE5M2, true>(a, sms, stream)
                         : launch_decode_inst<W, RB, kE5M2, false>(a, sms, stream);
}

template <bool kE5M2>
cudaError_t launch_decode_fmt(const DecodeArgs& a, int sms, cudaStream_t stream) {
  if (a.head_dim <= 64)
    return a.rows <= 8 ? launch_decode_one<64, 1, kE5M2>(a, sms, stream) : launch_decode_one<64, 2, kE5M2>(a, sms, stream);
  if (a.head_dim <= 128)
    return a.rows <= 8 ? launch_decode_one<128, 1, kE5M2>(a, sms, stream) : launch_decode_one<128, 2, kE5M2>(a, sms, stream);
  return launch_decode_one<256, 1, kE5M2>(a, sms, stream);
}

}  // namespace

// As many warps as one wave of the GPU holds, every one with at least a step of its own; among
// equals the smallest CTAs.  A second, partly filled wave costs more than the warps it adds
// (batch 16, 8 key/value heads, 8192 keys, head dim 128, an earlier form of the kernel: 57 us with
// three CTAs of four warps per slice, 384 of the 444 that fit; 70 with two, 77 with four).
// max_split: 8, the portable cluster size, or 16 where the device runs a cluster of sixteen for every
// item at once (batch 1, 32768 keys: one key/value head of 128 columns 21.7 -> 15.5 us, two of 64 14.5 -> 10.3).
int decode_split(int64_t items, int seqlen_k, int max_warps, int sms, int max_split, int* warps) {
  const int steps = (seqlen_k + kStepKeys - 1) / kStepKeys;
  int best_split = 1, best_warps = 4;
  int64_t best = 0;
  for (int nw : {4, 8, max_warps}) {
    if (nw > max_warps) continue;
    int64_t split = static_cast<int64_t>(sms) * (max_warps / nw) / items;
    if (split > max_split) split = max_split;
    if (split > steps / nw) split = steps / nw;
    if (split < 1) split = 1;
    const int64_t busy = items * split * (nw < steps ? nw : steps);
    // a CTA size that does not fit one wave is no gain
    if (nw > 4 && items * split > static_cast<int64_t>(sms) * (max_warps / nw)) continue;
    if (busy > best) { best = busy; best_split = static_cast<int>(split); best_warps = nw; }
  }
  *warps = best_warps;
  return best_split;
}

// Up to kDecodeRowsMax rows may come here.  A single block of rows always does.  Several blocks each
// read K and V (from L2, at the same rate per SM), so they do when the prefill kernel would leave SMs
// idle: it does not split a slice's keys.  Both sides' costs (us) are fits to launches of 4-160 slices of 16-56
// rows, 1024 and 8192 keys; a head dim costs as much as the width of the instance it runs in (64 slices of 16
// rows, 8192 keys, head dim 160 / 192 / 224: 103 / 106 / 109 us).  Measured, here against there: 16 slices of 56
// rows, 8192 keys, head dim 64: 17, 61; 64 of them at 128: 98, 73; 32 slices of 16 rows, 8192 keys at 256:
// 47, 70, 64 of them: 86, 71; of 1024 keys: 15.8, 14.8.
bool decode_takes(int64_t slices, int64_t rows, int seqlen_k, int head_dim, int sms) {
  const int width = head_dim <= 64 ? 64 : (head_dim <= 128 ? 128 : 256);
  const int64_t block = width == 256 ? 8 : 16;
  const int64_t row_blocks = (rows + block - 1) / block;
  if (rows > kDecodeRowsMax || slices * row_blocks * 8 > 0x7fffffff) return false;
  if (row_blocks == 1) return true;
  const double keys = seqlen_k;
  const double step = width == 64 ? 0.43 : (width == 128 ? 0.51 : 0.49);                // of 64 keys there
  const double here = static_cast<double>(row_blocks) * slices * keys * 2.0 * width / 4.7e6 + 3.0;
  const double there = static_cast<double>((slices + sms - 1) / sms) * (keys / 64.0 * step + 5.5);
  return here < there;
}

int current_sm_count(cudaError_t* e) {
  static std::atomic<int> sm_count[64];
  int dev = 0;
  *e = cudaGetDevice(&dev);
  if (*e != cudaSuccess) return 0;
  const bool cached = dev >= 0 && dev < 64;
  int sms = cached ? sm_count[dev].load(std::memory_order_acquire) : 0;
  if (sms == 0) {
    *e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (*e != cudaSuccess) return 0;
    if (cached) sm_count[dev].store(sms, std::memory_order_release);
  }
  return sms;
}

cudaError_t launch_decode(const DecodeArgs& a, bool e5m2, int sms, cudaStream_t stream) {
  return e5m2 ? launch_decode_fmt<true>(a, sms, stream) : launch_decode_fmt<false>(a, sms, stream);
}

}  // namespace fa8
