// Phases of the barriers of a tile's score buffers in the prefill kernel (fa8_fwd_sm100.cu).
//
// Every sub-block sb of a work item lives in buffer sb % kNB of its tile.  Buffer b has three barriers,
// each completing one phase per sub-block that goes through the buffer: s_full (its scores are there), p_full
// (its P is there) and o_done (its PV is complete).
//
// A wait by parity passes when the number of completed phases, seen modulo two, is the one after the
// awaited phase.  So it is right only while that number is known to be within one of it: with the awaited phase
// numbered p (from 0), p or p + 1 phases are complete.  Where the three are waited for:
//   s_full(sb)     p or more: the warp's own previous sub-block, sb - kW, had its scores, and kW <= kNB;
//                  p + 1 at most: the next scores in this buffer need PV(sb), which needs this warp's P(sb).
//   p_full(sb-1)   p or more: S(sb-1) lies before S(sb), which is there, and was issued after PV(sb-1-kNB), which
//                  needs P(sb-1-kNB); p + 1 at most: P(sb-1+kNB) follows P(sb) in the order of hand-overs.
//   o_done(sb-1)   p or more: S(sb-1) is there and was issued after PV(sb-1-kNB), and the tensor core completes
//                  a tile's products in order; p + 1 at most: PV(sb) needs P(sb).
// One barrier for all PVs of the tile (one phase each) would not do for o_done: with more than two buffers S(sb) says
// only that PV(sb-kNB) is complete (sb-kNB-1 where two sub-blocks share a product), which is two or more phases behind
// PV(sb-1), and the wait for that one passes on the parity of PV(sb-3).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FA8_HD __host__ __device__ __forceinline__
#else
#define FA8_HD inline
#endif

namespace fa8 {

// Parity to wait with for sub-block sb of the current item; bit b of ph_bits: parity of the phases buffer b has
// been through before the item.
template <int kNB>
FA8_HD uint32_t phase_parity(uint32_t ph_bits, int sb) {
  return ((ph_bits >> (sb % kNB)) ^ static_cast<uint32_t>(sb / kNB)) & 1u;
}

// Parity of the number of sub-blocks, of an item of n, that go through buffer b.
template <int kNB>
FA8_HD uint32_t phases_used(int b, int n) {
  return static_cast<uint32_t>((n + kNB - 1 - b) / kNB) & 1u;
}

}  // namespace fa8
