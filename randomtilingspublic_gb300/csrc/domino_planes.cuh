// What the bit-plane kernels of the domino sweep share (domino_cluster.cu, domino_grid.cu): access to
// the planes in shared memory, their load and write-back, and the draws of a warp's words.
//
// Planes: [rows][words][chains][VD0, VD1, HE, HO] 32-bit words; see domino_cluster.cu.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "rng.cuh"

namespace rt {

enum : int { kClTmt = 0, kClTmtParams = 1, kClFast = 2 };
constexpr int kClPad = 16;  // words of the scratch word and its neighbours

__device__ __forceinline__ uint32_t cl_lds(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 cl_lds2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 cl_lds4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ void cl_sts(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cl_xor(uint32_t a, uint32_t v) {
  asm volatile("red.shared.xor.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cl_xor_if(uint32_t a, uint32_t v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p red.shared.xor.b32 [%0], %1;\n\t}" ::"r"(a), "r"(v)
               : "memory");
}
// The CTA's barrier, met by the update warps and the draw warps at places of their own.
__device__ __forceinline__ void cl_cta_sync() { asm volatile("barrier.sync 0;" ::: "memory"); }
// Bits a, b, c, d from the least significant up.
__device__ __forceinline__ uint32_t cl_nibble(bool a, bool b, bool c, bool d) {
  return (a ? 1u : 0u) | (b ? 2u : 0u) | (c ? 4u : 0u) | (d ? 8u : 0u);
}

// A CTA's window of the chains at src as planes: rows i0 .. i0 + R - 1, words wlo .. wlo + wn - 1 (one
// warp per row and word: lane l reads cell 32 w + l of both colours).
template <int NCH>
__device__ __forceinline__ void cl_load_window(uint32_t* planes, const uint8_t* src, size_t chain_stride,
                                               size_t colour_stride, int P, int i0, int R, int wlo, int wn) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
  for (int it = warp; it < R * wn; it += nwarps) {
    const int ri = it / wn, wi = it - ri * wn;
    const int i = i0 + ri, w = wlo + wi, m = 32 * w + lane;
    const bool in = i >= 0 && w >= 0 && m < P;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const uint8_t* row = src + (size_t)c * chain_stride + (size_t)i * P;
      const uint32_t b0 = in ? row[m] : 0u, b1 = in ? row[colour_stride + m] : 0u;
      const uint32_t bo = (i & 1) ? b1 : b0;  // the colour whose cells sit at odd lattice columns
      const uint32_t vd0 = __ballot_sync(~0u, (b0 >> 1) & 1u), vd1 = __ballot_sync(~0u, (b1 >> 1) & 1u);
      const uint32_t he = __ballot_sync(~0u, (bo >> 2) & 1u), ho = __ballot_sync(~0u, (bo >> 3) & 1u);
      if (lane < 4) planes[(it * NCH + c) * 4 + lane] = lane == 0 ? vd0 : lane == 1 ? vd1 : lane == 2 ? he : ho;
    }
  }
}

// Window rows 1 .. R - 1 of both colours back to the chains as edge masks: cells m in [1, cols] of the
// window's inner words (the others keep their bytes, as the reference never rebuilds them).
template <int NCH>
__device__ __forceinline__ void cl_store_window(const uint32_t* planes, uint8_t* base, size_t chain_stride,
                                                size_t colour_stride, int P, int cols, int i0, int R, int wlo, int wn) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (int)(blockDim.x >> 5);
  for (int it = warp; it < (R - 1) * (wn - 2) * 2; it += nwarps) {
    const int t = it & 1, q = it >> 1;
    const int ri = 1 + q / (wn - 2), wi = 1 + q % (wn - 2);
    const int i = i0 + ri, w = wlo + wi, m = 32 * w + lane;
    if (m < 1 || m > cols || m >= P) continue;
    const bool aligned = ((i + 1 - t) & 1) != 0;
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const uint32_t* me = planes + ((ri * wn + wi) * NCH + c) * 4;
      const uint32_t up = (me[-4 * wn * NCH + 1 - t] >> lane) & 1u, dn = (me[t] >> lane) & 1u;
      const uint32_t he = (me[2] >> lane) & 1u;
      uint32_t lft, rgt;
      if (aligned) {
        lft = he;
        rgt = (me[3] >> lane) & 1u;
      } else {
        lft = lane ? (me[3] >> (lane - 1)) & 1u : me[3 - 4 * NCH] >> 31;
        rgt = he;
      }
      base[(size_t)c * chain_stride + (size_t)t * colour_stride + (size_t)i * P + m] =
          (uint8_t)(up | (dn << 1) | (lft << 2) | (rgt << 3));
    }
  }
}

// The moves of a run, one pair of words per slot: bit k of x (y) is set where cell k, in state 3 (12)
// at the start of the run, is in state 3 at its end.  They do not depend on the state.
//
// TinyMT: L half-sweeps of the warp's KS words (lane l: the generator of cell l of each); rl =
// {width up, low down, width down} times 2^9, params(s, m1, m2, tm) the generator's parameters.
template <int KS, class Params>
__device__ __forceinline__ void cl_moves_tmt(uint4 (&gen)[KS], uint4 rl, int L, uint2* out, Params params) {
  const int lane = threadIdx.x & 31;
  // Every lane composes the moves of all its warp's words (two logic operations a word) where
  // registers allow it, else lane s those of slot s (two selects more).
  constexpr bool kAll = KS <= 4;
  uint32_t x[kAll ? KS : 1], y[kAll ? KS : 1];
#pragma unroll
  for (int s = 0; s < (kAll ? KS : 1); ++s) x[s] = 0xffffffffu, y[s] = 0u;
  for (int hh = 0; hh < L; ++hh) {
    uint32_t um = 0u, dm = 0u;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      uint32_t m1, m2, tm;
      params(s, m1, m2, tm);
      const uint32_t t0 = tmt_next_t0_mad(gen[s], m1, m2, tm);
      const uint32_t bu = __ballot_sync(~0u, t0 < rl.x);
      const uint32_t bd = __ballot_sync(~0u, t0 - rl.y < rl.z);
      if constexpr (kAll) {
        x[s] ^= (x[s] & bu) | (~x[s] & bd);
        y[s] ^= (y[s] & bu) | (~y[s] & bd);
      } else {
        um = lane == s ? bu : um;
        dm = lane == s ? bd : dm;
      }
    }
    if constexpr (!kAll) {
      x[0] ^= (x[0] & um) | (~x[0] & dm);
      y[0] ^= (y[0] & um) | (~y[0] & dm);
    }
  }
  if constexpr (kAll) {
#pragma unroll
    for (int s = 0; s < KS; ++s)
      if (lane == s) out[s] = make_uint2(x[s], y[s]);
  } else {
    if (lane < KS) out[lane] = make_uint2(x[0], y[0]);
  }
}

// Fast mode: one half-sweep of four words, lane l quad l % 8 of word l / 8 (row, quad: its Philox
// counter); four tests each way as one nibble, two lanes' nibbles as one byte of the word's moves.
__device__ __forceinline__ void cl_moves_of(const uint4& d, uint4 rl, uint2* out) {
  const int lane = threadIdx.x & 31;
  const uint32_t u = cl_nibble(d.x < rl.x, d.y < rl.x, d.z < rl.x, d.w < rl.x);
  const uint32_t v = cl_nibble(d.x - rl.y < rl.z, d.y - rl.y < rl.z, d.z - rl.y < rl.z, d.w - rl.y < rl.z);
  const uint32_t mine = (u ^ 15u) | (v << 16);
  const uint32_t pair = mine | (__shfl_down_sync(~0u, mine, 1) << 4);
  if (!(lane & 1)) {
    uint8_t* to = reinterpret_cast<uint8_t*>(out + (lane >> 3)) + ((lane & 7) >> 1);
    to[0] = (uint8_t)pair;
    to[4] = (uint8_t)(pair >> 16);
  }
}
__device__ __forceinline__ void cl_moves_fast(uint64_t seed, uint32_t stream, int64_t h, uint32_t row, uint32_t quad,
                                              uint4 rl, uint2* out) {
  cl_moves_of(fast_quad(seed, stream, h, row, quad), rl, out);
}
// Two half-sweeps, h and h + 1, whose Philox blocks are computed side by side.
__device__ __forceinline__ void cl_moves_fast2(uint64_t seed, uint32_t stream, int64_t h, uint32_t row, uint32_t quad,
                                               uint4 rl0, uint4 rl1, uint2* out0, uint2* out1) {
  const uint4 d0 = fast_quad(seed, stream, h, row, quad), d1 = fast_quad(seed, stream, h + 1, row, quad);
  cl_moves_of(d0, rl0, out0);
  cl_moves_of(d1, rl1, out1);
}

}  // namespace rt
