// Pieces shared by the step kernel (amm_step.cu) and the set-up pass (amm_panel.cu): packed FP32x2
// arithmetic, the 16-byte vector unpacking and the branch-free body of one full column group.
#pragma once

#include "amm_device.cuh"
#include "amm_internal.h"

namespace amm {

// Packed FP32x2 arithmetic (Blackwell): two IEEE-rounded FMAs per instruction (the sm_100
// builtin, so the compiler allocates the register pairs itself).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// 16-byte vector -> E/2 float2 (exact for BF16: the 16 bits become the high half).
__device__ __forceinline__ void unpack2(const uint4& v, float2 (&o)[2]) {
  o[0] = make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
  o[1] = make_float2(__uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ void unpack2(const uint4& v, float2 (&o)[4]) {
  o[0] = make_float2(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u));
  o[1] = make_float2(__uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  o[2] = make_float2(__uint_as_float(v.z << 16), __uint_as_float(v.z & 0xffff0000u));
  o[3] = make_float2(__uint_as_float(v.w << 16), __uint_as_float(v.w & 0xffff0000u));
}

// Branch-free body of one full group: the axpy of group g (stage `cur`, coefficients `coef`)
// interleaved, slot by slot, with the partial dots of group g+1 (stage `nxt`) when NEXT.  Used
// when every column of both groups is present and every vector slot of every thread is valid.
template <typename Elem, int R, int GC, bool NEXT, int TC>
__device__ __forceinline__ void fused_block(const unsigned char* cur, const unsigned char* nxt,
                                            uint32_t col_bytes, int t, int T_rt,
                                            const float (&coef)[GC],
                                            const float2 (&dx)[R][8 / sizeof(Elem)],
                                            float2 (&yacc)[R][8 / sizeof(Elem)], float (&dn)[GC]) {
  constexpr int H = 8 / sizeof(Elem);
  // with a compile-time thread count (TC > 0) every shared-memory load uses an immediate offset
  const int T = TC > 0 ? TC : T_rt;
  const int colv = TC > 0 ? R * TC : (int)(col_bytes >> 4);  // vectors per column
  const uint4* c4 = reinterpret_cast<const uint4*>(cur) + t;
  const uint4* n4 = reinterpret_cast<const uint4*>(nxt) + t;
  float2 p[GC];
#pragma unroll
  for (int qq = 0; qq < GC; ++qq) p[qq] = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    uint4 vc[GC], vn[GC];
#pragma unroll
    for (int qq = 0; qq < GC; ++qq) {
      vc[qq] = c4[qq * colv + r * T];
      if (NEXT) vn[qq] = n4[qq * colv + r * T];
    }
#pragma unroll
    for (int qq = 0; qq < GC; ++qq) {
      float2 ac[H];
      unpack2(vc[qq], ac);
      const float2 c2 = make_float2(coef[qq], coef[qq]);
#pragma unroll
      for (int h = 0; h < H; ++h) yacc[r][h] = fma2(c2, ac[h], yacc[r][h]);
      if (NEXT) {
        float2 an[H];
        unpack2(vn[qq], an);
#pragma unroll
        for (int h = 0; h < H; ++h) p[qq] = fma2(an[h], dx[r][h], p[qq]);
      }
    }
  }
#pragma unroll
  for (int qq = 0; qq < GC; ++qq) dn[qq] = p[qq].x + p[qq].y;
}

// Sum over the 16 warps of NC partial values per warp (element (w, c) at base[w * stride + c]),
// computed identically by every warp: lane groups of L lanes own one value each and reduce by a
// fixed xor tree (deterministic).
template <typename V, int NC>
__device__ __forceinline__ void warp_partials_sum(const V* base, int stride, int lane,
                                                  V (&tot)[NC]) {
  constexpr int L = (32 / NC) < 16 ? (32 / NC) : 16;  // lanes per value
  constexpr int PER = 16 / L;                          // warp partials per lane
  constexpr int CPR = 32 / L;                          // values per round
  constexpr int ROUNDS = (NC + CPR - 1) / CPR;
#pragma unroll
  for (int rr = 0; rr < ROUNDS; ++rr) {
    const int q = rr * CPR + lane / L;
    const int w0 = lane % L;
    V v = V(0);
    if (q < NC) {
#pragma unroll
      for (int j = 0; j < PER; ++j) v += base[(w0 + j * L) * stride + q];
    }
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
#pragma unroll
    for (int c = 0; c < CPR; ++c)
      if (rr * CPR + c < NC) tot[rr * CPR + c] = __shfl_sync(0xffffffffu, v, c * L);
  }
}

}  // namespace amm
