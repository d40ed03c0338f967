// Batched power method: λ_max of C_b = A_b·A_bᵀ for many independent FP32 matrices of uneven
// sizes in ONE persistent launch (block power iteration with K vectors and Rayleigh–Ritz), and
// the batched backward ∂λ/∂A = 2·v(vᵀA).
//
// The reference handles one matrix per run (AMM.cu:74-95); this path batches the exact product
// of powerMethod_by_exact.cuh:37-53 with the Rayleigh step of dotProduct_and_generate_x
// (common.h:103-153) generalised to a block of K orthonormal vectors.
//
// Work split: one CTA (512 threads) per matrix at a time, matrices taken largest-first from an
// atomic queue.  A matrix of m rows is held by "teams" of P threads (P = smallest power of two
// >= m/4, at least 32), each thread owning 4 consecutive rows of the K vectors X and of the
// product Y in registers; the 512/P teams split the columns.  Per group of GC columns a team
// reads the columns once (coalesced 16-byte cp.async copies into a per-thread shared-memory
// ring that keeps two or more groups in flight), forms the K·GC partial dots A_jᵀX over its
// rows, reduces them across the team (warp butterfly, then shared memory for teams wider than a
// warp) and accumulates Y += A_j·(A_jᵀX): the fused single-pass product of the main kernel.
// Exact batches of 8 vectors take a tensor-core form of that product (TF32 mma.sync with a hi + lo
// split, column tiles copied by TMA; see batch_kernel) and, where it pays (plan_gram), go through
// C = A·Aᵀ, formed once per run on tcgen05 (amm_gram.cu), as C·X (cx_product).
// After the pass the team partials of Y are summed in a fixed order, the Gram matrices
// G = YᵀY and H = XᵀY are reduced in FP64, X <- Y·R⁻¹ (Cholesky QR), and every rr_period
// iterations (and at the end) H is diagonalised by a warp-parallel cyclic Jacobi in FP64: its
// largest eigenvalue is λ_max, its eigenvector q gives v = X·q.

#include <cooperative_groups.h>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <functional>
#include <queue>
#include <tuple>
#include <utility>
#include <vector>

#include "amm.h"
#include "amm_batch.h"
#include "amm_device.cuh"
#include "amm_internal.h"

namespace amm {
namespace batch {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxRows = 4 * kThreads;  // 2048
constexpr int kMaxK = 8;
constexpr int kJacobiSweeps = 16;

constexpr int kMaxCols = 8192;   // AMM mode: the CDF lives in shared memory
constexpr int kVrSlot = 3;       // VR scratch per CTA: X_memo, Y_memo, saved X
constexpr int kMaxPicks = 1024;  // AMM mode: c <= n / 8

struct Args {
  const Mat* mats;
  const int32_t* order;  // processing order (largest first), shared by the launches of a run
  int32_t count;
  int32_t max_iter;
  double tol;
  int32_t rr_period;
  int32_t count0;        // matrices of this launch's own list, taken before the shared one
  const int32_t* order0;
  uint64_t seed;
  uint32_t* states;  // AMM mode: xorshift32 states of every matrix (advanced in place)
  uint32_t* queue;  // [0]: next item of the shared list, [1]: of the own list; zero at the start
  double* lam;      // count x K Ritz values, descending ([0] = λ_max)
  float* vec;       // Σ m: v of each matrix (top Ritz vector, unit)
  int32_t* iters;   // iterations run (-1: rank-deficient block, no result)
  // AMM mode with variance reduction: product p is exact, and memoised, when
  // (p + 1) % vr_period == 0 and for the last product; the others estimate
  // C·X = Y_memo·S + Ĉ·(X − X_memo·S), S = X_memoᵀ·X (0: no variance reduction)
  int32_t vr_period;
  int32_t vr_base;   // first slot of this launch's CTAs in vr_mem (the second launch of a run
                     // is offset past the first one's CTAs)
  float* vr_mem;     // per CTA slot: X_memo, Y_memo, then X saved while a sampled product
                     // multiplies D in its place; kMaxRows x K floats each (see memo_load)
  // optional record for parity checks (null: none): each matrix's FP32 CDF at col_start[mi]
  // and the raw picks of its AMM product p < rec_products at st_off·rec_products + p·c + k
  float* rec_cdf;
  uint32_t* rec_picks;
  int32_t rec_products;
  const int64_t* col_start;
  // tensor-core kernel: one tensor map per matrix (FP32 {m rows, n columns}, 32 x 8 boxes,
  // 128-byte swizzle, zero fill outside the matrix), encoded on the host
  const CUtensorMap* tmaps;
  int32_t use_c;  // products as C·X where a matrix has its C (0: every product reads A)
};

// A shared-memory float4 load the compiler keeps in place (X is re-read per column group
// instead of being held in registers across the pass).
__device__ __forceinline__ float4 lds_f4(const float* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
  return v;
}

// Tensor-core product (exact mode, 8 vectors): X is stored [v][row] with a row stride of 2064
// floats (516 16-byte chunks, 4 mod 8: the 16-byte fragment loads of vector pairs land on
// disjoint banks).
constexpr int kXsStrideTC = kMaxRows + 16;

// Shared-memory position of X[row][v].  For an even block the vectors are interleaved in pairs
// ([v/2][row][2]) so that a thread's 4 rows of a vector pair are two 16-byte loads holding the
// float2 operands of the packed FMAs; the tensor-core kernel keeps [v][row].
template <int K, bool TC = false>
__device__ __forceinline__ int xs_idx(int v, int row) {
  if constexpr (TC)
    return v * kXsStrideTC + row;
  else if constexpr (K % 2 == 0)
    return (v >> 1) * (2 * kMaxRows) + row * 2 + (v & 1);
  else
    return v * kMaxRows + row;
}

// Shared-memory layout of Y (and of X by row): a thread's 4 rows x K vectors are K float4s (value
// e·K + v of row 4·slot + e in float4 (e·K + v) / 4), permuted by the slot so that 8 neighbouring
// threads' accesses of the same float4 fall on different banks (unpermuted, 128 bytes apart, they
// all fall on one).
template <int K>
__device__ __forceinline__ int yq(int slot, int i) {
  if constexpr (K == 8)
    return slot * 8 + (i ^ (slot & 7));
  else if constexpr (K == 4)
    return slot * 4 + (i ^ ((slot >> 1) & 3));
  else
    return slot * K + i;
}
// the same for one value (a float offset)
template <int K>
__device__ __forceinline__ int yat(int row, int v) {
  const int k = (row & 3) * K + v;
  return 4 * yq<K>(row >> 2, k >> 2) + (k & 3);
}
template <int K>
__device__ __forceinline__ void y_store(float* dst, int slot, const float (&Y)[4][K]) {
#pragma unroll
  for (int i = 0; i < K; ++i)
    reinterpret_cast<float4*>(dst)[yq<K>(slot, i)] =
        make_float4(Y[4 * i / K][4 * i % K], Y[(4 * i + 1) / K][(4 * i + 1) % K],
                    Y[(4 * i + 2) / K][(4 * i + 2) % K], Y[(4 * i + 3) / K][(4 * i + 3) % K]);
}
// Y = src (ADD: Y += src)
template <int K, bool ADD>
__device__ __forceinline__ void y_load(const float* src, int slot, float (&Y)[4][K]) {
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float4 v = reinterpret_cast<const float4*>(src)[yq<K>(slot, i)];
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float& y = Y[(4 * i + c) / K][(4 * i + c) % K];
      y = ADD ? y + w[c] : w[c];
    }
  }
}

// Start block: a counter-based hash of (seed, matrix, row, vector) -> uniform [-1, 1).
__device__ __forceinline__ float start_value(uint64_t seed, int mi, int row, int v) {
  uint64_t z = seed ^ (0x9E3779B97F4A7C15ull * (uint64_t)(mi + 1)) ^
               ((uint64_t)row << 20) ^ ((uint64_t)v << 52);
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (float)(int32_t)(uint32_t)(z >> 32) * (1.0f / 2147483648.0f);
}

// Pair (p, q), p < q, of slot s in round r of a round-robin over K (even) indices.
__device__ __forceinline__ void rr_pair(int K, int r, int s, int* p, int* q) {
  int a, b;
  if (s == 0) {
    a = K - 1;
    b = r;
  } else {
    a = (r + s) % (K - 1);
    b = (r - s + (K - 1)) % (K - 1);
  }
  *p = a < b ? a : b;
  *q = a < b ? b : a;
}

// The rotation (c, s) that annihilates h_pq: t = tan θ = sign(d)·b / (|d| + sqrt(d² + b²)), d = h_qq −
// h_pp, b = 2·h_pq, to FP32 accuracy from d and b scaled by an exact power of two (max(|d|, |b|) in
// [1, 2)); (c, s) = (1, t)/sqrt(1 + t²) in FP32, then two Newton steps x <- x·(3 − (c² + s²))/2 in FP64
// make the rotation orthogonal to FP64 rounding.  An angle off by FP32 rounding leaves h_pq at ~1e-7
// of its size instead of 0, which the next sweep removes; the eigenvalues depend only on the
// orthogonality.
__device__ __forceinline__ void jacobi_angle(double hpp, double hqq, double hpq, double* c,
                                             double* s) {
  const double dd = hqq - hpp, bb = 2.0 * hpq;
  const double mx = fmax(fabs(dd), fabs(bb));
  const int ex = (int)((__double_as_longlong(mx) >> 52) & 0x7ff);
  const double sc = __longlong_as_double((long long)(2046 - min(ex, 2045)) << 52);
  const float df = (float)(dd * sc), bf = (float)(bb * sc);
  const float tf = copysignf(1.f, df) * __fdividef(bf, fabsf(df) + sqrtf(fmaf(df, df, bf * bf)));
  const float cf = rsqrtf(fmaf(tf, tf, 1.f));
  double cc = (double)cf, ss = (double)(tf * cf);
#pragma unroll
  for (int nw = 0; nw < 2; ++nw) {
    const double f = fma(-0.5, fma(cc, cc, ss * ss), 1.5);
    cc *= f;
    ss *= f;
  }
  *c = hpq != 0.0 ? cc : 1.0;
  *s = hpq != 0.0 ? ss : 0.0;
}

// (a, b)·[c s; -s c], the rounding of each term stated: left to the compiler it would follow the code
// around it, and the blocks that sampled batches rotate can be singular to FP32 (see sampled_cluster)
__device__ __forceinline__ double rot_first(double c, double s, double a, double b) {
  return __fma_rn(c, a, -__dmul_rn(s, b));
}
__device__ __forceinline__ double rot_second(double c, double s, double a, double b) {
  return __fma_rn(s, a, __dmul_rn(c, b));
}

// Cyclic Jacobi on the symmetric K x K matrix H (FP64, shared memory) by one warp; V receives
// the eigenvectors (columns), H the eigenvalues on its diagonal.  The rotations of a round act on
// disjoint index pairs, so a round is applied at once: lane (a, b) holds the 2 x 2 block of H in
// rows of pair a and columns of pair b and rotates it from both sides; the lanes after those hold
// one row of V in two pairs each.  Every lane forms the two angles it needs itself, from entries
// loaded beside its block: a round is one shared-memory read, two interleaved angles, one write and
// two warp barriers.
template <int K>
__device__ void jacobi_warp(double* H, double* V, int lane) {
  __builtin_assume(__isShared(H));
  __builtin_assume(__isShared(V));
  for (int i = lane; i < K * K; i += 32) V[i] = (i / K == i % K) ? 1.0 : 0.0;
  __syncwarp();
  if constexpr (K > 1) {
    constexpr int NPR = K / 2;                      // pairs of a round
    constexpr int NH = NPR * NPR, NVL = K * NPR / 2;  // lanes on H and on V
    const bool on_h = lane < NH, act = lane < NH + NVL;
    const int vl = on_h ? 0 : (lane - NH) % NVL;  // (idle lanes repeat one that is not)
    const int row = vl % K;                          // lanes on V: the row
    const int sa = on_h ? lane / NPR : 2 * (vl / K) % NPR;
    const int sb = on_h ? lane % NPR : (2 * (vl / K) + 1) % NPR;
    // the pairs of slots sa and sb in every round, four bits an index (rounds 0-3, then 4-6)
    unsigned long long pairs_lo = 0, pairs_hi = 0;
#pragma unroll
    for (int r = 0; r < K - 1; ++r) {
      int pa, qa, pb, qb;
      rr_pair(K, r, sa, &pa, &qa);
      rr_pair(K, r, sb, &pb, &qb);
      const unsigned long long w = (unsigned long long)(pa | qa << 4 | pb << 8 | qb << 12)
                                   << (16 * (r & 3));
      if (r < 4)
        pairs_lo |= w;
      else
        pairs_hi |= w;
    }
#pragma unroll 1
    for (int sweep = 0; sweep < kJacobiSweeps; ++sweep) {
      double off = 0.0, dia = 0.0;
#pragma unroll
      for (int i = lane; i < K * K; i += 32) {
        const double h = H[i];
        if (i / K == i % K)
          dia += h * h;
        else
          off += h * h;
      }
      off = warp_sum(off);
      dia = warp_sum(dia);
      // off-diagonal entries below ~1e-13 of the matrix: the eigenvalue error left is their
      // square over the gap (the FP64 rounding floor of `off` is ~K²·eps²·dia, so a tighter test
      // would never be met and run every sweep); also stops on NaN
      if (!__any_sync(0xffffffffu, off > 1e-26 * dia)) break;  // (the same in every lane)
#pragma unroll 1
      for (int r = 0; r < K - 1; ++r) {
        const uint32_t pr = (uint32_t)((r < 4 ? pairs_lo : pairs_hi) >> (16 * (r & 3)));
        const int pa = pr & 15, qa = pr >> 4 & 15, pb = pr >> 8 & 15, qb = pr >> 12 & 15;
        double* const B = on_h ? H : V;
        __builtin_assume(__isShared(B));
        const int i00 = (on_h ? pa * K + pb : row * K + pa), i01 = (on_h ? pa * K + qb : row * K + qa);
        const int i10 = (on_h ? qa * K + pb : row * K + pb), i11 = (on_h ? qa * K + qb : row * K + qb);
        const double e00 = B[i00], e01 = B[i01], e10 = B[i10], e11 = B[i11];
        double ca, sna, cb, snb;
        jacobi_angle(H[pa * K + pa], H[qa * K + qa], H[pa * K + qa], &ca, &sna);
        jacobi_angle(H[pb * K + pb], H[qb * K + qb], H[pb * K + qb], &cb, &snb);
        __syncwarp();
        // H: columns by pair b, then rows by pair a (Jᵀ·H·J); V: (e00, e01) by pair a, (e10, e11) by
        // pair b.  Selects, no branch: lanes that part here stay parted for the rounds that follow
        const double c0 = on_h ? cb : ca, s0 = on_h ? snb : sna;
        const double cr = on_h ? ca : 1.0, sr = on_h ? sna : 0.0;
        const double t00 = rot_first(c0, s0, e00, e01), t01 = rot_second(c0, s0, e00, e01);
        const double t10 = rot_first(cb, snb, e10, e11), t11 = rot_second(cb, snb, e10, e11);
        if (act) {
          B[i00] = rot_first(cr, sr, t00, t10);
          B[i01] = rot_first(cr, sr, t01, t11);
          B[i10] = rot_second(cr, sr, t00, t10);
          B[i11] = rot_second(cr, sr, t01, t11);
        }
        __syncwarp();
      }
    }
  }
}

constexpr int align16(int x) { return (x + 15) & ~15; }
constexpr int align1024(int x) { return (x + 1023) & ~1023; }
constexpr int cmax(int a, int b) { return a > b ? a : b; }

// The column ring of the product pass: every thread copies its own 16 bytes of each column of
// a group (cp.async, no register staging) RingStages<GC> groups ahead and reads back only what it
// copied, so the ring needs no barrier.  96 KB: 64 KB in flight per SM at NST = 3.
constexpr int kRingBytes = 96 * 1024;
template <int GC>
struct Ring {
  static constexpr int stages = kRingBytes / (kThreads * GC * 16);
};

// Tensor-core product: per warp and stage, 8 columns x 128 rows (4 KB, four 32 x 8 TMA boxes);
// two stages.
constexpr int kTcCols = 8;
constexpr int kTcWarpFloats = kTcCols * 128;
constexpr int kTcStageFloats = kWarps * kTcWarpFloats;

template <int K, bool TC = false>
struct Smem {
  // byte offsets into dynamic shared memory, each 16-byte aligned
  static constexpr int part = 0;                  // float [2][kWarps][32] (TC: float2 per lane)
  static constexpr int bcast = align16(part + 2 * kWarps * 32 * 4 * (TC ? 2 : 1));
                                                                         // float [kWarps][32]
  static constexpr int gpart = align16(bcast + kWarps * 32 * 4);         // double [kWarps][2*K*K]
  static constexpr int gram = align16(gpart + kWarps * 2 * K * K * 8);   // double G[K*K], H[K*K]
  static constexpr int vmat = align16(gram + 2 * K * K * 8);             // double V[K*K]
  static constexpr int rinv = align16(vmat + K * K * 8);                 // float Rinv[K*K]
  static constexpr int qv = align16(rinv + K * K * 4);                   // float q[K]
  static constexpr int ritz = align16(qv + K * 4);                       // double θ[K], λ
  static constexpr int ctl = align16(ritz + (kMaxK + 1) * 8);            // int [4]
  static constexpr int tbar = align16(ctl + 16);  // uint64 [kWarps][2]: tensor-core tile copies
  static constexpr int xs = align16(tbar + kWarps * 2 * 8);              // float X[K][kMaxRows]
  static constexpr int xs_bytes = K * (TC ? kXsStrideTC : kMaxRows) * 4;
  // one region used in turn by: the column ring (tensor-core kernel: the tiles) during a product pass, or
  // the threads' run sums and X by row during a product through C; the team partials of Y after it, and
  // Y for the Gram sums (yred); the pick histogram of an AMM draw (hist, zeroed at the start of
  // every draw)
  // (tensor-core kernel: 1024-byte aligned, as the 128-byte swizzle of its tile copies needs)
  static constexpr int region = TC ? align1024(xs + xs_bytes) : align16(xs + xs_bytes);
  static constexpr int yred = region;                                    // float [4*kThreads][K]
  static constexpr int hist = align16(yred + 4 * kThreads * K * 4);      // uint32 [kMaxCols]
  static constexpr int xrow = hist;  // tensor-core kernel, a matrix multiplied as C·X: X by row (yq)
  static constexpr int region_bytes =
      TC ? cmax(2 * kTcStageFloats * 4, 4 * kThreads * K * 4)
         : cmax(hist + kMaxCols * 4 - region, kRingBytes);
  static constexpr int total = align16(region + region_bytes);           // exact mode ends here
  static constexpr int cdf = total;                                      // float [kMaxCols]
  static constexpr int lcol = align16(cdf + kMaxCols * 4);               // int32 [kMaxPicks]
  static constexpr int lw = align16(lcol + kMaxPicks * 4);             // float [kMaxPicks]
  static constexpr int scan = align16(lw + kMaxPicks * 4);             // uint32 [40], double[32]
  static constexpr int svr = align16(scan + 40 * 4 + 32 * 8);           // float S[K*K] (VR)
  static constexpr int total_amm = align16(svr + K * K * 4);
  static_assert(gpart % 8 == 0 && ritz % 8 == 0 && xs % 16 == 0 && region % 16 == 0,
                "shared-memory alignment");
  static_assert(!TC || xrow + kMaxRows * K * 4 <= region + region_bytes, "X by row fits the region");
  static_assert(!TC || total <= 227 * 1024, "the tensor-core layout exceeds a CTA's shared memory");
};

// One m16n8k8 TF32 tensor-core product D += A·B (FP32 accumulators), fragments as in the PTX
// ISA: lane = 4·g + t holds A(g, t), A(g+8, t), A(g, t+4), A(g+8, t+4), B(t, g), B(t+4, g) and
// D(g, 2t), D(g, 2t+1), D(g+8, 2t), D(g+8, 2t+1).
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, "
      "{%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// x = hi + lo with hi x rounded to TF32 (11 significant bits, to nearest, ties away: add half
// an ulp of TF32 to the bit pattern, then clear the 13 low bits) and lo = x - hi, exact in
// FP32; the tensor core reads lo to 11 bits, so hi + lo carries x to about 2^-21 relative.
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
  const uint32_t h = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  hi = h;
  lo = __float_as_uint(x - __uint_as_float(h));
}


// Sum of the NV values d over the team (P threads).  Returns, in every lane, the total of value
// lane / (32 / NV); the caller gathers value i from lane i·(32 / NV).  Fixed reduction order
// (deterministic).
template <int NV>
__device__ __forceinline__ float team_allreduce(float (&d)[NV], float* part, int buf, int warp,
                                                int lane, int P, int team, int team_warp0) {
  float r = warp_reduce_multi<float, NV>(d, lane);
  if (P > 32) {
    float* pb = part + buf * kWarps * 32;
    pb[warp * 32 + lane] = r;
    named_barrier_or(1 + team, P, false);
    float s = 0.f;
    for (int w = 0; w < P / 32; ++w) s += pb[(team_warp0 + w) * 32 + lane];
    r = s;
  }
  return r;
}

// Rayleigh–Ritz (every rr_period steps and at the end) and the next basis, by warp 0; kept out
// of line so that its FP64 scratch does not compete for registers with the product loop.
// H = XᵀCX is diagonalised (θ, V); λ = max θ, its Ritz vector v = X·q (q and the sorted θ go
// to shared memory for the residual test the whole CTA runs next).  The next basis is
// X <- Y·M, M = V·L⁻ᵀ with L·Lᵀ = VᵀGV: Cholesky QR of the block rotated into the Ritz basis,
// so the next H is nearly diagonal and the Jacobi sweeps are few.  ctl[1]: 0 go on, 2 failed
// (rank-deficient block or a non-finite λ); ctl[2]: a Ritz pair was formed.
template <int K>
__device__ __noinline__ void ritz_step(const Args& a, int mi, int it, double* Gm, double* Hm,
                                       double* Vm, double* ritz, float* Rinv, float* qv, int* ctl,
                                       double* scratch, int lane, bool writer, bool force_rr) {
  __builtin_assume(__isShared(Gm));
  __builtin_assume(__isShared(Hm));
  __builtin_assume(__isShared(Vm));
  __builtin_assume(__isShared(scratch));
  __builtin_assume(__isShared(ritz));
  __builtin_assume(__isShared(Rinv));
  const bool first = (it == 0);
  const bool rr = !first && ((K == 1) || ((it % a.rr_period) == 0) || (it >= a.max_iter) ||
                             force_rr);
  if (rr) jacobi_warp<K>(Hm, Vm, lane);
  // the Ritz values, descending: lane i < K places its own by its rank (ties in index order); the
  // first of the largest gives λ and its vector
  int st = 0;
  if (rr) {
    double mine = lane < K ? Hm[lane * K + lane] : 0.0;
    int rank = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const double o = __shfl_sync(0xffffffffu, mine, j);
      rank += (o > mine || (o == mine && j < lane)) ? 1 : 0;
    }
    // (a NaN ranks against nothing: such a block is reported below, whatever its order)
    if (!isfinite(mine)) rank = lane < K ? lane : 0;
    const uint32_t top = __ballot_sync(0xffffffffu, lane < K && rank == 0);
    const int best = top ? __ffs(top) - 1 : 0;
    const double lam = __shfl_sync(0xffffffffu, mine, best);
    if (lane < K) {
      ritz[rank] = mine;
      qv[lane] = (float)Vm[lane * K + best];
    }
    if (lane == 0) ritz[kMaxK] = lam;
    if (__any_sync(0xffffffffu, lane < K && !isfinite(mine))) st = 2;
  }
  if (lane == 0) ctl[2] = rr ? 1 : 0;
  // The next basis, by the whole warp; each entry is summed in the order of a sequential loop.
  double* Gp = scratch;              // VᵀGV (or G)
  double* T = scratch + K * K;       // G·V
  double* Li = scratch + 3 * K * K;  // L⁻¹ (lower)
  if (st == 0) {
    if (rr) {
#pragma unroll
      for (int idx = lane; idx < K * K; idx += 32) {
        const int i = idx / K, j = idx % K;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < K; ++k) acc += Gm[i * K + k] * Vm[k * K + j];
        T[idx] = acc;
      }
      __syncwarp();
#pragma unroll
      for (int idx = lane; idx < K * K; idx += 32) {
        const int i = idx / K, j = idx % K;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < K; ++k) acc += Vm[k * K + i] * T[k * K + j];
        Gp[idx] = acc;
      }
    } else {
      for (int idx = lane; idx < K * K; idx += 32) Gp[idx] = Gm[idx];
    }
    __syncwarp();
    double tr = 0.0;
#pragma unroll
    for (int i = 0; i < K; ++i) tr += Gp[i * K + i];
    bool ok = tr > 0.0 && isfinite(tr);
    // Cholesky L·Lᵀ = Gp in registers, lane i < K holding row i: per column one reciprocal square root
    // gives both L_jj = d·d^(-1/2) and 1/L_jj, so no step divides
    double l[K], ri[K];
#pragma unroll
    for (int k = 0; k < K; ++k) l[k] = lane < K ? Gp[lane * K + k] : 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const double d = __shfl_sync(0xffffffffu, l[j], j);
      const bool good = d > 1e-24 * tr;
      ok = ok && good;
      ri[j] = good ? rsqrt(d) : 0.0;
      l[j] = l[j] * ri[j];
#pragma unroll
      for (int k = j + 1; k < K; ++k) l[k] -= l[j] * __shfl_sync(0xffffffffu, l[j], k);
    }
    if (!ok) {  // rank-deficient block: no result for this matrix
      st = 2;
    } else {
      // L⁻¹, column j by lane j (forward substitution)
      double x[K];
#pragma unroll
      for (int i = 0; i < K; ++i) {
        double sv = 0.0;
#pragma unroll
        for (int k = 0; k < i; ++k) sv += __shfl_sync(0xffffffffu, l[k], i) * x[k];
        x[i] = i < lane ? 0.0 : i == lane ? ri[i] : -sv * ri[i];
      }
      if (lane < K) {
#pragma unroll
        for (int i = 0; i < K; ++i) Li[i * K + lane] = x[i];
      }
      __syncwarp();
      // M = V·L⁻ᵀ (or L⁻ᵀ without a rotation); (L⁻ᵀ)[k][j] = Li[j][k], zero for k > j
#pragma unroll
      for (int idx = lane; idx < K * K; idx += 32) {
        const int i = idx / K, j = idx % K;
        double sv = 0.0;
        if (rr) {
#pragma unroll
          for (int k = 0; k < K; ++k) sv += Vm[i * K + k] * Li[j * K + k];
        } else {
          sv = (i <= j) ? Li[j * K + i] : 0.0;
        }
        Rinv[i * K + j] = (float)sv;
      }
    }
  }
  if (lane == 0) {
    if (st == 2 && writer) {
      for (int i = 0; i < K; ++i) a.lam[(int64_t)mi * K + i] = nan("");
      a.iters[mi] = -1;
    }
    ctl[1] = st;
  }
  __syncwarp();
}

// ---- variance reduction helpers, out of line so that their registers do not compete with the
// product loop's ----
// S = X_memoᵀ·X (FP64 sums over team 0's rows, into Svr) and D = X − X_memo·S in place of X
// (X saved to Xsave, restored by vr_add_memo after the product); called by every thread of the CTA.
// The memo slots hold a thread's 4 rows as K float4s, float4 i of thread t at i·kThreads + t: every
// access is coalesced, and every thread reads back only what it wrote.  The sums of S: over a
// thread's 4 rows in turn, then a butterfly over the warp (K entries of S at a time), then over team 0's
// warps in turn.
template <int K>
__device__ __forceinline__ void memo_load(const float* p, int t, float (&v)[4][K]) {
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const float4 q = reinterpret_cast<const float4*>(p)[i * kThreads + t];
    const float w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) v[(4 * i + c) / K][(4 * i + c) % K] = w[c];
  }
}
template <int K>
__device__ __forceinline__ void memo_store(float* p, int t, const float (&v)[4][K]) {
#pragma unroll
  for (int i = 0; i < K; ++i)
    reinterpret_cast<float4*>(p)[i * kThreads + t] =
        make_float4(v[4 * i / K][4 * i % K], v[(4 * i + 1) / K][(4 * i + 1) % K],
                    v[(4 * i + 2) / K][(4 * i + 2) % K], v[(4 * i + 3) / K][(4 * i + 3) % K]);
}
template <int K>
__device__ __noinline__ void vr_difference(const float* Xm, float* Xs, float* Xsave, double* gpart,
                                           float* Svr, int P, int r0, int t, int warp, int lane,
                                           int team) {
  const int tw = P / 32;  // warps of team 0
  float xm[4][K];
  if (team == 0) {  // warp-uniform
    memo_load<K>(Xm, t, xm);
#pragma unroll 1
    for (int vb = 0; vb < K; ++vb) {
      double x[4], d[K];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = (double)Xs[xs_idx<K>(vb, r0 + e)];
#pragma unroll
      for (int va = 0; va < K; ++va) {
        d[va] = 0.0;
#pragma unroll
        for (int e = 0; e < 4; ++e) d[va] = fma((double)xm[e][va], x[e], d[va]);
      }
      const double r = warp_reduce_multi<double, K>(d, lane);  // value lane / (32 / K)
      if (lane % (32 / K) == 0) gpart[warp * K * K + lane / (32 / K) * K + vb] = r;
    }
  }
  __syncthreads();
  if (t < K * K) {
    double sv = 0.0;
    for (int w = 0; w < tw; ++w) sv += gpart[w * K * K + t];
    Svr[t] = (float)sv;
  }
  __syncthreads();
  if (team == 0) {
    float x[4][K];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int vb = 0; vb < K; ++vb) x[e][vb] = Xs[xs_idx<K>(vb, r0 + e)];
    memo_store<K>(Xsave, t, x);
#pragma unroll
    for (int vb = 0; vb < K; ++vb) {
      float sc[K];
#pragma unroll
      for (int va = 0; va < K; ++va) sc[va] = Svr[va * K + vb];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float d = x[e][vb];
#pragma unroll
        for (int va = 0; va < K; ++va) d = fmaf(-xm[e][va], sc[va], d);
        Xs[xs_idx<K>(vb, r0 + e)] = d;  // this thread alone reads and writes its rows here
      }
    }
  }
  __syncthreads();
}

// Y += Y_memo·S over this thread's rows (Y at Yp, laid out as the memo slots), and X back in place of
// D (team 0, once no team multiplies any more).
template <int K>
__device__ __noinline__ void vr_add_memo(float* Yp, const float* Ym, const float* Svr,
                                         const float* Xsave, float* Xs, int r0, int t) {
  float v4[4][K], Y[4][K];
  memo_load<K>(Xsave, t, v4);
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int v = 0; v < K; ++v) Xs[xs_idx<K>(v, r0 + e)] = v4[e][v];
  memo_load<K>(Ym, t, v4);
  memo_load<K>(Yp, t, Y);
#pragma unroll
  for (int vb = 0; vb < K; ++vb) {
    float sc[K];
#pragma unroll
    for (int va = 0; va < K; ++va) sc[va] = Svr[va * K + vb];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float acc = Y[e][vb];
#pragma unroll
      for (int va = 0; va < K; ++va) acc = fmaf(v4[e][va], sc[va], acc);
      Y[e][vb] = acc;
    }
  }
  memo_store<K>(Yp, t, Y);
}

// X_memo <- X over this thread's rows (team 0).
template <int K>
__device__ __noinline__ void vr_store_memo(float* Xm, const float* Xs, int r0, int t) {
  float x[4][K];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int v = 0; v < K; ++v) x[e][v] = Xs[xs_idx<K>(v, r0 + e)];
  memo_store<K>(Xm, t, x);
}

// One FP64 tensor-core product D += A·B (m8n8k4, FP64 accumulation), fragments as in the PTX
// ISA: lane = 4·g + t holds A(g, t), B(t, g), D(g, 2t) and D(g, 2t+1).
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// Gram matrices of the block, G = YᵀY and H = sym(XᵀY), in FP64 over team 0's rows (the only
// team holding the summed Y, here in shared memory as Ys, see yq); called by every thread of the
// CTA.  For 8 vectors each warp of team 0 multiplies its 128 rows on the FP64 tensor cores: per
// 4 rows one m8n8k4 product for G (A = Yᵀ, B = Y: lane 4·g + t supplies Y[row t][vector g] to
// both) and one for XᵀY (A = Xᵀ); FP32 × FP32 products are exact in FP64.  For fewer vectors
// each thread forms its FP64 partials over its 4 rows, 8 entries at a time, summed over the warp
// by one multi-value butterfly per 8 entries.  The team's warps are then summed in a fixed
// order.  Kept out of line so that its registers do not compete with the product loop's.
template <int K, bool TC>
__device__ __noinline__ void gram_step(const float* Xs, const float* Ys, double* gpart,
                                       double* Gm, double* Hm, int P, int r0, int t, int warp,
                                       int lane, int team) {
  constexpr int NP = K * (K + 1) / 2;
  const int tw = P / 32;  // warps of team 0
  if constexpr (K == 8) {
    // gpart[warp][0..63]: this warp's G (row-major), [64..127]: its XᵀY
    if (team == 0) {  // warp-uniform (P >= 32)
      __syncwarp();   // the warp's rows of Ys were written by its own lanes
      double dg[2] = {0.0, 0.0}, dh[2] = {0.0, 0.0};
      const int g = lane >> 2, tq = lane & 3;
      const int rb = 128 * warp;  // team 0's warp w holds rows [128w, 128w + 128)
#pragma unroll 4
      for (int k = 0; k < 32; ++k) {
        const int row = rb + 4 * k + tq;
        const double y = (double)Ys[yat<K>(row, g)];
        const double x = (double)Xs[xs_idx<K, TC>(g, row)];
        mma_f64(dg, y, y);
        mma_f64(dh, x, y);
      }
      double* gp = gpart + warp * 2 * K * K;
      gp[g * K + 2 * tq] = dg[0];
      gp[g * K + 2 * tq + 1] = dg[1];
      gp[K * K + g * K + 2 * tq] = dh[0];
      gp[K * K + g * K + 2 * tq + 1] = dh[1];
    }
    __syncthreads();
    if (t < 2 * NP) {
      const int which = t / NP, pi = t % NP;
      int a1 = 0, rem = pi;
      while (rem >= K - a1) {
        rem -= K - a1;
        ++a1;
      }
      const int b1 = a1 + rem;
      double s = 0.0;
      if (which == 0) {
        for (int w = 0; w < tw; ++w) s += gpart[w * 2 * K * K + a1 * K + b1];
      } else {
        double sa = 0.0, sb = 0.0;
        for (int w = 0; w < tw; ++w) {
          sa += gpart[w * 2 * K * K + K * K + a1 * K + b1];
          sb += gpart[w * 2 * K * K + K * K + b1 * K + a1];
        }
        s = 0.5 * (sa + sb);
      }
      double* D = which ? Hm : Gm;
      D[a1 * K + b1] = s;
      D[b1 * K + a1] = s;
    }
    __syncthreads();
  } else {
    constexpr int NV2 = 2 * NP;        // G entries (pair index), then H entries
    constexpr int NB = (NV2 + 7) / 8;  // batches of 8 entries
    if (team == 0) {                   // warp-uniform (P >= 32)
      float y[4][K];
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int v = 0; v < K; ++v) y[e][v] = Ys[yat<K>(r0 + e, v)];
#pragma unroll
      for (int bt = 0; bt < NB; ++bt) {
        double d[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) d[i] = 0.0;
        int pidx = 0;
#pragma unroll
        for (int a0 = 0; a0 < K; ++a0)
#pragma unroll
          for (int b0 = a0; b0 < K; ++b0, ++pidx) {
            if (pidx / 8 == bt) {
              double gg = 0.0;
#pragma unroll
              for (int e = 0; e < 4; ++e) gg = fma((double)y[e][a0], (double)y[e][b0], gg);
              d[pidx % 8] = gg;
            }
            if ((NP + pidx) / 8 == bt) {
              double h = 0.0;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float xa = Xs[xs_idx<K, TC>(a0, r0 + e)];
                const float xb = Xs[xs_idx<K, TC>(b0, r0 + e)];
                h = fma(0.5 * (double)xa, (double)y[e][b0], h);
                h = fma(0.5 * (double)xb, (double)y[e][a0], h);
              }
              d[(NP + pidx) % 8] = h;
            }
          }
        const double r = warp_reduce_multi<double, 8>(d, lane);  // entry 8·bt + lane/4
        const int vi = bt * 8 + (lane >> 2);
        if ((lane & 3) == 0 && vi < NV2) gpart[warp * NV2 + vi] = r;
      }
    }
    __syncthreads();
    if (t < NV2) {
      double s = 0.0;
      for (int w = 0; w < tw; ++w) s += gpart[w * NV2 + t];
      const int which = t / NP, pi = t % NP;
      int a1 = 0, rem = pi;
      while (rem >= K - a1) {
        rem -= K - a1;
        ++a1;
      }
      const int b1 = a1 + rem;
      double* D = which ? Hm : Gm;
      D[a1 * K + b1] = s;
      D[b1 * K + a1] = s;
    }
    __syncthreads();
  }
}

// Y = C·X over this team's share of C's columns (C = A·Aᵀ, ldc x ldc, zeros past m), this thread's
// rows r0 .. r0 + 3: per column one 16-byte load of C (coalesced over the team, four columns ahead in
// registers) against X's row (broadcast loads from `xrow`, see yq), in packed FP32 FMAs.  Bounded by the
// FMAs and by an SM's share of the L2 (16 packed FMAs per 16 bytes).  The sums are taken in runs of 16
// columns, added up in this thread's slot of shared memory (`slots`, [value / 4][thread]): one FP32 chain
// over a team's whole share made the rounding of Y the largest error of λ where the eigenvector sits on
// few rows (300 x 700 with lognormal row scales: rms 1.6e-7 -> 1.2e-7).  Out of line so that its
// registers do not compete with the other product loops'.
template <int K>
__device__ __noinline__ void cx_product(const float* __restrict__ C, int ldc, const float* xrow,
                                        float4* slots, int r0, int g0, int gstep) {
  constexpr int KP = K / 2;
  float2 run[4][KP];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int p = 0; p < KP; ++p) run[e][p] = make_float2(0.f, 0.f);
  const int ng = ldc >> 2;  // groups of 4 columns
  const float* base = C + r0;
  float4 c[4], cn[4];
  auto load = [&](int g, float4 (&o)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o[j] = __ldg(reinterpret_cast<const float4*>(base + (int64_t)(4 * g + j) * ldc));
  };
  bool some = false;  // the slot holds earlier runs
  float4* slot = slots + threadIdx.x;
  auto add_slot = [&]() {  // run += slot
    if (some)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int p = 0; p < KP; p += 2) {
          const float4 v = slot[(e * KP + p) / 2 * kThreads];
          run[e][p] = __fadd2_rn(run[e][p], make_float2(v.x, v.y));
          run[e][p + 1] = __fadd2_rn(run[e][p + 1], make_float2(v.z, v.w));
        }
  };
  if (r0 < ldc && g0 < ng) {
    load(g0, cn);
    int left = 4;  // groups of the run
#pragma unroll 1
    for (int g = g0; g < ng; g += gstep) {
#pragma unroll
      for (int j = 0; j < 4; ++j) c[j] = cn[j];
      if (g + gstep < ng) load(g + gstep, cn);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 x[KP];
#pragma unroll
        for (int p = 0; p < KP; p += 2) {
          const float4 v = reinterpret_cast<const float4*>(xrow)[yq<K>(g, j * (K / 4) + p / 2)];
          x[p] = make_float2(v.x, v.y);
          x[p + 1] = make_float2(v.z, v.w);
        }
        const float ce[4] = {c[j].x, c[j].y, c[j].z, c[j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 d = make_float2(ce[e], ce[e]);
#pragma unroll
          for (int p = 0; p < KP; ++p) run[e][p] = __ffma2_rn(d, x[p], run[e][p]);
        }
      }
      if (--left == 0 && g + gstep < ng) {
        add_slot();
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int p = 0; p < KP; p += 2) {
            slot[(e * KP + p) / 2 * kThreads] =
                make_float4(run[e][p].x, run[e][p].y, run[e][p + 1].x, run[e][p + 1].y);
            run[e][p] = run[e][p + 1] = make_float2(0.f, 0.f);
          }
        some = true;
        left = 4;
      }
    }
    add_slot();
  }
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int p = 0; p < KP; p += 2)
      slot[(e * KP + p) / 2 * kThreads] =
          make_float4(run[e][p].x, run[e][p].y, run[e][p + 1].x, run[e][p + 1].y);
}

template <int K, int GC, bool TC = false>
__global__ void __launch_bounds__(kThreads, 1) batch_kernel(const __grid_constant__ Args a) {
  constexpr int NV = K * GC;
  static_assert(TC || (NV <= 32 && (32 % NV) == 0), "K*GC must divide 32");
  static_assert(!TC || (K == 8 && GC == kTcCols), "the tensor-core product runs 8 vectors");
  using SL = Smem<K, TC>;
  extern __shared__ __align__(16) unsigned char smem[];
  float* yred = reinterpret_cast<float*>(smem + SL::yred);
  float* part = reinterpret_cast<float*>(smem + SL::part);
  float* bcast = reinterpret_cast<float*>(smem + SL::bcast);
  double* gpart = reinterpret_cast<double*>(smem + SL::gpart);
  double* Gm = reinterpret_cast<double*>(smem + SL::gram);
  double* Hm = Gm + K * K;
  double* Vm = reinterpret_cast<double*>(smem + SL::vmat);
  float* Rinv = reinterpret_cast<float*>(smem + SL::rinv);
  float* qv = reinterpret_cast<float*>(smem + SL::qv);
  double* ritz = reinterpret_cast<double*>(smem + SL::ritz);
  int* ctl = reinterpret_cast<int*>(smem + SL::ctl);
  float* Xs = reinterpret_cast<float*>(smem + SL::xs);  // X, one copy for all teams: [v][row]
  float* cdf = reinterpret_cast<float*>(smem + SL::cdf);
  uint32_t* hist = reinterpret_cast<uint32_t*>(smem + SL::hist);
  int32_t* lcol = reinterpret_cast<int32_t*>(smem + SL::lcol);
  float* lw = reinterpret_cast<float*>(smem + SL::lw);
  uint32_t* scan = reinterpret_cast<uint32_t*>(smem + SL::scan);
  double* dscan = reinterpret_cast<double*>(smem + SL::scan + 40 * 4);
  float* Svr = reinterpret_cast<float*>(smem + SL::svr);
  uint64_t* tbar = reinterpret_cast<uint64_t*>(smem + SL::tbar);

  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = (int)cluster.num_blocks();   // CTAs sharing one matrix
  const int crank = (int)cluster.block_rank();
  const bool writer = (crank == 0);           // rank 0 writes the results
  // tensor-core kernel: the warps' stage barriers of the tile copies (one arrival each: the
  // issuing lane's expect_tx).  The tiles' 128-byte swizzle is laid out for a 1024-byte aligned
  // region (true of a kernel without static shared memory); were it not, no copy is issued and
  // every matrix is reported without a result.
  uint32_t tph = 0;         // phase parity of this warp's two stages (alike in every lane)
  // no more copies in this warp (misaligned region, or a copy that timed out: the warp then
  // neither issues nor waits, so that later waits cannot time out one after another)
  bool tdead = TC && (smem_addr(smem + SL::region) & 1023u) != 0u;
  bool tfail = tdead;       // this pass's product is not to be trusted
  int tfail_mi = -1;        // the matrix of this CTA that gets no result for that reason
  if constexpr (TC) {
    if (t == 0) {
      for (int i = 0; i < 2 * kWarps; ++i) mbar_init(&tbar[i], 1);
      fence_barrier_init();
    }
    __syncthreads();
  }
  // the failure record, written once the cluster is done with the matrix (after the cluster
  // barrier of the next fetch), so that no result write of a peer comes after it
  auto record_tfail = [&]() {
    if (TC && tfail_mi >= 0 && t == 0) {
      for (int i = 0; i < K; ++i) a.lam[(int64_t)tfail_mi * K + i] = nan("");
      a.iters[tfail_mi] = -1;
    }
    tfail_mi = -1;
  };
  // a launch queued behind this one as a programmatic dependent may now take the SMs left
  griddep_launch_dependents();
  for (;;) {
    // rank 0 takes the next matrix, from this launch's own list first, then from the list it
    // shares with the other launch of the run; the cluster reads it from rank 0
    if (writer && t == 0) {
      int next = -1;
      if (a.count0 > 0) {
        const uint32_t k = atomicAdd(a.queue + 1, 1u);
        if (k < (uint32_t)a.count0) next = a.order0[k];
      }
      if (next < 0) {
        const uint32_t k = atomicAdd(a.queue, 1u);
        if (k < (uint32_t)a.count) next = a.order[k];
      }
      ctl[0] = next;
    }
    cluster.sync();
    const int mi = *cluster.map_shared_rank(&ctl[0], 0);
    cluster.sync();
    record_tfail();
    if (mi < 0) {
      // a launch queued behind another (programmatic dependent) ends only after it, so that
      // the work after it in the stream sees both; returns at once in any other launch
      griddep_wait();
      return;
    }
    const Mat M = a.mats[mi];
    const int m = M.m, n = M.n;
    int P = 32;
    while (P < kThreads && 4 * P < m) P <<= 1;
    const int NT = kThreads / P;
    const int team = t / P, tl = t % P;
    const int NTG = CL * NT;             // teams of the whole cluster split the columns
    const int gteam = crank * NT + team;
    const int team_warp0 = team * (P / 32);
    const int r0 = 4 * tl;
    const bool amm = !TC && M.c > 0;  // the tensor-core kernel runs exact batches only
    double total = 0.0;
    if (amm) {
      // ---- column norms² (get_norms, device_memory.h:34-59) into cdf[], then the CDF ----
      int buf = 0;
      for (int g0 = gteam * GC; g0 < n; g0 += NTG * GC, buf ^= 1) {
        float d[GC];
#pragma unroll
        for (int c = 0; c < GC; ++c) {
          float4 av = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r0 < m && g0 + c < n)
            av = __ldg(reinterpret_cast<const float4*>(M.A + r0 + (int64_t)(g0 + c) * M.ld));
          if (r0 + 1 >= m) av.y = 0.f;
          if (r0 + 2 >= m) av.z = 0.f;
          if (r0 + 3 >= m) av.w = 0.f;
          d[c] = fmaf(av.x, av.x, fmaf(av.y, av.y, fmaf(av.z, av.z, av.w * av.w)));
        }
        const float red = team_allreduce<GC>(d, part, buf, warp, lane, P, team, team_warp0);
        if (tl < GC * (32 / GC) && (lane % (32 / GC)) == 0) {
          const int c = lane / (32 / GC);
          if (g0 + c < n) cdf[g0 + c] = red;
        }
      }
      if (CL > 1) {  // norms of the columns the other CTAs of the cluster own
        cluster.sync();
        for (int j = t; j < n; j += kThreads) {
          const int owner = ((j / GC) % NTG) / NT;
          if (owner != crank) cdf[j] = *cluster.map_shared_rank(&cdf[j], owner);
        }
        cluster.sync();  // nobody overwrites its norms before every CTA has gathered
      }
      __syncthreads();
      // inclusive prefix in FP64, stored as FP32 (set_weights / CUB scan, common.h:34-40 and
      // powerMethod_by_previous.cuh:26-32); each thread owns a run of consecutive columns
      const int per = (n + kThreads - 1) / kThreads;
      const int j0 = t * per, j1 = min(n, j0 + per);
      double run = 0.0;
      for (int j = j0; j < j1; ++j) run += (double)cdf[j];
      // block exclusive scan of the run totals (FP64, fixed order)
      double incl = run;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) dscan[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        double w = lane < kWarps ? dscan[lane] : 0.0;
        double wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(0xffffffffu, wi, o);
          if (lane >= o) wi += y;
        }
        if (lane < kWarps) dscan[lane] = wi - w;
        if (lane == 31) dscan[kWarps] = wi;
      }
      __syncthreads();
      double pre = dscan[warp] + incl - run;
      total = dscan[kWarps];
      __syncthreads();
      for (int j = j0; j < j1; ++j) {
        const float nj = cdf[j];
        pre += (double)nj;
        cdf[j] = (float)pre;  // in place: this thread alone reads and writes cdf[j0, j1)
        hist[j] = 0u;
        if (a.rec_cdf && writer) a.rec_cdf[a.col_start[mi] + j] = cdf[j];
      }
      __syncthreads();
    }
    // AMM mode with variance reduction: this CTA's memo slot (CTA-private: every thread reads
    // back only the rows it wrote) and whether it holds an exact product of this matrix
    const bool vr = amm && a.vr_period > 0;
    float* Xm = a.vr_mem + (size_t)(a.vr_base + blockIdx.x) * (kVrSlot * kMaxRows * K);
    float* Ym = Xm + kMaxRows * K;
    float* Xsave = Ym + kMaxRows * K;
    bool memo = false;
    bool prev_exact = false;  // the product the Ritz step of this iteration uses was exact

    // ---- start block X0 (hash), orthonormalised below like every later Y ----
    float Y[4][K];
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int v = 0; v < K; ++v)
        Y[e][v] = (r0 + e < m) ? start_value(a.seed, mi, r0 + e, v) : 0.f;
    if (team == 0)
#pragma unroll
      for (int v = 0; v < K; ++v)
#pragma unroll
        for (int e = 0; e < 4; ++e) Xs[xs_idx<K, TC>(v, r0 + e)] = 0.f;
    __syncthreads();

    int it = 0, state = 0;  // state: 0 running, 1 converged / last, 2 degenerate
    for (;; ++it) {
      // ---- Gram matrices of the block: G = YᵀY, H = sym(XᵀY) (FP64, team 0's rows), from a
      // shared-memory copy of team 0's Y (each thread reads back only its own rows) ----
      if (team == 0) y_store<K>(yred, t, Y);
      gram_step<K, TC>(Xs, yred, gpart, Gm, Hm, P, r0, t, warp, lane, team);
      // (gpart, summed into Gm and Hm above, is the Ritz step's scratch)
      if (warp == 0)
        ritz_step<K>(a, mi, it, Gm, Hm, Vm, ritz, Rinv, qv, ctl, gpart, lane, writer,
                     vr && prev_exact);
      __syncthreads();
      // team 0's Y back from its shared-memory copy (not held in registers across the two
      // out-of-line steps, which then get the registers for themselves)
      if (team == 0) y_load<K, false>(yred, t, Y);
      if (ctl[2] && ctl[1] == 0) {
        // residual of the top Ritz pair, r = C·v − λ·v = (Y − λ·X)·q, over team 0's rows (FP64)
        const double lam = ritz[kMaxK];
        double r2 = 0.0;
        if (team == 0 && r0 < m) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float yq = 0.f, xq = 0.f;
#pragma unroll
            for (int v = 0; v < K; ++v) {
              yq = fmaf(Y[e][v], qv[v], yq);
              xq = fmaf(Xs[xs_idx<K, TC>(v, r0 + e)], qv[v], xq);
            }
            const double r = (double)yq - lam * (double)xq;
            r2 = fma(r, r, r2);
          }
        }
        r2 = warp_sum(r2);
        if (lane == 0) gpart[warp] = r2;
        __syncthreads();
        if (t == 0) {
          double s = 0.0;
          for (int w = 0; w < kWarps; ++w) s += gpart[w];
          // with variance reduction only an exact product's residual is the true one
          const bool done = (sqrt(s) <= a.tol * fabs(lam) && (!vr || prev_exact)) ||
                            it >= a.max_iter;
          if (done) {
            if (writer) {
              for (int i = 0; i < K; ++i) a.lam[(int64_t)mi * K + i] = ritz[i];
              a.iters[mi] = it;
            }
            ctl[1] = 1;
          }
        }
        __syncthreads();
      }
      state = ctl[1];
      if (state != 0) {
        if (state == 1 && team == 0 && writer) {  // v = X·q over this thread's rows
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (r0 + e < m) {
              float s = 0.f;
#pragma unroll
              for (int v = 0; v < K; ++v) s = fmaf(Xs[xs_idx<K, TC>(v, r0 + e)], qv[v], s);
              a.vec[M.out_off + r0 + e] = s;
            }
          }
        }
        break;
      }
      // ---- X <- Y·M (team 0 writes the shared copy) ----
      if (team == 0) {
        float X[4][K];
#pragma unroll
        for (int j = 0; j < K; ++j) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < K; ++i) s = fmaf(Y[e][i], Rinv[i * K + j], s);
            X[e][j] = s;
          }
        }
        if constexpr (TC) {  // [v][row]; and by row for a product with C (in the idle tile region)
#pragma unroll
          for (int j = 0; j < K; ++j)
            *reinterpret_cast<float4*>(Xs + xs_idx<K, true>(j, r0)) =
                make_float4(X[0][j], X[1][j], X[2][j], X[3][j]);
          if (a.use_c && M.C) y_store<K>(reinterpret_cast<float*>(smem + SL::xrow), t, X);
        } else if constexpr (K % 2 == 0) {  // interleaved pairs
#pragma unroll
          for (int j = 0; j < K; j += 2)
#pragma unroll
            for (int e = 0; e < 4; e += 2)
              *reinterpret_cast<float4*>(Xs + xs_idx<K>(j, r0 + e)) =
                  make_float4(X[e][j], X[e][j + 1], X[e + 1][j], X[e + 1][j + 1]);
        } else {
#pragma unroll
          for (int j = 0; j < K; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) Xs[xs_idx<K, TC>(j, r0 + e)] = X[e][j];
        }
      }
      __syncthreads();
      // kind of product `it`: exact in exact mode; in AMM mode with variance reduction exact
      // (and memoised) when (it + 1) % vr_period == 0 (powerMethod_by_previous.cuh:135-157)
      // and for the last product, so that the reported Ritz values come from an exact product
      const bool exact_p =
          !amm || (vr && ((it + 1) % a.vr_period == 0 || it + 1 >= a.max_iter));
      const bool wamm = amm && !exact_p;  // this product is sampled
      // ---- AMM: draw c columns (get_rand + pick_index, device_memory.h:506-545) and list the
      // distinct ones in ascending order with weight multiplicity / (c·p_j) ----
      int ncols = n;
      if (wamm) {
        // the histogram shares its memory with the column ring of the last product pass
        for (int j = t; j < n; j += kThreads) hist[j] = 0u;
        __syncthreads();
        const float total_f = cdf[n - 1];
        uint32_t* st = a.states + M.st_off;
        // every CTA of the cluster draws the same picks from the same states; rank 0 stores the
        // advanced states once all have read them
        uint32_t ys[kMaxPicks / kThreads];
#pragma unroll
        for (int u = 0; u < kMaxPicks / kThreads; ++u) {
          const int k = t + u * kThreads;
          ys[u] = k < M.c ? xorshift32(st[k]) : 0u;
        }
        if (CL > 1) cluster.sync();
#pragma unroll
        for (int u = 0; u < kMaxPicks / kThreads; ++u) {
          const int k = t + u * kThreads;
          if (k >= M.c) continue;
          const uint32_t y = ys[u];
          if (writer) st[k] = y;
          const float target = __fmul_rn(total_f, uniform_from(y));
          int lo = 0, hi = n;  // first i with cdf[i] > target, else n - 1
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (cdf[mid] <= target)
              lo = mid + 1;
            else
              hi = mid;
          }
          const int pick = lo < n ? lo : n - 1;
          atomicAdd(&hist[pick], 1u);
          if (a.rec_picks && writer && it < a.rec_products)
            a.rec_picks[M.st_off * a.rec_products + (int64_t)it * M.c + k] = (uint32_t)pick;
        }
        __syncthreads();
        const int per = (n + kThreads - 1) / kThreads;
        const int j0 = t * per, j1 = min(n, j0 + per);
        uint32_t nz = 0;
        for (int j = j0; j < j1; ++j) nz += hist[j] ? 1u : 0u;
        uint32_t cd = 0;
        uint32_t r = block_exclusive_scan(nz, scan, &cd);
        for (int j = j0; j < j1; ++j) {
          const uint32_t mult = hist[j];
          if (mult) {
            // the realised probability of column j is its FP32 CDF step over the total
            const double step = (double)cdf[j] - (j > 0 ? (double)cdf[j - 1] : 0.0);
            lcol[r] = j;
            lw[r] = (float)((double)mult * (double)total_f / ((double)M.c * step));
            ++r;
            hist[j] = 0u;
          }
        }
        ncols = (int)cd;
        __syncthreads();
      }
      // ---- variance reduction: S = X_memoᵀ·X (FP64 sums over team 0's rows) and the block
      // the sampled product multiplies, D = X − X_memo·S, in place of X; Y_memo·S is added,
      // and X put back, once the product is summed ----
      const bool use_d = wamm && memo;
      if (use_d) vr_difference<K>(Xm, Xs, Xsave, gpart, Svr, P, r0, t, warp, lane, team);
      const float* Xsrc = Xs;  // X, or D in its place
      // ---- Y = C·X (or its AMM estimate): the fused pass over the columns (team-local) ----
      const bool rows = r0 < m;
      int buf = 0;
      const bool by_c = TC && a.use_c && M.C != nullptr;  // the product as C·X
      if (by_c) {
        // (nothing that this kernel keeps in registers is passed to an out-of-line function by
        // address: it would live in local memory, and the L1 left beside the shared memory is
        // streamed through by the products)
        if constexpr (TC) {
          cx_product<K>(M.C, M.ldc, reinterpret_cast<const float*>(smem + SL::xrow),
                        reinterpret_cast<float4*>(yred), r0, gteam, NTG);
          memo_load<K>(yred, t, Y);
        }
        __syncthreads();  // the slots lie where Y is copied next
      } else if constexpr (TC) {
        // ---- tensor-core pass (exact mode, 8 vectors).  Warp wi of a team owns the team's
        // rows [128·wi, 128·wi + 128); per group of 8 columns its lane 0 copies those rows into
        // the warp's own 4 KB tile (two stages) with four TMA boxes of 32 rows x 8 columns
        // (128-byte swizzle: 16-byte chunk q of a column's 32-row line stored at q ^ (column
        // mod 8); rows past m and columns past n arrive as zeros), completing on the stage's
        // mbarrier.  Phase 1, per 16-row block: Tᵀ(16 x 8) += [X_hi | X_lo]ᵀ·A_blk, rows 0-7 of
        // the 16 holding X_hi, rows 8-15 X_lo, once with A_hi and once with A_lo (all four split
        // terms in two products); the rows of the block are ordered so that a lane's operands are
        // 4 consecutive rows (one 16-byte load each of A and X).  The team's warps sum their T
        // (fixed order).  Phase 2, per 16-row tile: Y += A_tile·T with the 8 columns ordered
        // 0,2,4,6 | 1,3,5,7 along k, so that the lane's T values are exactly its B operand; three
        // products (A_hi·T_hi, A_hi·T_lo, A_lo·T_hi). ----
        const int W = P / 32;               // warps of the team
        const int wi = tl >> 5;             // this warp's place in the team
        const int g = lane >> 2, tq = lane & 3;
        const int rbase = 128 * wi;         // first row of this warp
        const int nblk = max(0, min(8, (m - rbase + 15) >> 4));  // 16-row blocks below m
        const int nbox = (nblk + 1) >> 1;   // 32-row boxes below m
        float* wtile = reinterpret_cast<float*>(smem + SL::region) + warp * kTcWarpFloats;
        uint64_t* wbar = tbar + 2 * warp;   // this warp's stage barriers
        const CUtensorMap* tmap = a.tmaps + mi;
        float yacc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) yacc[i][j] = 0.f;
        auto issue = [&](int g0, int st) {
          // (the warp's reads of the stage ended before the __syncwarp that closed the group
          // which last used it); lane 0 announces the bytes, lanes 0..nbox-1 issue a box each
          if (nbox > 0 && !tdead) {
            if (lane == 0) mbar_arrive_expect_tx(&wbar[st], (uint32_t)nbox * 1024u);
            __syncwarp();
            if (lane < nbox)
              tma_load_2d(wtile + st * kTcStageFloats + lane * 256, tmap, rbase + 32 * lane, g0,
                          &wbar[st]);
          }
        };
        // every thread's earlier accesses of the tile region (the Gram step's copy of Y, the
        // team sums of the last pass, its tiles) are ordered before the first copies' writes
        fence_proxy_async_smem();
        __syncthreads();
        const int gstep = NTG * kTcCols;
        int st = 0;
        if (gteam * kTcCols < ncols) issue(gteam * kTcCols, 0);
#pragma unroll 1
        for (int g0 = gteam * kTcCols; g0 < ncols; g0 += gstep, buf ^= 1) {
          if (g0 + gstep < ncols) issue(g0 + gstep, st ^ 1);
          if (nbox > 0 && !tdead) {  // group g0 has landed (bounded wait; a timeout marks the matrix)
            const bool ok = mbar_wait_bounded(&wbar[st], (tph >> st) & 1u);
            tph ^= 1u << st;
            if (__any_sync(0xffffffffu, !ok)) tfail = tdead = true;
          }
          const float* tile = wtile + st * kTcStageFloats;
          // phase 1: T = AᵀX over this warp's rows
          float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
          for (int sb = 0; sb < nblk; ++sb) {
            const float4 av = lds_f4(tile + (sb >> 1) * 256 + g * 32 + 4 * ((4 * (sb & 1) + tq) ^ g));
            const float4 xv = lds_f4(Xs + g * kXsStrideTC + rbase + 16 * sb + 4 * tq);
            uint32_t ah[4], al[4], xh[4], xl[4];
            tf32_split(av.x, ah[0], al[0]);
            tf32_split(av.y, ah[1], al[1]);
            tf32_split(av.z, ah[2], al[2]);
            tf32_split(av.w, ah[3], al[3]);
            tf32_split(xv.x, xh[0], xl[0]);
            tf32_split(xv.y, xh[1], xl[1]);
            tf32_split(xv.z, xh[2], xl[2]);
            tf32_split(xv.w, xh[3], xl[3]);
            // k = tq <-> row 4·tq (+2), k = tq + 4 <-> row 4·tq + 1 (+2); the block's four
            // products start from zero and the block sums are added in FP32 with rounding to
            // nearest (the tensor core's own accumulation is not rounded to nearest, and a long
            // chain of it drifts: 1e-5 relative over a 2048-row pass)
            // (two independent chains of two, one per k-half, so that they overlap)
            float db0[4] = {0.f, 0.f, 0.f, 0.f}, db1[4] = {0.f, 0.f, 0.f, 0.f};
            mma_tf32(db0, xh[0], xl[0], xh[1], xl[1], ah[0], ah[1]);
            mma_tf32(db1, xh[2], xl[2], xh[3], xl[3], ah[2], ah[3]);
            mma_tf32(db0, xh[0], xl[0], xh[1], xl[1], al[0], al[1]);
            mma_tf32(db1, xh[2], xl[2], xh[3], xl[3], al[2], al[3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) d[j] += db0[j] + db1[j];
          }
          // lane (g, tq): T[col 2·tq][v g] and T[col 2·tq + 1][v g] (hi and lo rows summed)
          float t0 = d[0] + d[2], t1 = d[1] + d[3];
          if (W > 1) {
            float2* pb = reinterpret_cast<float2*>(part) + buf * kWarps * 32;
            pb[warp * 32 + lane] = make_float2(t0, t1);
            named_barrier_or(1 + team, P, false);
            t0 = 0.f;
            t1 = 0.f;
            for (int w = 0; w < W; ++w) {
              const float2 q = pb[(team_warp0 + w) * 32 + lane];
              t0 += q.x;
              t1 += q.y;
            }
          }
          uint32_t th0, tl0, th1, tl1;
          tf32_split(t0, th0, tl0);
          tf32_split(t1, th1, tl1);
          // phase 2: Y += A·T over this warp's 16-row tiles
          const int ce = 2 * tq, co = 2 * tq + 1;  // the lane's columns
          const float* pe = tile + ce * 32 + (g & 3);
          const float* po = tile + co * 32 + (g & 3);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (i >= nblk) break;
            // rows 16i + g and 16i + g + 8: box i/2, 16-byte chunks q0 and q0 + 2 of its lines
            const int q0 = 4 * (i & 1) + (g >> 2), q1 = q0 + 2;
            const int bo = (i >> 1) * 256;
            uint32_t ah[4], al[4];
            tf32_split(pe[bo + 4 * (q0 ^ ce)], ah[0], al[0]);
            tf32_split(pe[bo + 4 * (q1 ^ ce)], ah[1], al[1]);
            tf32_split(po[bo + 4 * (q0 ^ co)], ah[2], al[2]);
            tf32_split(po[bo + 4 * (q1 ^ co)], ah[3], al[3]);
            // three products from zero (small terms first), then one rounded FP32 add per
            // element into Y, which sums over every group of the pass
            float dt[4] = {0.f, 0.f, 0.f, 0.f};
            mma_tf32(dt, al[0], al[1], al[2], al[3], th0, th1);
            mma_tf32(dt, ah[0], ah[1], ah[2], ah[3], tl0, tl1);
            mma_tf32(dt, ah[0], ah[1], ah[2], ah[3], th0, th1);
#pragma unroll
            for (int j = 0; j < 4; ++j) yacc[i][j] += dt[j];
          }
          __syncwarp();  // every lane is done with this stage before it is refilled
          st ^= 1;
        }
        // (every copy issued was waited on: none can still be landing in the tiles)
        if (__syncthreads_or(tfail ? 1 : 0)) tfail_mi = mi;
        tfail = tdead;
        // the team partials of Y through yred (which shares the tiles' memory), summed over the
        // teams in a fixed order by team 0
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= nblk) break;
          const int row = team * 4 * P + rbase + 16 * i + g;
          *reinterpret_cast<float2*>(yred + yat<K>(row, 2 * tq)) =
              make_float2(yacc[i][0], yacc[i][1]);
          *reinterpret_cast<float2*>(yred + yat<K>(row + 8, 2 * tq)) =
              make_float2(yacc[i][2], yacc[i][3]);
        }
        __syncthreads();
        if (team == 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int v = 0; v < K; ++v) Y[e][v] = 0.f;
          if (rows) {
#pragma unroll 1
            for (int tm = 0; tm < NT; ++tm) y_load<K, true>(yred, tm * P + t, Y);
          }
        }
      } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int v = 0; v < K; ++v) Y[e][v] = 0.f;
      const float* __restrict__ Ab = M.A + r0;
      // one group of GC columns (weights in AMM mode): the team's dots A_jᵀX over its rows,
      // their sums over the team, and Y += A_j·(A_jᵀX)·w_j
      auto multiply = [&](const float4 (&av)[GC], const float (&wt)[GC]) {
        float d[NV];
        if constexpr (K % 2 == 0) {
          // packed FP32x2: a vector pair per instruction (X pairs interleaved in shared memory)
#pragma unroll
          for (int vp = 0; vp < K / 2; ++vp) {
            const float4 x01 = lds_f4(Xsrc + vp * 2 * kMaxRows + 2 * r0);      // rows 0, 1
            const float4 x23 = lds_f4(Xsrc + vp * 2 * kMaxRows + 2 * r0 + 4);  // rows 2, 3
            const float2 xr[4] = {make_float2(x01.x, x01.y), make_float2(x01.z, x01.w),
                                  make_float2(x23.x, x23.y), make_float2(x23.z, x23.w)};
#pragma unroll
            for (int c = 0; c < GC; ++c) {
              float2 s = __fmul2_rn(make_float2(av[c].x, av[c].x), xr[0]);
              s = __ffma2_rn(make_float2(av[c].y, av[c].y), xr[1], s);
              s = __ffma2_rn(make_float2(av[c].z, av[c].z), xr[2], s);
              s = __ffma2_rn(make_float2(av[c].w, av[c].w), xr[3], s);
              d[c * K + 2 * vp] = s.x;
              d[c * K + 2 * vp + 1] = s.y;
            }
          }
        } else {
#pragma unroll
          for (int v = 0; v < K; ++v) {
            const float4 xv = lds_f4(Xsrc + v * kMaxRows + r0);
#pragma unroll
            for (int c = 0; c < GC; ++c) {
              float s = av[c].x * xv.x;
              s = fmaf(av[c].y, xv.y, s);
              s = fmaf(av[c].z, xv.z, s);
              s = fmaf(av[c].w, xv.w, s);
              d[c * K + v] = s;
            }
          }
        }
        const float red = team_allreduce<NV>(d, part, buf, warp, lane, P, team, team_warp0);
        // the NV totals to every lane through this warp's shared-memory slot: one store and
        // broadcast loads instead of NV shuffles (measured on the B200: 7 % off the batch)
        float* bcw = bcast + warp * 32;
        __syncwarp();
        if ((lane % (32 / NV)) == 0) bcw[lane / (32 / NV)] = red;
        __syncwarp();
        if constexpr (K % 2 == 0) {
#pragma unroll
          for (int c = 0; c < GC; ++c)
#pragma unroll
            for (int vp = 0; vp < K / 2; ++vp) {
              float2 tc = *reinterpret_cast<const float2*>(bcw + c * K + 2 * vp);
              if (wamm) tc = __fmul2_rn(tc, make_float2(wt[c], wt[c]));
              const float ae[4] = {av[c].x, av[c].y, av[c].z, av[c].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 y2 = __ffma2_rn(make_float2(ae[e], ae[e]), tc,
                                             make_float2(Y[e][2 * vp], Y[e][2 * vp + 1]));
                Y[e][2 * vp] = y2.x;
                Y[e][2 * vp + 1] = y2.y;
              }
            }
        } else {
#pragma unroll
          for (int c = 0; c < GC; ++c)
#pragma unroll
            for (int v = 0; v < K; ++v) {
              const float tc = bcw[c * K + v] * wt[c];
              Y[0][v] = fmaf(av[c].x, tc, Y[0][v]);
              Y[1][v] = fmaf(av[c].y, tc, Y[1][v]);
              Y[2][v] = fmaf(av[c].z, tc, Y[2][v]);
              Y[3][v] = fmaf(av[c].w, tc, Y[3][v]);
            }
        }
      };
      // rows past m (the padding up to ld) are zero-filled, so are the slots past the list
      const int gstep = NTG * GC;
      constexpr int NST = Ring<GC>::stages;
      static_assert(NST >= 3, "the column ring needs at least 3 stages");
      // the ring: NST - 1 groups in flight while one is multiplied
      float4* ring = reinterpret_cast<float4*>(smem + SL::region);
      const int vbytes = rows ? 4 * min(4, m - r0) : 0;
      auto issue = [&](int g0, int slot) {
#pragma unroll
        for (int c = 0; c < GC; ++c) {
          const int col = (g0 + c < ncols) ? (wamm ? lcol[g0 + c] : g0 + c) : -1;
          const bool live = vbytes > 0 && col >= 0;
          cp_async16_zfill(ring + (slot * GC + c) * kThreads + t,
                           live ? Ab + (int64_t)col * M.ld : M.A, live ? vbytes : 0);
        }
      };
      int gi = gteam * GC;  // next group to copy
#pragma unroll 1
      for (int s = 0; s < NST - 1; ++s, gi += gstep) {
        if (gi < ncols) issue(gi, s);
        cp_async_commit();
      }
      int slot = 0;
#pragma unroll 1
      for (int g0 = gteam * GC; g0 < ncols; g0 += gstep, buf ^= 1) {
        cp_async_wait_group<NST - 2>();  // group g0 has landed (this thread's copies)
        // refill the slot this thread emptied in the previous group
        if (gi < ncols) issue(gi, slot == 0 ? NST - 1 : slot - 1);
        cp_async_commit();
        gi += gstep;
        float4 av[GC];
        float wt[GC];
#pragma unroll
        for (int c = 0; c < GC; ++c) {
          av[c] = lds_f4(reinterpret_cast<const float*>(ring + (slot * GC + c) * kThreads + t));
          wt[c] = (wamm && g0 + c < ncols) ? lw[g0 + c] : 1.f;
        }
        multiply(av, wt);
        slot = (slot + 1 == NST) ? 0 : slot + 1;
      }
      cp_async_wait_all();  // only empty groups can still be open here
      }
      // ---- sum the team partials of Y (fixed order), every team receives the total ----
      if ((!TC || by_c) && NT > 1) {
        __syncthreads();
        if (rows && team > 0) y_store<K>(yred, t, Y);  // (slot team·P + tl)
        __syncthreads();
        if (rows && team == 0) {  // only team 0 uses the summed Y (Gram, residual, X, v)
#pragma unroll 1
          for (int tm = 1; tm < NT; ++tm) y_load<K, true>(yred, tm * P + t, Y);
        }
      }
      // ---- sum the CTA partials of the cluster through distributed shared memory (fixed
      // rank order): every CTA receives the same Y ----
      if (CL > 1) {
        __syncthreads();
        if (team == 0 && rows) y_store<K>(yred, t, Y);
        cluster.sync();
        if (rows && team == 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int v = 0; v < K; ++v) Y[e][v] = 0.f;
#pragma unroll 1
          for (int rk = 0; rk < CL; ++rk)
            y_load<K, true>(cluster.map_shared_rank(yred, rk), t, Y);
        }
        cluster.sync();  // the buffers are rewritten by the next step
      }
      // ---- variance reduction: Y = Y_memo·S + Ĉ·D for a sampled product; an exact product
      // becomes the memo pair (team 0, its own rows, in every CTA of the cluster alike) ----
      if (use_d) {
        // no team reads X or D any more: every team passed a barrier after its product pass
        // (team sums, cluster sums) or team 0 is the only team
        __syncthreads();  // (the sums' slots are read; below: before Y is copied over these)
        if (team == 0) {
          memo_store<K>(yred, t, Y);  // (this thread's own words)
          vr_add_memo<K>(yred, Ym, Svr, Xsave, Xs, r0, t);
          memo_load<K>(yred, t, Y);
        }
        __syncthreads();
      }
      if (vr && exact_p) {
        if (team == 0) {
          memo_store<K>(Ym, t, Y);
          vr_store_memo<K>(Xm, Xs, r0, t);
        }
        memo = true;
      }
      prev_exact = exact_p;
    }
    __syncthreads();
  }
}

// ---- backward: grad_b = 2·v_b·(v_bᵀ·A_b), column-major like A_b, one warp per column ----
struct GradArgs {
  const Mat* mats;
  const int64_t* col_start;  // count + 1 prefix of column counts
  int32_t count;
  const float* vec;          // Σ m
  float* const* grads;       // count pointers
  const int64_t* grad_ld;    // count
  const float* scale;        // count (upstream gradient per matrix), or null (1)
  int32_t vs_len;            // floats of a warp's copy of v: the largest m, rounded up to 4
};

// Column prefixes a CTA of the backward keeps in shared memory (larger batches search global
// memory).
constexpr int kGradSmemMats = 4096;

// Each warp takes a contiguous range of columns (an even share of all the batch's columns), two
// adjacent columns at a time: both columns' loads are in flight together and their two dots
// share one warp reduction.  The matrix of a column is found in the column prefix (copied to
// shared memory once per CTA) by a search forward from the warp's previous matrix; when the warp
// enters a matrix it copies v into its own 16-byte aligned shared-memory slot, so that A, v and
// the gradient all move in 16-byte accesses (A and the gradient streaming; a gradient column
// that does not start 16-byte aligned takes 4-byte stores).
struct GradMat {
  Mat M;
  int64_t c0 = 0, c1 = 0;  // column range
  float* g = nullptr;
  int64_t gld = 0;
  float k = 1.f;  // 2·scale
  int mi = -1;
};

__device__ __forceinline__ void grad_store(const GradMat& G, const float* vs, int64_t j, float k,
                                           int lane) {
  const int m = G.M.m, m4 = m >> 2;
  float* g = G.g + j * G.gld;
  if ((reinterpret_cast<uintptr_t>(g) & 15u) == 0u) {
#pragma unroll 4
    for (int r4 = lane; r4 < m4; r4 += 32) {
      const float4 vv = reinterpret_cast<const float4*>(vs)[r4];
      __stcs(reinterpret_cast<float4*>(g) + r4, make_float4(k * vv.x, k * vv.y, k * vv.z, k * vv.w));
    }
    for (int r = 4 * m4 + lane; r < m; r += 32) g[r] = k * vs[r];
  } else {
    for (int r = lane; r < m; r += 32) g[r] = k * vs[r];
  }
}

// this lane's part of the dot of column j with v
__device__ __forceinline__ float grad_dot(const GradMat& G, const float* vs, int64_t j, int lane) {
  const int m = G.M.m, m4 = m >> 2;
  const float4* col4 = reinterpret_cast<const float4*>(G.M.A + j * G.M.ld);
  float s = 0.f;
#pragma unroll 4
  for (int r4 = lane; r4 < m4; r4 += 32) {
    const float4 c = __ldcs(col4 + r4);
    const float4 vv = reinterpret_cast<const float4*>(vs)[r4];
    s = fmaf(c.x, vv.x, s);
    s = fmaf(c.y, vv.y, s);
    s = fmaf(c.z, vv.z, s);
    s = fmaf(c.w, vv.w, s);
  }
  for (int r = 4 * m4 + lane; r < m; r += 32) s = fmaf(G.M.A[j * G.M.ld + r], vs[r], s);
  return s;
}

__global__ void __launch_bounds__(256, 4) grad_kernel(const __grid_constant__ GradArgs a) {
  // dynamic shared memory: 8 warp slots of vs_len floats (16-byte multiples), then the column
  // prefixes when count <= kGradSmemMats
  extern __shared__ __align__(16) unsigned char gsm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* vs = reinterpret_cast<float*>(gsm) + (size_t)warp * a.vs_len;
  int64_t* cs_s = reinterpret_cast<int64_t*>(gsm + sizeof(float) * 8 * (size_t)a.vs_len);
  const int count = a.count;
  const bool in_smem = count <= kGradSmemMats;
  if (in_smem)
    for (int i = threadIdx.x; i <= count; i += blockDim.x) cs_s[i] = a.col_start[i];
  __syncthreads();
  auto cstart = [&](int i) -> int64_t { return in_smem ? cs_s[i] : __ldg(a.col_start + i); };
  // the matrix holding column gc (gc not below the range of G): forward search from G's; on a
  // change v is copied into this warp's slot (every lane reads only after the __syncwarp)
  auto locate = [&](GradMat& G, int64_t gc) {
    if (gc < G.c1) return;
    int lo = G.mi + 1, hi = count - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (cstart(mid) <= gc)
        lo = mid;
      else
        hi = mid - 1;
    }
    G.mi = lo;
    G.M = a.mats[lo];
    G.c0 = cstart(lo);
    G.c1 = cstart(lo + 1);
    G.g = a.grads[lo];
    G.gld = a.grad_ld[lo];
    G.k = 2.f * (a.scale ? a.scale[lo] : 1.f);
    __syncwarp();  // every lane is done with the slot's previous vector
    const float* v = a.vec + G.M.out_off;
    for (int r = lane; r < G.M.m; r += 32) vs[r] = v[r];
    __syncwarp();
  };
  const int64_t total = cstart(count);
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t b0 = gw * total / nw, b1 = (gw + 1) * total / nw;  // this warp's columns
  GradMat G;
  for (int64_t gc = b0; gc < b1;) {
    locate(G, gc);
    const int64_t j = gc - G.c0;
    if (gc + 1 < b1 && gc + 1 < G.c1) {  // two columns of one matrix (the usual case)
      float d[2] = {grad_dot(G, vs, j, lane), grad_dot(G, vs, j + 1, lane)};
      const float s = warp_reduce_multi<float, 2>(d, lane);  // lane < 16: column j, else j + 1
      const float s0 = __shfl_sync(0xffffffffu, s, 0), s1 = __shfl_sync(0xffffffffu, s, 16);
      grad_store(G, vs, j, G.k * s0, lane);
      grad_store(G, vs, j + 1, G.k * s1, lane);
      gc += 2;
    } else {
      const float s0 = warp_sum(grad_dot(G, vs, j, lane));
      grad_store(G, vs, j, G.k * s0, lane);
      gc += 1;
    }
  }
}

using KernelFn = void (*)(Args);

struct Variant {
  int K, GC;
  KernelFn fn;
  bool tc;  // tensor-core product: exact batches only
};
constexpr int kClusterSizes[] = {1, 2, 4, 8};

static const Variant kVariants[] = {
    {1, 2, batch_kernel<1, 2>, false},
    {1, 4, batch_kernel<1, 4>, false},
    {4, 2, batch_kernel<4, 2>, false},
    {4, 4, batch_kernel<4, 4>, false},
    {8, 1, batch_kernel<8, 1>, false},
    {8, 2, batch_kernel<8, 2>, false},
    {8, 4, batch_kernel<8, 4>, false},
    {8, kTcCols, batch_kernel<8, kTcCols, true>, true},
};

static int smem_bytes(const Variant& V, bool amm) {
  if (V.tc) return Smem<8, true>::total;
  switch (V.K) {
    case 1: return amm ? Smem<1>::total_amm : Smem<1>::total;
    case 4: return amm ? Smem<4>::total_amm : Smem<4>::total;
    default: return amm ? Smem<8>::total_amm : Smem<8>::total;
  }
}

}  // namespace batch
}  // namespace amm

// ------------------------------------------------------------------------------------------
// Host side: the batch context
// ------------------------------------------------------------------------------------------
using amm::batch::Mat;

struct amm_batch {
  int device = 0;
  int nsm = 0;
  amm_batch_config cfg{};
  int64_t count = 0;
  std::vector<Mat> mats;
  int64_t vec_len = 0;
  int64_t total_cols = 0;
  int64_t n_states = 0;
  bool amm = false;
  // matrices multiplied as C·X: the tiles of their C = A·Aᵀ (longest first) and C's memory
  float* c_mem = nullptr;
  int64_t c_bytes = 0;
  amm::batch::GramTile* d_tiles = nullptr;
  int ntiles = 0;
  // costs per matrix and the processing order they give (largest first), [0] with every product
  // through A, [1] with products as C·X where planned
  std::vector<double> cost[2];
  std::vector<int32_t> order[2];
  // device memory (one allocation)
  void* mem = nullptr;
  Mat* d_mats = nullptr;
  int32_t* d_order = nullptr;  // both orders, one after the other
  uint32_t* d_queue = nullptr;
  int64_t* d_col_start = nullptr;
  float** d_grads = nullptr;
  int64_t* d_grad_ld = nullptr;
  uint32_t* d_states0 = nullptr;  // seeded xorshift states (AMM mode), copied per run
  uint32_t* d_states = nullptr;
  float* d_vr = nullptr;          // AMM mode with variance reduction: per-CTA memo pairs
  // exact batches of 8 vectors: one tensor map per matrix for the tensor-core kernel's tile
  // copies (null when they cannot be encoded; that kernel is then not a candidate)
  CUtensorMap* d_tmaps = nullptr;
  std::vector<CUtensorMap> h_tmaps;
  // optional record of the CDFs and picks (amm_batch_record)
  float* rec_cdf = nullptr;
  uint32_t* rec_picks = nullptr;
  int rec_products = 0;
  int variant = -1;  // chosen tile shape (index into kVariants)
  int cluster = 1;   // CTAs per matrix (cluster size)
  bool use_c = false;  // products as C·X where planned
  int grid = 0;      // CTAs of the persistent launch for that cluster size
  // The heaviest matrices on a wide-cluster launch (wide_count 0: one launch per run): it takes
  // the first wide_count matrices of the order on clusters of wide_cluster CTAs, then joins
  // the launch queued behind it (clusters of `cluster`, narrow_grid CTAs) on the rest.
  int wide_count = 0;
  int wide_cluster = 0;
  int wide_grid = 0;
  int narrow_grid = 0;
  float wide_ms = 0.f;   // the plan's time in the autotuner (0: not timed)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  cudaStream_t cap = nullptr;
  double* g_lam = nullptr;
  float* g_vec = nullptr;
  int32_t* g_iters = nullptr;
};

namespace {

int fail(cudaError_t e, const char* what) { return amm::record_cuda_failure(e, what); }

#define BATCH_CUDA(call)                            \
  do {                                              \
    cudaError_t e_ = (call);                        \
    if (e_ != cudaSuccess) return fail(e_, #call);  \
  } while (0)

struct Guard {
  int old = -1;
  explicit Guard(int dev) {
    cudaGetDevice(&old);
    if (old != dev) cudaSetDevice(dev);
  }
  ~Guard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (old >= 0 && cur != old) cudaSetDevice(old);
  }
};

// Clusters of cl CTAs of the given tile shape that are resident at once (one CTA per SM); 0 if
// that cluster size cannot run.
int max_clusters(amm_batch* b, int variant, int cl) {
  const auto& V = amm::batch::kVariants[variant];
  const int sm = amm::batch::smem_bytes(V, b->amm);
  if (cudaFuncSetAttribute(V.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess)
    return 0;
  if (cl > 1 &&
      cudaFuncSetAttribute(V.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl * b->nsm, 1, 1);
  cfg.blockDim = dim3(amm::batch::kThreads, 1, 1);
  cfg.dynamicSmemBytes = sm;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int nclusters = 0;
  if (cudaOccupancyMaxActiveClusters(&nclusters, (void*)V.fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nclusters > 0 ? nclusters : 0;
}

// CTAs of a persistent launch with clusters of cl CTAs: as many clusters as fit at once, and
// no more than there are matrices.  0 if that cluster size cannot run.
int persistent_grid(amm_batch* b, int variant, int cl) {
  const int nclusters = max_clusters(b, variant, cl);
  if (nclusters < 1) return 0;
  const int64_t use = std::min<int64_t>(nclusters, b->count);
  return (int)use * cl;
}

// C given back (no product reads it where use_c is off).
void drop_c(amm_batch* b) {
  if (b->c_mem) cudaFree(b->c_mem);
  b->c_mem = nullptr;
  b->ntiles = 0;
}

void drop_graph(amm_batch* b) {
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->gexec = nullptr;
  b->graph = nullptr;
}

// Start of a run: both work-list counters zeroed and, in AMM mode, the seeded states restored
// (every run draws the same picks); C formed where products go through it (gram).
int run_prologue(amm_batch* b, cudaStream_t s, bool gram) {
  BATCH_CUDA(cudaMemsetAsync(b->d_queue, 0, 4 * sizeof(uint32_t), s));
  if (b->amm)
    BATCH_CUDA(cudaMemcpyAsync(b->d_states, b->d_states0, sizeof(uint32_t) * b->n_states,
                               cudaMemcpyDeviceToDevice, s));
  if (gram)
    BATCH_CUDA(amm::batch::launch_gram(b->d_mats, b->d_tiles, b->ntiles, b->d_queue + 2, b->nsm, s));
  return AMM_OK;
}

// One persistent launch over the shared list (order, count), after its own list (order0,
// count0).  dependent: launched as a programmatic dependent of the launch before it in the
// stream, so that it starts on the SMs that launch leaves free.
int launch_kernel(amm_batch* b, int variant, int cl, int grid, double* d_lam, float* d_vec,
                  int32_t* d_iters, int max_iter, const int32_t* order, int count,
                  const int32_t* order0, int count0, bool dependent, bool use_c, cudaStream_t s,
                  int vr_base = 0) {
  const auto& V = amm::batch::kVariants[variant];
  const int sm = amm::batch::smem_bytes(V, b->amm);
  BATCH_CUDA(cudaFuncSetAttribute(V.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, sm));
  if (cl > 1)
    BATCH_CUDA(cudaFuncSetAttribute(V.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  amm::batch::Args a{};
  a.mats = b->d_mats;
  a.order = order;
  a.count = count;
  a.order0 = order0;
  a.count0 = count0;
  a.max_iter = max_iter;
  a.tol = b->cfg.tol;
  a.rr_period = b->cfg.rr_period > 0 ? b->cfg.rr_period : 1;
  a.seed = b->cfg.seed;
  a.queue = b->d_queue;
  a.states = b->d_states;
  a.lam = d_lam;
  a.vec = d_vec;
  a.iters = d_iters;
  a.vr_period = b->d_vr ? b->cfg.vr_period : 0;
  a.vr_base = vr_base;
  a.vr_mem = b->d_vr;
  a.rec_cdf = b->rec_cdf;
  a.rec_picks = b->rec_picks;
  a.rec_products = b->rec_products;
  a.col_start = b->d_col_start;
  a.tmaps = b->d_tmaps;
  a.use_c = use_c ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(amm::batch::kThreads, 1, 1);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cl;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = dependent ? 2 : 1;
  BATCH_CUDA(cudaLaunchKernelEx(&cfg, V.fn, a));
  amm::count_launch(1);
  BATCH_CUDA(cudaGetLastError());
  return AMM_OK;
}

// The device's order list for products with or without C.
const int32_t* order_of(const amm_batch* b, bool use_c) {
  return b->d_order + (use_c ? b->count : 0);
}

// A run as one launch over the order list (or a slice of it); gram: C is formed first.
int launch(amm_batch* b, int variant, int cl, int grid, double* d_lam, float* d_vec,
           int32_t* d_iters, int max_iter, const int32_t* order, int count, bool use_c, bool gram,
           cudaStream_t s) {
  const int rc = run_prologue(b, s, gram);
  if (rc) return rc;
  return launch_kernel(b, variant, cl, grid, d_lam, d_vec, d_iters, max_iter, order, count,
                       nullptr, 0, false, use_c, s);
}

// A run with the wide-cluster plan: the wide launch takes the heaviest matrices first, the
// launch queued behind it (programmatic dependent) takes the SMs left, and both share the rest
// of the order list.
int launch_wide(amm_batch* b, double* d_lam, float* d_vec, int32_t* d_iters, int max_iter,
                cudaStream_t s) {
  int rc = run_prologue(b, s, b->use_c);
  if (rc) return rc;
  const int32_t* first = order_of(b, b->use_c);
  const int32_t* rest = first + b->wide_count;
  const int nrest = (int)b->count - b->wide_count;
  rc = launch_kernel(b, b->variant, b->wide_cluster, b->wide_grid, d_lam, d_vec, d_iters,
                     max_iter, rest, nrest, first, b->wide_count, false, b->use_c, s);
  if (rc) return rc;
  return launch_kernel(b, b->variant, b->cluster, b->narrow_grid, d_lam, d_vec, d_iters,
                       max_iter, rest, nrest, nullptr, 0, true, b->use_c, s, b->wide_grid);
}

// The run of the chosen plan.
int launch_run(amm_batch* b, double* d_lam, float* d_vec, int32_t* d_iters, cudaStream_t s) {
  if (b->wide_count > 0) return launch_wide(b, d_lam, d_vec, d_iters, (int)b->cfg.max_iter, s);
  return launch(b, b->variant, b->cluster, b->grid, d_lam, d_vec, d_iters,
                (int)b->cfg.max_iter, order_of(b, b->use_c), (int)b->count, b->use_c, b->use_c, s);
}

// Exact products of `it` products of a sampled run with variance reduction.
int64_t exact_of_sampled(const amm_batch_config& cfg, int64_t it) {
  return cfg.vr_period > 0 ? it / cfg.vr_period + (it % cfg.vr_period != 0 ? 1 : 0) : 0;
}

// CTAs per matrix of a sampled batch of blocks (4 columns per group), from the sizes alone.
//
// A product sampled before the first memo has the rank of its distinct picks.  Where few columns carry
// a matrix's weight they are fewer than the block's vectors, and the block's last vectors are rounding:
// the order of the sums, which the cluster size and the group size set, shows in the Ritz values that
// follow (1e-3 of them over 111 matrices of 8 to 80 picks).  A tiling taken by the clock would make
// results follow the clock.  So the time of a run is estimated per cluster size, with the
// matrices handed to the clusters in order, each to the first that is free, and the smallest is taken:
// us per matrix and product, fixed part by team width (32 .. 512 threads), column groups, and what a
// cluster adds.  Fitted to the times of every cluster size over 502 batches of 8 to 600 matrices (m
// 16-2048, n 64-8192, c = n/4 .. n/32): the fastest size in 92 % of them, 0.5 % slower on average.
// (Times of the kernel while its tilings were still timed, 22.9 ms for the 512-matrix batch: other
// constants would give such batches other results.)
struct SampledCost {
  double fixed[5], group[5];   // by log2(threads of a team / 32)
  double draw, join, join_row; // a sampled product; a cluster's sums, per CTA and team width
  double distinct;             // distinct columns per pick
};
constexpr SampledCost kSampled4 = {{18.5, 18.3, 17.7, 21.6, 24.3}, {1.31, 1.60, 1.60, 1.68, 1.75},
                                   2.1, 4.6, 0.312, 0.3};
constexpr SampledCost kSampled8 = {{45.4, 50.0, 50.1, 63.2, 84.4}, {1.60, 1.89, 1.98, 2.17, 2.34},
                                   0.3, 11.9, 0.714, 0.4};

int sampled_cluster(const amm_batch* b, const std::vector<std::pair<int, int>>& sizes) {
  const SampledCost& k = b->cfg.nvec == 4 ? kSampled4 : kSampled8;
  const double it = (double)std::min<int64_t>(b->cfg.max_iter, 20);
  const double exact = (double)exact_of_sampled(b->cfg, (int64_t)it);
  int best = 0;
  double best_us = 0.0;
  for (const auto& size : sizes) {
    const int cl = size.first;  // CTAs of a cluster, and the clusters
    std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
    for (int i = 0; i < size.second; ++i) free_at.push(0.0);
    double end = 0.0;
    for (const int32_t i : b->order[0]) {
      const Mat& x = b->mats[i];
      int w = 0;
      while (w < 4 && 128 << w < x.m) ++w;
      const double teams = (double)((16 >> w) * cl);
      const double fixed = k.fixed[w] + (cl > 1 ? k.join + k.join_row * (double)(cl << w) : 0.0);
      const double groups = (double)x.n / (4.0 * teams);
      const double picked = k.distinct * (double)x.c / (4.0 * teams);
      const double us = (it + 1.0) * fixed + (exact + 0.1) * groups * k.group[w] +
                        (it - exact) * (k.draw + picked * k.group[w]);
      const double done = free_at.top() + us;
      free_at.pop();
      free_at.push(done);
      end = std::max(end, done);
    }
    if (best == 0 || end < best_us) {
      best = cl;
      best_us = end;
    }
  }
  return best;
}

// Whether the wide launch may take a matrix: in a sampled batch of blocks, unless the caller asked for
// the plan, one with picks enough that the order of its sums is rounding alone.
bool wide_may_take(const amm_batch* b, int32_t i) {
  return !b->amm || b->cfg.nvec == 1 || b->cfg.wide == 1 || b->mats[i].c >= 16 * b->cfg.nvec;
}

// Wide-cluster plan for a batch of uneven matrices.  With one cluster size for all, a matrix
// whose work alone, on one cluster, exceeds an even share of the whole batch per cluster sets
// the run's time (the queue hands it out first, but nothing can help with it).  Those leading
// matrices of the order go to a launch with clusters large enough for the heaviest (the next
// sizes up, at most 8) on at most half the SMs; it then helps with the rest.  Needs
// programmatic dependent launch (both launches resident at once).  With the default setting
// (wide = 0) only for an autotuned cluster size; wide = 1 plans it for a fixed one too, and
// wide = -1 never.
void plan_wide(amm_batch* b) {
  b->wide_count = 0;
  if (!amm::pdl_enabled() || b->cfg.wide < 0 || b->count < 2) return;
  if (b->cfg.cluster > 0 && b->cfg.wide == 0) return;
  const std::vector<double>& cost = b->cost[b->use_c];
  const std::vector<int32_t>& order = b->order[b->use_c];
  double total = 0.0;
  for (const double c : cost) total += c;
  // work per SM of an even split, with a margin: the per-CTA rate falls with the row count,
  // so the heaviest matrices are also the slowest per element
  const double share = 0.75 * total / (double)b->nsm;
  auto work = [&](int k) { return cost[order[k]]; };
  int nwide = 0;
  while (nwide < b->count && work(nwide) > (double)b->cluster * share &&
         wide_may_take(b, order[nwide]))
    ++nwide;
  if (nwide == 0) return;
  int wcl = 0;
  for (int cl : amm::batch::kClusterSizes) {
    if (cl <= b->cluster) continue;
    wcl = cl;
    if (work(0) <= (double)cl * share) break;
  }
  if (wcl == 0) return;
  int nclusters = std::min(max_clusters(b, b->variant, wcl), (b->nsm / 2) / wcl);
  nclusters = std::min(nclusters, nwide);
  if (nclusters < 1) return;
  const int wide_grid = nclusters * wcl;
  int narrow = (b->nsm - wide_grid) / b->cluster;
  narrow = std::min(narrow, max_clusters(b, b->variant, b->cluster));
  narrow = (int)std::min<int64_t>(narrow, b->count - nwide);
  if (narrow < 1) return;
  b->wide_count = nwide;
  b->wide_cluster = wcl;
  b->wide_grid = wide_grid;
  b->narrow_grid = narrow * b->cluster;
}

// Tile-shape autotuner: every (columns per group, cluster size) pair with the requested K runs
// the whole batch for up to 20 iterations (enough for the per-matrix set-up, which favours
// larger clusters, to weigh as it does in a real run); the fastest of two timed runs (CUDA
// events) is kept for the context.  A sampled batch of blocks is not timed (sampled_cluster).  Where
// products are planned as C·X and a tolerance ends the run, the run without C is timed too: whether
// forming C pays depends on how many products it takes to converge.
int autotune(amm_batch* b, double* d_lam, float* d_vec, int32_t* d_iters, cudaStream_t s) {
  if (b->variant >= 0) return AMM_OK;
  int best = -1, best_cl = 1, best_grid = 0;
  bool best_c = false;
  float best_ms = 0.f;
  cudaEvent_t e0, e1;
  BATCH_CUDA(cudaEventCreate(&e0));
  BATCH_CUDA(cudaEventCreate(&e1));
  const int n_var = (int)(sizeof(amm::batch::kVariants) / sizeof(amm::batch::kVariants[0]));
  // the candidates; a single one (tile and cluster size fixed by the caller, or a sampled batch of
  // blocks) is taken untimed
  std::vector<std::tuple<int, int, int, bool>> cand;  // (variant, cluster size, grid, with C)
  const bool sampled_blocks = b->amm && b->cfg.nvec > 1;
  for (int v = 0; v < n_var; ++v) {
    if (amm::batch::kVariants[v].K != b->cfg.nvec) continue;
    if (amm::batch::kVariants[v].tc && (b->amm || !b->d_tmaps)) continue;  // exact-only, maps
    // products as C·X are in the tensor-core kernel, whose product through A is the fastest exact one
    // as well (42 sizes with m 64-2048, n = m/4 .. 5m, 16 and 148 or 296 matrices)
    if (b->ntiles > 0 && !amm::batch::kVariants[v].tc) continue;
    if (b->cfg.tile_gc > 0 && amm::batch::kVariants[v].GC != b->cfg.tile_gc) continue;
    for (int cl : amm::batch::kClusterSizes) {
      if (b->cfg.cluster > 0 && cl != b->cfg.cluster) continue;
      const int grid = persistent_grid(b, v, cl);
      if (grid > 0) cand.emplace_back(v, cl, grid, b->ntiles > 0);
      if (grid > 0 && b->ntiles > 0 && b->cfg.tol > 0.0) cand.emplace_back(v, cl, grid, false);
    }
  }
  const bool fixed = cand.size() == 1;
  if (sampled_blocks && cand.size() > 1) {
    // Every tiling runs once, untimed: a run does not write the vector of a matrix whose block it finds
    // singular, and that vector is then the last one that another tiling found, as it was when the
    // tilings were timed (0.5 s of a first run of 512 matrices, where timing them took 1.4 s).
    const int iters = (int)std::min<int64_t>(b->cfg.max_iter, 20);
    for (const auto& cd : cand) {
      const int rc = launch(b, std::get<0>(cd), std::get<1>(cd), std::get<2>(cd), d_lam, d_vec, d_iters,
                            iters, order_of(b, false), (int)b->count, false, false, s);
      if (rc) return rc;
    }
    const int gc = b->cfg.tile_gc > 0 ? b->cfg.tile_gc : 4;
    std::vector<std::pair<int, int>> sizes;
    for (const auto& cd : cand)
      if (amm::batch::kVariants[std::get<0>(cd)].GC == gc)
        sizes.emplace_back(std::get<1>(cd), std::get<2>(cd) / std::get<1>(cd));
    const int cl = sampled_cluster(b, sizes);
    cand.erase(std::remove_if(cand.begin(), cand.end(),
                              [&](const auto& cd) {
                                return std::get<1>(cd) != cl ||
                                       amm::batch::kVariants[std::get<0>(cd)].GC != gc;
                              }),
               cand.end());
  }
  if (cand.size() == 1) {
    b->variant = std::get<0>(cand[0]);
    b->cluster = std::get<1>(cand[0]);
    b->grid = std::get<2>(cand[0]);
    b->use_c = std::get<3>(cand[0]);
    plan_wide(b);  // untimed with wide = 1, and where the cluster size is the caller's
    if (fixed || b->wide_count == 0 || b->cfg.wide == 1) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return AMM_OK;
    }
    b->variant = -1;  // the plan is timed below against the run without it
  }
  for (const auto& cd : cand) {
    const int v = std::get<0>(cd), cl = std::get<1>(cd), grid = std::get<2>(cd);
    const bool uc = std::get<3>(cd);
    const int iters = (int)std::min<int64_t>(b->cfg.max_iter, 20);
    int rc = launch(b, v, cl, grid, d_lam, d_vec, d_iters, iters, order_of(b, uc), (int)b->count, uc,
                    uc, s);
    if (rc) return rc;
    float ms = 0.f;
    for (int rep = 0; rep < 2; ++rep) {
      BATCH_CUDA(cudaEventRecord(e0, s));
      rc = launch(b, v, cl, grid, d_lam, d_vec, d_iters, iters, order_of(b, uc), (int)b->count, uc,
                  uc, s);
      if (rc) return rc;
      BATCH_CUDA(cudaEventRecord(e1, s));
      BATCH_CUDA(cudaEventSynchronize(e1));
      float t = 0.f;
      BATCH_CUDA(cudaEventElapsedTime(&t, e0, e1));
      ms = rep == 0 ? t : std::min(ms, t);
    }
    if (best < 0 || ms < best_ms) {
      best = v;
      best_cl = cl;
      best_grid = grid;
      best_c = uc;
      best_ms = ms;
    }
  }
  if (best < 0) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return AMM_ERR_UNSUPPORTED;
  }
  b->variant = best;
  b->cluster = best_cl;
  b->grid = best_grid;
  b->use_c = best_c;
  if (!best_c) drop_c(b);
  // the wide-cluster plan, kept only if it runs faster (same iterations, best of two), or
  // untimed with wide = 1
  plan_wide(b);
  if (b->wide_count > 0 && b->cfg.wide == 0) {
    const int iters = (int)std::min<int64_t>(b->cfg.max_iter, 20);
    int rc = launch_wide(b, d_lam, d_vec, d_iters, iters, s);
    float ms = 0.f;
    for (int rep = 0; rc == AMM_OK && rep < 2; ++rep) {
      BATCH_CUDA(cudaEventRecord(e0, s));
      rc = launch_wide(b, d_lam, d_vec, d_iters, iters, s);
      if (rc) break;
      BATCH_CUDA(cudaEventRecord(e1, s));
      BATCH_CUDA(cudaEventSynchronize(e1));
      float t = 0.f;
      BATCH_CUDA(cudaEventElapsedTime(&t, e0, e1));
      ms = rep == 0 ? t : std::min(ms, t);
    }
    b->wide_ms = ms;
    if (rc || !(ms < best_ms)) b->wide_count = 0;
    if (rc) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return rc;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return AMM_OK;
}

}  // namespace

extern "C" {

void amm_batch_config_default(amm_batch_config* c) {
  if (!c) return;
  std::memset(c, 0, sizeof(*c));
  c->nvec = 8;
  c->max_iter = 500;
  c->tol = 1e-6;
  c->rr_period = 1;
  c->use_graph = 1;
  c->seed = 1234;
  c->tile_gc = 0;
  c->c_divisor = 0;
  c->cluster = 0;
  c->wide = 0;
  c->vr_period = 0;
}

// The driver's tensor-map encoder (cuTensorMapEncodeTiled), looked up once through the
// runtime; null if the driver does not offer it.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// The tensor maps of the tensor-core kernel's tile copies, one per matrix: FP32, dims {m, n}
// (rows innermost; row stride ld·4 bytes, a multiple of 16 by the batch's alignment rule),
// boxes of 32 rows x 8 columns with the 128-byte swizzle, zeros outside the matrix.  False if
// any cannot be encoded.
static bool encode_tensor_maps(const std::vector<Mat>& ms, std::vector<CUtensorMap>& out) {
  const auto enc = tensor_map_encoder();
  if (!enc) return false;
  out.resize(ms.size());
  for (size_t i = 0; i < ms.size(); ++i) {
    const Mat& M = ms[i];
    const cuuint64_t dims[2] = {(cuuint64_t)M.m, (cuuint64_t)M.n};
    const cuuint64_t strides[1] = {(cuuint64_t)M.ld * sizeof(float)};
    const cuuint32_t box[2] = {32, (cuuint32_t)amm::batch::kTcCols};
    const cuuint32_t elem[2] = {1, 1};
    if (enc(&out[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(M.A), dims, strides,
            box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  return true;
}

// Estimated us of one SM for a matrix: a product through A (21 KB of A a us: the tensor-core product) and
// through C (45 KB of C a us, from L2 or HBM), each with two thirds of the idle rows of its teams (128,
// 256, .. 2048 rows); C itself by tiles of 128 x 256 (diagonal ones of an even row block: 128 x 128), and
// its slowest tile.
struct GramCost {
  double by_a, by_c, form, tile;
};
static GramCost gram_cost(const Mat& x) {
  const double m = (double)x.m, n = (double)x.n;
  double team = 128.0;
  while (team < m) team *= 2.0;
  const double rows = 0.65 * team + 0.35 * m;
  const int blocks = (x.m + 127) / 128;  // of 128 rows; block ti has ti / 2 + 1 tiles
  const double diag = (double)((blocks + 1) / 2);
  const double full = (double)((blocks / 2 + 1) * ((blocks + 1) / 2)) - diag;
  const double chunks = (double)((x.n + 31) / 32);
  const double t_full = 13.2 + 1.80 * chunks, t_diag = 13.2 + 1.46 * chunks;
  return {4.0 * rows * n / 21300.0, 4.0 * rows * m / 45000.0, diag * t_diag + full * t_full,
          full > 0.0 ? t_full : t_diag};
}

// Estimated us of a run of p products per matrix, those of `take` through C: C's tiles over all SMs, then
// the matrices on clusters of the best size, longest first.  An iteration costs 18 us beside its
// product, and 6.9 ns per row and further CTA of the cluster.  (Within 4.4 % rms of 900 measured
// runs, equal and uneven matrices, through A, through C and mixed.)
static double gram_run_us(const std::vector<Mat>& ms, const std::vector<GramCost>& cost,
                          const std::vector<char>& take, double p, int nsm) {
  double form = 0.0, tile = 0.0, best = 0.0;
  for (size_t i = 0; i < ms.size(); ++i)
    if (take[i]) {
      form += cost[i].form;
      tile = std::max(tile, cost[i].tile);
    }
  std::vector<double> us(ms.size());
  for (int cl : amm::batch::kClusterSizes) {
    for (size_t i = 0; i < ms.size(); ++i)
      us[i] = p * ((take[i] ? cost[i].by_c : cost[i].by_a) / cl + 17.7 +
                   0.0069 * (double)(cl - 1) * (double)ms[i].m);
    // (of 148 SMs 33 clusters of 4 and 15 of 8 are resident)
    const int clusters = std::max(1, (cl > 2 ? 9 * nsm / 10 : nsm) / cl);
    double end = 0.0;
    if (us.size() > 1024) {  // many: an even share, or the longest matrix
      double sum = 0.0;
      for (const double u : us) {
        sum += u;
        end = std::max(end, u);
      }
      end = std::max(end, sum / (double)clusters);
    } else {
      std::sort(us.begin(), us.end(), std::greater<double>());
      std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
      for (int k = 0; k < clusters; ++k) free_at.push(0.0);
      for (const double u : us) {
        const double done = free_at.top() + u;
        free_at.pop();
        free_at.push(done);
        end = std::max(end, done);
      }
    }
    if (cl == 1 || end < best) best = end;
  }
  return best + std::max(form / (double)nsm, tile);
}

// Which matrices are multiplied as C·X, C = A·Aᵀ formed once per run: those for which p products through
// C and a share w of forming it take less than p products through A, with the w, of a few, for
// which the run's estimate is least.  (w = 1 is right where the batch keeps every SM busy; in a small or
// an uneven batch the time of its longest matrices counts, and forming C, unlike their products, is
// spread over all SMs.)  Measured, 20 products of equal matrices, time through C over time through A: 296
// of 512 x 307 1.10, 512 x 512 0.85, 512 x 2560 0.35; 148 of 1024 x 614 1.26, 1024 x 1024 0.90; 16 of 2048 x
// 2048 0.80.  36 uneven batches of 11 to 512 matrices, m 16-2048, n 64-8192, 8 to 40 products: 0.5 % above
// the best of every product through A, every one through C, and C by work alone, at most 17 % (11 and 55
// matrices of up to 135 rows, where the routes lie that close); the 512-matrix batch 28.8 ms through
// A, 13.8 through C, 12.7 by this rule.  With a tolerance 16 products are counted, and the autotuner
// times the run without C as well.
// Only in exact batches of 8 vectors with the tile shape left to the library (a fixed one asks for its
// product): the order of a sampled batch's sums is fixed (see sampled_cluster), and the FP32 products
// of 4 vectors are the more accurate ones (λ's rms error against FP64 over 214 matrices: 6.6e-8
// through A, 7.8e-8 through C; 8 vectors: 1.4e-7 through A, 7.7e-8 through C).  None without `with_c`.
// Memory: all of C where an eighth of the device's free memory holds it; else the matrices that save most
// per byte, up to a 48th, so that the caller keeps the device's memory (free_bytes, asked for once).
// Returns C's floats in all; `cost`: per matrix, through A (m·n) and as planned (us a product).
static int64_t plan_gram(std::vector<Mat>& ms, const amm_batch_config& cfg, bool with_c, int nsm,
                         const std::function<size_t()>& free_bytes,
                         std::vector<double> (&cost)[2]) {
  for (auto& c : cost) c.resize(ms.size());
  for (size_t i = 0; i < ms.size(); ++i) {
    ms[i].C = nullptr;
    ms[i].ldc = (ms[i].m + 3) / 4 * 4;
    cost[0][i] = cost[1][i] = (double)ms[i].m * (double)ms[i].n;
  }
  if (!with_c) return 0;
  const double p = (double)(cfg.tol > 0.0 ? std::min<int64_t>(cfg.max_iter, 16) : cfg.max_iter);
  std::vector<GramCost> gc(ms.size());
  for (size_t i = 0; i < ms.size(); ++i) gc[i] = gram_cost(ms[i]);
  std::vector<char> take(ms.size(), 0), best = take, last = take;
  double best_us = gram_run_us(ms, gc, best, p, nsm);
  for (const double w : {1.0, 0.7, 0.5, 0.35, 0.2, 0.1}) {
    for (size_t i = 0; i < ms.size(); ++i)
      take[i] = w * gc[i].form + p * gc[i].by_c < p * gc[i].by_a;
    if (take == last) continue;
    last = take;
    const double us = gram_run_us(ms, gc, take, p, nsm);
    if (us < 0.99 * best_us) {
      best_us = us;
      best = take;
    }
  }
  auto c_bytes = [&](size_t i) { return sizeof(float) * (size_t)ms[i].ldc * (size_t)ms[i].ldc; };
  size_t planned = 0;
  for (size_t i = 0; i < ms.size(); ++i) planned += best[i] ? c_bytes(i) : 0;
  const size_t free_now = planned > 0 ? free_bytes() : 0;
  if (planned > free_now / 8) {
    std::vector<size_t> by_worth;
    std::vector<double> worth(ms.size());
    for (size_t i = 0; i < ms.size(); ++i) {
      if (best[i]) by_worth.push_back(i);
      worth[i] = (p * (gc[i].by_a - gc[i].by_c) - gc[i].form) / (double)c_bytes(i);
    }
    std::stable_sort(by_worth.begin(), by_worth.end(),
                     [&](size_t x, size_t y) { return worth[x] > worth[y]; });
    size_t room = free_now / 48;
    std::fill(best.begin(), best.end(), 0);
    for (const size_t i : by_worth) {
      if (c_bytes(i) > room || !(worth[i] > 0.0)) continue;
      room -= c_bytes(i);
      best[i] = 1;
    }
  }
  int64_t floats = 0;
  for (size_t i = 0; i < ms.size(); ++i) {
    cost[1][i] = 17.7 + (best[i] ? gc[i].by_c : gc[i].by_a);
    if (!best[i]) continue;
    ms[i].C = reinterpret_cast<float*>(1);  // placed by place_gram
    floats += (int64_t)ms[i].ldc * ms[i].ldc;
  }
  return floats;
}

// C of the planned matrices in `mem`, and their tiles, longest first.
static void place_gram(std::vector<Mat>& ms, float* mem, std::vector<amm::batch::GramTile>& tiles) {
  int64_t off = 0;
  for (size_t i = 0; i < ms.size(); ++i) {
    Mat& x = ms[i];
    if (!x.C) continue;
    x.C = mem + off;
    off += (int64_t)x.ldc * x.ldc;
    const int t = (x.m + 127) / 128;
    for (int ti = 0; ti < t; ++ti)
      for (int tj = 0; tj <= ti / 2; ++tj) tiles.push_back({(int32_t)i, ti, tj, 0});
  }
  std::stable_sort(tiles.begin(), tiles.end(),
                   [&](const amm::batch::GramTile& a, const amm::batch::GramTile& c) {
                     return ms[a.mat].n > ms[c.mat].n;
                   });
}

// with_c: matrices may be multiplied as C·X, with memory for C
static int batch_create(amm_batch** out, const amm_batch_matrix* mats, int64_t count,
                        const amm_batch_config* cfg, int device, bool with_c) {
  if (!out || !mats || !cfg || count < 1 || count > (1 << 20)) return AMM_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (cfg->nvec != 1 && cfg->nvec != 4 && cfg->nvec != 8) return AMM_ERR_UNSUPPORTED;
  if (cfg->max_iter < 1 || !(cfg->tol >= 0.0) || cfg->rr_period < 0 || cfg->c_divisor < 0 ||
      cfg->wide < -1 || cfg->wide > 1 || cfg->vr_period < 0)
    return AMM_ERR_INVALID_ARGUMENT;
  const bool amm_mode = cfg->c_divisor > 0;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return AMM_ERR_NO_DEVICE;
  if (device < 0 || device >= ndev) return AMM_ERR_INVALID_ARGUMENT;
  std::vector<Mat> ms((size_t)count);
  int64_t off = 0, cols = 0, nst = 0;
  for (int64_t i = 0; i < count; ++i) {
    const amm_batch_matrix& x = mats[i];
    if (!x.A || x.m < 1 || x.n < 1 || x.ld < x.m) return AMM_ERR_INVALID_ARGUMENT;
    if (x.m > amm::batch::kMaxRows || x.n > INT32_MAX) return AMM_ERR_UNSUPPORTED;
    if (x.m < cfg->nvec) return AMM_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(x.A) & 15) != 0 || (x.ld % 4) != 0) return AMM_ERR_ALIGNMENT;
    ms[i].A = static_cast<const float*>(x.A);
    ms[i].ld = x.ld;
    ms[i].m = (int32_t)x.m;
    ms[i].n = (int32_t)x.n;
    ms[i].out_off = off;
    ms[i].st_off = nst;
    ms[i].c = 0;
    if (amm_mode) {
      if (x.n > amm::batch::kMaxCols) return AMM_ERR_UNSUPPORTED;
      int64_t c = x.n / cfg->c_divisor;
      if (c < 1) c = 1;
      if (c > amm::batch::kMaxPicks) return AMM_ERR_UNSUPPORTED;
      ms[i].c = (int32_t)c;
      nst += c;
    }
    off += x.m;
    cols += x.n;
  }
  std::vector<double> cost[2];
  Guard g(device);
  int nsm = 1;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  // tensor maps when the tensor-core kernel can run: exact, 8 vectors
  std::vector<CUtensorMap> tmaps;
  const bool with_tmaps = !amm_mode && cfg->nvec == 8 && encode_tensor_maps(ms, tmaps);
  const int64_t c_floats = plan_gram(
      ms, *cfg, with_c && with_tmaps && cfg->tile_gc == 0, nsm,
      [] {
        size_t free_now = 0, all = 0;
        if (cudaMemGetInfo(&free_now, &all) != cudaSuccess) cudaGetLastError();
        return free_now;
      },
      cost);
  amm_batch* b = new amm_batch();
  b->nsm = nsm;
  b->device = device;
  b->cfg = *cfg;
  b->count = count;
  if (c_floats > 0) {
    b->c_bytes = (int64_t)sizeof(float) * c_floats;
    const cudaError_t ce = cudaMalloc(&b->c_mem, (size_t)b->c_bytes);
    if (ce != cudaSuccess) {
      cudaGetLastError();
      delete b;
      return ce == cudaErrorMemoryAllocation ? AMM_ERR_OUT_OF_MEMORY : fail(ce, "cudaMalloc");
    }
  }
  std::vector<amm::batch::GramTile> tiles;
  if (b->c_mem) place_gram(ms, b->c_mem, tiles);
  b->ntiles = (int)tiles.size();
  b->mats = ms;
  b->vec_len = off;
  b->total_cols = cols;
  b->n_states = nst;
  b->amm = amm_mode;
  // largest first, ties by index: the queue then balances like LPT scheduling
  std::vector<int32_t> both((size_t)(2 * count));
  for (int k = 0; k < 2; ++k) {
    b->cost[k].swap(cost[k]);
    b->order[k].resize((size_t)count);
    for (int64_t i = 0; i < count; ++i) b->order[k][i] = (int32_t)i;
    const std::vector<double>& c = b->cost[k];
    std::stable_sort(b->order[k].begin(), b->order[k].end(),
                     [&](int32_t x, int32_t y) { return c[x] > c[y]; });
    std::copy(b->order[k].begin(), b->order[k].end(), both.begin() + k * count);
  }
  size_t bytes = 0;
  auto carve = [&](size_t n, size_t align) {
    bytes = (bytes + align - 1) / align * align;
    const size_t o = bytes;
    bytes += n;
    return o;
  };
  const size_t o_mats = carve(sizeof(Mat) * count, 256);
  const size_t o_order = carve(sizeof(int32_t) * 2 * count, 256);
  const size_t o_queue = carve(sizeof(uint32_t) * 4, 256);
  const size_t o_cols = carve(sizeof(int64_t) * (count + 1), 256);
  const size_t o_grads = carve(sizeof(float*) * count, 256);
  const size_t o_gld = carve(sizeof(int64_t) * count, 256);
  const size_t o_st0 = carve(sizeof(uint32_t) * (nst > 0 ? nst : 1), 256);
  const size_t o_st = carve(sizeof(uint32_t) * (nst > 0 ? nst : 1), 256);
  // memo pairs of the variance reduction: one slot per CTA that can be resident at once (the
  // launches of a run hold at most one CTA per SM between them)
  const bool with_vr = amm_mode && cfg->vr_period > 0;
  const size_t vr_floats = (size_t)amm::batch::kVrSlot * amm::batch::kMaxRows * cfg->nvec;
  const size_t o_vr = with_vr ? carve(sizeof(float) * vr_floats * b->nsm, 256) : 0;
  b->h_tmaps.swap(tmaps);  // (64-byte aligned each on the device)
  const size_t o_tiles = carve(sizeof(amm::batch::GramTile) * (tiles.empty() ? 1 : tiles.size()), 256);
  const size_t o_tmaps = with_tmaps ? carve(sizeof(CUtensorMap) * count, 256) : 0;
  cudaError_t e = cudaMalloc(&b->mem, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (b->c_mem) cudaFree(b->c_mem);
    delete b;
    return e == cudaErrorMemoryAllocation ? AMM_ERR_OUT_OF_MEMORY : fail(e, "cudaMalloc");
  }
  char* base = static_cast<char*>(b->mem);
  b->d_mats = reinterpret_cast<Mat*>(base + o_mats);
  b->d_order = reinterpret_cast<int32_t*>(base + o_order);
  b->d_queue = reinterpret_cast<uint32_t*>(base + o_queue);
  b->d_col_start = reinterpret_cast<int64_t*>(base + o_cols);
  b->d_grads = reinterpret_cast<float**>(base + o_grads);
  b->d_grad_ld = reinterpret_cast<int64_t*>(base + o_gld);
  b->d_states0 = reinterpret_cast<uint32_t*>(base + o_st0);
  b->d_states = reinterpret_cast<uint32_t*>(base + o_st);
  b->d_vr = with_vr ? reinterpret_cast<float*>(base + o_vr) : nullptr;
  b->d_tmaps = with_tmaps ? reinterpret_cast<CUtensorMap*>(base + o_tmaps) : nullptr;
  b->d_tiles = reinterpret_cast<amm::batch::GramTile*>(base + o_tiles);
  std::vector<int64_t> cs((size_t)count + 1, 0);
  for (int64_t i = 0; i < count; ++i) cs[i + 1] = cs[i] + ms[i].n;
  e = cudaMemcpy(b->d_mats, ms.data(), sizeof(Mat) * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(b->d_order, both.data(), sizeof(int32_t) * 2 * count, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(b->d_col_start, cs.data(), sizeof(int64_t) * (count + 1),
                   cudaMemcpyHostToDevice);
  if (e == cudaSuccess && !tiles.empty())
    e = cudaMemcpy(b->d_tiles, tiles.data(), sizeof(tiles[0]) * tiles.size(),
                   cudaMemcpyHostToDevice);
  if (e == cudaSuccess && with_tmaps)
    e = cudaMemcpy(b->d_tmaps, b->h_tmaps.data(), sizeof(CUtensorMap) * count,
                   cudaMemcpyHostToDevice);
  if (e == cudaSuccess && nst > 0) {
    // xorshift32 states: a splitmix64 stream from the seed (never zero, a fixed point)
    std::vector<uint32_t> st((size_t)nst);
    uint64_t z = cfg->seed;
    for (int64_t k = 0; k < nst; ++k) {
      z += 0x9E3779B97F4A7C15ull;
      uint64_t x = z;
      x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
      x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
      x ^= x >> 31;
      const uint32_t v = (uint32_t)(x >> 32);
      st[(size_t)k] = v ? v : 0x6A09E667u;
    }
    e = cudaMemcpy(b->d_states0, st.data(), sizeof(uint32_t) * nst, cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    cudaFree(b->mem);
    if (b->c_mem) cudaFree(b->c_mem);
    delete b;
    return fail(e, "cudaMemcpy(batch descriptors)");
  }
  *out = b;
  return AMM_OK;
}

int amm_batch_create(amm_batch** out, const amm_batch_matrix* mats, int64_t count,
                     const amm_batch_config* cfg, int device) {
  const int rc = batch_create(out, mats, count, cfg, device, true);
  // without room for C every product reads A
  return rc == AMM_ERR_OUT_OF_MEMORY ? batch_create(out, mats, count, cfg, device, false) : rc;
}

int amm_batch_destroy(amm_batch* b) {
  if (!b) return AMM_ERR_INVALID_ARGUMENT;
  Guard g(b->device);
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->cap) cudaStreamDestroy(b->cap);
  if (b->mem) cudaFree(b->mem);
  if (b->c_mem) cudaFree(b->c_mem);
  delete b;
  return AMM_OK;
}

int amm_batch_vector_offsets(amm_batch* b, int64_t* offsets) {
  if (!b || !offsets) return AMM_ERR_INVALID_ARGUMENT;
  for (int64_t i = 0; i < b->count; ++i) offsets[i] = b->mats[i].out_off;
  offsets[b->count] = b->vec_len;
  return AMM_OK;
}

int amm_batch_run(amm_batch* b, double* d_lambda, float* d_vectors, int32_t* d_iters,
                  void* stream) {
  if (!b || !d_lambda || !d_vectors || !d_iters) return AMM_ERR_INVALID_ARGUMENT;
  Guard g(b->device);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc = autotune(b, d_lambda, d_vectors, d_iters, s);
  if (rc) return rc;
  if (!b->cfg.use_graph) return launch_run(b, d_lambda, d_vectors, d_iters, s);
  if (b->gexec && (b->g_lam != d_lambda || b->g_vec != d_vectors || b->g_iters != d_iters)) {
    cudaGraphExecDestroy(b->gexec);
    cudaGraphDestroy(b->graph);
    b->gexec = nullptr;
    b->graph = nullptr;
  }
  if (!b->gexec) {
    if (!b->cap) BATCH_CUDA(cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking));
    BATCH_CUDA(cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeRelaxed));
    const int64_t before = amm::launch_count();
    rc = launch_run(b, d_lambda, d_vectors, d_iters, b->cap);
    cudaGraph_t gr = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(b->cap, &gr);
    amm::count_launch(-(int)(amm::launch_count() - before));
    if (rc) {
      if (gr) cudaGraphDestroy(gr);
      return rc;
    }
    if (ce != cudaSuccess) return fail(ce, "cudaStreamEndCapture");
    const cudaError_t ie = cudaGraphInstantiate(&b->gexec, gr, 0);
    if (ie != cudaSuccess) {
      cudaGraphDestroy(gr);
      return fail(ie, "cudaGraphInstantiate");
    }
    b->graph = gr;
    b->g_lam = d_lambda;
    b->g_vec = d_vectors;
    b->g_iters = d_iters;
  }
  BATCH_CUDA(cudaGraphLaunch(b->gexec, s));
  amm::count_launch((b->wide_count > 0 ? 2 : 1) + (b->use_c ? 1 : 0));
  return AMM_OK;
}

int amm_batch_run_each(amm_batch* b, double* d_lambda, float* d_vectors, int32_t* d_iters,
                       void* stream) {
  if (!b || !d_lambda || !d_vectors || !d_iters) return AMM_ERR_INVALID_ARGUMENT;
  Guard g(b->device);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc = autotune(b, d_lambda, d_vectors, d_iters, s);
  if (rc) return rc;
  // one single-CTA launch per matrix; each reads its matrix index from a one-entry slice of
  // the order array; C of every matrix is formed ahead of the first
  for (int64_t i = 0; i < b->count; ++i) {
    rc = launch(b, b->variant, b->cluster, b->cluster, d_lambda, d_vectors, d_iters,
                (int)b->cfg.max_iter, order_of(b, false) + i, 1, b->use_c, b->use_c && i == 0, s);
    if (rc) return rc;
  }
  return AMM_OK;
}

int amm_batch_grad(amm_batch* b, const float* d_vectors, void* const* grad_ptrs,
                   const int64_t* grad_ld, const float* d_scale, void* stream) {
  if (!b || !d_vectors || !grad_ptrs || !grad_ld) return AMM_ERR_INVALID_ARGUMENT;
  for (int64_t i = 0; i < b->count; ++i) {
    if (!grad_ptrs[i] || grad_ld[i] < b->mats[i].m) return AMM_ERR_INVALID_ARGUMENT;
  }
  Guard g(b->device);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  BATCH_CUDA(cudaMemcpyAsync(b->d_grads, grad_ptrs, sizeof(void*) * b->count,
                             cudaMemcpyHostToDevice, s));
  BATCH_CUDA(cudaMemcpyAsync(b->d_grad_ld, grad_ld, sizeof(int64_t) * b->count,
                             cudaMemcpyHostToDevice, s));
  amm::batch::GradArgs a{};
  a.mats = b->d_mats;
  a.col_start = b->d_col_start;
  a.count = (int32_t)b->count;
  a.vec = d_vectors;
  a.grads = b->d_grads;
  a.grad_ld = b->d_grad_ld;
  a.scale = d_scale;
  // one warp per contiguous range of columns; a grid of the CTAs resident at once, 8 warps each
  int max_m = 1;
  for (const auto& M : b->mats) max_m = std::max(max_m, (int)M.m);
  a.vs_len = (max_m + 3) / 4 * 4;
  const size_t smem = sizeof(float) * 8 * (size_t)a.vs_len +
                      (b->count <= amm::batch::kGradSmemMats
                           ? sizeof(int64_t) * (size_t)(b->count + 1) : 0);
  if (smem > 48 * 1024)
    BATCH_CUDA(cudaFuncSetAttribute(amm::batch::grad_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  BATCH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, amm::batch::grad_kernel, 256,
                                                           smem));
  const int64_t warps = b->total_cols;  // at least one column per warp
  int64_t blocks = (warps + 7) / 8;
  blocks = std::min<int64_t>(blocks, (int64_t)b->nsm * std::max(per_sm, 1));
  amm::batch::grad_kernel<<<(int)blocks, 256, smem, s>>>(a);
  amm::count_launch(1);
  BATCH_CUDA(cudaGetLastError());
  // (the pointer arrays come from pageable host memory: the copies above were staged before
  // they returned, so the caller's arrays may go at once)
  return AMM_OK;
}

int amm_batch_set_matrices(amm_batch* b, const amm_batch_matrix* mats, int64_t count,
                           void* stream) {
  if (!b || !mats || count != b->count) return AMM_ERR_INVALID_ARGUMENT;
  for (int64_t i = 0; i < count; ++i) {
    const amm_batch_matrix& x = mats[i];
    if (!x.A || x.m != b->mats[i].m || x.n != b->mats[i].n || x.ld < x.m)
      return AMM_ERR_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(x.A) & 15) != 0 || (x.ld % 4) != 0) return AMM_ERR_ALIGNMENT;
  }
  // the new descriptors (and tensor maps) are formed first, so that a failure leaves the
  // context bound to the old matrices as a whole
  std::vector<Mat> ms = b->mats;
  for (int64_t i = 0; i < count; ++i) {
    ms[i].A = static_cast<const float*>(mats[i].A);
    ms[i].ld = mats[i].ld;
  }
  std::vector<CUtensorMap> tm;
  if (b->d_tmaps && !encode_tensor_maps(ms, tm)) return fail(cudaErrorInvalidValue, "tensor maps");
  b->mats.swap(ms);
  if (b->d_tmaps) b->h_tmaps.swap(tm);
  Guard g(b->device);
  // pageable sources: each copy is staged before the call returns, then stream-ordered
  BATCH_CUDA(cudaMemcpyAsync(b->d_mats, b->mats.data(), sizeof(Mat) * count,
                             cudaMemcpyHostToDevice, reinterpret_cast<cudaStream_t>(stream)));
  if (b->d_tmaps)
    BATCH_CUDA(cudaMemcpyAsync(b->d_tmaps, b->h_tmaps.data(), sizeof(CUtensorMap) * count,
                               cudaMemcpyHostToDevice, reinterpret_cast<cudaStream_t>(stream)));
  return AMM_OK;
}

int amm_batch_record(amm_batch* b, float* d_cdf, uint32_t* d_picks, int64_t products) {
  if (!b || products < 0 || products > (1 << 20) || (d_picks && products == 0))
    return AMM_ERR_INVALID_ARGUMENT;
  if ((d_cdf || d_picks) && !b->amm) return AMM_ERR_INVALID_ARGUMENT;
  b->rec_cdf = d_cdf;
  b->rec_picks = d_picks;
  b->rec_products = d_picks ? (int)products : 0;
  // the captured graph holds the launch arguments by value
  Guard g(b->device);
  drop_graph(b);
  return AMM_OK;
}

int amm_batch_tile_choice(amm_batch* b, int32_t* k_out, int32_t* gc_out, int32_t* cl_out) {
  if (!b || !k_out || !gc_out) return AMM_ERR_INVALID_ARGUMENT;
  if (b->variant < 0) return AMM_ERR_NOT_READY;
  *k_out = amm::batch::kVariants[b->variant].K;
  *gc_out = amm::batch::kVariants[b->variant].GC;
  if (cl_out) *cl_out = b->cluster;
  return AMM_OK;
}

int64_t amm_batch_c_bytes(amm_batch* b) { return b && b->c_mem ? b->c_bytes : 0; }

int amm_batch_release_c(amm_batch* b) {
  if (!b) return AMM_ERR_INVALID_ARGUMENT;
  if (!b->c_mem) return AMM_OK;
  Guard g(b->device);
  BATCH_CUDA(cudaDeviceSynchronize());
  drop_graph(b);  // it forms C and reads it
  drop_c(b);
  b->use_c = false;
  b->wide_count = 0;  // (planned and timed with C)
  return AMM_OK;
}

int amm_batch_wide_plan(amm_batch* b, int32_t* count, int32_t* cluster_size, int32_t* ctas,
                        float* ms) {
  if (!b || !count || !cluster_size || !ctas || !ms) return AMM_ERR_INVALID_ARGUMENT;
  if (b->variant < 0) return AMM_ERR_NOT_READY;
  *count = b->wide_count;
  *cluster_size = b->wide_count > 0 ? b->wide_cluster : 0;
  *ctas = b->wide_count > 0 ? b->wide_grid : 0;
  *ms = b->wide_ms;
  return AMM_OK;
}

}  // extern "C"
