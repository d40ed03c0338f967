// The persistent step kernel of a power-method call (sm_100a): steps [iter, iter_end) in one
// launch, one CTA per SM.
//
//   y = Σ_{k in the step's columns} coef_k · A_k,   coef_k = f(A_kᵀ·dx)
//
// Each CTA owns, per step, a contiguous slice of the step's sorted column list (all n columns for
// an exact step) and all m rows.  One warp streams the columns, GC per group, into a ring of NS
// shared-memory stages with 1-D TMA bulk copies; every thread holds dx and its rows of y in
// registers.  A slice that does not fit the ring is multiplied in a pipelined group loop (the
// axpy of group g beside the dots of group g + 1, one CTA barrier per group).  A slice that fits
// the ring is multiplied in two sweeps over the resident columns (all dots, one reduction, all
// axpys): three CTA barriers however many groups there are.  An exact step that follows another
// finds such a slice still in shared memory and copies nothing.
//
// The exchange between the CTAs.  A step needs the CTAs' partial y summed and the sum known to
// every CTA.  Both directions go through L2 in 16-byte packets of three floats and the step's
// epoch, written and read as single 128-bit accesses: the reader polls the packet itself, so
// there is neither a grid barrier nor a fence between the data and its flag.
//   1. every thread writes its rows of the CTA's partial as packets; thread 0 adds one packet
//      with the CTA's two scalars (Σ α_k t_k, z·dx);
//   2. CTA q owns an even share of the packets: it reads them from all G CTAs, sums in FP64 in a
//      fixed order and writes the packets of y it owns;
//   3. every thread of every CTA reads the packets of its own rows of y.  x·y, y·y and y·v* are
//      summed over all rows by every CTA in the same order, hence every CTA forms the same state,
//      scale and dx.  With more than 4 rows per thread the conversions to FP64 (measured: 17 a
//      clock and SM) cost more than another trip through L2: there the owners of step 2 also
//      write their rows' shares of the three sums, and every CTA sums the shares (8 rows per
//      thread, 4096 x 16384 with 1024 picks: 12.6 us a step against 13.3).
// An owner's packets and shares fill whole 128-byte lines of their own: where a line had two
// writers, some of the SMs polling it saw the second write 2 us late (10.0 -> 8.8 us a step at
// 1024 x 4096).  Several copies of y, each polled by a part of the SMs, gained nothing (8.8, 9.0
// and 9.1 us with 1, 4 and 8).
// No packet is overwritten early: a CTA writes partials of step i + 1 after it has read all
// packets of y_i, each written by a CTA that had read all its partials of step i; and packets of
// y_{i+1} are written after all partials of step i + 1, whose writers had read all of y_i.  The
// CTAs' scalars and shares have two places each, by step parity: a CTA that owns no packet (there
// are fewer packets than CTAs, or fewer owners) waits for no partial, so it may write its shares
// of step i + 1 before a slow CTA has read those of step i, and the scalars of a step may be
// rewritten before it has read them; two steps on, it has finished step i, for it wrote the partials
// of step i + 1 that the packets of y_{i+1} took.
//
// What bounds it: large steps the column stream (HBM); small ones the two trips through L2
// (write, poll: 0.5-0.7 us each from SM to SM) and the CTA-wide reductions between them.
// Measured against grid barriers (a counter per step, partial sums and shares read after it), us
// a step on one B200, before -> after: 256 x 1024 14.7 -> 7.0; 1024 x 4096 exact 19.2 -> 9.1;
// 4096 x 16384 with 1024 picks 14.7 -> 12.2; 3000 x 10007 BF16 18.8 -> 13.0; 16384 x 16384
// exact 157.9 -> 156.5; 16384 x 65536 BF16, mean of 9 steps, 73.1 -> 69.5.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "amm_device.cuh"
#include "amm_internal.h"
#include "amm_panel.cuh"

namespace amm {

// column groups of the next step issued ahead when its slice does not fit the ring
constexpr int kPrefetchGroups = 2;
constexpr int kMaxWarps = kMaxThreads / 32;
// dynamic shared memory a CTA may use: the opt-in maximum less the kernel's static variables
constexpr int kSmemBudget = 227 * 1024 - 1024;
constexpr int kMaxStages = 8;

struct StepArgs {
  Buffers b;
  PanelGeom g;
  CallCfg cc;
  int iter;      // first step of the launch
  int iter_end;  // steps [iter, iter_end) run in this launch
};

// ---- packets: three floats and the epoch, one 128-bit access each.  A reader uses all four
// words: where one was left unused the compiler narrowed the load to two, and a value from before
// the epoch's store was seen; a packet with fewer than three values repeats its last one. ----
__device__ __forceinline__ void packet_store(uint4* p, float a, float b, float c, uint32_t ep) {
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 q;\n\t"
      "mov.b64 lo, {%1, %2};\n\tmov.b64 hi, {%3, %4};\n\tmov.b128 q, {lo, hi};\n\t"
      "st.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
      "r"(__float_as_uint(a)), "r"(__float_as_uint(b)), "r"(__float_as_uint(c)), "r"(ep)
      : "memory");
}
__device__ __forceinline__ uint4 packet_load(const uint4* p) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .b64 lo, hi;\n\t.reg .b128 q;\n\t"
      "ld.relaxed.gpu.global.b128 q, [%4];\n\tmov.b128 {lo, hi}, q;\n\t"
      "mov.b64 {%0, %1}, lo;\n\tmov.b64 {%2, %3}, hi;\n\t}"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p)
      : "memory");
  return v;
}
// a double in a packet: (low, high, low)
__device__ __forceinline__ void packet_store(uint4* p, double d, uint32_t ep) {
  const float lo = __int_as_float(__double2loint(d));
  packet_store(p, lo, __int_as_float(__double2hiint(d)), lo, ep);
}
// U packets at p[k * stride], k < cnt, until each carries epoch ep (bounded; false: gave up);
// D: packets of a double
template <int U, bool D = false>
__device__ __forceinline__ bool packets_wait(const uint4* p, size_t stride, int cnt, uint32_t ep,
                                             uint4 (&v)[U]) {
  unsigned long long t0 = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = make_uint4(0u, 0u, 0u, ep);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (u < cnt) v[u] = packet_load(p + (size_t)u * stride);
  for (uint32_t it = 0;; ++it) {
    bool all = true;
#pragma unroll
    for (int u = 0; u < U; ++u) all = all && v[u].w == ep && (!D || v[u].z == v[u].x);
    if (all) return true;
    if ((it & 63u) == 63u) {
      const unsigned long long now = globaltimer_now();
      if (t0 == 0) t0 = now;
      if (now - t0 > kWaitLimitNs) return false;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v[u].w != ep || (D && v[u].z != v[u].x)) v[u] = packet_load(p + (size_t)u * stride);
  }
}

constexpr int kOwnBytes = 96;
constexpr int kOwnedMax = 64;   // packets a CTA owns at most: one per thread of two warps

// The same for packets at p[off[u]].
template <int U>
__device__ __forceinline__ bool packets_wait_at(const uint4* p, const int (&off)[U], int cnt,
                                                uint32_t ep, uint4 (&v)[U]) {
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = u < cnt ? packet_load(p + off[u]) : make_uint4(0u, 0u, 0u, ep);
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    bool all = true;
#pragma unroll
    for (int u = 0; u < U; ++u) all = all && v[u].w == ep;
    if (all) return true;
    if ((it & 63u) == 63u) {
      const unsigned long long now = globaltimer_now();
      if (t0 == 0) t0 = now;
      if (now - t0 > kWaitLimitNs) return false;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (v[u].w != ep) v[u] = packet_load(p + off[u]);
  }
}

// Shared memory carve (byte offsets), identical on host and device.
struct StepLayout {
  int stages, bars, redw, wl_idx, wl_w, wl_al, nxt, red, own, scr, coef, total;
};

// packets per thread, packets of a whole vector, packets a CTA owns at most
__host__ __device__ inline int step_packets_per_thread(const PanelGeom& g) {
  return (g.slots * g.elems + 2) / 3;
}
__host__ __device__ inline int step_packets(const PanelGeom& g) {
  return step_packets_per_thread(g) * g.threads;
}
// packets a CTA owns (the last owner fewer, CTAs past it none)
__host__ __device__ inline int step_owned_max(const PanelGeom& g) {
  return (step_packets(g) + g.grid - 1) / g.grid;
}
// A CTA's block of y packets: its packets, then by step parity and owner warp the shares of x·y, y·y
// and y·v*; whole 128-byte lines, so that no line has two writers
constexpr int kShareWarps = 2;
__host__ __device__ inline int step_block(const PanelGeom& g) {
  return (step_owned_max(g) + 2 * 3 * kShareWarps + 7) / 8 * 8;
}

__host__ __device__ inline StepLayout step_layout(const PanelGeom& g) {
  StepLayout L{};
  int o = 0;
  L.stages = o;
  o += g.stage_area;
  L.bars = o;
  o += kMaxStages * 16;
  L.redw = o;  // [max(2, stages)][16 warps][GC] partial dots
  o += kMaxStages * kMaxWarps * g.gc * 4;
  L.wl_idx = o;
  o += 4 * g.wl_cap;
  L.wl_w = o;
  o += 4 * g.wl_cap;
  L.wl_al = o;
  o += 4 * g.wl_cap;
  o = (o + 127) & ~127;
  L.nxt = o;  // first column indices of the next step's list
  o += 4 * kGcMax * kMaxStages;
  L.coef = o;  // coefficients of a resident slice
  o += 4 * kGcMax * kMaxStages;
  L.red = o;  // staging of the owned packets' sums: [3][threads] double
  o += 3 * 8 * g.threads;
  L.own = o;  // owned packets (kOwnBytes each): y_{i-1}, x_memo, y_memo, v, z (3 floats each), the
              // mask of real rows, v* (3 doubles)
  o += kOwnBytes * step_owned_max(g);
  o = (o + 15) & ~15;
  L.scr = o;  // [16 warps][4] double: x·y, y·y, y·v*; then [16] Σdx
  o += kMaxWarps * 5 * 8;
  L.total = (o + 127) & ~127;
  return L;
}

int step_smem(const PanelGeom& g) { return step_layout(g).total; }
int64_t step_partial_packets(const PanelGeom& g) { return step_packets(g) + 2; }
// y by owners' blocks
int64_t step_y_packets(const PanelGeom& g) { return (int64_t)step_block(g) * g.grid; }
// The packet exchange wants enough CTAs that one thread per owned packet is left; a device (or a
// partition) with fewer SMs, and the cluster variant, run the step kernel of amm_panel.cu.
bool step_supported(const PanelGeom& g) {
  return g.cluster == 1 && step_owned_max(g) <= std::min(g.threads, kOwnedMax) &&
         step_smem(g) <= kSmemBudget;
}

// Sum over the warps of the NC partial dots per warp (element (w, c) at base[w * NC + c]),
// identical in every warp: L lanes own one value, each adds every L-th warp, and a fixed xor tree
// joins them.
template <int NC>
__device__ __forceinline__ void warps_sum(const float* base, int ncw, int lane, float (&tot)[NC]) {
  constexpr int L = (32 / NC) < 16 ? (32 / NC) : 16;
  const int c = (lane / L) % NC;
  float v = 0.f;
  for (int w = lane % L; w < ncw; w += L) v += base[w * NC + c];
#pragma unroll
  for (int off = L / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
#pragma unroll
  for (int k = 0; k < NC; ++k) tot[k] = __shfl_sync(0xffffffffu, v, k * L);
}

template <typename Elem, int R, int GC>
__global__ void __launch_bounds__(kMaxThreads, 1)
    step_kernel(const __grid_constant__ StepArgs a) {
  constexpr int E = 16 / static_cast<int>(sizeof(Elem));
  constexpr int H = E / 2;             // float2 per vector
  constexpr int NV = R * E;            // rows of a thread
  constexpr int NP = (NV + 2) / 3;     // packets of a thread
  constexpr int kBatch = NP > 4 ? 6 : NP;  // packets of a thread read at once
  // x_memo of the next step is loaded before the Rayleigh sums where the registers allow it
  constexpr bool kXmAhead = NV <= 16;
  // the Rayleigh sums travel as the owners' shares (else every CTA sums all rows, x kept beside dx)
  constexpr bool kShares = NV > 4;
  const Buffers& b = a.b;
  const PanelGeom& g = a.g;
  const CallCfg& cc = a.cc;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int T = blockDim.x;
  const int ncw = T >> 5;
  const int G = gridDim.x;
  const int q = blockIdx.x;
  const int m = b.m;
  const int nvec = m / E;
  const int NS = g.nstages;
  const uint32_t col_bytes = (uint32_t)(m * sizeof(Elem));
  const bool full_slots = (T * R == nvec);  // every vector slot of every thread is a real row

  extern __shared__ __align__(128) unsigned char smem[];
  const StepLayout L = step_layout(g);
  unsigned char* stages = smem + L.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);
  float* redw = reinterpret_cast<float*>(smem + L.redw);
  uint32_t* wl_idx = reinterpret_cast<uint32_t*>(smem + L.wl_idx);
  float* wl_w = reinterpret_cast<float*>(smem + L.wl_w);
  float* wl_al = reinterpret_cast<float*>(smem + L.wl_al);
  uint32_t* nxt_cols = reinterpret_cast<uint32_t*>(smem + L.nxt);
  float* coef_s = reinterpret_cast<float*>(smem + L.coef);
  double* red = reinterpret_cast<double*>(smem + L.red);
  float* own = reinterpret_cast<float*>(smem + L.own);
  double* scr = reinterpret_cast<double*>(smem + L.scr);
  double* sdx_s = scr + 4 * kMaxWarps;
  __shared__ IterState st_s;           // state of the launch's first step, then of the step past its last
  // loop-carried values live in shared memory, so that the group loop keeps its registers
  __shared__ uint32_t ep0_s, iss_s;    // the launch's first epoch less one; groups issued so far
  __shared__ float scale_s[2];         // of step i at [i & 1], as the four below
  __shared__ int32_t mode_s[2], used_s[2], le_s[2];
  __shared__ int32_t memo_s[2];        // x_memo: 0 zero, 1 the context's, 2 this CTA's copy
  __shared__ double lam_s[2];          // λ of step i - 1 at [i & 1]
  __shared__ int32_t slo_s[kListWindow + 1], shi_s[kListWindow + 1];  // this CTA's slice of each
                                       // slot's list, and of all n columns
  __shared__ int32_t pre_s[2];         // groups of the current step issued ahead, and their list key
  __shared__ uint32_t cd_s[kListWindow];  // work-list lengths of the slots (fixed per launch)
  __shared__ int32_t nx_s[4];          // predicted next list: groups, key, length, sampled
  __shared__ int32_t nxlo_s;           // ... and its first index
  __shared__ int32_t wlkey_s;          // slot of the coefficient slice copied ahead (-2: none)
  __shared__ double zdx_s;             // this CTA's share of z·dx
  __shared__ double sum_s[2];          // Σ over the CTAs of Σ α_k t_k, and z·dx

  // The launch is a programmatic dependent of the grid before it: its CTAs start on the SMs that
  // grid leaves and wait for it to complete before touching global memory.  Every CTA of this
  // grid is resident by the time it lets the next grid be scheduled (one CTA per SM), so the
  // exchanges below cannot starve.
  griddep_launch_dependents();
  if (t == 0) {
    for (int s = 0; s < NS; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  __syncthreads();
  griddep_wait();

  // epochs of this launch: ep0 + 1 for its first step; CTA 0 leaves a fresh start on the way out
  if (t <= kListWindow) {  // T >= 32 > kListWindow
    const uint32_t total = t < kListWindow ? __ldg(b.wl_count + t) : (uint32_t)b.n;
    if (t < kListWindow) cd_s[t] = total;
    slo_s[t] = (int32_t)((int64_t)q * total / G);
    shi_s[t] = (int32_t)((int64_t)(q + 1) * total / G);
  }
  if (t == 0) {
    st_s = b.st[a.iter & 1];
    ep0_s = *reinterpret_cast<const volatile uint32_t*>(b.epoch);
    iss_s = 0u;
    scale_s[a.iter & 1] = st_s.scale;
    mode_s[a.iter & 1] = st_s.mode;
    used_s[a.iter & 1] = st_s.used;
    le_s[a.iter & 1] = st_s.last_exact;
    memo_s[a.iter & 1] = st_s.memo_zero ? 0 : 1;
    lam_s[a.iter & 1] = st_s.lam_prev;
    pre_s[0] = 0;
    pre_s[1] = -2;
    wlkey_s = -2;
    zdx_s = 0.0;
  }
  // the owned packets [p0, p1): packet p holds values 3·(p / T) .. +2 of thread p % T, whose
  // value v is row (p % T + (v / E)·T)·E + v % E
  const int NPT = NP * T;
  struct Geo {  // the exchange's sizes: read from shared memory where they are used
    int32_t own_n, blk, p0, npk, rec_warps;
    uint32_t own_div;  // p / own_n = umulhi(p, own_div) for p < 2^16, own_n > 1
  };
  __shared__ Geo geo_s;
  const volatile Geo& geo = geo_s;
  if (t == 0) {
    Geo x;
    x.own_n = step_owned_max(g);
    x.blk = step_block(g);
    x.p0 = min(NPT, q * x.own_n);
    x.npk = min(NPT, x.p0 + x.own_n) - x.p0;
    x.rec_warps = x.own_n > 32 ? 2 : 1;
    x.own_div = (uint32_t)((0x100000000ull + x.own_n - 1) / x.own_n);
    geo_s = x;
  }
  __syncthreads();
  auto packet_row = [&](int p, int e) -> int {
    const int v = 3 * (p / T) + e, vi = p % T + (v / E) * T;
    return (v < NV && vi < nvec) ? vi * E + v % E : -1;
  };
  constexpr int kOwn = kOwnBytes / 4;  // words of an owned packet's record
  for (int k = t, npk = geo.npk, p0 = geo.p0; k < npk; k += T) {
    int mask = 0;
    for (int e = 0; e < 3; ++e) mask |= packet_row(p0 + k, e) >= 0 ? 1 << e : 0;
    mask |= (NV - 3 * ((p0 + k) / T)) << 8;  // values of the packet (3 or more: full)
    own[kOwn * k + 15] = __int_as_float(mask);
  }
  for (int k = t, npk = geo.npk, p0 = geo.p0; k < 3 * npk; k += T) {
    const int row = packet_row(p0 + k / 3, k % 3);
    float* o = own + kOwn * (k / 3) + k % 3;
    reinterpret_cast<double*>(own + kOwn * (k / 3) + 16)[k % 3] =
        row >= 0 && b.has_vstar ? __ldcg(b.vstar + row) : 0.0;
    o[0] = row >= 0 ? __ldcg(b.y[(a.iter + 1) & 1] + row) : 0.f;
    o[3] = row >= 0 ? __ldcg(b.x_memo + row) : 0.f;
    o[6] = row >= 0 ? __ldcg(b.y_memo + row) : 0.f;
    o[9] = row >= 0 ? __ldcg(b.v + row) : 0.f;
    o[12] = row >= 0 ? __ldcg(b.z + row) : 0.f;
  }
  uint4* const ll1 = b.pk_part;                              // [G][NPT + 2]
  const size_t ll1_stride = (size_t)NPT + 2;
  // x_memo of this thread's rows: the context's copy until the launch's first variance-reduction
  // step, then this CTA's own (each thread reads back what it wrote)
  auto xm_at = [&](int memo) -> float* {
    return memo == 2 ? b.partials + (size_t)q * m : b.x_memo;
  };

  // a vector's rows of this thread from row-ordered global memory
  auto load_rows = [&](const float* src, float2 (&o)[R][H]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int vi = t + r * T;
#pragma unroll
      for (int h4 = 0; h4 < E / 4; ++h4) {
        const float4 v = vi < nvec ? __ldcg(reinterpret_cast<const float4*>(src) + vi * (E / 4) + h4)
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
        o[r][2 * h4] = make_float2(v.x, v.y);
        o[r][2 * h4 + 1] = make_float2(v.z, v.w);
      }
    }
  };
  auto store_rows = [&](float* dst, const float2 (&o)[R][H]) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int vi = t + r * T;
      if (vi < nvec) {
#pragma unroll
        for (int h4 = 0; h4 < E / 4; ++h4)
          reinterpret_cast<float4*>(dst)[vi * (E / 4) + h4] =
              make_float4(o[r][2 * h4].x, o[r][2 * h4].y, o[r][2 * h4 + 1].x, o[r][2 * h4 + 1].y);
      }
    }
  };
  // value v of a thread's rows (v is a compile-time constant after unrolling)
  auto val = [](float2 (&o)[R][H], int v) -> float& {
    float2& f = o[v / E][(v % E) / 2];
    return (v & 1) ? f.y : f.x;
  };
  // packets [k0, k0 + kBatch) of a thread into its rows
  auto unpack_rows = [&](const uint4 (&pk)[kBatch], int k0, float2 (&o)[R][H]) {
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int v = 3 * (k0 + k);
      if (v + 2 < NV) {
        val(o, v) = __uint_as_float(pk[k].x);
        val(o, v + 1) = __uint_as_float(pk[k].y);
        val(o, v + 2) = __uint_as_float(pk[k].z);
      } else if (v + 1 < NV) {  // (x, y, y)
        val(o, v) = __uint_as_float(pk[k].x);
        val(o, v + 1) = __uint_as_float(pk[k].y & pk[k].z);
      } else if (v < NV) {  // (x, x, x)
        val(o, v) = __uint_as_float(pk[k].x & pk[k].y & pk[k].z);
      }
    }
  };

  // Stage ring: group number `pos` (counted over the whole launch) lives in stage pos % NS and
  // completes phase (pos / NS) of that stage's barrier; (s_cur, ph_cur) are the stage and phase
  // parity of the current step's first group.  One warp issues: lane 0 announces each group's
  // bytes, then the lanes issue one column each.  A stage is refilled once every thread is past
  // the group that last used it (a CTA barrier).
  const int iw = ncw - 1;  // the issuing warp
  // columns [k0, k1) of a list (shared memory; null: columns first + k), k0 a multiple of GC, as
  // groups from stage s on
  auto issue = [&](int s, int k0, int k1, const uint32_t* cols, int first) {
    if (lane == 0) {
      int sg = s;
      for (int k = k0; k < k1; k += GC) {
        mbar_arrive_expect_tx(&full[sg], (uint32_t)min(GC, k1 - k) * col_bytes);
        sg = sg + 1 == NS ? 0 : sg + 1;
      }
    }
    __syncwarp();
    const uint64_t policy = l2_evict_first_policy();
    const unsigned char* Abase = reinterpret_cast<const unsigned char*>(b.A);
    for (int k = k0 + lane; k < k1; k += 32) {
      int sg = s + (k - k0) / GC;
      sg = sg >= NS ? sg - NS : sg;
      const uint32_t col = cols ? cols[k] : (uint32_t)(first + k);
      bulk_g2s(stages + ((size_t)sg * GC + (k - k0) % GC) * col_bytes,
               Abase + (size_t)col * ((size_t)b.ld * sizeof(Elem)), col_bytes, &full[sg], policy);
    }
    if (lane == 0) iss_s += (uint32_t)((k1 - k0 + GC - 1) / GC);
  };
  int s_cur = 0;
  uint32_t ph_cur = 0;
  auto advance = [&](int k) {  // k <= NS groups on
    s_cur += k;
    if (s_cur >= NS) {
      s_cur -= NS;
      ph_cur ^= 1u;
    }
  };
  bool ok = true;
  // on the way out: no copy may still be landing in this CTA's shared memory (the last NS issued
  // groups cover every stage; waits are bounded), and CTA 0 leaves the next launch its epochs
  auto leave = [&](bool failed, int ran) {  // ran: steps begun
    if (warp == iw && lane == 0) {
      const uint32_t issued = iss_s;
      for (uint32_t p = issued > (uint32_t)NS ? issued - (uint32_t)NS : 0u; p < issued; ++p)
        mbar_wait_bounded(&full[p % (uint32_t)NS], (p / (uint32_t)NS) & 1u);
      if (failed) atomicOr(b.status, (uint32_t)kDevTimeout);
      // (a CTA is at most one step ahead of another, and each has read its first epoch before CTA 0 is past
      // its first step; a launch that runs no step uses no epoch)
      if (q == 0) *b.epoch = ep0_s + (uint32_t)ran + 4u;
    }
  };

  // ---- everything step j needs that does not depend on the product of the step before ----
  // dx = x_j − x_memo on this thread's rows (x_j = scale·y_{j−1}, FP32 multiply; `yv` holds
  // y_{j-1}, `xm` x_memo) and Σdx over all rows; this CTA's share of z·dx (dots,
  // common.h:55-87); the coefficient slice of the step's list; and the list predicted for step
  // j+1 (exact unless the adaptive VR switch, which needs step j's cosine, changes the kind).
  float2 dx[R][H];
  float2 xv[kShares ? 1 : R][H];  // x_j, where the Rayleigh sums are formed from all rows
  double sum_dx = 0.0;
  auto prepare = [&](int j, int jmode, int jused, int jlast_exact, int jmemo, float jscale,
                     double jcos, float2 (&yv)[R][H], float2 (&xm)[R][H]) {
    const bool jamm = jmode == kPrevious || jmode == kProposed;
    const bool jcentred = jmode == kProposed;
    const bool jsampled = jamm && !cc.sanity;
    const int jslot = jused % kListWindow;
    if (warp == (ncw > 2 ? 2 : 0) && jcentred) {
      double zp = 0.0;
      for (int k = lane, npk = geo.npk; k < npk; k += 32) {
        const float* o = own + kOwn * k;
#pragma unroll
        for (int e = 0; e < 3; ++e)
          zp = fma((double)__fsub_rn(__fmul_rn(jscale, o[e]), o[3 + e]), (double)o[12 + e], zp);
      }
      zp = warp_sum(zp);
      if (lane == 0) zdx_s = zp;
    }
    // the coefficient slice, unless copied ahead on the right prediction (the warps after warp
    // 0, all of a one-warp CTA)
    if (jamm && !(jsampled && wlkey_s == jslot)) {
      const int jl = jsampled ? jslot : kListWindow, jlo = slo_s[jl], jnb = shi_s[jl] - jlo;
      cp_async_wait_all();  // no copy ahead may still land in wl_*
      const int t1 = T > 32 ? t - 32 : t, T1 = T > 32 ? T - 32 : T;
      for (int k = t1; k >= 0 && k < jnb; k += T1) {
        if (jsampled) {
          wl_idx[k] = __ldg(b.wl_col[jslot] + jlo + k);
          wl_w[k] = __ldg(b.wl_wm[jslot] + jlo + k);
          wl_al[k] = __ldg(b.wl_al[jslot] + jlo + k);
        } else {  // sanity mode: identity list, weight 1
          wl_w[k] = 1.0f;
          wl_al[k] = __ldg(b.alpha + jlo + k);
        }
      }
    }
    if (warp == (ncw > 1 ? 1 : 0)) {
      int groups = 0, nkey = -2, nnb = 0, nsmp = 0, nlo = 0;
      if (j + 1 < a.iter_end) {
        int le;
        const int nmode = decide_mode(cc, j + 1, jcos, jlast_exact, &le);
        const int nslot = (jused + (jsampled ? 1 : 0)) % kListWindow;
        nsmp = ((nmode == kPrevious || nmode == kProposed) && !cc.sanity) ? 1 : 0;
        const int nl = nsmp ? nslot : kListWindow;
        nlo = slo_s[nl];
        nnb = shi_s[nl] - nlo;
        groups = (nnb + GC - 1) / GC;
        nkey = nsmp ? nslot : -1;
        if (nsmp) {
          const int nf = min(NS * GC, nnb);
          for (int k = lane; k < nf; k += 32) cp_async4(nxt_cols + k, b.wl_col[nslot] + nlo + k);
        }
      }
      if (lane == 0) {
        nx_s[0] = groups;
        nx_s[1] = nkey;
        nx_s[2] = nnb;
        nx_s[3] = nsmp;
        nxlo_s = nlo;
      }
    }
    const bool sub = jamm && jmemo != 0;
    if (!kXmAhead && sub) load_rows(xm_at(jmemo), dx);
    double sdx = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float2 xs = kXmAhead ? xm[r][h] : dx[r][h];
        const float x0 = sub ? xs.x : 0.f, x1 = sub ? xs.y : 0.f;
        const float2 xj = make_float2(__fmul_rn(jscale, yv[r][h].x), __fmul_rn(jscale, yv[r][h].y));
        const float d0 = __fsub_rn(xj.x, x0), d1 = __fsub_rn(xj.y, x1);
        dx[r][h] = make_float2(d0, d1);
        if constexpr (!kShares) xv[r][h] = xj;
        if (jcentred) sdx += (double)d0 + (double)d1;
      }
    }
    sum_dx = 0.0;
    if (jcentred) {  // Σdx over all m rows (dots, common.h:55-87), identical in every CTA
      sdx = warp_sum(sdx);
      if (lane == 0) sdx_s[warp] = sdx;
      __syncthreads();
      for (int w = 0; w < ncw; ++w) sum_dx += sdx_s[w];
    }
  };
  __syncthreads();  // st_s, the slices, own
  bool done = st_s.done != 0;
  if (a.iter < a.iter_end && !done) {  // uniform over the grid
    float2 yv[R][H], xm[R][H];
    load_rows(b.y[(a.iter + 1) & 1], yv);
    if constexpr (kXmAhead) load_rows(b.x_memo, xm);
    const int p = a.iter & 1;
    prepare(a.iter, mode_s[p], used_s[p], le_s[p], memo_s[p], scale_s[p], st_s.cos_prev, yv, xm);
  }
  cp_async_wait_all();
  __syncthreads();

  int i = a.iter;
  for (; i < a.iter_end && !done; ++i) {
    const int mode = mode_s[i & 1], slot = used_s[i & 1] % kListWindow;
    const bool amm = mode == kPrevious || mode == kProposed;
    const bool centred = mode == kProposed;
    const bool sampled = amm && !cc.sanity;
    const int key = sampled ? slot : -1;  // which columns the step reads

    // ---- this CTA's column list: a contiguous slice of the sorted work list ----------------
    const int lo = slo_s[sampled ? slot : kListWindow];
    const int nb = shi_s[sampled ? slot : kListWindow] - lo;
    if (sampled && q == 0 && t == 0) b.distinct_hist[i] = (int32_t)cd_s[slot];
    const int ngroups = (nb + GC - 1) / GC;

    // the groups of this step already in the ring (issued at the end of the previous step on the
    // predicted list, or left there by it); a misprediction is drained and the ring moves on.  No
    // thread may wait for a new group before the drain is over: where the drained groups filled the
    // ring, a new one takes the stage of one still landing, and a wait for that stage's next phase
    // would see the phase before it complete and go through at once.
    int pre = 0;
    {
      const int pn = pre_s[0];
      if (pn > 0) {
        if (pre_s[1] == key) {
          pre = pn;
        } else {
          bool drained = true;
          if (warp == iw && lane == 0) {
            int sg = s_cur;
            uint32_t ph = ph_cur;
            for (int k = 0; k < pn && drained; ++k) {
              drained = mbar_wait_bounded(&full[sg], ph);
              if (++sg == NS) {
                sg = 0;
                ph ^= 1u;
              }
            }
          }
          if (named_barrier_or(1, T, !drained)) {
            leave(true, i - a.iter + 1);
            return;
          }
          advance(pn);
        }
      }
    }
    if (warp == iw && ngroups > pre) {  // the first NS groups not already in flight
      int sg = s_cur + pre;
      sg = sg >= NS ? sg - NS : sg;
      issue(sg, pre * GC, min(NS * GC, nb), sampled ? wl_idx : nullptr, lo);
    }

    float2 yacc[R][H];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int h = 0; h < H; ++h) yacc[r][h] = make_float2(0.f, 0.f);
    const float sum_dx_f = (float)sum_dx;

    const uint32_t stage_bytes = (uint32_t)GC * col_bytes;
    // guarded partial dots of a group of cnt columns in stage s
    auto dot_group = [&](int cnt, int s, float (&d)[GC]) {
      const unsigned char* sb = stages + (size_t)s * stage_bytes;
#pragma unroll
      for (int qq = 0; qq < GC; ++qq) {
        d[qq] = 0.f;
        if (qq < cnt) {
          const uint4* col = reinterpret_cast<const uint4*>(sb + (size_t)qq * col_bytes);
          float2 pa = make_float2(0.f, 0.f), pb = make_float2(0.f, 0.f);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const int vi = t + r * T;
            if (vi < nvec) {
              float2 av[H];
              unpack2(col[vi], av);
#pragma unroll
              for (int h = 0; h < H; h += 2) {
                pa = fma2(av[h], dx[r][h], pa);
                if (h + 1 < H) pb = fma2(av[h + 1], dx[r][h + 1], pb);
              }
            }
          }
          d[qq] = (pa.x + pa.y) + (pb.x + pb.y);
        }
      }
    };
    // y += coef · A of one column over this thread's rows
    auto axpy_col = [&](int qq, int s, float coef) {
      const uint4* col =
          reinterpret_cast<const uint4*>(stages + (size_t)s * stage_bytes + (size_t)qq * col_bytes);
      const float2 c2 = make_float2(coef, coef);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int vi = t + r * T;
        if (vi < nvec) {
          float2 av[H];
          unpack2(col[vi], av);
#pragma unroll
          for (int h = 0; h < H; ++h) yacc[r][h] = fma2(c2, av[h], yacc[r][h]);
        }
      }
    };
    // this warp's sums of the group's dots, to slot `buf` of redw ([warp][GC])
    auto publish = [&](int cnt, int buf, float (&d)[GC]) {
      float* slotp = redw + (buf * kMaxWarps + warp) * GC;
      if constexpr (GC >= 2) {
        const float r = warp_reduce_multi<float, GC>(d, lane);
        constexpr int LL = 32 / GC;
        const int qv = lane / LL;
        if (lane % LL == 0 && qv < cnt) slotp[qv] = r;
      } else {
        const float v = warp_sum(d[0]);
        if (lane == 0) slotp[0] = v;
      }
    };
    // coefficient of column k of the slice from its dot
    float sacc = 0.f;  // Σ α_k t_k (proposed)
    auto coef_of = [&](int k, float tot) -> float {
      if (!amm) return tot;
      if (centred) {
        const float al = wl_al[k];
        const float tq = __fmul_rn(__fsub_rn(tot, __fmul_rn(al, sum_dx_f)), wl_w[k]);
        sacc = fmaf(al, tq, sacc);
        return tq;
      }
      return __fmul_rn(tot, wl_w[k]);
    };

    if (ngroups <= NS) {
      // ---- a resident slice: all dots, one reduction, all axpys ----
      int s = s_cur;
      uint32_t ph = ph_cur;
      for (int grp = 0; grp < ngroups && ok; ++grp) {
        ok = mbar_wait_bounded(&full[s], ph);
        if (++s == NS) {
          s = 0;
          ph ^= 1u;
        }
      }
      s = s_cur;
#pragma unroll 1
      for (int grp = 0; grp < ngroups; ++grp) {
        const int cnt = min(GC, nb - grp * GC);
        float d[GC];
        dot_group(cnt, s, d);
        publish(cnt, grp, d);
        if (++s == NS) s = 0;
      }
      if (named_barrier_or(1, T, !ok)) ok = false;
      if (warp == 0 && ok) {
        for (int k = lane; k < nb; k += 32) {
          const float* base = redw + (k / GC) * kMaxWarps * GC + k % GC;
          float tot = base[0];
          for (int w = 1; w < ncw; ++w) tot += base[w * GC];
          coef_s[k] = coef_of(k, tot);
        }
        if (centred) sacc = warp_sum(sacc);  // (thread 0 sends it)
      }
      __syncthreads();
      if (ok) {
        s = s_cur;
        for (int grp = 0; grp < ngroups; ++grp) {
          const int cnt = min(GC, nb - grp * GC);
#pragma unroll
          for (int qq = 0; qq < GC; ++qq)
            if (qq < cnt) axpy_col(qq, s, coef_s[grp * GC + qq]);
          if (++s == NS) s = 0;
        }
      }
    } else {
      // ---- pipelined group loop ----
      float dn[GC];
      ok = mbar_wait_bounded(&full[s_cur], ph_cur);
      if (ok) {
        dot_group(min(GC, nb), s_cur, dn);
        publish(min(GC, nb), 0, dn);
      }
      if (named_barrier_or(1, T, !ok)) ok = false;
      for (int grp = 0; ok && grp < ngroups; ++grp) {
        const int cnt = min(GC, nb - grp * GC);
        float coef[GC], tots[GC];
        // coefficients of this group (every warp sums the warp partials in the same order)
        warps_sum<GC>(redw + (grp & 1) * kMaxWarps * GC, ncw, lane, tots);
#pragma unroll
        for (int qq = 0; qq < GC; ++qq) coef[qq] = qq < cnt ? coef_of(grp * GC + qq, tots[qq]) : 0.f;
        const bool more = grp + 1 < ngroups;
        const int cnt_n = more ? min(GC, nb - (grp + 1) * GC) : 0;
        const int s_nxt = s_cur + 1 == NS ? 0 : s_cur + 1;
        const uint32_t ph_nxt = s_nxt == 0 ? ph_cur ^ 1u : ph_cur;
        if (more && !mbar_wait_bounded(&full[s_nxt], ph_nxt)) ok = false;
        const unsigned char* sb = stages + (size_t)s_cur * stage_bytes;
        if (full_slots && cnt == GC && (!more || cnt_n == GC) && ok) {
          const unsigned char* sn = more ? stages + (size_t)s_nxt * stage_bytes : sb;
          if (more) {
            if (T == 512)
              fused_block<Elem, R, GC, true, 512>(sb, sn, col_bytes, t, T, coef, dx, yacc, dn);
            else
              fused_block<Elem, R, GC, true, 0>(sb, sn, col_bytes, t, T, coef, dx, yacc, dn);
          } else {
            if (T == 512)
              fused_block<Elem, R, GC, false, 512>(sb, sb, col_bytes, t, T, coef, dx, yacc, dn);
            else
              fused_block<Elem, R, GC, false, 0>(sb, sb, col_bytes, t, T, coef, dx, yacc, dn);
          }
        } else if (ok) {
          if (more) dot_group(cnt_n, s_nxt, dn);
#pragma unroll
          for (int qq = 0; qq < GC; ++qq)
            if (qq < cnt) axpy_col(qq, s_cur, coef[qq]);
        }
        if (more && ok) publish(cnt_n, (grp + 1) & 1, dn);
        // partials of grp+1 published; every thread is done with stage grp: the issuing warp refills it
        if (named_barrier_or(1, T, !ok)) ok = false;
        if (warp == iw && ok && grp + NS < ngroups) {
          const int c0 = (grp + NS) * GC;
          issue(s_cur, c0, min(c0 + GC, nb), sampled ? wl_idx : nullptr, lo);
        }
        s_cur = s_nxt;
        ph_cur = ph_nxt;
      }
    }
    if (!ok) {
      leave(true, i - a.iter + 1);
      return;
    }
    // The next step's first groups go out now.  A step that reads all columns after one that did,
    // on a slice that fits the ring, finds them in place.  Otherwise every stage is free (past
    // one more barrier for a resident slice): all groups of a slice that fits the ring, else two
    // (about 128 KB per CTA; measured on the B200 at m = 16384: a third one slows the packet
    // writes that follow by more than it saves).
    const int ngn = nx_s[0], nkey = nx_s[1];
    const bool stay = ngroups <= NS && key == -1 && nkey == -1 && ngn == ngroups;
    if (!stay) {
      if (ngroups <= NS) {
        __syncthreads();
        advance(ngroups);
      }
      if (warp == iw) {
        const int groups = ngn <= NS ? ngn : kPrefetchGroups;
        if (groups > 0)
          issue(s_cur, 0, min(groups * GC, nx_s[2]), nx_s[3] ? nxt_cols : nullptr, nxlo_s);
        if (lane == 0) {
          pre_s[0] = groups;
          pre_s[1] = nkey;
        }
      }
    } else if (warp == iw && lane == 0) {
      pre_s[0] = ngroups;
      pre_s[1] = -1;
    }

    // ---- 1. this CTA's partial y and its scalars, as packets ----
    const uint32_t ep = ep0_s + (uint32_t)(i - a.iter) + 1u;
    {
      uint4* out = ll1 + (size_t)q * ll1_stride + t;
#pragma unroll
      for (int k = 0; k < NP; ++k)
        packet_store(out + k * T, val(yacc, 3 * k), 3 * k + 1 < NV ? val(yacc, 3 * k + 1 < NV ? 3 * k + 1 : 0) : 0.f,
                     3 * k + 2 < NV ? val(yacc, 3 * k + 2 < NV ? 3 * k + 2 : 0) : 0.f, ep);
      if (t == 0) {
        const double zd = centred ? zdx_s : 0.0;
        packet_store(out + NPT + (i & 1), sacc, __int_as_float(__double2loint(zd)),
                     __int_as_float(__double2hiint(zd)), ep);
      }
    }
    if (sampled) {
      // The picks are consumed: their histogram entries and chunk totals are cleared for the
      // next draw into this slot (several CTAs may zero one chunk total: the same value).
      const int cs = b.chunk_shift;
      uint32_t* cnt = b.count[slot];
      uint32_t* chk = b.chunk[slot];
      for (int k = t; k < nb; k += T) {
        const uint32_t col = wl_idx[k];  // written before the barriers of the product
        cnt[col] = 0u;
        chk[col >> cs] = 0u;
      }
    }
    // ---- 2. the owned packets from every CTA: thread t reads packet p0 + t % npk of CTAs
    // t / npk, t / npk + S, ... (S = T / npk), sums in FP64 and stages the sums ----
    const float scale = scale_s[i & 1];
    const int npk = geo.npk, p0 = geo.p0, own_n = geo.own_n, blk = geo.blk;
    const int rec_warps = geo.rec_warps;
    if (npk > 0) {
      const int S = T / npk, pa = t % npk, ps = t / npk;
      if (ps < S) {
        double sx = 0.0, sy = 0.0, sz = 0.0;
        const uint4* src = ll1 + p0 + pa;
        constexpr int U = 6;
        for (int j = ps; j < G && ok; j += S * U) {
          uint4 v[U];
          const int cnt = (G - j + S - 1) / S;
          ok = packets_wait<U>(src + (size_t)j * ll1_stride, (size_t)S * ll1_stride, cnt, ep, v);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (u >= cnt) break;
            sx += (double)__uint_as_float(v[u].x);
            sy += (double)__uint_as_float(v[u].y);
            sz += (double)__uint_as_float(v[u].z);
          }
        }
        red[t] = sx;
        red[T + t] = sy;
        red[2 * T + t] = sz;
      }
    }
    if (centred && warp == ncw - 1) {  // the CTAs' scalars, summed lane-strided, then a butterfly
      double sa = 0.0, sz = 0.0;
      constexpr int U = 5;
      for (int j = lane; j < G && ok; j += 32 * U) {
        uint4 v[U];
        const int cnt = (G - j + 31) / 32;
        ok = packets_wait<U>(ll1 + (size_t)j * ll1_stride + NPT + (i & 1), 32 * ll1_stride, cnt,
                             ep, v);
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u < cnt) {
            sa += (double)__uint_as_float(v[u].x);
            sz += __hiloint2double((int)v[u].z, (int)v[u].y);
          }
      }
      __syncwarp();
      sa = warp_sum(sa);
      sz = warp_sum(sz);
      if (lane == 0) {
        sum_s[0] = sa;
        sum_s[1] = sz;
      }
    }
    // (past this barrier no thread of the CTA reads wl_* of this step any more)
    if (named_barrier_or(1, T, !ok)) {
      leave(true, i - a.iter + 1);
      return;
    }
    if (warp < rec_warps) {
      // L lanes per owned packet in warp 0, or one thread per packet when there are more than 32
      int Lp = 1;
      if (rec_warps == 1 && npk > 0)
        while (2 * Lp * npk <= 32) Lp *= 2;
      const int pa = t / Lp, l = t % Lp;
      double sum[3] = {0.0, 0.0, 0.0};
      if (pa < npk) {
        const int S = T / npk;
        for (int s = l; s < S; s += Lp)
#pragma unroll
          for (int e = 0; e < 3; ++e) sum[e] += red[e * T + s * npk + pa];
      }
      for (int off = Lp / 2; off > 0; off >>= 1)
#pragma unroll
        for (int e = 0; e < 3; ++e) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], off);
      float* o = own + kOwn * (pa < npk ? pa : 0);
      float yo[3] = {0.f, 0.f, 0.f};
      if (pa < npk) {  // (all L lanes hold the sums; the first writes)
        const double S_a = centred ? sum_s[0] : 0.0, zdx = centred ? sum_s[1] : 0.0;
        const int mask = __float_as_int(o[15]);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const double tv = sum[e];
          if (!amm) {
            yo[e] = (float)tv;
          } else if (!centred) {  // previous: y_memo + A_S·tmp (core_previousAMM.cuh:225-232)
            yo[e] = (float)((double)o[6 + e] + tv);
          } else {
            // y_memo + Σdx·v + z·dx in FP64, rounded (core_proposedAMM.cuh:198-212)
            const float base = (float)(fma(sum_dx, (double)o[9 + e], zdx) + (double)o[6 + e]);
            yo[e] = (float)((double)base + (tv - S_a));
          }
          if (!(mask >> e & 1)) yo[e] = 0.f;  // past row m, or no value at all
        }
        // (values past the thread's last one repeat it, see packets)
        const int left = mask >> 8;
        const float y1 = left > 1 ? yo[1] : yo[0], y2 = left > 2 ? yo[2] : y1;
        if (l == 0) packet_store(b.pk_y + (size_t)q * blk + pa, yo[0], y1, y2, ep);
      }
      __syncwarp();  // every lane has read its packet's record
      double xy = 0.0, yy = 0.0, yd = 0.0;
      if (pa < npk && l == 0) {
        const double* vs = reinterpret_cast<const double*>(o + 16);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const float xa = __fmul_rn(scale, o[e]);
          if constexpr (kShares) {  // (dotProduct_and_generate_x, common.h:103-153)
            const double yd0 = (double)yo[e];
            xy = fma(yd0, (double)xa, xy);
            yy = fma(yd0, yd0, yy);
            if (b.has_vstar) yd = fma(yd0, vs[e], yd);
          }
          if (mode == kExactMemo) {
            o[3 + e] = xa;
            o[6 + e] = yo[e];
          }
          o[e] = yo[e];
        }
      }
      if constexpr (kShares) {
        __syncwarp();
        xy = warp_sum(xy);
        yy = warp_sum(yy);
        if (b.has_vstar) yd = warp_sum(yd);
        if (lane == 0) {
          uint4* out = b.pk_y + (size_t)q * blk + own_n + 3 * (kShareWarps * (i & 1) + warp);
          packet_store(out, xy, ep);
          packet_store(out + 1, yy, ep);
          if (b.has_vstar) packet_store(out + 2, yd, ep);
        }
      }
    }
    if (i + 1 < a.iter_end && (T == 32 || warp > 0)) {
      // the coefficient slice of the predicted next list, copied ahead (checked in prepare)
      const bool smp = nx_s[3] != 0;
      const int t1 = T > 32 ? t - 32 : t, T1 = T > 32 ? T - 32 : T;
      if (smp) {
        const int nslot = nx_s[1];
        const int64_t nlo = nxlo_s;
        const int nnb = nx_s[2];
        for (int k = t1; k < nnb; k += T1) {
          cp_async4(wl_idx + k, b.wl_col[nslot] + nlo + k);
          cp_async4(wl_w + k, b.wl_wm[nslot] + nlo + k);
          cp_async4(wl_al + k, b.wl_al[nslot] + nlo + k);
        }
      }
      if (t1 == 0) wlkey_s = smp ? nx_s[1] : -2;
    }

    // ---- 3. y of this thread's rows; the shares, summed in every CTA alike; λ and the next
    // step's state ----
    float2 yv[R][H], xm[R][H];
    const uint4* const ll2 = b.pk_y;
    const uint32_t own_div = geo.own_div;
#pragma unroll
    for (int k0 = 0; k0 < NP; k0 += kBatch) {
      uint4 pk[kBatch];
      int off[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        const int p = min((k0 + k) * T + t, NPT - 1);
        const int o = own_n == 1 ? p : (int)__umulhi((uint32_t)p, own_div);
        off[k] = o * blk + (p - o * own_n);
      }
      ok = packets_wait_at<kBatch>(ll2, off, NP - k0, ep, pk) && ok;
      unpack_rows(pk, k0, yv);
    }
    int memo = memo_s[i & 1];
    if (mode == kExactMemo) {
      memo = 2;
      store_rows(xm_at(2), dx);  // dx = x in an exact step
      if (q == 0) {  // for the next launch
        store_rows(b.x_memo, dx);
        store_rows(b.y_memo, yv);
      }
    }
    if (kXmAhead && memo && cc.uses_amm) load_rows(xm_at(memo), xm);
    // the Rayleigh sums (dotProduct_and_generate_x, common.h:103-153), alike in every CTA
    double xy = 0.0, yy = 0.0, yd = 0.0;
    const int nrec = rec_warps * G;
    if constexpr (kShares) {
      auto records = [&](const uint4* p) -> double {  // this thread's records
        double d = 0.0;
        for (int r = t; r < nrec && ok; r += T) {
          uint4 v[1];
          const int w = r >= G ? 1 : 0;
          ok = packets_wait<1, true>(p + (r - w * G) * blk + 3 * (kShareWarps * (i & 1) + w), 0, 1,
                                     ep, v);
          d += __hiloint2double((int)v[0].y, (int)v[0].x);
        }
        return d;
      };
      xy = records(ll2 + own_n);
      yy = records(ll2 + own_n + 1);
      if (b.has_vstar) yd = records(ll2 + own_n + 2);
      __syncwarp();
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const double y0 = (double)yv[r][h].x, y1 = (double)yv[r][h].y;
          xy = fma(y0, (double)xv[r][h].x, xy);
          xy = fma(y1, (double)xv[r][h].y, xy);
          yy = fma(y0, y0, yy);
          yy = fma(y1, y1, yy);
        }
      if (b.has_vstar) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int vi = t + r * T;
          if (vi < nvec) {
#pragma unroll
            for (int e = 0; e < E; ++e)
              yd = fma((double)val(yv, r * E + e), __ldg(b.vstar + (size_t)vi * E + e), yd);
          }
        }
      }
    }
    if (!kShares || 32 * warp < nrec) {
      xy = warp_sum(xy);
      yy = warp_sum(yy);
      if (b.has_vstar) yd = warp_sum(yd);
    }
    if (lane == 0) {
      scr[4 * warp + 0] = xy;
      scr[4 * warp + 1] = yy;
      scr[4 * warp + 2] = yd;
    }
    if (named_barrier_or(1, T, !ok)) {
      leave(true, i - a.iter + 1);
      return;
    }
    // every warp forms the state of the next step (next_state) from the same sums
    xy = lane < ncw ? scr[4 * lane + 0] : 0.0;
    yy = lane < ncw ? scr[4 * lane + 1] : 0.0;
#pragma unroll
    for (int off = kMaxWarps / 2; off > 0; off >>= 1) {
      xy += __shfl_xor_sync(0xffffffffu, xy, off);
      yy += __shfl_xor_sync(0xffffffffu, yy, off);
    }
    xy = __shfl_sync(0xffffffffu, xy, 0);  // (lanes 16.. summed nothing)
    yy = __shfl_sync(0xffffffffu, yy, 0);
    const double rs = rsqrt(yy), cosv = xy * rs, lam_prev = lam_s[i & 1];
    const float nscale = (float)rs;
    const int nused = used_s[i & 1] + (amm && !cc.sanity ? 1 : 0);
    done = !isfinite(xy) || !isfinite(rs);
    if (cc.tol > 0.0 && i >= 1 && fabs(xy - lam_prev) <= cc.tol * fabs(xy)) done = true;
    int nle;
    const int nmode = decide_mode(cc, i + 1, cosv, le_s[i & 1], &nle);
    if (i + 1 < a.iter_end && !done) {
      prepare(i + 1, nmode, nused, nle, memo, nscale, cosv, yv, xm);
    } else if (q == 0) {
      store_rows(b.y[i & 1], yv);  // the last step of the launch: y for what runs next
    }
    if (t == 0) {
      const int p = (i + 1) & 1;
      scale_s[p] = nscale;
      mode_s[p] = nmode;
      used_s[p] = nused;
      le_s[p] = nle;
      memo_s[p] = memo;
      lam_s[p] = xy;
    }
    if (q == 0 && t == T - 1) {  // the trace, and the state as the next launch reads it
      yd = 0.0;
      for (int w = 0; w < ncw; ++w) yd += scr[4 * w + 2];
      IterState cur = st_s;
      StepScalars sc;
      st_s = next_state(cc, i, cur, xy, yy, yd, &sc);
      record_step(b, cc, i, cur, sc);
    }
    cp_async_wait_all();  // the slice and the next-list indices copied ahead
    __syncthreads();  // the next step's state, wl_*, nx_s, wlkey_s, pre_s
  }
  // past the last step of the launch (or the early stop): the state the next launch (or the
  // call's end) reads, and no copy still in flight
  leave(false, i - a.iter);
  __syncthreads();
  if (q == 0 && t == 0) b.st[a.iter_end & 1] = st_s;
}

// ------------------------------------------------------------------------------------------
// Launch
// ------------------------------------------------------------------------------------------
using StepFn = void (*)(StepArgs);

static StepFn pick_step(int dtype, int R, int GC) {
#define AMM_PICK(EL, RR, GG) \
  if (R == RR && GC == GG) return step_kernel<EL, RR, GG>;
  if (dtype == 1) {
    AMM_PICK(__nv_bfloat16, 1, 8)
    AMM_PICK(__nv_bfloat16, 1, 4)
    AMM_PICK(__nv_bfloat16, 2, 4)
    AMM_PICK(__nv_bfloat16, 2, 2)
    AMM_PICK(__nv_bfloat16, 4, 2)
    AMM_PICK(__nv_bfloat16, 4, 1)
  } else {
    AMM_PICK(float, 1, 8)
    AMM_PICK(float, 1, 4)
    AMM_PICK(float, 2, 4)
    AMM_PICK(float, 2, 2)
    AMM_PICK(float, 4, 2)
    AMM_PICK(float, 4, 1)
    AMM_PICK(float, 8, 1)
  }
#undef AMM_PICK
  return nullptr;
}

// One CTA of the step kernel fits on an SM with the geometry's carve.
bool step_coresident(const PanelGeom& g) {
  const StepFn fn = pick_step(g.dtype, g.slots, g.gc);
  const int smem = step_smem(g);
  int per_sm = 0;
  if (!fn ||
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, g.threads, (size_t)smem) !=
          cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return per_sm >= 1;
}

// The failure path of the packet waits, on purpose (after wait_probe_kernel, whose `out` it goes on
// with): one warp waits in each of their three forms for an epoch that nothing writes.
__global__ void packet_probe_kernel(const uint4* p, uint32_t* status, uint32_t* out) {
  const unsigned long long t0 = globaltimer_now();
  const uint32_t never = packet_load(p).w + 1u;
  uint4 v[1];
  const int off[1] = {0};
  bool through = packets_wait<1>(p, 0, 1, never, v);
  through = packets_wait<1, true>(p, 0, 1, never, v) || through;
  through = packets_wait_at<1>(p, off, 1, never, v) || through;
  if (threadIdx.x == 0) {
    if (through) out[1] = 1u;
    out[2] += (uint32_t)((globaltimer_now() - t0) / 1000ull);
    if (!through) atomicOr(status, (uint32_t)kDevTimeout);
  }
}

cudaError_t launch_packet_probe(const Buffers& b, uint32_t* out, cudaStream_t s) {
  packet_probe_kernel<<<1, 32, 0, s>>>(b.pk_y, b.status, out);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_step(const Buffers& b, const PanelGeom& g, const CallCfg& cc, int iter,
                        int iter_end, cudaStream_t s) {
  StepArgs a{};
  a.b = b;
  a.g = g;
  a.cc = cc;
  a.iter = iter;
  a.iter_end = iter_end;
  const StepFn fn = pick_step(g.dtype, g.slots, g.gc);
  if (!fn) return cudaErrorInvalidValue;
  const int smem = step_smem(g);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(g.grid);
  cfg.blockDim = dim3(g.threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  int na = 0;
  const bool dep = pdl_enabled();
  if (dep) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (!dep || coop_with_pdl()) {
    at[na].id = cudaLaunchAttributeCooperative;
    at[na].val.cooperative = 1;
    ++na;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  e = cudaLaunchKernelEx(&cfg, fn, a);
  count_launch();
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace amm
