// C = A·Aᵀ of many FP32 matrices (column-major, uneven sizes) on the 5th-generation tensor cores, for
// the batched solver: a matrix whose block product is taken many times is multiplied as C·X (m·m
// entries from L2) instead of A·(AᵀX) (twice m·n products on the legacy tensor pipe).
//
// FP32 from BF16 products.  x = b0 + b1 + b2 (each the nearest BF16 of what is left: 24 bits), and
// A·Aᵀ is summed from b0·b0, b0·b1, b1·b0, b1·b1, b0·b2 and b2·b0; the dropped terms are below
// 2^-26 of the product.  The tensor core does not round its running sum to nearest, and a long chain
// of products in tensor memory drifts (about 3e-6 of the terms after 128 products).  So each chunk
// of 32 columns starts from zero, takes its 10 small products first and its 2 large ones last,
// and the chunks are summed in FP32 registers with rounding to nearest.  λ's rms error against FP64 (384
// matrices each, products through A -> through C): 512 x 2048 1.2e-7 -> 7.2e-8, 640 x 640 1.3e-7
// -> 7.3e-8, 128 x 800 1.2e-7 -> 7.1e-8, 300 x 700 with lognormal row scales 1.4e-7 -> 1.3e-7.
// (Summing eight chunks at a time into C instead: the same errors, 15.5 -> 27 ms a run.)
//
// One CTA of 512 threads per tile of 128 rows x up to 256 columns on or below the diagonal, tiles
// taken from a queue, longest first.  256 columns because a product of 128 x N x 16 takes about as
// long for N = 128 as for N = 256 (476 matrices of the 512-matrix batch: 6.7 ms with 128 x 128 tiles, 6.3
// with these, before the steps below).  Per chunk every thread converts 2 + 4 float4 (4 consecutive
// rows of a column: one coalesced 16-byte load, three 8-byte stores into the 128-byte-swizzled
// MN-major planes), one thread issues the 12 products, and while they run the threads add the chunk before from
// tensor memory (two accumulators, two stages of planes).  The next chunk's loads are issued before
// the barrier, so that their latency passes while the warps meet.
// What bounds it: the converting threads (64 accumulators and 24 loaded values of 128 registers
// each), then the products, about 150 clocks each, and shared-memory bandwidth (per chunk 72 KB of
// planes written, 144 KB read, at 128 bytes a clock).  The whole run of the 512-matrix batch: loads
// after the barrier, 16 tensor-memory columns at a time 14.3 ms; loads before it 14.2; 8 columns at a
// time (fewer spills) 13.2, with the loads after the barrier 13.9; 32-bit shared-memory addresses and
// one column pointer 12.8.  148 matrices of 512 x 2560: 0.92 ms, 810 TFLOP/s of products, the tensor
// cores active in 43 % of the cycles, issue in 51 %, DRAM at 12 %.
#include <cuda_runtime.h>

#include <cstdint>

#include "amm_batch.h"
#include "amm_device.cuh"
#include "amm_internal.h"

namespace amm {
namespace batch {

namespace {

constexpr int kRows = 128;       // rows of a tile
constexpr int kCols = 256;       // columns of a tile at most
constexpr int kChunk = 32;       // columns of A per stage
constexpr int kGramThreads = 512;
constexpr int kPlaneA = kRows * kChunk * 2;            // bytes of a BF16 plane of the row operand
constexpr int kPlaneB = kCols * kChunk * 2;            // ... of the column operand
constexpr int kStage = 3 * (kPlaneA + kPlaneB);
constexpr int kGramSmem = 2 * kStage + 1024;           // (aligned to 1024 inside)
constexpr uint32_t kAccCols = 2 * kCols;               // tensor-memory columns: two accumulators

// Shared-memory descriptor of an MN-major BF16 operand of `rows` rows with the 128-byte swizzle:
// atoms of 64 rows x 8 columns (1024 bytes), row blocks 1024 bytes apart, column groups 16·rows.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr, uint32_t rows) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)(1024 >> 4) << 16) |
         ((uint64_t)rows << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16, FP32 accumulators, BF16 operands, both MN-major, M = 128
constexpr uint32_t kInstr = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                            ((uint32_t)(kRows >> 4) << 24);

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t instr,
                                         bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(instr), "r"((uint32_t)add)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void st_shared(uint32_t addr, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(x), "r"(y) : "memory");
}
// 8 columns of this warp's 32 tensor-memory lanes, added to acc
__device__ __forceinline__ void tmem_add8(uint32_t addr, float* acc) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] += __uint_as_float(r[i]);
}

// two floats to BF16 (nearest), x in the low half
__device__ __forceinline__ uint32_t to_bf16x2(float x, float y) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
// the three BF16 parts of (x, y); each remainder is exact in FP32
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
  p[0] = to_bf16x2(x, y);
  float rx = x - __uint_as_float(p[0] << 16), ry = y - __uint_as_float(p[0] & 0xffff0000u);
  p[1] = to_bf16x2(rx, ry);
  rx -= __uint_as_float(p[1] << 16);
  ry -= __uint_as_float(p[1] & 0xffff0000u);
  p[2] = to_bf16x2(rx, ry);
}

__global__ void __launch_bounds__(kGramThreads, 1)
    gram_kernel(const Mat* __restrict__ mats, const GramTile* __restrict__ tiles, int ntiles,
                uint32_t* queue) {
  extern __shared__ __align__(16) unsigned char gram_smem[];
  const uint32_t planes = (smem_addr(gram_smem) + 1023u) & ~1023u;
  __shared__ uint64_t bar[2];     // products of a stage done
  __shared__ uint32_t tmem_s;
  __shared__ int tile_s;
  // of the products: the instruction; the column operand's first byte, rows and bytes per plane
  __shared__ uint32_t op_s[4];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(&tmem_s)),
                 "r"(kAccCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = tmem_s;
  uint32_t ph = 0u;           // phase parity of the two stages, a bit each (alike in every thread)
  bool dead = false;          // a wait gave up: no more products, every tile is NaN
  // this thread's part of an accumulator: lane quarter warp % 4, columns 64·(warp / 4) ..
  const int seg = 64 * (warp >> 2);
  const uint32_t acc_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)seg;
  // this thread's part of a chunk: rows 4·lane .. +3 (of each 128), columns 2·warp, 2·warp + 1; the
  // 8-byte half of the 16-byte piece (row / 8) ^ (column mod 8) of its 128-byte line
  const uint32_t mb = (uint32_t)lane >> 4, piece = ((uint32_t)lane >> 1) & 7u, half = lane & 1u;
  const uint32_t kg = (uint32_t)warp >> 2, kr = (2u * (uint32_t)warp) & 7u;

  for (;;) {
    __syncthreads();  // tile_s was read
    if (t == 0) tile_s = (int)atomicAdd(queue, 1u);
    __syncthreads();
    if (tile_s >= ntiles) break;
    const GramTile tl = tiles[tile_s];
    const Mat M = mats[tl.mat];
    const int m = M.m, n = M.n;
    // an even row block's last tile is its diagonal block alone: the rows serve as both operands
    const bool diag = 2 * tl.tj == tl.ti;
    const int ncol = diag ? kRows : min(kCols, (M.ldc - kCols * tl.tj + 15) & ~15);
    // (what only the issuing thread or the tile's end needs is kept out of the registers)
    if (t == 0) {
      op_s[0] = kInstr | ((uint32_t)(ncol >> 3) << 17);
      op_s[1] = diag ? 0u : 3u * kPlaneA;
      op_s[2] = diag ? kRows : kCols;
      op_s[3] = diag ? kPlaneA : kPlaneB;
    }
    const int nchunk = (n + kChunk - 1) / kChunk;
    const int ra0 = kRows * tl.ti + 4 * lane, rb0 = kCols * tl.tj + 4 * lane;
    // rows r0 .. r0 + 3 of a column at p (zeros outside the matrix; left: rows from r0 to the end)
    auto load4 = [](const float* p, int left) -> float4 {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (left >= 4) {
        v = __ldg(reinterpret_cast<const float4*>(p));
      } else if (left > 0) {  // the last rows: nothing past row m is read
        v.x = __ldg(p);
        if (left > 1) v.y = __ldg(p + 1);
        if (left > 2) v.z = __ldg(p + 2);
      }
      return v;
    };
    // this thread's rows of the chunk's first column of its two
    const float* pa = M.A + (int64_t)(2 * warp) * M.ld + ra0;
    const int ab = rb0 - ra0;  // (from the row operand's rows to the column operand's)
    const int64_t ld = M.ld;
    const int la = m - ra0, lb = diag ? 0 : m - rb0;
    int left_k = n - 2 * warp;  // columns from this thread's first one to the end
    float4 ra[2], rb[2][2];  // [column], [128 rows][column]
    auto load_chunk = [&]() {  // the chunks in turn
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bool in = j < left_k;
        ra[j] = load4(pa + j * ld, in ? la : 0);
        rb[0][j] = load4(pa + ab + j * ld, in ? lb : 0);
        rb[1][j] = load4(pa + ab + j * ld + 128, in ? lb - 128 : 0);
      }
      pa += kChunk * ld;
      left_k -= kChunk;
    };
    // 128 rows of an operand of `rows` rows, from its row block `blk` (of 64) on
    auto convert = [&](const float4 (&r)[2], uint32_t base, uint32_t rows, uint32_t blk,
                       uint32_t plane) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        uint32_t lo[3], hi[3];
        split3(r[j].x, r[j].y, lo);
        split3(r[j].z, r[j].w, hi);
        const uint32_t c = kr + (uint32_t)j;  // column within its group
        const uint32_t off = kg * 16u * rows + (blk + mb) * 1024u + c * 128u +
                             ((piece ^ c) << 4) + half * 8u;
#pragma unroll
        for (int p = 0; p < 3; ++p)
          st_shared(base + p * plane + off, lo[p], hi[p]);
      }
    };
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    // add chunk kc's accumulator once its products are done
    auto promote = [&](int kc) {
      const int s = kc & 1;
      if (!dead && !mbar_wait_bounded(&bar[s], (ph >> s) & 1u)) dead = true;
      ph ^= 1u << s;
      tmem_fence_after();
      __syncwarp();
      if (seg < ncol) {  // warp-uniform
#pragma unroll
        for (int h = 0; h < 8; ++h)
          tmem_add8(acc_addr + (uint32_t)(s * kCols + 8 * h), acc + 8 * h);
      }
      tmem_fence_before();
    };
    load_chunk();
#pragma unroll 1
    for (int kc = 0; kc < nchunk; ++kc) {
      const int s = kc & 1;
      const uint32_t st = planes + (uint32_t)(s * kStage);
      convert(ra, st, kRows, 0, kPlaneA);  // (the stage's last products were waited for)
      if (!diag) {
        convert(rb[0], st + 3 * kPlaneA, kCols, 0, kPlaneB);
        if (ncol > 128) convert(rb[1], st + 3 * kPlaneA, kCols, 2, kPlaneB);
      }
      fence_proxy_async_smem();
      if (kc + 1 < nchunk) load_chunk();
      dead = __syncthreads_or(dead ? 1 : 0) != 0;
      if (t == 0 && !dead) {
        tmem_fence_after();
        const uint32_t d = *const_cast<volatile uint32_t*>(&tmem_s) + (uint32_t)(s * kCols);
        const volatile uint32_t* op = op_s;
        const uint32_t instr = op[0], a0 = st, b0 = a0 + op[1];
        const uint32_t brows = op[2], bplane = op[3];
        // (plane of A, plane of B), the small products first
        constexpr int pa[6] = {1, 0, 2, 0, 1, 0}, pb[6] = {1, 2, 0, 1, 0, 0};
        bool add = false;
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int ks = 0; ks < kChunk / 16; ++ks) {
            mma_bf16(d, operand_desc(a0 + pa[p] * kPlaneA + ks * 32 * kRows, kRows),
                     operand_desc(b0 + pb[p] * bplane + ks * 32 * brows, brows), instr, add);
            add = true;
          }
        mma_commit(&bar[s]);
      }
      if (kc > 0) promote(kc - 1);
    }
    promote(nchunk - 1);
    dead = __syncthreads_or(dead ? 1 : 0) != 0;
    if (dead) {
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = __int_as_float(0x7fffffff);
    }
    // row r, columns c0 .. c0 + 63 of C (what lies in the tile but past ldc is left out), and their
    // mirror image unless in the diagonal block (rows and columns of [m, ldc) are zeros, computed from
    // zero rows)
    const GramTile te = tiles[*const_cast<volatile int*>(&tile_s)];
    float* const C = mats[te.mat].C;
    const int ldc = mats[te.mat].ldc;
    const int r = kRows * te.ti + 32 * (warp & 3) + lane, c0 = kCols * te.tj + seg;
    if (r < ldc && seg < ncol) {
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (c0 + i < ldc) C[(int64_t)(c0 + i) * ldc + r] = acc[i];
      if (c0 / kRows != te.ti) {
#pragma unroll
        for (int i = 0; i < 64; i += 4)
          if (c0 + i < ldc)
            *reinterpret_cast<float4*>(C + (int64_t)r * ldc + c0 + i) =
                make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      }
    }
  }
  tmem_fence_before();
  __syncthreads();
  if (warp == 0) {
    tmem_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAccCols)
                 : "memory");
  }
}

}  // namespace

cudaError_t launch_gram(const Mat* mats, const GramTile* tiles, int ntiles, uint32_t* queue,
                        int nsm, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kGramSmem);
  if (e != cudaSuccess) return e;
  gram_kernel<<<ntiles < nsm ? ntiles : nsm, kGramThreads, kGramSmem, s>>>(mats, tiles, ntiles,
                                                                           queue);
  count_launch();
  return cudaGetLastError();
}

}  // namespace batch
}  // namespace amm
