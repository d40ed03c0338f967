// Declarations shared by the batched solver (amm_batch.cu) and its Gram products (amm_gram.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace amm {
namespace batch {

struct Mat {
  const float* A;  // column-major, ld % 4 == 0, 16-byte aligned
  int64_t ld;
  int32_t m, n;
  int64_t out_off;  // first row of this matrix's vector in the output
  int64_t st_off;   // AMM mode: first of this matrix's c xorshift states
  int32_t c;        // AMM mode: samples per product (0: exact)
  int32_t ldc;      // m rounded up to 4: leading dimension and columns of C
  float* C;         // A·Aᵀ (ldc x ldc, zeros past m), formed at the start of every run; null: the
                    // exact products of this matrix read A
};

// Rows 128·ti .. +127 and columns 256·tj .. +255 of a matrix's C, tj <= ti / 2: what lies below the
// diagonal block is written with its mirror image.
struct GramTile {
  int32_t mat, ti, tj, pad;
};

// C = A·Aᵀ of every matrix in the tile list; `queue` is a zeroed counter.
cudaError_t launch_gram(const Mat* mats, const GramTile* tiles, int ntiles, uint32_t* queue,
                        int nsm, cudaStream_t s);

}  // namespace batch
}  // namespace amm
