// Internal interface of the blockwise row gradients (slotscan_rowadj.cu).
#pragma once
#include <cuda_runtime.h>

namespace slotscan {

constexpr int RA_NMAX = 256;         // rows (threads) per CTA

struct RowAdjTensor {                // one tensor (keys or values) of width D; dbuf may be NULL (zeros)
    const void* x;
    const float* x0;
    const float* dbuf;
    void* dx;
    int D;
};
struct RowAdjArgs {
    int N, T, H, G, hard, hard_gate;
    const float* as;                 // [nbh][T][N] softmax address (soft address only)
    const int* am;                   // [nbh][T] address (hard address only)
    const int* lim;                  // [nbh][NB] last candidate row at the block's first token, NULL: all rows
    const float* gate;
    float* dp;                       // [slices][nbh][T][N]
    int bh0, nbh;                    // the sequences of this launch
    int nsl0;                        // slices of the first tensor
    RowAdjTensor t0, t1;
};

static inline int row_adjoint_ds(int N) { return N <= 64 ? 16 : 32; }
static inline int row_adjoint_slices(int N, int D) { return (D + row_adjoint_ds(N) - 1) / row_adjoint_ds(N); }

// in_dtype as in slotscan_params: type of x and dx.  D of every slice lands in A.dp; sum the slices with run_row_dsum.
cudaError_t run_row_adjoint(const RowAdjArgs& A, int in_dtype, cudaStream_t st);
// table[0] += table[1] + ... + table[slices - 1] over n elements, in this order
cudaError_t run_row_dsum(float* dp, size_t n, int slices, cudaStream_t st);

}  // namespace slotscan
