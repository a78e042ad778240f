/*
 * eg_transpose.cuh -- transpose of a CSR matrix in one launch.
 */
#ifndef EG_TRANSPOSE_CUH
#define EG_TRANSPOSE_CUH

#include <cuda_runtime.h>

namespace eg {

/* Zeros before the launch. */
struct TransposeCtrl {
    unsigned arrivals;            /* of the grid's barriers                                */
    int bad;                      /* an offset decreases or a column is out of range       */
    int skewed;                   /* columns too long to be ordered here: nothing is out   */
    int abort;                    /* a barrier gave up                                     */
    unsigned long long squares;   /* sum of the columns' squared lengths                   */
    unsigned long long pad;
};

struct TransposeParams {
    int nrows, ncols, nnz;
    int chunk_shift;              /* columns a CTA scans, as a power of two                */
    const long long *row_ptr;
    const int *col, *val;
    int *count;                   /* [ncols + 1]: lengths, then offsets in a CTA's chunk   */
    int *totals;                  /* [kTransposeGrid]                                      */
    int *rank;                    /* [nnz] arrival of an edge in its column                */
    int4 *rec;                    /* [nnz] edge, column, row, value, by column             */
    long long *csc_ptr;           /* [ncols + 1]                                           */
    int *csc_row, *csc_val;       /* [nnz]                                                 */
    TransposeCtrl *ctrl;
    unsigned long long wait_limit_ns;
};

constexpr int kTransposeGrid = 512;   /* most CTAs */

/* The CTAs of a launch on a device of `sms` SMs. */
int transpose_grid(int nrows, int ncols, long long nnz, int sms);
/* An error where the grid does not fit the device at once. */
cudaError_t launch_transpose(TransposeParams p, int grid, cudaStream_t st);

}  // namespace eg

#endif
