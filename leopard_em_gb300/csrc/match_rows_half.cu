// Row pass of the long rows (match_rows_half.cuh).
#include "match_rows_half.cuh"

#include "match_launch.h"

namespace lgb {

// row length, threads per row, rows and resident CTAs, radices of the half-length transform.
// Largest first radix that leaves the last pass 8 to 16 outputs a thread: its
// statistics then fit registers at 12 or more warps per SM.
#define LGB_ROW_HALF(n, threads, rows, per_sm, ...)                                                                \
  int launch_rowpass_##n(const void* Y, int H, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,         \
                         const int* o0_dev, float* mip, int* best, double* s1, double* s2, cudaStream_t s) {       \
    return rowpass_half_t<RowHalf<n / 2, threads, rows, Radices<__VA_ARGS__>, per_sm>>(                            \
        Y, H, y_rows, Wcp, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, s);                                   \
  }
LGB_ROW_HALF(512, 32, 2, 8, 8, 8, 4)
LGB_ROW_HALF(1024, 32, 1, 12, 16, 8, 4)
LGB_ROW_HALF(2048, 64, 1, 6, 16, 8, 8)
LGB_ROW_HALF(2880, 160, 1, 3, 16, 9, 10)
LGB_ROW_HALF(3072, 128, 1, 3, 16, 8, 12)
LGB_ROW_HALF(3840, 128, 1, 3, 16, 15, 8)
LGB_ROW_HALF(4096, 128, 1, 3, 16, 16, 8)
LGB_ROW_HALF(5760, 192, 1, 2, 16, 12, 15)
#undef LGB_ROW_HALF

}  // namespace lgb
