// Row pass of the long rows (match_rows_half.cuh).
#include "match_rows_half.cuh"

#include "match_launch.h"

namespace lgb {

// row length, threads per row, rows and resident CTAs, radices of the half-length transform.
// Largest first radix that leaves the last pass 8 to 16 outputs a thread: its
// statistics then fit registers at 12 or more warps per SM.
// The short rows' split forms (8 and 4 groups a row at 512, 6 and 3 at 1024, 3
// at 2048) keep the resident threads: below about 600 rows the unsplit form
// leaves most of them without a row.  Unsplit -> split, microseconds a batch:
//   512 x 512 26.3 -> 22.0 (32 correlograms), 88.9 -> 53.3 (96)   256 x 512 25.6 -> 16.1 (32)
//   288 x 1024 40.9 -> 30.4 (32)   512 x 1024 46.8 -> 43.8 (32)   288 x 2048 49.6 -> 45.6 (32)
#define LGB_ROW_HALF(n, ...)                                                                                       \
  int launch_rowpass_##n(const void* Y, int H, int y_rows, int Wcp, int n_c, int nb, int n_orient, int o0,         \
                         const int* o0_dev, float* mip, int* best, double* s1, double* s2, cudaStream_t s) {       \
    return rowpass_half_t<__VA_ARGS__>(Y, H, y_rows, Wcp, n_c, nb, n_orient, o0, o0_dev, mip, best, s1, s2, s);     \
  }
using R512 = Radices<8, 8, 4>;
using R1024 = Radices<16, 8, 4>;
using R2048 = Radices<16, 8, 8>;
LGB_ROW_HALF(512, RowHalf<256, 32, 2, R512, 8>, RowHalf<256, 32, 1, R512, 2, 8>, RowHalf<256, 32, 1, R512, 4, 4>)
LGB_ROW_HALF(1024, RowHalf<512, 32, 1, R1024, 12>, RowHalf<512, 32, 1, R1024, 2, 6>, RowHalf<512, 32, 1, R1024, 4, 3>)
LGB_ROW_HALF(2048, RowHalf<1024, 64, 1, R2048, 6>, RowHalf<1024, 64, 1, R2048, 2, 3>)
LGB_ROW_HALF(2880, RowHalf<1440, 160, 1, Radices<16, 9, 10>, 3>)
LGB_ROW_HALF(3072, RowHalf<1536, 128, 1, Radices<16, 8, 12>, 3>)
LGB_ROW_HALF(3840, RowHalf<1920, 128, 1, Radices<16, 15, 8>, 3>)
LGB_ROW_HALF(4096, RowHalf<2048, 128, 1, Radices<16, 16, 8>, 3>)
LGB_ROW_HALF(5760, RowHalf<2880, 192, 1, Radices<16, 12, 15>, 2>)
#undef LGB_ROW_HALF

}  // namespace lgb
