// Padded rfft of projection rows, the longer rows (match_pad_reg.cuh).
#include "match_launch.h"
#include "match_pad_reg.cuh"

namespace lgb {

// row length, threads per row, rows at once, radices of the half-length
// transform (those of the row pass)
#define LGB_PAD_REG(n, threads, rows, ...)                                                                         \
  int launch_pad_rfft_##n(const float* proj, const double* rowstats, int h, int norm_h, int norm_w, int Wcp, int n_c, \
                          void* A, cudaStream_t s, bool norm_ready) {                                              \
    return pad_rfft_reg_t<PadReg<n / 2, threads, rows, Radices<__VA_ARGS__>>>(proj, rowstats, h, norm_h, norm_w, Wcp, \
                                                                              n_c, A, s, norm_ready);              \
  }
LGB_PAD_REG(512, 32, 4, 8, 8, 4)
LGB_PAD_REG(1024, 64, 2, 16, 8, 4)
LGB_PAD_REG(2048, 64, 2, 16, 8, 8)
LGB_PAD_REG(2880, 96, 1, 16, 9, 10)
LGB_PAD_REG(3072, 96, 1, 16, 8, 12)
LGB_PAD_REG(3840, 128, 1, 16, 15, 8)
LGB_PAD_REG(4096, 128, 1, 16, 16, 8)
LGB_PAD_REG(5760, 128, 1, 16, 12, 15)
#undef LGB_PAD_REG

}  // namespace lgb
