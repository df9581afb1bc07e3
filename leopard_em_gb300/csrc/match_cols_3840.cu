// Column pass in two register passes (match_cols_reg.cuh): column lengths 3840 and 1024.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

int launch_colpass_3840(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows, int waves, void* Y,
                        cudaStream_t s) {
  return colpass_reg_t<ColReg<8, 8, 4, 15, 64, 4, 1>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

int launch_colpass_1024(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows, int waves, void* Y,
                        cudaStream_t s) {
  return colpass_reg_t<ColReg<4, 8, 4, 8, 32, 8, 2>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
