// Column pass in two register passes (match_cols_reg.cuh): column length 4096.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

int launch_colpass_4096(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<8, 8, 8, 8, 64, 4, 1>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
