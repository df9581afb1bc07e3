// Column pass in two register passes (match_cols_reg.cuh): column length 5760.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

int launch_colpass_5760(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<10, 8, 9, 8, 80, 4, 1, true>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
