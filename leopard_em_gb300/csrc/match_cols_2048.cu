// Column pass in two register passes (match_cols_reg.cuh): column lengths 2048 and 576.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

// 576 rows, templates of 193 to 288: 12 sparse inputs instead of a dense first
// pass (289 columns, 96 correlograms: 0.9 -> 0.7 us each).
int launch_colpass_2048(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<4, 8, 8, 8, 32, 4, 2>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

int launch_colpass_576(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<3, 8, 3, 8, 24, 8, 3>,
                       ColReg<2, 12, 3, 8, 24, 8, 3>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
