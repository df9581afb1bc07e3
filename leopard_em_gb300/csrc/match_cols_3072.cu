// Column pass in two register passes (match_cols_reg.cuh): column lengths 3072 and 2880.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

// Templates beyond 384 rows: a split with 16 sparse inputs instead of a dense
// first pass (3072 x 2049, h 512: 39.3 -> 30.0 us a correlogram).
int launch_colpass_3072(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<8, 8, 3, 16, 64, 4, 1>,
                       ColReg<4, 16, 3, 16, 64, 4, 1>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

int launch_colpass_2880(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<3, 16, 4, 15, 60, 4, 1>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
