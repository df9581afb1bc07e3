// Column pass in two register passes (match_cols_reg.cuh): column lengths 3840 and 1024.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

// Templates beyond the first split's sparse rows (480 of 3840, 256 of 1024): a
// second split with 16 sparse inputs instead of a dense first pass, which
// spills.  h 512: 3840 x 2049 51.6 -> 35.4 us a correlogram, 1024 x 2049 10.2 -> 9.6.
int launch_colpass_3840(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<8, 8, 4, 15, 64, 4, 1>,
                       ColReg<4, 16, 4, 15, 64, 4, 1>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

int launch_colpass_1024(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  return colpass_reg_t<ColReg<4, 8, 4, 8, 32, 8, 2>,
                       ColReg<2, 16, 4, 8, 32, 8, 2>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
