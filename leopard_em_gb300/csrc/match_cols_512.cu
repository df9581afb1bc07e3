// Column pass in two register passes (match_cols_reg.cuh): column length 512.
#include "match_cols_reg.cuh"
#include "match_launch.h"

namespace lgb {

// Two splits of the first radix: 8 x 4 skips all but the first 64 rows, 2 x 8
// all but the first 256 (rows beyond: the dense first pass).  Against three
// radix-8 passes of 64 threads a column, microseconds a batch before -> now:
// h 64: 32 correlograms 32.0 -> 26.9, 8: 18.0 -> 16.0, 1: 13.2 -> 13.9;
// h 256: 32: 35 -> 31, 1: 13.5 -> 16.4; h 384, 80 per image: 320: 233 -> 171.
// (The split may not depend on the batch: a correlogram's bits would.)
int launch_colpass_512(const void* A, const void* Ip, int ips, int h, int Wcp, int n_c, int cpi, int y_rows,
                        int waves, void* Y, cudaStream_t s) {
  if (h <= 64)
    return colpass_reg_launch<ColReg<8, 4, 2, 8, 32, 8, 2>, true>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
  return colpass_reg_t<ColReg<2, 8, 4, 8, 16, 8, 4>>(A, Ip, ips, h, Wcp, n_c, cpi, y_rows, waves, Y, s);
}

}  // namespace lgb
