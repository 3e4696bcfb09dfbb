// Grid kernels of the chemistry operator instantiated for mechanism cracmm2
// (device code generated from CCTM/src/MECHS/cracmm2 by cmaq_gb300.mechgen).
#include "gen/cracmm2_mech.cuh"
#include "gen/cracmm2_coop.cuh"
#include "mech_ops.cuh"

namespace mech_cracmm2 {
// Calls of at most this many cells take the cooperative ROS3 kernel: from the initial state
// 10,881 cells take 267 ms there and 701 ms one cell per lane, 50,000 cells 1,190 and 962 ms; a
// later call of the hour 26 and 232 ms, 116 and 282 ms.
constexpr long long COOP_LIMIT = 40000;
// Adjoint windows of at most this many cells take the cooperative kernels: two steps and their
// reverse take 744 ms there and 2,865 ms one cell per lane for 5,000 cells, 2,870 and 3,626 ms for
// 20,000, 4,304 and 4,586 ms for 30,000.
constexpr long long ADJ_COOP_LIMIT = 30000;
}

DEFINE_MECH_OPS(mech_cracmm2, mech_ops_cracmm2)
