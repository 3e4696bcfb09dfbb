// Grid kernels of the chemistry operator instantiated for mechanism cracmm2
// (device code generated from CCTM/src/MECHS/cracmm2 by cmaq_gb300.mechgen).
#include "gen/cracmm2_mech.cuh"
#include "gen/cracmm2_coop.cuh"
#include "mech_ops.cuh"

namespace mech_cracmm2 {
// Calls of at most this many cells take the cooperative ROS3 kernel, larger ones the work queue,
// which hands its last cells over to it: the first, second and third call of 20,000 cells take 449 /
// 81 / 56 ms there and 559 / 100 / 115 ms by the queue, of 40,000 cells 877 / 148 / 99 and 673 /
// 134 / 120.
constexpr long long COOP_LIMIT = 27000;
// Adjoint windows of at most this many cells take the cooperative kernels: two steps and their
// reverse take 744 ms there and 2,865 ms one cell per lane for 5,000 cells, 2,870 and 3,626 ms for
// 20,000, 4,304 and 4,586 ms for 30,000.
constexpr long long ADJ_COOP_LIMIT = 30000;
}

DEFINE_MECH_OPS(mech_cracmm2, mech_ops_cracmm2)
