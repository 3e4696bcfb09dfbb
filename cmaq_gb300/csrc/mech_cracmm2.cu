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
// The adjoint's sweeps over at most this many cells take the cooperative kernels: two steps forward
// take 793 ms there and 1,113 ms one cell per lane for 20,000 cells, 1,061 and 1,348 ms for 27,000,
// 1,138 and 1,213 ms for 29,000; their reverse, with three cells to an SM instead of five, 2,224 and
// 2,522 ms for 20,000, 2,452 and 2,761 for 22,000, 2,672 and 2,435 for 24,000, 3,218 and 2,557 for
// 29,000 (at rtol 1e-5 6,050 and 6,922 ms for 22,000, 7,453 and 7,045 for 27,000).
constexpr long long ADJ_COOP_LIMIT = 30000, ADJ_REVERSE_COOP_LIMIT = 22000;
}

DEFINE_MECH_OPS(mech_cracmm2, mech_ops_cracmm2)
