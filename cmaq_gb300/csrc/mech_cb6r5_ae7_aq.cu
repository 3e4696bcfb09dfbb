// Grid kernels of the chemistry operator instantiated for mechanism cb6r5_ae7_aq
// (device code generated from CCTM/src/MECHS/cb6r5_ae7_aq by cmaq_gb300.mechgen).
#include "gen/cb6r5_ae7_aq_mech.cuh"
#include "gen/cb6r5_ae7_aq_coop.cuh"
#include "mech_ops.cuh"

namespace mech_cb6r5_ae7_aq {
// Calls of at most this many cells take the cooperative ROS3 kernel, larger ones the work queue,
// which hands its last cells over to it: the first, second and third call of 36,000 cells take 182 /
// 36 / 29 ms there and 197 / 48 / 35 ms by the queue, of 54,000 cells 270 / 54 / 43 and 265 / 52 / 42.
constexpr long long COOP_LIMIT = 50000;
// The adjoint's sweeps over at most this many cells take the cooperative kernels: two steps forward
// take 289 ms there and 449 ms one cell per lane for 40,000 cells, 388 and 470 ms for 54,000, both
// sweeps 1,553 and 1,582 ms for 60,000 and 2,062 and 1,716 ms for 80,000; their reverse 781 and
// 993 ms for 40,000, 976 and 1,001 for 50,000, 1,059 and 1,057 for 54,000 (2,314 and 2,682 ms at
// rtol 1e-5).
constexpr long long ADJ_COOP_LIMIT = 55000, ADJ_REVERSE_COOP_LIMIT = 55000;
}

DEFINE_MECH_OPS(mech_cb6r5_ae7_aq, mech_ops_cb6r5_ae7_aq)
