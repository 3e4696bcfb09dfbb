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
// Adjoint windows of at most this many cells take the cooperative kernels: two steps and their
// reverse take 221 ms there and 1,102 ms one cell per lane for 8,000 cells, 1,296 and 1,591 ms for
// 50,000, 1,553 and 1,582 ms for 60,000, 2,062 and 1,716 ms for 80,000.
constexpr long long ADJ_COOP_LIMIT = 55000;
}

DEFINE_MECH_OPS(mech_cb6r5_ae7_aq, mech_ops_cb6r5_ae7_aq)
