// Grid kernels of the chemistry operator instantiated for mechanism cb6r5_ae7_aq
// (device code generated from CCTM/src/MECHS/cb6r5_ae7_aq by cmaq_gb300.mechgen).
#include "gen/cb6r5_ae7_aq_mech.cuh"
#include "gen/cb6r5_ae7_aq_coop.cuh"
#include "mech_ops.cuh"

namespace mech_cb6r5_ae7_aq {
// Calls of at most this many cells take the cooperative ROS3 kernel: from the initial state
// 36,000 cells take 202 ms there and 271 ms one cell per lane, 126,000 cells 707 and 386 ms; a
// later call of the hour 30 and 53 ms, 104 and 81 ms.
constexpr long long COOP_LIMIT = 60000;
}

DEFINE_MECH_OPS(mech_cb6r5_ae7_aq, mech_ops_cb6r5_ae7_aq)
