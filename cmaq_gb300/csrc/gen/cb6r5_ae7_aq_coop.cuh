// Generated by cmaq_gb300.mechgen.coop from mechs/cb6r5_ae7_aq/manifest.json.  Do not edit.
// Sizes and tables of the cooperative ROS3 kernel (csrc/coop.cuh).
#pragma once
#include <cuda_runtime.h>
namespace mech_cb6r5_ae7_aq {
extern __device__ const double c_coop_const[264];
extern __device__ const uint2 c_coop_rows[38528];
struct Coop {
    static constexpr int ELEMS = 3223, NCONST = 264, MAX_CELLS = 8;
    static constexpr int Y = 0, V = 149, K1 = 298, K2 = 447, T = 596;
    static constexpr int RKI = 745, G = 3132, Z = 3133;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static __device__ __forceinline__ const double* constants() { return c_coop_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coop_rows; }
    static constexpr int STAGE1_ROWS = 708, RHS_ROWS = 172, SOLVE_ROWS = 280;
};
}  // namespace mech_cb6r5_ae7_aq
