// Generated by cmaq_gb300.mechgen.coop from mechs/cracmm2/manifest.json.  Do not edit.
// Sizes and tables of the cooperative ROS3 kernel (csrc/coop.cuh).
#pragma once
#include <cuda_runtime.h>
namespace mech_cracmm2 {
extern __device__ const double c_coop_const[544];
extern __device__ const uint2 c_coop_rows[69888];
struct Coop {
    static constexpr int ELEMS = 5304, NCONST = 544, MAX_CELLS = 5;
    static constexpr int Y = 0, V = 189, K1 = 378, K2 = 567, T = 756;
    static constexpr int RKI = 945, G = 5291, Z = 5292;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static __device__ __forceinline__ const double* constants() { return c_coop_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coop_rows; }
    static constexpr int STAGE1_ROWS = 1416, RHS_ROWS = 324, SOLVE_ROWS = 420;
};
}  // namespace mech_cracmm2
