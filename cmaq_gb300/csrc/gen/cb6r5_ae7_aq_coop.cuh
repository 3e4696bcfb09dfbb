// Generated by cmaq_gb300.mechgen.coop from mechs/cb6r5_ae7_aq/manifest.json and gen/cb6r5_ae7_aq_ebi.cu.  Do not edit.
// Sizes and tables of the cooperative kernels (csrc/coop.cuh, csrc/ebi_coop.cuh).
#pragma once
#include <cuda_runtime.h>
namespace mech_cb6r5_ae7_aq {
extern __device__ const double c_coop_const[264];
extern __device__ const uint2 c_coop_rows[38528];
extern __device__ const double c_coopadj_const[264];
extern __device__ const uint2 c_coopadj_rows[67200];
extern __device__ const double c_coopebi_const[264];
extern __device__ const uint2 c_coopebi_rows[7168];
extern __device__ const double c_coopgear_const[264];
extern __device__ const uint2 c_coopgear_rows[29184];
struct Coop {
    static constexpr int ELEMS = 3223, NCONST = 264, MAX_CELLS = 8;
    static constexpr int Y = 0, V = 149, K1 = 298, K2 = 447, T = 596, RKI = 745, G = 3132, Z = 3133;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int STAGE1_ROWS = 708, RHS_ROWS = 172, SOLVE_ROWS = 280;
    // chunks of one pass through the programs (stage1, rhs, solve, solve), and where each lies
    static constexpr int PASS = 53;
    static __device__ __forceinline__ int chunk(int k) { return k < 43 ? k : k - 10; }
    static __device__ __forceinline__ const double* constants() { return c_coop_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coop_rows; }
};
struct CoopAdj {
    static constexpr int ELEMS = 4377, NCONST = 264, MAX_CELLS = 6;
    static constexpr int Y = 0, V = 149, K1 = 298, K2 = 447, T = 596, K3 = 745, NU2 = 894, NU3 = 1043, PHI = 1192, LAM = 1341, EMIS = 1490, RKI = 1639, GK = 2337, G = 4375, Z = 4376;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int STAGE1_ROWS = 712, RHS_ROWS = 172, SOLVE_ROWS = 280, TSOLVE_ROWS = 372, JTV_ROWS = 104, GRADIENT_ROWS = 372;
    // chunks of one pass through the programs (stage1, rhs, solve, solve, tsolve, tsolve, jtv, tsolve, gradient), and where each lies
    static constexpr int PASS = 113;
    static __device__ __forceinline__ int chunk(int k) { return k < 43 ? k : k < 67 ? k - 10 : k < 85 ? k - 24 : k < 99 ? k - 42 : k - 38; }
    static __device__ __forceinline__ const double* constants() { return c_coopadj_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopadj_rows; }
};
// the forward pass's programs of the same tables: stage1, rhs, solve, solve
struct CoopAdjForward : CoopAdj {
    static constexpr int PASS = 53;
    static __device__ __forceinline__ int chunk(int k) { return k < 43 ? k : k - 10; }
};
struct CoopEbi {
    static constexpr int ELEMS = 2464, NCONST = 264, MAX_CELLS = 10;
    static constexpr int YC = 0, YC0 = 149, YCP = 298, PROD = 447, LOSS = 596, PNEG = 745, RKI = 894, DTC = 1592, Z = 1593, ONE = 1594;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int ITERATION_ROWS = 216;
    // chunks of one pass through the programs (iteration), and where each lies
    static constexpr int PASS = 8;
    static __device__ __forceinline__ int chunk(int k) { return k; }
    static __device__ __forceinline__ const double* constants() { return c_coopebi_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopebi_rows; }
};
struct CoopGear {
    static constexpr int ELEMS = 5312, NCONST = 264, MAX_CELLS = 5;
    static constexpr int Q = 4120, R1 = 0, Z = 1, ONE = 2, WORKSPACE = 4;
    static constexpr int CHUNK = 16, TABLE_SMEM = 9792;
    static constexpr int PREDICTOR_ROWS = 440, RHS_ROWS = 168, SOLVE_ROWS = 280;
    // chunks of one pass through the programs (predictor, rhs, solve), and where each lies
    static constexpr int PASS = 57;
    static __device__ __forceinline__ int chunk(int k) { return k; }
    static __device__ __forceinline__ const double* constants() { return c_coopgear_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopgear_rows; }
};
}  // namespace mech_cb6r5_ae7_aq
