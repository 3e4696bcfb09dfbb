// Generated by cmaq_gb300.mechgen.coop from mechs/cracmm2/manifest.json and gen/cracmm2_ebi.cu.  Do not edit.
// Sizes and tables of the cooperative kernels (csrc/coop.cuh, csrc/ebi_coop.cuh).
#pragma once
#include <cuda_runtime.h>
namespace mech_cracmm2 {
extern __device__ const double c_coop_const[544];
extern __device__ const uint2 c_coop_rows[69888];
extern __device__ const double c_coopadj_const[544];
extern __device__ const uint2 c_coopadj_rows[120064];
extern __device__ const double c_coopebi_const[550];
extern __device__ const uint2 c_coopebi_rows[13440];
extern __device__ const double c_coopgear_const[544];
extern __device__ const uint2 c_coopgear_rows[57088];
struct Coop {
    static constexpr int ELEMS = 5304, NCONST = 544, MAX_CELLS = 5;
    static constexpr int Y = 0, V = 189, K1 = 378, K2 = 567, T = 756, RKI = 945, G = 5291, Z = 5292;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int STAGE1_ROWS = 1416, RHS_ROWS = 324, SOLVE_ROWS = 420;
    // chunks of one pass through the programs (stage1, rhs, solve, solve), and where each lies
    static constexpr int PASS = 93;
    static __device__ __forceinline__ int chunk(int k) { return k < 78 ? k : k - 15; }
    static __device__ __forceinline__ const double* constants() { return c_coop_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coop_rows; }
};
struct CoopAdj {
    static constexpr int ELEMS = 6958, NCONST = 544, MAX_CELLS = 3;
    static constexpr int Y = 0, V = 189, K1 = 378, K2 = 567, T = 756, K3 = 945, NU2 = 1134, NU3 = 1323, PHI = 1512, LAM = 1701, EMIS = 1890, RKI = 2079, GK = 3141, G = 6956, Z = 6957;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int STAGE1_ROWS = 1408, RHS_ROWS = 324, SOLVE_ROWS = 420, TSOLVE_ROWS = 684, JTV_ROWS = 180, GRADIENT_ROWS = 652;
    // chunks of one pass through the programs (stage1, rhs, solve, solve, tsolve, tsolve, jtv, tsolve, gradient), and where each lies
    static constexpr int PASS = 199;
    static __device__ __forceinline__ int chunk(int k) { return k < 78 ? k : k < 118 ? k - 15 : k < 150 ? k - 40 : k < 175 ? k - 72 : k - 65; }
    static __device__ __forceinline__ const double* constants() { return c_coopadj_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopadj_rows; }
};
// the forward pass's programs of the same tables: stage1, rhs, solve, solve
struct CoopAdjForward : CoopAdj {
    static constexpr int PASS = 93;
    static __device__ __forceinline__ int chunk(int k) { return k < 78 ? k : k - 15; }
};
struct CoopEbi {
    static constexpr int ELEMS = 3067, NCONST = 550, MAX_CELLS = 8;
    static constexpr int YC = 0, YC0 = 189, YCP = 378, PROD = 567, LOSS = 756, PNEG = 945, RKI = 1134, DTC = 2196, Z = 2197, ONE = 2198;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int ITERATION_ROWS = 416;
    // chunks of one pass through the programs (iteration), and where each lies
    static constexpr int PASS = 15;
    static __device__ __forceinline__ int chunk(int k) { return k; }
    static __device__ __forceinline__ const double* constants() { return c_coopebi_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopebi_rows; }
};
struct CoopGear {
    static constexpr int ELEMS = 8285, NCONST = 544, MAX_CELLS = 3;
    static constexpr int Q = 6773, R1 = 0, Z = 1, ONE = 2, WORKSPACE = 4;
    static constexpr int CHUNK = 8, TABLE_SMEM = 5696;
    static constexpr int PREDICTOR_ROWS = 1040, RHS_ROWS = 320, SOLVE_ROWS = 420;
    // chunks of one pass through the programs (predictor, rhs, solve), and where each lies
    static constexpr int PASS = 223;
    static __device__ __forceinline__ int chunk(int k) { return k; }
    static __device__ __forceinline__ const double* constants() { return c_coopgear_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_coopgear_rows; }
};
}  // namespace mech_cracmm2
