// Generated by cmaq_gb300.mechgen.coop from gen/kmt2_aq.cuh.  Do not edit.
// Sizes and tables of the cooperative KMT2 kernels (csrc/kmt2_coop.cuh).
#pragma once
#include <cuda_runtime.h>
namespace kmt2_coop {
extern __device__ const double c_kmt2_const[9];
extern __device__ const uint2 c_kmt2_rows[17920];
extern __device__ const short c_kmt2_diag[161];
struct Rate { int kind, r, i0, i1, i2; double p0, p1, p2; };   // 0 DISF, 1 DISB, 2 KRXN, 3 KIEPOX
extern __device__ const Rate c_kmt2_rate[123];
struct Coop {
    static constexpr int ELEMS = 3353, NCONST = 9, MAX_CELLS = 8;
    static constexpr int WS_ELEMS = 2876, FACTOR = 2876, CELL = 2999, CELL_DOUBLES = 64, Z = 3351, ONE = 3352, NRATE = 123;
    static constexpr int CHUNK = 28, TABLE_SMEM = 15936;
    static constexpr int FJAC_ROWS = 80, DECOMP_ROWS = 136, SOLVE_ROWS = 244, FUN_ROWS = 64;
    // chunks of one pass (fjac, decomp, solve, solve, fun, solve, fun, solve), and where each lies
    static constexpr int PASS = 50;
    static __device__ __forceinline__ int chunk(int k) { return k < 3 ? k + 0 : k < 8 ? k + 0 : k < 17 ? k + 0 : k < 26 ? k + -9 : k < 29 ? k + -9 : k < 38 ? k + -21 : k < 41 ? k + -21 : k + -33; }
    static __device__ __forceinline__ const double* constants() { return c_kmt2_const; }
    static __device__ __forceinline__ const uint2* rows() { return c_kmt2_rows; }
};
}  // namespace kmt2_coop
