// Cooperative adjoint of ROS3: the lanes of a warp go through one cell's steps, forward and in
// reverse, on its state in shared memory (coop.cuh; the programs: mechgen/coop.py's
// adjoint_programs, the method: adjoint.cuh).
//
// The one-cell-per-lane kernels leave a call of some thousand cells bound by the latency of one
// lane: two synchronisation steps and their reverse take 430 ms for 30 CB6r5 cells and 1,100 ms
// for 8,000.  Here a reverse step is 3,036 rows on a cell's 35.0 KB in shared memory
// (6 cells per SM; CRACMM2 5,456 rows, 55.7 KB, 3 cells).  Measured: 36 ms for 30 cells, 70 (779) for 900, 221 (1,102) for 8,000, 1,039
// (1,429) for 40,000; CRACMM2 127 (1,640) for 100 and 744 (2,865) for 5,000.  As in coop.cuh the
// latency of a row bounds the small calls, the FP64 pipe the large ones.
//
// The state and its gradients go through the same operations in the same order as there; the
// rate gradients are summed over a warp's cells in the order that it takes them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "adjoint.cuh"
#include "coop.cuh"

namespace coop {

// Next queue position of a warp without a cell; the same in all lanes.
__device__ __forceinline__ bool adj_next(const adj::Args& a, bool need, long long& cell)
{
    unsigned long long pos = 0;
    if (need && (threadIdx.x & 31) == 0) pos = atomicAdd(a.head, 1ull);
    pos = __shfl_sync(0xffffffffu, pos, 0);
    const unsigned long long qlen = (unsigned long long)(a.queue_len > 0 ? a.queue_len : a.ncell);
    if (!need || pos >= qlen) return false;
    cell = a.order ? a.order[pos] : a.cell0 + (long long)pos;
    return true;
}

template <class M, class C>
__device__ __forceinline__ void adj_inputs(const adj::Args& a, long long cell, double* x)
{
    const int sub = threadIdx.x & 31;
    for (int r = sub; r < M::NRXNS; r += 32) {
        const double k = a.rki[(size_t)r * a.ncell + cell];
        x[C::RKI + r] = a.kmult ? k * a.kmult[r] : k;
    }
    for (int i = sub; i < M::ISCHAN; i += 32) x[C::EMIS + i] = a.emis ? a.emis[(size_t)i * a.ncell + cell] : 0.0;
}

// adj::k_adj_forward, with `attempt` of coop.cuh
template <class M, class C>
__global__ void __launch_bounds__(C::MAX_CELLS * 32, 1) k_adj_forward_coop(adj::Args a)
{
    extern __shared__ __align__(128) char coop_smem[];
    const int sub = threadIdx.x & 31;
    double* cst = (double*)(coop_smem + C::TABLE_SMEM);
    double* x = cst + C::NCONST + (size_t)(threadIdx.x / 32) * C::ELEMS;
    for (int i = threadIdx.x; i < C::NCONST; i += blockDim.x) cst[i] = C::constants()[i];
    for (int i = sub; i < C::ELEMS; i += 32) x[i] = 0.0;
    Stream<C> rows;
    rows.start(coop_smem);
    const bool taping = a.tape_off != nullptr;
    const bool pooling = !taping && a.pool_y != nullptr;
    ros3::CellState s;
    ros3::start(s);
    long long cell = -1, base = 0, blk = -1;
    int cap = 0, written = -1, fill = adj::TAPE_BLOCK;
    bool pool_ok = true, drained = false;
    unsigned long long overruns = 0, failed = 0;
    for (;;) {
        const bool need = cell < 0 && !drained;
        if (__any_sync(0xffffffffu, need)) {
            if (adj_next(a, need, cell)) {
                for (int i = sub; i < M::ISCHAN; i += 32) x[C::Y + i] = a.y_in[(size_t)i * a.ncell + cell];
                adj_inputs<M, C>(a, cell, x);
                ros3::start(s);
                written = -1;
                if (taping) {
                    base = a.tape_off[cell] - a.tape_base;
                    cap = a.nsteps[cell];
                }
                blk = -1;
                fill = adj::TAPE_BLOCK;
                pool_ok = true;
            } else if (need) {
                drained = true;
            }
            __syncwarp();
        }
        const bool busy = cell >= 0;
        if (!__syncthreads_or(busy)) break;
        const int nacc = s.st.nsteps;
        double h = s.dt;
        if (s.tnow + h > a.chemstep) h = a.chemstep - s.tnow;
        // Y changes only when a step is accepted: its place on the tape is filled once per accepted step
        double* t = nullptr;
        if (busy && taping && written != nacc && nacc < cap) {
            t = a.tape_y + (size_t)(base + nacc) * M::ISCHAN;
        } else if (busy && pooling && pool_ok && written != nacc) {
            if (fill == adj::TAPE_BLOCK) {
                unsigned long long nb = 0;
                if (sub == 0) nb = atomicAdd(a.pool_head, 1ull);
                nb = __shfl_sync(0xffffffffu, nb, 0);
                if ((long long)nb < a.pool_blocks) {
                    if (sub == 0) a.pool_prev[nb] = blk;
                    blk = (long long)nb;
                    fill = 0;
                } else {
                    pool_ok = false;
                }
            }
            if (pool_ok) t = a.pool_y + (size_t)(blk * adj::TAPE_BLOCK + fill) * M::ISCHAN;
        }
        if (t) {
            for (int i = sub; i < M::ISCHAN; i += 32) t[i] = x[C::Y + i];
            written = nacc;
        }
        __syncwarp();
        attempt<M, C, true>(x, rows, (uint32_t)__cvta_generic_to_shared(cst), s, a.chemstep, a.tol, a.max_iter, busy,
                               nullptr, 0);
        if (!rows.ok) s.st.status |= ros3::ST_NONFINITE;   // a table chunk did not arrive: the cell fails
        if (busy) {
            if (s.st.nsteps != nacc) {
                if (taping) {
                    if (nacc >= cap) overruns++;
                    else if (sub == 0) a.tape_h[base + nacc] = h;
                }
                if (pooling && pool_ok) {
                    if (sub == 0) a.pool_h[blk * adj::TAPE_BLOCK + fill] = h;
                    fill++;
                }
            }
            if (ros3::finished(s, a.chemstep)) {
                if (a.y_out)
                    for (int i = sub; i < M::ISCHAN; i += 32) a.y_out[(size_t)i * a.ncell + cell] = x[C::Y + i];
                if (sub == 0) {
                    if (!taping) a.nsteps[cell] = s.st.nsteps;
                    if (pooling && pool_ok) {
                        a.last_block[cell] = blk;
                        a.last_fill[cell] = fill;
                    } else if (pooling) {
                        atomicAdd(a.pool_ovf, 1u);
                    }
                    if (a.status) a.status[cell] = s.st.status;
                }
                failed += s.st.status != ros3::ST_OK;
                cell = -1;
            }
        }
        __syncwarp();
    }
    rows.drain();
    if (a.counters && sub == 0) {
        if (overruns) atomicAdd(&a.counters[0], overruns);
        if (failed) atomicAdd(&a.counters[2], failed);
    }
}

// adj::reverse_step on the warp's cell: Y and the step size h to LAM, GK and ge (dL/dE of
// the lane's species).  Every warp of the block calls it.
template <class M, class C>
__device__ __forceinline__ void reverse_step(double* __restrict__ x, Stream<C>& rows, uint32_t cst, double h, bool work,
                                             double (&ge)[(M::NSPEC + 31) / 32])
{
    using namespace ros3;
    constexpr int N = M::NSPEC, TRIPS = (N + 31) / 32;
    static_assert(M::ISCHAN == M::NSPEC, "every species is integrated");
    const int sub = threadIdx.x & 31;
    const uint32_t cell = (uint32_t)__cvta_generic_to_shared(x);
    const double dtinv = fpdiv::div(1.0, h);
    const double x21 = C21 * dtinv, x31 = C31 * dtinv, x32 = C32 * dtinv;
    // f(n) for the lane's species, with the same trips in every lane; a warp without work (a cell
    // without steps passes its gradient on) only keeps up with the block
    auto each = [&](auto f) {
#pragma unroll
        for (int i = 0; i < TRIPS; ++i) {
            const int n = sub + i * 32;
            if (work && n < N) f(n, i);
        }
        __syncwarp();
    };
    if (sub == 0) x[C::G] = dtinv * RGAM;
    __syncwarp();
    run<C>(rows, C::STAGE1_ROWS, cell, cst, work);       // the stages as the forward step formed them
    each([&](int n, int) {
        const double k1 = -x[C::V + n];
        x[C::K1 + n] = k1;
        x[C::T + n] = x[C::Y + n] + k1;
    });
    run<C>(rows, C::RHS_ROWS, cell, cst, work);
    each([&](int n, int) { x[C::V + n] = fma(-x21, x[C::K1 + n], -x[C::T + n]); });
    run<C>(rows, C::SOLVE_ROWS, cell, cst, work);
    each([&](int n, int) {
        const double k2 = x[C::V + n];
        x[C::K2 + n] = k2;
        x[C::V + n] = fma(-x32, k2, fma(-x31, x[C::K1 + n], -x[C::T + n]));
    });
    run<C>(rows, C::SOLVE_ROWS, cell, cst, work);
    each([&](int n, int) {                               // clipped components of Y' pass no gradient
        const double k1 = x[C::K1 + n], k3 = x[C::V + n], y = x[C::Y + n];
        x[C::K3 + n] = k3;
        x[C::T + n] = y + k1;
        double yn = fma(B1, k1, y);
        yn = fma(B2, x[C::K2 + n], yn);
        yn = fma(B3, k3, yn);
        const double lam = yn > CONMIN ? x[C::LAM + n] : 0.0;
        x[C::LAM + n] = lam;
        x[C::V + n] = B3 * lam;
    });
    run<C>(rows, C::TSOLVE_ROWS, cell, cst, work);
    each([&](int n, int) {
        const double nu3 = x[C::V + n];
        x[C::NU3 + n] = nu3;
        x[C::V + n] = fma(-x32, nu3, B2 * x[C::LAM + n]);
    });
    run<C>(rows, C::TSOLVE_ROWS, cell, cst, work);
    each([&](int n, int i) {
        const double nu2 = x[C::V + n], phi = -x[C::NU3 + n] - nu2;
        x[C::NU2 + n] = nu2;
        x[C::PHI + n] = phi;
        ge[i] = ge[i] + phi;
        x[C::V + n] = 0.0;
    });
    run<C>(rows, C::JTV_ROWS, cell, cst, work);
    each([&](int n, int) {
        const double lam = x[C::LAM + n], t = x[C::V + n];
        const double mu = fma(-x21, x[C::NU2 + n], fma(-x31, x[C::NU3 + n], B1 * lam));
        x[C::V + n] = mu + t;
        x[C::LAM + n] = lam + t;
    });
    run<C>(rows, C::TSOLVE_ROWS, cell, cst, work);
    each([&](int n, int i) {
        const double phi = -x[C::V + n];
        x[C::PHI + n] = phi;
        ge[i] = ge[i] + phi;
    });
    run<C>(rows, C::GRADIENT_ROWS, cell, cst, work);
    __syncwarp();
}

// adj::k_adj_reverse
template <class M, class C>
__global__ void __launch_bounds__(C::MAX_CELLS * 32, 1) k_adj_reverse_coop(adj::Args a)
{
    constexpr int TRIPS = (M::NSPEC + 31) / 32;
    extern __shared__ __align__(128) char coop_smem[];
    const int sub = threadIdx.x & 31;
    double* cst = (double*)(coop_smem + C::TABLE_SMEM);
    double* x = cst + C::NCONST + (size_t)(threadIdx.x / 32) * C::ELEMS;
    for (int i = threadIdx.x; i < C::NCONST; i += blockDim.x) cst[i] = C::constants()[i];
    for (int i = sub; i < C::ELEMS; i += 32) x[i] = 0.0;
    Stream<C> rows;
    rows.start(coop_smem);
    double ge[TRIPS];
#pragma unroll
    for (int i = 0; i < TRIPS; ++i) ge[i] = 0.0;
    long long cell = -1, base = 0, blk = -1;
    int left = 0, fill = 0;
    const bool pooled = a.last_block != nullptr;
    bool drained = false;
    unsigned long long ncells = 0;
    for (;;) {
        const bool need = cell < 0 && !drained;
        if (__any_sync(0xffffffffu, need)) {
            if (adj_next(a, need, cell)) {
                adj_inputs<M, C>(a, cell, x);
                for (int i = sub; i < M::ISCHAN; i += 32) x[C::LAM + i] = a.lam[(size_t)i * a.ncell + cell];
#pragma unroll
                for (int i = 0; i < TRIPS; ++i) ge[i] = 0.0;
                left = a.nsteps[cell];
                if (pooled) {
                    blk = a.last_block[cell];
                    fill = a.last_fill[cell];
                } else {
                    base = a.tape_off[cell] - a.tape_base;
                }
            } else if (need) {
                drained = true;
            }
            __syncwarp();
        }
        const bool busy = cell >= 0;
        if (!__syncthreads_or(busy)) break;
        const bool work = busy && left > 0;
        double h = 1.0;
        if (work) {
            --left;
            size_t e;
            if (pooled) {
                if (fill == 0) {
                    blk = a.pool_prev[blk];
                    fill = adj::TAPE_BLOCK;
                }
                --fill;
                e = (size_t)(blk * adj::TAPE_BLOCK + fill);
            } else {
                e = (size_t)(base + left);
            }
            const double* t = (pooled ? a.pool_y : a.tape_y) + e * M::ISCHAN;
            for (int i = sub; i < M::ISCHAN; i += 32) x[C::Y + i] = t[i];
            h = (pooled ? a.pool_h : a.tape_h)[e];
        }
        __syncwarp();
        reverse_step<M, C>(x, rows, (uint32_t)__cvta_generic_to_shared(cst), h, work, ge);
        __syncwarp();
        if (busy && left == 0) {
#pragma unroll
            for (int i = 0; i < TRIPS; ++i) {
                const int n = sub + i * 32;
                if (n < M::ISCHAN) {
                    const size_t at = (size_t)n * a.ncell + cell;
                    a.lam[at] = rows.ok ? x[C::LAM + n] : NAN;   // a table chunk did not arrive
                    if (a.grad_emis) a.grad_emis[at] = a.grad_emis[at] + ge[i];
                }
            }
            ncells++;
            cell = -1;
        }
        __syncwarp();
    }
    rows.drain();
    for (int r = sub; r < M::NRXNS; r += 32) {
        const double v = rows.ok ? x[C::GK + r] : NAN;
        if (v != 0.0) atomicAdd(&a.grad_logk[r], v);
    }
    if (a.counters && ncells && sub == 0) atomicAdd(&a.counters[1], ncells);
}

}  // namespace coop
