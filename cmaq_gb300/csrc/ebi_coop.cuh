// Cooperative EBI: the lanes of a warp integrate one cell whose state lies in shared memory.
//
// One Backward-Euler iteration is one pass through the cell's program (coop.cuh: HRRATES,
// HRG1-HRG4 and HRPRODLOSS dealt out to the lanes by mechgen/coop.py: 156 rows and 15 blocks of
// divisions, square roots and maxima for CB6r5, 356 and 15 for CRACMM2), then HRSOLVER's species loops over the
// lanes with votes for convergence.  Every value is computed with the same operations in the
// same order as in ebi::iterate and the oracle: same bits.
//
// An EBI call lasts as long as its slowest cell (thousands of iterations), so what counts is
// the latency of an iteration: 26 us, about half of it the rows' (130 cycles each, as in
// coop.cuh), the rest divisions and the species loops.  The earlier warp kernel walked index
// tables in global memory and ran the group solutions HRG1-HRG4 on one lane: 0.2 ms.  A first
// call of 27,880 CB6r5 cells took 862-901 ms with it and the one-cell-per-lane kernel for the
// quick cells, and takes 252-290 ms here (by the inputs).
#pragma once
#include "coop.cuh"
#include "ebi.cuh"

namespace chem {

// Rate constants and sunlight flags of cells [c0, c1) by whole warps, for the cooperative kernel
template <class M>
__global__ void __launch_bounds__(THREADS_PER_BLOCK, 1) k_ebi_rconst_pass(GridArgs a, long long c0, long long c1,
                                                                          double* rki, uint8_t* sunlit)
{
    const long long nwarps = (long long)gridDim.x * WARPS_PER_BLOCK;
    const long long warp = (long long)blockIdx.x * WARPS_PER_BLOCK + (threadIdx.x >> 5);
    double* ws = warp_ws<M>(a.ws, warp);
    for (long long base = c0 + warp * 32; base < c1; base += nwarps * 32) {
        const long long c = base + (threadIdx.x & 31);
        if (c < c1) {
            const bool sun = rconst_cell_ebi<M>(a, c, ws);
            for (int r = 0; r < M::NRXNS; ++r) rki[(size_t)r * a.ncell + c] = ws[(M::OFF_RKI + r) * 32];
            sunlit[c] = sun ? 1 : 0;
        }
    }
}

// The rate constants of the warp's cell without that pass, by its first lane; returns the sunlight
// flag.  Out of line: the iterations' code stays as it is.
template <class M>
__device__ __noinline__ bool ebi_rates_of_cell(const GridArgs& a, long long cell, double* __restrict__ rki)
{
    const int lane = threadIdx.x & 31;
    const size_t warp = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    double* ws = a.ws + warp * ((size_t)M::WS_ELEMS * 32);   // the first lane's column
    int sun = 0;
    if (lane == 0) sun = rconst_cell_ebi<M>(a, cell, ws) ? 1 : 0;
    sun = __shfl_sync(0xffffffffu, sun, 0);
    __syncwarp();
    for (int r = lane; r < M::NRXNS; r += 32) rki[r] = ws[(M::OFF_RKI + r) * 32];
    return sun != 0;
}

// What follows an iteration's program in ebi::iterate: the species updates, the convergence
// test and HRSOLVER's bookkeeping.  notmax: the lane's species' NOTMAX flags (bit i: species
// lane + 32 i).
template <class M, class E>
__device__ __forceinline__ void ebi_coop_update(double* __restrict__ x, ebi::State& s, uint32_t notmax, double* yv,
                                                long long ystride)
{
    using namespace ebi;
    constexpr int TRIPS = (M::NSPEC + 31) / 32, ETRIPS = (M::EBI_N_EBISP + 31) / 32;
    const int lane = threadIdx.x & 31;
    const double dtc = s.dtc;
#pragma unroll 1
    for (int i = 0; i < ETRIPS; ++i) {
        const int sp = M::ebi_ebisp(min(lane + 32 * i, M::EBI_N_EBISP - 1));   // lanes past the end repeat the last
        const double yc = x[E::YC + sp];
        const double ycp = yc * fpdiv::div(x[E::YC0 + sp] + x[E::PROD + sp] * dtc, yc + x[E::LOSS + sp] * dtc);
        __syncwarp();
        x[E::YCP + sp] = ycp;
    }
    __syncwarp();
    for (int k = 0; k < M::EBI_NPNEG; ++k) {   // negative product stoichiometry: all lanes the same
        const int p = M::ebi_pneg(k);
        const double pneg = x[E::PNEG + p];
        if (pneg > 0.0) {
            const double fxdloss = pneg * dtc;
            const double yc0 = x[E::YC0 + p], prod = x[E::PROD + p];
            double ycp = 0.0;
            if (!(fxdloss >= yc0 + prod * dtc)) {
                const double varloss = fmax(x[E::LOSS + p] - pneg, ZERO);
                ycp = fpdiv::div(yc0 + prod * dtc - fxdloss, 1.0 + fpdiv::div(varloss * dtc, x[E::YC + p]));
            }
            __syncwarp();
            x[E::YCP + p] = ycp;
        }
    }
    __syncwarp();
    bool conv = true, mxfl = false;
#pragma unroll 1
    for (int i = 0; i < TRIPS; ++i) {
        const int sp = min(lane + 32 * i, M::NSPEC - 1);
        const double ycp = fmax(ZERO, x[E::YCP + sp]);
        const double yc = x[E::YC + sp];
        const double aerror = fmax(fabs(yc - ycp), EPSLON);
        const double rerror = fpdiv::div(aerror, fmax(FLOOR, fabs(yc + ycp)));
        if (rerror > M::ebi_rtol(sp) || aerror > 1.0e-5) conv = false;
        if (ycp > MAXPRED && (notmax >> i & 1u)) {
            mxfl = true;
            conv = false;
        }
        __syncwarp();
        x[E::YC + sp] = ycp;
    }
    __syncwarp();
    conv = __all_sync(0xffffffffu, conv);
    mxfl = __any_sync(0xffffffffu, mxfl);
    s.lebi_conv = conv;
    if (conv) {
        if (yv)   // each lane its own species
            for (int i = lane; i < M::NSPEC; i += 32) {
                double& y = yv[(size_t)M::iold2new(i) * ystride];
                y = fma(0.5 * dtc, x[E::YC + i] + x[E::YC0 + i], y);
            }
        s.ninr++;
        s.substep_start = true;
        if (s.ninr > s.n_inr_steps) {
            s.nebi++;
            if (s.nebi > s.n_ebi_steps) {
                s.done = true;
            } else {
                if (s.nbkups != 0) {
                    s.nbkups = 0;
                    s.n_inr_steps = 1;
                    s.dtc = s.tmstep;
                }
                s.ninr = 1;
            }
        }
    } else if (mxfl || s.iter >= M::EBI_NEBITER) {
        s.nbkups++;
        if (s.dtc > DTMIN) {
            for (int i = lane; i < M::NSPEC; i += 32) x[E::YC + i] = x[E::YC0 + i];
            s.dtc = 0.5 * s.dtc;
            s.n_inr_steps = 1 << (s.nbkups < 30 ? s.nbkups : 30);
            s.ninr = 1;
            s.substep_start = true;
        } else {
            s.status |= ST_DT_UNDERFLOW;
            s.done = true;
        }
    }
    __syncwarp();
}

// One EBI CHEM call, a cell per warp from the work queue.  Rates come from k_ebi_rconst_pass or,
// without its arrays, from the warp's first lane in its column of the workspace, while the block
// waits.  The block's warps go through the iterations together.  Dynamic shared memory as k_chem_ros3_coop's.
template <class M, class E>
__global__ void __launch_bounds__(E::MAX_CELLS * 32, 1) k_chem_ebi_warp(GridArgs a, QueueArgs q, EbiArgs e)
{
    extern __shared__ __align__(128) char coop_smem[];
    const int lane = threadIdx.x & 31;
    double* cst = (double*)(coop_smem + E::TABLE_SMEM);
    double* x = cst + E::NCONST + (size_t)(threadIdx.x >> 5) * E::ELEMS;
    for (int i = threadIdx.x; i < E::NCONST; i += blockDim.x) cst[i] = E::constants()[i];
    for (int i = lane; i < E::ELEMS; i += 32) x[i] = i == E::Z ? 0.0 : 1.0;   // a warp without a cell: finite numbers
    coop::Stream<E> rows;
    rows.start(coop_smem);
    const uint32_t cell0 = (uint32_t)__cvta_generic_to_shared(x), cst0 = (uint32_t)__cvta_generic_to_shared(cst);
    const unsigned long long qlen = queue_len(q, a.ncell);
    ebi::State s;
    s.done = true;
    long long cell = -1;
    uint32_t notmax = 0;
    bool sun = false, drained = false;
    double* yv = nullptr;
    unsigned long long iters = 0, failed = 0, sunlit = 0;
    for (;;) {
        if (cell < 0 && !drained) {   // the same in all lanes
            unsigned long long pos = 0;
            if (lane == 0) pos = atomicAdd(q.head, 1ull);
            pos = __shfl_sync(0xffffffffu, pos, 0);
            if (pos < qlen) {
                cell = q.cell0 + (q.order ? q.order[pos] : (long long)pos);
                const float inv_dens = __fdiv_rn(1.0f, a.dens[cell]);
                notmax = 0;
                for (int i = lane; i < M::NSPEC; i += 32) {
                    const double v = gather_conc_ebi(a, e, cell, i, inv_dens);
                    x[E::YC + i] = v;
                    x[E::YC0 + i] = x[E::YCP + i] = x[E::PROD + i] = x[E::LOSS + i] = x[E::PNEG + i] = 0.0;
                    if (v <= ebi::MAXPRED) notmax |= 1u << (i >> 5);
                }
                if (a.rki_all) {
                    for (int r = lane; r < M::NRXNS; r += 32) x[E::RKI + r] = a.rki_all[(size_t)r * a.ncell + cell];
                    sun = a.sun_all[cell] != 0;
                } else {
                    sun = ebi_rates_of_cell<M>(a, cell, x + E::RKI);
                }
                s.tmstep = e.tmstep;
                s.dtc = e.tmstep;
                s.n_ebi_steps = e.n_ebi_steps;
                s.nebi = 1;
                s.ninr = 1;
                s.n_inr_steps = 1;
                s.nbkups = 0;
                s.iter = 0;
                s.total_iter = 0;
                s.lebi_conv = true;
                s.substep_start = true;
                s.done = false;
                s.status = ebi::ST_OK;
                yv = a.yave ? a.yave + cell : nullptr;
                if (yv) ycddm_zero<M>(yv, a.ncell, lane, 32);
            } else {
                drained = true;
            }
            __syncwarp();
        }
        const bool busy = cell >= 0;
        if (!__syncthreads_or(busy)) break;
        bool go = busy;
        if (go && s.total_iter >= a.max_iter) {
            s.status |= ebi::ST_MAXITER;
            s.done = true;
            go = false;
        }
        if (go) {
            if (s.substep_start) {
                if (s.lebi_conv)
                    for (int i = lane; i < M::NSPEC; i += 32) x[E::YC0 + i] = x[E::YC + i];
                s.substep_start = false;
                s.iter = 0;
            }
            s.iter++;
            s.total_iter++;
            if (lane == 0) x[E::DTC] = s.dtc;
        }
        __syncwarp();
        coop::run<E>(rows, E::ITERATION_ROWS, cell0, cst0, go);
        if (!rows.ok) {   // a table chunk did not arrive: the cell fails
            s.status |= ebi::ST_MAXITER;
            s.done = true;
        } else if (go) {
            ebi_coop_update<M, E>(x, s, notmax, yv, a.ncell);
        }
        __syncwarp();
        if (busy && s.done) {
            if (yv) ycddm_finish<M>(yv, a.ncell, a.chemstep, lane, 32);
            const float dens = a.dens[cell];
            for (int sp = lane; sp < M::NSPEC; sp += 32) {   // write-back (hrdriver.F:446-454)
                const double y = fmax(x[E::YC + sp], 1.0e-30);
                const float v = a.convert[sp] ? (float)((double)__fmul_rn(e.rev[sp], dens) * y) : (float)y;
                a.cgrid[(size_t)a.cgrid_index[sp] * a.ncell + cell] = v;
            }
            if (lane == 0) {
                iters += s.total_iter;
                failed += s.status != ebi::ST_OK;
                sunlit += sun;
                if (a.cell_status) a.cell_status[cell] = s.status;
                if (a.cell_steps) a.cell_steps[cell] = s.total_iter;
            }
            cell = -1;
        }
        __syncwarp();
    }
    rows.drain();
    if (a.counters && lane == 0) {
        if (iters) atomicAdd(&a.counters[0], iters);
        if (failed) atomicAdd(&a.counters[2], failed);
        if (sunlit) atomicAdd(&a.counters[3], sunlit);
    }
}

}  // namespace chem
