// Cooperative SMVGEAR: the lanes of a warp integrate one cell whose workspace lies in shared memory.
//
// SMVGEAR's stiffest cells need tens of thousands of Newton iterations in one call, a call
// lasts as long as its slowest cell, and on this GPU one FP64 warp instruction takes 64
// cycles whatever its number of active lanes, so a lone cell must spread its FP64 work over
// the lanes to advance.  The control flow (gear::advance) runs in every lane; the predictor
// matrix and its factors, f and the corrector's solve are programs of coop.cuh (for CB6r5
// 440, 168 and 280 rows).  One-warp blocks, 4 per SM for CB6r5 and 3 for CRACMM2, so that
// cells at different points of SMVGEAR do not wait for one another; each block has its own
// feed of rows.  Cells come from the work queue; results equal k_gear's bit for bit.
//
// Measured: a first call of 252 CB6r5 cells (its stiffest cell alone) 680 -> 226 ms, 8,000 cells
// 953 ms (4,000 took 6.6 s); the table-driven routines before walked index tables in global memory.
#pragma once
#include "coop.cuh"
#include "gear.cuh"

namespace chem {

template <class M, class G, bool GRID>
__global__ void __launch_bounds__(32) k_gear_warp(GridArgs a, QueueArgs q, GearArgs g)
{
    extern __shared__ __align__(128) char gear_smem[];
    const int lane = threadIdx.x & 31;
    double* cst = (double*)(gear_smem + G::TABLE_SMEM);
    double* x = cst + G::NCONST;           // R1DELT, 0, 1, then the cell's workspace
    double* sm = x + G::WORKSPACE;
    for (int i = lane; i < G::NCONST; i += 32) cst[i] = G::constants()[i];
    if (lane == 0) {
        x[G::Z] = 0.0;
        x[G::ONE] = 1.0;
    }
    const uint32_t cell0 = (uint32_t)__cvta_generic_to_shared(x), cst0 = (uint32_t)__cvta_generic_to_shared(cst);
    coop::Feed<G> rows;
    rows.init(gear_smem);
    constexpr int RHS0 = (G::PREDICTOR_ROWS + G::CHUNK - 1) / G::CHUNK;   // the rhs program's first chunk
    // lane 0's slot of this warp's global workspace, for the gather (stride 32)
    double* wsg = a.ws + (size_t)blockIdx.x * ((size_t)M::WS_ELEMS * 32);
    const gear::Coef* K = g.coef;
    const unsigned long long qlen = queue_len(q, a.ncell);
    unsigned long long acc = 0, rej = 0, failed = 0, sunlit = 0, sun_att = 0;
    for (;;) {
        unsigned long long pos = 0;
        if (lane == 0) pos = atomicAdd(q.head, 1ull);
        pos = __shfl_sync(0xffffffffu, pos, 0);
        if (pos >= qlen) break;
        const long long cell = q.cell0 + (q.order ? q.order[pos] : (long long)pos);
        bool sun;
        if (GRID) {
            if (a.rki_all) {   // rates from the rate-constant pass; concentrations as gather_cell
                const float svol = __fdiv_rn(1.0f, a.dens[cell]);
                for (int i = lane; i < M::ISCHAN; i += 32) {
                    const float conc = a.cgrid[(size_t)a.cgrid_index[i] * a.ncell + cell];
                    const float v = a.convert[i] ? __fmul_rn(__fmul_rn(a.fwd_conv[i], svol), conc) : conc;
                    sm[M::GEAR_CNEW + M::iold2new(i)] = fmax((double)v, 1.0e-30);
                }
                for (int r = lane; r < M::NRXNS; r += 32) sm[M::OFF_RKI + r] = a.rki_all[(size_t)r * a.ncell + cell];
                sun = a.sun_all[cell] != 0;
            } else {
                int sflag = 0;
                if (lane == 0) sflag = gather_cell<M>(a, cell, wsg, true) ? 1 : 0;
                sun = __shfl_sync(0xffffffffu, sflag, 0) != 0;
                __syncwarp();
                for (int i = lane; i < M::NSPEC; i += 32) sm[M::GEAR_CNEW + i] = wsg[(M::OFF_Y + i) * 32];
                for (int r = lane; r < M::NRXNS; r += 32) sm[M::OFF_RKI + r] = wsg[(M::OFF_RKI + r) * 32];
            }
        } else {
            for (int i = lane; i < M::NSPEC; i += 32) sm[M::GEAR_CNEW + i] = g.y[(size_t)i * a.ncell + cell];
            for (int r = lane; r < M::NRXNS; r += 32) sm[M::OFF_RKI + r] = g.rk[(size_t)r * a.ncell + cell];
            sun = g.night[cell] == 0;
        }
        __syncwarp();
        gear::State s;
        gear::start<M, 1, true>(s, sm, sun, K, GRID && a.yave != nullptr);
        for (;;) {
            // the rows of f and of the corrector's solve travel while the control flow runs
            rows.begin(RHS0, G::PASS);
            const bool more = gear::advance<M, 1, true>(sm, s, K, a.chemstep) == gear::NEED_F;
            __syncwarp();
            if (!more) break;
            if (s.need_jac) {
                rows.cancel();
                rows.begin(0, G::PASS);
                for (int b = 0; b < M::ISCHAN; b += 32) {   // CEFF of grpderiv.F:147-155
                    const int i = min(b + lane, M::ISCHAN - 1);
                    const double y = sm[M::GEAR_CNEW + i];
                    x[G::Q + i] = y <= 1.0e-30 ? 0.0 : y;
                }
                if (lane == 0) x[G::R1] = s.r1delt;
                coop::run<G>(rows, G::PREDICTOR_ROWS, cell0, cst0);
            }
            coop::run<G>(rows, G::RHS_ROWS, cell0, cst0);
            gear::floor_gloss<M, 1, true>(sm);
            if (s.label == gear::L_ITER_POST) {
                gear::corrector_rhs<M, 1, true>(sm, s.delt);
                coop::run<G>(rows, G::SOLVE_ROWS, cell0, cst0);
            }
            rows.cancel();
            if (!rows.ok) {   // a table chunk did not arrive: the cell fails
                s.st.status |= gear::ST_NONFINITE;
                break;
            }
        }
        rows.cancel();
        if (GRID) {   // write-back as scatter_cell
            const double densd = (double)a.dens[cell];
            for (int i = lane; i < M::ISCHAN; i += 32) {
                const int old = M::inew2old(i);
                const double y = sm[M::GEAR_CNEW + i];
                const float v = a.convert[old] ? (float)((a.rev_conv[old] * densd) * y) : (float)y;
                a.cgrid[(size_t)a.cgrid_index[old] * a.ncell + cell] = v;
                if (a.yave) a.yave[(size_t)i * a.ncell + cell] = sm[M::GEAR_CAVEG + i];
            }
        } else {
            for (int i = lane; i < M::NSPEC; i += 32) g.y[(size_t)i * a.ncell + cell] = sm[M::GEAR_CNEW + i];
            if (g.cell_stats && lane == 0) {
                int* o = g.cell_stats + (size_t)8 * cell;
                o[0] = s.st.nsteps; o[1] = s.st.ncfail; o[2] = s.st.nefail; o[3] = s.st.npderiv;
                o[4] = s.st.nsubfun; o[5] = s.st.nnewt; o[6] = s.st.maxord; o[7] = s.st.status;
            }
        }
        __syncwarp();   // the next cell overwrites the shared workspace
        if (lane == 0) {
            const int att = s.st.nsteps + s.st.ncfail + s.st.nefail;
            acc += s.st.nsteps;
            rej += s.st.ncfail + s.st.nefail;
            failed += s.st.status != gear::ST_OK;
            sunlit += s.lsun;
            if (s.lsun) sun_att += att;
            if (a.cell_status) a.cell_status[cell] = s.st.status;
            if (a.cell_steps) a.cell_steps[cell] = att;
        }
    }
    if (a.counters && lane == 0) {
        atomicAdd(&a.counters[0], acc);
        atomicAdd(&a.counters[1], rej);
        atomicAdd(&a.counters[2], failed);
        atomicAdd(&a.counters[3], sunlit);
        atomicAdd(&a.counters[4], sun_att);
    }
}

}  // namespace chem
