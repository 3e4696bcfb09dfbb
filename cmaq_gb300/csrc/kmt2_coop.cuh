// Cooperative KMT2: the lanes of a warp integrate one cloudy cell whose workspace lies in shared
// memory.
//
// Fun, Jac_SP, KppDecomp and KppSolve are programs of coop.cuh (mechgen/coop.py, from the
// generated straight-line routines; a step takes 988 rows and 83 blocks of divisions with its
// two f, J, factorisation and four solves), the rate laws of Update_RCONST go to a lane each with their
// temperature factors formed once per cell, and the vectors of Rodas3 are formed over the
// lanes.  Set-up, mapping and redistribution of a cell (kmt2.cuh with stride 1) run in one
// lane.  Every operation of a cell, and its order, is the integrator's: same bits.
//
// The one-cell-per-lane kernels step a cell in 3 ms however few cells there are; a step here
// takes 0.14 ms alone on an SM and 0.23 ms with eight cells, half of it the solves, whose
// divisions follow one another row by row.
#pragma once
#include "coop.cuh"
#include "gen/kmt2_coop_tables.cuh"

#undef KMT2_NS
#undef KMT2_STRIDE
#define KMT2_NS kmt2w
#define KMT2_STRIDE 1
#include "kmt2.cuh"

namespace kmt2_coop {

using namespace kmt2w;
static_assert(Coop::WS_ELEMS == WS_ELEMS, "workspace layout");
static_assert(sizeof(Cell) <= sizeof(double) * Coop::CELL_DOUBLES, "room for the cell's scalars");

constexpr int TRIPS = (NVAR + 31) / 32, W_V = W_K + 3 * NVAR;

// The temperature factors of Update_RCONST's rates, each formed by one lane once per cell
__device__ __forceinline__ void factors(double* ws, const Cell& c)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int i = 0; i < (Coop::NRATE + 31) / 32; ++i) {
        const Rate q = c_kmt2_rate[min(lane + 32 * i, Coop::NRATE - 1)];
        const double keq = q.kind == 0 ? q.p0 : 1.0, kr = q.kind == 0 ? q.p2 : q.p0;
        const double e = kq_exp((q.kind == 0 || q.kind == 2 ? q.p1 : 0.0) * c.delinvt);
        // DISF: KB * ( KEQ * EXP ), KRXN: KR * EXP (KEQ = 1: the product is exact)
        ws[Coop::FACTOR + min(lane + 32 * i, Coop::NRATE - 1)] = kr * (keq * e);
    }
}

// Update_RCONST from the state y: rates of one kind to a lane each; what limits diffusion is
// evaluated together for the two kinds that need it
__device__ __forceinline__ void rates(double* ws, const Cell& c, const double* e3)
{
    const int lane = threadIdx.x & 31;
    const double* y = ws + W_Y;
    const double* f = ws + W_F;
#pragma unroll 1
    for (int i = 0; i < (Coop::NRATE + 31) / 32; ++i) {
        const int j = min(lane + 32 * i, Coop::NRATE - 1);
        const Rate q = c_kmt2_rate[j];
        double k = ws[Coop::FACTOR + j], kt = 0.0;
        bool limited = false;
        if (q.kind == 0) {
            if (q.i0 == 1) k = k * c.gm1;
        } else if (q.kind == 1) {
            k = kq_disb(c, q.p0, q.i0);
        } else if (q.kind == 2) {
            k = kq_krxn_k(c, y, k, q.i0, q.i2);
            if (q.i1 >= 1) {
                kt = kq_kt_qy(c, y, e3[0], e3[1], e3[2]);
                limited = true;
            }
        } else if (kq_iepox_off(c, q.i0)) {
            k = 0.0;
        } else {
            kt = kq_kt_iepox(c, y, f, q.p0, q.p1, q.i0, &k);
            limited = true;
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, limited)) {
            const double d = kq_diffusion_factor(c, kt);
            if (limited) k = k * d;
        }
        if (q.kind >= 2) k = k * c.phi2;
        __syncwarp();
        ws[W_R + q.r] = k;
    }
    __syncwarp();
}

// kq_next without the evaluations at a new step: 0 the cell is finished (L.ierr), 1 another
// attempt of the step, 2 the first attempt of a new one.  The same in all lanes.
__device__ __forceinline__ int next_attempt(const Cell& c, Lane& L, long long* st)
{
    const double roundoff = DBL_EPSILON;
    for (;;) {
        if (L.phase == KL_DONE) {
            st[S_IERR] = L.ierr;
            return 0;
        }
        if (L.phase == KL_ATTEMPT) return 1;
        if (L.phase == KL_PASS) {
            if (!(L.tc < c.tend)) {
                L.phase = KL_DONE;
                continue;
            }
            if (st[S_NKRON] >= 16) {
                L.ierr = -100;
                L.phase = KL_DONE;
                continue;
            }
            st[S_NKRON]++;
            const double tstart = L.tc;
            L.tend = tstart + c.dt;
            L.hmax = fabs(L.tend - tstart);
            L.nstp = L.nacc = 0;
            L.t = tstart;
            L.h = fmin(1.0e-5, L.hmax);
            L.texit = 0.0;
            if (fabs(L.h) <= 10.0 * roundoff) L.h = 1.0e-5;
            L.reject_last = L.reject_more = false;
            L.phase = KL_STEP;
        }
        if (!(fabs(L.t - L.tend) >= roundoff)) {
            kq_return(L, 1);
            continue;
        }
        if (L.nstp > 200000) {
            kq_return(L, -6);
            continue;
        }
        if ((L.t + 0.1 * L.h) == L.t || L.h <= roundoff) {
            kq_return(L, -7);
            continue;
        }
        L.h = fmin(L.h, fabs(L.tend - L.t));
        st[S_NFUN]++;
        st[S_NJAC]++;
        L.phase = KL_ATTEMPT;
        return 2;
    }
}

// ros_PrepareMatrix up to the factorisation, which follows as a program (KppDecomp tests each
// pivot before it works on its row, so the test sees the matrix as it comes in)
__device__ __forceinline__ bool prepare(double* ws, Lane& L, long long* st)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 4
    for (int b = 0; b < LU_NONZERO; b += 32) {
        const int i = min(b + lane, LU_NONZERO - 1);
        ws[W_GHIMJ + i] = -ws[W_JAC0 + i];
    }
    __syncwarp();
    for (int nsing = 0;;) {
        const double ghinv = fpdiv::div(1.0, L.h * 0.5);
        bool singular = false;
#pragma unroll 1
        for (int b = 0; b < NVAR; b += 32) {
            const int d = c_kmt2_diag[min(b + lane, NVAR - 1)];
            const double g = -ws[W_JAC0 + d] + ghinv;
            singular = singular || fabs(g) < DBL_MIN;
            ws[W_GHIMJ + d] = g;
        }
        __syncwarp();
        st[S_NDEC]++;
        if (!__any_sync(0xffffffffu, singular)) return true;
        st[S_NSNG]++;
        if (++nsing > 5) {
            kq_return(L, -8);
            return false;
        }
        L.h = L.h * 0.5;
    }
}

// the error norm and the accept / reject decision of kq_decide; K4 is V, YNEW the new state
__device__ __forceinline__ void decide(double* ws, Lane& L, long long* st)
{
    const int lane = threadIdx.x & 31;
    double* q2 = ws + W_K;   // K1 is not needed any more
#pragma unroll 1
    for (int b = 0; b < NVAR; b += 32) {
        const int i = min(b + lane, NVAR - 1);
        const double ymax = fmax(fabs(ws[W_Y + i]), fabs(ws[W_YNEW + i]));
        const double q = fpdiv::div(0.0 + ws[W_V + i], kq_atol(i) + kq_rtol(i) * ymax);
        __syncwarp();
        q2[i] = q * q;
    }
    __syncwarp();
    double err = 0.0;
#pragma unroll 8
    for (int i = 0; i < NVAR; ++i) err = err + q2[i];
    err = sqrt(err / (double)NVAR);
    err = err > 1.0e-10 ? err : 1.0e-10;
    const double h = L.h;
    double hnew = h * fmin(6.0, fmax(0.2, 0.9 / kq_pow(err, 1.0 / 3.0)));
    L.nstp++;
    st[S_NSTP]++;
    if (err <= 1.0) {
        L.nacc++;
        st[S_NACC]++;
        for (int b = 0; b < NVAR; b += 32) {
            const int i = min(b + lane, NVAR - 1);
            ws[W_Y + i] = ws[W_YNEW + i];
        }
        L.t = L.t + h;
        hnew = fmax(0.0, fmin(hnew, L.hmax));
        if (L.reject_last) hnew = fmin(hnew, h);
        L.texit = L.t;
        L.reject_last = L.reject_more = false;
        L.h = hnew;
        L.phase = KL_STEP;
    } else {
        if (L.reject_more) hnew = h * 0.1;
        L.reject_more = L.reject_last;
        L.reject_last = true;
        L.h = hnew;
        if (L.nacc >= 1) st[S_NREJ]++;
    }
    __syncwarp();
}

// v[i] = EXPR(i) for the species over the lanes (lanes past the end repeat the last; EXPR must
// not read what another lane's assignment writes)
#define KC_FORM(...)                                         \
    _Pragma("unroll") for (int b = 0; b < TRIPS; ++b)        \
    {                                                        \
        const int i = threadIdx.x % 32 + 32 * b;             \
        if (i < NVAR) { __VA_ARGS__ }                        \
    }

// The cells of a call: the block's warps take cells from the queue of `count` and go through the steps
// together.  begin(cell, ws): lane 0's set-up of a new cell, its status; finish(cell, c, L, st, ws): its
// write-back, by the whole warp.  resuming: the queue's positions are lanes that may have left a
// cell, which resume(pos, c, L, st, ws) brings here (-1: none).
template <class Resume, class Begin, class Finish>
__device__ __forceinline__ void integrate(char* smem, unsigned long long* next, long long count, Resume resume,
                                          bool resuming, Begin begin, Finish finish)
{
    const int lane = threadIdx.x & 31;
    double* cst = (double*)(smem + Coop::TABLE_SMEM);
    double* ws = cst + Coop::NCONST + (size_t)(threadIdx.x >> 5) * Coop::ELEMS;
    for (int i = threadIdx.x; i < Coop::NCONST; i += blockDim.x) cst[i] = Coop::constants()[i];
    for (int i = lane; i < Coop::ELEMS; i += 32) ws[i] = i == Coop::ONE ? 1.0 : 0.0;
    coop::Stream<Coop> rows;
    rows.start(smem);
    const uint32_t w0 = (uint32_t)__cvta_generic_to_shared(ws), c0 = (uint32_t)__cvta_generic_to_shared(cst);
    Cell& shared_cell = *(Cell*)(ws + Coop::CELL);
    Cell c{};
    Lane L{};
    long long st[NSTAT];
    double e3[3] = {0.0, 0.0, 0.0};
    long long cell = -1;
    bool drained = false;
    for (;;) {
        if (cell < 0 && !drained) {   // the same in all lanes
            unsigned long long pos = 0;
            do {
                if (lane == 0) pos = atomicAdd(next, 1ull);
                pos = __shfl_sync(0xffffffffu, pos, 0);
                if (resuming && pos < (unsigned long long)count) cell = resume(pos, c, L, st, ws);
            } while (resuming && cell < 0 && pos < (unsigned long long)count);
            if (pos < (unsigned long long)count) {
                int e = 0;
                if (!resuming) {
                    cell = (long long)pos;
                    if (lane == 0) e = begin(cell, shared_cell, ws);
                    e = __shfl_sync(0xffffffffu, e, 0);
                    __syncwarp();
                    c = shared_cell;
                    for (int i = 0; i < NSTAT; ++i) st[i] = 0;
                    L.tc = 0.0;
                    L.ierr = e != 0 ? e - 100 : 1;
                    L.phase = e != 0 ? KL_DONE : KL_PASS;
                }
                if (e == 0) {
                    factors(ws, c);
                    e3[0] = kq_exp(0.0 * c.delinvt);
                    e3[1] = kq_exp(-5530.88 * c.delinvt);
                    e3[2] = kq_exp(-5280.56 * c.delinvt);
                }
            } else {
                drained = true;
            }
            __syncwarp();
        }
        if (!__syncthreads_or(cell >= 0)) break;
        int what = 0;
        if (cell >= 0) {
            what = next_attempt(c, L, st);
            if (what == 0) {
                finish(cell, c, L, st, ws);
                cell = -1;
            } else if (what == 2) {
                // kq_ionic, its two powers in two lanes
                const double lg1 = kq_log_gm1(c, ws + W_Y);
                const double g = kq_rpow(10.0, lane & 1 ? lg1 * 4.0 : lg1);
                c.gm1 = __shfl_sync(0xffffffffu, g, 0);
                const double gm2 = __shfl_sync(0xffffffffu, g, 1);
                c.gm2 = gm2 > 1.0e-30 ? gm2 : 1.0e-30;
                rates(ws, c, e3);
            }
        }
        __syncwarp();
        coop::run<Coop>(rows, Coop::FJAC_ROWS, w0, c0, what == 2);
        bool on = what != 0;
        if (on) on = prepare(ws, L, st);
        __syncwarp();
        coop::run<Coop>(rows, Coop::DECOMP_ROWS, w0, c0, on);
        KC_FORM(ws[W_V + i] = ws[W_FCN0 + i];)
        coop::run<Coop>(rows, Coop::SOLVE_ROWS, w0, c0, on);
        const double h = on ? L.h : 1.0;
        const double c21 = fpdiv::div(4.0, h), c31 = fpdiv::div(1.0, h), c32 = fpdiv::div(-1.0, h),
                     c43 = fpdiv::div(-(8.0 / 3.0), h);
        KC_FORM(const double k1 = ws[W_V + i]; double t = ws[W_FCN0 + i]; if (c21 != 0.0) t = t + c21 * k1;
                ws[W_K + i] = k1; ws[W_V + i] = t; ws[W_YNEW + i] = ws[W_Y + i] + 2.0 * k1;)
        coop::run<Coop>(rows, Coop::SOLVE_ROWS, w0, c0, on);
        KC_FORM(ws[W_K + NVAR + i] = ws[W_V + i];)
        coop::run<Coop>(rows, Coop::FUN_ROWS, w0, c0, on);
        KC_FORM(double t = ws[W_V + i]; if (c31 != 0.0) t = t + c31 * ws[W_K + i];
                if (c32 != 0.0) t = t + c32 * ws[W_K + NVAR + i]; ws[W_V + i] = t;)
        coop::run<Coop>(rows, Coop::SOLVE_ROWS, w0, c0, on);
        KC_FORM(const double k3 = ws[W_V + i]; ws[W_K + 2 * NVAR + i] = k3; ws[W_YNEW + i] = ws[W_YNEW + i] + k3;)
        coop::run<Coop>(rows, Coop::FUN_ROWS, w0, c0, on);
        KC_FORM(double t = ws[W_V + i]; if (c31 != 0.0) t = t + c31 * ws[W_K + i];
                if (c32 != 0.0) t = t + c32 * ws[W_K + NVAR + i];
                if (c43 != 0.0) t = t + c43 * ws[W_K + 2 * NVAR + i]; ws[W_V + i] = t;)
        coop::run<Coop>(rows, Coop::SOLVE_ROWS, w0, c0, on);
        if (on) {
            st[S_NFUN] += 2;
            st[S_NSOL] += 4;
            KC_FORM(ws[W_YNEW + i] = ws[W_YNEW + i] + ws[W_V + i];)
            __syncwarp();
            decide(ws, L, st);
        }
        if (!rows.ok && cell >= 0) {   // a table chunk did not arrive: the cell fails
            L.ierr = -100;
            L.phase = KL_DONE;
        }
        __syncwarp();
    }
    rows.drain();
}
#undef KC_FORM

}  // namespace kmt2_coop
