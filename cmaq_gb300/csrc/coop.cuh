// Cooperative ROS3: the lanes of a warp integrate one cell whose state lies in shared memory.
//
// The one-cell-per-lane kernels stream a 34 KB workspace per cell from DRAM and need ten
// thousands of cells to fill the device: a warp's step attempt takes 1.3 ms however few cells
// there are, because a lone warp issues one FP64 instruction per 64 cycles on GB300.  Here
// the operations of an attempt (f, the iteration matrix and its factors, the solves) are
// dealt out to the 32 lanes by a schedule made with the mechanism (mechgen/coop.py: rows of
// one operation per lane, gen/<mech>_coop.cu), so an attempt of a CB6r5 cell takes 1,440 rows
// (19,954 operations in their 46,080 places), and the state (25.8 KB, 8 cells per SM; CRACMM2
// 42.4 KB, 5) stays in shared memory.
//
// Measured (CB6r5): an attempt takes 212,000 cycles for one warp per SM and 285,000 for eight
// (0.10 and 0.14 ms; the one-cell-per-lane kernel's takes 1.3 ms).  What bounds it: with one
// warp the latency of a row (126-135 cycles, 64 of them the FP64 instruction's), with eight
// the FP64 pipe (168 cycles per row of eight warps, 152 at its measured rate).  CHEM calls from
// the initial state, one cell per lane and here: 105 cells 125 and 11 ms, 11,200 cells 286 and 62 ms,
// 36,000 cells 392 and 179 ms; CRACMM2 11,200 cells 632 and 250 ms.
//
// Every element of a cell's state goes through the same operations in the same order as in
// the generated sequential routines, and the vector updates below repeat ros3.cuh's, so the
// results have the same bits as the one-cell-per-lane kernels'.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "chem_kernels.cuh"
#include "fpdiv.cuh"
#include "queue_kernels.cuh"

namespace coop {

constexpr int UNROLL = 4, AHEAD = 3;
// operation encoding of mechgen/coop.py: acc = +-a * b + c
constexpr uint32_t A_SPECIAL = 1u, C_LOAD = 1u, C_KEEP = 2u, C_MULACC = 4u, D_STORE = 1u << 16, B_CONST = 1u << 17,
                   A_NEG = 1u << 31;

// Shared memory by its 32-bit addresses and predicated instructions: with generic pointers
// and branches a row took ten times its time.
__device__ __forceinline__ double lds(uint32_t p)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p));
    return v;
}
__device__ __forceinline__ double lds_if(uint32_t p, uint32_t on, double other)
{
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q ld.shared.f64 %0, [%1]; }" : "+d"(other) : "r"(p), "r"(on));
    return other;
}
__device__ __forceinline__ void sts_if(uint32_t p, uint32_t on, double v)
{
    asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q st.shared.f64 [%0], %1; }" : : "r"(p), "d"(v), "r"(on) : "memory");
}
__device__ __forceinline__ uint2 ldw(uint32_t p)
{
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(p));
    return v;
}

__device__ __forceinline__ bool try_parity(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{ .reg .pred q; mbarrier.try_wait.parity.shared.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// The chunk of turn t was not there at once: whether it arrives within some `limit` cycles, the same in
// all lanes of the warp.  When it does not, what is in flight to the two buffers has had that time again
// when this returns, and the mark behind the block's barriers spares its warps later waits.
static __device__ __noinline__ bool wait_longer(uint32_t bar, uint32_t t, long long limit)
{
    uint32_t mark;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(mark) : "r"(bar + 16) : "memory");
    if (__any_sync(0xffffffffu, mark != 0)) return false;
    const auto wait = [&](bool both) {
        // looked for once more after the time is up: a warp that was kept from running has not waited
        for (const long long t0 = clock64();;) {
            const bool late = __any_sync(0xffffffffu, clock64() - t0 >= limit);
            bool there = try_parity(bar + 8 * (t & 1u), t >> 1 & 1u);
            if (both) there = try_parity(bar + 8 * ((t + 1) & 1u), (t + 1) >> 1 & 1u) && there;
            there = __all_sync(0xffffffffu, there);
            if (there || late) return there;
        }
    };
    if (wait(false)) return true;
    wait(true);
    asm volatile("st.shared.u32 [%0], %1;" : : "r"(bar + 16), "r"(1u) : "memory");
    return false;
}

// How a chunk of a table travels: one bulk copy, whose arrival completes the barrier's phase.
struct BulkCopy {
    static constexpr long long LIMIT = 1ll << 31;   // a wait gives up after a second
    __device__ __forceinline__ void operator()(uint32_t to, const uint2* from, uint32_t bytes, uint32_t bar)
    {
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" : : "r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     : : "r"(to), "l"(from), "r"(bytes), "r"(bar) : "memory");
    }
};

// The block's stream of table rows: chunks of CHUNK rows, fetched by one bulk copy each into
// two buffers in shared memory that all warps read, in the order of one pass through the
// programs (C::chunk), and again.  A warp that fetched its rows itself waited for the L2 on
// every row.
//
// A chunk that does not arrive ends the stream: `ok` turns false in all lanes of a warp at once
// (no lane waits in a vote of the warp for one that gave up), and the kernels report every cell that the
// warp takes from then on as failed.  Thread 0 fetches only while its own warp has seen every chunk,
// so no buffer is fetched into while a copy to it is under way; when it stops, the other warps' next
// waits end too.  All warps keep to the block's barriers throughout.  What a chunk that is there does
// not need lies out of line (with `ok` tested before the wait, a vote of the block at the release, or
// the wait inline, some calls took up to 5 % more time).
template <class C, class Copy = BulkCopy>
struct Stream {
    static constexpr int W = 32;
    static constexpr uint32_t BYTES = C::CHUNK * W * 8;
    static constexpr uint32_t PITCH = (C::CHUNK + AHEAD) * W * 8;   // rows of zeros end a buffer: looked ahead at only
    uint32_t buf, bar;   // shared addresses: two buffers; two barriers and the mark of wait_longer
    int k;               // chunk of the pass
    uint32_t turn;       // chunks taken so far
    bool ok;             // false: a copy did not arrive (the wait gave up)
    Copy copy;

    __device__ __forceinline__ static int wrap(int c) { return c >= C::PASS ? c - C::PASS : c; }

    // thread 0: the copy of the pass's chunk c into buffer i
    __device__ __forceinline__ void fetch(int c, uint32_t i)
    {
        copy(buf + PITCH * i, C::rows() + (size_t)C::chunk(c) * (C::CHUNK * W), BYTES, bar + 8 * i);
    }

    // smem: C::TABLE_SMEM bytes, 128-byte aligned.  Called by the whole block.
    __device__ __forceinline__ void start(void* smem)
    {
        buf = (uint32_t)__cvta_generic_to_shared(smem);
        bar = buf + 2 * PITCH;
        k = 0;
        turn = 0;
        ok = true;
        for (uint32_t j = threadIdx.x; j < 2 * AHEAD * W; j += blockDim.x)
            *(uint2*)((char*)smem + PITCH * (j / (AHEAD * W)) + BYTES + 8 * (j % (AHEAD * W))) = make_uint2(0u, 0u);
        if (threadIdx.x == 0) {
            asm volatile("st.shared.u32 [%0], %1;" : : "r"(bar + 16), "r"(0u) : "memory");
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(bar) : "memory");
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(bar + 8) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
            asm volatile("fence.proxy.async.shared::cta;" : : : "memory");
            fetch(0, 0);
            fetch(1, 1);
        }
        __syncthreads();
    }

    // whether the chunk of turn t has arrived, the same in all lanes of the warp
    __device__ __forceinline__ bool arrived(uint32_t t)
    {
        if (__all_sync(0xffffffffu, try_parity(bar + 8 * (t & 1u), t >> 1 & 1u))) return true;
        return wait_longer(bar, t, Copy::LIMIT);
    }

    // waits (with a limit) for the current chunk and returns its shared address
    __device__ __forceinline__ uint32_t wait()
    {
        if (!arrived(turn)) ok = false;
        return buf + PITCH * (turn & 1u);
    }

    // the block is through with the current chunk: its buffer takes the one after the next
    __device__ __forceinline__ void release()
    {
        __syncthreads();
        if (threadIdx.x == 0 && ok) {
            asm volatile("fence.proxy.async.shared::cta;" : : : "memory");
            fetch(wrap(k + 2), turn & 1u);
        }
        ++turn;
        k = wrap(k + 1);
    }

    // the copies in flight have arrived (a block must not end before them)
    __device__ __forceinline__ void drain()
    {
        if (!ok) return;
        arrived(turn);
        arrived(turn + 1);
    }
};

// The rows of a one-warp block that goes through its programs by demand: begin names the
// chunks to come, cancel drops those not taken.  It ends as a Stream does.
template <class C, class Copy = BulkCopy>
struct Feed {
    static constexpr int W = 32;
    static constexpr uint32_t BYTES = C::CHUNK * W * 8, PITCH = (C::CHUNK + AHEAD) * W * 8;
    uint32_t buf, bar, turn;
    int next, end;       // chunk to take next, end of what was begun
    bool ok;
    Copy copy;

    __device__ __forceinline__ void fetch(int c, uint32_t i)
    {
        asm volatile("fence.proxy.async.shared::cta;" : : : "memory");
        copy(buf + PITCH * i, C::rows() + (size_t)c * (C::CHUNK * W), BYTES, bar + 8 * i);
    }

    __device__ __forceinline__ void init(void* smem)
    {
        buf = (uint32_t)__cvta_generic_to_shared(smem);
        bar = buf + 2 * PITCH;
        turn = 0;
        next = end = 0;
        ok = true;
        for (uint32_t j = threadIdx.x; j < 2 * AHEAD * W; j += W)
            *(uint2*)((char*)smem + PITCH * (j / (AHEAD * W)) + BYTES + 8 * (j % (AHEAD * W))) = make_uint2(0u, 0u);
        if (threadIdx.x == 0) {
            asm volatile("st.shared.u32 [%0], %1;" : : "r"(bar + 16), "r"(0u) : "memory");
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(bar) : "memory");
            asm volatile("mbarrier.init.shared.b64 [%0], 1;" : : "r"(bar + 8) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
        }
        __syncwarp();
    }

    // chunks [c0, c1): the first two are on their way when it returns
    __device__ __forceinline__ void begin(int c0, int c1)
    {
        if (!ok) return;
        next = c0;
        end = c1;
        __syncwarp();
        if (threadIdx.x == 0) {
            fetch(c0, turn & 1u);
            if (c0 + 1 < c1) fetch(c0 + 1, (turn + 1) & 1u);
        }
    }

    __device__ __forceinline__ bool arrived(uint32_t t)
    {
        if (__all_sync(0xffffffffu, try_parity(bar + 8 * (t & 1u), t >> 1 & 1u))) return true;
        return wait_longer(bar, t, Copy::LIMIT);
    }

    __device__ __forceinline__ uint32_t wait()
    {
        if (!arrived(turn)) ok = false;
        return buf + PITCH * (turn & 1u);
    }

    __device__ __forceinline__ void release()
    {
        __syncwarp();
        if (!ok) return;
        if (threadIdx.x == 0 && next + 2 < end) fetch(next + 2, turn & 1u);
        ++turn;
        ++next;
    }

    __device__ __forceinline__ void cancel()
    {
        for (int n = min(2, end - next); n > 0; --n) {
            if (!arrived(turn)) ok = false;
            ++turn;
        }
        next = end = 0;
        __syncwarp();
    }
};

struct Operands {
    double a, b, c;
};

__device__ __forceinline__ Operands operands(uint2 w, uint32_t cell, uint32_t cst)
{
    Operands o;
    o.a = lds(cell + (w.x & 0xfff8u));
    o.b = lds((w.y & B_CONST ? cst : cell) + (w.x >> 16));
    o.c = lds_if(cell + (w.y & 0xfff8u), w.y & C_LOAD, -0.0);
    return o;
}

// A row of special operations (mechgen/coop.py); lanes without one have kind 0.
static __device__ __noinline__ void special_row(uint2 w, uint32_t cell, uint32_t cst)
{
    enum { RCP = 1, DIV, SQRT, MAX, SIGN };
    const uint32_t kind = w.y & 7u;
    const double a = lds(cell + (w.x & 0xfff8u));
    const double b = lds((w.y & B_CONST ? cst : cell) + (w.x >> 16));
    double r = 0.0;
    if (__any_sync(0xffffffffu, kind == RCP || kind == DIV)) {
        const bool on = kind == RCP || kind == DIV;
        r = fpdiv::div(kind == DIV ? a : 1.0, on ? b : 1.0);
    }
    __syncwarp();
    if (kind == SQRT) r = sqrt(b);
    if (kind == MAX) r = fmax(a, b);
    if (kind == SIGN) r = copysign(1.0, b);
    __syncwarp();   // every lane has read its operands
    sts_if(cell + (w.y & 0xfff8u), w.y & D_STORE, r);
}

// The rows of a program on the warp's cell; every warp of the block calls it (S: Stream or Feed;
// on, the same in all lanes: false to stay with the block without going through the rows).  While row t's FMA is under way, row t - 1's results are stored and then the
// operands of row t + 2 loaded, so that a row waits for neither (with the operands of row
// t + 1 loaded there it waited for them: 135 cycles a row); the schedule knows that a row's
// results can be loaded three rows later.
template <class C, class S>
__device__ __forceinline__ void run(S& st, int rows, uint32_t cell, uint32_t cst, bool on = true)
{
    constexpr int W = 32;
    double acc = 0.0;
    for (int r0 = 0; r0 < rows; r0 += C::CHUNK) {
        const int nr = min(C::CHUNK, rows - r0);
        uint32_t p = st.wait() + (threadIdx.x & 31) * 8;
        __syncwarp();
        uint32_t pending = 0;   // word 1 of the row whose result acc has not been stored yet
        if (st.ok && on) {
            uint2 w = ldw(p), w1 = ldw(p + W * 8), w2 = ldw(p + 2 * W * 8);
            Operands o = operands(w, cell, cst), o1 = operands(w1, cell, cst);
            for (int r = 0; r < nr; r += UNROLL) {   // programs are padded to a multiple of UNROLL rows
                if (__any_sync(0xffffffffu, w.x & A_SPECIAL)) {   // all lanes or none
                    sts_if(cell + (pending & 0xfff8u), pending & D_STORE, acc);
                    pending = 0;
                    __syncwarp();
                    special_row(w, cell, cst);
                    __syncwarp();
                    p += UNROLL * W * 8;
                    w = ldw(p);
                    w1 = ldw(p + W * 8);
                    w2 = ldw(p + 2 * W * 8);
                    o = operands(w, cell, cst);
                    o1 = operands(w1, cell, cst);
                    continue;
                }
#pragma unroll
                for (int j = 0; j < UNROLL; ++j) {
                    const uint2 w3 = ldw(p + (j + 3) * (W * 8));
                    double a = w.y & C_MULACC ? acc : o.a;
                    const double c = w.y & C_KEEP ? acc : o.c;
                    a = __hiloint2double(__double2hiint(a) ^ (int)(w.y & A_NEG), __double2loint(a));
                    const double before = acc;
                    acc = fma(a, o.b, c);
                    sts_if(cell + (pending & 0xfff8u), pending & D_STORE, before);
                    __syncwarp();
                    o = o1;
                    o1 = operands(w2, cell, cst);
                    pending = w.y;
                    w = w1;
                    w1 = w2;
                    w2 = w3;
                }
                p += UNROLL * W * 8;
            }
        }
        sts_if(cell + (pending & 0xfff8u), pending & D_STORE, acc);
        st.release();
    }
}

// One attempt of ros3::attempt_phased (rbsolver.F:344-589) on the warp's cell; the scalar state
// is kept identically by the lanes.  Every warp of the block calls it; one with
// active == false leaves the FP64 pipe to the others (27,880 EBI cells 270 -> 259 ms, 12 ROS3 calls of
// 10,527 cells 148 -> 146 ms).  yave: the cell's
// time integral of Y in global memory (stride ystride), or nullptr.  ADJ: of the adjoint's forward pass.
template <class M, class C, bool ADJ = false>
__device__ __forceinline__ void attempt(double* __restrict__ x, Stream<C>& rows, uint32_t cst, ros3::CellState& s,
                                        double chemstep, ros3::Tol tol, int max_iter, bool active, double* yave,
                                        long long ystride)
{
    using namespace ros3;
    constexpr int W = 32, N = M::NSPEC, TRIPS = (N + W - 1) / W;
    static_assert(M::ISCHAN == M::NSPEC, "every species is integrated");
    const int sub = threadIdx.x & 31;
    const uint32_t cell = (uint32_t)__cvta_generic_to_shared(x);
    bool go = active;
    if (go && s.iter >= max_iter) { s.st.status |= ST_MAXITER; go = false; }
    double dt = 1.0, tend = 0.0;
    if (go) {
        s.iter++;
        dt = s.dt;
        tend = s.tnow + dt;
        if (tend > chemstep) { dt = chemstep - s.tnow; tend = chemstep; }
    }
    __syncwarp();
    const double dtinv = fpdiv::div(1.0, dt);
    if (sub == 0) x[C::G] = dtinv * RGAM;
    // f(Y), the factors, stage 1: V = -K1
    run<C>(rows, C::STAGE1_ROWS, cell, cst, active);
    // The species loops run the same trips in every lane: lanes that left a loop early went
    // through the rows that follow apart from the others, at twice the time.
#pragma unroll
    for (int i = 0; i < TRIPS; ++i) {   // stage 2
        const int n = sub + i * W;
        if (n < N) {
            const double k1 = -x[C::V + n];
            x[C::K1 + n] = k1;
            x[C::T + n] = x[C::Y + n] + k1;
        }
    }
    run<C>(rows, C::RHS_ROWS, cell, cst, active);
    {
        const double x1 = C21 * dtinv;
#pragma unroll
        for (int i = 0; i < TRIPS; ++i) {
            const int n = sub + i * W;
            if (n < N) x[C::V + n] = fma(-x1, x[C::K1 + n], -x[C::T + n]);
        }
    }
    run<C>(rows, C::SOLVE_ROWS, cell, cst, active);
    {   // stage 3
        const double x1 = C31 * dtinv;
        const double x2 = C32 * dtinv;
#pragma unroll
        for (int i = 0; i < TRIPS; ++i) {
            const int n = sub + i * W;
            if (n < N) {
                const double k2 = x[C::V + n];
                x[C::K2 + n] = k2;
                const double t = fma(-x1, x[C::K1 + n], -x[C::T + n]);
                x[C::V + n] = fma(-x2, k2, t);
            }
        }
    }
    run<C>(rows, C::SOLVE_ROWS, cell, cst, active);
    // solution (T) and weighted error (K1) of each species, then the norm in species order
    int bad = 0;
#pragma unroll 1
    for (int i = 0; i < TRIPS; ++i) {
        const int n = min(sub + i * W, N - 1);   // lanes past the end repeat the last species
        const double k1 = x[C::K1 + n];
        const double k2 = x[C::K2 + n];
        const double k3 = x[C::V + n];
        double yp = fma(B1, k1, x[C::Y + n]);
        yp = fma(B2, k2, yp);
        yp = fma(B3, k3, yp);
        const double ytol = fma(tol.rtol, fabs(yp), tol.atol);
        double e = D1 * k1;
        e = fma(D2, k2, e);
        e = fma(D3, k3, e);
        const double qn = fpdiv::div(e, ytol);
        __syncwarp();
        x[C::T + n] = yp;
        x[C::K1 + n] = qn;
        bad |= !isfinite(yp);
        __syncwarp();
    }
    for (int o = W / 2; o > 0; o >>= 1) bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    double err = 0.0;
#pragma unroll 8
    for (int n = 0; n < N; ++n) {
        const double q = x[C::K1 + n];
        err = fma(q, q, err);
    }
    const double maxerr = fmax_keepnan(fmax(0.0, UROUND), sqrt(err * tol.rnspec));
    const bool accept = go && maxerr <= 1.0;
#pragma unroll
    for (int i = 0; i < TRIPS; ++i) {
        const int n = sub + i * W;
        if (accept && n < N) {
            const double yn = fmax(x[C::T + n], CONMIN);
            if (yave) yave[(size_t)n * ystride] = yave[(size_t)n * ystride] + 0.5 * (x[C::Y + n] + yn) * dt;
            x[C::Y + n] = yn;
        }
    }
    if (accept) {
        double dtfac = step_factor<ADJ>(maxerr);
        s.st.nsteps++;
        if (bad) s.st.status |= ST_NONFINITE;
        s.tnow = tend;
        dtfac = s.lpass ? fmax(FACMIN, fmin(dtfac, FACMAX)) : fmax(FACMIN, fmin(dtfac, FACONE));
        s.dt = fmin(DTMAX, fmax(tol.dtmin, dtfac * dt));
        s.lpass = true;
    } else if (go) {
        if (s.st.nfails == 0 && s.tnow == 0.0) s.st.nbad_starts++;
        s.st.nfails++;
        s.dt = FACMIN * dt;
        s.lpass = false;
        if (s.dt < tol.dtmin) s.st.status |= ST_DT_UNDERFLOW;
    }
    __syncwarp();
}

// One CHEM call on the cells of the work queue (rates from the rate-constant pass).  The
// block's warps go through the attempts together.  Dynamic shared memory: the table chunks,
// the constants, then ELEMS doubles per cell.
template <class M, class C>
__global__ void __launch_bounds__(C::MAX_CELLS * 32, 1) k_chem_ros3_coop(chem::GridArgs a, chem::QueueArgs q)
{
    constexpr int W = 32;
    extern __shared__ __align__(128) char coop_smem[];
    const int sub = threadIdx.x & 31;
    double* cst = (double*)(coop_smem + C::TABLE_SMEM);
    double* x = cst + C::NCONST + (size_t)(threadIdx.x / W) * C::ELEMS;
    for (int i = threadIdx.x; i < C::NCONST; i += blockDim.x) cst[i] = C::constants()[i];
    for (int i = sub; i < C::ELEMS; i += W) x[i] = 0.0;
    Stream<C> rows;
    rows.start(coop_smem);
    const bool unfinished = q.over.count != nullptr;   // goes on with the cells that were handed over
    const unsigned long long qlen = unfinished ? *q.over.count : chem::queue_len(q, a.ncell);
    ros3::CellState s;
    ros3::start(s);
    long long cell = -1;
    bool sun = false, drained = false;
    unsigned long long acc_steps = 0, rej_steps = 0, failed = 0, sunlit = 0, sun_att = 0;
    for (;;) {
        const bool need = cell < 0 && !drained;
        if (__any_sync(0xffffffffu, need)) {
            unsigned long long pos = 0;
            if (need && sub == 0) pos = atomicAdd(q.head, 1ull);
            pos = __shfl_sync(0xffffffffu, pos, 0);
            if (need && pos < qlen && unfinished) {
                cell = q.over.cell[pos];
                const int slot = q.over.slot[pos];
                const double* ws = a.ws + (size_t)(slot >> 5) * ((size_t)M::WS_ELEMS * 32) + (slot & 31);
                for (int i = sub; i < M::ISCHAN; i += W) x[C::Y + i] = ws[(M::OFF_Y + i) * 32];
                for (int r = sub; r < M::NRXNS; r += W) x[C::RKI + r] = a.rki_all[(size_t)r * a.ncell + cell];
                if (a.yave)
                    for (int i = sub; i < M::ISCHAN; i += W) a.yave[(size_t)i * a.ncell + cell] = ws[(M::OFF_YAVE + i) * 32];
                sun = a.sun_all[cell] != 0;
                s = q.over.state[pos];
            } else if (need && pos < qlen) {
                cell = q.cell0 + (q.order ? q.order[pos] : (long long)pos);
                const float svol = __fdiv_rn(1.0f, a.dens[cell]);
                for (int i = sub; i < M::ISCHAN; i += W) {   // as gather_cell_pass
                    const float conc = a.cgrid[(size_t)a.cgrid_index[i] * a.ncell + cell];
                    const float v = a.convert[i] ? __fmul_rn(__fmul_rn(a.fwd_conv[i], svol), conc) : conc;
                    x[C::Y + M::iold2new(i)] = (double)fmaxf(v, chem::CONCMIN_F);
                }
                for (int r = sub; r < M::NRXNS; r += W) x[C::RKI + r] = a.rki_all[(size_t)r * a.ncell + cell];
                if (a.yave)
                    for (int i = sub; i < M::ISCHAN; i += W) a.yave[(size_t)i * a.ncell + cell] = 0.0;
                sun = a.sun_all[cell] != 0;
                ros3::start(s);
            } else if (need) {
                drained = true;
            }
        }
        const bool busy = cell >= 0;
        if (!__syncthreads_or(busy)) break;
        attempt<M, C>(x, rows, (uint32_t)__cvta_generic_to_shared(cst), s, a.chemstep, a.tol, a.max_iter, busy,
                         busy && a.yave ? a.yave + cell : nullptr, a.ncell);
        if (!rows.ok) s.st.status |= ros3::ST_NONFINITE;   // a table chunk did not arrive: the cell fails
        const bool end = busy && ros3::finished(s, a.chemstep);
        if (__any_sync(0xffffffffu, end) && end) {
            const double densd = (double)a.dens[cell];
            for (int i = sub; i < M::ISCHAN; i += W) {   // as scatter_cell, store_yave
                const int old = M::inew2old(i);
                const double y = x[C::Y + i];
                const float v = a.convert[old] ? (float)((a.rev_conv[old] * densd) * y) : (float)y;
                a.cgrid[(size_t)a.cgrid_index[old] * a.ncell + cell] = v;
                if (a.yave) {
                    double& yv = a.yave[(size_t)i * a.ncell + cell];
                    yv = yv / a.chemstep;
                }
            }
            if (sub == 0) {
                acc_steps += s.st.nsteps;
                rej_steps += s.st.nfails;
                failed += s.st.status != ros3::ST_OK;
                sunlit += sun;
                if (sun) sun_att += s.st.nsteps + s.st.nfails;
                if (a.cell_status) a.cell_status[cell] = s.st.status;
                if (a.cell_steps) a.cell_steps[cell] = s.st.nsteps + s.st.nfails;
            }
            cell = -1;
        }
        __syncwarp();
    }
    rows.drain();
    if (a.counters && sub == 0) {
        if (acc_steps) atomicAdd(&a.counters[0], acc_steps);
        if (rej_steps) atomicAdd(&a.counters[1], rej_steps);
        if (failed) atomicAdd(&a.counters[2], failed);
        if (sunlit) atomicAdd(&a.counters[3], sunlit);
        if (sun_att) atomicAdd(&a.counters[4], sun_att);
    }
}

// A launch asks for its cells' bytes; the kernel's limit is always set to MAX_CELLS' (a limit per
// launch would be another thread's, which launches on a handle of its own).
template <class C>
inline size_t smem_bytes(int cells)
{
    return C::TABLE_SMEM + sizeof(double) * ((size_t)C::NCONST + (size_t)cells * C::ELEMS);
}

}  // namespace coop
