// Device-driven gauge-eliminated PCG (PressureWorkspace::solve_loaded,
// src/pressure.rs:577-740) on the sealed-box operator.
//
// One PCG iteration of the Jacobi method is two slab passes:
//   pass 1  d <- z + beta*d, q = K d, curvature = d.q           (24N bytes)
//   pass 2  q = K d re-applied from d, p += alpha*d, r -= alpha*q,
//           z = r/D stored, r.r and r.z                         (48N bytes)
// instead of the four array passes of the reference (88N); q is never stored. Scalars never leave
// the device: the last block of each pass takes solve_loaded's decision
// (alpha, beta, breakdown, candidate, restart) and writes it to SolveState.
// The true-residual check and the restart run as flag-gated kernels at the end
// of each captured chunk of iterations, so the host only launches graphs and
// polls one word per chunk.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "pcg.hpp"
#include "pcg_device.cuh"
#include "resident.hpp"
#include "slab.cuh"
#include "solve_state.cuh"
#include "stencil.cuh"

namespace rb200 {

constexpr int EW = 256;
constexpr int EW_CAP = 148 * 8;

// ------------------------------------------------------------------ init
__global__ void __launch_bounds__(EW) k_init_sums(GridDev g, SolveState* st, const double* __restrict__ b,
                                                  double* __restrict__ p, Partials part) {
    init_sums_body(g, st, b, p, part, whole_launch());
}

template <int KIND>
__global__ void __launch_bounds__(EW) k_load_residual(GridDev g, SolveState* st, const double* b,
                                                      double* d0, double* d1, double* __restrict__ r,
                                                      double* __restrict__ z, int mode, Partials part,
                                                      rb200_trace* trace) {
    load_residual_body<KIND>(g, st, b, d0, d1, r, z, mode, part, trace, whole_launch());
}

// precondition_jacobi (src/pressure.rs:534-575) as a primitive: z = r/D on
// every row but the eliminated gauge row (z[0] = 0), and r.z over rows >= 1.
__global__ void __launch_bounds__(EW) k_precondition_jacobi(GridDev g, const double* __restrict__ r,
                                                            double* __restrict__ z, Partials part,
                                                            double* __restrict__ rz_out) {
    __shared__ BlockReduce<1, 0> sm;
    Neu acc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.cells; c += gridDim.x * blockDim.x) {
        if (c == 0) {
            z[0] = 0.0;
            continue;
        }
        int i, j, k;
        cell_coords(g, c, i, j, k);
        const int m = diag_mask(g, i, j, k);
        const double rc = r[c];
        const double zc = div_diag(rc, g.diag[m], g.rdiag[m]);
        z[c] = zc;
        acc.add(rc * zc);
    }
    dd sums[1] = {acc.as_dd()};
    double none[1];
    block_reduce<1, 0>(sm, sums, none);
    if (publish_and_check_last<1, 0>(part, blockIdx.x, gridDim.x, sums, none)) {
        fold_partials<1, 0>(part, gridDim.x, sm, sums, none);
        if (threadIdx.x == 0) *rz_out = dd_value(sums[0]);
    }
}

// ------------------------------------------------------------ slab staging
// Stage one or two slabs of the block's brick into shared memory.
template <int ZC>
__device__ __forceinline__ void stage_issue(const GridDev& g, const TmaMaps& maps, uint64_t* bar, double* sm0,
                                            const double* src0, const CUtensorMap* m0, double* sm1,
                                            const double* src1, const CUtensorMap* m1, int x0, int y0, int k0) {
    const int tid = threadIdx.x + TX * threadIdx.y;
    if (maps.use) {
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
        }
        __syncthreads();
        if (tid == 0) {
            mbar_expect_tx(bar, (sm1 ? 2u : 1u) * Slab<ZC>::BYTES);
            tma_load_slab(sm0, m0, x0 - 2, y0 - 1, k0 - 1, bar);
            if (sm1) tma_load_slab(sm1, m1, x0 - 2, y0 - 1, k0 - 1, bar);
        }
    } else {
        slab_issue_rows<ZC>(g, sm0, src0, x0, y0, k0);
        if (sm1) slab_issue_rows<ZC>(g, sm1, src1, x0, y0, k0);
        cp_async_commit();
    }
}

// Wait for the staged slabs. A TMA wait that runs out records an execution
// error in the solver state, waits once more for the copy in flight, and the
// whole block returns false (the decision is block-uniform).
__device__ __forceinline__ bool stage_wait(const TmaMaps& maps, uint64_t* bar, SolveState* st) {
    bool ok = true;
    if (maps.use)
        ok = mbar_wait_bounded(bar, 0);
    else
        cp_async_wait_all();
    ok = __syncthreads_and(ok) != 0;
    if (!ok) {
        if (threadIdx.x == 0 && threadIdx.y == 0) {
            st->status = RB200_EXECUTION;
            st->flags = st->flags | F_DONE | F_STOP;
        }
        mbar_wait_bounded(bar, 0);
        __syncthreads();
    }
    return ok;
}

// ------------------------------------------------------------ pass 1
// Direction update fused with q = K d and the curvature d.q
// (src/pressure.rs:657-668, :720-731). The slabs hold z and the old direction;
// the new direction d = z (restart) or z + beta*d is formed in shared memory
// for the whole slab (out-of-domain and gauge entries are 0 in both inputs, so
// they stay 0), then each cell's row of K d is applied.
template <int ZC>
__global__ void __launch_bounds__(TILE_THREADS) k_pass1(GridDev g, SolveState* st, const double* __restrict__ zarr,
                                                        double* d0, double* d1, double* __restrict__ qout,
                                                        const __grid_constant__ TmaMaps maps, Partials part,
                                                        rb200_trace* trace) {
    using S = Slab<ZC>;
    extern __shared__ __align__(128) double smem[];
    __shared__ BlockReduce<1, 0> red;
    __shared__ __align__(8) uint64_t bar;
    double* sz = smem;
    double* sd = smem + S::SIZE;
    const int flags = st->flags;
    if (flags & F_STOP) return;
    const bool fresh = (flags & F_REPLACED) != 0;
    const double beta = st->beta;
    const int dsel = st->dsel;
    const double* __restrict__ src = dsel ? d1 : d0;
    double* __restrict__ dst = dsel ? d0 : d1;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, k0 = blockIdx.z * ZC;
    stage_issue<ZC>(g, maps, &bar, sz, zarr, &maps.z, fresh ? nullptr : sd, src, dsel ? &maps.d1 : &maps.d0, x0,
                    y0, k0);
    if (!stage_wait(maps, &bar, st)) return;
    const int tid = threadIdx.x + TX * threadIdx.y;
    if (!fresh)
        for (int e = tid; e < S::SIZE; e += TILE_THREADS) sz[e] = sz[e] + beta * sd[e];
    __syncthreads();
    Neu acc;
    const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
    if (i < g.n[0] && j < g.n[1]) {
        const int kend = min(ZC, g.n[2] - k0);
        int e = S::own(threadIdx.x, threadIdx.y, 0);
        int c = cell_idx(g, i, j, k0);
        const int plane = g.n[0] * g.n[1];
        for (int q = 0; q < kend; ++q, e += S::PLANE, c += plane) {
            Neigh v = slab_neigh<ZC>(sz, e);
            double qv = c == 0 ? 0.0 : apply_row(g, i, j, k0 + q, v);
            dst[c] = v.c;
            if (qout) qout[c] = qv;
            acc.add(v.c * qv);
        }
    }
    dd sums[1] = {acc.as_dd()};
    double none[1];
    block_reduce<1, 0>(red, sums, none);
    const int nb = nblocks3();
    if (publish_and_check_last<1, 0>(part, block_id3(), nb, sums, none)) {
        fold_partials<1, 0>(part, nb, red, sums, none);
        if (tid3() == 0) decide_pass1(st, trace, dd_value(sums[0]), flags, dsel);
    }
}

// ------------------------------------------------------------ pass 2
// p += alpha*d, r -= alpha*K d (src/pressure.rs:669-680) with K d re-applied
// from the direction slab, the recursive norm, and the preconditioner's local
// part: Jacobi z = r/D with r.z (precondition_jacobi, :534-575); red-black SGS
// stores y = r/D on the red cells.
// PRE: 0 Jacobi (z = r/D and r.z here), 1 red-black SGS (y = r/D on red
// cells), 2 none (lexicographic SGS forms z in its sweeps).
template <int ZC, int PRE>
__global__ void __launch_bounds__(TILE_THREADS) k_pass2(GridDev g, SolveState* st, double* __restrict__ p,
                                                        double* __restrict__ r, double* __restrict__ z,
                                                        const double* d0, const double* d1,
                                                        const __grid_constant__ TmaMaps maps, Partials part,
                                                        rb200_trace* trace) {
    using S = Slab<ZC>;
    extern __shared__ __align__(128) double smem[];
    __shared__ BlockReduce<2, 0> red;
    __shared__ __align__(8) uint64_t bar;
    const int flags = st->flags;
    if (flags & F_STOP) return;
    const double alpha = st->alpha;
    const int dsel = st->dsel;
    const double* __restrict__ d = dsel ? d1 : d0;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, k0 = blockIdx.z * ZC;
    stage_issue<ZC>(g, maps, &bar, smem, d, dsel ? &maps.d1 : &maps.d0, nullptr, nullptr, nullptr, x0, y0, k0);
    const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
    const bool own = i < g.n[0] && j < g.n[1];
    const int kend = own ? min(ZC, g.n[2] - k0) : 0;
    const int plane = g.n[0] * g.n[1];
    const int c0 = own ? cell_idx(g, i, j, k0) : 0;
    double pv[ZC], rv[ZC];
#pragma unroll
    for (int q = 0; q < ZC; ++q) {
        if (q < kend) {
            pv[q] = p[c0 + q * plane];
            rv[q] = r[c0 + q * plane];
        }
    }
    if (!stage_wait(maps, &bar, st)) return;
    Neu acc_rr, acc_rz;
#pragma unroll
    for (int q = 0; q < ZC; ++q) {
        if (q >= kend) break;
        const int c = c0 + q * plane;
        if (c == 0) continue;  // gauge row: p[0], r[0] stay 0
        Neigh v = slab_neigh<ZC>(smem, S::own(threadIdx.x, threadIdx.y, q));
        const int k = k0 + q;
        double qv = apply_row(g, i, j, k, v);
        p[c] = pv[q] + alpha * v.c;
        double rc = rv[q] - alpha * qv;
        r[c] = rc;
        acc_rr.add(rc * rc);
        if (PRE == 0) {
            const int m = diag_mask(g, i, j, k);
            double zc = div_diag(rc, g.diag[m], g.rdiag[m]);
            z[c] = zc;
            acc_rz.add(rc * zc);
        } else if (PRE == 1 && ((i + j + k) & 1) == 0) {
            z[c] = rc / diag_at(g, i, j, k);
        }
    }
    dd sums[2] = {acc_rr.as_dd(), acc_rz.as_dd()};
    double none[1];
    block_reduce<2, 0>(red, sums, none);
    const int nb = nblocks3();
    if (publish_and_check_last<2, 0>(part, block_id3(), nb, sums, none)) {
        fold_partials<2, 0>(part, nb, red, sums, none);
        if (tid3() == 0) decide_pass2(st, trace, dd_value(sums[0]), dd_value(sums[1]), flags, PRE == 0);
    }
}

// ------------------------------------------------------------ true residual
// true_report (src/pressure.rs:432-456): t = b - K p on every cell (the gauge
// row included), |t|_2, max|t|, max|t|*dt/V; then the acceptance and restart
// decisions of solve_loaded (:686-715). t is kept in the spare direction
// buffer for a restart.
template <int ZC>
__global__ void __launch_bounds__(TILE_THREADS) k_true_residual(GridDev g, SolveState* st, const double* __restrict__ b,
                                                                const double* __restrict__ p, double* d0, double* d1,
                                                                const __grid_constant__ TmaMaps maps, Partials part,
                                                                rb200_trace* trace) {
    using S = Slab<ZC>;
    extern __shared__ __align__(128) double smem[];
    __shared__ BlockReduce<3, 1> red;
    __shared__ __align__(8) uint64_t bar;
    const int flags = st->flags;
    if (!(flags & F_NEED_TRUE)) return;
    double* __restrict__ spare = st->dsel ? d0 : d1;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, k0 = blockIdx.z * ZC;
    stage_issue<ZC>(g, maps, &bar, smem, p, &maps.p, nullptr, nullptr, nullptr, x0, y0, k0);
    if (!stage_wait(maps, &bar, st)) return;
    Neu acc;
    double total = 0.0;
    double gauge_sq = 0.0;  // t[0]^2 when this thread holds cell 0
    double mx[1] = {0.0};
    const int i = x0 + threadIdx.x, j = y0 + threadIdx.y;
    if (i < g.n[0] && j < g.n[1]) {
        const int kend = min(ZC, g.n[2] - k0);
        const int plane = g.n[0] * g.n[1];
        int c = cell_idx(g, i, j, k0);
        int e = S::own(threadIdx.x, threadIdx.y, 0);
        for (int q = 0; q < kend; ++q, e += S::PLANE, c += plane) {
            Neigh v = slab_neigh<ZC>(smem, e);
            double t = b[c] - apply_row(g, i, j, k0 + q, v);
            spare[c] = t;
            acc.add(t * t);
            total += t;
            if (c == 0) gauge_sq = t * t;
            mx[0] = fmax(mx[0], fabs(t));
        }
    }
    // the second sum leaves out the gauge row: |t[1..]|^2; the third is of t itself
    dd sums[3] = {acc.as_dd(), dd_add1(acc.as_dd(), -gauge_sq), dd{total, 0.0}};
    block_reduce<3, 1>(red, sums, mx);
    const int nb = nblocks3();
    if (publish_and_check_last<3, 1>(part, block_id3(), nb, sums, mx)) {
        fold_partials<3, 1>(part, nb, red, sums, mx);
        if (tid3() == 0) {
            extra_of(st).load_mean = dd_value(sums[2]) / g.cells;
            decide_true(st, trace, dd_value(sums[0]), dd_value(sums[1]), mx[0], flags, g.volume);
        }
    }
}

// ------------------------------------------------------------ multigrid outer passes
// Flexible CG around the FP32 multigrid preconditioner: q = K d is formed by
// pass 1 for d.q and recomputed from d where the update and the finish need it
// (no q vector); the finish pass takes the FP32 V-cycle output as z (FP64),
// reduces r.z and z.r_old and takes the decision with the
// Polak-Ribiere beta = (z.r - z.r_old) / (z_old.r_old) (tolerant of a
// preconditioner that is symmetric only up to FP32 rounding). The residual
// before the update stays available in a second buffer. This update serves
// grids whose finest level is solved inside the cluster kernel: r stays in the
// first buffer (the V-cycle's first half-sweep reads it there) and r_old is
// copied to the second.
__global__ void __launch_bounds__(EW) k_mg_update(GridDev g, SolveState* st, double* __restrict__ p,
                                                  double* __restrict__ r, double* __restrict__ r_old,
                                                  const double* d0, const double* d1, Partials part,
                                                  rb200_trace* trace) {
    __shared__ BlockReduce<2, 0> red;
    const int flags = st->flags;
    if (flags & F_STOP) return;
    const double alpha = st->alpha, mean = extra_of(st).mean;
    const double* __restrict__ d = st->dsel ? d1 : d0;
    Neu acc;
    double total = 0.0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.cells; c += gridDim.x * blockDim.x) {
        int i, j, k;
        cell_coords(g, c, i, j, k);
        p[c] = p[c] + alpha * d[c];
        const double ro = r[c];
        double rc = (ro - mean) - alpha * kd_at(g, d, i, j, k, c);
        r_old[c] = ro;
        r[c] = rc;
        acc.add(rc * rc);
        total += rc;
    }
    dd sums[2] = {acc.as_dd(), dd{total, 0.0}};
    double none[1];
    block_reduce<2, 0>(red, sums, none);
    if (publish_and_check_last<2, 0>(part, blockIdx.x, gridDim.x, sums, none)) {
        fold_partials<2, 0>(part, gridDim.x, red, sums, none);
        if (threadIdx.x == 0) {
            if (flags & F_PROFILE) return;
            extra_of(st).mean = dd_value(sums[1]) / g.cells;
            int it = st->it + 1;
            st->it = it;
            double recursive_l2 = sqrt(dd_value(sums[0]));
            st->recursive_l2 = recursive_l2;
            if (trace) trace[it - 1].recursive_l2 = recursive_l2;
            if (recursive_l2 <= st->threshold || it == st->max_it) st->flags = flags | F_CANDIDATE;
        }
    }
}

// ------------------------------------------------------------ lexicographic SGS
// precondition_sgs (src/pressure.rs:467-532): forward
//   y_i = (r_i + sum_{lower d} w_d y_{i-s_d}) / D_i    (d = X, Y, Z in order)
// then reverse
//   z_i = y_i + (sum_{upper d} w_d z_{i+s_d}) / D_i
// over rows 1..N-1 (row 0 is the eliminated gauge row, z_0 = 0). Each row
// depends only on its lower (upper) neighbours, so any order that respects
// those dependencies computes the reference's lexicographic sweep bit for bit
// (the reference's own tiled wavefront, src/sgs.rs:56-104, uses the same
// fact).
//
// One launch runs both sweeps over units of 16 x 8 lines along x. A thread
// owns a line: at step t of a unit, line (j, k) of it does cell i = t - j - k of
// its direction, so that the x neighbour is the thread's own last value, and the
// y and z neighbours' are in shared memory since the step before; one barrier a
// step. What bounds a sweep is that serial chain: n0 + n1 + n2 steps of 160 to
// 240 cycles (shared load, the sums, each rounded, the division, shared store,
// barrier), and some 3 us for each unit boundary on the way. So a
// line's step holds nothing else: a missing neighbour is a -0.0 (adding its
// product changes no bit), the ends of a line have a path of their own, two
// warps fetch the next 16 steps' values and store the last 16's through shared
// memory, 16 consecutive cells of a line at a time, and two warps fetch the
// unit's incoming faces SGS_AHEAD steps before their use and send the outgoing
// ones a step after it.
//
// A boundary value crosses as two 64-bit words, each a 32-bit half under a tag
// that holds the sweep's number, which makes a word its own flag. The words lie
// in the direction buffer that the iteration does not hold (the next pass
// overwrites it whole); the tags are the bits of signalling NaNs, which no
// arithmetic leaves there, and both buffers start as zeros. A number returns
// after 131072 applications, and the words of a solve's last one may lie there
// that long: they are the reverse sweep's (each of its words takes the place of
// the forward sweep's word of that face cell), and a reverse sweep's reads come
// after its own unit's forward sweep, which has written those words again.
//
// A block takes the next slot of a queue (slots 0..U-1: the units in wave order
// jb + kb ascending; U..2U-1: the same list backwards for the reverse sweep). A
// slot only waits for slots taken before it, by blocks that are running, so the
// queue cannot deadlock whatever the number of resident blocks. A unit's
// reverse sweep reads the z of its own forward sweep, published by a state word
// (release); it starts after the forward sweep of every unit, since its upper
// neighbours' reverse sweeps come after the forward sweep of the last unit,
// which comes after every other forward sweep.
//
// us per iteration of a solve, tiles of 8^3 cells with a block barrier for each
// of their 22 hyperplanes / this: 32^3 138 / 83, 63x48x37 226 / 102, 96^3
// 453 / 208, 256x20x20 417 / 124. Units of 16 x 16 lines took 113, 222 and 148
// for the last three (two line warps to a scheduler); with face words in flight
// left as they were after a wait, each to be waited for in turn, 108, 207 and 124.
//
// Every wait is bounded: a wait that runs out raises the abort word, which
// ends every other wait, and marks the solve as failed (execution error).
constexpr int SGS_UJ = 16, SGS_UK = 8;         // lines of a unit along y and z
constexpr int SGS_C = 16;                      // steps of a chunk
constexpr int SGS_P = SGS_C + 1;               // pitch of a line's chunk (bank conflicts)
constexpr int SGS_LINES = SGS_UJ * SGS_UK;
constexpr int SGS_MOVERS = 64;                 // threads that move the chunks
constexpr int SGS_STEPPERS = SGS_LINES + 64;   // the lines and the faces' two warps: they share the step barrier
constexpr int SGS_THREADS = SGS_STEPPERS + SGS_MOVERS;
constexpr int SGS_AHEAD = 6;                   // steps between a face word's load and its use
constexpr int SGS_VP = SGS_UJ + 2;             // pitch of the step values
constexpr int SGS_VALS = (SGS_UK + 1) * SGS_VP;
constexpr int SGS_CHUNK = SGS_LINES * SGS_P;
constexpr int SGS_RING = 8;                    // steps of face words in shared memory
constexpr size_t kSmemSgs = (3 * SGS_CHUNK + 2 * SGS_VALS + SGS_RING * 64) * sizeof(double);
constexpr unsigned kSgsSpins = 1u << 22;
constexpr unsigned kSgsTag = 0x7ff40000u;      // | sweep number mod 2^18

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void ld_pair(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_tagged(unsigned long long* p, double v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(p), "l"(t | unsigned(__double2loint(v))),
                 "l"(t | unsigned(__double2hiint(v)))
                 : "memory");
}
// Without a branch: 8 bytes or nothing read (zeros written then); a store or none.
__device__ __forceinline__ void cp_async8_if(bool on, double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(on ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void st_cg_if(bool on, double* p, double v) {
    asm volatile("{\n.reg .pred q;\nsetp.ne.s32 q, %0, 0;\n@q st.global.cg.f64 [%1], %2;\n}\n" ::"r"(int(on)), "l"(p),
                 "d"(v)
                 : "memory");
}
// Kept out of the step's code, which rarely needs it.
__device__ __noinline__ double sgs_divide(double a, double b) { return a / b; }

// The steppers' barrier; at the end of a chunk the whole block's.
__device__ __forceinline__ void sgs_step_barrier() {
    asm volatile("bar.sync 1, %0;\n" ::"n"(SGS_STEPPERS) : "memory");
}
__device__ __forceinline__ void sgs_step_end(int t, int steps) {
    if (t + 1 == steps || t % SGS_C == SGS_C - 1)
        __syncthreads();
    else
        sgs_step_barrier();
}

// A unit: its place among the units, its first line and its lines.
struct SgsUnit {
    int jb, kb, nj, nk, j0, k0;
};
// The incoming face words of line `line` of axis y or z (face f lies between
// units f and f + 1 of that axis).
__device__ __forceinline__ size_t sgs_word(const GridDev& g, const SgsFlow& f, bool z, int face, int line) {
    const size_t row = z ? size_t(f.nj - 1) * g.n[2] + size_t(face) * g.n[1] + line
                         : size_t(face) * g.n[2] + line;
    return 2 * row * g.n[0];
}

// Polls a face word until it holds the tag; all lanes of a warp. False when the
// wait ran out or another did.
__device__ __noinline__ bool sgs_poll(const unsigned long long* p, unsigned tag, bool want, unsigned* ctl,
                                      unsigned long long* lo, unsigned long long* hi) {
    for (unsigned n = 1;; ++n) {
        unsigned long long a = 0, b = 0;
        if (want) ld_pair(p, a, b);
        if (__all_sync(0xffffffffu, !want || (unsigned(a >> 32) == tag && unsigned(b >> 32) == tag))) {
            *lo = a;
            *hi = b;
            return true;
        }
        const bool out = n > kSgsSpins || ((n & 7u) == 0u && *(volatile const unsigned*)(ctl + 1) != 0u);
        if (__any_sync(0xffffffffu, out)) return false;
    }
}

// The slot of the step values (first buffer) that line q of an incoming face
// fills: beside row q + 1 for the y face, above column q + 1 for the z face. A
// face has as many slots as a unit has lines across it.
__host__ __device__ constexpr int sgs_face_slots(bool z) { return z ? SGS_UJ : SGS_UK; }
__host__ __device__ constexpr int sgs_face_slot(bool z, int q) { return z ? q + 1 : (q + 1) * SGS_VP; }
constexpr bool sgs_face_slots_fit() {
    for (int z = 0; z < 2; ++z)
        for (int q = 0; q < sgs_face_slots(z != 0); ++q)
            if (q >= 16 || sgs_face_slot(z != 0, q) >= SGS_VALS) return false;
    return true;
}
static_assert(sgs_face_slots_fit(), "a face has at most 16 lanes, its slots lie inside one buffer of step values");

// The incoming faces' warp of a unit: lane q fetches line q of the y face, lane
// 16 + q of the z face, one step of the unit at a time. The words come through
// asynchronous copies, since a load into registers would be waited for at the
// next branch (with strong loads into registers, 63x48x37 takes 29.2 ms a solve
// for 17.4). Such a copy is a weak access that nothing orders after the other
// block's relaxed store. It needs no order: it goes to L2, where that store is
// performed, it returns an old or a new word, each word tells by itself which,
// and an old one is polled for with strong loads, after which the copies behind
// it are made again.
template <bool REV>
__device__ __forceinline__ void sgs_faces(const GridDev& g, const SgsFlow& f, const SgsUnit& U, int steps,
                                          const unsigned long long* words, unsigned tag, double* vals,
                                          unsigned long long* ring, int* s_fail) {
    const int lane = threadIdx.x & 31, q = lane & 15, n0 = g.n[0];
    const bool zf = lane >= 16;
    const int b = zf ? U.kb : U.jb, nb = zf ? f.nk : f.nj, lines = zf ? U.nj : U.nk;
    const bool has = q < lines && (REV ? b + 1 < nb : b > 0);
    const int line = (zf ? U.j0 : U.k0) + (REV ? lines - 1 - q : q);
    const unsigned long long* base = words + (has ? sgs_word(g, f, zf, REV ? b : b - 1, line) : 0);
    double* const to = vals + sgs_face_slot(zf, q);
    if (!has && q < sgs_face_slots(zf)) to[0] = to[SGS_VALS] = -0.0;
    if (!__any_sync(0xffffffffu, has)) {
        __syncthreads();
        for (int t = 0; t < steps; ++t) sgs_step_end(t, steps);
        return;
    }
    const unsigned len = has ? unsigned(n0) : 0u;
    auto wanted = [&](int t) { return unsigned(t - q) < len; };
    auto word = [&](int t) { return base + 2 * (REV ? n0 - 1 - (t - q) : t - q); };
    auto fetch = [&](int t) {
        if (wanted(t)) cp_async16_cg(ring + (t % SGS_RING) * 64 + 2 * lane, word(t));
        cp_async_commit();
    };
    unsigned long long lo, hi;  // the word pair of the next step
    auto read = [&](int t) {
        lo = ring[(t % SGS_RING) * 64 + 2 * lane];
        hi = ring[(t % SGS_RING) * 64 + 2 * lane + 1];
    };
    bool dead = false;
    auto deliver = [&](int t) {
        const bool want = wanted(t);
        const bool ok = !want || (unsigned(lo >> 32) == tag && unsigned(hi >> 32) == tag);
        if (!__all_sync(0xffffffffu, ok) && !dead) {
            if (sgs_poll(want ? word(t) : words, tag, want, f.ctl, &lo, &hi)) {
                for (int e = 1; e < SGS_AHEAD - 1; ++e) fetch(t + e);  // those in flight came too early as well
            } else {
                dead = true;
                if (lane == 0) {
                    atomicExch(f.ctl + 1, 1u);
                    *s_fail = 1;
                }
            }
        }
        if (want) to[((t + 1) & 1) * SGS_VALS] = __hiloint2double(int(unsigned(hi)), int(unsigned(lo)));
    };
    for (int t = 0; t < SGS_AHEAD; ++t) fetch(t);
    asm volatile("cp.async.wait_group %0;\n" ::"n"(SGS_AHEAD - 2) : "memory");
    read(0);
    deliver(0);
    read(1);
    __syncthreads();
    for (int t = 0; t < steps; ++t) {
        deliver(t + 1);
        fetch(t + SGS_AHEAD);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(SGS_AHEAD - 2) : "memory");
        read(t + 2);
        sgs_step_end(t, steps);
    }
    cp_async_wait_all();
}

// The outgoing faces' warp of a unit, one step behind the lines: lane q sends
// line q of the y face, lane 16 + q of the z face.
template <bool REV>
__device__ __forceinline__ void sgs_send(const GridDev& g, const SgsFlow& f, const SgsUnit& U, int steps,
                                         unsigned long long* words, unsigned tag, const double* vals) {
    const int lane = threadIdx.x & 31, q = lane & 15, n0 = g.n[0];
    const bool zf = lane >= 16;
    const int b = zf ? U.kb : U.jb, nb = zf ? f.nk : f.nj, lines = zf ? U.nj : U.nk;
    const bool has = q < lines && (REV ? b > 0 : b + 1 < nb);
    const int line = (zf ? U.j0 : U.k0) + (REV ? lines - 1 - q : q);
    unsigned long long* const base = words + (has ? sgs_word(g, f, zf, REV ? b - 1 : b, line) : 0);
    const double* const from = vals + (zf ? U.nk * SGS_VP + q + 1 : (q + 1) * SGS_VP + U.nj);
    const int back = q + (zf ? U.nk : U.nj) - 1;
    auto send = [&](int t) {
        const int i = t - back;
        if (has && unsigned(i) < unsigned(n0))
            st_tagged(base + 2 * (REV ? n0 - 1 - i : i), from[(t & 1) * SGS_VALS], tag);
    };
    __syncthreads();
    for (int t = 0; t < steps; ++t) {
        if (t > 0) send(t - 1);
        sgs_step_end(t, steps);
    }
    send(steps - 1);
}

// The movers of a unit: chunk c + 1 comes in (r, in reverse z) and chunk c - 1
// goes out to z while chunk c is computed.
template <bool REV>
__device__ __forceinline__ void sgs_move(const GridDev& g, const SgsUnit& U, int steps, const double* __restrict__ r,
                                         double* z, double* chunks) {
    constexpr int ROWS = SGS_MOVERS / SGS_C, PASSES = SGS_UJ / ROWS;
    const int x = threadIdx.x - SGS_STEPPERS, n0 = g.n[0], sz = n0 * g.n[1];
    const int ts = x % SGS_C, row = x / SGS_C;
    const double* __restrict__ src = REV ? z : r;
    // slot ts of line (tj, tk) of a chunk is cell i = 16 chunk + ts - tj - tk of
    // the line in its direction; from one tk to the next it moves by `hop`
    const int hop = REV ? 1 - sz : sz - 1;
    auto start = [&](int chunk, int tj, int& i) {
        i = chunk * SGS_C + ts - tj;
        return (REV ? n0 - 1 - i : i) + n0 * (U.j0 + (REV ? U.nj - 1 - tj : tj)) +
               sz * (U.k0 + (REV ? U.nk - 1 : 0));
    };
    auto load = [&](int chunk) {
        for (int h = 0; h < PASSES; ++h) {
            const int tj = row + h * ROWS;
            int i, c = start(chunk, tj, i);
            double* const dst = chunks + (chunk % 3) * SGS_CHUNK + tj * SGS_P + ts;
            const unsigned lines = tj < U.nj ? unsigned(U.nk) : 0u;
#pragma unroll
            for (int tk = 0; tk < SGS_UK; ++tk) {
                const bool on = unsigned(tk) < lines && unsigned(i - tk) < unsigned(n0);
                cp_async8_if(on, dst + tk * SGS_UJ * SGS_P, on ? src + (c + tk * hop) : src);
            }
        }
        cp_async_commit();
    };
    auto store = [&](int chunk) {
        for (int h = 0; h < PASSES; ++h) {
            const int tj = row + h * ROWS;
            int i, c = start(chunk, tj, i);
            const double* const from = chunks + (chunk % 3) * SGS_CHUNK + tj * SGS_P + ts;
            const unsigned lines = tj < U.nj ? unsigned(U.nk) : 0u;
            double v[SGS_UK];
#pragma unroll
            for (int tk = 0; tk < SGS_UK; ++tk) v[tk] = from[tk * SGS_UJ * SGS_P];
#pragma unroll
            for (int tk = 0; tk < SGS_UK; ++tk)
                st_cg_if(unsigned(tk) < lines && unsigned(i - tk) < unsigned(n0) && c + tk * hop != 0, z + (c + tk * hop), v[tk]);
        }
    };
    const int nchunks = (steps + SGS_C - 1) / SGS_C;
    load(0);
    cp_async_wait_all();
    if (!REV && x == 0 && U.jb == 0 && U.kb == 0) chunks[0] = 0.0;  // the gauge row
    __syncthreads();
    for (int ch = 0; ch < nchunks; ++ch) {
        if (ch + 1 < nchunks) load(ch + 1);
        if (ch > 0) store(ch - 1);
        cp_async_wait_all();
        __syncthreads();
    }
    store(nchunks - 1);
}

// The lines of a unit.
template <bool REV>
__device__ __forceinline__ void sgs_lines(const GridDev& g, const SgsUnit& U, int steps, double* chunks,
                                          double* vals) {
    const int tid = threadIdx.x, n0 = g.n[0];
    const int j = tid % SGS_UJ, k = tid / SGS_UJ;
    const bool line = j < U.nj && k < U.nk;
    // the divisors at the line's first cell, inside it and at its last cell
    double D0 = 1.0, y0 = 1.0, D1 = 1.0, y1 = 1.0, Dm = 1.0, ym = 1.0;
    if (line) {
        const int jg = U.j0 + (REV ? U.nj - 1 - j : j), kg = U.k0 + (REV ? U.nk - 1 - k : k);
        const int first = diag_mask(g, REV ? n0 - 1 : 0, jg, kg), end = diag_mask(g, REV ? 0 : n0 - 1, jg, kg);
        D0 = g.diag[first];
        y0 = g.rdiag[first];
        D1 = g.diag[end];
        y1 = g.rdiag[end];
        Dm = g.diag[first | 3];
        ym = g.rdiag[first | 3];
    }
    // div_diag_fast_ok on the sum's bits without its sign; no range where a
    // divisor has no reciprocal (a zero sum is a zero either way)
    const unsigned range = y0 != 0.0 && y1 != 0.0 && ym != 0.0 ? 901u << 21 : 0u;
    const double w0 = g.weight[0], w1 = g.weight[1], w2 = g.weight[2];
    double* const mine = vals + (k + 1) * SGS_VP + j + 1;
    double last = -0.0;
    const int back = j + k;
    // the steps with work for a warp, and the groups of 4 whose cells are all inside
    const int low = __shfl_sync(0xffffffffu, back, 0), high = __shfl_sync(0xffffffffu, back, 31);
    const int active = __any_sync(0xffffffffu, line) ? n0 + high - low : 0;
    const int inside = active ? max(0, n0 - 5 - (high - low)) : 0;
    auto step = [&](int s, int t, double* cell, bool edge) {
        const double* const prev = mine + ((s + 1) & 1) * SGS_VALS;
        const double in = *cell, zy = prev[-1], zz = prev[-SGS_VP];
        const int i = t - back;
        const bool on = line && (!edge || unsigned(i) < unsigned(n0));
        double D = Dm, y = ym;
        if (edge) {
            D = i == 0 ? D0 : (i == n0 - 1 ? D1 : Dm);
            y = i == 0 ? y0 : (i == n0 - 1 ? y1 : ym);
        }
        // (r + x + y + z) / D, in reverse y + (0 + x + y + z) / D
        const double sum = (((REV ? 0.0 : in) + w0 * last) + w1 * zy) + w2 * zz;
        double v = div_diag_fast(sum, D, y);
        const unsigned top = unsigned(__double2hiint(sum)) << 1;
        const bool fast = top - (573u << 21) < range || (top | unsigned(__double2loint(sum))) == 0u;
        if (on && !fast) v = sgs_divide(sum, D);
        if (REV) v = in + v;
        mine[(s & 1) * SGS_VALS] = v;
        *cell = v;
        if (on) last = v;
    };
    __syncthreads();
    for (int t0 = 0; t0 < steps; t0 += SGS_C) {
        double* const cur = chunks + ((t0 / SGS_C) % 3) * SGS_CHUNK + tid * SGS_P;
        const int se = min(SGS_C, steps - t0);
        for (int s0 = 0; s0 < se; s0 += 4) {
            if (unsigned(t0 + s0 - high - 1) < unsigned(inside)) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    step(e, 0, cur + s0 + e, false);
                    if (e < 3) sgs_step_barrier();
                }
            } else {
                for (int s = s0; s < s0 + 4 && s < se; ++s) {
                    if (unsigned(t0 + s - low) < unsigned(active)) step(s, t0 + s, cur + s, true);
                    if (s < s0 + 3 && s + 1 < se) sgs_step_barrier();
                }
            }
            if (s0 + 4 < se) sgs_step_barrier();
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(SGS_THREADS, 2) k_sgs_flow(const __grid_constant__ GridDev g, SolveState* st,
                                                             const double* __restrict__ r, double* z, double* d0,
                                                             double* d1, SgsFlow f, int mode) {
    extern __shared__ __align__(16) double sgs_smem[];
    double* const chunks = sgs_smem;
    double* const vals = sgs_smem + 3 * SGS_CHUNK;
    unsigned long long* const ring =
        reinterpret_cast<unsigned long long*>(vals + 2 * SGS_VALS);  // on a 16-byte boundary
    __shared__ int s_slot, s_fail;
    if (!gate(st->flags, mode)) return;
    unsigned long long* const words = reinterpret_cast<unsigned long long*>(st->dsel ? d0 : d1);
    const int units = f.nj * f.nk, slots = 2 * units;
    const unsigned number = f.ctl[2 + units];
    const int role = threadIdx.x < SGS_LINES ? 0 : (threadIdx.x < SGS_STEPPERS - 32 ? 1 : (threadIdx.x < SGS_STEPPERS ? 2 : 3));
    if (threadIdx.x == 0) {
        s_slot = int(atomicAdd(f.ctl, 1u));
        s_fail = 0;
    }
    __syncthreads();
    int slot = s_slot;
    while (slot < slots) {
        // the next slot is taken now, its atomic overlapping this unit
        unsigned next_slot = 0;
        if (threadIdx.x == 0) next_slot = atomicAdd(f.ctl, 1u);
        const bool reverse = slot >= units;
        const int unit = f.order[reverse ? slots - 1 - slot : slot];
        SgsUnit U;
        U.jb = unit % f.nj;
        U.kb = unit / f.nj;
        U.j0 = U.jb * SGS_UJ;
        U.k0 = U.kb * SGS_UK;
        U.nj = min(SGS_UJ, g.n[1] - U.j0);
        U.nk = min(SGS_UK, g.n[2] - U.k0);
        const int steps = g.n[0] + U.nj + U.nk - 2;
        const unsigned tag = kSgsTag | ((2u * number + (reverse ? 1u : 0u)) & 0x3ffffu);
        if (reverse) {
            if (threadIdx.x == 0) {
                unsigned n = 0;
                while (ld_acquire_u32(f.ctl + 2 + unit) == 0u) {
                    ++n;
                    const bool over = n > kSgsSpins;
                    if (over) atomicExch(f.ctl + 1, 1u);
                    if (over || ((n & 7u) == 0u && *(volatile const unsigned*)(f.ctl + 1) != 0u)) {
                        s_fail = 1;
                        break;
                    }
                    if (n > 256u) __nanosleep(64);
                }
            }
            __syncthreads();
            if (!s_fail) {
                if (role == 0) sgs_lines<true>(g, U, steps, chunks, vals);
                else if (role == 1) sgs_faces<true>(g, f, U, steps, words, tag, vals, ring, &s_fail);
                else if (role == 2) sgs_send<true>(g, f, U, steps, words, tag, vals);
                else sgs_move<true>(g, U, steps, r, z, chunks);
            }
        } else {
            if (role == 0) sgs_lines<false>(g, U, steps, chunks, vals);
            else if (role == 1) sgs_faces<false>(g, f, U, steps, words, tag, vals, ring, &s_fail);
            else if (role == 2) sgs_send<false>(g, f, U, steps, words, tag, vals);
            else sgs_move<false>(g, U, steps, r, z, chunks);
        }
        __syncthreads();
        if (s_fail) {
            if (threadIdx.x == 0) {
                atomicExch(f.ctl + 1, 1u);
                st->status = RB200_EXECUTION;
                st->flags = (st->flags | F_DONE | F_STOP) & ~F_NEED_REPLACE;
            }
            return;
        }
        if (threadIdx.x == 0) {
            if (!reverse) {
                __threadfence();
                st_release_u32(f.ctl + 2 + unit, 1u);
            }
            s_slot = int(next_slot);
        }
        __syncthreads();
        slot = s_slot;
    }
}

__global__ void __launch_bounds__(EW) k_sgs_dot(GridDev g, SolveState* st, const double* __restrict__ r,
                                                const double* __restrict__ z, int mode, Partials part,
                                                rb200_trace* trace, unsigned* sgs_ctl, int sgs_words) {
    __shared__ BlockReduce<1, 0> sm;
    // the sweep kernel before this one has ended: its queue starts over
    // and its number moves on (the word after the states)
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= sgs_words; t += gridDim.x * blockDim.x)
        sgs_ctl[t] = t < sgs_words ? 0u : sgs_ctl[t] + 1u;
    if (!gate(st->flags, mode)) return;
    Neu acc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.cells; c += gridDim.x * blockDim.x)
        if (c != 0) acc.add(r[c] * z[c]);
    dd sums[1] = {acc.as_dd()};
    double none[1];
    block_reduce<1, 0>(sm, sums, none);
    if (publish_and_check_last<1, 0>(part, blockIdx.x, gridDim.x, sums, none)) {
        fold_partials<1, 0>(part, gridDim.x, sm, sums, none);
        if (threadIdx.x == 0) decide_rz(st, trace, dd_value(sums[0]), mode);
    }
}

// ------------------------------------------------------------ red-black SGS
// Symmetric Gauss-Seidel preconditioner in red-black order on the
// gauge-eliminated system (cell 0, red, is removed): forward reds then blacks,
// backward blacks then reds. With reds first, the forward red solve and the
// backward black solve are diagonal, so M^-1 r is
//   red:    y_r = r_r/D_r                     (stored by the pass that forms r)
//   black:  z_b = (r_b + sum_nb w * y_nb) / D_b
//   red:    z_r = y_r + (sum_nb w * z_nb) / D_r
// A symmetric M, as PCG needs; new (the reference sweeps lexicographically).
__device__ __forceinline__ bool is_black(int i, int j, int k) { return ((i + j + k) & 1) != 0; }

// Work mapping of the two passes: thread t takes cell pair m = t mod half of
// row t / half (row = j + n1 k), i.e. cells 2m and 2m + 1 of the row, one of
// each colour (half = ceil(n0 / 2); 2m + 1 may be n0 on an odd row length).
struct PairMap {
    int half, pairs;
    FastDiv by_half, by_n1;
};

static PairMap pair_map(const GridDev& g) {
    PairMap p;
    p.half = (g.n[0] + 1) / 2;
    p.pairs = p.half * g.n[1] * g.n[2];
    p.by_half = make_fastdiv(unsigned(p.half));
    p.by_n1 = make_fastdiv(unsigned(g.n[1]));
    return p;
}

// Neighbour sum of cell (i, j, k), x-, x+, y-, y+, z-, z+ (one order for both colours).
__device__ __forceinline__ double rb_neighbours(const GridDev& g, const double* __restrict__ z, int c, int i, int j,
                                                int k, double init) {
    double y = init;
    if (i > 0) y += g.weight[0] * z[c - 1];
    if (i + 1 < g.n[0]) y += g.weight[0] * z[c + 1];
    if (j > 0) y += g.weight[1] * z[c - g.n[0]];
    if (j + 1 < g.n[1]) y += g.weight[1] * z[c + g.n[0]];
    const int sz = g.n[0] * g.n[1];
    if (k > 0) y += g.weight[2] * z[c - sz];
    if (k + 1 < g.n[2]) y += g.weight[2] * z[c + sz];
    return y;
}

__global__ void __launch_bounds__(EW) k_rbsgs_black(GridDev g, PairMap pm, SolveState* st,
                                                    const double* __restrict__ r, double* __restrict__ z, int mode) {
    if (!gate(st->flags, mode)) return;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < pm.pairs; t += gridDim.x * blockDim.x) {
        const int row = fast_div(t, pm.by_half);
        const int m = t - row * pm.half;
        const int k = fast_div(row, pm.by_n1);
        const int j = row - k * g.n[1];
        const int i = 2 * m + ((j + k + 1) & 1);  // the black cell of the pair
        if (i >= g.n[0]) continue;
        const int c = i + g.n[0] * row;
        const int mask = diag_mask(g, i, j, k);
        z[c] = div_diag(rb_neighbours(g, z, c, i, j, k, r[c]), g.diag[mask], g.rdiag[mask]);
    }
}

__global__ void __launch_bounds__(EW) k_rbsgs_red_dot(GridDev g, PairMap pm, SolveState* st,
                                                      const double* __restrict__ r, double* __restrict__ z, int mode,
                                                      Partials part, rb200_trace* trace) {
    __shared__ BlockReduce<1, 0> sm;
    if (!gate(st->flags, mode)) return;
    Neu acc;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < pm.pairs; t += gridDim.x * blockDim.x) {
        const int row = fast_div(t, pm.by_half);
        const int m = t - row * pm.half;
        const int k = fast_div(row, pm.by_n1);
        const int j = row - k * g.n[1];
        const int ired = 2 * m + ((j + k) & 1), iblk = 2 * m + ((j + k + 1) & 1);
        const int cred = ired + g.n[0] * row, cblk = iblk + g.n[0] * row;
        if (ired < g.n[0] && cred != 0) {  // z[0] = 0 is kept by k_load_residual
            const int mask = diag_mask(g, ired, j, k);
            const double corr = rb_neighbours(g, z, cred, ired, j, k, 0.0);
            const double zc = z[cred] + div_diag(corr, g.diag[mask], g.rdiag[mask]);
            z[cred] = zc;
            acc.add(r[cred] * zc);
        }
        if (iblk < g.n[0] && cblk != 0) acc.add(r[cblk] * z[cblk]);
    }
    dd sums[1] = {acc.as_dd()};
    double none[1];
    block_reduce<1, 0>(sm, sums, none);
    if (publish_and_check_last<1, 0>(part, blockIdx.x, gridDim.x, sums, none)) {
        fold_partials<1, 0>(part, gridDim.x, sm, sums, none);
        if (threadIdx.x == 0) decide_rz(st, trace, dd_value(sums[0]), mode);
    }
}

// ------------------------------------------------------------ graph embedding
// Device-side reset of the solver state (what solve() uploads from the host).
// The seeded start of the resident carrier: p = the accepted previous
// pressure when `warm` is set.
__global__ void __launch_bounds__(EW) k_seed_pressure(int n, double* __restrict__ p, const double* __restrict__ seed,
                                                      const int* __restrict__ warm) {
    if (!*warm) return;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) p[c] = seed[c];
}

__global__ void k_solve_reset(SolveState* st, rb200_settings s, const double* __restrict__ dt_dev,
                              const int* __restrict__ skip, int flexible, const int* __restrict__ warm) {
    SolveState init{};
    init.dt = *dt_dev;
    init.relative = s.relative_residual;
    init.absolute = s.absolute_residual;
    init.divergence_limit = s.divergence_limit;
    init.max_it = s.max_iterations > 0x7fffffffull ? 0x7fffffff : int(s.max_iterations);
    init.status = ST_RUNNING;
    init.flexible = flexible;
    if (warm && *warm != 0) init.flags = F_WARM;
    if (skip && *skip != 0) init.flags = F_DONE | F_STOP;
    *st = init;
}

// Condition of the restart branch of a loop trip (an IF node): the true
// residual asked for a restart.
__global__ void k_replace_cond(const SolveState* st, cudaGraphConditionalHandle handle) {
    cudaGraphSetConditional(handle, (st->flags & F_NEED_REPLACE) ? 1u : 0u);
}

// Condition of the WHILE node: repeat while the solve is running. The trip
// count is bounded; running out of trips ends the solve with an execution
// error instead of looping on.
__global__ void k_loop_cond(SolveState* st, cudaGraphConditionalHandle handle, int max_trips) {
    const int trips = st->trips + 1;
    st->trips = trips;
    unsigned go = (st->flags & F_DONE) ? 0u : 1u;
    if (go && trips >= max_trips) {
        st->status = RB200_EXECUTION;
        st->flags = st->flags | F_DONE | F_STOP;
        go = 0u;
    }
    cudaGraphSetConditional(handle, go);
}

// ------------------------------------------------------------ host side
constexpr int ZC = 8;
constexpr size_t kSmemPass1 = 2 * size_t(Slab<ZC>::SIZE) * sizeof(double);
constexpr size_t kSmemSlab = size_t(Slab<ZC>::SIZE) * sizeof(double);

static dim3 slab_grid(const GridDev& g) {
    return dim3((g.n[0] + TX - 1) / TX, (g.n[1] + TY - 1) / TY, (g.n[2] + ZC - 1) / ZC);
}
int slab_blocks(const GridDev& g) {
    dim3 d = slab_grid(g);
    return int(d.x * d.y * d.z);
}

static int ew_blocks(int n) {
    int b = (n + EW - 1) / EW;
    return b < 1 ? 1 : (b < EW_CAP ? b : EW_CAP);
}

// Dynamic shared memory above 48 KB must be opted into per kernel.
static int set_smem_attrs() {
    RB200_CUDA(cudaFuncSetAttribute(k_pass1<ZC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemPass1)));
    RB200_CUDA(cudaFuncSetAttribute(k_pass2<ZC, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemSlab)));
    RB200_CUDA(cudaFuncSetAttribute(k_pass2<ZC, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemSlab)));
    RB200_CUDA(cudaFuncSetAttribute(k_pass2<ZC, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemSlab)));
    RB200_CUDA(cudaFuncSetAttribute(k_true_residual<ZC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    int(kSmemSlab)));
    return RB200_OK;
}

struct Bufs {
    double *b, *p, *r, *z, *d0, *d1, *r1;  // r1: the multigrid method's second residual buffer
    SolveState* st;
    Partials part;
    rb200_trace* trace;
    TmaMaps maps;
    SgsFlow sgs{};
    const DirectSolver* direct = nullptr;  // the mixed method by fast diagonalisation (d0: the second p buffer)
};

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against libcuda). The encoder validates base, strides and box on the host.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    });
    return fn;
}

// TMA slabs need a row pitch that is a multiple of 16 bytes (nx even) and, to
// stay well inside the encoder's documented limits, a grid at least one box
// large in every direction. Other grids take the cp.async path.
static bool tma_eligible(const GridDev& g) {
    return (g.n[0] % 2) == 0 && g.n[0] >= Slab<ZC>::SX && g.n[1] >= Slab<ZC>::SY && g.n[2] >= Slab<ZC>::SZ;
}

static bool encode_map(CUtensorMap* m, const double* base, const GridDev& g, const cuuint32_t box[3]) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    cuuint64_t dims[3] = {cuuint64_t(g.n[0]), cuuint64_t(g.n[1]), cuuint64_t(g.n[2])};
    cuuint64_t strides[2] = {cuuint64_t(g.n[0]) * 8, cuuint64_t(g.n[0]) * cuuint64_t(g.n[1]) * 8};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(base), dims, strides,
                     const_cast<cuuint32_t*>(box), estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

static bool encode_slab_map(CUtensorMap* m, const double* base, const GridDev& g) {
    const cuuint32_t box[3] = {cuuint32_t(Slab<ZC>::SX), cuuint32_t(Slab<ZC>::SY), cuuint32_t(Slab<ZC>::SZ)};
    return encode_map(m, base, g, box);
}

static bool encode_box_map(CUtensorMap* m, const double* base, const GridDev& g) {
    const cuuint32_t box[3] = {cuuint32_t(TX), cuuint32_t(TY), cuuint32_t(ZC)};
    return encode_map(m, base, g, box);
}

// The maps of a solver's vectors. The encoder takes a null address, and a load
// through such a map reads address 0: a solver without z or a second direction
// (the direct method) has no maps, and without r (its timing run) no map of r,
// which the direction pass does not read.
static TmaMaps make_maps(const GridDev& g, const double* z, const double* d0, const double* d1, const double* p,
                         const double* r) {
    TmaMaps m;
    std::memset(&m, 0, sizeof(m));
    if (z && d0 && d1 && p && tma_eligible(g) && encode_slab_map(&m.z, z, g) && encode_slab_map(&m.d0, d0, g) &&
        encode_slab_map(&m.d1, d1, g) && encode_slab_map(&m.p, p, g) && encode_box_map(&m.p_box, p, g) &&
        (!r || encode_box_map(&m.r_box, r, g)))
        m.use = 1;
    else
        std::memset(&m, 0, sizeof(m));
    return m;
}

// One lexicographic SGS application: both sweeps in one launch, then r.z.
static int launch_sgs(const GridDev& g, const Bufs& B, int mode, cudaStream_t s) {
    k_sgs_flow<<<B.sgs.blocks, SGS_THREADS, kSmemSgs, s>>>(g, B.st, B.r, B.z, B.d0, B.d1, B.sgs, mode);
    k_sgs_dot<<<ew_blocks(g.cells), EW, 0, s>>>(g, B.st, B.r, B.z, mode, B.part, B.trace, B.sgs.ctl,
                                                B.sgs.nj * B.sgs.nk + 2);
    return 2;
}

// Initial residual and preconditioned start (src/pressure.rs:603-650).
// `mg` is the multigrid hierarchy of the mixed method (nullptr otherwise).
static int launch_start(const GridDev& g, int method, const Bufs& B, const Multigrid* mg, cudaStream_t s) {
    const int eb = ew_blocks(g.cells);
    k_init_sums<<<eb, EW, 0, s>>>(g, B.st, B.b, B.p, B.part);
    if (B.direct) return 1;  // a seeded solve adds the seed's residual
    if (method == RB200_JACOBI_PCG_V1) {
        k_load_residual<KIND_JACOBI><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_INIT, B.part,
                                                       B.trace);
        return 2;
    }
    if (method == RB200_RBSGS_PCG) {
        k_load_residual<KIND_RBSGS><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_INIT, B.part,
                                                      B.trace);
        const PairMap pm = pair_map(g);
        const int pb = ew_blocks(pm.pairs);
        k_rbsgs_black<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_INIT);
        k_rbsgs_red_dot<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_INIT, B.part, B.trace);
        return 4;
    }
    k_load_residual<KIND_MG><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_INIT, B.part, B.trace);
    if (method == RB200_SGS_PCG_V1) return 2 + launch_sgs(g, B, MODE_INIT, s);
    int n = 2 + mg->enqueue(B.r, B.st, MODE_INIT, s);
    return n + mg->enqueue_finish(B.st, B.r, B.r1, MODE_INIT, B.part, B.trace, s);
}

// One PCG iteration (src/pressure.rs:651-734).
static int launch_iteration(const GridDev& g, int method, const Bufs& B, const Multigrid* mg, cudaStream_t s) {
    if (B.direct) return B.direct->enqueue_iteration(g, B.st, B.b, B.p, B.d0, B.part, B.trace, s);
    const dim3 grid = slab_grid(g), block(TX, TY, 1);
    const int eb = ew_blocks(g.cells);
    const bool flexible = method == RB200_MG_MIXED;
    if (flexible)
        mg->enqueue_pass1(g, B.st, B.d0, B.d1, B.part, B.trace, s);
    else
        k_pass1<ZC><<<grid, block, kSmemPass1, s>>>(g, B.st, B.z, B.d0, B.d1, nullptr, B.maps, B.part, B.trace);
    if (method == RB200_JACOBI_PCG_V1) {
        k_pass2<ZC, 0><<<grid, block, kSmemSlab, s>>>(g, B.st, B.p, B.r, B.z, B.d0, B.d1, B.maps, B.part,
                                                         B.trace);
        return 2;
    }
    if (method == RB200_RBSGS_PCG) {
        k_pass2<ZC, 1><<<grid, block, kSmemSlab, s>>>(g, B.st, B.p, B.r, B.z, B.d0, B.d1, B.maps, B.part,
                                                          B.trace);
        const PairMap pm = pair_map(g);
        const int pb = ew_blocks(pm.pairs);
        k_rbsgs_black<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_ITER);
        k_rbsgs_red_dot<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_ITER, B.part, B.trace);
        return 4;
    }
    if (method == RB200_SGS_PCG_V1) {
        k_pass2<ZC, 2><<<grid, block, kSmemSlab, s>>>(g, B.st, B.p, B.r, B.z, B.d0, B.d1, B.maps, B.part,
                                                          B.trace);
        return 2 + launch_sgs(g, B, MODE_ITER, s);
    }
    int n = 2;
    if (mg->fuses_update()) {
        mg->enqueue_update_first(g, B.st, B.p, B.r, B.r1, B.d0, B.d1, B.part, B.trace, s);
        n += mg->enqueue(B.r, B.st, MODE_ITER, s, true);
    } else {
        k_mg_update<<<eb, EW, 0, s>>>(g, B.st, B.p, B.r, B.r1, B.d0, B.d1, B.part, B.trace);
        n += mg->enqueue(B.r, B.st, MODE_ITER, s);
    }
    return n + mg->enqueue_finish(B.st, B.r, B.r1, MODE_ITER, B.part, B.trace, s);
}

// The gated true-residual check and restart (src/pressure.rs:686-715).
static int launch_check(const GridDev& g, int method, const Bufs& B, const Multigrid* mg, cudaStream_t s) {
    if (B.direct) return B.direct->enqueue_settle(g, B.st, B.p, B.d0, s);  // every iteration ends in the check
    const dim3 grid = slab_grid(g), block(TX, TY, 1);
    const int eb = ew_blocks(g.cells);
    k_true_residual<ZC><<<grid, block, kSmemSlab, s>>>(g, B.st, B.b, B.p, B.d0, B.d1, B.maps, B.part, B.trace);
    if (method == RB200_JACOBI_PCG_V1) {
        k_load_residual<KIND_JACOBI><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_REPLACE, B.part,
                                                       B.trace);
        return 2;
    }
    if (method == RB200_RBSGS_PCG) {
        k_load_residual<KIND_RBSGS><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_REPLACE, B.part,
                                                      B.trace);
        const PairMap pm = pair_map(g);
        const int pb = ew_blocks(pm.pairs);
        k_rbsgs_black<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_REPLACE);
        k_rbsgs_red_dot<<<pb, EW, 0, s>>>(g, pm, B.st, B.r, B.z, MODE_REPLACE, B.part, B.trace);
        return 4;
    }
    k_load_residual<KIND_MG><<<eb, EW, 0, s>>>(g, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_REPLACE, B.part, B.trace);
    if (method == RB200_SGS_PCG_V1) return 2 + launch_sgs(g, B, MODE_REPLACE, s);
    int n = 2 + mg->enqueue(B.r, B.st, MODE_REPLACE, s);
    return n + mg->enqueue_finish(B.st, B.r, B.r1, MODE_REPLACE, B.part, B.trace, s);
}

static SolveState initial_state(double dt, const rb200_settings& s) {
    SolveState init{};
    init.dt = dt;
    init.relative = s.relative_residual;
    init.absolute = s.absolute_residual;
    init.divergence_limit = s.divergence_limit;
    init.max_it = s.max_iterations > 0x7fffffffull ? 0x7fffffff : int(s.max_iterations);
    init.status = ST_RUNNING;
    return init;
}

static void fill_report(const SolveState& f, rb200_report* report) {
    if (!report) return;
    std::memset(report, 0, sizeof(*report));
    report->iterations = uint64_t(f.it);
    report->true_residual_l2 = f.true_l2;
    report->true_residual_max = f.true_max;
    report->predicted_divergence_max = f.true_div;
    report->incompatible_sum = f.incompatible_sum;
    report->incompatible_budget = f.incompatible_budget;
    report->breakdown_iteration = uint64_t(f.breakdown_it);
}

PcgSolver::~PcgSolver() {
    if (chunk_exec_) cudaGraphExecDestroy(chunk_exec_);
    if (beside_chunk_exec_) cudaGraphExecDestroy(beside_chunk_exec_);
    for (auto& e : ev_)
        if (e) cudaEventDestroy(e);
    cudaFree(b_);
    cudaFree(p_);
    cudaFree(r_);
    cudaFree(d_[0]);
    cudaFree(d_[1]);
    cudaFree(z_);
    cudaFree(r1_);
    cudaFree(part_.data);
    cudaFree(part_.ticket);
    cudaFree(st_);
    cudaFree(d_trace_);
    cudaFree(gbar_);
    cudaFree(ppart_);
    cudaFree(rwords_);
    cudaFree(const_cast<int*>(sgs_.order));
    cudaFree(sgs_.ctl);
    if (h_st_) cudaFreeHost(h_st_);
}

// Whether a cooperative launch of the solver's kernel can sit in a CUDA graph,
// inside the body of a WHILE conditional node (the resident carrier's form).
// Checked once per process for the resident kernel and once for the streaming
// ones, by capturing and instantiating such a graph (nothing is launched).
static bool persistent_graphs_supported(PcgSolver& solver, bool resident) {
    static std::once_flag onces[2];
    static bool answers[2] = {false, false};
    bool& supported = answers[resident];
    std::call_once(onces[resident], [&] {
        cudaStream_t outer = nullptr, body_stream = nullptr;
        if (cudaStreamCreateWithFlags(&outer, cudaStreamNonBlocking) != cudaSuccess) return;
        if (cudaStreamCreateWithFlags(&body_stream, cudaStreamNonBlocking) != cudaSuccess) {
            cudaStreamDestroy(outer);
            return;
        }
        bool ok = cudaStreamBeginCapture(outer, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
        cudaGraph_t graph = nullptr;
        if (ok) {
            cudaStreamCaptureStatus status;
            const cudaGraphNode_t* deps = nullptr;
            size_t ndeps = 0;
            cudaGraph_t g = nullptr;
            ok = cudaStreamGetCaptureInfo(outer, &status, nullptr, &g, &deps, &ndeps) == cudaSuccess;
            cudaGraphConditionalHandle handle;
            ok = ok && cudaGraphConditionalHandleCreate(&handle, g, 0, cudaGraphCondAssignDefault) == cudaSuccess;
            cudaGraphNodeParams cp{};
            cp.type = cudaGraphNodeTypeConditional;
            cp.conditional.handle = handle;
            cp.conditional.type = cudaGraphCondTypeWhile;
            cp.conditional.size = 1;
            cudaGraphNode_t node;
            ok = ok && cudaGraphAddNode(&node, g, deps, ndeps, &cp) == cudaSuccess;
            if (ok) {
                cudaGraph_t body = cp.conditional.phGraph_out[0];
                ok = cudaStreamBeginCaptureToGraph(body_stream, body, nullptr, nullptr, 0,
                                                   cudaStreamCaptureModeRelaxed) == cudaSuccess;
                if (ok) {
                    cudaError_t le = solver.launch_persistent_chunk(body_stream, 1);
                    cudaGraph_t captured = nullptr;
                    cudaError_t ee = cudaStreamEndCapture(body_stream, &captured);
                    ok = le == cudaSuccess && ee == cudaSuccess;
                }
                ok = ok && cudaStreamUpdateCaptureDependencies(outer, &node, 1, cudaStreamSetCaptureDependencies) ==
                               cudaSuccess;
            }
        }
        cudaError_t end = cudaStreamEndCapture(outer, &graph);
        ok = ok && end == cudaSuccess;
        if (ok) {
            cudaGraphExec_t exec = nullptr;
            ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
            if (exec) cudaGraphExecDestroy(exec);
        }
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        cudaStreamDestroy(body_stream);
        cudaStreamDestroy(outer);
        supported = ok;
    });
    return supported;
}

// The lexicographic SGS queue: unit ids in wave order, the zeroed state
// words, and the sweep kernel's resident block count.
int PcgSolver::sgs_setup() {
    sgs_.nj = (g_.n[1] + SGS_UJ - 1) / SGS_UJ;
    sgs_.nk = (g_.n[2] + SGS_UK - 1) / SGS_UK;
    std::vector<int> order;
    order.reserve(size_t(sgs_.nj) * sgs_.nk);
    for (int w = 0; w <= sgs_.nj + sgs_.nk - 2; ++w)
        for (int kb = std::max(0, w - sgs_.nj + 1); kb <= std::min(w, sgs_.nk - 1); ++kb)
            order.push_back(w - kb + sgs_.nj * kb);
    const size_t units = order.size(), words = units + 3;
    int* d_order = nullptr;
    RB200_CUDA(cudaMalloc(&d_order, units * sizeof(int)));
    sgs_.order = d_order;
    RB200_CUDA(cudaMalloc(&sgs_.ctl, words * sizeof(unsigned)));
    bytes_ += units * sizeof(int) + words * sizeof(unsigned);
    RB200_CUDA(cudaMemcpyAsync(d_order, order.data(), units * sizeof(int), cudaMemcpyHostToDevice, stream_));
    RB200_CUDA(cudaMemsetAsync(sgs_.ctl, 0, words * sizeof(unsigned), stream_));
    for (double* d : d_) RB200_CUDA(cudaMemsetAsync(d, 0, size_t(g_.cells) * sizeof(double), stream_));
    RB200_CUDA(cudaStreamSynchronize(stream_));
    int dev = 0, sms = 0, per_sm = 0;
    RB200_CUDA(cudaGetDevice(&dev));
    RB200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    RB200_CUDA(cudaFuncSetAttribute(k_sgs_flow, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemSgs)));
    RB200_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sgs_flow, SGS_THREADS, kSmemSgs));
    sgs_.blocks = int(std::min<long long>(2ll * (long long)units, std::max(1ll, (long long)sms * per_sm)));
    return RB200_OK;
}

int PcgSolver::init(const GridDev& g, int method, cudaStream_t stream) {
    g_ = g;
    method_ = method;
    stream_ = stream;
    RB200_CUDA(cudaGetDevice(&device_));
    if (method < RB200_JACOBI_PCG_V1 || method > RB200_MG_MIXED) return RB200_UNSUPPORTED;
    int rc = set_smem_attrs();
    if (rc) return rc;
    part_blocks_ = std::max(slab_blocks(g), EW_CAP);
    const size_t n = size_t(g.cells);
    auto alloc = [&](double** ptr, size_t count) -> int {
        cudaError_t e = cudaMalloc(ptr, count * sizeof(double));
        if (e != cudaSuccess) {
            set_error(std::string("cudaMalloc: ") + cudaGetErrorString(e));
            return RB200_OUT_OF_MEMORY;
        }
        bytes_ += count * sizeof(double);
        return RB200_OK;
    };
    use_direct_ = method == RB200_MG_MIXED && direct_supported(g);
    if ((rc = alloc(&b_, n)) || (rc = alloc(&p_, n)) || (rc = alloc(&d_[0], n))) return rc;
    if (use_direct_) {
        if ((rc = direct_.init(g, stream_))) return rc;
        bytes_ += direct_.bytes();
    } else if ((rc = alloc(&r_, n)) || (rc = alloc(&z_, n)) || (rc = alloc(&d_[1], n))) {
        return rc;
    }
    if (multigrid()) {
        if ((rc = alloc(&r1_, n))) return rc;
        RB200_CUDA(cudaMemsetAsync(r1_, 0, n * sizeof(double), stream_));
        if ((rc = mg_.init(g, stream_))) return rc;
        bytes_ += mg_.bytes();
    }
    // up to 2K + M = 9 doubles per block (the init sums)
    if ((rc = alloc(&part_.data, size_t(part_blocks_) * 12))) return rc;
    RB200_CUDA(cudaMalloc(&part_.ticket, sizeof(unsigned)));
    RB200_CUDA(cudaMemsetAsync(part_.ticket, 0, sizeof(unsigned), stream_));
    RB200_CUDA(cudaMalloc(reinterpret_cast<void**>(&st_), sizeof(SolveStates)));
    RB200_CUDA(cudaMemsetAsync(st_, 0, sizeof(SolveStates), stream_));
    RB200_CUDA(cudaMallocHost(&h_st_, 2 * sizeof(SolveState)));
    for (auto& e : ev_) RB200_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    maps_ = make_maps(g, z_, d_[0], d_[1], p_, r_);
    if (method == RB200_SGS_PCG_V1 && (rc = sgs_setup())) return rc;
    // the direct method takes two iterations to 1e-8, the multigrid one six or seven
    chunk_ = use_direct_ ? 2 : method == RB200_MG_MIXED ? 4 : (g.cells >= (1 << 20) ? 32 : 16);
    // RB200_PERSISTENT=0 in the environment keeps the per-pass kernels (a
    // diagnostic switch: both paths compute the same iteration).
    const char* persist_env = std::getenv("RB200_PERSISTENT");
    const bool persist_allowed = !(persist_env && persist_env[0] == '0');
    // Jacobi-PCG keeps its direction on the chip where every brick of 32 x 16 x 32
    // cells has an SM (up to 128^3); larger grids stream their vectors through
    // the persistent kernel. us per iteration, resident / before: 32^3 5.4 / 24
    // (per-pass kernels), 64^3 7.7 / 12.9, 80x48x45 7.7 / 12.9, 96^3 13.3 / 21.4,
    // 128^3 22.6 / 34.6.
    if (method == RB200_JACOBI_PCG_V1 && persist_allowed && (rc = resident_setup(g, &resident_))) return rc;
    if (resident_.q) {
        RB200_CUDA(cudaMalloc(&gbar_, sizeof(GridBarrier)));
        const size_t words = resident_words(resident_);
        RB200_CUDA(cudaMalloc(&rwords_, words * sizeof(unsigned long long)));
        bytes_ += words * sizeof(unsigned long long);
        RB200_CUDA(reset_persistent(stream_));
        persist_blocks_ = resident_.blocks;
        if (!persistent_graphs_supported(*this, true)) {
            persist_blocks_ = 0;
            resident_.q = 0;
        } else {
            chunk_ = 64;
            // Carriers stepped together run two at a time where each takes two
            // lanes (coop.cu), so where the plan takes more there is a second
            // one, a longer run of cells a thread: slower alone (us per
            // iteration 37^3 7.7 / 8.1, 45^3 8.1 / 8.4, 63^3 8.7 / 10.1, 75^3
            // 14.4 / 23.1), faster two at a time (ms for eight carriers stepped
            // together, one at a time / two: 37^3 20.1 / 10.7, 45^3 26.3 / 13.7,
            // 63^3 39.8 / 23.2, 75^3 81 / 64, 95^3 102 / 91). Its blocks hold
            // half the SMs or fewer, or there is none (above about 96^3).
            int sms = 0;
            RB200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_));
            const int half = (sms / kCoopLanes) * (kCoopLanes / 2);
            if (resident_.blocks > half && (rc = resident_setup(g, &beside_, half))) return rc;
        }
    } else if ((method == RB200_JACOBI_PCG_V1 || method == RB200_RBSGS_PCG) && maps_.use && persist_allowed) {
        persist_pre_ = method == RB200_RBSGS_PCG ? 1 : 0;
        int blocks = 0;
        if ((rc = persistent_setup(g, &blocks))) return rc;
        if (blocks > 0) {
            RB200_CUDA(cudaMalloc(&gbar_, sizeof(GridBarrier)));
            RB200_CUDA(cudaMemsetAsync(gbar_, 0, sizeof(GridBarrier), stream_));
            if ((rc = alloc(&ppart_, persistent_partial_doubles(blocks)))) return rc;
            persist_blocks_ = blocks;
            if (!persistent_graphs_supported(*this, false)) persist_blocks_ = 0;
            else chunk_ = 64;
        }
    }
    return capture_chunk(&chunk_exec_, false);
}

cudaError_t PcgSolver::launch_persistent_chunk(cudaStream_t s, int budget, rb200_trace* trace, bool beside) {
    if (resident_.q)
        return launch_resident(beside ? beside_ : resident_, g_, st_, b_, p_, r_, z_, d_[0], d_[1], rwords_, gbar_, trace, budget, s);
    return launch_persistent(g_, st_, b_, p_, r_, z_, d_[0], d_[1], ppart_, gbar_, trace, maps_, persist_blocks_,
                             budget, s, persist_pre_);
}

cudaError_t PcgSolver::reset_persistent(cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(gbar_, 0, sizeof(GridBarrier), s);
    if (e == cudaSuccess && rwords_)
        e = cudaMemsetAsync(rwords_, 0, resident_words(resident_) * sizeof(unsigned long long), s);
    return e;
}

int PcgSolver::set_trace(rb200_trace* host, size_t capacity) {
    if (d_trace_) {
        cudaFree(d_trace_);
        d_trace_ = nullptr;
    }
    h_trace_ = host;
    trace_cap_ = host ? capacity : 0;
    if (trace_cap_) RB200_CUDA(cudaMalloc(&d_trace_, trace_cap_ * sizeof(rb200_trace)));
    for (cudaGraphExec_t* exec : {&chunk_exec_, &beside_chunk_exec_})
        if (*exec) {
            cudaGraphExecDestroy(*exec);
            *exec = nullptr;
        }
    return capture_chunk(&chunk_exec_, false);
}

// One chunk: `chunk_` iterations, then the gated true-residual and restart.
int PcgSolver::capture_chunk(cudaGraphExec_t* exec, bool beside) {
    const Bufs B{b_, p_, r_, z_, d_[0], d_[1], r1_, st_, part_, d_trace_, maps_, sgs_, direct()};
    const Multigrid* mg = multigrid();
    cudaGraph_t graph = nullptr;
    RB200_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    int nodes = 0;
    cudaError_t launch_err = cudaSuccess;
    if (persist_blocks_) {
        launch_err = launch_persistent_chunk(stream_, chunk_, d_trace_, beside);
        nodes = 1;
    } else {
        for (int q = 0; q < chunk_; ++q) nodes += launch_iteration(g_, method_, B, mg, stream_);
        nodes += launch_check(g_, method_, B, mg, stream_);
    }
    nodes_per_chunk_ = nodes;
    if (launch_err == cudaSuccess) launch_err = cudaGetLastError();
    cudaError_t end_err = cudaStreamEndCapture(stream_, &graph);
    if (launch_err != cudaSuccess || end_err != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        set_error(std::string("chunk capture: ") +
                  cudaGetErrorString(launch_err != cudaSuccess ? launch_err : end_err));
        return RB200_EXECUTION;
    }
    cudaError_t e = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        set_error(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
        return RB200_EXECUTION;
    }
    return RB200_OK;
}

int PcgSolver::launch_chunk(int slot) {
    // a chunk that is a cooperative kernel takes its lanes, as a carrier's step does
    CoopTurn turn;
    int rc = turn.begin(stream_, persistent_blocks(beside_now_), user_);
    if (rc) return rc;
    RB200_CUDA(cudaGraphLaunch(beside_now_ ? beside_chunk_exec_ : chunk_exec_, stream_));
    if ((rc = turn.end())) return rc;
    launches_ += uint64_t(nodes_per_chunk_);
    return record_flags(slot);
}

int PcgSolver::record_flags(int slot) {
    RB200_CUDA(cudaMemcpyAsync(&h_st_[slot], st_, sizeof(SolveState), cudaMemcpyDeviceToHost, stream_));
    RB200_CUDA(cudaEventRecord(ev_[slot], stream_));
    return RB200_OK;
}

int PcgSolver::solve(double dt, const rb200_settings& s, rb200_report* report, rb200_cancel_fn cancelled,
                     void* ctx, const double* initial) {
    if (report) std::memset(report, 0, sizeof(*report));
    SolveState init = initial_state(dt, s);
    init.flexible = method_ == RB200_MG_MIXED ? 1 : 0;
    if (initial) {
        RB200_CUDA(cudaMemcpyAsync(p_, initial, size_t(g_.cells) * sizeof(double), cudaMemcpyDefault, stream_));
        init.flags |= F_WARM;
    }
    if (d_trace_ && uint64_t(init.max_it) > trace_cap_) {
        set_error("trace capacity is smaller than max_iterations");
        return RB200_INVALID_ARGUMENT;
    }
    h_st_[0] = init;
    RB200_CUDA(cudaMemcpyAsync(st_, &h_st_[0], sizeof(SolveState), cudaMemcpyHostToDevice, stream_));
    if (d_trace_) RB200_CUDA(cudaMemsetAsync(d_trace_, 0, trace_cap_ * sizeof(rb200_trace), stream_));
    RB200_CUDA(cudaMemsetAsync(part_.ticket, 0, sizeof(unsigned), stream_));
    if (persist_blocks_) RB200_CUDA(reset_persistent(stream_));
    // in flight until this function returns
    struct Active {
        std::atomic<int>* n;
        explicit Active(std::atomic<int>* count) : n(count) {
            if (n) ++*n;
        }
        ~Active() {
            if (n) --*n;
        }
    } active(persist_blocks_ ? &coop_active(device_) : nullptr);
    launches_ += uint64_t(launch_start(g_, method_, Bufs{b_, p_, r_, z_, d_[0], d_[1], r1_, st_, part_, d_trace_, maps_, sgs_, direct()},
                                       multigrid(), stream_));
    if (use_direct_ && initial) launches_ += uint64_t(direct_.enqueue_seed(g_, st_, b_, p_, d_[0], part_, stream_));
    RB200_CUDA(cudaGetLastError());
    // The host copy of the state must be stable before the chunk copies reuse
    // h_st_ slots.
    RB200_CUDA(cudaStreamSynchronize(stream_));
    int rc;
    if ((rc = record_flags(0))) return rc;
    // A chunk ahead of the flags keeps the device busy through long solves. The
    // direct method's usual solve is one chunk, so it launches none ahead. Nor
    // does a cooperative solve beside others, which keep the device busy: the
    // last chunk would wait for their turns to do nothing.
    const bool others = persist_blocks_ && coop_active(device_) > 1;
    const bool ahead = !use_direct_ && !others;
    // Beside others the solve takes half of the lanes where it can, from its first
    // chunk to its last: a launch leaves z on the surfaces of its bricks only.
    beside_now_ = others && has_beside();
    if (beside_now_ && !beside_chunk_exec_ && capture_chunk(&beside_chunk_exec_, true)) beside_now_ = false;
    if (ahead && (rc = launch_chunk(1))) return rc;
    int slot = 0, last_it = -1, stalls = 0;
    bool cancelled_now = false;
    for (;;) {
        RB200_CUDA(cudaEventSynchronize(ev_[slot]));
        const SolveState& h = h_st_[slot];
        if (h.flags & F_DONE) break;
        if (cancelled && cancelled(ctx)) {
            cancelled_now = true;
            break;
        }
        if (h.it == last_it) {
            if (++stalls > 4) {
                RB200_CUDA(cudaStreamSynchronize(stream_));
                set_error("pressure solve made no progress");
                return RB200_EXECUTION;
            }
        } else {
            stalls = 0;
            last_it = h.it;
        }
        if ((rc = launch_chunk(slot))) return rc;
        if (ahead) slot ^= 1;
    }
    RB200_CUDA(cudaStreamSynchronize(stream_));
    RB200_CUDA(cudaMemcpy(&h_st_[0], st_, sizeof(SolveState), cudaMemcpyDeviceToHost));
    const SolveState& f = h_st_[0];
    if (d_trace_ && h_trace_) {
        size_t n = std::min(trace_cap_, size_t(f.it));
        RB200_CUDA(cudaMemcpy(h_trace_, d_trace_, n * sizeof(rb200_trace), cudaMemcpyDeviceToHost));
    }
    fill_report(f, report);
    if (cancelled_now) return RB200_CANCELLED;
    return f.status;
}

int PcgSolver::enqueue_reset(const double* dt_dev, const int* skip, const rb200_settings& settings, cudaStream_t s,
                             const int* warm, const double* seed) {
    if (warm && seed) {
        k_seed_pressure<<<ew_blocks(g_.cells), EW, 0, s>>>(g_.cells, p_, seed, warm);
        launches_ += 1;
    }
    k_solve_reset<<<1, 1, 0, s>>>(st_, settings, dt_dev, skip, method_ == RB200_MG_MIXED ? 1 : 0,
                                  (warm && seed) ? warm : nullptr);
    RB200_CUDA(cudaMemsetAsync(part_.ticket, 0, sizeof(unsigned), s));
    if (persist_blocks_) RB200_CUDA(reset_persistent(s));
    launches_ += 1;
    const Bufs B{b_, p_, r_, z_, d_[0], d_[1], r1_, st_, part_, d_trace_, maps_, sgs_, direct()};
    launch_start(g_, method_, B, multigrid(), s);
    if (use_direct_ && warm && seed) direct_.enqueue_seed(g_, st_, b_, p_, d_[0], part_, s);
    RB200_CUDA(cudaGetLastError());
    return RB200_OK;
}

int PcgSolver::enqueue_reset_fused(const double* dt_dev, const int* skip, const rb200_settings& settings,
                                   cudaStream_t s) {
    k_solve_reset<<<1, 1, 0, s>>>(st_, settings, dt_dev, skip, 1, nullptr);
    RB200_CUDA(cudaMemsetAsync(part_.ticket, 0, sizeof(unsigned), s));
    launches_ += 1;
    RB200_CUDA(cudaGetLastError());
    return RB200_OK;
}

int PcgSolver::enqueue_loop(cudaStream_t cs, cudaStream_t body_stream, const rb200_settings& settings, bool beside) {
    cudaStreamCaptureStatus status;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    RB200_CUDA(cudaStreamGetCaptureInfo(cs, &status, nullptr, &graph, &deps, &ndeps));
    if (status != cudaStreamCaptureStatusActive) {
        set_error("enqueue_loop needs an active stream capture");
        return RB200_EXECUTION;
    }
    cudaGraphConditionalHandle handle;
    RB200_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    RB200_CUDA(cudaGraphAddNode(&node, graph, deps, ndeps, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    // The loop body: one chunk of iterations, the gated check, the condition.
    RB200_CUDA(cudaStreamBeginCaptureToGraph(body_stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    const Bufs B{b_, p_, r_, z_, d_[0], d_[1], r1_, st_, part_, d_trace_, maps_, sgs_, direct()};
    const Multigrid* mg = multigrid();
    if (persist_blocks_) {
        RB200_CUDA(launch_persistent_chunk(body_stream, chunk_, d_trace_, beside));
    } else if (mg) {
        // The multigrid restart (a whole V-cycle) as an IF node after the
        // true-residual check: its launches run only in trips that restart.
        int nodes = 0;
        for (int q = 0; q < chunk_; ++q) nodes += launch_iteration(g_, method_, B, mg, body_stream);
        const dim3 grid = slab_grid(g_), block(TX, TY, 1);
        k_true_residual<ZC><<<grid, block, kSmemSlab, body_stream>>>(g_, B.st, B.b, B.p, B.d0, B.d1, B.maps, B.part,
                                                                      B.trace);
        cudaStreamCaptureStatus bst;
        const cudaGraphNode_t* bdeps = nullptr;
        size_t nbdeps = 0;
        cudaGraph_t bodyg = nullptr;
        RB200_CUDA(cudaStreamGetCaptureInfo(body_stream, &bst, nullptr, &bodyg, &bdeps, &nbdeps));
        cudaGraphConditionalHandle rh;
        RB200_CUDA(cudaGraphConditionalHandleCreate(&rh, bodyg, 0, cudaGraphCondAssignDefault));
        k_replace_cond<<<1, 1, 0, body_stream>>>(st_, rh);
        RB200_CUDA(cudaStreamGetCaptureInfo(body_stream, &bst, nullptr, &bodyg, &bdeps, &nbdeps));
        cudaGraphNodeParams ip{};
        ip.type = cudaGraphNodeTypeConditional;
        ip.conditional.handle = rh;
        ip.conditional.type = cudaGraphCondTypeIf;
        ip.conditional.size = 1;
        cudaGraphNode_t inode;
        RB200_CUDA(cudaGraphAddNode(&inode, bodyg, bdeps, nbdeps, &ip));
        cudaStream_t rs = nullptr;
        RB200_CUDA(cudaStreamCreateWithFlags(&rs, cudaStreamNonBlocking));
        cudaError_t ce = cudaStreamBeginCaptureToGraph(rs, ip.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                       cudaStreamCaptureModeRelaxed);
        if (ce == cudaSuccess) {
            const int eb = ew_blocks(g_.cells);
            k_load_residual<KIND_MG><<<eb, EW, 0, rs>>>(g_, B.st, B.b, B.d0, B.d1, B.r, B.z, MODE_REPLACE, B.part,
                                                        B.trace);
            mg->enqueue(B.r, B.st, MODE_REPLACE, rs);
            mg->enqueue_finish(B.st, B.r, B.r1, MODE_REPLACE, B.part, B.trace, rs);
            cudaGraph_t rbody = nullptr;
            ce = cudaStreamEndCapture(rs, &rbody);
        }
        cudaStreamDestroy(rs);
        if (ce != cudaSuccess) {
            set_error(std::string("restart branch capture: ") + cudaGetErrorString(ce));
            return RB200_EXECUTION;
        }
        RB200_CUDA(cudaStreamUpdateCaptureDependencies(body_stream, &inode, 1, cudaStreamSetCaptureDependencies));
        nodes_per_chunk_ = nodes + 2;  // the check and the branch condition (the restart runs rarely)
    } else {
        for (int q = 0; q < chunk_; ++q) launch_iteration(g_, method_, B, mg, body_stream);
        launch_check(g_, method_, B, mg, body_stream);
    }
    const uint64_t mi = settings.max_iterations;
    // Every trip of a running solve does at least one iteration (a candidate
    // stops the rest of its trip for the true-residual check), so the
    // iteration limit ends a solve before this bound does, as in the
    // reference, however often it restarts.
    const uint64_t trips = mi + 64;
    k_loop_cond<<<1, 1, 0, body_stream>>>(st_, handle, trips > (1u << 24) ? (1 << 24) : int(trips));
    cudaError_t le = cudaGetLastError();
    cudaGraph_t captured = nullptr;
    cudaError_t ee = cudaStreamEndCapture(body_stream, &captured);
    if (le != cudaSuccess || ee != cudaSuccess) {
        set_error(std::string("loop body capture: ") + cudaGetErrorString(le != cudaSuccess ? le : ee));
        return RB200_EXECUTION;
    }
    RB200_CUDA(cudaStreamUpdateCaptureDependencies(cs, &node, 1, cudaStreamSetCaptureDependencies));
    return RB200_OK;
}

int PcgSolver::profile(int which, int launches, double* avg_ms) {
    if (launches < 1 || which < 0 || which > 2) return RB200_INVALID_ARGUMENT;
    if (method_ == RB200_MG_MIXED && which == 1) return RB200_UNSUPPORTED;
    if (which == 2 && !persist_blocks_) return RB200_UNSUPPORTED;
    SolveState prof{};
    prof.rz = 1.0;
    prof.alpha = 1e-6;
    prof.beta = 0.5;
    prof.threshold = -1.0;
    prof.max_it = 0x7fffffff;
    prof.flags = F_PROFILE;
    prof.status = ST_RUNNING;
    h_st_[0] = prof;
    RB200_CUDA(cudaMemcpyAsync(st_, &h_st_[0], sizeof(SolveState), cudaMemcpyHostToDevice, stream_));
    const bool jac = method_ == RB200_JACOBI_PCG_V1;
    const dim3 grid = slab_grid(g_), block(TX, TY, 1);
    // the direct method keeps no z and no second direction: the timed pass gets
    // some for this call
    struct Lent {
        double** v = nullptr;
        ~Lent() {
            if (!v) return;
            cudaFree(*v);
            *v = nullptr;
        }
    } lent[2];
    int lends = 0;
    for (double** v : {&z_, &d_[1]})
        if (!*v) {
            if (cudaMalloc(v, size_t(g_.cells) * sizeof(double)) != cudaSuccess) {
                cudaGetLastError();
                *v = nullptr;
                return RB200_OUT_OF_MEMORY;
            }
            lent[lends++].v = v;
            RB200_CUDA(cudaMemsetAsync(*v, 0, size_t(g_.cells) * sizeof(double), stream_));
        }
    const TmaMaps maps = use_direct_ ? make_maps(g_, z_, d_[0], d_[1], p_, r_) : maps_;
    if (which == 2) {
        // one warm iteration, then `launches` iterations in one launch
        RB200_CUDA(reset_persistent(stream_));
        CoopTurn turn;
        int rc = turn.begin(stream_, persist_blocks_, user_);
        if (rc) return rc;
        RB200_CUDA(launch_persistent_chunk(stream_, 1, nullptr));
        cudaEvent_t a, b;
        RB200_CUDA(cudaEventCreate(&a));
        RB200_CUDA(cudaEventCreate(&b));
        RB200_CUDA(cudaEventRecord(a, stream_));
        RB200_CUDA(launch_persistent_chunk(stream_, launches, nullptr));
        RB200_CUDA(cudaEventRecord(b, stream_));
        if ((rc = turn.end())) return rc;
        RB200_CUDA(cudaEventSynchronize(b));
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, a, b);
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        RB200_CUDA(cudaGetLastError());
        RB200_CUDA(cudaMemcpy(&h_st_[0], st_, sizeof(SolveState), cudaMemcpyDeviceToHost));
        if (h_st_[0].status == RB200_EXECUTION) {
            set_error("persistent solver timing run failed");
            return RB200_EXECUTION;
        }
        *avg_ms = double(ms) / launches;
        return RB200_OK;
    }
    auto launch = [&]() {
        if (which == 0)
            k_pass1<ZC><<<grid, block, kSmemPass1, stream_>>>(g_, st_, z_, d_[0], d_[1], nullptr, maps, part_, nullptr);
        else if (jac)
            k_pass2<ZC, 0><<<grid, block, kSmemSlab, stream_>>>(g_, st_, p_, r_, z_, d_[0], d_[1], maps, part_,
                                                                   nullptr);
        else if (method_ == RB200_SGS_PCG_V1)
            k_pass2<ZC, 2><<<grid, block, kSmemSlab, stream_>>>(g_, st_, p_, r_, z_, d_[0], d_[1], maps, part_,
                                                                   nullptr);
        else
            k_pass2<ZC, 1><<<grid, block, kSmemSlab, stream_>>>(g_, st_, p_, r_, z_, d_[0], d_[1], maps, part_,
                                                                    nullptr);
    };
    launch();  // warm
    cudaEvent_t a, b;
    RB200_CUDA(cudaEventCreate(&a));
    RB200_CUDA(cudaEventCreate(&b));
    RB200_CUDA(cudaEventRecord(a, stream_));
    for (int q = 0; q < launches; ++q) launch();
    RB200_CUDA(cudaEventRecord(b, stream_));
    RB200_CUDA(cudaEventSynchronize(b));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    RB200_CUDA(cudaGetLastError());
    *avg_ms = double(ms) / launches;
    return RB200_OK;
}

// ProviderWorkspace's qualification of a candidate pressure
// (src/solver_provider.rs:239-270) in one pass: t = b - K p, |t|^2 and |b|^2
// (compensated), max|t|, and flags for a non-finite pressure (1) or product
// (2). out = {|t|^2, |b|^2, max|t|, flags, p[0]}.
__global__ void __launch_bounds__(EW) k_qualify_pressure(GridDev g, const double* __restrict__ b,
                                                         const double* __restrict__ p, Partials part,
                                                         double* __restrict__ out) {
    __shared__ BlockReduce<2, 2> sm;
    Neu tt, bb;
    double m[2] = {0.0, 0.0};
    const int sy = g.n[0], sz = g.n[0] * g.n[1];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < g.cells; c += gridDim.x * blockDim.x) {
        int i, j, k;
        cell_coords(g, c, i, j, k);
        Neigh v;
        v.c = p[c];
        v.xm = i > 0 ? p[c - 1] : 0.0;
        v.xp = i + 1 < g.n[0] ? p[c + 1] : 0.0;
        v.ym = j > 0 ? p[c - sy] : 0.0;
        v.yp = j + 1 < g.n[1] ? p[c + sy] : 0.0;
        v.zm = k > 0 ? p[c - sz] : 0.0;
        v.zp = k + 1 < g.n[2] ? p[c + sz] : 0.0;
        if (!isfinite(v.c)) m[1] = fmax(m[1], 1.0);
        const double q = apply_row(g, i, j, k, v);
        if (!isfinite(q)) m[1] = fmax(m[1], 2.0);
        const double bc = b[c];
        const double t = bc - q;
        tt.add(t * t);
        bb.add(bc * bc);
        m[0] = fmax(m[0], fabs(t));
    }
    dd sums[2] = {tt.as_dd(), bb.as_dd()};
    block_reduce<2, 2>(sm, sums, m);
    if (publish_and_check_last<2, 2>(part, blockIdx.x, gridDim.x, sums, m)) {
        fold_partials<2, 2>(part, gridDim.x, sm, sums, m);
        if (threadIdx.x == 0) {
            out[0] = dd_value(sums[0]);
            out[1] = dd_value(sums[1]);
            out[2] = m[0];
            out[3] = m[1];
            out[4] = p[0];
        }
    }
}

int launch_qualify_pressure(const GridDev& g, const double* b, const double* p, Partials part, double* out,
                            cudaStream_t s) {
    k_qualify_pressure<<<ew_blocks(g.cells), EW, 0, s>>>(g, b, p, part, out);
    RB200_CUDA(cudaGetLastError());
    return RB200_OK;
}

int launch_precondition_jacobi(const GridDev& g, const double* r, double* z, Partials part, double* rz_out,
                               cudaStream_t s) {
    k_precondition_jacobi<<<ew_blocks(g.cells), EW, 0, s>>>(g, r, z, part, rz_out);
    RB200_CUDA(cudaGetLastError());
    return RB200_OK;
}
int precondition_partials_blocks() { return EW_CAP; }

// ------------------------------------------------------------ allocation-free solve
// A Jacobi-PCG solve for callers that cannot allocate device memory: a host
// application whose device memory is owned by its own allocator under a fixed
// budget, so that a plug-in may not grow its footprint while it runs. Its
// scratch (residual, two direction buffers, preconditioned residual,
// reduction partials, solver state and ticket) lives in this fixed file-scope
// device array, which every GPU that loads the library holds until the process
// exits. It has no counterpart in the reference.
constexpr int kStaticMaxCells = 32768;   // 32^3 cells
constexpr int kStaticMaxBlocks = 2048;   // blocks of the widest pass of a solve
// Doubles of one block's reduction partials in the widest stage of a solve:
// k_init_sums publishes 3 double-double sums and 3 maxima (2 * 3 + 3); the
// other stages publish fewer (true residual 7, pass 2 4, pass 1 and the
// residual load 2).
constexpr int kStaticSlotDoubles = 2 * 3 + 3;
constexpr size_t kStaticStateDoubles = 64;
constexpr size_t kStaticPartialDoubles = size_t(kStaticMaxBlocks) * kStaticSlotDoubles;
constexpr size_t kStaticDoubles = 4 * size_t(kStaticMaxCells) + kStaticPartialDoubles + kStaticStateDoubles;
static __device__ __align__(256) double g_static_scratch[kStaticDoubles];

static_assert(sizeof(SolveStates) + sizeof(unsigned) <= kStaticStateDoubles * sizeof(double),
              "state does not fit the static scratch");

// Device address of g_static_scratch per device, resolved once per device
// with that device current. In host code the symbol itself is only a host-side
// stand-in, never a device address. The cached address belongs to the
// device's primary context: after cudaDeviceReset the array may be loaded at
// another address, so a process that resets a device must not call the
// allocation-free solve on it again.
static double* static_scratch_address(int device, int* rc) {
    static std::mutex mu;
    static double* addr[64] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= 64) {
        *rc = RB200_INVALID_ARGUMENT;
        return nullptr;
    }
    if (!addr[device]) {
        void* ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_static_scratch);
        if (e != cudaSuccess || !ptr) {
            set_error(std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
            *rc = RB200_EXECUTION;
            return nullptr;
        }
        addr[device] = static_cast<double*>(ptr);
    }
    *rc = RB200_OK;
    return addr[device];
}

int static_solve_jacobi(const GridDev& g, const double* rhs, double* pressure, double dt, const rb200_settings& s,
                        rb200_report* report, cudaStream_t stream) {
    if (g.cells > kStaticMaxCells) {
        set_error("grid exceeds the 32768-cell limit of the allocation-free solve");
        return RB200_UNSUPPORTED;
    }
    // every stage's partials (at most kStaticSlotDoubles per block) must fit
    // the reserved region
    if (size_t(std::max(slab_blocks(g), ew_blocks(g.cells))) * kStaticSlotDoubles > kStaticPartialDoubles) {
        set_error("grid shape needs more reduction blocks than the allocation-free solve holds");
        return RB200_UNSUPPORTED;
    }
    int device = 0;
    RB200_CUDA(cudaGetDevice(&device));
    int rc = RB200_OK;
    double* base = static_scratch_address(device, &rc);
    if (rc) return rc;
    if ((rc = set_smem_attrs())) return rc;
    Bufs B;
    B.b = const_cast<double*>(rhs);  // read only
    B.p = pressure;
    B.r = base;
    B.d0 = B.r + kStaticMaxCells;
    B.d1 = B.d0 + kStaticMaxCells;
    B.z = B.d1 + kStaticMaxCells;
    B.r1 = nullptr;
    B.part.data = B.z + kStaticMaxCells;
    double* state_slot = B.part.data + kStaticPartialDoubles;
    B.st = reinterpret_cast<SolveState*>(state_slot);
    B.part.ticket = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(state_slot) + sizeof(SolveStates));
    B.trace = nullptr;
    B.maps = make_maps(g, B.z, B.d0, B.d1, B.p, B.r);

    SolveState init = initial_state(dt, s);
    // The array keeps the previous call's contents: the ticket must start at 0.
    RB200_CUDA(cudaMemsetAsync(B.part.ticket, 0, sizeof(unsigned), stream));
    RB200_CUDA(cudaMemcpyAsync(B.st, &init, sizeof(SolveState), cudaMemcpyHostToDevice, stream));
    launch_start(g, RB200_JACOBI_PCG_V1, B, nullptr, stream);
    RB200_CUDA(cudaGetLastError());
    const int chunk = 16;
    int last_it = -1, stalls = 0;
    SolveState h{};
    for (;;) {
        RB200_CUDA(cudaMemcpyAsync(&h, B.st, sizeof(SolveState), cudaMemcpyDeviceToHost, stream));
        RB200_CUDA(cudaStreamSynchronize(stream));
        if (h.flags & F_DONE) break;
        if (h.it == last_it) {
            if (++stalls > 4) {
                set_error("pressure solve made no progress");
                return RB200_EXECUTION;
            }
        } else {
            stalls = 0;
            last_it = h.it;
        }
        for (int q = 0; q < chunk; ++q) launch_iteration(g, RB200_JACOBI_PCG_V1, B, nullptr, stream);
        launch_check(g, RB200_JACOBI_PCG_V1, B, nullptr, stream);
        RB200_CUDA(cudaGetLastError());
    }
    fill_report(h, report);
    return h.status;
}

}  // namespace rb200

extern "C" int rb200_pressure_solve_static(const rb200_grid* grid, double density, const double* rhs_device,
                                           double* pressure_device, size_t len, double dt,
                                           const rb200_settings* settings, rb200_report* report, void* stream) {
    using namespace rb200;
    if (!grid || !rhs_device || !pressure_device || !settings) return RB200_INVALID_ARGUMENT;
    GridDev g;
    int rc = make_grid_dev(grid, density, &g);
    if (rc) return rc;
    if (len != size_t(g.cells)) return RB200_LENGTH_MISMATCH;
    if (!std::isfinite(dt) || dt <= 0.0 || !settings_valid(settings)) return RB200_INVALID_ARGUMENT;
    return static_solve_jacobi(g, rhs_device, pressure_device, dt, *settings, report, (cudaStream_t)stream);
}
