// Resident Jacobi-PCG: one cooperative kernel runs a chunk of iterations of
// PressureWorkspace::solve_loaded (src/pressure.rs:577-740, jacobi-pcg-v1) on
// grids whose direction fits the chip. Same iteration, decisions and bounds on
// every wait as the streaming kernel of persist.cu; what differs is where the
// vectors live.
//
// Each block (one per SM) owns one brick of 32 x 16 x Q cells for the whole
// launch. The direction d stays in shared memory with a one-cell halo (128^3:
// 34 x 18 x 34 doubles, 166 KB), the residual r in registers (Q cells of a z run
// per thread), and z = r/D is formed where it is used. Per iteration a block
// moves its p (read and written, 16 bytes per cell), the z of its brick's
// surface, and its halo's z: about 20 bytes per cell against the streaming
// kernel's 72, all of it L2 traffic.
//
//   1  own cells d <- z + beta d; halo d <- z_halo + beta d_halo (the
//      neighbour's surface z, read after the barrier that published it)
//      q = K d, d.q                                       -> alpha
//   2  r -= alpha K d, z = r/D, r.r, r.z, surface z out   -> beta
//      p += alpha d while the other blocks' partials travel
//
// The grid reduction is a barrier and an all-to-all in one: a block publishes
// its double-double partials as 64-bit words that carry a 32-bit half of the
// value and the barrier's number, so a word that has the number is the data and
// needs no flag, no counter and no second read; every block polls all words
// with one or two per thread and folds them in the same order. Two word sets
// alternate: a block that posts barrier m + 2 has passed m + 1, so every block
// has read m.
//
// Bound by FP64 issue at 16 warps per SM (70 operations per cell and iteration
// without contraction: 9.2 us at 128^3 on the 128 SMs its bricks occupy, 22.6 us
// measured) and, on small grids, by the two reductions (about 2.3 us each of the
// 5.4 at 32^3: butterflies of dependent FP64 additions in the block and in the
// fold, 0.5 us one way between SMs).
#include <algorithm>
#include <type_traits>

#include "resident.hpp"
#include "slab.cuh"
#include "solve_state.cuh"

namespace rb200 {

namespace {

constexpr int RT = 512;                  // threads
constexpr int RW = RT / 32;              // warps
constexpr int RY = RW;                   // rows of a brick: one warp each
constexpr int RX = 34;                   // shared row: 32 cells and a halo cell on either side
constexpr int SP = RX * (RY + 2);        // shared plane
constexpr int RWORDS = 10;               // words of one block's widest partials (two sums, one maximum)
constexpr int RMAXB = 160;               // blocks of a grid at most (the fold's reach)
constexpr unsigned kSpins = 1u << 24;
// Cells of a thread's run whose residual waits in shared memory.
__host__ __device__ constexpr int resident_shared_cells(int q) { return q == 32 ? 12 : 0; }

struct ResidentArgs {
    GridDev g;
    SolveState* st;
    const double* b;
    double *p, *r, *z, *d0, *d1;
    unsigned long long* words;  // [2][blocks][RWORDS]
    GridBarrier* bar;           // count: barriers passed by earlier launches of the solve
    rb200_trace* trace;
    int budget;
    int nbx, nby;               // bricks along x and y
};

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

struct RCtx {
    int tid, lane, warp;
    unsigned seq;             // number of the last barrier
    BlockReduce<2, 1>* red;   // shared
    unsigned* halves;         // shared: the received words' value halves
};

// Row of K at one cell (apply_full, src/operator.rs:400-416): X lower, X upper,
// Y lower, Y upper, Z lower, Z upper. In the place of a neighbour outside the
// box the caller gives the cell's own value: its term is an exact zero, and the
// row needs no masks.
__device__ __forceinline__ double row_at(const GridDev& g, double cv, double xm, double xp, double ym, double yp,
                                         double zm, double zp) {
    double q = g.weight[0] * (cv - xm);
    q += g.weight[0] * (cv - xp);
    q += g.weight[1] * (cv - ym);
    q += g.weight[1] * (cv - yp);
    q += g.weight[2] * (cv - zm);
    q += g.weight[2] * (cv - zp);
    return q;
}

struct Neu2 {
    Neu a, b;
    __device__ __forceinline__ dd as_dd() const { return pair_add(dd{a.s, a.c}, dd{b.s, b.c}); }
};

// Reduces this block's K sums and M maxima, publishes them, runs `between`
// (work that needs no other block), waits for every block's partials and folds
// them, in the same order everywhere. RELEASE: the block's
// global stores so far are visible to every block afterwards. The result is
// valid in warp 0. False when a wait ran out or a block gave up.
struct Nothing {
    __device__ __forceinline__ void operator()() const {}
};
template <int K, int M, bool RELEASE, class Between = Nothing>
__device__ __forceinline__ bool reduce_all(RCtx& c, const ResidentArgs& A, dd (&sums)[K > 0 ? K : 1],
                                           double (&maxs)[M > 0 ? M : 1], Between between = Between()) {
    constexpr int W = 2 * (2 * K + M);
    constexpr int PER = RMAXB / 32;
    BlockReduce<2, 1>& red = *c.red;
    unsigned* const halves = c.halves;
    const int nb = int(gridDim.x);
#pragma unroll
    for (int q = 0; q < K; ++q) sums[q] = lanes_sum<32>(sums[q]);
#pragma unroll
    for (int q = 0; q < M; ++q) maxs[q] = warp_reduce_max(maxs[q]);
    if (c.lane == 0) {
#pragma unroll
        for (int q = 0; q < K; ++q) red.s[c.warp][q] = sums[q];
#pragma unroll
        for (int q = 0; q < M; ++q) red.m[c.warp][q] = maxs[q];
    }
    __syncthreads();
    const unsigned seq = ++c.seq;
    unsigned long long* base = A.words + size_t(seq & 1u) * nb * RWORDS;
    if (c.warp == 0) {
        if (RELEASE) __threadfence();
#pragma unroll
        for (int q = 0; q < K; ++q) sums[q] = lanes_sum<RW>(red.s[c.lane & (RW - 1)][q]);
#pragma unroll
        for (int q = 0; q < M; ++q) maxs[q] = warp_reduce_max(red.m[c.lane & (RW - 1)][q]);
        // every lane has the result: lane l posts word l
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < K; ++q) {
            if ((c.lane >> 1) == 2 * q) v = sums[q].hi;
            if ((c.lane >> 1) == 2 * q + 1) v = sums[q].lo;
        }
#pragma unroll
        for (int q = 0; q < M; ++q)
            if ((c.lane >> 1) == 2 * K + q) v = maxs[q];
        if (c.lane < W) {
            const unsigned half = (c.lane & 1) ? unsigned(__double2hiint(v)) : unsigned(__double2loint(v));
            st_word(base + size_t(blockIdx.x) * W + c.lane, ((unsigned long long)seq << 32) | half);
        }
    }
    between();
    // whole warps poll together, so that they stay converged for what follows
    bool ok = true;
    for (int t0 = c.warp * 32; t0 < nb * W; t0 += RT) {
        const int t = min(t0 + c.lane, nb * W - 1);
        unsigned n = 0;
        unsigned long long w;
        for (;;) {
            w = ld_word(base + t);
            if (__all_sync(0xffffffffu, unsigned(w >> 32) == seq)) break;
            if ((++n & 63u) == 0u &&
                __any_sync(0xffffffffu, *(volatile unsigned*)&A.bar->abort != 0u || n > kSpins)) {
                ok = false;
                break;
            }
        }
        halves[t] = unsigned(w);
    }
    if (!__syncthreads_and(ok)) return false;
    if (c.warp == 0) {
        const double* vals = reinterpret_cast<const double*>(halves);
        dd v[PER][K > 0 ? K : 1];
#pragma unroll
        for (int q = 0; q < M; ++q) maxs[q] = 0.0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int b = c.lane + 32 * u;
            const bool have = b < nb;
#pragma unroll
            for (int q = 0; q < K; ++q)
                v[u][q] = have ? dd{vals[b * (W / 2) + 2 * q], vals[b * (W / 2) + 2 * q + 1]} : dd{0.0, 0.0};
#pragma unroll
            for (int q = 0; q < M; ++q) maxs[q] = have ? fmax(maxs[q], vals[b * (W / 2) + 2 * K + q]) : maxs[q];
        }
#pragma unroll
        for (int w = 1; w < PER; w *= 2)
#pragma unroll
            for (int u = 0; u + w < PER; u += 2 * w) {
                if (32 * (u + w) >= nb) continue;
#pragma unroll
                for (int q = 0; q < K; ++q) v[u][q] = pair_add(v[u][q], v[u + w][q]);
            }
#pragma unroll
        for (int q = 0; q < K; ++q) sums[q] = lanes_sum<32>(v[0][q]);
#pragma unroll
        for (int q = 0; q < M; ++q) maxs[q] = warp_reduce_max(maxs[q]);
    }
    return true;
}

template <int Q>
__global__ void __launch_bounds__(RT, 1) k_jacobi_resident(const __grid_constant__ ResidentArgs A) {
    extern __shared__ __align__(16) double sd[];
    __shared__ SolveState sst;
    __shared__ double sdiag[64], srdiag[64];
    __shared__ BlockReduce<2, 1> red;
    __shared__ __align__(16) unsigned halves[RMAXB * RWORDS];
    const GridDev& g = A.g;
    RCtx c;
    c.red = &red;
    c.halves = halves;
    c.tid = threadIdx.x;
    c.lane = c.tid & 31;
    c.warp = c.tid >> 5;
    if (c.tid < 64) {
        sdiag[c.tid] = g.diag[c.tid];
        srdiag[c.tid] = g.rdiag[c.tid];
    }
    if (c.tid == 0) sst = *A.st;
    const unsigned seq0 = unsigned(*(volatile unsigned long long*)&A.bar->count);
    c.seq = seq0;
    __syncthreads();
    rb200_trace* trace = blockIdx.x == 0 ? A.trace : nullptr;
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2], plane = n0 * n1;
    const int x0 = int(blockIdx.x % unsigned(A.nbx)) * 32;
    const int y0 = int((blockIdx.x / unsigned(A.nbx)) % unsigned(A.nby)) * RY;
    const int k0 = int(blockIdx.x / unsigned(A.nbx * A.nby)) * Q;
    // this thread's z run: cells (i, j, k0 .. k0 + kend - 1)
    const int i = x0 + c.lane, j = y0 + c.warp;
    const bool own = i < n0 && j < n1;
    const int kend = own ? min(Q, n2 - k0) : 0;
    const int e0 = (c.lane + 1) + RX * (c.warp + 1) + SP;
    // shared elements of the x and y neighbours; outside the box the cell
    // itself, whose term in the row is an exact zero
    const int exm = e0 - (i > 0 ? 1 : 0), exp = e0 + (i + 1 < n0 ? 1 : 0);
    const int eym = e0 - (j > 0 ? RX : 0), eyp = e0 + (j + 1 < n1 ? RX : 0);
    const int c0 = i + n0 * (j + n1 * k0);
    const int mxy = int(i > 0) | (int(i + 1 < n0) << 1) | (int(j > 0) << 2) | (int(j + 1 < n1) << 3);
    const bool surface = c.lane == 0 || c.lane == 31 || c.warp == 0 || c.warp == RY - 1;  // of the brick, in x or y
    const bool gauge = own && c0 == 0;
    auto mask_of = [&](int k) { return mxy | (int(k > 0) << 4) | (int(k + 1 < n2) << 5); };

    // the residual of the run: in registers, the last cells of a long run in
    // shared memory (64 registers of residuals leave too few for the phases)
    constexpr int RR = Q - resident_shared_cells(Q);
    double r[RR];
    double* const rs = sd + SP * (Q + 2) + c.tid;
    auto get_r = [&](int u) { return u < RR ? r[u < RR ? u : 0] : rs[(u - RR) * RT]; };
    auto set_r = [&](int u, double v) {
        if (u < RR)
            r[u < RR ? u : 0] = v;
        else
            rs[(u - RR) * RT] = v;
    };
#pragma unroll
    for (int u = 0; u < Q; ++u) set_r(u, u < kend ? __ldcg(A.r + c0 + u * plane) : 0.0);
    // Updates the halo cells inside the box: sd[element] = f(value at the cell
    // of src, sd[element]). A warp's items are rows of the z and y faces (lanes
    // along x) and planes of the x faces (lanes along y, half a warp per face),
    // eight at a time so that the loads overlap.
    const int hz = min(Q, n2 - k0), hy = min(RY, n1 - y0), hx = min(32, n0 - x0);
    const int itz = (2 * hy + RW - 1) / RW, ity = (2 * hz + RW - 1) / RW, itx = (hz + RW - 1) / RW;
    auto halo = [&](const double* src, auto f) {
        constexpr int H = 8;
        for (int t0 = 0; t0 < itz + ity + itx; t0 += H) {
            int e[H];
            double v[H];
#pragma unroll
            for (int q = 0; q < H; ++q) {
                int t = t0 + q, cc = 0;
                bool in = false;
                e[q] = 0;
                if (t < itz) {
                    const int w = c.warp + RW * t, y = w >> 1, up = w & 1;
                    const int k = up ? k0 + hz : k0 - 1;
                    in = w < 2 * hy && c.lane < hx && k >= 0 && k < n2;
                    cc = (x0 + c.lane) + n0 * (y0 + y + n1 * k);
                    e[q] = (c.lane + 1) + RX * (y + 1) + SP * (up ? hz + 1 : 0);
                } else if (t < itz + ity) {
                    const int w = c.warp + RW * (t - itz), z = w >> 1, up = w & 1;
                    const int jj = up ? y0 + hy : y0 - 1;
                    in = w < 2 * hz && c.lane < hx && jj >= 0 && jj < n1;
                    cc = (x0 + c.lane) + n0 * (jj + n1 * (k0 + z));
                    e[q] = (c.lane + 1) + RX * (up ? hy + 1 : 0) + SP * (z + 1);
                } else if (t < itz + ity + itx) {
                    const int z = c.warp + RW * (t - itz - ity), y = c.lane & 15, up = c.lane >> 4;
                    const int ii = up ? x0 + hx : x0 - 1;
                    in = z < hz && y < hy && ii >= 0 && ii < n0;
                    cc = ii + n0 * (y0 + y + n1 * (k0 + z));
                    e[q] = (up ? hx + 1 : 0) + RX * (y + 1) + SP * (z + 1);
                }
                v[q] = in ? __ldcg(src + cc) : 0.0;
                e[q] = in ? e[q] : -1;
            }
#pragma unroll
            for (int q = 0; q < H; ++q)
                if (e[q] >= 0) sd[e[q]] = f(v[q], sd[e[q]]);
        }
    };
    {
        const double* cur = sst.dsel ? A.d1 : A.d0;
        const bool fresh = (sst.flags & F_REPLACED) != 0;  // the next direction is z: the old one is not read
        for (int u = 0; u < kend; ++u) sd[e0 + u * SP] = fresh ? 0.0 : __ldcg(cur + c0 + u * plane);
        halo(cur, [&](double v, double) { return fresh ? 0.0 : v; });
    }
    __syncthreads();

    bool ok = true;
    int iters = 0;
    constexpr int G = Q < 4 ? Q : 4;  // cells whose loads are in flight together
    // p += alpha d: long runs do it inside phase 2, where the traffic overlaps
    // the arithmetic; short ones while the partials travel
    constexpr bool PIN = Q >= 16;
    // diagonals (and reciprocals) of the run's first, inner and last cells: the
    // inner ones have both z neighbours
    const int m0 = mask_of(k0), m1 = mask_of(k0 + max(kend, 1) - 1), mz = mxy | 0x30;
    const double Da = sdiag[m0], ya = srdiag[m0], Dz = sdiag[mz], yz = srdiag[mz], Db = sdiag[m1], yb = srdiag[m1];
    const bool yok = !own || (ya != 0.0 && yz != 0.0 && yb != 0.0);
    const bool full = kend == Q;
    // the diagonal of cell u; a whole run's last cell is known at compile time
    auto pick = [&](bool whole, int u, double a, double mid, double b) {
        if (whole) return u == 0 ? a : u == Q - 1 ? b : mid;
        const double d = u == 0 ? a : mid;
        return u == kend - 1 ? b : d;
    };
    using T = std::true_type;
    using F = std::false_type;
    for (;;) {
        const int flags = sst.flags;
        if (flags & F_DONE) break;
        if (flags & F_NEED_TRUE) {
            // ------------------------------------------ true residual t = b - K p
            // a barrier first: every block's p is complete
            dd s0[1] = {{0.0, 0.0}};
            double none[1] = {0.0};
            if (!(ok = reduce_all<1, 0, true>(c, A, s0, none))) break;
            double* spare = sst.dsel ? A.d0 : A.d1;
            Neu acc;
            double gauge_sq = 0.0, mx = 0.0;
            for (int u = 0; u < kend; ++u) {
                const int k = k0 + u, cc = c0 + u * plane;
                const double* p = A.p + cc;
                const int m = mask_of(k);
                const double pc = __ldcg(p);
                const double kp = row_at(g, pc, m & 1 ? __ldcg(p - 1) : pc, m & 2 ? __ldcg(p + 1) : pc,
                                         m & 4 ? __ldcg(p - n0) : pc, m & 8 ? __ldcg(p + n0) : pc,
                                         m & 16 ? __ldcg(p - plane) : pc, m & 32 ? __ldcg(p + plane) : pc);
                const double t = __ldcg(A.b + cc) - kp;
                spare[cc] = t;
                acc.add(t * t);
                if (cc == 0) gauge_sq = t * t;
                mx = fmax(mx, fabs(t));
            }
            dd sums[2] = {acc.as_dd(), dd_add1(acc.as_dd(), -gauge_sq)};
            double maxs[1] = {mx};
            if (!(ok = reduce_all<2, 1, false>(c, A, sums, maxs))) break;
            if (c.tid == 0) decide_true(&sst, trace, dd_value(sums[0]), dd_value(sums[1]), maxs[0], flags, g.volume);
            __syncthreads();
            continue;
        }
        if (flags & F_NEED_REPLACE) {
            // ------------------------------------------ restart: r = t, z = r/D
            const double* spare = sst.dsel ? A.d0 : A.d1;
            Neu acc;
#pragma unroll
            for (int u = 0; u < Q; ++u) {
                if (u >= kend) continue;
                const int cc = c0 + u * plane;
                const double rc = cc == 0 ? 0.0 : __ldcg(spare + cc);
                set_r(u, rc);
                const int m = mask_of(k0 + u);
                const double zc = cc == 0 ? 0.0 : div_diag(rc, sdiag[m], srdiag[m]);
                if (surface || u == 0 || u == kend - 1) A.z[cc] = zc;
                acc.add(rc * zc);
            }
            dd sums[1] = {acc.as_dd()};
            double none[1] = {0.0};
            if (!(ok = reduce_all<1, 0, true>(c, A, sums, none))) break;
            if (c.tid == 0) decide_rz(&sst, trace, dd_value(sums[0]), MODE_REPLACE);
            __syncthreads();
            continue;
        }
        if (flags & F_STOP) break;
        if (iters >= A.budget) break;

        // ---------------------------------------------- 1: direction, K d, d.q
        {
            // a fresh direction is z: beta = 0 (the old one is finite, or zero at the start)
            const double beta = (flags & F_REPLACED) ? 0.0 : sst.beta;
            const int dsel = sst.dsel;
            halo(A.z, [&](double zc, double dv) { return zc + beta * dv; });
            auto direction = [&](auto full_t) {
                constexpr bool FULL = decltype(full_t)::value;
#pragma unroll
                for (int u0 = 0; u0 < Q; u0 += G) {
                    if (!FULL && u0 >= kend) break;
                    double v[G], rv[G];
                    bool bad = !yok;
#pragma unroll
                    for (int t = 0; t < G; ++t) {
                        v[t] = sd[e0 + (u0 + t) * SP];
                        rv[t] = get_r(u0 + t);
                    }
#pragma unroll
                    for (int t = 0; t < G; ++t) {
                        const int u = u0 + t;
                        const double zc = div_diag_fast(rv[t], pick(FULL, u, Da, Dz, Db), pick(FULL, u, ya, yz, yb));
                        bad |= !div_diag_range_ok(rv[t]);
                        v[t] = zc + beta * v[t];
                    }
                    if (bad) {
                        // a quotient outside the fast division's range
#pragma unroll 1
                        for (int t = 0; t < G; ++t) {
                            double rc = 0.0;
#pragma unroll
                            for (int q = 0; q < G; ++q) rc = q == t ? rv[q] : rc;
                            const double D = sdiag[mask_of(k0 + u0 + t)];
                            const double nv = rc / D + beta * sd[e0 + (u0 + t) * SP];
#pragma unroll
                            for (int q = 0; q < G; ++q) v[q] = q == t ? nv : v[q];
                        }
                    }
#pragma unroll
                    for (int t = 0; t < G; ++t)
                        if (FULL || u0 + t < kend) sd[e0 + (u0 + t) * SP] = v[t];
                    asm volatile("" ::: "memory");  // one group's values live at a time
                }
            };
            if (full)
                direction(T{});
            else
                direction(F{});
            // the z ghosts: a copy of the boundary cell
            if (own && k0 == 0) sd[e0 - SP] = sd[e0];
            if (own && k0 + kend == n2) sd[e0 + kend * SP] = sd[e0 + (kend - 1) * SP];
            __syncthreads();
            Neu2 acc;
            auto cells = [&](auto full_t) {
                constexpr bool FULL = decltype(full_t)::value;
                double vm = sd[e0 - SP], vc = sd[e0];
#pragma unroll
                for (int u = 0; u < Q; ++u) {
                    if (u % G == 0) {
                        if (!FULL && u >= kend) break;
                        asm volatile("" ::: "memory");
                    }
                    const int o = u * SP;
                    const double vp = sd[e0 + o + SP];
                    double qv = row_at(g, vc, sd[exm + o], sd[exp + o], sd[eym + o], sd[eyp + o], vm, vp);
                    if (u == 0 && gauge) qv = 0.0;  // gauge row
                    const double term = vc * qv;
                    (u & 1 ? acc.b : acc.a).add(FULL || u < kend ? term : 0.0);
                    vm = vc;
                    vc = vp;
                }
            };
            if (full)
                cells(T{});
            else
                cells(F{});
            dd sums[1] = {acc.as_dd()};
            double none[1] = {0.0};
            if (!(ok = reduce_all<1, 0, false>(c, A, sums, none))) break;
            if (c.tid == 0) decide_pass1(&sst, trace, dd_value(sums[0]), flags, dsel);
            __syncthreads();
            if (sst.flags & F_DONE) continue;
        }
        // ---------------------------------------------- 2: p, r, z, r.r, r.z
        {
            const int flags2 = sst.flags;
            const double alpha = sst.alpha;
            Neu2 acc_rr, acc_rz;
            bool bad = !yok;
            auto cells = [&](auto full_t) {
                constexpr bool FULL = decltype(full_t)::value;
                auto ld_p = [&](int u) { return PIN && u < Q && (FULL || u < kend) ? __ldcg(A.p + c0 + u * plane) : 0.0; };
                double vm = sd[e0 - SP], vc = sd[e0];
                double pv[G];
#pragma unroll
                for (int t = 0; t < G; ++t) pv[t] = ld_p(t);
#pragma unroll
                for (int u0 = 0; u0 < Q; u0 += G) {
                    if (!FULL && u0 >= kend) break;
                    double pn[G];  // the next group's p travels while this one computes
#pragma unroll
                    for (int t = 0; t < G; ++t) pn[t] = ld_p(u0 + G + t);
#pragma unroll
                    for (int t = 0; t < G; ++t) {
                        const int u = u0 + t, o = u * SP;
                        const double vp = sd[e0 + o + SP];
                        const double qv = row_at(g, vc, sd[exm + o], sd[exp + o], sd[eym + o], sd[eyp + o], vm, vp);
                        double rc = get_r(u) - alpha * qv;
                        if (u == 0 && gauge) rc = 0.0;  // gauge row: r[0], z[0] stay 0
                        if (!FULL && u >= kend) rc = 0.0;
                        set_r(u, rc);
                        (u & 1 ? acc_rr.b : acc_rr.a).add(rc * rc);
                        const double zc = div_diag_fast(rc, pick(FULL, u, Da, Dz, Db), pick(FULL, u, ya, yz, yb));
                        bad |= !div_diag_range_ok(rc);
                        if (FULL || u < kend) {
                            if (surface || u == 0 || (FULL ? u == Q - 1 : u == kend - 1)) A.z[c0 + u * plane] = zc;
                            // p[0] + alpha d[0] = p[0]: d[0] = 0
                            if (PIN) A.p[c0 + u * plane] = pv[t] + alpha * vc;
                        }
                        (u & 1 ? acc_rz.b : acc_rz.a).add(rc * zc);
                        vm = vc;
                        vc = vp;
                    }
#pragma unroll
                    for (int t = 0; t < G; ++t) pv[t] = pn[t];
                    asm volatile("" ::: "memory");
                }
            };
            if (full)
                cells(T{});
            else
                cells(F{});
            if (bad && own) {
                // z by division (r is complete)
                acc_rz = Neu2{};
#pragma unroll
                for (int u = 0; u < Q; ++u) {
                    if (u >= kend) continue;
                    const double rc = get_r(u);
                    const double zc = rc / sdiag[mask_of(k0 + u)];
                    if (surface || u == 0 || u == kend - 1) A.z[c0 + u * plane] = zc;
                    (u & 1 ? acc_rz.b : acc_rz.a).add(rc * zc);
                }
            }
            dd sums[2] = {acc_rr.as_dd(), acc_rz.as_dd()};
            double none[1] = {0.0};
            auto update_p = [&] {
                if (PIN) return;
                double pv[Q];
#pragma unroll
                for (int u = 0; u < Q; ++u) pv[u] = u < kend ? __ldcg(A.p + c0 + u * plane) : 0.0;
#pragma unroll
                for (int u = 0; u < Q; ++u)
                    if (u < kend) A.p[c0 + u * plane] = pv[u] + alpha * sd[e0 + u * SP];
            };
            if (!(ok = reduce_all<2, 0, true>(c, A, sums, none, update_p))) break;
            if (c.tid == 0) decide_pass2(&sst, trace, dd_value(sums[0]), dd_value(sums[1]), flags2, true);
            __syncthreads();
            ++iters;
        }
    }
    if (!ok) {
        if (c.tid == 0) {
            atomicExch(&A.bar->abort, 1u);
            A.st->status = RB200_EXECUTION;
            A.st->flags = A.st->flags | F_DONE | F_STOP;
        }
        return;
    }
    // the vectors of the next launch
    if (c.seq != seq0 && !(sst.flags & F_DONE)) {
        double* cur = sst.dsel ? A.d1 : A.d0;
#pragma unroll
        for (int u = 0; u < Q; ++u) {
            if (u >= kend) continue;
            A.r[c0 + u * plane] = get_r(u);
            cur[c0 + u * plane] = sd[e0 + u * SP];
        }
    }
    if (blockIdx.x == 0 && c.tid == 0) {
        *A.st = sst;
        A.bar->count = c.seq;
    }
}

const void* resident_kernel(int q) {
    switch (q) {
        case 1: return (const void*)k_jacobi_resident<1>;
        case 2: return (const void*)k_jacobi_resident<2>;
        case 4: return (const void*)k_jacobi_resident<4>;
        case 8: return (const void*)k_jacobi_resident<8>;
        case 16: return (const void*)k_jacobi_resident<16>;
        default: return (const void*)k_jacobi_resident<32>;
    }
}

constexpr size_t kResidentSmemMax = 212 * 1024;  // beside the static arrays

}  // namespace

// ------------------------------------------------------------ host side
int resident_setup(const GridDev& g, ResidentPlan* plan, int blocks) {
    *plan = ResidentPlan{};
    int dev = 0, sms = 0, coop = 0;
    RB200_CUDA(cudaGetDevice(&dev));
    RB200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    RB200_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return RB200_OK;
    sms = std::min(sms, RMAXB);
    if (blocks > 0) sms = std::min(sms, blocks);
    // the shortest run whose bricks all have an SM: the most SMs at work
    for (int q : {1, 2, 4, 8, 16, 32}) {
        const long long nbx = (g.n[0] + 31) / 32, nby = (g.n[1] + RY - 1) / RY, nbz = (g.n[2] + q - 1) / q;
        const size_t smem = (size_t(SP) * (q + 2) + size_t(RT) * resident_shared_cells(q)) * sizeof(double);
        if (nbx * nby * nbz > sms || smem > kResidentSmemMax) continue;
        RB200_CUDA(cudaFuncSetAttribute(resident_kernel(q), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        int(kResidentSmemMax)));
        int per_sm = 0;
        RB200_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, resident_kernel(q), RT, smem));
        if (per_sm < 1) continue;
        plan->q = q;
        plan->nbx = int(nbx);
        plan->nby = int(nby);
        plan->blocks = int(nbx * nby * nbz);
        plan->smem = smem;
        return RB200_OK;
    }
    return RB200_OK;
}

size_t resident_words(const ResidentPlan& plan) { return 2 * size_t(plan.blocks) * RWORDS; }

cudaError_t launch_resident(const ResidentPlan& plan, const GridDev& g, SolveState* st, const double* b, double* p,
                            double* r, double* z, double* d0, double* d1, unsigned long long* words, GridBarrier* bar,
                            rb200_trace* trace, int budget, cudaStream_t s) {
    ResidentArgs A{g, st, b, p, r, z, d0, d1, words, bar, trace, budget, plan.nbx, plan.nby};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(plan.blocks), 1, 1);
    cfg.blockDim = dim3(RT, 1, 1);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {&A};
    return cudaLaunchKernelExC(&cfg, resident_kernel(plan.q), args);
}

}  // namespace rb200
