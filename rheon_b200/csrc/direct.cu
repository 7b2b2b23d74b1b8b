// Fast diagonalisation of the sealed box (direct.hpp): the cosine-transform
// passes and the FP64 refinement pass of one grid.
#include <algorithm>
#include <cmath>
#include <vector>

#include "direct_device.cuh"
#include "pdl.hpp"

namespace rb200 {

// One transform pass: a block per tile of lines.
template <bool ROW, int OP>
__global__ void __launch_bounds__(DCT_THREADS, 2) k_dct(const __grid_constant__ DctJob J, const SolveState* st) {
    pdl_wait();
    extern __shared__ float4 dct_smem[];
    const int flags = st->flags;
    if (flags & F_DONE) return;
    const bool cold = J.src64 != nullptr && st->it == 0 && !(flags & F_WARM);
    const float scale = ROW ? transform_scale(flags, OP != DCT_FORWARD) : 1.0f;
    dct_tile_any<ROW, OP>(J, blockIdx.x, cold, scale, reinterpret_cast<float*>(dct_smem));
}

__global__ void __launch_bounds__(MG_THREADS, 3) k_refine(GridDev g, SolveState* st, const double* b, double* pa,
                                                       double* pb, const float* z, float* r32, Partials part,
                                                       rb200_trace* trace, int seed, int kc_len) {
    pdl_wait();
    refine_body(g, st, b, pa, pb, z, r32, part, trace, seed != 0, kc_len, whole_launch());
}

__global__ void __launch_bounds__(256) k_settle(int cells, const SolveState* st, double* __restrict__ pa,
                                                const double* __restrict__ pb) {
    pdl_wait();
    if (!(st->flags & F_DONE)) return;
    const bool zero = settle_zero(st);
    if (!zero && !st->dsel) return;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < cells; c += gridDim.x * blockDim.x)
        pa[c] = zero ? 0.0 : pb[c];
}

// ------------------------------------------------------------ host side
bool direct_supported(const GridDev& g) {
    int longest = 0;
    double top = 0.0, low = 0.0, wmax = 0.0;
    for (int d = 0; d < 3; ++d) {
        longest = std::max(longest, g.n[d]);
        const double s = std::sin(CUDART_PI / (2.0 * g.n[d]));
        const double first = 4.0 * g.weight[d] * s * s;  // the axis' smallest nonzero eigenvalue
        if (g.n[d] > 1) {
            top += 4.0 * g.weight[d];
            low = low > 0.0 ? std::min(low, first) : first;
        }
        wmax = std::max(wmax, g.weight[d]);
    }
    // Where it applies it is the faster of the two (us per carrier step, direct /
    // multigrid: 32^3 177 / 521, 64^3 227 / 734, 128^3 495 / 1752, 512x64x64
    // 584 / 3060, 256^3 2894 / 7198). Larger axes do not fit the transform's
    // tile. The FP32 rounding of z comes back through K as noise spread over
    // the whole spectrum, which the next iteration reduces by 10^5 or more, so
    // uneven spacings cost an iteration where point relaxation stalls
    // (iterations to 1e-8, direct / multigrid: 96x16x16 with h = (1, 0.02,
    // 0.02), condition 2 10^7, 3 / 262; 64^3 with h = (1, 0.01, 1), condition
    // 2 10^7, 3 / more than 300). Up to 10^9 it also holds where the FP64
    // residual's own rounding is the limit, of either method: that floor grows
    // with the condition and is highest for smooth right-hand sides, which end at
    // 1e-8 from a condition of 3 10^8 on and at 2 to 4e-8 near 10^9, where noise
    // still takes 4 iterations to 1e-8. Weights near the ends of the FP32 range
    // stay with the multigrid method too.
    return longest > 8 && longest <= kDctMaxAxis && top <= 1e9 * low && wmax > 1e-12 && wmax < 1e12;
}

DctTables::~DctTables() { cudaFree(data_); }

int DctTables::init(const GridDev& g, cudaStream_t s) {
    std::vector<float> host;
    size_t at[3][5];
    for (int d = 0; d < 3; ++d) {
        DctAxis& A = axis[d];
        const int n = g.n[d];
        A.n = n;
        A.ne = (n + 1) / 2;
        A.no = n / 2;
        A.neP = (A.ne + 3) & ~3;
        A.noP = (A.no + 3) & ~3;
        // outputs per thread: the least padding, then the larger block
        A.mP = 0;
        for (int rm : {8, 6, 4}) {
            const int mb = (A.ne + 4 * rm - 1) / (4 * rm);
            if (mb <= 8 && (A.mP == 0 || 4 * rm * mb < A.mP)) {
                A.RM = rm;
                A.MB = mb;
                A.mP = 4 * rm * mb;
            }
        }
        int same = -1;
        for (int e = 0; e < d; ++e)
            if (g.n[e] == n) same = e;
        if (same >= 0) {
            for (int q = 0; q < 4; ++q) at[d][q] = at[same][q];
        } else {
            auto basis = [&](int q, int i) {
                // cos(pi q (2i + 1) / 2n), the angle reduced in integers
                const long long a = (long long)q * (2 * i + 1) % (4ll * n);
                return std::cos(CUDART_PI * double(a) / (2.0 * n)) * std::sqrt((q ? 2.0 : 1.0) / n);
            };
            auto table = [&](int which, int K, int KP, bool odd, bool inverse) {
                at[d][which] = host.size();
                host.resize(host.size() + size_t(KP) * A.mP, 0.0f);
                float* t = host.data() + at[d][which];
                for (int k = 0; k < K; ++k)
                    for (int m = 0; m < K; ++m)
                        t[size_t(k) * A.mP + m] = float(inverse ? basis(2 * k + odd, m) : basis(2 * m + odd, k));
            };
            table(0, A.ne, A.neP, false, false);
            table(1, A.no, A.noP, true, false);
            table(2, A.ne, A.neP, false, true);
            table(3, A.no, A.noP, true, true);
        }
        at[d][4] = host.size();
        host.resize(host.size() + size_t((n + 3) & ~3), 0.0f);
        for (int q = 0; q < n; ++q) {
            const double sn = std::sin(CUDART_PI * q / (2.0 * n));
            host[at[d][4] + (q & 1 ? A.ne + q / 2 : q / 2)] = float(4.0 * g.weight[d] * sn * sn);
        }
    }
    RB200_CUDA(cudaMalloc(&data_, host.size() * sizeof(float)));
    bytes_ = host.size() * sizeof(float);
    RB200_CUDA(cudaMemcpyAsync(data_, host.data(), bytes_, cudaMemcpyHostToDevice, s));
    RB200_CUDA(cudaStreamSynchronize(s));
    for (int d = 0; d < 3; ++d) {
        axis[d].fe = data_ + at[d][0];
        axis[d].fo = data_ + at[d][1];
        axis[d].ie = data_ + at[d][2];
        axis[d].io = data_ + at[d][3];
        axis[d].lam = data_ + at[d][4];
    }
    return RB200_OK;
}

size_t direct_job_smem(const DctJob& J) {
    const size_t tc = 32 * size_t(J.nb), k = size_t(J.A.neP + J.A.noP);
    const size_t tile = J.inner == 1 ? tc * dct_row_pitch(J.A.neP, J.A.noP) : tc * k;
    return (2 * size_t(DCT_KB) * J.A.mP + tc + tile) * sizeof(float);
}

void direct_jobs(const DctTables& T, const GridDev& g, const double* b, const float* r32, float* z, bool alone,
                 DctJob (&jobs)[5]) {
    const int axis_of[5] = {0, 1, 2, 1, 0};
    for (int q = 0; q < 5; ++q) {
        DctJob& J = jobs[q];
        const int d = axis_of[q];
        J = DctJob{};
        J.A = T.axis[d];
        J.inner = d == 0 ? 1 : (d == 1 ? g.n[0] : g.n[0] * g.n[1]);
        J.lines = g.cells / g.n[d];
        J.n0 = g.n[0];
        J.src = q == 0 ? r32 : z;
        J.src64 = q == 0 ? b : nullptr;
        J.dst = z;
        J.lam0 = T.axis[0].lam;
        J.lam1 = T.axis[1].lam;
        // Tiles as wide as eight warps allow while two blocks per SM all have
        // one; narrower ones on small grids.
        // Few lines leave the SMs without warps to hide the shared reads: below
        // six warps an SM a thread takes 4 outputs, and a transform up to twice
        // the warps (us per solve of two iterations, 6 or 8 outputs / 4: 64^3
        // 175 / 148, 90x75x63 279 / 227, 96^3 206 / 195, 112^3 266 / 247; at
        // seven warps an SM 128^3 302 / 302, 512x64x64 414 / 448). A batch fills
        // the chip with its instances: 64 boxes 2.55 / 2.77 ms of a step.
        if (alone && J.A.RM > 4 && (J.lines + 31) / 32 * J.A.MB < 6 * 148 && J.A.mP % 16 == 0 && J.A.mP <= 128) {
            J.A.RM = 4;
            J.A.MB = J.A.mP / 16;
        }
        J.nb = std::max(1, 8 / J.A.MB);
        while (J.nb > 1 && (J.lines + 32 * J.nb - 1) / (32 * J.nb) < 2 * 148) --J.nb;
        J.tiles = (J.lines + 32 * J.nb - 1) / (32 * J.nb);
    }
}

DirectSolver::~DirectSolver() {
    cudaFree(r32_);
    cudaFree(z_);
}

int DirectSolver::init(const GridDev& g, cudaStream_t s) {
    int rc = tables_.init(g, s);
    if (rc) return rc;
    const size_t n = size_t(g.cells) * sizeof(float);
    if (cudaMalloc(&r32_, n) != cudaSuccess || cudaMalloc(&z_, n) != cudaSuccess) {
        cudaGetLastError();
        set_error("direct preconditioner: out of device memory");
        return RB200_OUT_OF_MEMORY;
    }
    bytes_ = tables_.bytes() + 2 * n;
    const int smem = int(kDctSmemMax);
    RB200_CUDA(cudaFuncSetAttribute(k_dct<true, DCT_FORWARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    RB200_CUDA(cudaFuncSetAttribute(k_dct<true, DCT_INVERSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    RB200_CUDA(cudaFuncSetAttribute(k_dct<false, DCT_FORWARD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    RB200_CUDA(cudaFuncSetAttribute(k_dct<false, DCT_INVERSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    RB200_CUDA(cudaFuncSetAttribute(k_dct<false, DCT_SOLVE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return RB200_OK;
}

// Blocks and z-march length of the refinement pass: one warp per line of 32
// quads and 8 planes, less where that leaves SMs without work.
static void refine_shape(const GridDev& g, int* blocks, int* kc_len) {
    if (g.n[0] & 3) {
        *kc_len = 1;
        *blocks = std::max(1, std::min((g.cells + MG_THREADS - 1) / MG_THREADS, 148 * 8));
        return;
    }
    const long long segs = ((long long)(g.n[0] / 4) * g.n[1] + 31) / 32;
    int kc = 16;
    while (kc > 1 && segs * ((g.n[2] + kc - 1) / kc) < 148ll * 16) kc /= 2;
    const long long lines = segs * ((g.n[2] + kc - 1) / kc);
    *kc_len = kc;
    *blocks = int(std::max(1ll, std::min((lines + MG_THREADS / 32 - 1) / (MG_THREADS / 32), 148ll * 8)));
}

int DirectSolver::enqueue_seed(const GridDev& g, SolveState* st, const double* b, double* p, double* p2, Partials part,
                               cudaStream_t s) const {
    int blocks, kc;
    refine_shape(g, &blocks, &kc);
    k_refine<<<blocks, MG_THREADS, 0, s>>>(g, st, b, p, p2, z_, r32_, part, nullptr, 1, kc);
    return 1;
}

int DirectSolver::enqueue_iteration(const GridDev& g, SolveState* st, const double* b, double* p, double* p2,
                                    Partials part, rb200_trace* trace, cudaStream_t s) const {
    DctJob jobs[5];
    direct_jobs(tables_, g, b, r32_, z_, true, jobs);
    auto go = [&](void (*kernel)(const DctJob, const SolveState*), const DctJob& J) {
        pdl_launch(kernel, dim3(J.tiles), dim3(32 * J.A.MB * J.nb), direct_job_smem(J), s, J,
                   static_cast<const SolveState*>(st));
    };
    go(k_dct<true, DCT_FORWARD>, jobs[0]);
    go(k_dct<false, DCT_FORWARD>, jobs[1]);
    go(k_dct<false, DCT_SOLVE>, jobs[2]);
    go(k_dct<false, DCT_INVERSE>, jobs[3]);
    go(k_dct<true, DCT_INVERSE>, jobs[4]);
    int blocks, kc;
    refine_shape(g, &blocks, &kc);
    pdl_launch(k_refine, dim3(blocks), dim3(MG_THREADS), 0, s, g, st, b, p, p2, static_cast<const float*>(z_), r32_,
               part, trace, 0, kc);
    return 6;
}

int DirectSolver::enqueue_settle(const GridDev& g, SolveState* st, double* p, const double* p2, cudaStream_t s) const {
    const int blocks = std::max(1, std::min((g.cells + 255) / 256, 148 * 8));
    pdl_launch(k_settle, dim3(blocks), dim3(256), 0, s, g.cells, static_cast<const SolveState*>(st), p, p2);
    return 1;
}

}  // namespace rb200
