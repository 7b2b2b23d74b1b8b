// Device bodies of the direct preconditioner (direct.hpp): one tile of a
// cosine transform and the FP64 refinement pass. Shared by the single-grid
// kernels (direct.cu) and the packed batch kernels (batch.cu).
#pragma once

#include "direct.hpp"
#include "mg_device.cuh"
#include "pcg_device.cuh"
#include "project.cuh"

namespace rb200 {

constexpr int DCT_THREADS = 256;
// Table rows staged at a time, with a block barrier for each lot (us per solve,
// 16 rows / 32: 256^3 1979 / 1872, 128^3 302 / 295, 512x64x64 413 / 392; 64 boxes
// 2.55 / 2.45 ms of a step).
constexpr int DCT_KB = 32;

__host__ __device__ __forceinline__ int dct_row_pitch(int neP, int noP) { return ((neP + noP + 31) & ~31) + 4; }

enum DctOp : int { DCT_FORWARD = 0, DCT_INVERSE = 1, DCT_SOLVE = 2 };

// Two floats as one register pair, and the pair's multiply-add (each rounded as
// fmaf rounds it).
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// The register block's inner product over one staged table chunk: RM outputs x
// 4 lines per thread. Lines along x (ROW) keep their elements contiguous in
// shared memory and are read four contraction steps at a time; other lines are
// stored line-fastest and read as a quad of lines per step.
template <int RM, bool ROW>
__device__ __forceinline__ void dct_chunk(float (&acc)[RM][4], const float* __restrict__ sT, int mP,
                                          const float* __restrict__ sX, int pitch, int lstep, int rows) {
    unsigned long long p[RM / 2][4];
#pragma unroll
    for (int r = 0; r < RM / 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) p[r][j] = pack2(acc[2 * r][j], acc[2 * r + 1][j]);
#pragma unroll 1
    for (int k = 0; k < rows; k += 4) {
        float b[4][4];  // [step][line]
        if (ROW) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(sX + j * lstep * pitch + k);
                b[0][j] = v.x;
                b[1][j] = v.y;
                b[2][j] = v.z;
                b[3][j] = v.w;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 v = *reinterpret_cast<const float4*>(sX + (k + u) * pitch);
                b[u][0] = v.x;
                b[u][1] = v.y;
                b[u][2] = v.z;
                b[u][3] = v.w;
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            unsigned long long a[RM / 2], w[4];
            const float* t = sT + (k + u) * mP;
            if (RM % 4 == 0) {
#pragma unroll
                for (int r = 0; r < RM / 4; ++r) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(t + 4 * r);
                    a[2 * r] = v.x;
                    a[2 * r + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int r = 0; r < RM / 2; ++r) a[r] = *reinterpret_cast<const unsigned long long*>(t + 2 * r);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = pack2(b[u][j], b[u][j]);
#pragma unroll
            for (int r = 0; r < RM / 2; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) fma2(p[r][j], a[r], w[j]);
        }
    }
#pragma unroll
    for (int r = 0; r < RM / 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(p[r][j], acc[2 * r][j], acc[2 * r + 1][j]);
}

// Both halves of a transform from the staged tile (even part in the first neP
// contraction steps, odd part after it). Table chunks are staged one ahead by
// cp.async; the first barrier also publishes the tile.
template <int RM, bool ROW>
__device__ __forceinline__ void dct_product(float (&ae)[RM][4], float (&ao)[RM][4], const DctAxis& A, const float* te,
                                            const float* to, float* sT, const float* sX, int pitch, int lstep, int m0,
                                            bool active) {
    const int ce = (A.neP + DCT_KB - 1) / DCT_KB, co = (A.noP + DCT_KB - 1) / DCT_KB;
    const int mP = A.mP;
    auto issue = [&](int c) {
        const bool odd = c >= ce;
        const int k0 = (odd ? c - ce : c) * DCT_KB;
        const int rows = min(DCT_KB, (odd ? A.noP : A.neP) - k0);
        const float* src = (odd ? to : te) + size_t(k0) * mP;
        float* dst = sT + (c & 1) * DCT_KB * mP;
        for (int t = threadIdx.x; t < rows * mP / 4; t += blockDim.x) cp_async16_cg(dst + 4 * t, src + 4 * t);
        cp_async_commit();
    };
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) ae[r][j] = ao[r][j] = 0.0f;
    issue(0);
    for (int c = 0; c < ce; ++c) {
        cp_async_wait_all();
        __syncthreads();
        if (c + 1 < ce + co) issue(c + 1);
        if (active)
            dct_chunk<RM, ROW>(ae, sT + (c & 1) * DCT_KB * mP + m0, mP, sX + c * DCT_KB * (ROW ? 1 : pitch), pitch,
                               lstep, min(DCT_KB, A.neP - c * DCT_KB));
    }
    for (int c = 0; c < co; ++c) {
        cp_async_wait_all();
        __syncthreads();
        if (ce + c + 1 < ce + co) issue(ce + c + 1);
        if (active)
            dct_chunk<RM, ROW>(ao, sT + ((ce + c) & 1) * DCT_KB * mP + m0, mP,
                               sX + (A.neP + c * DCT_KB) * (ROW ? 1 : pitch), pitch, lstep,
                               min(DCT_KB, A.noP - c * DCT_KB));
    }
}

// One tile of 32 nb lines (k_dct, k_b_dct). Bound by shared-memory reads and the
// FP32 pipes: n / 2 multiply-adds per element and transform against 8 bytes
// moved, and the tables come from L2. A whole line set per block (a 64 KB tile
// at n = 256) keeps the element traffic at one read and one write a pass; 8 x 4
// outputs a thread take three 16-byte reads for 32 multiply-adds, issued two at
// a time (paired: the five passes of 256^3 857 us against 936 one at a time, in
// a step 3436 against 3610). 8 x 8 outputs, three quarters of the reads but half
// the warps, took 5% longer on a step of 256^3 and 7% on one of 128^3.
// The whole lines of the tile are staged in shared
// memory before anything is written, so src and dst may be the same array.
// `cold`: read src64 instead of src. `scale`: of what the first pass (ROW forward)
// reads and of what the last one (ROW inverse) writes.
template <int RM, bool ROW, int OP>
__device__ __forceinline__ void dct_tile(const DctJob& J, int tile, bool cold, float scale, float* smem) {
    const DctAxis& A = J.A;
    const int n = A.n, ne = A.ne, no = A.no, neP = A.neP, noP = A.noP;
    const int TC = 32 * J.nb, inner = J.inner;
    const int tid = threadIdx.x, nth = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int wm = warp % A.MB, wn = warp / A.MB;
    const bool active = wn < J.nb;
    const int m0 = (4 * wm + (lane & 3)) * RM;
    const int cn = 8 * wn + (lane >> 2);
    float* const sT = smem;
    int* const sB = reinterpret_cast<int*>(sT + 2 * DCT_KB * A.mP);  // first element of each line, -1 past the end
    float* const sX = reinterpret_cast<float*>(sB + TC);
    const int pitch = ROW ? dct_row_pitch(neP, noP) : TC;
    const int line0 = tile * TC;
    for (int t = tid; t < TC; t += nth) {
        const int line = line0 + t;
        int base = -1;
        if (line < J.lines) {
            const int o = line / inner;
            base = ROW ? line * n : o * inner * n + (line - o * inner);
        }
        sB[t] = base;
    }
    __syncthreads();
    const float4 z4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const bool vec = ROW ? (n & 7) == 0 : (inner & 3) == 0;
    const float* __restrict__ src = J.src;
    const double* __restrict__ s64 = J.src64;
    // ---- stage the tile
    if (ROW) {
        auto ld4f = [&](int at) -> float4 {
            if (cold) {
                const double2 a = *reinterpret_cast<const double2*>(s64 + at);
                const double2 b = *reinterpret_cast<const double2*>(s64 + at + 2);
                return make_float4(float(a.x) * scale, float(a.y) * scale, float(b.x) * scale, float(b.y) * scale);
            }
            const float4 v = *reinterpret_cast<const float4*>(src + at);
            return make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
        };
        auto ld1 = [&](int at) -> float { return (cold ? float(s64[at]) : src[at]) * scale; };
        if (vec && OP == DCT_FORWARD) {
            const int iq = ne >> 2;
#pragma unroll 4
            for (int t = tid; t < TC * iq; t += nth) {
                const int r = t / iq, q = t - r * iq, base = sB[r];
                float4 a = z4, b = z4;
                if (base >= 0) {
                    a = ld4f(base + 4 * q);
                    b = ld4f(base + n - 4 - 4 * q);
                }
                float* d = sX + r * pitch + 4 * q;
                *reinterpret_cast<float4*>(d) = make_float4(a.x + b.w, a.y + b.z, a.z + b.y, a.w + b.x);
                *reinterpret_cast<float4*>(d + neP) = make_float4(a.x - b.w, a.y - b.z, a.z - b.y, a.w - b.x);
            }
        } else if (vec) {
            const int iq = n >> 2;
#pragma unroll 4
            for (int t = tid; t < TC * iq; t += nth) {
                const int r = t / iq, q = t - r * iq, base = sB[r];
                const float4 a = base >= 0 ? *reinterpret_cast<const float4*>(src + base + 4 * q) : z4;
                *reinterpret_cast<float4*>(sX + r * pitch + 4 * q) = a;
            }
        } else {
            for (int t = tid; t < TC * neP; t += nth) {
                const int r = t / neP, i = t - r * neP, base = sB[r];
                float e = 0.0f, o = 0.0f;
                if (base >= 0) {
                    if (OP == DCT_FORWARD) {
                        if (i < no) {
                            const float a = ld1(base + i), b = ld1(base + n - 1 - i);
                            e = a + b;
                            o = a - b;
                        } else if (i < ne) {
                            e = ld1(base + i);
                        }
                    } else {
                        if (i < ne) e = src[base + i];
                        if (i < no) o = src[base + ne + i];
                    }
                }
                sX[r * pitch + i] = e;
                if (i < noP) sX[r * pitch + neP + i] = o;
            }
        }
    } else if (vec) {
        const int qt = TC >> 2;
#pragma unroll 4
        for (int t = tid; t < neP * qt; t += nth) {
            const int i = t / qt, q = t - i * qt, base = sB[4 * q];
            float4 e = z4, o = z4;
            if (base >= 0) {
                if (OP == DCT_INVERSE) {
                    if (i < ne) e = *reinterpret_cast<const float4*>(src + base + i * inner);
                    if (i < no) o = *reinterpret_cast<const float4*>(src + base + (ne + i) * inner);
                } else if (i < no) {
                    const float4 a = *reinterpret_cast<const float4*>(src + base + i * inner);
                    const float4 b = *reinterpret_cast<const float4*>(src + base + (n - 1 - i) * inner);
                    e = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
                    o = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
                } else if (i < ne) {
                    e = *reinterpret_cast<const float4*>(src + base + i * inner);
                }
            }
            *reinterpret_cast<float4*>(sX + i * pitch + 4 * q) = e;
            if (i < noP) *reinterpret_cast<float4*>(sX + (neP + i) * pitch + 4 * q) = o;
        }
    } else {
#pragma unroll 4
        for (int t = tid; t < neP * TC; t += nth) {
            const int i = t / TC, q = t - i * TC, base = sB[q];
            float e = 0.0f, o = 0.0f;
            if (base >= 0) {
                if (OP == DCT_INVERSE) {
                    if (i < ne) e = src[base + i * inner];
                    if (i < no) o = src[base + (ne + i) * inner];
                } else if (i < no) {
                    const float a = src[base + i * inner], b = src[base + (n - 1 - i) * inner];
                    e = a + b;
                    o = a - b;
                } else if (i < ne) {
                    e = src[base + i * inner];
                }
            }
            sX[i * pitch + q] = e;
            if (i < noP) sX[(neP + i) * pitch + q] = o;
        }
    }
    // ---- products
    float ae[RM][4], ao[RM][4];
    const int lstep = 8 * J.nb;  // ROW: a thread's lines cn, cn + lstep, ...
    const float* const sXt = ROW ? sX + cn * pitch : sX + 4 * cn;
    dct_product<RM, ROW>(ae, ao, A, OP == DCT_INVERSE ? A.ie : A.fe, OP == DCT_INVERSE ? A.io : A.fo, sT, sXt, pitch,
                         lstep, m0, active);
    if (OP == DCT_SOLVE) {
        // divide by the eigenvalues and transform back, in place in the tile
        __syncthreads();
        if (active) {
            float lxy[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int line = line0 + 4 * cn + j;
                const int y = line / J.n0;
                lxy[j] = line < J.lines ? J.lam0[line - y * J.n0] + J.lam1[y] : 1.0f;
            }
#pragma unroll
            for (int r = 0; r < RM; ++r) {
                const int m = m0 + r;
                if (m < ne) {
                    const float lz = A.lam[m];
                    float v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float l = lxy[j] + lz;
                        v[j] = l > 0.0f ? ae[r][j] / l : 0.0f;
                    }
                    *reinterpret_cast<float4*>(sX + m * pitch + 4 * cn) = make_float4(v[0], v[1], v[2], v[3]);
                }
                if (m < no) {
                    const float lz = A.lam[ne + m];
                    float v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = ao[r][j] / (lxy[j] + lz);
                    *reinterpret_cast<float4*>(sX + (neP + m) * pitch + 4 * cn) = make_float4(v[0], v[1], v[2], v[3]);
                }
            }
        }
        dct_product<RM, ROW>(ae, ao, A, A.ie, A.io, sT, sXt, pitch, lstep, m0, active);
    }
    // ---- results
    float* __restrict__ dst = J.dst;
    if (ROW) {
        __syncthreads();
        if (active) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float* row = sX + (cn + j * lstep) * pitch;
#pragma unroll
                for (int r = 0; r < RM; ++r) {
                    const int m = m0 + r;
                    if (OP == DCT_FORWARD) {
                        if (m < ne) row[m] = ae[r][j];
                        if (m < no) row[ne + m] = ao[r][j];
                    } else if (m < no) {
                        row[m] = (ae[r][j] + ao[r][j]) * scale;
                        row[n - 1 - m] = (ae[r][j] - ao[r][j]) * scale;
                    } else if (m < ne) {
                        row[m] = ae[r][j] * scale;
                    }
                }
            }
        }
        __syncthreads();
        if (vec) {
            const int iq = n >> 2;
            for (int t = tid; t < TC * iq; t += nth) {
                const int r = t / iq, q = t - r * iq, base = sB[r];
                if (base >= 0)
                    *reinterpret_cast<float4*>(dst + base + 4 * q) =
                        *reinterpret_cast<const float4*>(sX + r * pitch + 4 * q);
            }
        } else {
            for (int t = tid; t < TC * n; t += nth) {
                const int r = t / n, i = t - r * n, base = sB[r];
                if (base >= 0) dst[base + i] = sX[r * pitch + i];
            }
        }
    } else if (active) {
        auto put = [&](int i, const float (&v)[4]) {
            if (vec) {
                const int base = sB[4 * cn];
                if (base >= 0) *reinterpret_cast<float4*>(dst + base + i * inner) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int base = sB[4 * cn + j];
                    if (base >= 0) dst[base + i * inner] = v[j];
                }
            }
        };
#pragma unroll
        for (int r = 0; r < RM; ++r) {
            const int m = m0 + r;
            if (OP == DCT_FORWARD) {
                if (m < ne) put(m, ae[r]);
                if (m < no) put(ne + m, ao[r]);
            } else if (m < no) {
                float lo[4], hi[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    lo[j] = ae[r][j] + ao[r][j];
                    hi[j] = ae[r][j] - ao[r][j];
                }
                put(m, lo);
                put(n - 1 - m, hi);
            } else if (m < ne) {
                put(m, ae[r]);
            }
        }
    }
}

template <bool ROW, int OP>
__device__ __forceinline__ void dct_tile_any(const DctJob& J, int tile, bool cold, float scale, float* smem) {
    if (J.A.RM == 8)
        dct_tile<8, ROW, OP>(J, tile, cold, scale, smem);
    else if (J.A.RM == 6)
        dct_tile<6, ROW, OP>(J, tile, cold, scale, smem);
    else
        dct_tile<4, ROW, OP>(J, tile, cold, scale, smem);
}

// build_rhs (project.cuh) with the start of a cold solve on it (the sums of b,
// |b| and b^2, max|b| and the decision of init_sums_body, pcg_device.cuh) in
// one pass: b is written once and not read back, and p is not zeroed (a solve
// that ends at iteration 0 has it zeroed by k_settle). Rows of a multiple of 4
// cells take quads and march along z as correct_divergence_quads does. Bound by
// HBM (20 bytes a cell in f32). The two passes it replaces took 101 + 97 us at
// 256^3 on a B200 and 0.28 + 0.25 ms over 64 boxes of 32^3 to 96^3; this one
// about 100 us and 0.26 ms.
template <class T>
__device__ __forceinline__ void rhs_init_body(const GridDev& g, const T* __restrict__ u, const T* __restrict__ v,
                                              const T* __restrict__ w, double dt, double* __restrict__ out, int* vflags,
                                              SolveState* st, Partials part, Span sp) {
    __shared__ BlockReduce<3, 3> sm;
    const double rdt = div_reciprocal(dt);
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    Neu sum[3];
    double m[3] = {0.0, 0.0, 0.0};
    int local = 0;
    auto value = [&](T xl, T xh, T yl, T yh, T zl, T zh) {
        double flux = 0.0;
        flux += g.area[0] * (double(xl) - double(xh));
        flux += g.area[1] * (double(yl) - double(yh));
        flux += g.area[2] * (double(zl) - double(zh));
        const double b = div_diag(flux, dt, rdt);
        if (!isfinite(b)) {
            local |= VF_ARITH;
            m[1] = 1.0;
        }
        const double a = fabs(b);
        sum[0].add(b);
        sum[1].add(a);
        sum[2].add(b * b);
        m[0] = a > m[0] ? a : m[0];
        return b;
    };
    if ((n0 & 3) == 0) {
        const int quads = n0 >> 2, sz = n0 * n1;
        const int items = quads * n1, segs = (items + 31) >> 5;
        const int lane = threadIdx.x & 31, nw = sp.blocks * int(blockDim.x >> 5);
        const int kc = march_planes(segs, n2, nw), kcs = (n2 + kc - 1) / kc;
        for (int line = sp.block * int(blockDim.x >> 5) + int(threadIdx.x >> 5); line < segs * kcs; line += nw) {
            const int seg = line % segs, kb = (line / segs) * kc, ke = min(n2, kb + kc);
            const int it = seg * 32 + lane;
            if (it >= items) continue;
            const int j = it / quads, i0 = 4 * (it - j * quads);
            int c = i0 + n0 * (j + n1 * kb);
            T wl[4];
            ld4(w + c, wl);
            for (int k = kb; k < ke; ++k, c += sz) {
                const int fu = i0 + (n0 + 1) * (j + n1 * k), fv = i0 + n0 * (j + (n1 + 1) * k);
                T x[5], vl[4], vh[4], wh[4];
#pragma unroll
                for (int e = 0; e < 5; ++e) x[e] = u[fu + e];
                ld4(v + fv, vl);
                ld4(v + fv + n0, vh);
                ld4(w + c + sz, wh);
                double b[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    b[e] = value(x[e], x[e + 1], vl[e], vh[e], wl[e], wh[e]);
                    wl[e] = wh[e];
                }
                st4(out + c, b);
            }
        }
    } else {
        for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
            int i, j, k;
            cell_coords(g, c, i, j, k);
            out[c] = value(u[face_idx(g, 0, i, j, k)], u[face_idx(g, 0, i + 1, j, k)], v[face_idx(g, 1, i, j, k)],
                           v[face_idx(g, 1, i, j + 1, k)], w[face_idx(g, 2, i, j, k)], w[face_idx(g, 2, i, j, k + 1)]);
        }
    }
    if (local) atomicOr(vflags, local);
    dd s[3] = {sum[0].as_dd(), sum[1].as_dd(), sum[2].as_dd()};
    block_reduce<3, 3>(sm, s, m);
    if (publish_and_check_last<3, 3>(part, sp.block, sp.blocks, s, m)) {
        fold_partials<3, 3>(part, sp.blocks, sm, s, m);
        if (threadIdx.x == 0) decide_init(g, st, s, m, false, nullptr);
    }
}

// Whether a finished solve left p untouched: it ended on the right-hand side,
// and p = 0 is its result.
__device__ __forceinline__ bool settle_zero(const SolveState* st) {
    return st->it == 0 && !(st->flags & F_WARM) && st->status != ST_RUNNING;
}

// Decision after a refinement iteration's true residual (`squared`, `maximum`
// over every row): solve_loaded's acceptance and iteration limit
// (src/pressure.rs:686-715); the residual is the true one, so there is no
// candidate and no restart.
__device__ __forceinline__ void decide_refined(SolveState* st, rb200_trace* trace, double squared, double maximum,
                                               int flags, double volume, bool seed) {
    const int it = seed ? 0 : st->it + 1;
    if (!seed) {
        st->it = it;
        st->dsel ^= 1;
    }
    const double div = maximum * st->dt / volume;
    const double l2 = sqrt(squared);
    st->recursive_l2 = l2;
    if (trace && it >= 1) {
        rb200_trace& t = trace[it - 1];
        t.alpha = 1.0;  // p += z
        t.recursive_l2 = l2;
        t.checked = 1;
    }
    flags = with_transform_scale(flags & ~(F_STOP | F_NEED_TRUE), maximum);
    if (!isfinite(squared) || !isfinite(div)) {
        breakdown(st, it, flags);
        return;
    }
    // what FP32 holds of a residual below its normal range has nothing more to
    // give than an iteration that did not halve it
    const bool spent = !seed && maximum < 0x1p-126 && !(maximum < 0.5 * st->true_max);
    st->true_l2 = l2;
    st->true_max = maximum;
    st->true_div = div;
    if (l2 <= st->threshold && div <= st->divergence_limit)
        finish(st, RB200_OK, flags);
    else if (it == st->max_it)
        finish(st, RB200_ITERATION_LIMIT, flags);
    else if (spent)
        breakdown(st, it, flags);
    else
        st->flags = flags;
}

// The refinement pass: p_new = p + (z - z[0]) (z alone in a cold solve's first
// iteration; p itself for the seed's residual), t = b - K p_new in FP64,
// r32 = f32(t), |t|^2 and max|t|. p_new goes to the other p buffer, because
// neighbours read the old one. A warp takes a line of quads of one row and
// marches along z with the z neighbours in registers.
__device__ __forceinline__ void refine_body(const GridDev& g, SolveState* st, const double* __restrict__ b, double* pa,
                                            double* pb, const float* __restrict__ z, float* __restrict__ r32,
                                            Partials part, rb200_trace* trace, bool seed, int kc_len, Span sp) {
    __shared__ BlockReduce<1, 1> red;
    const int flags = st->flags;
    if (flags & F_DONE) return;
    if (seed != ((flags & F_NEED_TRUE) != 0)) return;
    const bool old = seed || st->it > 0 || (flags & F_WARM);
    const int sel = st->dsel;
    const double* __restrict__ po = sel ? pb : pa;
    double* __restrict__ pn = sel ? pa : pb;
    const double z0 = seed ? 0.0 : double(z[0]);
    auto val = [&](int c) -> double {
        const double zc = seed ? 0.0 : double(z[c]) - z0;
        return old ? po[c] + zc : zc;
    };
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2], sy = n0, sz = n0 * n1;
    Neu acc;
    double mx[1] = {0.0};
    const Warps W = span_warps(sp);
    if ((n0 & 3) == 0) {
        const int quads = n0 >> 2;
        auto val4 = [&](int c0, double (&o)[4]) {
            if (old)
                ld_quad(po + c0, o);
            else
                o[0] = o[1] = o[2] = o[3] = 0.0;
            if (!seed) {
                const float4 zv = *reinterpret_cast<const float4*>(z + c0);
                o[0] += double(zv.x) - z0;
                o[1] += double(zv.y) - z0;
                o[2] += double(zv.z) - z0;
                o[3] += double(zv.w) - z0;
            }
        };
        // lanes are dealt (row, quad) pairs of one plane, consecutive in memory
        const int items = quads * n1, segs = (items + 31) >> 5;
        const int kcs = (n2 + kc_len - 1) / kc_len;
        for (int line = W.w0; line < segs * kcs; line += W.nw) {
            const int seg = line % segs, kb = (line / segs) * kc_len, ke = min(n2, kb + kc_len);
            const int it = seg * 32 + W.lane;
            if (it >= items) continue;
            const int j = it / quads, i0 = 4 * (it - j * quads);
            double prev[4] = {0, 0, 0, 0}, cur[4], next[4];
            const int base = n0 * (j + n1 * kb) + i0;
            if (kb > 0) val4(base - sz, prev);
            val4(base, cur);
            for (int k = kb; k < ke; ++k) {
                const int c0 = base + (k - kb) * sz;
                double ym[4] = {0, 0, 0, 0}, yp[4] = {0, 0, 0, 0};
                double bv[4];
                ld_quad(b + c0, bv);
#pragma unroll
                for (int e = 0; e < 4; ++e) next[e] = 0.0;
                if (k + 1 < n2) val4(c0 + sz, next);
                if (j > 0) val4(c0 - sy, ym);
                if (j + 1 < n1) val4(c0 + sy, yp);
                const double xl = i0 > 0 ? val(c0 - 1) : 0.0;
                const double xr = i0 + 4 < n0 ? val(c0 + 4) : 0.0;
                float4 rq;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    Neigh v;
                    v.c = cur[e];
                    v.xm = e == 0 ? xl : cur[e - 1];
                    v.xp = e == 3 ? xr : cur[e + 1];
                    v.ym = ym[e];
                    v.yp = yp[e];
                    v.zm = prev[e];
                    v.zp = next[e];
                    const double t = bv[e] - apply_row(g, i0 + e, j, k, v);
                    acc.add(t * t);
                    mx[0] = fmax(mx[0], fabs(t));
                    f4put(rq, e, float(t));
                }
                if (!seed) {
                    *reinterpret_cast<double2*>(pn + c0) = make_double2(cur[0], cur[1]);
                    *reinterpret_cast<double2*>(pn + c0 + 2) = make_double2(cur[2], cur[3]);
                }
                *reinterpret_cast<float4*>(r32 + c0) = rq;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    prev[e] = cur[e];
                    cur[e] = next[e];
                }
            }
        }
    } else {
        for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
            int i, j, k;
            cell_coords(g, c, i, j, k);
            Neigh v;
            v.c = val(c);
            v.xm = i > 0 ? val(c - 1) : 0.0;
            v.xp = i + 1 < n0 ? val(c + 1) : 0.0;
            v.ym = j > 0 ? val(c - sy) : 0.0;
            v.yp = j + 1 < n1 ? val(c + sy) : 0.0;
            v.zm = k > 0 ? val(c - sz) : 0.0;
            v.zp = k + 1 < n2 ? val(c + sz) : 0.0;
            const double t = b[c] - apply_row(g, i, j, k, v);
            acc.add(t * t);
            mx[0] = fmax(mx[0], fabs(t));
            if (!seed) pn[c] = v.c;
            r32[c] = float(t);
        }
    }
    // a NaN anywhere leaves |t|^2 NaN, which decides; fmax alone would drop it
    dd sums[1] = {acc.as_dd()};
    block_reduce<1, 1>(red, sums, mx);
    if (publish_and_check_last<1, 1>(part, sp.block, sp.blocks, sums, mx)) {
        fold_partials<1, 1>(part, sp.blocks, red, sums, mx);
        if (threadIdx.x == 0) decide_refined(st, trace, dd_value(sums[0]), mx[0], flags, g.volume, seed);
    }
}

}  // namespace rb200
