// Device bodies of the operator steps the resident carrier shares with the
// standalone primitives: build_rhs, the actual divergence, the gradient
// correction and the fused correction/divergence/velocity-rate epilogue.
#pragma once

#include "internal.hpp"

namespace rb200 {

constexpr int EW_THREADS = 256;
constexpr int EW_BLOCKS_CAP = 148 * 8;
constexpr float kF32Max = 3.40282346638528859811704183484516925440e+38f;

// ------------------------------------------------------------ build_rhs
// build_rhs (src/operator.rs:460-509) / build_rhs_f64 (:672-708):
//   flux = 0; flux += area_d * (f64(u_lo) - f64(u_hi)) for d = X,Y,Z; b = flux/dt
// RN(1/x) where div_diag may use it (2^-500 < x < 2^500), else 0.
__device__ __forceinline__ double div_reciprocal(double x) { return (x > 0x1p-500 && x < 0x1p500) ? 1.0 / x : 0.0; }

// The flags of a cell's lower faces and, at the end of an axis, its upper wall.
__device__ __forceinline__ int face_checks(const GridDev& g, int i, int j, int k, const double lo[3],
                                           const double hi[3]) {
    const int p[3] = {i, j, k};
    int f = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (!isfinite(lo[a])) f |= VF_NONFINITE;
        if (p[a] == 0 && lo[a] != 0.0) f |= VF_WALL;
        if (p[a] + 1 == g.n[a]) {
            if (!isfinite(hi[a])) f |= VF_NONFINITE;
            if (hi[a] != 0.0) f |= VF_WALL;
        }
    }
    return f;
}

// CHECK: validate_velocity (src/operator.rs:850-875) on the way, every face by
// the cell it is the lower face of (the upper walls by the last cells): finite,
// wall-normal faces zero.
template <class T, bool CHECK = false>
__device__ __forceinline__ void build_rhs_body(const GridDev& g, const T* __restrict__ u, const T* __restrict__ v,
                                               const T* __restrict__ w, double dt, double* __restrict__ out,
                                               int* flags, Span sp) {
    // flux / dt correctly rounded through RN(1/dt) and one exact remainder
    const double rdt = div_reciprocal(dt);
    int local = 0;
    for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
        int i, j, k;
        cell_coords(g, c, i, j, k);
        const double lo[3] = {double(u[face_idx(g, 0, i, j, k)]), double(v[face_idx(g, 1, i, j, k)]),
                              double(w[face_idx(g, 2, i, j, k)])};
        const double hi[3] = {double(u[face_idx(g, 0, i + 1, j, k)]), double(v[face_idx(g, 1, i, j + 1, k)]),
                              double(w[face_idx(g, 2, i, j, k + 1)])};
        if (CHECK) local |= face_checks(g, i, j, k, lo, hi);
        double flux = 0.0;
        flux += g.area[0] * (lo[0] - hi[0]);
        flux += g.area[1] * (lo[1] - hi[1]);
        flux += g.area[2] * (lo[2] - hi[2]);
        double value = div_diag(flux, dt, rdt);
        if (!isfinite(value)) local |= VF_ARITH;
        out[c] = value;
    }
    if (local) atomicOr(flags, local);
}

// ------------------------------------------------------------ divergence
// f32 faces (src/operator.rs:543-567): ((dx/h0 + dy/h1) + dz/h2).
// f64 faces (src/operator.rs:711-742): value = 0; value += diff_d/h_d.
// The quotients are correctly rounded through RN(1/h_d) and one exact
// remainder (div_diag): the bits of the divisions.
template <class T>
__device__ __forceinline__ double cell_divergence(const GridDev& g, double xl, double xh, double yl,
                                                  double yh, double zl, double zh) {
    const double qx = div_diag(xh - xl, g.h[0], g.rh[0]);
    const double qy = div_diag(yh - yl, g.h[1], g.rh[1]);
    const double qz = div_diag(zh - zl, g.h[2], g.rh[2]);
    if (sizeof(T) == 4) {
        return qx + qy + qz;
    } else {
        double value = 0.0;
        value += qx;
        value += qy;
        value += qz;
        return value;
    }
}

// ------------------------------------------------------------ correction
// f32: u <- f32( f64(u) - (dt*accel_d)*(p_c - p_l) )   (src/operator.rs:651-662)
// f64: u <- u - dt*(accel_d*(p_c - p_l))               (src/operator.rs:767-775)
template <class T>
__device__ __forceinline__ T corrected(const GridDev& g, int a, T u, double pc, double pl, double dt,
                                       int& flag) {
    if (sizeof(T) == 4) {
        double value = double(u) - dt * g.accel[a] * (pc - pl);
        if (!(fabs(value) <= double(kF32Max))) flag |= VF_ARITH;  // not finite, or beyond f32
        return T(value);
    } else {
        double gradient = g.accel[a] * (pc - pl);
        double value = double(u) - dt * gradient;
        if (!isfinite(value)) flag |= VF_ARITH;
        return T(value);
    }
}

// Four consecutive values (16-byte aligned) as doubles, and back.
__device__ __forceinline__ void ld4(const float* p, float (&o)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
}
__device__ __forceinline__ void ld4(const double* p, double (&o)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    o[0] = a.x;
    o[1] = a.y;
    o[2] = b.x;
    o[3] = b.y;
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void st4(double* p, const double (&v)[4]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
}

// Lines of 32 quads of a plane marched along z: how many planes a line takes,
// so that a launch of `warps` warps has one line each where the box allows it.
__device__ __forceinline__ int march_planes(int segs, int n2, int warps) {
    return max(1, min(16, int((long long)segs * n2 / warps)));
}

// ------------------------------------------------------------ fused epilogue
// correct_divergence_body for rows of a multiple of 4 cells: a thread takes a
// quad of cells and marches along z, with 16-byte accesses and the corrected
// upper z faces and the pressure kept as the next plane's lower ones: 17
// corrections and 22 loads per quad and plane instead of 24 and 52. The
// operations on a value are the same. Bound by HBM (32 bytes a cell in f32) and
// issue. On a B200: 256^3 f32 308 us cell by cell, 171 in quads; 64 boxes of
// 32^3 to 96^3 0.98 and 0.41 ms. Other rows keep the cell-by-cell loop: their
// quads would not be aligned.
template <class T>
__device__ __forceinline__ void correct_divergence_quads(const GridDev& g, const double* __restrict__ p, double dt,
                                                         const T* __restrict__ iu, const T* __restrict__ iv,
                                                         const T* __restrict__ iw, T* __restrict__ ou,
                                                         T* __restrict__ ov, T* __restrict__ ow, T (&mxf)[3],
                                                         double& mxd, int& local, Span sp) {
    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2], sz = n0 * n1, quads = n0 >> 2;
    const int items = quads * n1, segs = (items + 31) >> 5;
    const int lane = threadIdx.x & 31, nw = sp.blocks * int(blockDim.x >> 5);
    const int kc = march_planes(segs, n2, nw), kcs = (n2 + kc - 1) / kc;
    auto seen = [&](int a, T v) {
        const T m = v < T(0) ? -v : v;
        mxf[a] = m > mxf[a] ? m : mxf[a];
    };
    for (int line = sp.block * int(blockDim.x >> 5) + int(threadIdx.x >> 5); line < segs * kcs; line += nw) {
        const int seg = line % segs, kb = (line / segs) * kc, ke = min(n2, kb + kc);
        const int it = seg * 32 + lane;
        if (it >= items) continue;
        const int j = it / quads, i0 = 4 * (it - j * quads);
        const bool ylo = j > 0, yhi = j + 1 < n1, xlo = i0 > 0, xhi = i0 + 4 < n0;
        int c = i0 + n0 * (j + n1 * kb);  // also the w face below the cell
        double pm[4], pc[4], pp[4];
        T wl[4];
        ld4(p + c, pc);
        ld4(iw + c, wl);
        if (kb > 0) {
            ld4(p + c - sz, pm);
#pragma unroll
            for (int e = 0; e < 4; ++e) wl[e] = corrected<T>(g, 2, wl[e], pc[e], pm[e], dt, local);
        }
        for (int k = kb; k < ke; ++k, c += sz) {
            const int fu = i0 + (n0 + 1) * (j + n1 * k), fv = i0 + n0 * (j + (n1 + 1) * k);
            T u[5], vl[4], vh[4], wh[4];
            double pl[4], ph[4];
            const bool up = k + 1 < n2;
#pragma unroll
            for (int e = 0; e < 5; ++e) u[e] = iu[fu + e];
            ld4(iv + fv, vl);
            ld4(iv + fv + n0, vh);
            ld4(iw + c + sz, wh);
            const double px = xlo ? p[c - 1] : 0.0, pxh = xhi ? p[c + 4] : 0.0;
            if (ylo) ld4(p + c - n0, pl);
            if (yhi) ld4(p + c + n0, ph);
            if (up) ld4(p + c + sz, pp);
            if (xlo) u[0] = corrected<T>(g, 0, u[0], pc[0], px, dt, local);
#pragma unroll
            for (int e = 1; e < 4; ++e) u[e] = corrected<T>(g, 0, u[e], pc[e], pc[e - 1], dt, local);
            if (xhi) u[4] = corrected<T>(g, 0, u[4], pxh, pc[3], dt, local);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (ylo) vl[e] = corrected<T>(g, 1, vl[e], pc[e], pl[e], dt, local);
                if (yhi) vh[e] = corrected<T>(g, 1, vh[e], ph[e], pc[e], dt, local);
                if (up) wh[e] = corrected<T>(g, 2, wh[e], pp[e], pc[e], dt, local);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ou[fu + e] = u[e];
                seen(0, u[e]);
                seen(1, vl[e]);
                seen(2, wl[e]);
                const double div = cell_divergence<T>(g, double(u[e]), double(u[e + 1]), double(vl[e]), double(vh[e]),
                                                      double(wl[e]), double(wh[e]));
                if (!isfinite(div)) local |= VF_ARITH;
                mxd = fmax(mxd, fabs(div));
            }
            st4(ov + fv, vl);
            st4(ow + c, wl);
            if (!xhi) {
                ou[fu + 4] = u[4];
                seen(0, u[4]);
            }
            if (!yhi) {
                st4(ov + fv + n0, vh);
#pragma unroll
                for (int e = 0; e < 4; ++e) seen(1, vh[e]);
            }
            if (!up) {
                st4(ow + c + sz, wh);
#pragma unroll
                for (int e = 0; e < 4; ++e) seen(2, wh[e]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                wl[e] = wh[e];
                pc[e] = pp[e];
            }
        }
    }
}

// One thread per cell: corrects the three lower faces the cell owns (writes
// them, wall faces copied through), recomputes its three upper faces to form
// the actual divergence of the stored values (actual_divergence_max,
// src/pressure.rs:330-342), and reduces max|div| and max|u_d| per axis
// (velocity_rate, src/simulation.rs:1415-1429).
template <class T>
__device__ __forceinline__ void correct_divergence_body(const GridDev& g, const double* __restrict__ p, double dt,
                                                        const T* __restrict__ iu, const T* __restrict__ iv,
                                                        const T* __restrict__ iw, T* __restrict__ ou,
                                                        T* __restrict__ ov, T* __restrict__ ow, Partials part,
                                                        double* out_scalars, int* flags, Span sp) {
    __shared__ BlockReduce<0, 4> sm;
    const T* in[3] = {iu, iv, iw};
    T* out[3] = {ou, ov, ow};
    const int s[3] = {1, g.n[0], g.n[0] * g.n[1]};
    double mx[4] = {0.0, 0.0, 0.0, 0.0};
    int local = 0;
    if ((g.n[0] & 3) == 0) {
        T mxf[3] = {T(0), T(0), T(0)};
        correct_divergence_quads<T>(g, p, dt, iu, iv, iw, ou, ov, ow, mxf, mx[0], local, sp);
#pragma unroll
        for (int a = 0; a < 3; ++a) mx[1 + a] = double(mxf[a]);
    } else
    for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
        int ijk[3];
        cell_coords(g, c, ijk[0], ijk[1], ijk[2]);
        double lo[3], hi[3];
        const double pc = p[c];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            int flo = face_idx(g, a, ijk[0], ijk[1], ijk[2]);
            int fhi = flo + (a == 0 ? 1 : (a == 1 ? g.fc[1][0] : g.fc[2][0] * g.fc[2][1]));
            T vlo = in[a][flo];
            if (ijk[a] > 0) vlo = corrected<T>(g, a, vlo, pc, p[c - s[a]], dt, local);
            out[a][flo] = vlo;
            T vhi = in[a][fhi];
            if (ijk[a] + 1 < g.n[a]) {
                vhi = corrected<T>(g, a, vhi, p[c + s[a]], pc, dt, local);
            } else {
                out[a][fhi] = vhi;
                mx[1 + a] = fmax(mx[1 + a], fabs(double(vhi)));
            }
            mx[1 + a] = fmax(mx[1 + a], fabs(double(vlo)));
            lo[a] = double(vlo);
            hi[a] = double(vhi);
        }
        double div = cell_divergence<T>(g, lo[0], hi[0], lo[1], hi[1], lo[2], hi[2]);
        if (!isfinite(div)) local |= VF_ARITH;
        mx[0] = fmax(mx[0], fabs(div));
    }
    if (local) atomicOr(flags, local);
    dd none[1];
    block_reduce<0, 4>(sm, none, mx);
    if (publish_and_check_last<0, 4>(part, sp.block, sp.blocks, none, mx)) {
        fold_partials<0, 4>(part, sp.blocks, sm, none, mx);
        if (threadIdx.x == 0)
            for (int q = 0; q < 4; ++q) out_scalars[q] = mx[q];
    }
}

}  // namespace rb200
