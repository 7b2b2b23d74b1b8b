// Device bodies of the semi-Lagrangian advection (src/advection.rs,
// src/sampling.rs), shared by the standalone kernels (advection.cu) and the
// resident carrier step (carrier.cu). One thread per face or cell; the
// arithmetic type R is double (the reference's f64 arithmetic, bit for bit on
// f32 or f64 storage) or float (the mixed-precision path).
#pragma once

#include <type_traits>

#include "internal.hpp"

namespace rb200 {

constexpr int ADV_THREADS = 256;


__device__ __forceinline__ double clampd(double x, double lo, double hi) {
    // f64::clamp: if x < min { min } then if x > max { max }.
    if (x < lo) x = lo;
    if (x > hi) x = hi;
    return x;
}

// (x - o_d) / h_d correctly rounded, through the reciprocal of h_d and one
// exact remainder (common.cuh) instead of a division: the same bits.
__device__ __forceinline__ double div_h(double r, const GridDev& g, int d) { return div_diag(r, g.h[d], g.rh[d]); }

// The integer value of an integer-valued fq in [0, 2^31).
__device__ __forceinline__ int cell_of(double fq) { return __double2loint(fq + 0x1p52); }

// The scaled coordinate (x - o_d) / h_d of a position in the box, of
// ScalarSampler::sample (src/sampling.rs:74-122; its clamp to the box is done
// where the position is formed). It depends on the position only, so the three
// components of a velocity sample share it.
__device__ __forceinline__ void scaled_position(const GridDev& g, const double pos[3], double xh[3]) {
#pragma unroll
    for (int d = 0; d < 3; ++d) xh[d] = div_h(pos[d] - g.o[d], g, d);
}

// The cell and fraction of a scaled coordinate on a lattice of top + 1 points:
// q = clamp(x, 0, top), its floor (q >= 0: the truncation, an integer below
// 2^31 read from the mantissa of fq + 2^52) and the rest.
struct Lattice {
    int lo, hi;
    double t;
};
__device__ __forceinline__ Lattice lattice(double x, int top) {
    const double q = clampd(x, 0.0, double(top));
    const double fq = trunc(q);
    Lattice l;
    l.lo = cell_of(fq);
    l.hi = min(l.lo + 1, top);
    l.t = q - fq;
    return l;
}

// ScalarSampler::sample (src/sampling.rs:74-122) from the lattice cells of the
// three axes: the eight corners weighted ((1 * w_x) * w_y) * w_z in the
// reference's z, y, x order, the sum clamped to the corners' range. 1 * w_x is
// w_x exactly, so the products w_x w_y are formed once per (x, y) pair; the
// values and every rounding are the reference's. Minimum and maximum are plain
// comparisons (in float for f32 values): the fields are finite.
template <class T>
__device__ __forceinline__ double sample_at(const T* __restrict__ values, const Lattice& X, const Lattice& Y,
                                            const Lattice& Z, int s1, int s2) {
    const double wx[2] = {1.0 - X.t, X.t};
    const double wy[2] = {1.0 - Y.t, Y.t};
    const double wz[2] = {1.0 - Z.t, Z.t};
    const double wxy[2][2] = {{wx[0] * wy[0], wx[1] * wy[0]}, {wx[0] * wy[1], wx[1] * wy[1]}};
    const int px[2] = {X.lo, X.hi};
    const int py[2] = {s1 * Y.lo, s1 * Y.hi};
    const int pz[2] = {s2 * Z.lo, s2 * Z.hi};
    double result = 0.0;
    T minimum{}, maximum{};
#pragma unroll
    for (int z = 0; z < 2; ++z)
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const double weight = wxy[y][x] * wz[z];
                const T value = __ldg(values + (px[x] + py[y] + pz[z]));
                if (x + y + z == 0) {
                    minimum = maximum = value;
                } else {
                    minimum = value < minimum ? value : minimum;
                    maximum = value > maximum ? value : maximum;
                }
                result += weight * double(value);
            }
    return clampd(result, double(minimum), double(maximum));
}

template <class T>
struct Faces {
    const T* f[3];
};

// The velocity at a position in the box. A component's lattice has n + 1
// points along its own axis and n along the others, where it is offset by 1/2:
// two lattice cells per axis serve the three components.
template <class T>
__device__ __forceinline__ void velocity_sample(const GridDev& g, const Faces<T>& vel, const double pos[3],
                                                double out[3]) {
    double xh[3];
    scaled_position(g, pos, xh);
    Lattice own[3], off[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        own[d] = lattice(xh[d], g.n[d]);
        off[d] = lattice(xh[d] - 0.5, g.n[d] - 1);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
        out[a] = sample_at<T>(vel.f[a], a == 0 ? own[0] : off[0], a == 1 ? own[1] : off[1], a == 2 ? own[2] : off[2],
                              g.fc[a][0], g.fc[a][0] * g.fc[a][1]);
}

// VelocitySampler::departure (src/sampling.rs:160-175). A value that is not
// finite is flagged (the step or call fails) and replaced, so that the samples
// stay in range.
__device__ __forceinline__ void departure(const GridDev& g, const double pos[3], const double vel[3], double dt,
                                          double out[3], int& flag) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double value = pos[d] - dt * vel[d];
        if (!isfinite(value)) {
            flag |= VF_ARITH;
            value = g.o[d];
        }
        out[d] = clampd(value, g.o[d], g.up[d]);
    }
}

// The second half of VelocitySampler::backtrace (src/sampling.rs:151-159),
// midpoint RK2, from the velocity at the start point.
template <class T>
__device__ __forceinline__ void backtrace_from(const GridDev& g, const Faces<T>& vel, const double pos[3],
                                               const double initial[3], double dt, double out[3], int& flag) {
    double mid[3], v1[3];
    departure(g, pos, initial, 0.5 * dt, mid, flag);
    velocity_sample<T>(g, vel, mid, v1);
    departure(g, pos, v1, dt, out, flag);
}

// VelocitySampler::backtrace (src/sampling.rs:151-159): midpoint RK2.
template <class T>
__device__ __forceinline__ void backtrace(const GridDev& g, const Faces<T>& vel, const double pos[3], double dt,
                                          double out[3], int& flag) {
    double initial[3];
    velocity_sample<T>(g, vel, pos, initial);
    backtrace_from<T>(g, vel, pos, initial, dt, out, flag);
}

// The velocity at the centre of face p of axis a. There the sampler's
// fractions are 0 or 1/2 (exactly so where the grid's centres are exact; the
// FP32 path takes the exact face position in any case), so the face's own
// component is its value and each other component c is the mean of the four
// c-faces around it in the a-c plane: the corners of weight 1/4, summed from 0
// in the sampler's z, y, x order. The corners of weight 0 add only zeros,
// which change no sum that starts from +0, and the mean lies within the
// corners' range, so the result has the bits of the eight-corner sample, with
// four loads per component instead of eight and none for the own one.
template <class T, class R>
__device__ __forceinline__ void face_velocity(const GridDev& g, const Faces<T>& vel, const int p[3], int a, R out[3],
                                              int& flag) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int s1 = g.fc[c][0], s2 = g.fc[c][0] * g.fc[c][1];
        const int at = p[0] + s1 * p[1] + s2 * p[2];
        const T* f = vel.f[c];
        if (c == a) {
            out[c] = R(0) + R(f[at]);
            if (!isfinite(out[c])) flag |= VF_ARITH;
            continue;
        }
        // c-faces: the corners are p_a - 1 and p_a along a, p_c and p_c + 1
        // along c; the higher of the two axes is the outer one of the sum
        auto stride = [&](int d) { return d == 0 ? 1 : (d == 1 ? s1 : s2); };
        const int su = stride(min(a, c)), sv = stride(max(a, c));
        const int base = at - stride(a);
        const R w = R(0.25);
        R r = R(0);
        r += w * R(f[base]);
        r += w * R(f[base + su]);
        r += w * R(f[base + sv]);
        r += w * R(f[base + su + sv]);
        if (!isfinite(r)) flag |= VF_ARITH;
        out[c] = r;
    }
}

// ------------------------------------------------------------ FP32 arithmetic
// The mixed-precision path of the same scheme, in scaled coordinates
// (x - o) / h throughout: a face or cell centre is p or p + 1/2 exactly, the
// departure point x - (dt / h) v is one multiply-add per axis, and no division,
// origin or second clamp is needed. A lattice is offset by 0 or 1/2 along each
// axis, so a position has two (cell, fraction) pairs per axis, shared by the
// three velocity components. Interpolation is nested (1 - t) a + t b in
// multiply-adds; the stored value is clamped to its corners' range, as the
// reference's sample is. Bound by L1 gathers (40 per face) and issue, about
// 350 instructions a face where the FP64-style arithmetic in float spent 1270: at
// 256^3 1780 us before, 777 now for the velocity (issue slots 73 % busy), 748
// and 300 for the tracer.
struct LatticeF {
    float top, last;  // dims - 1, max(dims - 2, 0)
};

// The cell below q and the fraction within it, q clamped to [0, top]. The cell
// is q - 1/2 rounded to nearest (an exact integer may give t = 1 in the cell
// below it: the same value) and at most `last`, so that its upper neighbour
// exists. BIG: axes beyond the reach of the rounding constant.
template <bool BIG>
__device__ __forceinline__ void lattice_cell(float x, const LatticeF& l, int& lo, float& t) {
    const float q = fminf(fmaxf(x, 0.0f), l.top);
    if (BIG) {
        const float f = fminf(floorf(q), l.last);
        lo = int(f);
        t = q - f;
    } else {
        constexpr float M = 12582912.0f;  // 1.5 2^23
        const float f = fminf(((q - 0.5f) + M) - M, l.last);
        lo = __float_as_int(f + M) - 0x4B400000;
        t = q - f;
    }
}

__device__ __forceinline__ float lerp_f(float t, float a, float b) { return fmaf(t, b, fmaf(-t, a, a)); }

// Trilinear value at cell offset `at` of a lattice with strides s1, s2; sx, sy,
// sz: the upper neighbours' offsets (0 along a one-point axis). CLAMP: to the
// range of the eight corners.
template <class T, bool CLAMP>
__device__ __forceinline__ float trilinear(const T* __restrict__ f, int at, int sx, int sy, int sz, float tx, float ty,
                                           float tz) {
    const T* p0 = f + at;
    const T* p1 = p0 + sy;
    const T* p2 = p0 + sz;
    const T* p3 = p2 + sy;
    const float a0 = float(__ldg(p0)), b0 = float(__ldg(p0 + sx));
    const float a1 = float(__ldg(p1)), b1 = float(__ldg(p1 + sx));
    const float a2 = float(__ldg(p2)), b2 = float(__ldg(p2 + sx));
    const float a3 = float(__ldg(p3)), b3 = float(__ldg(p3 + sx));
    float r = lerp_f(tz, lerp_f(ty, lerp_f(tx, a0, b0), lerp_f(tx, a1, b1)),
                     lerp_f(ty, lerp_f(tx, a2, b2), lerp_f(tx, a3, b3)));
    if (CLAMP) {
        const float lo = fminf(fminf(fminf(a0, b0), fminf(a1, b1)), fminf(fminf(a2, b2), fminf(a3, b3)));
        const float hi = fmaxf(fmaxf(fmaxf(a0, b0), fmaxf(a1, b1)), fmaxf(fmaxf(a2, b2), fmaxf(a3, b3)));
        // not through fmin/fmax: a NaN stays one
        if (r < lo) r = lo;
        if (r > hi) r = hi;
    }
    return r;
}

// Strides and lattices of the box, uniform over the launch.
struct BoxF {
    LatticeF face[3], cell[3];  // along axis d: the lattice of axis-d faces, and of every other component
    int up[3];                  // offset factor of the upper neighbour (0 along a one-cell axis)
};
__device__ __forceinline__ BoxF box_f(const GridDev& g) {
    BoxF b;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        b.face[d] = LatticeF{float(g.n[d]), float(g.n[d] - 1)};
        b.cell[d] = LatticeF{float(g.n[d] - 1), float(max(g.n[d] - 2, 0))};
        b.up[d] = g.n[d] > 1 ? 1 : 0;
    }
    return b;
}

// The velocity at scaled position x.
template <class T, bool BIG>
__device__ __forceinline__ void velocity_f(const GridDev& g, const BoxF& b, const Faces<T>& vel, const float x[3],
                                           float out[3]) {
    int lf[3], lc[3];
    float tf[3], tc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        lattice_cell<BIG>(x[d], b.face[d], lf[d], tf[d]);
        lattice_cell<BIG>(x[d] - 0.5f, b.cell[d], lc[d], tc[d]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int s1 = g.fc[a][0], s2 = g.fc[a][0] * g.fc[a][1];
        const int lx = a == 0 ? lf[0] : lc[0], ly = a == 1 ? lf[1] : lc[1], lz = a == 2 ? lf[2] : lc[2];
        const int ux = a == 0 ? 1 : b.up[0], uy = a == 1 ? 1 : b.up[1], uz = a == 2 ? 1 : b.up[2];
        out[a] = trilinear<T, false>(vel.f[a], lx + s1 * ly + s2 * lz, ux, s1 * uy, s2 * uz, a == 0 ? tf[0] : tc[0],
                                     a == 1 ? tf[1] : tc[1], a == 2 ? tf[2] : tc[2]);
    }
}

// The departure point (scaled) of the scaled position x0 with velocity v0
// there: midpoint RK2. sc: dt / h per axis.
template <class T, bool BIG>
__device__ __forceinline__ void departure_f(const GridDev& g, const BoxF& b, const Faces<T>& vel, const float x0[3],
                                            const float v0[3], const float sc[3], float x[3], int& flag) {
    float mid[3], v1[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) mid[d] = fmaf(-0.5f * sc[d], v0[d], x0[d]);
    if (!isfinite(mid[0] + mid[1] + mid[2])) flag |= VF_ARITH;
    // the sampler clamps to the lattices, which covers the clamp to the box
    velocity_f<T, BIG>(g, b, vel, mid, v1);
#pragma unroll
    for (int d = 0; d < 3; ++d) x[d] = fmaf(-sc[d], v1[d], x0[d]);
    if (!isfinite(x[0] + x[1] + x[2])) flag |= VF_ARITH;
}

// dt / h per axis, rounded once from double, by three threads of the block.
__device__ __forceinline__ void step_scale(const GridDev& g, double dt, float sc[3]) {
    __shared__ float s[3];
    if (threadIdx.x < 3) s[threadIdx.x] = float(dt / g.h[threadIdx.x]);
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 3; ++d) sc[d] = s[d];
}

// The lower faces of cell (p0, p1, p2) along axis A.
template <class T, bool BIG, int A>
__device__ __forceinline__ void advect_face_f(const GridDev& g, const BoxF& b, const Faces<T>& vel, const int p[3],
                                              const float sc[3], double dt, T* __restrict__ out,
                                              const float* __restrict__ tracer, double gb, int& flag) {
    const int s1 = g.fc[A][0], s2 = g.fc[A][0] * g.fc[A][1];
    const int at = p[0] + s1 * p[1] + s2 * p[2];
    // the upper wall belongs to the last cell
    if (p[A] + 1 == g.n[A]) out[at + (A == 0 ? 1 : A == 1 ? s1 : s2)] = T(0);
    if (p[A] == 0) {
        out[at] = T(0);
        return;
    }
    float v[3];
    face_velocity<T, float>(g, vel, p, A, v, flag);
    float x0[3], x[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) x0[d] = float(p[d]) + (d == A ? 0.0f : 0.5f);
    departure_f<T, BIG>(g, b, vel, x0, v, sc, x, flag);
    int lo[3];
    float t[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) lattice_cell<BIG>(d == A ? x[d] : x[d] - 0.5f, d == A ? b.face[d] : b.cell[d], lo[d], t[d]);
    const float r = trilinear<T, true>(vel.f[A], lo[0] + s1 * lo[1] + s2 * lo[2], A == 0 ? 1 : b.up[0],
                                       s1 * (A == 1 ? 1 : b.up[1]), s2 * (A == 2 ? 1 : b.up[2]), t[0], t[1], t[2]);
    if (!isfinite(r)) flag |= VF_ARITH;
    T value = T(r);
    if (A == 1 && tracer != nullptr && gb != 0.0) {
        // Buoyancy hook (new): interior Y face, after advection, before pressure.
        const int below = cell_idx(g, p[0], p[1] - 1, p[2]), above = cell_idx(g, p[0], p[1], p[2]);
        const double c = 0.5 * (double(tracer[below]) + double(tracer[above]));
        const double forced = double(value) + dt * (gb * c);
        if (!isfinite(forced)) flag |= VF_ARITH;
        value = T(forced);
    }
    out[at] = value;
}

template <class T, bool BIG>
__device__ __forceinline__ void advect_velocity_cells_f(const GridDev& g, const Faces<T>& vel, double dt,
                                                        const float sc[3], T* ou, T* ov, T* ow,
                                                        const float* __restrict__ tracer, double gb, int* flags,
                                                        Span sp) {
    const BoxF b = box_f(g);
    int local = 0;
    for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
        int p[3];
        cell_coords(g, c, p[0], p[1], p[2]);
        advect_face_f<T, BIG, 0>(g, b, vel, p, sc, dt, ou, tracer, gb, local);
        advect_face_f<T, BIG, 1>(g, b, vel, p, sc, dt, ov, tracer, gb, local);
        advect_face_f<T, BIG, 2>(g, b, vel, p, sc, dt, ow, tracer, gb, local);
    }
    if (local) atomicOr(flags, local);
}

template <class T, bool BIG>
__device__ __forceinline__ void advect_tracer_cells_f(const GridDev& g, const float* __restrict__ old,
                                                      const Faces<T>& vel, const float sc[3], float* __restrict__ out,
                                                      int* flags, Span sp) {
    const BoxF b = box_f(g);
    const int s1 = g.n[0], s2 = g.n[0] * g.n[1];
    int local = 0;
    for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
        int p[3];
        cell_coords(g, c, p[0], p[1], p[2]);
        float x0[3], v[3], x[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            // at a cell centre a component is the mean of the cell's two faces
            const int f1 = g.fc[d][0], f2 = g.fc[d][0] * g.fc[d][1];
            const T* f = vel.f[d] + (p[0] + f1 * p[1] + f2 * p[2]);
            v[d] = 0.5f * float(f[0]) + 0.5f * float(f[d == 0 ? 1 : d == 1 ? f1 : f2]);
            x0[d] = float(p[d]) + 0.5f;
        }
        departure_f<T, BIG>(g, b, vel, x0, v, sc, x, local);
        int lo[3];
        float t[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) lattice_cell<BIG>(x[d] - 0.5f, b.cell[d], lo[d], t[d]);
        const float r = trilinear<float, true>(old, lo[0] + s1 * lo[1] + s2 * lo[2], b.up[0], s1 * b.up[1],
                                               s2 * b.up[2], t[0], t[1], t[2]);
        if (!isfinite(r)) local |= VF_ARITH;
        out[c] = r;
    }
    if (local) atomicOr(flags, local);
}

// Axes that the rounding constant of lattice_cell does not reach.
__device__ __forceinline__ bool big_axes(const GridDev& g) { return max(max(g.n[0], g.n[1]), g.n[2]) >= (1 << 21); }

// ------------------------------------------------------------ FP64 arithmetic
// The lower face of cell p along axis A (and the upper wall of the last cell).
template <class T, int A>
__device__ __forceinline__ void advect_face_d(const GridDev& g, const Faces<T>& vel, const int p[3], double dt,
                                              T* __restrict__ out, const float* __restrict__ tracer, double gb,
                                              int& flag) {
    const int s1 = g.fc[A][0], s2 = g.fc[A][0] * g.fc[A][1];
    const int f = p[0] + s1 * p[1] + s2 * p[2];
    if (p[A] + 1 == g.n[A]) out[f + (A == 0 ? 1 : A == 1 ? s1 : s2)] = T(0);
    if (p[A] == 0) {
        out[f] = T(0);
        return;
    }
    double pos[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) pos[d] = g.o[d] + (double(p[d]) + (d == A ? 0.0 : 0.5)) * g.h[d];
    double dep[3], xh[3];
    if (g.exact_centres) {
        double initial[3];
        face_velocity<T, double>(g, vel, p, A, initial, flag);
        backtrace_from<T>(g, vel, pos, initial, dt, dep, flag);
    } else {
        backtrace<T>(g, vel, pos, dt, dep, flag);
    }
    scaled_position(g, dep, xh);
    Lattice at[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) at[d] = lattice(d == A ? xh[d] : xh[d] - 0.5, d == A ? g.n[d] : g.n[d] - 1);
    const double sampled = sample_at<T>(vel.f[A], at[0], at[1], at[2], s1, s2);
    if (!isfinite(sampled)) flag |= VF_ARITH;
    T value = T(sampled);
    if (A == 1 && tracer != nullptr && gb != 0.0) {
        // Buoyancy hook (new): interior Y face, after advection, before pressure.
        const int below = cell_idx(g, p[0], p[1] - 1, p[2]), above = cell_idx(g, p[0], p[1], p[2]);
        const double c = 0.5 * (double(tracer[below]) + double(tracer[above]));
        const double forced = double(value) + dt * (gb * c);
        if (!isfinite(forced)) flag |= VF_ARITH;
        value = T(forced);
    }
    out[f] = value;
}

// advect_velocity (src/advection.rs:28-68): wall-normal faces are exactly 0,
// every other face samples its own component at the RK2 departure point. A
// thread advects the lower faces of a cell, axis by axis, so that an axis is a
// constant in the code (one face a thread, of whichever axis, kept its
// per-axis values in local memory). Bound by issue and the FP64 pipe, about 320
// operations a face: 128^3 in f64 227 us (108 us of FP64 issue; 417 us with nine
// lattice cells a sample instead of six, clamps and finite tests repeated per
// component, and fmin and fmax).
template <class T, class R>
__device__ __forceinline__ void advect_velocity_body(const GridDev& g, const Faces<T>& vel, double dt, T* ou, T* ov,
                                                     T* ow, const float* __restrict__ tracer, double gb, int* flags,
                                                     Span sp) {
    if constexpr (std::is_same<R, float>::value) {
        float sc[3];
        step_scale(g, dt, sc);
        if (big_axes(g))
            advect_velocity_cells_f<T, true>(g, vel, dt, sc, ou, ov, ow, tracer, gb, flags, sp);
        else
            advect_velocity_cells_f<T, false>(g, vel, dt, sc, ou, ov, ow, tracer, gb, flags, sp);
    } else {
        int local = 0;
        for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
            int p[3];
            cell_coords(g, c, p[0], p[1], p[2]);
            advect_face_d<T, 0>(g, vel, p, dt, ou, tracer, gb, local);
            advect_face_d<T, 1>(g, vel, p, dt, ov, tracer, gb, local);
            advect_face_d<T, 2>(g, vel, p, dt, ow, tracer, gb, local);
        }
        if (local) atomicOr(flags, local);
    }
}

// advect_tracer (src/advection.rs:72-102), evaluated densely; the reference's
// zero-support skip produces the same bits (tests/advection_contract.rs:7-41).
template <class T, class R>
__device__ __forceinline__ void advect_tracer_body(const GridDev& g, const float* __restrict__ old,
                                                   const Faces<T>& vel, double dt, float* __restrict__ out,
                                                   int* flags, Span sp) {
    if constexpr (std::is_same<R, float>::value) {
        float sc[3];
        step_scale(g, dt, sc);
        if (big_axes(g))
            advect_tracer_cells_f<T, true>(g, old, vel, sc, out, flags, sp);
        else
            advect_tracer_cells_f<T, false>(g, old, vel, sc, out, flags, sp);
        return;
    }
    int local = 0;
    for (int c = sp.block * blockDim.x + threadIdx.x; c < g.cells; c += sp.blocks * blockDim.x) {
        int p[3];
        cell_coords(g, c, p[0], p[1], p[2]);
        double pos[3], dep[3], xh[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) pos[d] = g.o[d] + (double(p[d]) + 0.5) * g.h[d];
        backtrace<T>(g, vel, pos, dt, dep, local);
        scaled_position(g, dep, xh);
        Lattice at[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) at[d] = lattice(xh[d] - 0.5, g.n[d] - 1);
        const double sampled = sample_at<float>(old, at[0], at[1], at[2], g.n[0], g.n[0] * g.n[1]);
        if (!isfinite(sampled)) local |= VF_ARITH;
        out[c] = float(sampled);
    }
    if (local) atomicOr(flags, local);
}

}  // namespace rb200
