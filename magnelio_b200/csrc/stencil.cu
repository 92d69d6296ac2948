// Leapfrog curl updates with the CFS-PML psi recursion fused in: the direct
// form, 16 bytes of cells per thread and no march (one cell per thread on small
// meshes).
//
//   E^{n+1} = aE * E^n + bE * (C^T h)      then, on CPML slabs,
//             E += +-bE * (ck * dH + psi_E),  psi_E = air * (b psi_E + c dH)
//   H^{n+3/2} = aH * H - bH * (C e)        then, on CPML slabs,
//             H += +-bH * (ck * dE + psi_H),  psi_H = air * (b psi_H + c dE)
//
// Reference semantics: the fused Numba/CUDA kernels
// (src/magnelio/_operators/numba_kernels.py:36-127, :281-434) followed by
// CPMLBoundary.update_E / update_H (src/magnelio/boundaries/cpml.py:343-516).
// The in-thread curl order is the reference's: curl = +H_a - H_a' - H_b + H_b'.
//
// Thread mapping: a thread owns 16 bytes of consecutive k (4 float, 2 double
// cells) of one field set; threads run along the flattened rows of one i plane
// (the padded row pitch is a multiple of 8), blockIdx.y is the plane (np planes
// per thread), threadIdx.y the field set: the sets of a cell share its
// coefficients through the L1.  Nothing is staged and no thread waits for
// another, so meshes whose state stays in the L2 (up to about 1.5 M cells in
// float32: latency and instructions bound them, not HBM) keep the whole chip
// busy where a march along i (the stream, tile and slab forms) leaves most of
// it idle; large meshes stream at the HBM rate (256^3 without CPML, float32:
// 262 us per step, 96 B per cell at 0.95 of the measured copy rate).  Cells
// per second, direct / stream / slab step's lists: 39 / 14.5 / 17.0 G at 0.9 M
// cells, 49 / 28 / 33.7 G at 5.8 M, 57.7 / 41.0 / 46.7 G at 105 M (CPML all
// round); four field sets of 5.8 M cells 55 / 37 / 44 G.
#include "direct.cuh"
#include "lumped.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

namespace fitb {

namespace {

constexpr int kDirectThreads = 128;

// V consecutive cells of one array.
template <typename T, int V>
struct Vec {
    T v[V];
};

template <int V>
__device__ __forceinline__ Vec<float, V> ldv(const float* p) {
    static_assert(V == 1 || V == 4, "16 bytes or one cell");
    if constexpr (V == 1) return {{*p}};
    if constexpr (V == 4) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        return {{q.x, q.y, q.z, q.w}};
    }
}
template <int V>
__device__ __forceinline__ Vec<double, V> ldv(const double* p) {
    static_assert(V == 1 || V == 2, "16 bytes or one cell");
    if constexpr (V == 1) return {{*p}};
    if constexpr (V == 2) {
        const double2 q = *reinterpret_cast<const double2*>(p);
        return {{q.x, q.y}};
    }
}
template <int V>
__device__ __forceinline__ void stv(float* p, const Vec<float, V>& a) {
    if constexpr (V == 1) *p = a.v[0];
    if constexpr (V == 4) *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
template <int V>
__device__ __forceinline__ void stv(double* p, const Vec<double, V>& a) {
    if constexpr (V == 1) *p = a.v[0];
    if constexpr (V == 2) *reinterpret_cast<double2*>(p) = make_double2(a.v[0], a.v[1]);
}

template <typename T, int CK>
__device__ __forceinline__ T decode16(unsigned short u, float scale) {
    if constexpr (CK == kCoefF16) return (T)__half2float(__ushort_as_half(u)) * (T)scale;
    return (T)__bfloat162float(__ushort_as_bfloat16(u)) * (T)scale;
}

// Entry o of one stored coefficient array.
template <typename T, int CK>
__device__ __forceinline__ T coef_at(const T* __restrict__ a, const unsigned short* __restrict__ q, float scale,
                                     long long o) {
    if constexpr (CK == kCoefNative) return __ldg(a + o);
    return decode16<T, CK>(__ldg(q + o), scale);
}

template <typename T, int V, int CK>
__device__ __forceinline__ Vec<T, V> coef_vec(const T* a, const unsigned short* q, float scale, long long o) {
    if constexpr (CK == kCoefNative) {
        return ldv<V>(a + o);
    } else {
        Vec<T, V> r;
        unsigned short u[V];
        if constexpr (V == 4) {
            const ushort4 w = *reinterpret_cast<const ushort4*>(q + o);
            u[0] = w.x, u[1] = w.y, u[2] = w.z, u[3] = w.w;
        } else if constexpr (V == 2) {
            const ushort2 w = *reinterpret_cast<const ushort2*>(q + o);
            u[0] = w.x, u[1] = w.y;
        } else {
            u[0] = q[o];
        }
#pragma unroll
        for (int c = 0; c < V; ++c) r.v[c] = decode16<T, CK>(u[c], scale);
        return r;
    }
}

// The update coefficients of a thread's cells and side (0: E, 1: H).  UA:
// alpha is one wherever beta is not zero and a0 elsewhere, so it is not read.
template <typename T, int V, int CK, bool UA>
__device__ __forceinline__ void load_cell_coef(const StencilArgs<T>& p, int side, int o, Vec<T, V> a[3],
                                               Vec<T, V> b[3]) {
    const T* A = side == 0 ? p.aE : p.aH;
    const T* Bp = side == 0 ? p.bE : p.bH;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        b[c] = coef_vec<T, V, CK>(Bp, p.cq[2 * side + 1], p.cs[8 * side + 4 + c], c * p.g.vol + o);
        if constexpr (!UA) a[c] = coef_vec<T, V, CK>(A, p.cq[2 * side], p.cs[8 * side + c], c * p.g.vol + o);
    }
}

template <typename T, int V, bool UA>
__device__ __forceinline__ T alpha_of(const Vec<T, V>& a, T b, float a0, int c) {
    if constexpr (UA) return b != T(0) ? T(1) : (T)a0;
    return a.v[c];
}

// The roundings of the update, spelled out: which product of a sum of two the
// compiler contracts into the FMA depends on the code around it.  These are
// the ones the stream kernels compile to (Ex: fma(beta, curl, alpha E), the
// other components fma(alpha, f, +-beta curl)), so a cell at a time and 16 bytes
// give the same bits, and the stream kernels' bits wherever no two slabs of an
// axis overlap (cell_psi takes all near faces before the far ones there).
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }

// CPML of one axis at a thread's cells: psi <- air (b psi + c d) and the
// corrections f1 += s1 b1 (ck d1 + psi1), f2 += s2 b2 (ck d2 + psi2) with
// (s1, s2) = (-1, +1) when NEG1, else (+1, -1).  The axis is a template
// argument and its two faces are picked by selects: a loop over the face
// table with the axis read from it cost 436 instructions per warp on a box
// with CPML all round.  SIDE: -1 picks the face by the coordinate; 0 and 1
// are the two faces of an axis whose slabs overlap.
template <typename T, int V, int A, int SIDE, bool NEG1>
__device__ __forceinline__ void axis_psi(const AxisSlabs& x, int b, int i, int j, int k, const T d1[V], const T d2[V],
                                         const Vec<T, V>& b1, const Vec<T, V>& b2, Vec<T, V>& f1, Vec<T, V>& f2) {
    // V entries with one layer (x, y), or cell by cell along z: there
    // the psi loads of all the cells go out before the first is used
    constexpr int NC = A == 2 ? V : 1, W = A == 2 ? 1 : V;
    Vec<T, W> p1[NC], p2[NC];
    bool on[NC];
    bool any = false;
#pragma unroll
    for (int m = 0; m < NC; ++m) {
        const int c = A == 0 ? i : (A == 1 ? j : k + m);
        const bool hi = SIDE < 0 ? c >= x.lo1 : SIDE == 1;
        const int l = hi ? c - x.lo1 : c, n = hi ? x.n[1] : x.n[0];
        on[m] = (unsigned)l < (unsigned)n;
        any = any || on[m];
        if (!on[m]) continue;
        const int s = (A == 0 ? l : i) * (hi ? x.s0[1] : x.s0[0]) + (A == 1 ? l : j) * (hi ? x.s1[1] : x.s1[0]) +
                      (A == 2 ? l : k);
        const T* q = static_cast<const T*>(hi ? x.psi[1] : x.psi[0]) +
                     ((size_t)(unsigned)b * (hi ? x.set[1] : x.set[0]) + s);
        p1[m] = ldv<W>(q);
        p2[m] = ldv<W>(q + (hi ? x.slab[1] : x.slab[0]));
    }
    if (!any) return;
#pragma unroll
    for (int m = 0; m < NC; ++m) {
        if (!on[m]) continue;
        const int c = A == 0 ? i : (A == 1 ? j : k + m);
        const bool hi = SIDE < 0 ? c >= x.lo1 : SIDE == 1;
        const int l = hi ? c - x.lo1 : c, n = hi ? x.n[1] : x.n[0];
        const int s = (A == 0 ? l : i) * (hi ? x.s0[1] : x.s0[0]) + (A == 1 ? l : j) * (hi ? x.s1[1] : x.s1[0]) +
                      (A == 2 ? l : k);
        const T* __restrict__ t = static_cast<const T*>(hi ? x.bcc[1] : x.bcc[0]) + l;
        const T cb = __ldg(t), cc = __ldg(t + n), ck = __ldg(t + 2 * n);
        const unsigned slab = hi ? x.slab[1] : x.slab[0];
        const unsigned char* air = hi ? x.air[1] : x.air[0];
#pragma unroll
        for (int w = 0; w < W; ++w) {
            p1[m].v[w] = fma_(cc, d1[m + w], mul_(p1[m].v[w], cb));
            p2[m].v[w] = fma_(cc, d2[m + w], mul_(p2[m].v[w], cb));
            if (air) {
                if (!air[s + w]) p1[m].v[w] = T(0);
                if (!air[slab + s + w]) p2[m].v[w] = T(0);
            }
            const T c1 = fma_(ck, d1[m + w], p1[m].v[w]), c2 = fma_(ck, d2[m + w], p2[m].v[w]);
            f1.v[m + w] = fma_(NEG1 ? -b1.v[m + w] : b1.v[m + w], c1, f1.v[m + w]);
            f2.v[m + w] = fma_(NEG1 ? b2.v[m + w] : -b2.v[m + w], c2, f2.v[m + w]);
        }
        T* out = static_cast<T*>(hi ? x.psi_out[1] : x.psi_out[0]) +
                 ((size_t)(unsigned)b * (hi ? x.set[1] : x.set[0]) + s);
        stv<W>(out, p1[m]);
        stv<W>(out + slab, p2[m]);
    }
}

// The CPML corrections of a thread's cells, x, y, z faces in that order.
// E side: Ey += x, Ez -= x; Ex -= y, Ez += y; Ex += z, Ey -= z; the H side the
// other way round.  dab: difference along axis a of component b; zs: the
// thread's cells may lie in a z slab (uniform per warp).
template <typename T, int V, int SIDE, bool E>
__device__ __forceinline__ void cell_psi(const AxisSlabs ax[3], int b, int i, int j, int k, bool zs,
                                         const Vec<T, V> bc[3], const T dxz[V], const T dxy[V], const T dyz[V],
                                         const T dyx[V], const T dzy[V], const T dzx[V], Vec<T, V>& fx, Vec<T, V>& fy,
                                         Vec<T, V>& fz) {
    axis_psi<T, V, 0, SIDE, !E>(ax[0], b, i, j, k, dxz, dxy, bc[1], bc[2], fy, fz);
    axis_psi<T, V, 1, SIDE, E>(ax[1], b, i, j, k, dyz, dyx, bc[0], bc[2], fx, fz);
    if (zs) axis_psi<T, V, 2, SIDE, !E>(ax[2], b, i, j, k, dzy, dzx, bc[0], bc[1], fx, fy);
}

// Row pads beyond k = nz stay +0 whatever their neighbours hold.
template <typename T, int V>
__device__ __forceinline__ void keep_pad(Vec<T, V>& f, int k, int nz) {
#pragma unroll
    for (int c = 1; c < V; ++c)
        if (k + c > nz) f.v[c] = T(0);
}

// Row j, first cell k and z-slab flag of thread t of a plane: the vectors
// clear of the z slabs of every row first, then (from a warp boundary on) the
// others, so that only warps full of z-slab cells run that part.  False: no
// cell.
__device__ __forceinline__ bool direct_cell(const DirectArgs& d, int ny, unsigned t, int V, int& j, int& k, bool& zs) {
    zs = t >= d.mid_threads;
    if (!zs) {
        j = (int)(__umulhi(2 * t, d.mid_div.m) >> d.mid_div.s);
        k = (d.n_low + (int)t - j * d.n_mid) * V;
    } else {
        if (d.n_edge == 0) return false;  // the last block's spare threads
        t -= d.mid_threads;
        j = (int)(__umulhi(2 * t, d.edge_div.m) >> d.edge_div.s);
        const int e = (int)t - j * d.n_edge;
        k = (e < d.n_low ? e : e + d.n_mid) * V;
    }
    return j <= ny;
}

// Resident CTAs per SM asked of the compiler: 128 registers for the vector
// form, 64 (float) and 85 (double) for one cell per thread.  Measured with the
// vector form at 97 x 104 x 89 / 251 x 187 x 233 / 81 x 75 x 90 float64 (us
// per step): 4 CTAs of 128 threads 31.7 / 215 / 28.7, 5 of 128 (102
// registers) 32.6 / 216 / 31.0, 2 of 256 33.6 / 224 / 29.9, 3 of 256 (85
// registers, spills) 36.3 / 228 / 35.3.
template <typename T, int V>
constexpr int direct_min_ctas() {
    return V == 1 ? (sizeof(T) == 4 ? 8 : 6) : 4;
}

// E_new of a thread's cells at plane i of field set b.  hz_im, hy_im: H of
// plane i - 1; on return H of plane i.  ES: the roundings of the slab step (all
// components fma(beta, curl, alpha E)) instead of the stream kernels'.
template <typename T, int V, int CK, bool UA, bool OV, bool ES>
__device__ __forceinline__ void cell_E(const StencilArgs<T>& p, const DirectArgs& d, const T* E, const T* H, T* Eo,
                                       int b, int i, int j, int k, int o, bool zs, Vec<T, V>& hz_im,
                                       Vec<T, V>& hy_im) {
    const Geom& g = p.g;
    const long long vol = g.vol;
    const int sj = (int)g.sj;
    Vec<T, V> a[3], bc[3];
    load_cell_coef<T, V, CK, UA>(p, 0, o, a, bc);
    const Vec<T, V> hx = ldv<V>(H + o), hy = ldv<V>(H + vol + o), hz = ldv<V>(H + 2 * vol + o);
    const Vec<T, V> hz_jm = ldv<V>(H + 2 * vol + o - sj), hx_jm = ldv<V>(H + o - sj);
    const T hy_km = H[vol + o - 1], hx_km = H[o - 1];
    Vec<T, V> ex = ldv<V>(E + o), ey = ldv<V>(E + vol + o), ez = ldv<V>(E + 2 * vol + o);
    T dxz[V], dxy[V], dyz[V], dyx[V], dzy[V], dzx[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const T hyk = c ? hy.v[c - (c > 0)] : hy_km, hxk = c ? hx.v[c - (c > 0)] : hx_km;
        // Same accumulation order as the reference kernels.
        const T cx = ((hz.v[c] - hz_jm.v[c]) - hy.v[c]) + hyk;
        const T cy = ((hx.v[c] - hxk) - hz.v[c]) + hz_im.v[c];
        const T cz = ((hy.v[c] - hy_im.v[c]) - hx.v[c]) + hx_jm.v[c];
        const T ax = alpha_of<T, V, UA>(a[0], bc[0].v[c], p.a0[0], c);
        const T ay = alpha_of<T, V, UA>(a[1], bc[1].v[c], p.a0[0], c);
        const T az = alpha_of<T, V, UA>(a[2], bc[2].v[c], p.a0[0], c);
        ex.v[c] = fma_(bc[0].v[c], cx, mul_(ax, ex.v[c]));
        ey.v[c] = ES ? fma_(bc[1].v[c], cy, mul_(ay, ey.v[c])) : fma_(ay, ey.v[c], mul_(bc[1].v[c], cy));
        ez.v[c] = ES ? fma_(bc[2].v[c], cz, mul_(az, ez.v[c])) : fma_(az, ez.v[c], mul_(bc[2].v[c], cz));
        dxz[c] = hz.v[c] - hz_im.v[c];
        dxy[c] = hy.v[c] - hy_im.v[c];
        dyz[c] = hz.v[c] - hz_jm.v[c];
        dyx[c] = hx.v[c] - hx_jm.v[c];
        dzy[c] = hy.v[c] - hyk;
        dzx[c] = hx.v[c] - hxk;
    }
    cell_psi<T, V, OV ? 0 : -1, true>(d.ax[0], b, i, j, k, zs, bc, dxz, dxy, dyz, dyx, dzy, dzx, ex, ey, ez);
    if constexpr (OV) cell_psi<T, V, 1, true>(d.ax[0], b, i, j, k, zs, bc, dxz, dxy, dyz, dyx, dzy, dzx, ex, ey, ez);
    // lumped ports of one edge: the thread that owns the edge steps the
    // element on the value it is about to store
    for (int q = 0; q < d.n_lumped; ++q) {
        const int4 at = d.lumped[q];
        if (at.x != i || at.y != j || (unsigned)(at.z - k) >= (unsigned)V) continue;
#pragma unroll
        for (int c = 0; c < V; ++c) {
            if (at.z != k + c) continue;
            const T v =
                lumped_edge_step<T>(d.ports[q], d.pa, b, at.w == 0 ? ex.v[c] : (at.w == 1 ? ey.v[c] : ez.v[c]));
            if (at.w == 0) ex.v[c] = v;
            if (at.w == 1) ey.v[c] = v;
            if (at.w == 2) ez.v[c] = v;
        }
    }
    if (k + V - 1 > g.nz) {
        keep_pad(ex, k, g.nz);
        keep_pad(ey, k, g.nz);
        keep_pad(ez, k, g.nz);
    }
    stv<V>(Eo + o, ex);
    stv<V>(Eo + vol + o, ey);
    stv<V>(Eo + 2 * vol + o, ez);
    hz_im = hz;
    hy_im = hy;
}

// H_new of a thread's cells at plane i from E_new.  ez_ip, ey_ip: E of plane
// i + 1; on return E of plane i.
template <typename T, int V, int CK, bool UA, bool OV>
__device__ __forceinline__ void cell_H(const StencilArgs<T>& p, const DirectArgs& d, const T* E, const T* H, T* Ho,
                                       int b, int i, int j, int k, int o, bool zs, Vec<T, V>& ez_ip,
                                       Vec<T, V>& ey_ip) {
    const Geom& g = p.g;
    const long long vol = g.vol;
    const int sj = (int)g.sj;
    Vec<T, V> a[3], bc[3];
    load_cell_coef<T, V, CK, UA>(p, 1, o, a, bc);
    const Vec<T, V> ex = ldv<V>(E + o), ey = ldv<V>(E + vol + o), ez = ldv<V>(E + 2 * vol + o);
    const Vec<T, V> ez_jp = ldv<V>(E + 2 * vol + o + sj), ex_jp = ldv<V>(E + o + sj);
    const T ey_kp = E[vol + o + V], ex_kp = E[o + V];
    Vec<T, V> hx = ldv<V>(H + o), hy = ldv<V>(H + vol + o), hz = ldv<V>(H + 2 * vol + o);
    T dxz[V], dxy[V], dyz[V], dyx[V], dzy[V], dzx[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        const T eyk = c < V - 1 ? ey.v[(c + 1) % V] : ey_kp, exk = c < V - 1 ? ex.v[(c + 1) % V] : ex_kp;
        const T cx = ((ez_jp.v[c] - ez.v[c]) - eyk) + ey.v[c];
        const T cy = ((exk - ex.v[c]) - ez_ip.v[c]) + ez.v[c];
        const T cz = ((ey_ip.v[c] - ey.v[c]) - ex_jp.v[c]) + ex.v[c];
        hx.v[c] = fma_(alpha_of<T, V, UA>(a[0], bc[0].v[c], p.a0[1], c), hx.v[c], -mul_(bc[0].v[c], cx));
        hy.v[c] = fma_(alpha_of<T, V, UA>(a[1], bc[1].v[c], p.a0[1], c), hy.v[c], -mul_(bc[1].v[c], cy));
        hz.v[c] = fma_(alpha_of<T, V, UA>(a[2], bc[2].v[c], p.a0[1], c), hz.v[c], -mul_(bc[2].v[c], cz));
        dxz[c] = ez_ip.v[c] - ez.v[c];
        dxy[c] = ey_ip.v[c] - ey.v[c];
        dyz[c] = ez_jp.v[c] - ez.v[c];
        dyx[c] = ex_jp.v[c] - ex.v[c];
        dzy[c] = eyk - ey.v[c];
        dzx[c] = exk - ex.v[c];
    }
    cell_psi<T, V, OV ? 0 : -1, false>(d.ax[1], b, i, j, k, zs, bc, dxz, dxy, dyz, dyx, dzy, dzx, hx, hy, hz);
    if constexpr (OV) cell_psi<T, V, 1, false>(d.ax[1], b, i, j, k, zs, bc, dxz, dxy, dyz, dyx, dzy, dzx, hx, hy, hz);
    if (k + V - 1 > g.nz) {
        keep_pad(hx, k, g.nz);
        keep_pad(hy, k, g.nz);
        keep_pad(hz, k, g.nz);
    }
    stv<V>(Ho + o, hx);
    stv<V>(Ho + vol + o, hy);
    stv<V>(Ho + 2 * vol + o, hz);
    ez_ip = ez;
    ey_ip = ey;
}

template <typename T, int V, int CK, bool UA, bool OV, bool ES>
__global__ void __launch_bounds__(kDirectThreads, direct_min_ctas<T, V>())
    k_update_E(const __grid_constant__ StencilArgs<T> p, const __grid_constant__ DirectArgs d) {
    const Geom& g = p.g;
    int j, k;
    bool zs;
    if (!direct_cell(d, g.ny, blockIdx.x * blockDim.x + threadIdx.x, V, j, k, zs)) return;
    const long long vol = g.vol;
    const int si = (int)g.si;
    const int i0 = blockIdx.y * d.np, i1 = min(i0 + d.np, g.nx + 1);
    for (int b = threadIdx.y; b < p.B; b += blockDim.y) {
        const long long fs = (long long)b * 3 * vol;
        const T* H = p.h + fs;
        int o = (int)pidx(g, i0, j, k);  // offset within a component: below 2^31 on any GPU this fits
        Vec<T, V> hz_im = ldv<V>(H + 2 * vol + o - si), hy_im = ldv<V>(H + vol + o - si);
        for (int i = i0; i < i1; ++i, o += si)
            cell_E<T, V, CK, UA, OV, ES>(p, d, p.e + fs, H, p.e_next + fs, b, i, j, k, o, zs, hz_im, hy_im);
    }
}

template <typename T, int V, int CK, bool UA, bool OV>
__global__ void __launch_bounds__(kDirectThreads, direct_min_ctas<T, V>())
    k_update_H(const __grid_constant__ StencilArgs<T> p, const __grid_constant__ DirectArgs d) {
    const Geom& g = p.g;
    // the step counter, when nothing after this kernel reads it
    if (d.advance && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) *d.advance += 1;
    int j, k;
    bool zs;
    if (!direct_cell(d, g.ny, blockIdx.x * blockDim.x + threadIdx.x, V, j, k, zs)) return;
    const long long vol = g.vol;
    const int si = (int)g.si;
    const int i0 = blockIdx.y * d.np, i1 = min(i0 + d.np, g.nx + 1);
    for (int b = threadIdx.y; b < p.B; b += blockDim.y) {
        const long long fs = (long long)b * 3 * vol;
        const T* E = p.e_next + fs;
        int o = (int)pidx(g, i1 - 1, j, k);
        Vec<T, V> ez_ip = ldv<V>(E + 2 * vol + o + si), ey_ip = ldv<V>(E + vol + o + si);
        for (int i = i1 - 1; i >= i0; --i, o -= si)
            cell_H<T, V, CK, UA, OV>(p, d, E, p.h + fs, p.h_next + fs, b, i, j, k, o, zs, ez_ip, ey_ip);
    }
}

// bits 0 / 1 of flags[side]: some entry has alpha != (beta != 0) / alpha != 1
// (so an unset bit 0 means alpha follows from beta with a0 = 0, an unset
// bit 1 with a0 = 1); over the entries of the component's own sub-box.
template <typename T, int CK>
__global__ void __launch_bounds__(256) k_unit_alpha(const StencilArgs<T> p, int* flags) {
    const Geom& g = p.g;
    const int side = blockIdx.y / 3, c = blockIdx.y % 3;
    int ni, nj, nk;
    comp_shape(g, 3 * side + c, ni, nj, nk);
    const T* __restrict__ A = side == 0 ? p.aE : p.aH;
    const T* __restrict__ Bp = side == 0 ? p.bE : p.bH;
    int bad = 0;
    for (long long row = blockIdx.x; row < (long long)ni * nj; row += gridDim.x) {
        const long long o = c * g.vol + pidx(g, (int)(row / nj), (int)(row % nj), 0);
        for (int k = threadIdx.x; k < nk; k += blockDim.x) {
            const T b = coef_at<T, CK>(Bp, p.cq[2 * side + 1], p.cs[8 * side + 4 + c], o + k);
            const T a = coef_at<T, CK>(A, p.cq[2 * side], p.cs[8 * side + c], o + k);
            if (a != (b != T(0) ? T(1) : T(0))) bad |= 1;
            if (a != T(1)) bad |= 2;
        }
    }
    if (bad) atomicOr(flags + side, bad);
}

template <typename T>
__global__ void k_pack(const T* __restrict__ flat, T* __restrict__ padded, Geom g, int comp) {
    int ni, nj, nk;
    comp_shape(g, comp, ni, nj, nk);
    const long long n = (long long)ni * nj * nk;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % nk);
        const long long r = t / nk;
        const int j = (int)(r % nj);
        const int i = (int)(r / nj);
        padded[pidx(g, i, j, k)] = flat[t];
    }
}

template <typename T>
__global__ void k_unpack(const T* __restrict__ padded, T* __restrict__ flat, Geom g, int comp) {
    int ni, nj, nk;
    comp_shape(g, comp, ni, nj, nk);
    const long long n = (long long)ni * nj * nk;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n;
         t += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(t % nk);
        const long long r = t / nk;
        const int j = (int)(r % nj);
        const int i = (int)(r / nj);
        flat[t] = padded[pidx(g, i, j, k)];
    }
}

__global__ void k_advance(long long* step) { step[0] += 1; }

template <typename T>
__global__ void k_energy_partial(const T* __restrict__ e, const T* __restrict__ h,
                                 const T* __restrict__ meps, const T* __restrict__ mmu,
                                 long long n3, double* __restrict__ partials) {
    double acc = 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n3;
         t += (long long)gridDim.x * blockDim.x) {
        const double ev = (double)e[t], hv = (double)h[t];
        acc += (double)meps[t] * ev * ev + (double)mmu[t] * hv * hv;
    }
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) partials[blockIdx.x] = red[0];
}

__global__ void k_energy_final(const double* __restrict__ partials, int n, double* out) {
    __shared__ double red[256];
    double acc = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) acc += partials[t];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = 0.5 * red[0];
}

}  // namespace

// t / n for t < 2^31 as mulhi(2 t, m) >> s.
static DirectDiv direct_div(int n) {
    int s = 0;
    while ((1u << s) < (unsigned)n) ++s;
    return {(unsigned)(((1ull << (31 + s)) / (unsigned)n) + 1), s};
}

constexpr int kGridRows = 65535;  // gridDim.y at most

// Grid of the direct kernels: V cells and np planes per thread, 128 threads,
// the field sets of a cell in threadIdx.y (as many as there are warps).
// Returns whether both faces of an axis reach one cell.
template <typename T>
static bool direct_grid(const StencilArgs<T>& a, DirectArgs& d, int V, dim3& grid, dim3& block) {
    bool overlap = false;
    for (int side = 0; side < 2; ++side) {
        for (auto& x : d.ax[side]) x = AxisSlabs{};
        for (auto& x : d.ax[side]) x.lo1 = 0x7fffffff;
        for (int q = 0; q < a.nfaces; ++q) {
            const FaceDev& f = a.f[q];
            AxisSlabs& x = d.ax[side][f.axis];
            const int hi = f.lo > 0 || x.n[0] > 0 ? 1 : 0;  // a face of the whole axis first, then the far side
            if (hi) x.lo1 = f.lo;
            x.n[hi] = f.n;
            x.s0[hi] = f.dJ * f.pk;
            x.s1[hi] = f.pk;
            x.slab[hi] = (unsigned)f.slab;
            x.set[hi] = 4 * f.slab;
            x.psi[hi] = static_cast<T*>(f.psi) + 2 * side * f.slab;  // E1, E2 or H1, H2
            x.psi_out[hi] = static_cast<T*>(d.ping_pong ? f.psi_next : f.psi) + 2 * side * f.slab;
            x.bcc[hi] = f.bcc;
            x.air[hi] = f.masked ? f.air + 2 * side * f.slab : nullptr;
        }
        for (const AxisSlabs& x : d.ax[side]) overlap = overlap || x.n[0] > x.lo1;
    }
    const int nset = std::min(a.B, kDirectThreads / 32);
    block = dim3(kDirectThreads / nset / 32 * 32, nset, 1);
    // one plane per thread, more on meshes with more planes than a grid has
    // rows of blocks
    d.np = std::max({1, d.np, (a.g.nx + kGridRows) / kGridRows});
    const AxisSlabs& z = d.ax[0][2];
    const int nvec = a.g.nz / V + 1;
    d.n_low = std::min(nvec, (z.n[0] + V - 1) / V);
    const int high = z.n[1] > 0 ? nvec - std::min(nvec, z.lo1 / V) : 0;
    d.n_mid = std::max(0, nvec - d.n_low - high);
    d.n_edge = nvec - d.n_mid;
    const long long rows = a.g.ny + 1;
    d.mid_threads = (unsigned)((rows * d.n_mid + 31) / 32 * 32);
    d.mid_div = direct_div(std::max(1, d.n_mid));
    d.edge_div = direct_div(std::max(1, d.n_edge));
    grid = dim3((unsigned)((d.mid_threads + rows * d.n_edge + block.x - 1) / block.x),
                (unsigned)((a.g.nx + d.np) / d.np), 1);
    return overlap;
}

template <typename T, int V, int CK, bool ES>
static void direct_launch(const StencilArgs<T>& a, DirectArgs d, int which, cudaStream_t s) {
    dim3 grid, block;
    const bool overlap = direct_grid<T>(a, d, V, grid, block);
    // alpha read from memory: conductive or mixed coefficients, and small
    // meshes whose thick slabs overlap
    const auto go = [&](auto kE, auto kH) {
        if (which == 0)
            kE<<<grid, block, 0, s>>>(a, d);
        else
            kH<<<grid, block, 0, s>>>(a, d);
    };
    if (overlap)
        go(k_update_E<T, V, CK, false, true, ES>, k_update_H<T, V, CK, false, true>);
    else if (a.unit_alpha)
        go(k_update_E<T, V, CK, true, false, ES>, k_update_H<T, V, CK, true, false>);
    else
        go(k_update_E<T, V, CK, false, false, ES>, k_update_H<T, V, CK, false, false>);
}

// Meshes up to this many cells take one cell per thread: their step is the
// latency of one short thread.  The line is where one field set with CPML all
// round crosses (float32 and float64).  Measured, one cell against 16 bytes per
// thread, us per step with CPML: 7.1 / 9.1 at 11 thousand cells, 8.4 / 9.0 at 101
// thousand, 10.0 / 10.6 at 148 thousand, 12.1 / 11.3 at 226 thousand; float64
// 7.4 / 8.3, 9.3 / 9.5, 11.7 / 11.8, 13.8 / 13.7.  Without CPML the two cross at
// about 50 thousand cells (4.6 / 4.6; 6.0 / 5.4 at 148 thousand), and so do
// batches in float32 (four sets with CPML 9.1 / 10.5 at 21 thousand, 12.9 / 10.9
// at 54 thousand, 22.0 / 18.9 at 148 thousand; eight 37.0 / 32.7 there); the rule
// does not look at either.
constexpr long long kScalarCells = 150000;

template <typename T>
static bool direct_wide(const StencilArgs<T>& a) {
    return (long long)(a.g.nx + 1) * (a.g.ny + 1) * (a.g.nz + 1) > kScalarCells;
}

template <typename T>
void launch_direct_half(const StencilArgs<T>& a0, const DirectArgs& d, int which, cudaStream_t s) {
    constexpr int W = 16 / (int)sizeof(T);
    StencilArgs<T> a = a0;
    if (!d.ping_pong) {
        a.e_next = a.e;
        a.h_next = a.h;
    }
    const bool wide = direct_wide(a);
    const auto kind = [&](auto ck, auto es) {
        constexpr int CK = decltype(ck)::value;
        constexpr bool ES = decltype(es)::value;
        wide ? direct_launch<T, W, CK, ES>(a, d, which, s) : direct_launch<T, 1, CK, ES>(a, d, which, s);
    };
    using Native = std::integral_constant<int, kCoefNative>;
    using F16 = std::integral_constant<int, kCoefF16>;
    using BF16 = std::integral_constant<int, kCoefBF16>;
    if (d.slab_bits)  // the slab step takes no bfloat16
        a.coef_kind == kCoefF16 ? kind(F16(), std::true_type()) : kind(Native(), std::true_type());
    else if (a.coef_kind == kCoefF16)
        kind(F16(), std::false_type());
    else if (a.coef_kind == kCoefBF16)
        kind(BF16(), std::false_type());
    else
        kind(Native(), std::false_type());
}

template <typename T>
void direct_shape(const StencilArgs<T>& a, int np, int* out) {
    DirectArgs d{};
    d.np = np;
    dim3 grid, block;
    direct_grid<T>(a, d, direct_wide(a) ? 16 / (int)sizeof(T) : 1, grid, block);
    out[0] = d.np;
    out[1] = (int)grid.x;
    out[2] = (int)grid.y;
    out[3] = (int)grid.z;
}

template <typename T>
void launch_unit_alpha(const StencilArgs<T>& a, int* flags, cudaStream_t s) {
    const dim3 grid(592, 6);
    if (a.coef_kind == kCoefF16)
        k_unit_alpha<T, kCoefF16><<<grid, 256, 0, s>>>(a, flags);
    else if (a.coef_kind == kCoefBF16)
        k_unit_alpha<T, kCoefBF16><<<grid, 256, 0, s>>>(a, flags);
    else
        k_unit_alpha<T, kCoefNative><<<grid, 256, 0, s>>>(a, flags);
}

template <typename T>
void launch_pack(const T* flat, T* padded, const Geom& g, int comp, long long flat_off,
                 cudaStream_t s) {
    k_pack<T><<<1184, 256, 0, s>>>(flat + flat_off, padded, g, comp);
}

template <typename T>
void launch_unpack(const T* padded, T* flat, const Geom& g, int comp, long long flat_off,
                   cudaStream_t s) {
    k_unpack<T><<<1184, 256, 0, s>>>(padded, flat + flat_off, g, comp);
}

void launch_advance(long long* step, cudaStream_t s) { k_advance<<<1, 1, 0, s>>>(step); }

template <typename T>
void launch_energy(const T* e, const T* h, const T* meps, const T* mmu, const Geom& g, int b,
                   long long e_block, double* partials, int nblocks, double* out,
                   cudaStream_t s) {
    const T* eb = e + (long long)b * e_block;
    const T* hb = h + (long long)b * e_block;
    k_energy_partial<T><<<nblocks, 256, 0, s>>>(eb, hb, meps, mmu, e_block, partials);
    k_energy_final<<<1, 256, 0, s>>>(partials, nblocks, out);
}

#define FITB_INST(T)                                                                           \
    template void launch_direct_half<T>(const StencilArgs<T>&, const DirectArgs&, int, cudaStream_t); \
    template void direct_shape<T>(const StencilArgs<T>&, int, int*);                           \
    template void launch_unit_alpha<T>(const StencilArgs<T>&, int*, cudaStream_t);             \
    template void launch_pack<T>(const T*, T*, const Geom&, int, long long, cudaStream_t);     \
    template void launch_unpack<T>(const T*, T*, const Geom&, int, long long, cudaStream_t);   \
    template void launch_energy<T>(const T*, const T*, const T*, const T*, const Geom&, int,    \
                                   long long, double*, int, double*, cudaStream_t);
FITB_INST(float)
FITB_INST(double)
#undef FITB_INST

}  // namespace fitb
