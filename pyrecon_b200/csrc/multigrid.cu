// Full-multigrid solve of the RSD-modified Poisson equation on a periodic mesh.
//
// Operator, for cell c with p = i + offset / h (local line of sight) or p = los / h (global),
// g = beta / (h^2 |p|^2), G_a = 1/h_a^2 + g p_a^2 (reference src/multigrid.c:63-104):
//   (A v)_c = 2 (G_x + G_y + G_z) v_c - S(v)_c
//   S(v)_c  = sum_a G_a (v_{c+a} + v_{c-a})
//           + g/2 sum_{a<b} p_a p_b (v_{c+a+b} + v_{c-a-b} - v_{c-a+b} - v_{c+a-b})
//           + [local] g sum_a p_a (v_{c+a} - v_{c-a})
// Damped Jacobi: v <- (1 - w) v + w (f + S(v)) / (2 sum G), one fused kernel per sweep
// (the reference writes jac then blends in a second pass).
//
// Schedule = the reference's fixed FMG (src/multigrid.c:270-328): restrict f to the coarsest
// level (while every n > 4 and even), then per level prolong the coarse solution and run
// `vcycle_niterations` V-cycles of `jacobi_niterations` pre- and post-sweeps.
//
// Mixed precision (f32 entry with mixed_precision = 1): the V-cycle is affine and consistent,
// so V(v, f) = v + V(0, f - A v) exactly; each V-cycle is run as an FP64 residual of the FP64
// iterate, an FP32 V-cycle from zero on that defect, and an FP64 correction.
#include "common.cuh"

#include <algorithm>
#include <list>
#include <map>
#include <mutex>
#include <stdlib.h>
#include <string>
#include <tuple>
#include <vector>

namespace prc {

template <typename T> struct Stencil {
    int n[3];
    T h2[3], ih2[3], off[3], losh[3];
    T beta;
    int local;
};

template <typename T>
static Stencil<T> make_stencil(const int n[3], const double boxsize[3], const double boxcenter[3], double beta,
                               const double* los) {
    Stencil<T> s;
    s.local = los == nullptr;
    s.beta = (T)beta;
    for (int d = 0; d < 3; d++) {
        s.n[d] = n[d];
        T bs = (T)boxsize[d], bc = (T)boxcenter[d];
        T h = bs / (T)n[d];                                  // FLOAT / size_t in the reference
        s.h2[d] = h * h;
        s.ih2[d] = (T)(1. / (double)s.h2[d]);
        s.off[d] = (T)(((double)bc - (double)bs / 2.) / (double)h);
        s.losh[d] = s.local ? (T)0 : (T)los[d] / h;
    }
    return s;
}

// Operator forms of the quad kernels (template argument MODE).  MG_LOCAL: p = position / h, 19 points
// with the first-derivative term.  MG_GLOBAL: p = los / h, 19 points.  MG_AXIS0..2: a line of sight
// along one axis, where every edge coefficient p_a p_b and all but one p_a^2 are exactly zero, so the
// operator reads 7 points; the terms it leaves out are exact zeros in the 19-point form, so the two agree
// up to the compiler's contraction of the kept terms into multiply-adds (run-time knob mg_axis_stencil = 0
// keeps the 19-point form for comparison).
enum { MG_GLOBAL = 0, MG_LOCAL = 1, MG_AXIS0 = 2, MG_AXIS1 = 3, MG_AXIS2 = 4 };

template <typename T> static int mg_mode(const Stencil<T>& s) {
    if (s.local) return MG_LOCAL;
    int zeros = 0, axis = 0;
    for (int d = 0; d < 3; d++) {
        if (s.losh[d] == (T)0) zeros++;
        else axis = d;
    }
    return zeros == 2 && tune_get("mg_axis_stencil", 0, 1) != 0 ? MG_AXIS0 + axis : MG_GLOBAL;
}

template <typename T, typename S>
__device__ __forceinline__ void coeffs(const Stencil<S>& s, int x, int y, int z, T p[3], T& g, T G[3]) {
    if (s.local) {
        p[0] = (T)x + (T)s.off[0];
        p[1] = (T)y + (T)s.off[1];
        p[2] = (T)z + (T)s.off[2];
    } else {
        p[0] = (T)s.losh[0];
        p[1] = (T)s.losh[1];
        p[2] = (T)s.losh[2];
    }
    g = (T)s.beta / ((T)s.h2[0] * p[0] * p[0] + (T)s.h2[1] * p[1] * p[1] + (T)s.h2[2] * p[2] * p[2]);
#pragma unroll
    for (int d = 0; d < 3; d++) G[d] = (T)s.ih2[d] + g * p[d] * p[d];
}

// S(v) from the six axis neighbours and the three edge combinations e_ab = v(+a+b) + v(-a-b) -
// v(-a+b) - v(+a-b); every kernel evaluates it through this one expression.
template <typename A>
__device__ __forceinline__ A stencil_terms(A vxp, A vxm, A vyp, A vym, A vzp, A vzm, A exy, A exz, A eyz, const A p[3],
                                           A g, const A G[3], int local) {
    A s = G[0] * (vxp + vxm) + G[1] * (vyp + vym) + G[2] * (vzp + vzm);
    s += g / (A)2 * (p[0] * p[1] * exy + p[0] * p[2] * exz + p[1] * p[2] * eyz);
    if (local) s += g * (p[0] * (vxp - vxm) + p[1] * (vyp - vym) + p[2] * (vzp - vzm));
    return s;
}

// The neighbour terms of S(v) at one cell, accumulated in type A from a mesh of type V (read-only global
// memory, or shared memory when SMEM).
template <typename A, typename V, bool SMEM = false>
__device__ __forceinline__ A neighbour_sum(const V* __restrict__ v, const int n[3], int x, int y, int z, const A p[3],
                                           A g, const A G[3], int local) {
    const int xp = wrap_up(x, n[0]), xm = wrap_dn(x, n[0]);
    const int yp = wrap_up(y, n[1]), ym = wrap_dn(y, n[1]);
    const int zp = wrap_up(z, n[2]), zm = wrap_dn(z, n[2]);
    const int64_t sx = (int64_t)n[1] * n[2], sy = n[2];
    const int64_t X0 = x * sx, Xp = xp * sx, Xm = xm * sx;
    const int64_t Y0 = y * sy, Yp = yp * sy, Ym = ym * sy;
#define L(a, b, c) ((A)(SMEM ? v[(a) + (b) + (c)] : __ldg(v + (a) + (b) + (c))))
    const A vxp = L(Xp, Y0, z), vxm = L(Xm, Y0, z);
    const A vyp = L(X0, Yp, z), vym = L(X0, Ym, z);
    const A vzp = L(X0, Y0, zp), vzm = L(X0, Y0, zm);
    const A exy = L(Xp, Yp, z) + L(Xm, Ym, z) - L(Xm, Yp, z) - L(Xp, Ym, z);
    const A exz = L(Xp, Y0, zp) + L(Xm, Y0, zm) - L(Xm, Y0, zp) - L(Xp, Y0, zm);
    const A eyz = L(X0, Yp, zp) + L(X0, Ym, zm) - L(X0, Ym, zp) - L(X0, Yp, zm);
#undef L
    return stencil_terms<A>(vxp, vxm, vyp, vym, vzp, vzm, exy, exz, eyz, p, g, G, local);
}

// Kernels run one thread per cell of a 3D launch: (z, y) over the block's (x, y) threads, x over
// blockIdx.z.  A batch of `count` problems of the same shape, stored one after the other, is one
// launch with count n0 planes along blockIdx.z: problem blockIdx.z / n0, plane blockIdx.z % n0.
__device__ __forceinline__ bool cell3(const int n[3], int& x, int& y, int& z) {
    z = blockIdx.x * blockDim.x + threadIdx.x;
    y = blockIdx.y * blockDim.y + threadIdx.y;
    x = gridDim.z == (unsigned)n[0] ? (int)blockIdx.z : (int)(blockIdx.z % n[0]);   // no division unbatched
    return z < n[2] && y < n[1];
}

// Offset of this block's problem in a batch of meshes of shape n.
__device__ __forceinline__ int64_t batch_offset(const int n[3]) {
    if (gridDim.z == (unsigned)n[0]) return 0;
    return (int64_t)(blockIdx.z / n[0]) * ((int64_t)n[0] * n[1] * n[2]);
}

// One damped-Jacobi sweep: vout = (1 - w) v + w (f + S(v)) / (2 sum G).  zero_v: v is
// identically zero (first sweep of a V-cycle started from zero), so S(v) = 0 and v is not read.
template <typename T, typename FT>
__global__ void __launch_bounds__(256) jacobi_sweep(const T* __restrict__ v, const FT* __restrict__ f,
                                                    T* __restrict__ vout, Stencil<T> s, T w, int zero_v) {
    pdl_trigger();
    pdl_wait();
    int x, y, z;
    if (!cell3(s.n, x, y, z)) return;
    const int64_t bo = batch_offset(s.n);
    v += bo, f += bo, vout += bo;
    const int64_t i = ((int64_t)x * s.n[1] + y) * s.n[2] + z;
    T p[3], g, G[3];
    coeffs<T>(s, x, y, z, p, g, G);
    T jac = (T)f[i];
    T vc = (T)0;
    if (!zero_v) {
        jac += neighbour_sum<T>(v, s.n, x, y, z, p, g, G, s.local);
        vc = v[i];
    }
    jac /= (T)2 * (G[0] + G[1] + G[2]);
    vout[i] = ((T)1 - w) * vc + w * jac;
}

// ---- four cells along z per thread (n2 % 4 == 0, 16-byte aligned meshes) ----
// The thread loads the nine (x +- 1, y +- 1) columns it needs once as vectors (the five that need
// z - 1 and z + 4 as well), so a cell costs ~5 loads instead of 19 and the index arithmetic is
// shared.  Same expression per cell as the one-cell kernels.
template <typename T> __device__ __forceinline__ void load4(const T* __restrict__ p, T (&o)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 q = __ldg((const float4*)p);
        o[0] = q.x, o[1] = q.y, o[2] = q.z, o[3] = q.w;
    } else {
        const double2 a = __ldg((const double2*)p), b = __ldg((const double2*)p + 1);
        o[0] = a.x, o[1] = a.y, o[2] = b.x, o[3] = b.y;
    }
}
// values at z0 - 1 .. z0 + 4 of one column (periodic in z)
template <typename T> __device__ __forceinline__ void load6(const T* __restrict__ col, int z0, int n2, T (&o)[6]) {
    T m[4];
    load4(col + z0, m);
    o[0] = __ldg(col + (z0 == 0 ? n2 - 1 : z0 - 1));
    o[1] = m[0], o[2] = m[1], o[3] = m[2], o[4] = m[3];
    o[5] = __ldg(col + (z0 + 4 == n2 ? 0 : z0 + 4));
}

struct Quad {
    int x, y, z0;
    int64_t c;        // offset of (x, y, 0)
};
__device__ __forceinline__ bool quad_of(const int n[3], Quad& q) {
    q.z0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    q.y = blockIdx.y * blockDim.y + threadIdx.y;
    q.x = gridDim.z == (unsigned)n[0] ? (int)blockIdx.z : (int)(blockIdx.z % n[0]);
    q.c = ((int64_t)q.x * n[1] + q.y) * n[2];
    return q.z0 < n[2] && q.y < n[1];
}

// The nine columns a quad's operator reads: the centre and the four axis neighbours at z0 - 1 .. z0 + 4,
// the four (x +- 1, y +- 1) edge columns at z0 .. z0 + 3.
template <typename V> struct QuadCols {
    V c[6], XP[6], XM[6], YP[6], YM[6], PP[4], MM[4], MP[4], PM[4];
};

// Axis modes read the centre column at z0 - 1 .. z0 + 4 and the four axis neighbours at z0 .. z0 + 3
// (entries 1..4 of their arrays), nothing else.
template <int MODE, typename V, typename S>
__device__ __forceinline__ void quad_load(const V* __restrict__ v, const Stencil<S>& s, const Quad& q, QuadCols<V>& Q) {
    const int n0 = s.n[0], n1 = s.n[1], n2 = s.n[2];
    const int64_t sx = (int64_t)n1 * n2;
    const int64_t xp = (int64_t)wrap_up(q.x, n0) * sx, xm = (int64_t)wrap_dn(q.x, n0) * sx, x0 = (int64_t)q.x * sx;
    const int64_t yp = (int64_t)wrap_up(q.y, n1) * n2, ym = (int64_t)wrap_dn(q.y, n1) * n2, y0 = (int64_t)q.y * n2;
    load6(v + x0 + y0, q.z0, n2, Q.c);
    if constexpr (MODE >= MG_AXIS0) {
        V t[4];
        load4(v + xp + y0 + q.z0, t);
#pragma unroll
        for (int k = 0; k < 4; k++) Q.XP[k + 1] = t[k];
        load4(v + xm + y0 + q.z0, t);
#pragma unroll
        for (int k = 0; k < 4; k++) Q.XM[k + 1] = t[k];
        load4(v + x0 + yp + q.z0, t);
#pragma unroll
        for (int k = 0; k < 4; k++) Q.YP[k + 1] = t[k];
        load4(v + x0 + ym + q.z0, t);
#pragma unroll
        for (int k = 0; k < 4; k++) Q.YM[k + 1] = t[k];
        return;
    }
    load6(v + xp + y0, q.z0, n2, Q.XP);
    load6(v + xm + y0, q.z0, n2, Q.XM);
    load6(v + x0 + yp, q.z0, n2, Q.YP);
    load6(v + x0 + ym, q.z0, n2, Q.YM);
    load4(v + xp + yp + q.z0, Q.PP);
    load4(v + xm + ym + q.z0, Q.MM);
    load4(v + xm + yp + q.z0, Q.MP);
    load4(v + xp + ym + q.z0, Q.PM);
}

}  // namespace prc

#include "mg_march.cuh"

namespace prc {

// U, W, q and P (op_terms) of a quad's cell i from its columns, one cell at a time: pairs would start at an odd column, and
// the moves and registers they cost (80 against 64 in the FP32 sweep: 512 x 512 x 8 9.3 and 8.7 us) take warps from kernels
// that wait on memory.
template <bool LOCAL, typename T>
__device__ __forceinline__ void quad_terms(const QuadCols<T>& Q, const OpCoef<T>& k, const XYCoef<T>& c, int z0, int i,
                                           T& U, T& W, T& q, T& PP) {
    const T p2 = z_p2<LOCAL>(k, z0 + i), s2 = rn_mul(p2, p2);
    const T exy = rn_sub(rn_add(Q.PP[i], Q.MM[i]), rn_add(Q.MP[i], Q.PM[i]));
    const T exz = rn_sub(rn_add(Q.XP[i + 2], Q.XM[i]), rn_add(Q.XM[i + 2], Q.XP[i]));
    const T eyz = rn_sub(rn_add(Q.YP[i + 2], Q.YM[i]), rn_add(Q.YM[i + 2], Q.YP[i]));
    op_terms<LOCAL, One<T>>(k, c, p2, s2, Q.XP[i + 1], Q.XM[i + 1], Q.YP[i + 1], Q.YM[i + 1], Q.c[i + 2], Q.c[i], exy, exz, eyz,
                            U, W, q, PP);
}

// U, W, q and P of the axis modes, which leave out terms that are exact zeros, and the damped-Jacobi values from them.  The
// expressions are left to the compiler, for all four cells before the divisions: in pairs of cells, spelled out as op_terms,
// they took 40 registers instead of 32 in the FP32 sweep and 70 instead of 64 in the FP64 one (a sweep at 256^3: FP32 33.8 us
// and 37.3 in pairs, FP64 along y 78 and 95; one cell at a time, spelled out, 38.7 and 85).  They come out as vcycle_coarse
// spells them (the tests compare the bits).
template <int MODE, typename T>
__device__ __forceinline__ void axis_terms(const QuadCols<T>& Q, const Stencil<T>& s, T (&U)[4], T (&W)[4], T (&qq)[4],
                                           T (&P)[4]) {
    const T ih0 = s.ih2[0], ih1 = s.ih2[1], ih2 = s.ih2[2];
    const T p0 = s.losh[0], p1 = s.losh[1], p2 = s.losh[2];
    const T s0 = p0 * p0, s1 = p1 * p1;
    const T q01 = s.h2[0] * s0 + s.h2[1] * s1, P01 = s0 + s1;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const T s2 = p2 * p2;
        const T xpv = Q.XP[k + 1], xmv = Q.XM[k + 1], ypv = Q.YP[k + 1], ymv = Q.YM[k + 1], zpv = Q.c[k + 2], zmv = Q.c[k];
        U[k] = ih0 * (xpv + xmv) + ih1 * (ypv + ymv) + ih2 * (zpv + zmv);
        if constexpr (MODE == MG_AXIS0) W[k] = s0 * (xpv + xmv);
        else if constexpr (MODE == MG_AXIS1) W[k] = s1 * (ypv + ymv);
        else W[k] = s2 * (zpv + zmv);
        qq[k] = q01 + s.h2[2] * s2;
        P[k] = P01 + s2;
    }
}
// The same where v is identically zero.
template <typename T>
__device__ __forceinline__ void axis_zero_terms(const Stencil<T>& s, T (&U)[4], T (&W)[4], T (&qq)[4], T (&P)[4], T (&vc)[4]) {
    const T p0 = s.losh[0], p1 = s.losh[1], p2 = s.losh[2];
    const T s0 = p0 * p0, s1 = p1 * p1;
    const T q01 = s.h2[0] * s0 + s.h2[1] * s1, P01 = s0 + s1;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const T s2 = p2 * p2;
        qq[k] = q01 + s.h2[2] * s2;
        P[k] = P01 + s2;
        U[k] = W[k] = vc[k] = (T)0;
    }
}
template <typename T> __device__ __forceinline__ T quotient(T a, T b) {
    if constexpr (sizeof(T) == 4) return __fdividef(a, b);
    else return a / b;
}
template <typename T>
__device__ __forceinline__ void axis_blend(const Stencil<T>& s, T w, const T (&fv)[4], const T (&vc)[4], const T (&U)[4],
                                           const T (&W)[4], const T (&qq)[4], const T (&P)[4], T (&o)[4]) {
    const T sih = s.ih2[0] + s.ih2[1] + s.ih2[2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const T jac = quotient<T>(qq[k] * (fv[k] + U[k]) + s.beta * W[k], (T)2 * (qq[k] * sih + s.beta * P[k]));
        o[k] = vc[k] + w * (jac - vc[k]);
    }
}

// The damped-Jacobi values of a quad from its columns (19-point operator).
template <bool LOCAL, typename T>
__device__ __forceinline__ void quad_jacobi(const QuadCols<T>& Q, const OpCoef<T>& k, T w, int x, int y, int z0,
                                            const T (&f)[4], T (&o)[4]) {
    const XYCoef<T> c = xy_coef<LOCAL>(k, x, y);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        T U, W, q, PP;
        quad_terms<LOCAL>(Q, k, c, z0, i, U, W, q, PP);
        o[i] = op_jacobi<One<T>>(k, f[i], Q.c[i + 1], U, W, q, PP, w);
    }
}

// The sums of a quad's cells 2 j, 2 j + 1 in a pair, FP32 meshes below MARCH_MIN_BYTES: fewer instructions, and there no
// sweep waits on memory bandwidth (60 sweeps and their residuals at 100 x 60 x 44 in a solve of 1.00 ms: 0.94 in pairs).
// The same operations: the same bits.
template <bool LOCAL, typename T, typename P2 = typename Pair<T>::T>
__device__ __forceinline__ void quad_pair_terms(const QuadCols<T>& Q, const OpCoef<T>& k, const XYCoef<T>& c, int z0, int i,
                                                P2& U, P2& W, P2& q, P2& PP) {
    typedef Pair<T> P;
    auto two = [](const T* a) { return P::make(a[0], a[1]); };
    const P2 p2 = P::make(z_p2<LOCAL>(k, z0 + i), z_p2<LOCAL>(k, z0 + i + 1)), s2 = P::mul(p2, p2);
    const P2 exy = P::sub(P::add(two(Q.PP + i), two(Q.MM + i)), P::add(two(Q.MP + i), two(Q.PM + i)));
    const P2 exz = P::sub(P::add(two(Q.XP + i + 2), two(Q.XM + i)), P::add(two(Q.XM + i + 2), two(Q.XP + i)));
    const P2 eyz = P::sub(P::add(two(Q.YP + i + 2), two(Q.YM + i)), P::add(two(Q.YM + i + 2), two(Q.YP + i)));
    op_terms<LOCAL, P>(k, c, p2, s2, two(Q.XP + i + 1), two(Q.XM + i + 1), two(Q.YP + i + 1), two(Q.YM + i + 1),
                       two(Q.c + i + 2), two(Q.c + i), exy, exz, eyz, U, W, q, PP);
}
template <bool LOCAL, typename T>
__device__ __forceinline__ void quad_pairs_jacobi(const QuadCols<T>& Q, const OpCoef<T>& k, T w, int x, int y, int z0,
                                                  const T (&f)[4], T (&o)[4]) {
    typedef Pair<T> P;
    const XYCoef<T> c = xy_coef<LOCAL>(k, x, y);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        typename P::T U, W, q, PP;
        quad_pair_terms<LOCAL>(Q, k, c, z0, i, U, W, q, PP);
        const typename P::T r = op_jacobi<P>(k, P::make(f[i], f[i + 1]), P::make(Q.c[i + 1], Q.c[i + 2]), U, W, q, PP, w);
        o[i] = r.x, o[i + 1] = r.y;
    }
}

// The same where v is identically zero (the first sweep of a V-cycle started from zero): w q f / den, with q and P
// summed in their own order (local: h_0^2 p_0^2 and h_1^2 p_1^2 as (h^2 p) p).
template <bool LOCAL, typename T>
__device__ __forceinline__ void quad_zero(const OpCoef<T>& k, T w, int x, int y, int z0, const T (&f)[4], T (&o)[4]) {
    typedef Pair<T> P;
    typedef typename P::T P2;
    XYCoef<T> c = xy_coef<LOCAL>(k, x, y);
    if (LOCAL) {
        const T p0 = rn_add((T)x, k.off0), p1 = rn_add((T)y, k.off1);
        c.q01 = fma_rn(rn_mul(k.h21, p1), p1, rn_mul(rn_mul(k.h20, p0), p0));
        c.P01 = fma_rn(p1, p1, c.s0);
    }
    const P2 zero = both((T)0);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const P2 p2 = LOCAL ? P::make(rn_add((T)(z0 + 2 * j), k.off2), rn_add((T)(z0 + 2 * j + 1), k.off2)) : both(k.off2);
        const P2 s2 = P::mul(p2, p2), q = P::fma(both(k.h22), s2, both(c.q01)), PP = P::add(both(c.P01), s2);
        const P2 r = op_jacobi<P>(k, P::make(f[2 * j], f[2 * j + 1]), zero, zero, zero, q, PP, w);
        o[2 * j] = r.x, o[2 * j + 1] = r.y;
    }
}

template <typename T> __device__ __forceinline__ void store4(T* p, const T (&o)[4]) {
    if constexpr (sizeof(T) == 4) {
        *(float4*)p = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        ((double2*)p)[0] = make_double2(o[0], o[1]);
        ((double2*)p)[1] = make_double2(o[2], o[3]);
    }
}

// Damped-Jacobi sweep of four cells per thread: the axis modes, the 19-point ones where march_ok leaves them here (short
// rows, small meshes), and (zero_v) every sweep from an identically zero v.
// ADD: the sweep's result is added to acc instead of being stored (OP_JACOBI_ADD).  PAIRS: 19-point, by quad_pair_terms.
template <typename T, int MODE, bool ADD, bool PAIRS>
__global__ void __launch_bounds__(256) jacobi_sweep4(const T* __restrict__ v, const T* __restrict__ f,
                                                     T* __restrict__ vout, double* __restrict__ acc, Stencil<T> s, T w,
                                                     int zero_v) {
    pdl_trigger();
    pdl_wait();
    Quad q;
    if (!quad_of(s.n, q)) return;
    const int64_t bo = batch_offset(s.n);
    v += bo, f += bo, vout += bo;
    T fv[4], o[4];
    load4(f + q.c + q.z0, fv);
    if constexpr (MODE >= MG_AXIS0) {
        T U[4], W[4], qq[4], P[4], vc[4];
        if (zero_v) {
            axis_zero_terms(s, U, W, qq, P, vc);
        } else {
            QuadCols<T> Q;
            quad_load<MODE>(v, s, q, Q);
            axis_terms<MODE>(Q, s, U, W, qq, P);
            load4(v + q.c + q.z0, vc);
        }
        axis_blend(s, w, fv, vc, U, W, qq, P, o);
    } else if (zero_v) {
        quad_zero<MODE == MG_LOCAL>(op_coef<MODE == MG_LOCAL>(s), w, q.x, q.y, q.z0, fv, o);
    } else {
        QuadCols<T> Q;
        quad_load<MODE>(v, s, q, Q);
        if constexpr (PAIRS) quad_pairs_jacobi<MODE == MG_LOCAL>(Q, op_coef<MODE == MG_LOCAL>(s), w, q.x, q.y, q.z0, fv, o);
        else quad_jacobi<MODE == MG_LOCAL>(Q, op_coef<MODE == MG_LOCAL>(s), w, q.x, q.y, q.z0, fv, o);
    }
    if constexpr (ADD) {
        double* a = acc + bo + q.c + q.z0;
        double t[4];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const double2 d = *(const double2*)(a + j);
            t[j] = d.x + (double)o[j], t[j + 1] = d.y + (double)o[j + 1];
        }
        store4(a, t);
    } else {
        store4(vout + q.c + q.z0, o);
    }
}

// ---- two sweeps per pass (temporal blocking) ----
// A block owns a tile of TY rows (y) x 4 TQ cells (z) and marches along x through a slab of planes.  At
// plane step x it stages plane x + 1 of v (the tile grown by two rows and eight cells on each side;
// planes x - 1 and x are already there), runs the first sweep at plane x over the tile grown by one
// row and one quad on each side into a ring of three planes in shared memory, then the second sweep at
// plane x - 1 over the tile from the ring's planes x - 2 .. x.  v and f are read from DRAM once and the
// result written once per two sweeps (the halo of the first sweep is recomputed by the neighbouring
// tiles).  Every quad goes through quad_jacobi, the arithmetic of jacobi_sweep4, so two
// sweeps here equal two jacobi_sweep4 launches bit for bit.  Periodic in every axis: staged rows and
// 4-cell chunks wrap (n2 % 4 == 0 keeps every chunk contiguous and aligned).
template <typename T, int TY, int TQ> struct TbShape {
    static constexpr int ZP = 4 * TQ + 16;         // row pitch: cells z0 - 8 .. z0 + 4 TQ + 8
    static constexpr int R0 = TY + 4;              // rows of a staged v plane: y0 - 2 .. y0 + TY + 1
    static constexpr int R1 = TY + 2;              // rows of a first-sweep plane: y0 - 1 .. y0 + TY
    static constexpr int Q1 = TQ + 2;              // quads of a first-sweep row: z0 - 4 .. z0 + 4 TQ + 3
    static constexpr int THREADS = TQ * TY;
};

__device__ __forceinline__ int wrap_mod(int i, int n) {
    i %= n;
    return i < 0 ? i + n : i;
}

template <typename T>
__device__ __forceinline__ void smem_quad6(const T* row, int i, T (&o)[6]) {   // cells i - 1 .. i + 4, i % 4 == 0
    T m[4];
    if constexpr (sizeof(T) == 4) {
        const float4 a = *(const float4*)(row + i);
        m[0] = a.x, m[1] = a.y, m[2] = a.z, m[3] = a.w;
    } else {
        const double2 a = *(const double2*)(row + i), b = *(const double2*)(row + i + 2);
        m[0] = a.x, m[1] = a.y, m[2] = b.x, m[3] = b.y;
    }
    o[0] = row[i - 1], o[1] = m[0], o[2] = m[1], o[3] = m[2], o[4] = m[3], o[5] = row[i + 4];
}
template <typename T> __device__ __forceinline__ void smem_quad4(const T* row, int i, T (&o)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 a = *(const float4*)(row + i);
        o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w;
    } else {
        const double2 a = *(const double2*)(row + i), b = *(const double2*)(row + i + 2);
        o[0] = a.x, o[1] = a.y, o[2] = b.x, o[3] = b.y;
    }
}
template <typename T> __device__ __forceinline__ void smem_store4(T* row, int i, const T (&o)[4]) {
    if constexpr (sizeof(T) == 4) {
        *(float4*)(row + i) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        *(double2*)(row + i) = make_double2(o[0], o[1]);
        *(double2*)(row + i + 2) = make_double2(o[2], o[3]);
    }
}

// The columns of the quad at (row r, cell index i) of plane `mid`, its neighbours in planes `lo` (x - 1)
// and `hi` (x + 1), all with row pitch ZP.
template <typename T, int ZP>
__device__ __forceinline__ void smem_cols(const T* lo, const T* mid, const T* hi, int r, int i, QuadCols<T>& Q) {
    smem_quad6(mid + r * ZP, i, Q.c);
    smem_quad6(hi + r * ZP, i, Q.XP);
    smem_quad6(lo + r * ZP, i, Q.XM);
    smem_quad6(mid + (r + 1) * ZP, i, Q.YP);
    smem_quad6(mid + (r - 1) * ZP, i, Q.YM);
    smem_quad4(hi + (r + 1) * ZP, i, Q.PP);
    smem_quad4(lo + (r - 1) * ZP, i, Q.MM);
    smem_quad4(lo + (r + 1) * ZP, i, Q.MP);
    smem_quad4(hi + (r - 1) * ZP, i, Q.PM);
}

template <typename T, bool LOCAL, int TY, int TQ>
__global__ void __launch_bounds__(TQ * TY, (sizeof(T) == 4 ? 6 : 4)) jacobi_sweep2_tb(const T* __restrict__ v, const T* __restrict__ f,
                                                             T* __restrict__ vout, Stencil<T> s, T w, int zero_v,
                                                             int slab, int nslab) {
    pdl_trigger();
    pdl_wait();
    typedef TbShape<T, TY, TQ> SH;
    constexpr int ZP = SH::ZP;
    constexpr int PL0 = SH::R0 * ZP, PL1 = SH::R1 * ZP;
    __shared__ __align__(16) T v0s[3 * PL0];       // planes x - 1, x, x + 1 of v (ring)
    __shared__ __align__(16) T v1s[3 * PL1];       // first-sweep planes x - 2, x - 1, x (ring)
    const int n0 = s.n[0], n1 = s.n[1], n2 = s.n[2];
    const int64_t N = (int64_t)n0 * n1 * n2;
    const int prob = blockIdx.z / nslab;
    const int x0 = (blockIdx.z % nslab) * slab, x1 = min(x0 + slab, n0);
    v += prob * N, f += prob * N, vout += prob * N;
    const int y0 = blockIdx.y * TY, z0 = blockIdx.x * (4 * TQ);
    const int tid = threadIdx.x;
    const int64_t sx = (int64_t)n1 * n2;
    const OpCoef<T> kc = op_coef<LOCAL>(s);

    // stage plane x (periodic) of v into ring slot x mod 3
    auto stage = [&](int x) {
        T* dst = v0s + wrap_mod(x, 3) * PL0;
        const int64_t xo = (int64_t)wrap_mod(x, n0) * sx;
        constexpr int CH = ZP / 4;                 // 4-cell chunks per staged row
        for (int q = tid; q < SH::R0 * CH; q += SH::THREADS) {
            const int r = q / CH, ch = q % CH;
            const int gy = wrap_mod(y0 - 2 + r, n1), gz = wrap_mod(z0 - 8 + 4 * ch, n2);
            T m[4];
            load4(v + xo + (int64_t)gy * n2 + gz, m);
            smem_store4(dst + r * ZP, 4 * ch, m);
        }
    };
    if (!zero_v) {
        stage(x0 - 2);
        stage(x0 - 1);
    }
    for (int x = x0 - 1; x <= x1; x++) {
        if (!zero_v) stage(x + 1);
        __syncthreads();
        // first sweep at plane x over rows y0 - 1 .. y0 + TY, quads z0 - 4 .. z0 + 4 TQ
        {
            const int gx = wrap_mod(x, n0);
            const T* lo = v0s + wrap_mod(x - 1, 3) * PL0;
            const T* mid = v0s + wrap_mod(x, 3) * PL0;
            const T* hi = v0s + wrap_mod(x + 1, 3) * PL0;
            T* out = v1s + wrap_mod(x, 3) * PL1;
            for (int q = tid; q < SH::R1 * SH::Q1; q += SH::THREADS) {
                const int r = q / SH::Q1, k = q % SH::Q1;
                const int gy = wrap_mod(y0 - 1 + r, n1), gz = wrap_mod(z0 - 4 + 4 * k, n2);
                T fv[4], o[4];
                load4(f + (int64_t)gx * sx + (int64_t)gy * n2 + gz, fv);
                if (zero_v) {
                    quad_zero<LOCAL>(kc, w, gx, gy, gz, fv, o);
                } else {
                    QuadCols<T> Q;
                    smem_cols<T, ZP>(lo, mid, hi, r + 1, 4 * k + 4, Q);
                    quad_jacobi<LOCAL>(Q, kc, w, gx, gy, gz, fv, o);
                }
                smem_store4(out + r * ZP, 4 * k + 4, o);
            }
        }
        __syncthreads();
        // second sweep at plane x - 1 over the tile
        const int xo = x - 1;
        if (xo >= x0) {
            const T* lo = v1s + wrap_mod(xo - 1, 3) * PL1;
            const T* mid = v1s + wrap_mod(xo, 3) * PL1;
            const T* hi = v1s + wrap_mod(xo + 1, 3) * PL1;
            const int r = tid / TQ, k = tid % TQ;
            const int gy = y0 + r, gz = z0 + 4 * k;
            if (gy < n1 && gz < n2) {
                const int64_t at = (int64_t)xo * sx + (int64_t)gy * n2 + gz;
                T fv[4], o[4];
                load4(f + at, fv);
                QuadCols<T> Q;
                smem_cols<T, ZP>(lo, mid, hi, r + 1, 4 * k + 8, Q);
                quad_jacobi<LOCAL>(Q, kc, w, xo, gy, gz, fv, o);
                if constexpr (sizeof(T) == 4) {
                    *(float4*)(vout + at) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
                    ((double2*)(vout + at))[0] = make_double2(o[0], o[1]);
                    ((double2*)(vout + at))[1] = make_double2(o[2], o[3]);
                }
            }
        }
    }
}

// r = f - A v of four cells per thread, evaluated in type A and stored as R: the axis modes, and the 19-point ones where
// march_ok leaves them here.
template <typename A, typename R, int MODE>
__global__ void __launch_bounds__(256) residual_kernel4(const A* __restrict__ v, const A* __restrict__ f,
                                                        R* __restrict__ r, Stencil<A> s) {
    pdl_trigger();
    pdl_wait();
    Quad q;
    if (!quad_of(s.n, q)) return;
    const int64_t bo = batch_offset(s.n);
    v += bo, f += bo, r += bo;
    QuadCols<A> Q;
    R o[4];
    quad_load<MODE>(v, s, q, Q);
    if constexpr (MODE >= MG_AXIS0) {
        A U[4], W[4], qq[4], P[4], vc[4], fv[4];
        axis_terms<MODE>(Q, s, U, W, qq, P);
        load4(v + q.c + q.z0, vc);
        load4(f + q.c + q.z0, fv);
        const A sih2 = (A)2 * (s.ih2[0] + s.ih2[1] + s.ih2[2]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const A g = quotient<A>(s.beta, qq[k]);
            const A x = vc[k];
            o[k] = (R)((fv[k] + U[k] - sih2 * x) + g * (W[k] - (A)2 * P[k] * x));
        }
    } else {
        A fv[4];
        load4(f + q.c + q.z0, fv);
        const OpCoef<A> k = op_coef<MODE == MG_LOCAL>(s);
        const XYCoef<A> c = xy_coef<MODE == MG_LOCAL>(k, q.x, q.y);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            A U, W, qq, PP;
            quad_terms<MODE == MG_LOCAL>(Q, k, c, q.z0, i, U, W, qq, PP);
            o[i] = (R)op_residual<One<A>>(k, fv[i], Q.c[i + 1], U, W, qq, PP);
        }
    }
    store4(r + q.c + q.z0, o);
}

// r = f - A v, evaluated in type A (double for the mixed-precision defect), stored as R.
template <typename A, typename V, typename FT, typename R, typename S>
__global__ void __launch_bounds__(256) residual_kernel(const V* __restrict__ v, const FT* __restrict__ f,
                                                       R* __restrict__ r, Stencil<S> s) {
    pdl_trigger();
    pdl_wait();
    int x, y, z;
    if (!cell3(s.n, x, y, z)) return;
    const int64_t bo = batch_offset(s.n);
    v += bo, f += bo, r += bo;
    const int64_t i = ((int64_t)x * s.n[1] + y) * s.n[2] + z;
    A p[3], g, G[3];
    coeffs<A>(s, x, y, z, p, g, G);
    const A nb = neighbour_sum<A>(v, s.n, x, y, z, p, g, G, s.local);
    const A av = (A)2 * (G[0] + G[1] + G[2]) * (A)v[i] - nb;
    r[i] = (R)((A)f[i] - av);
}

// The quad kernels' instance for an operator form (mg_mode).
template <typename T, bool ADD> static decltype(&jacobi_sweep4<T, MG_GLOBAL, ADD, false>) sweep4_kernel(int mode, bool small) {
    constexpr bool PAIRS = sizeof(T) == 4;
    switch (mode) {
    case MG_LOCAL: return small ? jacobi_sweep4<T, MG_LOCAL, ADD, PAIRS> : jacobi_sweep4<T, MG_LOCAL, ADD, false>;
    case MG_AXIS0: return jacobi_sweep4<T, MG_AXIS0, ADD, false>;
    case MG_AXIS1: return jacobi_sweep4<T, MG_AXIS1, ADD, false>;
    case MG_AXIS2: return jacobi_sweep4<T, MG_AXIS2, ADD, false>;
    default: return small ? jacobi_sweep4<T, MG_GLOBAL, ADD, PAIRS> : jacobi_sweep4<T, MG_GLOBAL, ADD, false>;
    }
}
template <typename A, typename R> static decltype(&residual_kernel4<A, R, MG_GLOBAL>) residual4_kernel(int mode) {
    switch (mode) {
    case MG_LOCAL: return residual_kernel4<A, R, MG_LOCAL>;
    case MG_AXIS0: return residual_kernel4<A, R, MG_AXIS0>;
    case MG_AXIS1: return residual_kernel4<A, R, MG_AXIS1>;
    case MG_AXIS2: return residual_kernel4<A, R, MG_AXIS2>;
    default: return residual_kernel4<A, R, MG_GLOBAL>;
    }
}

// 27-point full weighting, coarse cell (x, y, z) centred on fine (2x, 2y, 2z).
template <typename A, typename TI, typename TO>
__global__ void __launch_bounds__(256) reduce_kernel(const TI* __restrict__ fine, TO* __restrict__ coarse, Dims nf) {
    pdl_trigger();
    pdl_wait();
    const int nc[3] = {nf.n[0] / 2, nf.n[1] / 2, nf.n[2] / 2};
    {
        int x, y, z;
        if (!cell3(nc, x, y, z)) return;
        const int64_t bc = batch_offset(nc);
        fine += 8 * bc, coarse += bc;
        const int64_t i = ((int64_t)x * nc[1] + y) * nc[2] + z;
        const int X[3] = {wrap_dn(2 * x, nf.n[0]), 2 * x, wrap_up(2 * x, nf.n[0])};
        const int Y[3] = {wrap_dn(2 * y, nf.n[1]), 2 * y, wrap_up(2 * y, nf.n[1])};
        const int Z[3] = {wrap_dn(2 * z, nf.n[2]), 2 * z, wrap_up(2 * z, nf.n[2])};
        A acc = 0;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const TI* row = fine + ((int64_t)X[a] * nf.n[1] + Y[b]) * nf.n[2];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const int side = (a != 1) + (b != 1) + (c != 1);
                    acc += (A)(8 >> side) * (A)__ldg(row + Z[c]);
                }
            }
        coarse[i] = (TO)(acc / (A)64);
    }
}

// Trilinear prolongation of a coarse mesh (nc) onto the fine mesh (2 nc): fine node 2c + e is
// the mean of the coarse nodes c + e' over e' <= e.  ADD: fine += value (V-cycle correction),
// else fine = value.
template <typename A, typename TI, typename TO, bool ADD>
__global__ void __launch_bounds__(256) prolong_kernel(const TI* __restrict__ coarse, TO* __restrict__ fine, Dims nc) {
    pdl_trigger();
    pdl_wait();
    const int nf1 = 2 * nc.n[1], nf2 = 2 * nc.n[2];
    {
        int x, y, z;
        if (!cell3(nc.n, x, y, z)) return;
        const int64_t bc = batch_offset(nc.n);
        coarse += bc, fine += 8 * bc;
        const int xs[2] = {x, wrap_up(x, nc.n[0])}, ys[2] = {y, wrap_up(y, nc.n[1])}, zs[2] = {z, wrap_up(z, nc.n[2])};
        A c[2][2][2];
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int d = 0; d < 2; d++)
                    c[a][b][d] = (A)__ldg(coarse + ((int64_t)xs[a] * nc.n[1] + ys[b]) * nc.n[2] + zs[d]);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int ex = (e >> 2) & 1, ey = (e >> 1) & 1, ez = e & 1;
            A s = 0;
#pragma unroll
            for (int a = 0; a <= ex; a++)
#pragma unroll
                for (int b = 0; b <= ey; b++)
#pragma unroll
                    for (int d = 0; d <= ez; d++) s += c[a][b][d];
            s /= (A)((1 + ex) * (1 + ey) * (1 + ez));
            TO* dst = fine + ((int64_t)(2 * x + ex) * nf1 + (2 * y + ey)) * nf2 + (2 * z + ez);
            if (ADD) *dst = (TO)((A)*dst + s);
            else *dst = (TO)s;
        }
    }
}

// ---- restriction and prolongation, two coarse cells along z per thread (fine n2 % 4 == 0, aligned meshes) ----
// Bound by memory: a fine mesh is read (and written) in 16-byte vectors, four fine cells a row instead of one.
template <typename T> __device__ __forceinline__ void load2(const T* __restrict__ p, T (&o)[2]) {
    if constexpr (sizeof(T) == 4) {
        const float2 q = __ldg((const float2*)p);
        o[0] = q.x, o[1] = q.y;
    } else {
        const double2 q = __ldg((const double2*)p);
        o[0] = q.x, o[1] = q.y;
    }
}

// Launch over (n0, n1, n2 / 2) of the coarse shape; nc: the coarse shape.
__device__ __forceinline__ bool coarse_pair(const int nc[3], int& x, int& y, int& z) {
    z = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
    y = blockIdx.y * blockDim.y + threadIdx.y;
    x = gridDim.z == (unsigned)nc[0] ? (int)blockIdx.z : (int)(blockIdx.z % nc[0]);
    return z < nc[2] && y < nc[1];
}

// The order of the sum is reduce_kernel's (its weights are powers of two: every product is exact).
template <typename T>
__global__ void __launch_bounds__(256) reduce_pair(const T* __restrict__ fine, T* __restrict__ coarse, Dims nf) {
    pdl_trigger();
    pdl_wait();
    const int nc[3] = {nf.n[0] / 2, nf.n[1] / 2, nf.n[2] / 2};
    int x, y, z;
    if (!coarse_pair(nc, x, y, z)) return;
    const int64_t bc = batch_offset(nc);
    fine += 8 * bc, coarse += bc;
    const int X[3] = {wrap_dn(2 * x, nf.n[0]), 2 * x, wrap_up(2 * x, nf.n[0])};
    const int Y[3] = {wrap_dn(2 * y, nf.n[1]), 2 * y, wrap_up(2 * y, nf.n[1])};
    const int zm = z == 0 ? nf.n[2] - 1 : 2 * z - 1;
    T acc[2] = {0, 0};
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const T* row = fine + ((int64_t)X[a] * nf.n[1] + Y[b]) * nf.n[2];
            T m[4];
            load4(row + 2 * z, m);
            const T left = __ldg(row + zm);
            const int side = (a != 1) + (b != 1);
            const T wc = (T)(8 >> side), we = (T)(4 >> side);
            acc[0] = fma_rn(we, m[1], fma_rn(wc, m[0], fma_rn(we, left, acc[0])));
            acc[1] = fma_rn(we, m[3], fma_rn(wc, m[2], fma_rn(we, m[1], acc[1])));
        }
    T* o = coarse + ((int64_t)x * nc[1] + y) * nc[2] + z;
    if constexpr (sizeof(T) == 4) *(float2*)o = make_float2(acc[0] / 64, acc[1] / 64);
    else *(double2*)o = make_double2(acc[0] / 64, acc[1] / 64);
}

// ADD: fine += the prolonged coarse mesh, else fine = it.
template <typename T, bool ADD>
__global__ void __launch_bounds__(256) prolong_pair(const T* __restrict__ coarse, T* __restrict__ fine, Dims nc) {
    pdl_trigger();
    pdl_wait();
    int x, y, z;
    if (!coarse_pair(nc.n, x, y, z)) return;
    const int64_t bc = batch_offset(nc.n);
    coarse += bc, fine += 8 * bc;
    const int64_t nf1 = 2 * nc.n[1], nf2 = 2 * nc.n[2];
    const int xs[2] = {x, wrap_up(x, nc.n[0])}, ys[2] = {y, wrap_up(y, nc.n[1])}, zn = z + 2 == nc.n[2] ? 0 : z + 2;
    T c[2][2][3];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const T* row = coarse + ((int64_t)xs[a] * nc.n[1] + ys[b]) * nc.n[2];
            T t[2];
            load2(row + z, t);
            c[a][b][0] = t[0], c[a][b][1] = t[1], c[a][b][2] = __ldg(row + zn);
        }
#pragma unroll
    for (int ex = 0; ex < 2; ex++)
#pragma unroll
        for (int ey = 0; ey < 2; ey++) {
            T* dst = fine + ((2 * x + ex) * nf1 + (2 * y + ey)) * nf2 + 2 * z;
            T o[4];
            if constexpr (ADD) {
                if constexpr (sizeof(T) == 4) {
                    const float4 q = *(const float4*)dst;
                    o[0] = q.x, o[1] = q.y, o[2] = q.z, o[3] = q.w;
                } else {
                    const double2 q = *(const double2*)dst, w = *((const double2*)dst + 1);
                    o[0] = q.x, o[1] = q.y, o[2] = w.x, o[3] = w.y;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                // the mean of the corners, summed in prolong_kernel's order
                const int d = j / 2, ez = j & 1;
                T t = 0;
#pragma unroll
                for (int a = 0; a <= ex; a++)
#pragma unroll
                    for (int b = 0; b <= ey; b++)
#pragma unroll
                        for (int e = 0; e <= ez; e++) t = rn_add(t, c[a][b][d + e]);
                t = rn_mul(t, (T)1 / (T)((1 + ex) * (1 + ey) * (1 + ez)));
                o[j] = ADD ? rn_add(o[j], t) : t;
            }
            store4(dst, o);
        }
}

template <typename TI, typename TO>
__global__ void convert_kernel(const TI* __restrict__ in, TO* __restrict__ out, int64_t n) {
    pdl_trigger();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (TO)in[i];
}

template <typename TA, typename TB>
__global__ void add_kernel(TA* __restrict__ acc, const TB* __restrict__ x, int64_t n) {
    pdl_trigger();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        acc[i] = acc[i] + (TA)x[i];
}

static int grid_for(int64_t n) {
    int64_t blocks = (n + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(blocks, (int64_t)device_sm_count() * 16));
}

// 3D launch over an (n0, n1, n2) mesh for the cell3 kernels: up to 32 z x 8 y threads per block.
struct Grid3 {
    dim3 grid, block;
};
// `count` problems of that shape: count n0 blocks along z (see cell3).
static Grid3 grid3(const int n[3], int count = 1) {
    int bx = 1, by = 1;
    while (bx < n[2] && bx < 32) bx <<= 1;
    while (by < n[1] && bx * by < 256) by <<= 1;
    Grid3 g;
    g.block = dim3(bx, by, 1);
    g.grid = dim3((n[2] + bx - 1) / bx, (n[1] + by - 1) / by, n[0] * count);
    return g;
}
static Grid3 grid3_coarse(const int nf[3], int count = 1) {
    const int nc[3] = {nf[0] / 2, nf[1] / 2, nf[2] / 2};
    return grid3(nc, count);
}
// Launch of the four-cells-per-thread kernels, usable when n2 % 4 == 0 and the meshes are
// 16-byte aligned.
static Grid3 grid3_quad(const int n[3], int count = 1) {
    const int nq[3] = {n[0], n[1], n[2] / 4};
    return grid3(nq, count);
}
static bool quad_ok(const int n[3], const void* a, const void* b, const void* c) {
    return n[2] % 4 == 0 && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
}

// March kernels: usable for the 19-point operator (local or oblique line of sight) where the quad kernels are
// and a row holds a tile.
// Below MARCH_MIN_BYTES of v the quad kernels are as fast (64^3 FP32, 1 MB: 3.2 against 3.7 us, the march's pipeline
// fill; 96^3 FP32, 3.5 MB: 6.0 against 4.7 us; 64^3 FP64, 2 MB: 4.2 against 4.0 us).
// FP32 rows that segments cover badly (march_lanes computes more than 29 / 20 of their cells): sweeps need MARCH_WIDE_BYTES
// and go to the quad kernels beyond 9 / 5, residuals (a write-only output more to gain) beyond 2.  A sweep, quad kernel and
// march: 128 x 128 x 44 (1.64) 5.0 and 5.5 us, 80^3 (1.5) 4.3 and 4.6, 300 x 200 x 52 (1.54, 12 MB) 14.1 and 13.2, 252 x 100
// x 36 (2.0) 7.1 and 8.2, 1000 x 200 x 20 (2.4) 22.6 and 26.5; a residual of 80^3 5.9 and 4.7, 1000 x 200 x 20 27.5 and
// 30.7.  In FP64 the march is ahead wherever a row holds a tile (1000 x 200 x 20: 60 and 44 us).
// Where half the rows of the tiles lie past the mesh, or a third of 32 and more, the quad kernels stay: solves in FP64 by them
// and marched, 640 x 24 x 24 (24 rows of 64) 1.78 and 2.03 ms, 2000 x 20 x 16 (20 of 32) 1.45 and 1.54.
constexpr int64_t MARCH_MIN_BYTES = 3 << 19, MARCH_WIDE_BYTES = 4 << 20;
template <typename A> static bool march_ok(const Stencil<A>& s, int count, int op) {
    int cells;
    const int lz = march_lanes<A>(s.n[2], &cells);
    if (mg_mode(s) > MG_LOCAL || lz == 0 || (int64_t)s.n[0] * count > 65535) return false;
    const int rows = MARCH_THREADS / lz;
    if (2 * ((s.n[1] + rows - 1) / rows * rows) >= (rows >= 32 ? 3 : 4) * s.n[1]) return false;
    const int64_t bytes = (int64_t)s.n[0] * s.n[1] * s.n[2] * count * (int64_t)sizeof(A);
    if (bytes < MARCH_MIN_BYTES) return false;
    if (sizeof(A) == 8 || 20 * cells <= 29 * s.n[2]) return true;
    if (op == OP_RESIDUAL) return cells <= 2 * s.n[2];
    return 5 * cells <= 9 * s.n[2] && bytes >= MARCH_WIDE_BYTES;
}

template <typename A, typename OT, int OP>
static cudaError_t launch_march(const A* v, const A* f, OT* out, double* acc, const Stencil<A>& s, A w, int count,
                                cudaStream_t st) {
    const MarchSplit sp = march_split<A>(s.n, count);
    void (*kernel)(const A*, const A*, OT*, double*, Stencil<A>, A, MarchSplit) = nullptr;
    size_t smem = 0;
#define MARCH_CASE(LZ)                                                                                  \
    case LZ:                                                                                            \
        kernel = s.local ? march_kernel<A, OT, LZ, true, OP> : march_kernel<A, OT, LZ, false, OP>;      \
        smem = (size_t)MARCH_STAGES * MarchTile<A, LZ>::STAGE;                                          \
        break;
    switch (sp.lz) {
        MARCH_CASE(32)
        MARCH_CASE(16)
        MARCH_CASE(8)
        MARCH_CASE(4)
        default: return cudaErrorInvalidValue;
    }
#undef MARCH_CASE
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(kernel, dim3(sp.zsegs, sp.ytiles, sp.nslab * count), dim3(MARCH_THREADS), smem, st, v, f, out, acc,
                      s, w, sp);
}

// Coarse (nf / 2) from fine, and fine (2 nc) from coarse, over `count` meshes.
template <typename T>
static cudaError_t launch_reduce(const T* fine, T* coarse, const int nf[3], int count, cudaStream_t st) {
    const Dims d = {{nf[0], nf[1], nf[2]}};
    const int half[3] = {nf[0] / 2, nf[1] / 2, nf[2] / 4};
    const bool pair = nf[2] % 4 == 0 && (((uintptr_t)fine | (uintptr_t)coarse) & 15) == 0;
    const Grid3 g = pair ? grid3(half, count) : grid3_coarse(nf, count);
    return launch_pdl(pair ? reduce_pair<T> : reduce_kernel<T, T, T>, g.grid, g.block, 0, st, fine, coarse, d);
}
template <typename T, bool ADD>
static cudaError_t launch_prolong(const T* coarse, T* fine, const int nc[3], int count, cudaStream_t st) {
    const Dims d = {{nc[0], nc[1], nc[2]}};
    // an FP64 mesh that is only written: one coarse cell a thread is faster (256^3 27 us, two 39)
    if constexpr (ADD || sizeof(T) == 4) {
        if (nc[2] % 2 == 0 && (((uintptr_t)fine | (uintptr_t)coarse) & 15) == 0) {
            const int half[3] = {nc[0], nc[1], nc[2] / 2};
            const Grid3 g = grid3(half, count);
            return launch_pdl(prolong_pair<T, ADD>, g.grid, g.block, 0, st, coarse, fine, d);
        }
    }
    const Grid3 g = grid3(nc, count);
    return launch_pdl(prolong_kernel<T, T, T, ADD>, g.grid, g.block, 0, st, coarse, fine, d);
}

// Tile of the temporal-blocked sweeps: TB_TY rows x 4 TB_TQ cells.
constexpr int TB_TY = 8, TB_TQ = 16;

// Slab length of the temporal-blocked sweeps for a level with no tuning-table entry (0: one sweep per
// pass).
static int mg_tb_default(const int n[3], size_t tsize) {
    (void)n;
    (void)tsize;
    return 0;
}

__device__ __forceinline__ int cells_of(const int n[3]) { return n[0] * n[1] * n[2]; }

__device__ __forceinline__ void cell_xyz(int i, const int n[3], int& x, int& y, int& z) {
    z = i % n[2];
    y = (i / n[2]) % n[1];
    x = i / (n[1] * n[2]);
}

}  // namespace prc

#include "mg_coarse.cuh"

namespace prc {

// ---------------------------------------------------------------------------------------------
// Level hierarchy and the FMG / V-cycle drivers
// ---------------------------------------------------------------------------------------------
struct Level {
    int n[3];
    int64_t size() const { return (int64_t)n[0] * n[1] * n[2]; }
};

static bool coarsenable(const int n[3]) {
    for (int d = 0; d < 3; d++)
        if (!(n[d] > 4 && n[d] % 2 == 0)) return false;
    return true;
}

static std::vector<Level> hierarchy(const int32_t nmesh[3]) {
    std::vector<Level> L;
    Level l;
    for (int d = 0; d < 3; d++) l.n[d] = nmesh[d];
    L.push_back(l);
    while (coarsenable(L.back().n)) {
        Level c;
        for (int d = 0; d < 3; d++) c.n[d] = L.back().n[d] / 2;
        L.push_back(c);
    }
    return L;
}

static size_t al(size_t b) { return (b + 255) & ~(size_t)255; }

// Per-level buffers of one precision.
template <typename T> struct LevelBufs {
    T *v, *f, *r, *tmp;
};

struct Params {
    double boxsize[3], boxcenter[3], los[3];
    int has_los;
    double beta, damping;
    int jn, vn;
};

template <typename T> struct MGRunner {
    std::vector<Level> L;
    std::vector<LevelBufs<T>> B;     // per level: count problems one after the other in each buffer
    Params P;
    cudaStream_t st;
    int count = 1;

    Stencil<T> stencil(int l) const {
        return make_stencil<T>(L[l].n, P.boxsize, P.boxcenter, P.beta, P.has_los ? P.los : nullptr);
    }

    // niter sweeps ping-ponging between v and tmp; on return v points at the result and tmp at the
    // other buffer (the pointers are swapped instead of copying back).  zero_first: v known zero.
    // Pairs of sweeps run as one temporal-blocked pass when the tuning table's "mg_jacobi" (FP32) or
    // "mg_jacobi_f64" entry for the level (keyed by n0) is a slab length > 0 (mg_tb_default otherwise).
    // acc (optional): the last sweep adds its result to acc, and nothing is left in v.
    int jacobi(int l, T*& v, const T* f, T*& tmp, int niter, bool zero_first, double* acc = nullptr) {
        Stencil<T> s = stencil(l);
        const int64_t N = L[l].size() * count;
        const Grid3 g = grid3(L[l].n, count);
        if (niter == 0 && zero_first && cudaMemsetAsync(v, 0, N * sizeof(T), st) != cudaSuccess) return PRC_ERR_CUDA;
        const bool quad = quad_ok(L[l].n, v, f, tmp);
        const Grid3 gq = grid3_quad(L[l].n, count);
        const bool small = N * (int64_t)sizeof(T) < MARCH_MIN_BYTES;
        int it = 0;
        const int slab =
            quad ? tune_get(sizeof(T) == 4 ? "mg_jacobi" : "mg_jacobi_f64", L[l].n[0], mg_tb_default(L[l].n, sizeof(T)))
                 : 0;
        if (slab > 0) {
            const int nslab = (L[l].n[0] + slab - 1) / slab;
            const dim3 grid((L[l].n[2] + 4 * TB_TQ - 1) / (4 * TB_TQ), (L[l].n[1] + TB_TY - 1) / TB_TY, nslab * count);
            if ((int64_t)nslab * count <= 65535) {
                for (; it + 1 < (acc != nullptr ? niter - 1 : niter); it += 2) {
                    const bool z0 = zero_first && it == 0;
                    PRC_LAUNCH_B("mg_jacobi2", st, (double)N * sizeof(T) * (z0 ? 2 : 3),
                                 launch_pdl((s.local ? jacobi_sweep2_tb<T, true, TB_TY, TB_TQ>
                                          : jacobi_sweep2_tb<T, false, TB_TY, TB_TQ>), grid, TB_TY * TB_TQ, 0, st, v, f, tmp, s, (T)P.damping, z0, slab, nslab));
                    std::swap(v, tmp);
                }
            }
        }
        for (; it < niter; it++) {
            const bool z0 = zero_first && it == 0;
            double* a = it + 1 == niter ? acc : nullptr;
            const double bytes = (double)N * (sizeof(T) * (z0 ? 1 : 2) + (a != nullptr ? 16 : sizeof(T)));
            if (quad && !z0 && march_ok(s, count, OP_JACOBI)) {
                if (a != nullptr)
                    PRC_LAUNCH_B("mg_jacobi_add", st, bytes,
                                 (launch_march<T, T, OP_JACOBI_ADD>(v, f, tmp, a, s, (T)P.damping, count, st)));
                else
                    PRC_LAUNCH_B("mg_jacobi", st, bytes,
                                 (launch_march<T, T, OP_JACOBI>(v, f, tmp, nullptr, s, (T)P.damping, count, st)));
            } else if (quad) {
                PRC_LAUNCH_B(a != nullptr ? "mg_jacobi_add" : "mg_jacobi", st, bytes,
                             launch_pdl(a != nullptr ? sweep4_kernel<T, true>(mg_mode(s), small) : sweep4_kernel<T, false>(mg_mode(s), small), gq.grid, gq.block, 0, st, v, f, tmp, a, s, (T)P.damping, z0));
            } else {
                PRC_LAUNCH_B("mg_jacobi", st, (double)N * sizeof(T) * (z0 ? 2 : 3),
                             launch_pdl(jacobi_sweep<T, T>, g.grid, g.block, 0, st, v, f, tmp, s, (T)P.damping, z0));
                if (a != nullptr)
                    PRC_LAUNCH_B("mg_correct_fp64", st, (16.0 + sizeof(T)) * N,
                                 launch_pdl(add_kernel<double, T>, grid_for(N), 256, 0, st, a, tmp, N));
            }
            std::swap(v, tmp);
        }
        PRC_CHECK_LAUNCH();
        return PRC_OK;
    }

    // Clusters of cl blocks of a coarse kernel that run on the device at once, looked up once for each shared-memory size.
    template <typename K> static int clusters_at_once(K kernel, int cl, size_t smem) {
        typedef std::tuple<const void*, int, int, size_t> Key;
        static std::mutex mu;
        static std::map<Key, int> known;
        int dev = 0;
        cudaGetDevice(&dev);
        std::lock_guard<std::mutex> lock(mu);
        const Key key((const void*)kernel, dev, cl, smem);
        const auto it = known.find(key);
        if (it != known.end()) return it->second;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl);
        cfg.blockDim = dim3(MG_COARSE_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = cl;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        return known[key] = n;
    }

    // The V-cycle from level l down as one vcycle_coarse launch, when level l has at most "mg_small_cells"
    // cells (run-time knob, key 0; 0 runs every step as its own kernel) and its levels fit in shared memory.
    // Of cubes the largest it takes is 20^3: a block has threads for 1024 pairs of cells of its top level, and of 24^3, dealt
    // as twice the planes of 12^3, one would hold four planes, 1152 pairs.
    int coarse_vcycle(int l, T* v, const T* f, bool v_zero, bool* done) {
        *done = false;
        const int limit = tune_get("mg_small_cells", 0, MG_COARSE_DEFAULT_CELLS);
        const int nl = (int)L.size() - l;
        if (limit <= 0 || L[l].size() > limit || nl > MG_COARSE_LEVELS) return PRC_OK;
        CoarseCycle<T> c;
        c.nl = nl;
        c.ndist = 0;
        // rows of four cells are dealt (the quad kernels' arithmetic, by pairs); the rest stays in block 0
        const int slots = MG_COARSE_SLOTS * MG_COARSE_THREADS;
        while (c.ndist < nl && L[l + c.ndist].size() > MG_SINGLE_CELLS && L[l + c.ndist].n[2] % 4 == 0) c.ndist++;
        if (c.ndist < nl && L[l + c.ndist].size() > slots) return PRC_OK;
        // a lone level has only its ten sweeps to save, and in FP64 or with the seven terms of an axis a launched sweep is
        // short: solves by launches and in a cluster, 512 x 64 x 16 (128 x 16 x 4 the coarsest) FP64 1.26 and 1.30 ms, along
        // y 0.93 and 1.00, 2000 x 20 x 16 FP32 along y 0.70 and 0.77; but 64 x 512 x 16 FP32 oblique 0.87 and 0.84
        if (nl == 1 && c.ndist == 1 && (sizeof(T) == 8 || mg_mode(stencil(l)) >= MG_AXIS0)) return PRC_OK;
        c.base = c.ndist > 0 ? L[l + c.ndist - 1].n[0] : 0;
        int cl = 1;
        while (c.ndist > 0 && 2 * cl <= std::min(c.base, MG_COARSE_CLUSTER)) cl *= 2;
        if (c.ndist > 0 &&
            ((int64_t)((c.base + cl - 1) / cl) << (c.ndist - 1)) * L[l].n[1] * (L[l].n[2] / 2) > slots)
            return PRC_OK;
        size_t at = 0;
        for (int j = 0; j < nl; j++) {
            const Level& lv = L[l + j];
            c.s[j] = stencil(l + j);
            const int64_t planes = j < c.ndist ? (int64_t)((c.base + cl - 1) / cl) << (c.ndist - 1 - j) : lv.n[0];
            const int64_t pl = (int64_t)lv.n[1] * lv.n[2], own = (planes * pl + 3) & ~3ll;
            c.vsize[j] = (int)(((planes + (j < c.ndist ? 2 : 0)) * pl + 3) & ~3ll);
            c.at[j] = (int)at;
            at += 2 * (size_t)c.vsize[j] + own;
            if (at * sizeof(T) > MG_COARSE_MAX_SMEM) return PRC_OK;
        }
        const size_t smem = at * sizeof(T);
        c.w = (T)P.damping;
        c.jn = P.jn;
        c.zero_v = v_zero ? 1 : 0;
        c.axis = mg_mode(c.s[0]) >= MG_AXIS0 ? mg_mode(c.s[0]) - MG_AXIS0 : -1;
        const auto kernel = c.s[0].local ? vcycle_coarse<T, true> : vcycle_coarse<T, false>;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MG_COARSE_MAX_SMEM) != cudaSuccess)
            return PRC_ERR_CUDA;
        // A batch whose clusters do not run at once takes the dealt levels by launches (same bits) and comes back with the
        // levels of one block: whole solves by clusters and so, 14 of 32^3 FP32 0.89 and 1.06 ms, 16 1.18 and 1.06, 32 of
        // 40^3 FP64 along z 3.43 and 2.57, 16 of 64^3 FP64 4.84 and 4.62.
        if (c.ndist > 0 && clusters_at_once(kernel, cl, smem) < count) return PRC_OK;
        PRC_LAUNCH_B("mg_vcycle_coarse", st, (double)L[l].size() * count * sizeof(T) * (v_zero ? 2 : 3),
                     launch_cluster_pdl(kernel, dim3(cl * count), dim3(MG_COARSE_THREADS), cl, smem, st, f, v, c));
        PRC_CHECK_LAUNCH();
        *done = true;
        return PRC_OK;
    }

    // Recursive V-cycle on level l: v (B[l].v, or the caller's level-0 pointer) with right-hand side f.
    // acc (optional): the cycle's result is added to it; where the last step could do so itself, v holds nothing.
    int vcycle(int l, T*& v, const T* f, bool v_zero, double* acc = nullptr) {
        bool small = false;
        PRC_TRY(coarse_vcycle(l, v, f, v_zero, &small));
        if (small || P.jn == 0) {
            if (!small) PRC_TRY(vcycle_steps(l, v, f, v_zero, nullptr));
            if (acc != nullptr) {
                const int64_t N = L[l].size() * count;
                PRC_LAUNCH_B("mg_correct_fp64", st, 20.0 * N,
                             launch_pdl(add_kernel<double, T>, grid_for(N), 256, 0, st, acc, v, N));
                PRC_CHECK_LAUNCH();
            }
            return PRC_OK;
        }
        return vcycle_steps(l, v, f, v_zero, acc);
    }

    int vcycle_steps(int l, T*& v, const T* f, bool v_zero, double* acc) {
        PRC_TRY(jacobi(l, v, f, B[l].tmp, P.jn, v_zero));
        if (l + 1 < (int)L.size()) {
            Stencil<T> s = stencil(l);
            const int64_t N = L[l].size() * count;
            const Grid3 g = grid3(L[l].n, count);
            if (quad_ok(L[l].n, v, f, B[l].r) && march_ok(s, count, OP_RESIDUAL)) {
                PRC_LAUNCH_B("mg_residual", st, 3.0 * N * sizeof(T),
                             (launch_march<T, T, OP_RESIDUAL>(v, f, B[l].r, nullptr, s, (T)0, count, st)));
            } else if (quad_ok(L[l].n, v, f, B[l].r)) {
                const Grid3 gq = grid3_quad(L[l].n, count);
                PRC_LAUNCH_B("mg_residual", st, 3.0 * N * sizeof(T),
                             launch_pdl(residual4_kernel<T, T>(mg_mode(s)), gq.grid, gq.block, 0, st, v, f, B[l].r, s));
            } else {
                PRC_LAUNCH_B("mg_residual", st, 3.0 * N * sizeof(T),
                             launch_pdl(residual_kernel<T, T, T, T, T>, g.grid, g.block, 0, st, v, f, B[l].r, s));
            }
            PRC_LAUNCH_B("mg_reduce", st, (double)(N + L[l + 1].size() * count) * sizeof(T),
                         launch_reduce(B[l].r, B[l + 1].f, L[l].n, count, st));
            PRC_CHECK_LAUNCH();
            PRC_TRY(vcycle(l + 1, B[l + 1].v, B[l + 1].f, true));
            PRC_LAUNCH_B("mg_prolong_add", st, (double)(2 * N + L[l + 1].size() * count) * sizeof(T),
                         (launch_prolong<T, true>(B[l + 1].v, v, L[l + 1].n, count, st)));
            PRC_CHECK_LAUNCH();
        }
        return jacobi(l, v, f, B[l].tmp, P.jn, false, acc);
    }
};

// Plain FMG in precision T (the reference schedule); f0 is the level-0 right-hand side.
template <typename T> static int fmg_plain(MGRunner<T>& R, const T* f0, T* v0) {
    const int nl = (int)R.L.size();
    cudaStream_t st = R.st;
    // right-hand sides at every level
    R.B[0].f = const_cast<T*>(f0);
    const int cnt = R.count;
    for (int l = 0; l + 1 < nl; l++) {
        PRC_LAUNCH_B("mg_reduce", st, (double)(R.L[l].size() + R.L[l + 1].size()) * cnt * sizeof(T),
                     launch_reduce(R.B[l].f, R.B[l + 1].f, R.L[l].n, cnt, st));
    }
    PRC_CHECK_LAUNCH();
    // the FMG solution of level l >= 1 lives in B[l].v; level 0 starts in v0 and may end in
    // B[0].tmp (pointer swaps), in which case it is copied to v0 once at the end
    T* v0cur = v0;
    for (int l = nl - 1; l >= 0; l--) {
        T*& v = l == 0 ? v0cur : R.B[l].v;
        if (l == nl - 1) {
            if (cudaMemsetAsync(v, 0, R.L[l].size() * cnt * sizeof(T), st) != cudaSuccess) return PRC_ERR_CUDA;
        } else {
            PRC_LAUNCH_B("mg_prolong", st, (double)(R.L[l].size() + R.L[l + 1].size()) * cnt * sizeof(T),
                         (launch_prolong<T, false>(R.B[l + 1].v, v, R.L[l + 1].n, cnt, st)));
            PRC_CHECK_LAUNCH();
        }
        for (int it = 0; it < R.P.vn; it++) PRC_TRY(R.vcycle(l, v, R.B[l].f, l == nl - 1 && it == 0));
    }
    if (v0cur != v0 &&
        cudaMemcpyAsync(v0, v0cur, R.L[0].size() * cnt * sizeof(T), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return PRC_ERR_CUDA;
    return PRC_OK;
}

}  // namespace prc

using namespace prc;

namespace {

// Workspace layout for plain FMG in precision T: per level v, f, r, tmp (level 0's f and v receive the
// caller's right-hand side and return the solution, so the solve itself touches the workspace only).
template <typename T> size_t plain_layout(const int32_t nmesh[3], char* base, std::vector<LevelBufs<T>>* out,
                                          std::vector<Level>* lv, int count = 1) {
    std::vector<Level> L = hierarchy(nmesh);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += al(bytes);
        return p;
    };
    std::vector<LevelBufs<T>> B(L.size());
    for (size_t l = 0; l < L.size(); l++) {
        size_t b = (size_t)L[l].size() * count * sizeof(T);
        B[l].v = (T*)take(b);
        B[l].f = (T*)take(b);
        B[l].r = (T*)take(b);
        B[l].tmp = (T*)take(b);
    }
    if (out) *out = B;
    if (lv) *lv = L;
    return off;
}

// Mixed layout: FP64 f and v per level, plus the FP32 plain buffers for the inner V-cycles.
struct MixedBufs {
    std::vector<double*> f64, v64;
    std::vector<LevelBufs<float>> b32;
    std::vector<Level> L;
};

size_t mixed_layout(const int32_t nmesh[3], char* base, MixedBufs* mb, int count = 1) {
    std::vector<Level> L = hierarchy(nmesh);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += al(bytes);
        return p;
    };
    MixedBufs m;
    m.L = L;
    m.f64.resize(L.size());
    m.v64.resize(L.size());
    m.b32.resize(L.size());
    for (size_t l = 0; l < L.size(); l++) {
        size_t n = (size_t)L[l].size() * count;
        m.f64[l] = (double*)take(n * 8);
        m.v64[l] = (double*)take(n * 8);
        m.b32[l].v = (float*)take(n * 4);
        m.b32[l].f = (float*)take(n * 4);
        m.b32[l].r = (float*)take(n * 4);
        m.b32[l].tmp = (float*)take(n * 4);
    }
    if (mb) *mb = m;
    return off;
}

Params make_params(const double boxsize[3], const double boxcenter[3], double beta, double damping, int jn, int vn,
                   const double* los) {
    Params P;
    for (int d = 0; d < 3; d++) {
        P.boxsize[d] = boxsize[d];
        P.boxcenter[d] = boxcenter[d];
        P.los[d] = los ? los[d] : 0.;
    }
    P.has_los = los != nullptr;
    P.beta = beta;
    P.damping = damping;
    P.jn = jn;
    P.vn = vn;
    return P;
}

bool mg_args_ok(const void* delta, const void* phi, const int32_t nmesh[3], const double* boxsize,
                const double* boxcenter, int jn, int vn) {
    if (!delta || !phi || !nmesh || !boxsize || !boxcenter || jn < 0 || vn < 0) return false;
    for (int d = 0; d < 3; d++)
        if (nmesh[d] < 1 || !(boxsize[d] > 0)) return false;
    return true;
}

// Plain solve of the right-hand side held in the workspace's level-0 f into its level-0 v.
template <typename T> int solve_plain(const int32_t nmesh[3], const Params& P, void* ws, cudaStream_t st,
                                      int count = 1) {
    MGRunner<T> R;
    plain_layout<T>(nmesh, (char*)ws, &R.B, &R.L, count);
    R.P = P;
    R.st = st;
    R.count = count;
    T* f0 = R.B[0].f;
    T* v0 = R.B[0].v;
    return fmg_plain<T>(R, f0, v0);
}

// Mixed precision FMG: every V-cycle is v64 += V32(0, f64 - A v64); the FP64 right-hand side is in the
// workspace's level-0 f64 and the solution is left in its level-0 v64.
int solve_mixed(const int32_t nmesh[3], const Params& P, void* ws, cudaStream_t st, int count = 1) {
    MixedBufs m;
    mixed_layout(nmesh, (char*)ws, &m, count);
    const int nl = (int)m.L.size();
    MGRunner<float> R;
    R.L = m.L;
    R.B = m.b32;
    R.P = P;
    R.st = st;
    R.count = count;
    for (int l = 0; l + 1 < nl; l++) {
        PRC_LAUNCH_B("mg_reduce", st, 8.0 * (m.L[l].size() + m.L[l + 1].size()) * count,
                     launch_reduce(m.f64[l], m.f64[l + 1], m.L[l].n, count, st));
    }
    PRC_CHECK_LAUNCH();
    for (int l = nl - 1; l >= 0; l--) {
        const int64_t N = m.L[l].size() * count;
        const Grid3 g = grid3(m.L[l].n, count);
        if (l == nl - 1) {
            if (cudaMemsetAsync(m.v64[l], 0, N * 8, st) != cudaSuccess) return PRC_ERR_CUDA;
        } else {
            PRC_LAUNCH_B("mg_prolong", st, 8.0 * (m.L[l].size() + m.L[l + 1].size()) * count,
                         (launch_prolong<double, false>(m.v64[l + 1], m.v64[l], m.L[l + 1].n, count, st)));
        }
        Stencil<double> s64 = make_stencil<double>(m.L[l].n, P.boxsize, P.boxcenter, P.beta,
                                                   P.has_los ? P.los : nullptr);
        for (int it = 0; it < P.vn; it++) {
            // defect in FP64 (stored FP32 as the inner V-cycle's right-hand side)
            if (quad_ok(m.L[l].n, m.v64[l], m.f64[l], R.B[l].f) && march_ok(s64, count, OP_RESIDUAL)) {
                PRC_LAUNCH_B("mg_residual_fp64", st, 20.0 * N,
                             (launch_march<double, float, OP_RESIDUAL>(m.v64[l], m.f64[l], R.B[l].f, nullptr,
                                                                               s64, 0., count, st)));
            } else if (quad_ok(m.L[l].n, m.v64[l], m.f64[l], R.B[l].f)) {
                const Grid3 gq = grid3_quad(m.L[l].n, count);
                PRC_LAUNCH_B("mg_residual_fp64", st, 20.0 * N,
                             launch_pdl(residual4_kernel<double, float>(mg_mode(s64)), gq.grid, gq.block, 0, st, m.v64[l], m.f64[l], R.B[l].f, s64));
            } else {
                PRC_LAUNCH_B("mg_residual_fp64", st, 20.0 * N,
                             launch_pdl(residual_kernel<double, double, double, float, double>, g.grid, g.block, 0, st, m.v64[l], m.f64[l], R.B[l].f, s64));
            }
            PRC_CHECK_LAUNCH();
            PRC_TRY(R.vcycle(l, R.B[l].v, R.B[l].f, true, m.v64[l]));
        }
    }
    return PRC_OK;
}

// ---- the whole solve as a CUDA graph ----
//
// A solve is a fixed sequence of some thousands of small launches (most on the coarse levels),
// set by the mesh, the parameters and the workspace address (the caller's right-hand side and
// solution are copied in and out around it, so they are not part of it).  It is captured once into a CUDA graph
// and replayed while those stay the same (a small cache keyed on all of them), on the caller's stream
// (on a library stream joined to it by events when the caller gives the legacy default stream, which
// cannot be captured).  PRC_MG_GRAPH=0 launches directly.
struct GraphEntry {
    std::string key;
    int device;
    cudaGraphExec_t exec;
    unsigned long long launches;
    double bytes;
};
struct SideStream {
    cudaStream_t s = nullptr;
    cudaEvent_t in = nullptr, out = nullptr;
};
std::mutex g_graph_mutex;
std::list<GraphEntry> g_graphs;
std::map<int, SideStream> g_side;
constexpr size_t GRAPH_CACHE = 64;

bool graphs_enabled() {
    static int cached = -1;
    if (cached < 0) {
        const char* v = getenv("PRC_MG_GRAPH");
        cached = (v != nullptr && v[0] == '0') ? 0 : 1;
    }
    return cached == 1;
}

template <typename V> void key_add(std::string& k, const V& v) { k.append((const char*)&v, sizeof(V)); }

std::string solve_key(int tsize, int mixed, const int32_t nmesh[3], const Params& P, const void* ws, size_t wsb,
                      int count) {
    std::string k;
    key_add(k, tsize);
    key_add(k, mixed);
    key_add(k, count);
    for (int d = 0; d < 3; d++) {
        key_add(k, nmesh[d]);
        key_add(k, P.boxsize[d]);
        key_add(k, P.boxcenter[d]);
        key_add(k, P.los[d]);
    }
    key_add(k, P.has_los);
    key_add(k, P.beta);
    key_add(k, P.damping);
    key_add(k, P.jn);
    key_add(k, P.vn);
    key_add(k, ws);
    key_add(k, wsb);
    key_add(k, tune_generation());   // kernel choices of the tuning table
    return k;
}

template <typename F> int run_graph(const std::string& key, cudaStream_t st, F body) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (!graphs_enabled() || cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return body(st);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return PRC_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_graph_mutex);
    const bool legacy = st == nullptr || st == cudaStreamLegacy;
    SideStream& side = g_side[dev];
    if (legacy && side.s == nullptr) {
        if (cudaStreamCreateWithFlags(&side.s, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&side.in, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&side.out, cudaEventDisableTiming) != cudaSuccess) {
            side = SideStream();
            return body(st);
        }
    }
    const cudaStream_t run_st = legacy ? side.s : st;
    if (legacy &&
        (cudaEventRecord(side.in, st) != cudaSuccess || cudaStreamWaitEvent(side.s, side.in, 0) != cudaSuccess))
        return PRC_ERR_CUDA;
    auto it = g_graphs.begin();
    for (; it != g_graphs.end(); ++it)
        if (it->device == dev && it->key == key) break;
    if (it != g_graphs.end()) {
        g_graphs.splice(g_graphs.begin(), g_graphs, it);
    } else {
        capture_tally(nullptr, nullptr);
        if (cudaStreamBeginCapture(run_st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return PRC_ERR_CUDA;
        const int r = body(run_st);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(run_st, &g);
        GraphEntry ent;
        capture_tally(&ent.launches, &ent.bytes);
        if (r != PRC_OK || e != cudaSuccess || g == nullptr) {
            if (g != nullptr) cudaGraphDestroy(g);
            cudaGetLastError();
            return r != PRC_OK ? r : PRC_ERR_CUDA;
        }
        const cudaError_t ei = cudaGraphInstantiate(&ent.exec, g, 0);
        cudaGraphDestroy(g);
        if (ei != cudaSuccess) return PRC_ERR_CUDA;
        ent.key = key;
        ent.device = dev;
        g_graphs.push_front(ent);
        while (g_graphs.size() > GRAPH_CACHE) {
            const GraphEntry& old = g_graphs.back();
            int cur = dev;
            if (old.device != cur) cudaSetDevice(old.device);
            cudaDeviceSynchronize();
            cudaGraphExecDestroy(old.exec);
            if (old.device != cur) cudaSetDevice(cur);
            g_graphs.pop_back();
        }
    }
    const GraphEntry& ent = g_graphs.front();
    {
        KernelScope scope("mg_solve_graph", run_st, ent.bytes, false);
        if (cudaGraphLaunch(ent.exec, run_st) != cudaSuccess) return PRC_ERR_CUDA;
    }
    add_launches(ent.launches);
    if (legacy &&
        (cudaEventRecord(side.out, side.s) != cudaSuccess || cudaStreamWaitEvent(st, side.out, 0) != cudaSuccess))
        return PRC_ERR_CUDA;
    return PRC_OK;
}

// Solve through the workspace: each problem's right-hand side is copied into its slot of level 0's f
// (FP64 f for the mixed precision solve), the (graph-captured) solve runs on the workspace alone,
// and each slot of level 0's v is copied out.
template <typename T>
int run_plain_io(const T* const* delta, T* const* phi, int count, const int32_t nmesh[3], const Params& P, void* ws,
                 const std::string& key, cudaStream_t st) {
    std::vector<LevelBufs<T>> B;
    plain_layout<T>(nmesh, (char*)ws, &B, nullptr, count);
    const int64_t N = (int64_t)nmesh[0] * nmesh[1] * nmesh[2];
    for (int b = 0; b < count; b++)
        if (cudaMemcpyAsync(B[0].f + b * N, delta[b], N * sizeof(T), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return PRC_ERR_CUDA;
    PRC_TRY(run_graph(key, st, [&](cudaStream_t s) { return solve_plain<T>(nmesh, P, ws, s, count); }));
    for (int b = 0; b < count; b++)
        if (cudaMemcpyAsync(phi[b], B[0].v + b * N, N * sizeof(T), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return PRC_ERR_CUDA;
    return PRC_OK;
}

int run_mixed_io(const float* const* delta, float* const* phi, double* const* phi64, int count, const int32_t nmesh[3],
                 const Params& P, void* ws, const std::string& key, cudaStream_t st) {
    MixedBufs m;
    mixed_layout(nmesh, (char*)ws, &m, count);
    const int64_t N = (int64_t)nmesh[0] * nmesh[1] * nmesh[2];
    for (int b = 0; b < count; b++)
        PRC_LAUNCH_B("mg_convert", st, 12.0 * N,
                     convert_kernel<float, double><<<grid_for(N), 256, 0, st>>>(delta[b], m.f64[0] + b * N, N));
    PRC_CHECK_LAUNCH();
    PRC_TRY(run_graph(key, st, [&](cudaStream_t s) { return solve_mixed(nmesh, P, ws, s, count); }));
    for (int b = 0; b < count; b++) {
        PRC_LAUNCH_B("mg_convert", st, 12.0 * N,
                     convert_kernel<double, float><<<grid_for(N), 256, 0, st>>>(m.v64[0] + b * N, phi[b], N));
        if (phi64 && phi64[b] &&
            cudaMemcpyAsync(phi64[b], m.v64[0] + b * N, N * sizeof(double), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return PRC_ERR_CUDA;
    }
    PRC_CHECK_LAUNCH();
    return PRC_OK;
}

// The batch shares one launch per step along z: count n0 planes (see cell3).
bool batch_ok(const int32_t nmesh[3], int count) { return count >= 1 && (int64_t)nmesh[0] * count <= 65535; }

}  // namespace

extern "C" {

size_t prc_multigrid_batch_workspace_bytes(const int32_t nmesh[3], int mesh_bytes, int mixed_precision, int count) {
    if (!nmesh || count < 1) return 0;
    for (int d = 0; d < 3; d++)
        if (nmesh[d] < 1) return 0;
    if (mesh_bytes == 4 && mixed_precision) return mixed_layout(nmesh, nullptr, nullptr, count);
    if (mesh_bytes == 4) return plain_layout<float>(nmesh, nullptr, nullptr, nullptr, count);
    return plain_layout<double>(nmesh, nullptr, nullptr, nullptr, count);
}

size_t prc_multigrid_workspace_bytes(const int32_t nmesh[3], int mesh_bytes, int mixed_precision) {
    return prc_multigrid_batch_workspace_bytes(nmesh, mesh_bytes, mixed_precision, 1);
}

prc_status_t prc_multigrid_batch_f32(const float* const* delta, float* const* phi, int count, const int32_t nmesh[3],
                                     const double boxsize[3], const double boxcenter[3], double beta, double damping,
                                     int jacobi_niterations, int vcycle_niterations, const double* los,
                                     int mixed_precision, void* workspace, size_t workspace_bytes, void* stream) {
    if (!delta || !phi || !batch_ok(nmesh, count)) return PRC_ERR_ARG;
    for (int b = 0; b < count; b++)
        if (!mg_args_ok(delta[b], phi[b], nmesh, boxsize, boxcenter, jacobi_niterations, vcycle_niterations))
            return PRC_ERR_ARG;
    Params P = make_params(boxsize, boxcenter, beta, damping, jacobi_niterations, vcycle_niterations, los);
    if (!workspace || workspace_bytes < prc_multigrid_batch_workspace_bytes(nmesh, 4, mixed_precision, count))
        return PRC_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const std::string key = solve_key(4, mixed_precision ? 1 : 0, nmesh, P, workspace, workspace_bytes, count);
    if (mixed_precision) return run_mixed_io(delta, phi, nullptr, count, nmesh, P, workspace, key, st);
    return run_plain_io<float>(delta, phi, count, nmesh, P, workspace, key, st);
}

prc_status_t prc_multigrid_batch_mixed_f32(const float* const* delta, float* const* phi, double* const* phi64,
                                           int count, const int32_t nmesh[3], const double boxsize[3],
                                           const double boxcenter[3], double beta, double damping,
                                           int jacobi_niterations, int vcycle_niterations, const double* los,
                                           void* workspace, size_t workspace_bytes, void* stream) {
    if (!delta || !phi || !batch_ok(nmesh, count)) return PRC_ERR_ARG;
    for (int b = 0; b < count; b++)
        if (!mg_args_ok(delta[b], phi[b], nmesh, boxsize, boxcenter, jacobi_niterations, vcycle_niterations))
            return PRC_ERR_ARG;
    Params P = make_params(boxsize, boxcenter, beta, damping, jacobi_niterations, vcycle_niterations, los);
    if (!workspace || workspace_bytes < prc_multigrid_batch_workspace_bytes(nmesh, 4, 1, count))
        return PRC_ERR_WORKSPACE;
    const std::string key = solve_key(4, 1, nmesh, P, workspace, workspace_bytes, count);
    return run_mixed_io(delta, phi, phi64, count, nmesh, P, workspace, key, (cudaStream_t)stream);
}

prc_status_t prc_multigrid_mixed_f32(const float* delta, float* phi, double* phi64, const int32_t nmesh[3],
                                     const double boxsize[3], const double boxcenter[3], double beta, double damping,
                                     int jacobi_niterations, int vcycle_niterations, const double* los,
                                     void* workspace, size_t workspace_bytes, void* stream) {
    return prc_multigrid_batch_mixed_f32(&delta, &phi, &phi64, 1, nmesh, boxsize, boxcenter, beta, damping,
                                         jacobi_niterations, vcycle_niterations, los, workspace, workspace_bytes,
                                         stream);
}

prc_status_t prc_multigrid_batch_f64(const double* const* delta, double* const* phi, int count,
                                     const int32_t nmesh[3], const double boxsize[3], const double boxcenter[3],
                                     double beta, double damping, int jacobi_niterations, int vcycle_niterations,
                                     const double* los, void* workspace, size_t workspace_bytes, void* stream) {
    if (!delta || !phi || !batch_ok(nmesh, count)) return PRC_ERR_ARG;
    for (int b = 0; b < count; b++)
        if (!mg_args_ok(delta[b], phi[b], nmesh, boxsize, boxcenter, jacobi_niterations, vcycle_niterations))
            return PRC_ERR_ARG;
    Params P = make_params(boxsize, boxcenter, beta, damping, jacobi_niterations, vcycle_niterations, los);
    if (!workspace || workspace_bytes < prc_multigrid_batch_workspace_bytes(nmesh, 8, 0, count)) return PRC_ERR_WORKSPACE;
    const std::string key = solve_key(8, 0, nmesh, P, workspace, workspace_bytes, count);
    return run_plain_io<double>(delta, phi, count, nmesh, P, workspace, key, (cudaStream_t)stream);
}

prc_status_t prc_multigrid_f32(const float* delta, float* phi, const int32_t nmesh[3], const double boxsize[3],
                               const double boxcenter[3], double beta, double damping, int jacobi_niterations,
                               int vcycle_niterations, const double* los, int mixed_precision, void* workspace,
                               size_t workspace_bytes, void* stream) {
    return prc_multigrid_batch_f32(&delta, &phi, 1, nmesh, boxsize, boxcenter, beta, damping, jacobi_niterations,
                                   vcycle_niterations, los, mixed_precision, workspace, workspace_bytes, stream);
}

prc_status_t prc_multigrid_f64(const double* delta, double* phi, const int32_t nmesh[3], const double boxsize[3],
                               const double boxcenter[3], double beta, double damping, int jacobi_niterations,
                               int vcycle_niterations, const double* los, void* workspace, size_t workspace_bytes,
                               void* stream) {
    return prc_multigrid_batch_f64(&delta, &phi, 1, nmesh, boxsize, boxcenter, beta, damping, jacobi_niterations,
                                   vcycle_niterations, los, workspace, workspace_bytes, stream);
}

#define MG_COMPONENTS(SUF, T)                                                                                        \
    prc_status_t prc_mg_jacobi_##SUF(T* v, const T* f, T* scratch, const int32_t nmesh[3], const double boxsize[3], \
                                     const double boxcenter[3], double beta, double damping, int niterations,       \
                                     const double* los, void* stream) {                                             \
        if (!v || !f || !scratch || !nmesh || !boxsize || !boxcenter || niterations < 0) return PRC_ERR_ARG;        \
        MGRunner<T> R;                                                                                               \
        R.L = hierarchy(nmesh);                                                                                      \
        R.P = make_params(boxsize, boxcenter, beta, damping, niterations, 0, los);                                  \
        R.st = (cudaStream_t)stream;                                                                                 \
        T *cur = v, *other = scratch;                                                                                \
        PRC_TRY(R.jacobi(0, cur, f, other, niterations, false));                                                     \
        if (cur != v && cudaMemcpyAsync(v, cur, (size_t)R.L[0].size() * sizeof(T), cudaMemcpyDeviceToDevice,       \
                                        (cudaStream_t)stream) != cudaSuccess)                                        \
            return PRC_ERR_CUDA;                                                                                     \
        return PRC_OK;                                                                                               \
    }                                                                                                                \
    prc_status_t prc_mg_residual_##SUF(const T* v, const T* f, T* r, const int32_t nmesh[3],                        \
                                       const double boxsize[3], const double boxcenter[3], double beta,             \
                                       const double* los, void* stream) {                                           \
        if (!v || !f || !r || !nmesh || !boxsize || !boxcenter) return PRC_ERR_ARG;                                 \
        int n[3] = {nmesh[0], nmesh[1], nmesh[2]};                                                                   \
        Stencil<T> s = make_stencil<T>(n, boxsize, boxcenter, beta, los);                                            \
        const double bytes = 3.0 * sizeof(T) * n[0] * n[1] * n[2];                                                   \
        if (quad_ok(n, v, f, r) && march_ok(s, 1, OP_RESIDUAL))                                                             \
            PRC_LAUNCH_B("mg_residual", (cudaStream_t)stream, bytes,                                                 \
                         (launch_march<T, T, OP_RESIDUAL>(v, f, r, nullptr, s, (T)0, 1, (cudaStream_t)stream)));   \
        else if (quad_ok(n, v, f, r))                                                                                     \
            PRC_LAUNCH_B("mg_residual", (cudaStream_t)stream, bytes,                                                 \
                         residual4_kernel<T, T>(mg_mode(s))                                              \
                             <<<grid3_quad(n).grid, grid3_quad(n).block, 0, (cudaStream_t)stream>>>(v, f, r, s));     \
        else                                                                                                         \
            PRC_LAUNCH_B("mg_residual", (cudaStream_t)stream, bytes,                                                 \
                         residual_kernel<T, T, T, T, T><<<grid3(n).grid, grid3(n).block, 0, (cudaStream_t)stream>>>(  \
                             v, f, r, s));                                                                           \
        PRC_CHECK_LAUNCH();                                                                                          \
        return PRC_OK;                                                                                               \
    }                                                                                                                \
    prc_status_t prc_mg_reduce_##SUF(const T* fine, T* coarse, const int32_t nf[3], void* stream) {                 \
        if (!fine || !coarse || !nf) return PRC_ERR_ARG;                                                             \
        const int n[3] = {nf[0], nf[1], nf[2]};                                                                       \
        PRC_LAUNCH("mg_reduce", (cudaStream_t)stream,                                                                \
                   launch_reduce(fine, coarse, n, 1, (cudaStream_t)stream)); \
        PRC_CHECK_LAUNCH();                                                                                          \
        return PRC_OK;                                                                                               \
    }                                                                                                                \
    prc_status_t prc_mg_prolong_##SUF(const T* coarse, T* fine, const int32_t nc[3], void* stream) {                \
        if (!fine || !coarse || !nc) return PRC_ERR_ARG;                                                             \
        const int n[3] = {nc[0], nc[1], nc[2]};                                                                       \
        PRC_LAUNCH("mg_prolong", (cudaStream_t)stream,                                                               \
                   (launch_prolong<T, false>(coarse, fine, n, 1, (cudaStream_t)stream))); \
        PRC_CHECK_LAUNCH();                                                                                          \
        return PRC_OK;                                                                                               \
    }

MG_COMPONENTS(f32, float)
MG_COMPONENTS(f64, double)

}  // extern "C"
