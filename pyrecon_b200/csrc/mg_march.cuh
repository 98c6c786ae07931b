// The 19-point operator (local or oblique line of sight) at a cell, and the kernel that marches it along x (included by
// multigrid.cu).
//
// With q = sum_a h_a^2 p_a^2 (so g = beta / q), P = sum_a p_a^2, s_a = p_a^2:
//   U = sum_a (v+a + v-a) / h_a^2
//   W = sum_a s_a (v+a + v-a) + 1/2 sum_{a<b} p_a p_b e_ab [+ sum_a p_a (v+a - v-a), local]
//   S(v) = U + g W,   2 sum_a G_a = 2 (sum_a 1/h_a^2 + g P),
//   damped Jacobi: v + w (num / den - v), num = q (f + U) + beta W, den = 2 (q sum 1/h^2 + beta P),
//   residual: (f + U - 2 v sum 1/h^2) + g (W - 2 P v).
// Every product that meets an addition is an explicit fma and every other one is kept from contraction, in one order, so
// every kernel (four cells a thread, marched, two sweeps a pass) gives the same bits per cell, FP32 and FP64.
#pragma once

namespace prc {

__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// Scalars of a level.
template <typename A> struct OpCoef {
    A ih0, ih1, ih2, h20, h21, h22, off0, off1, off2, beta, beta2, sih2;   // 2 beta, 2 sum 1/h^2
};
// Terms that depend on x and y only.
template <typename A> struct XYCoef {
    A s0, s1, ap, am, bp, bm, q01, P01, e01, hp0, hp1;
};

template <bool LOCAL, typename A> __device__ __forceinline__ OpCoef<A> op_coef(const Stencil<A>& s) {
    OpCoef<A> k;
    k.ih0 = s.ih2[0], k.ih1 = s.ih2[1], k.ih2 = s.ih2[2];
    k.h20 = s.h2[0], k.h21 = s.h2[1], k.h22 = s.h2[2];
    k.off0 = LOCAL ? s.off[0] : s.losh[0];
    k.off1 = LOCAL ? s.off[1] : s.losh[1];
    k.off2 = LOCAL ? s.off[2] : s.losh[2];
    k.beta = s.beta;
    k.beta2 = rn_mul((A)2, s.beta);
    k.sih2 = rn_mul((A)2, rn_add(rn_add(s.ih2[0], s.ih2[1]), s.ih2[2]));
    return k;
}

template <bool LOCAL, typename A> __device__ __forceinline__ XYCoef<A> xy_coef(const OpCoef<A>& k, int x, int y) {
    XYCoef<A> c;
    const A p0 = LOCAL ? rn_add((A)x, k.off0) : k.off0;
    const A p1 = LOCAL ? rn_add((A)y, k.off1) : k.off1;
    c.s0 = rn_mul(p0, p0), c.s1 = rn_mul(p1, p1);
    c.ap = rn_add(c.s0, p0), c.am = rn_sub(c.s0, p0);
    c.bp = rn_add(c.s1, p1), c.bm = rn_sub(c.s1, p1);
    c.q01 = fma_rn(k.h21, c.s1, rn_mul(k.h20, c.s0));
    c.P01 = rn_add(c.s0, c.s1);
    c.hp0 = rn_mul((A)0.5, p0), c.hp1 = rn_mul((A)0.5, p1);
    c.e01 = rn_mul(c.hp0, p1);
    return c;
}

// p2 of a cell, counted from the multiple of four cells below it.
template <bool LOCAL, typename A> __device__ __forceinline__ A z_p2(const OpCoef<A>& k, int z) {
    return LOCAL ? rn_add(rn_add((A)(z & ~3), k.off2), (A)(z & 3)) : k.off2;
}

// FP32: the hardware reciprocal (1 ulp; its argument is a sum of squares of cell numbers, far from the subnormals).
__device__ __forceinline__ float rcp_approx(float a) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// ---- two cells at once ----
// FP32 pairs go through the packed instructions (one issue slot for two cells, the same rounding per cell; a 512^3
// sweep 330 us against 350 with scalar ones), FP64 pairs through two scalar ones.
template <typename A> struct Pair;
template <> struct Pair<float> {
    typedef float2 T;
    static __device__ __forceinline__ T make(float a, float b) { return make_float2(a, b); }
    static __device__ __forceinline__ T all(float a) { return make_float2(a, a); }
    static __device__ __forceinline__ T div_sub(T a, T b, T c) { return fma(a, make(rcp_approx(b.x), rcp_approx(b.y)), make(-c.x, -c.y)); }
    static __device__ __forceinline__ T div(float a, T b) { return mul(all(a), make(rcp_approx(b.x), rcp_approx(b.y))); }
    static __device__ __forceinline__ T add(T a, T b) { return __fadd2_rn(a, b); }
    static __device__ __forceinline__ T sub(T a, T b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
    static __device__ __forceinline__ T mul(T a, T b) { return __fmul2_rn(a, b); }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return __ffma2_rn(a, b, c); }
};
template <> struct Pair<double> {
    typedef double2 T;
    static __device__ __forceinline__ T make(double a, double b) { return make_double2(a, b); }
    static __device__ __forceinline__ T all(double a) { return make_double2(a, a); }
    static __device__ __forceinline__ T div_sub(T a, T b, T c) { return sub(make(a.x / b.x, a.y / b.y), c); }
    static __device__ __forceinline__ T div(double a, T b) { return make(a / b.x, a / b.y); }
    static __device__ __forceinline__ T add(T a, T b) { return make(rn_add(a.x, b.x), rn_add(a.y, b.y)); }
    static __device__ __forceinline__ T sub(T a, T b) { return make(rn_sub(a.x, b.x), rn_sub(a.y, b.y)); }
    static __device__ __forceinline__ T mul(T a, T b) { return make(rn_mul(a.x, b.x), rn_mul(a.y, b.y)); }
    static __device__ __forceinline__ T fma(T a, T b, T c) { return make(fma_rn(a.x, b.x, c.x), fma_rn(a.y, b.y, c.y)); }
};
// One cell, with the same operations.
template <typename A> struct One {
    typedef A T;
    static __device__ __forceinline__ A all(A a) { return a; }
    static __device__ __forceinline__ A add(A a, A b) { return rn_add(a, b); }
    static __device__ __forceinline__ A sub(A a, A b) { return rn_sub(a, b); }
    static __device__ __forceinline__ A mul(A a, A b) { return rn_mul(a, b); }
    static __device__ __forceinline__ A fma(A a, A b, A c) { return fma_rn(a, b, c); }
    static __device__ __forceinline__ A div_sub(A a, A b, A c) {
        if constexpr (sizeof(A) == 4) return fma_rn(a, rcp_approx(b), -c);
        else return rn_sub(a / b, c);
    }
    static __device__ __forceinline__ A div(A a, A b) {
        if constexpr (sizeof(A) == 4) return rn_mul(a, rcp_approx(b));
        else return a / b;
    }
};
template <typename A> __device__ __forceinline__ typename Pair<A>::T both(A a) { return Pair<A>::make(a, a); }

// U, W, q and P of the cells of ops O from their neighbours (xp .. zm) and edge sums e_ab.
template <bool LOCAL, typename O, typename A, typename V = typename O::T>
__device__ __forceinline__ void op_terms(const OpCoef<A>& k, const XYCoef<A>& c, V p2, V s2, V xp, V xm, V yp, V ym, V zp,
                                         V zm, V exy, V exz, V eyz, V& U, V& W, V& q, V& PP) {
    const V Sx = O::add(xp, xm), Sy = O::add(yp, ym), Sz = O::add(zp, zm);
    U = O::fma(O::all(k.ih0), Sx, O::mul(O::all(k.ih1), Sy));
    U = O::fma(O::all(k.ih2), Sz, U);
    if (LOCAL) {
        W = O::fma(O::all(c.ap), xp, O::mul(O::all(c.am), xm));
        W = O::fma(O::all(c.bp), yp, W);
        W = O::fma(O::all(c.bm), ym, W);
        W = O::fma(O::add(s2, p2), zp, W);
        W = O::fma(O::sub(s2, p2), zm, W);
    } else {
        W = O::fma(O::all(c.s0), Sx, O::mul(O::all(c.s1), Sy));
        W = O::fma(s2, Sz, W);
    }
    W = O::fma(O::all(c.e01), exy, W);
    W = O::fma(O::mul(O::all(c.hp0), p2), exz, W);
    W = O::fma(O::mul(O::all(c.hp1), p2), eyz, W);
    q = O::fma(O::all(k.h22), s2, O::all(c.q01));
    PP = O::add(O::all(c.P01), s2);
}

// The damped-Jacobi values v + w (num / den - v).
template <typename O, typename A, typename V = typename O::T>
__device__ __forceinline__ V op_jacobi(const OpCoef<A>& k, V f, V v, V U, V W, V q, V PP, A w) {
    const V num = O::fma(q, O::add(f, U), O::mul(O::all(k.beta), W));
    const V den = O::fma(q, O::all(k.sih2), O::mul(O::all(k.beta2), PP));
    return O::fma(O::all(w), O::div_sub(num, den, v), v);
}

// f - A v; t2 = W - 2 P v.
template <typename O, typename A, typename V = typename O::T>
__device__ __forceinline__ V op_residual_from(const OpCoef<A>& k, V f, V v, V U, V t2, V q) {
    const V t1 = O::fma(O::all(-k.sih2), v, O::add(f, U));
    return O::fma(O::div(k.beta, q), t2, t1);
}
template <typename O, typename A, typename V = typename O::T>
__device__ __forceinline__ V op_residual(const OpCoef<A>& k, V f, V v, V U, V W, V q, V PP) {
    return op_residual_from<O>(k, f, v, U, O::fma(O::mul(O::all((A)-2), PP), v, W), q);
}

// ---- the march ----
// One damped-Jacobi sweep or residual, 12 bytes of DRAM a cell in FP32.  The quad kernels it replaces were bound by
// instructions (nine columns of loads and their addresses).  Measured, local line of sight, FP32 sweep: 512^3 504 -> 330 us
// (4.9 TB/s, 75 % of the copy rate), 384^3 234 -> 154, 256^3 72 -> 52, 192^3 40 -> 22, 128^3 9.6 -> 8.7; FP64 sweep 384^3
// 560 -> 388, 256^3 167 -> 141; FP64 residual 384^3 615 -> 430.  Planes reach shared memory by 16-byte copies of the block's
// own threads: bulk copies issued by one thread of a computing warp held that warp, and through the release of stages the
// others, back (484 us at 512^3), one per row from a warp of its own was limited by their number (950 us).
// A thread owns VZ adjacent cells along z (one 16-byte vector) of one row y and walks a slab of planes, so per plane only
// the three rows y - 1, y, y + 1 of plane x + 1 are read (the rows of planes x - 1 and x are in registers): a quad that
// loads its nine columns spends ~100 instructions a cell, a marched one ~50.  z neighbours come by shuffle; the first
// and last lane of a segment read their outer neighbour's column.
// ---- vectors of VZ cells ----
template <typename A, int NP> __device__ __forceinline__ void smem_pairs(const A* p, typename Pair<A>::T (&o)[NP]) {
    if constexpr (sizeof(A) == 4) {
        const float4 a = *(const float4*)p;
        o[0] = make_float2(a.x, a.y), o[1] = make_float2(a.z, a.w);
    } else {
        o[0] = *(const double2*)p;
    }
}
template <typename T, int VZ> __device__ __forceinline__ void smem_vec(const T* p, T (&o)[VZ]) {
    if constexpr (sizeof(T) == 4) {
        static_assert(VZ == 4, "vector of four floats");
        const float4 a = *(const float4*)p;
        o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w;
    } else {
        static_assert(VZ == 2, "vector of two doubles");
        const double2 a = *(const double2*)p;
        o[0] = a.x, o[1] = a.y;
    }
}
template <typename T, int VZ> __device__ __forceinline__ void storev(T* p, const T (&o)[VZ]) {
    if constexpr (sizeof(T) * VZ == 16 && sizeof(T) == 4) *(float4*)p = make_float4(o[0], o[1], o[2], o[3]);
    else if constexpr (sizeof(T) * VZ == 16) *(double2*)p = make_double2(o[0], o[1]);
    else *(float2*)p = make_float2(o[0], o[1]);
}

enum { OP_JACOBI = 0, OP_RESIDUAL = 1, OP_JACOBI_ADD = 2 };

template <typename A> struct MarchVZ { static constexpr int value = 16 / (int)sizeof(A); };

constexpr int MARCH_THREADS = 256;
constexpr int MARCH_STAGES = 5;           // ring of planes in shared memory
constexpr int MARCH_FILL = 4;             // plane steps a wave of blocks costs beside its slab (march_split)

// How a march is split (march_split): a tile is TZ = LZ VZ cells along z (the last segment of a row ends with the row)
// of 256 / LZ rows, a block a tile through a slab of `slab` planes (the last slab ends with the mesh).
struct MarchSplit {
    int lz, zsegs, ytiles, slab, nslab;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <typename A, int LZ> struct MarchTile {
    static constexpr int VZ = MarchVZ<A>::value, TZ = LZ * VZ, ROWS = MARCH_THREADS / LZ;
    static constexpr int PITCH = (TZ + 2 * VZ) * (int)sizeof(A);      // bytes of a staged row: halo, segment, halo
    static constexpr int F_AT = (ROWS + 2) * PITCH, STAGE = F_AT + MARCH_THREADS * 16;
};

// Step k stages plane x0 - 1 + k of v (the tile's rows and the two beside them, with a vector of halo on either side
// unless the segment is the whole row) and, from k = 2 on, the tile's cells of plane x0 - 2 + k of f, by 16-byte
// asynchronous copies of the block's threads, MARCH_STAGES - 1 steps ahead; one block barrier a step.
// OP_JACOBI: out = damped-Jacobi value.  OP_RESIDUAL: out = f - A v.  OP_JACOBI_ADD: acc += the damped-Jacobi
// value (the last sweep of a correction V-cycle adds its result to the FP64 iterate), out unused.
template <typename A, typename OT, int LZ, bool LOCAL, int OP>
__global__ void __launch_bounds__(MARCH_THREADS, 2)
    march_kernel(const A* __restrict__ v, const A* __restrict__ f, OT* __restrict__ out, double* __restrict__ acc,
                 Stencil<A> s, A w, MarchSplit sp) {
    pdl_trigger();
    typedef MarchTile<A, LZ> T;
    constexpr int VZ = T::VZ, TZ = T::TZ, PITCH = T::PITCH;
    extern __shared__ __align__(128) unsigned char march_smem[];
    const int n0 = s.n[0], n1 = s.n[1], n2 = s.n[2];
    const int tid = threadIdx.x, lane = tid % LZ, rr = tid / LZ;
    const int64_t sx = (int64_t)n1 * n2, N = n0 * sx;
    const int prob = blockIdx.z / sp.nslab, is = blockIdx.z - prob * sp.nslab;
    const int x_own = is * sp.slab, x0 = min(x_own, n0 - sp.slab), x1 = x0 + sp.slab;
    const int y0 = blockIdx.y * T::ROWS, y = y0 + rr;
    const int z_own = blockIdx.x * TZ, zs = min(z_own, n2 - TZ), z0 = zs + lane * VZ;
    const bool mine = y < n1 && z0 >= z_own;
    auto wrap_row = [&](int r) {       // row of the mesh at staged row r (rows past the mesh wrap, and are not used)
        int q = y0 - 1 + r;
        if (q < 0) q += n1;
        while (q >= n1) q -= n1;
        return q;
    };
    // this thread's copies of a plane: its own cell vector of v and f, and (the first threads) one of the outer ones
    const int64_t own_off = (int64_t)wrap_row(rr + 1) * n2 + z0;
    const int own_at = (rr + 1) * PITCH + (lane + 1) * 16;
    int64_t ext_off = 0;
    int ext_at = -1;
    if (tid < 2 * LZ) {
        const int r = tid < LZ ? 0 : T::ROWS + 1;
        ext_off = (int64_t)wrap_row(r) * n2 + z0;
        ext_at = r * PITCH + (lane + 1) * 16;
    } else if (sp.zsegs > 1 && tid < 2 * LZ + 2 * (T::ROWS + 2)) {
        const int e = tid - 2 * LZ, r = e >> 1;
        const int z = (e & 1) ? (zs + TZ == n2 ? 0 : zs + TZ) : (zs == 0 ? n2 - VZ : zs - VZ);
        ext_off = (int64_t)wrap_row(r) * n2 + z;
        ext_at = r * PITCH + ((e & 1) ? (LZ + 1) * 16 : 0);
    }
    const int steps = sp.slab + 2;
    int xs = x0 == 0 ? n0 - 1 : x0 - 1, issued = 0, ist = 0;
    const A* vp = v + prob * N + xs * sx;
    const A* fp = f + prob * N + (x0 - 2) * sx + own_off;
    pdl_wait();
    auto issue = [&]() {
        if (issued < steps) {
            unsigned char* dst = march_smem + ist * T::STAGE;
            cp_async16(dst + own_at, vp + own_off);
            if (ext_at >= 0) cp_async16(dst + ext_at, vp + ext_off);
            if (issued >= 2) cp_async16(dst + T::F_AT + tid * 16, fp);
            vp += sx;
            fp += sx;
            if (++xs == n0) xs = 0, vp -= N;
            issued++;
            if (++ist == MARCH_STAGES) ist = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < MARCH_STAGES - 1; i++) issue();
    const bool edge_l = lane == 0, edge_r = lane == LZ - 1, edge = edge_l || edge_r;
    // the edge lanes' outer column, relative to their own vector
    const int zh = (edge_l ? (sp.zsegs == 1 ? TZ - 1 : -1) : (sp.zsegs == 1 ? 0 : TZ)) - lane * VZ;
    typedef Pair<A> P;
    typedef typename P::T P2;
    constexpr int NP = VZ / 2;
    const OpCoef<A> k = op_coef<LOCAL>(s);

    // planes in flight, by plane index mod 3: the rows y, y + 1, y - 1 and the cells beside this thread's in each
    P2 C[3][NP], Yp[3][NP], Ym[3][NP];
    A cl[3], cr[3], pl[3], pr[3], ml[3], mr[3];
    int stage = 0;
    // reads the next plane into slot i (and its f cells into fv), and sends for the one MARCH_STAGES - 1 steps ahead into
    // the stage that every thread read before this step's barrier
    auto take = [&](int i, P2 (&fv)[NP], bool with_f) {
        asm volatile("cp.async.wait_group %0;" ::"n"(MARCH_STAGES - 2) : "memory");
        __syncthreads();
        issue();
        const unsigned char* r = march_smem + stage * T::STAGE + own_at;
        smem_pairs<A, NP>((const A*)r, C[i]);
        smem_pairs<A, NP>((const A*)(r + PITCH), Yp[i]);
        smem_pairs<A, NP>((const A*)(r - PITCH), Ym[i]);
        A hc = (A)0, hp = (A)0, hm = (A)0;
        if (edge) {
            const A* h = (const A*)r + zh;
            hc = h[0];
            hp = h[PITCH / (int)sizeof(A)];
            hm = h[-(PITCH / (int)sizeof(A))];
        }
        if (with_f) smem_pairs<A, NP>((const A*)(march_smem + stage * T::STAGE + T::F_AT + tid * 16), fv);
        auto beside = [&](const P2 (&a)[NP], A h, A& l, A& g) {
            l = __shfl_up_sync(0xffffffffu, a[NP - 1].y, 1, LZ);
            g = __shfl_down_sync(0xffffffffu, a[0].x, 1, LZ);
            if (edge_l) l = h;
            if (edge_r) g = h;
        };
        beside(C[i], hc, cl[i], cr[i]);
        beside(Yp[i], hp, pl[i], pr[i]);
        beside(Ym[i], hm, ml[i], mr[i]);
        if (++stage == MARCH_STAGES) stage = 0;
    };
    P2 fv[NP], p2[NP], s2[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
        p2[i] = P::make(z_p2<LOCAL>(k, z0 + 2 * i), z_p2<LOCAL>(k, z0 + 2 * i + 1));
        s2[i] = P::mul(p2[i], p2[i]);
    }
    take(2, fv, false);
    take(0, fv, false);
    int64_t io = prob * N + x0 * sx + (int64_t)y * n2 + z0;
    for (int xb = x0; xb < x1; xb += 3) {
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const int x = xb + u;
            if (x >= x1) break;
            const int im = (u + 2) % 3, ip = (u + 1) % 3;
            take(ip, fv, true);
            const XYCoef<A> c = xy_coef<LOCAL>(k, x, y);
            A o[VZ];
#pragma unroll
            for (int j = 0; j < NP; j++) {
                // cells j - 1 and j + 2 of a row: the next pair's, or the neighbour thread's
                auto before = [&](const P2 (&a)[NP], A l) { return j == 0 ? l : a[j == 0 ? 0 : j - 1].y; };
                auto after = [&](const P2 (&a)[NP], A g) { return j == NP - 1 ? g : a[j == NP - 1 ? 0 : j + 1].x; };
                const P2 zp = P::make(C[u][j].y, after(C[u], cr[u])), zm = P::make(before(C[u], cl[u]), C[u][j].x);
                const P2 exy = P::sub(P::add(Yp[ip][j], Ym[im][j]), P::add(Yp[im][j], Ym[ip][j]));
                const A xpl = before(C[ip], cl[ip]), xpr = after(C[ip], cr[ip]);
                const A xml = before(C[im], cl[im]), xmr = after(C[im], cr[im]);
                const P2 exz = P::make(rn_sub(rn_add(C[ip][j].y, xml), rn_add(C[im][j].y, xpl)),
                                       rn_sub(rn_add(xpr, C[im][j].x), rn_add(xmr, C[ip][j].x)));
                const A ypl = before(Yp[u], pl[u]), ypr = after(Yp[u], pr[u]);
                const A yml = before(Ym[u], ml[u]), ymr = after(Ym[u], mr[u]);
                const P2 eyz = P::make(rn_sub(rn_add(Yp[u][j].y, yml), rn_add(Ym[u][j].y, ypl)),
                                       rn_sub(rn_add(ypr, Ym[u][j].x), rn_add(ymr, Yp[u][j].x)));
                P2 U, W, q, PP;
                op_terms<LOCAL, P>(k, c, p2[j], s2[j], C[ip][j], C[im][j], Yp[u][j], Ym[u][j], zp, zm, exy, exz, eyz, U, W, q,
                                PP);
                const P2 r = OP == OP_RESIDUAL ? op_residual<P>(k, fv[j], C[u][j], U, W, q, PP)
                                               : op_jacobi<P>(k, fv[j], C[u][j], U, W, q, PP, w);
                o[2 * j] = r.x, o[2 * j + 1] = r.y;
            }
            if (mine && x >= x_own) {
                if constexpr (OP == OP_JACOBI_ADD) {
                    double* a = acc + io;
#pragma unroll
                    for (int j = 0; j < VZ; j += 2) {
                        double2 t = *(double2*)(a + j);
                        t.x += (double)o[j], t.y += (double)o[j + 1];
                        *(double2*)(a + j) = t;
                    }
                } else {
                    OT oo[VZ];
#pragma unroll
                    for (int j = 0; j < VZ; j++) oo[j] = (OT)o[j];
                    storev<OT, VZ>(out + io, oo);
                }
            }
            io += sx;
        }
    }
}

// Lanes a row of a march over rows of n2 cells: the power of two that computes the least, each segment's halo counted (a
// segment that is the whole row has none); 0 where a row does not hold a tile.  cells: what a row then computes and stages.
template <typename A> static int march_lanes(int n2, int* cells) {
    constexpr int VZ = MarchVZ<A>::value;
    int best = 0;
    *cells = 0;
    for (int lz = 32; lz >= 4; lz >>= 1) {
        const int tz = lz * VZ, c = (n2 + tz - 1) / tz * (tz + 2 * VZ);
        if (tz <= n2 && (best == 0 || c < *cells)) best = lz, *cells = c;
    }
    if (best * VZ == n2) *cells = n2;
    return best;
}

// The split of a march over `count` meshes of shape n, or lz = 0 where a row does not hold a tile.
template <typename A> static MarchSplit march_split(const int n[3], int count) {
    MarchSplit sp = {};
    constexpr int VZ = MarchVZ<A>::value;
    int cells;
    sp.lz = march_lanes<A>(n[2], &cells);
    if (sp.lz == 0) return sp;
    const int tz = sp.lz * VZ, rows = MARCH_THREADS / sp.lz;
    sp.zsegs = (n[2] + tz - 1) / tz;
    sp.ytiles = (n[1] + rows - 1) / rows;
    // the slab length whose waves of blocks (two a SM) take the fewest plane steps; a block's two outer planes and the
    // fill of its pipeline count MARCH_FILL.  Each length once, from the longest down: 2 sqrt(n0) of them, on every launch.
    const int64_t slots = 2 * (int64_t)device_sm_count(), tiles = (int64_t)sp.zsegs * sp.ytiles * count;
    int64_t best = 0;
    for (int slab = n[0];;) {
        const int real = (n[0] + slab - 1) / slab;
        const int64_t cost = (tiles * real + slots - 1) / slots * (slab + MARCH_FILL);
        if (best == 0 || cost < best) best = cost, sp.slab = slab, sp.nslab = real;
        if (slab == 1) break;
        const int more = (n[0] + slab - 2) / (slab - 1);       // the fewest slabs shorter than this one
        slab = (n[0] + more - 1) / more;
    }
    return sp;
}

}  // namespace prc
