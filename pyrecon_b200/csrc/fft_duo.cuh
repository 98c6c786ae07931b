// FP32 strided passes on pairs of columns (included by fft.cu after fft_tma.cuh).
//
// The TMA-fed passes of fft_tma.cuh hold one column's 8 points in a thread and are bound by shared-memory instructions
// and barriers, not by DRAM.  Here a thread holds the same 8 points t + i N / 8 of two adjacent columns: an exchange
// moves 16 bytes an access (half the shared-memory instructions a point), twiddles and addresses serve two columns,
// and a tile has half the threads, so two or more blocks with their own barriers share an SM.  The arithmetic of a
// column, its order included, is that of pass_regs and the kernels of fft_tma.cuh: the same bits.
//
// Measured per nmesh-512 reconstruction of the local-line-of-sight iteration, against one column a thread:
// k-space pass 4.29 -> 3.45 ms (3.1 TB/s), Hessian pass 3.80 -> 3.15 ms (3.1 TB/s), y forward 1.41 -> 1.18 and y inverse
// 1.15 -> 0.98 ms (5.5 TB/s).  The strided pass is within a fifth of a copy; the other two are bound by issue slots and
// shared memory (46 instructions a point and transform, issue slots 53 to 57 % busy, then stalls on shared-memory
// results), not by DRAM.
#pragma once

namespace fast {

struct alignas(16) Duo {
    float2 a, b;       // columns 2 q and 2 q + 1 of a tile
};

// pass_regs on two columns.
template <int N, int R, int NS, int DIR>
__device__ __forceinline__ void pass_duo(float2 (&va)[8], float2 (&vb)[8], int t, const float2* __restrict__ tw) {
    typedef float2 C;
    constexpr int T = N / 8, NB = 8 / R;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        C ua[R], ub[R];
#pragma unroll
        for (int r = 0; r < R; r++) ua[r] = va[b + r * NB], ub[r] = vb[b + r * NB];
        if constexpr (NS > 1) {
            const int k = (t + b * T) & (NS - 1);
            const C* row = tw + k * (R - 1);
            if constexpr (R == 8 && PRC_TW_RECUR) {
                C w[8];
                w[1] = row[0];
                w[2] = row[1];
                w[4] = row[3];
                if (DIR > 0) {
                    w[1] = cconj(w[1]);
                    w[2] = cconj(w[2]);
                    w[4] = cconj(w[4]);
                }
                w[3] = cmul(w[1], w[2]);
                w[5] = cmul(w[1], w[4]);
                w[6] = cmul(w[2], w[4]);
                w[7] = cmul(w[3], w[4]);
#pragma unroll
                for (int r = 1; r < 8; r++) ua[r] = cmul(ua[r], w[r]), ub[r] = cmul(ub[r], w[r]);
            } else {
#pragma unroll
                for (int r = 1; r < R; r++) {
                    C w = row[r - 1];
                    if (DIR > 0) w = cconj(w);
                    ua[r] = cmul(ua[r], w), ub[r] = cmul(ub[r], w);
                }
            }
        }
        dftR<C, DIR, R>(ua);
        dftR<C, DIR, R>(ub);
#pragma unroll
        for (int r = 0; r < R; r++) va[b + r * NB] = ua[r], vb[b + r * NB] = ub[r];
    }
}

// exchange_pp on two columns.
template <int N, int R, int NS, class Addr>
__device__ __forceinline__ void exchange_duo(float2 (&va)[8], float2 (&vb)[8], int t, Duo* s, const Addr& addr) {
    constexpr int T = N / 8, NB = 8 / R;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        const int j = t + b * T;
        const int k = j & (NS - 1);
        const int base = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) s[addr(base + r * NS)] = Duo{va[b + r * NB], vb[b + r * NB]};
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const Duo d = s[addr(t + i * T)];
        va[i] = d.a, vb[i] = d.b;
    }
}

template <int N, int DIR, int P> struct PassesDuo {
    template <class Addr0, class Addr1>
    static __device__ __forceinline__ void run(float2 (&va)[8], float2 (&vb)[8], int t, Duo* s0, const Addr0& addr0,
                                               Duo* s1, const Addr1& addr1, const float2* tw) {
        constexpr int R = TwLayout<N>::radix(P);
        constexpr int NS = ipow8(P);
        pass_duo<N, R, NS, DIR>(va, vb, t, tw + TwLayout<N>::offset(P));
        if constexpr (P + 1 < Plan<N>::NPASS) {
            if constexpr (P % 2 == 0) exchange_duo<N, R, NS>(va, vb, t, s0, addr0);
            else exchange_duo<N, R, NS>(va, vb, t, s1, addr1);
            PassesDuo<N, DIR, P + 1>::run(va, vb, t, s0, addr0, s1, addr1, tw);
        }
    }
};

// fft_regs_pp on two columns (the same contract for s0 and s1).
template <int N, int DIR, class Addr0, class Addr1>
__device__ __forceinline__ void fft_duo(float2 (&va)[8], float2 (&vb)[8], int t, Duo* s0, const Addr0& addr0, Duo* s1,
                                        const Addr1& addr1, const float2* tw) {
    PassesDuo<N, DIR, 0>::run(va, vb, t, s0, addr0, s1, addr1, tw);
}

// Pairs of a tile: BP pairs a row of BP * 16 bytes.  A tile of 64-byte rows pads the buffer of the first exchange
// (PadAddr: the first Stockham pass writes rows 8 t + r).
template <int BP> struct PairAddr {
    int q;
    __device__ __forceinline__ int operator()(int k) const { return k * BP + q; }
};
template <int BP> struct PadPairAddr {
    int q;
    __device__ __forceinline__ int operator()(int k) const { return (k + (k >> 3)) * BP + q; }
};
template <int N, int BP> struct DuoTile {
    static constexpr int ELEMS = N * BP, PADDED = BP <= 4 ? (N + N / 8) * BP : N * BP;      // Duo values
    static constexpr int THREADS = N / 8 * BP;
};

// Columns 2 q and 2 q + 1 of a row stored at g, the ones below the spectrum's width.
__device__ __forceinline__ void store_duo(float2* g, float2 a, float2 b, bool oka, bool okb) {
    if (okb) *(float4*)g = make_float4(a.x, a.y, b.x, b.y);
    else if (oka) *g = a;
}

// ---- x pass with the k-space step (x_kspace_tma on pairs) ----
// One stage: a tile is in registers after the first exchange, and the next one arrives while this one's outputs are
// transformed back.  Shared memory: the stage, two exchange buffers, the twiddles.
template <int N, int BP> struct KSpaceDuoSmem {
    typedef DuoTile<N, BP> DT;
    static constexpr size_t BYTES = (size_t)(2 * DT::ELEMS + DT::PADDED) * sizeof(Duo) + (size_t)N * sizeof(float2) + 16;
};

// KLine's multipliers m (or i m) of one column, one real number a point, with the roundings that the one-column kernel
// gets from the compiler written out (a change of them moves the displacements by 1e-7).  A line has N points, so point
// t + i N / 8 has the wavenumber index t + i N / 8 (- N from i = 4 on) and the Nyquist point is t = 0, i = 4.
template <int N, int KT> struct KDuo {
    static constexpr bool IMAG = KT == KOP_PSI || KT == KOP_PP;
    float ky, kz, a[8], b[KT == KOP_PP ? 8 : 1];
    bool nyqy, nyqz;

    static __device__ __forceinline__ float kx(const KOp& op, int t, int i) {
        return __fmul_rn((float)6.283185307179586, __fmul_rn((float)t + (float)(i * (N / 8) - (i < 4 ? 0 : N)), (float)op.fscale[0]));
    }
    static __device__ __forceinline__ float dot(const KOp& op, float x, float y, float z) {
        return __fadd_rn(__fmul_rn(z, (float)op.los[2]), __fmaf_rn(x, (float)op.los[0], __fmul_rn(y, (float)op.los[1])));
    }
    __device__ __forceinline__ void setup(const KOp& op, const Dims& dims, int t, int iy, int iz) {
        const float norm = (float)op.norm, beta = (float)op.beta;
        ky = kval<float>(iy, dims.n[1], (float)op.fscale[1]);
        kz = kval<float>(iz, dims.n[2], (float)op.fscale[2]);
        nyqy = nyquist(iy, dims.n[1]), nyqz = nyquist(iz, dims.n[2]);
        const float ky2 = __fmul_rn(ky, ky), kz2 = __fmul_rn(kz, kz);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float x = kx(op, t, i);
            const float k2 = KT == KOP_HESS3 ? __fadd_rn(kz2, __fadd_rn(ky2, __fmul_rn(x, x)))
                                             : __fadd_rn(kz2, __fmaf_rn(x, x, ky2));
            const bool zero = i == 0 && t == 0 && iy == 0 && iz == 0;
            if constexpr (KT == KOP_PP) {
                const float tx = i == 4 && t == 0 ? x : -x;
                const float kl = dot(op, x, ky, kz), klt = dot(op, tx, nyqy ? ky : -ky, nyqz ? kz : -kz);
                a[i] = zero ? 0.f : 1.f / __fmaf_rn(beta, __fmul_rn(kl, kl), k2);
                b[i] = zero ? 0.f : 1.f / __fmaf_rn(beta, __fmul_rn(klt, klt), k2);
            } else {
                a[i] = zero ? 0.f : norm / k2;
            }
        }
    }
    __device__ __forceinline__ void multipliers(const KOp& op, int t, int o, float (&m)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float x = kx(op, t, i);
            const bool nyqx = i == 4 && t == 0;
            if constexpr (KT == KOP_PSI) {
                // (k - t) / 2, t = -k but k on the Nyquist index
                m[i] = __fmul_rn(o == 0 ? (nyqx ? 0.f : x) : o == 1 ? (nyqy ? 0.f : ky) : (nyqz ? 0.f : kz), a[i]);
            } else if constexpr (KT == KOP_HESS3) {
                m[i] = o == 0 ? a[i] : __fmul_rn(o == 1 ? (nyqx ? 0.f : x) : __fmul_rn(x, x), a[i]);
            } else {
                const float k = o == 0 ? x : o == 1 ? ky : kz;
                const bool nyq = o == 0 ? nyqx : o == 1 ? nyqy : nyqz;
                m[i] = __fmul_rn(0.5f * __fmaf_rn(k, a[i], -__fmul_rn(nyq ? k : -k, b[i])), (float)op.norm);
            }
        }
    }
    // The radix-8 butterfly of m v (i m v): the products are part of its first additions.
    static __device__ __forceinline__ void first_pass(const float (&m)[8], const float2 (&v)[8], float2 (&u)[8]) {
        typedef float2 C;
        C s[4], d[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float p = m[i], q = m[i + 4];
            const C x = IMAG ? make_float2(-v[i].y, v[i].x) : v[i], y = IMAG ? make_float2(-v[i + 4].y, v[i + 4].x) : v[i + 4];
            const C qy = make_float2(__fmul_rn(q, y.x), __fmul_rn(q, y.y));
            s[i] = make_float2(__fmaf_rn(p, x.x, qy.x), __fmaf_rn(p, x.y, qy.y));
            d[i] = make_float2(__fmaf_rn(p, x.x, -qy.x), __fmaf_rn(p, x.y, -qy.y));
        }
        C e[4], o[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            C* w = h == 0 ? e : o;
            const C t0 = s[h], t1 = d[h], t2 = s[h + 2], t3 = cmul_i(d[h + 2], 1);
            w[0] = cadd(t0, t2), w[2] = csub(t0, t2), w[1] = cadd(t1, t3), w[3] = csub(t1, t3);
        }
        const float r = 0.70710678118654752440f;
        const C o1 = o[1], o3 = o[3];
        o[1] = make_float2(r * (o1.x - o1.y), r * (o1.y + o1.x));
        o[2] = cmul_i(o[2], 1);
        o[3] = make_float2(r * (-o3.x - o3.y), r * (-o3.y + o3.x));
#pragma unroll
        for (int k = 0; k < 4; k++) u[k] = cadd(e[k], o[k]), u[k + 4] = csub(e[k], o[k]);
    }
};

template <int N, int BP, int KT, int MINB>
__global__ void __launch_bounds__(N / 8 * BP, MINB)
    x_kspace_duo(const __grid_constant__ prc::tma::Maps maps, int nin, Specs<float2> out, Dims dims, int pitch, KOp op) {
    typedef float2 C;
    typedef DuoTile<N, BP> DT;
    constexpr int TL = N / 8, B = 2 * BP;
    // consecutive transforms of an odd number of exchanges would start on the buffer the previous one read last
    constexpr bool SYNC = Shape<N>::NX % 2 == 1;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Duo* stage = (Duo*)smem_raw;
    Duo* ybuf = stage + DT::ELEMS;
    Duo* xbuf = ybuf + DT::ELEMS;
    C* tw = (C*)(xbuf + DT::PADDED);
    uint64_t* bar = (uint64_t*)(tw + N);
    const int tid = threadIdx.x, q = tid % BP, t = tid / BP;
    const PairAddr<BP> addr{q};
    typedef typename std::conditional<(BP <= 4), PadPairAddr<BP>, PairAddr<BP>>::type XAddr;
    const XAddr xaddr{q};
    if (tid == 0) {
        prc::tma::barrier_init(bar, 1);
        prc::tma::fence_barrier_init();
    }
    fill_pass_twiddles<C, N>(tw);
    const int n1 = dims.n[1], nh = dims.n[2] / 2 + 1;
    const int64_t ls = (int64_t)n1 * pitch;
    const int ctiles = (nh + B - 1) / B;
    const int64_t tiles_per = (int64_t)n1 * ctiles;
    const int64_t ntiles = tiles_per * nin;
    __syncthreads();
    if ((prc::tma::smem_addr(stage) & 127) != 0) {
        if (tid == 0) atomicOr(&prc::g_fault, prc::tma::FAULT_SMEM_ALIGN);
        return;
    }
    auto issue = [&](int64_t tile) {
        if (tile >= ntiles) return;
        const TileAt a = tile_at(tile, tiles_per, ctiles, B);
        issue_tile<float, N, B>((C*)stage, &maps.m[a.bi], bar, 0, a.o, a.c0);
    };
    if (tid == 0) issue(blockIdx.x);
    unsigned phase = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, phase ^= 1) {
        const bool ok = prc::tma::wait(bar, phase);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                atomicOr(&prc::g_fault, prc::tma::FAULT_WAIT_TIMEOUT);
                prc::tma::wait(bar, phase);      // the copy in flight lands before the block leaves
            }
            return;
        }
        const TileAt a = tile_at(tile, tiles_per, ctiles, B);
        const int iy = a.o, iz = a.c0 + 2 * q;
        C va[8], vb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const Duo d = stage[(t + i * TL) * BP + q];
            va[i] = d.a, vb[i] = d.b;
        }
        // the stage is free once every thread is past the first exchange's barrier
        fft_duo<N, -1>(va, vb, t, xbuf, xaddr, ybuf, addr, tw);
        if constexpr (SYNC) __syncthreads();
        if (tid == 0) {
            prc::tma::fence_proxy_async();
            issue(tile + gridDim.x);
        }
        constexpr bool WRITTEN = KT == KOP_PSI || KT == KOP_HESS3 || KT == KOP_PP;
        typename std::conditional<WRITTEN, KDuo<N, KT>, KLine<float, N, KT>>::type ka, kb;
        ka.setup(op, dims, t, iy, iz);
        kb.setup(op, dims, t, iy, iz + 1);
        if constexpr (KT == KOP_HESS3) {
            if (t == 0 && op.side != nullptr) {
                KLine<float, N, KT> line;
                line.kp[4].a = ka.a[4];
                line.ky = ka.ky, line.kz = ka.kz;
                line.nyquist_lines(op, dims, t, iy, iz, va);
                line.kp[4].a = kb.a[4];
                line.kz = kb.kz;
                line.nyquist_lines(op, dims, t, iy, iz + 1, vb);
            }
        }
        const int64_t off = (int64_t)iy * pitch + iz;
        for (int o = 0; o < op.nper; o++) {
            C ua[8], ub[8];
            if constexpr (WRITTEN) {
                float m[8];
                ka.multipliers(op, t, o, m);
                KDuo<N, KT>::first_pass(m, va, ua);
                kb.multipliers(op, t, o, m);
                KDuo<N, KT>::first_pass(m, vb, ub);
                exchange_duo<N, 8, 1>(ua, ub, t, xbuf, xaddr);
                PassesDuo<N, +1, 1>::run(ua, ub, t, xbuf, xaddr, ybuf, addr, tw);
            } else {
                ka.apply(op, dims, t, o, va, ua);
                kb.apply(op, dims, t, o, vb, ub);
                fft_duo<N, +1>(ua, ub, t, xbuf, xaddr, ybuf, addr, tw);
            }
            if constexpr (SYNC) __syncthreads();
            C* go = out.p[a.bi * op.nper + o] + off;
#pragma unroll
            for (int i = 0; i < 8; i++) store_duo(go + (int64_t)(t + i * TL) * ls, ua[i], ub[i], iz < nh, iz + 1 < nh);
        }
    }
}

// ---- strided pass (strided_tma on pairs), in place ----
template <int N, int BP, int S> struct StridedDuoSmem {
    typedef DuoTile<N, BP> DT;
    static constexpr size_t BYTES = (size_t)(S * DT::ELEMS + DT::PADDED) * sizeof(Duo) + (size_t)N * sizeof(float2) + S * 8 + 16;
};

template <int N, int BP, int S, int DIR, int MINB>
__global__ void __launch_bounds__(N / 8 * BP, MINB)
    strided_duo(const __grid_constant__ prc::tma::Maps maps, Specs<float2> data, int nbatch, Strided s, int axis) {
    typedef float2 C;
    typedef DuoTile<N, BP> DT;
    constexpr int TL = N / 8, B = 2 * BP;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Duo* stages = (Duo*)smem_raw;
    Duo* xscr = stages + S * DT::ELEMS;
    C* tw = (C*)(xscr + DT::PADDED);
    uint64_t* bars = (uint64_t*)(tw + N);
    const int tid = threadIdx.x, q = tid % BP, t = tid / BP;
    const PairAddr<BP> addr{q};
    typedef typename std::conditional<(BP <= 4), PadPairAddr<BP>, PairAddr<BP>>::type XAddr;
    const XAddr xaddr{q};
    if (tid == 0) {
        for (int i = 0; i < S; i++) prc::tma::barrier_init(&bars[i], 1);
        prc::tma::fence_barrier_init();
    }
    fill_pass_twiddles<C, N>(tw);
    const int ctiles = (s.ncols + B - 1) / B;
    const int64_t tiles_per = (int64_t)s.outer * ctiles;
    const int64_t ntiles = tiles_per * nbatch;
    __syncthreads();
    if ((prc::tma::smem_addr(stages) & 127) != 0) {
        if (tid == 0) atomicOr(&prc::g_fault, prc::tma::FAULT_SMEM_ALIGN);
        return;
    }
    auto issue = [&](int64_t j) {
        const int64_t tile = blockIdx.x + j * gridDim.x;
        if (tile >= ntiles) return;
        const TileAt a = tile_at(tile, tiles_per, ctiles, B);
        issue_tile<float, N, B>((C*)(stages + (j % S) * DT::ELEMS), &maps.m[a.bi], &bars[j % S], axis, a.o, a.c0);
    };
    if (tid == 0)
        for (int j = 0; j < S; j++) issue(j);
    for (int64_t j = 0;; j++) {
        const int64_t tile = blockIdx.x + j * gridDim.x;
        if (tile >= ntiles) break;
        const int st = (int)(j % S);
        const bool ok = prc::tma::wait(&bars[st], (uint32_t)((j / S) & 1));
        if (__syncthreads_or(!ok)) {
            if (tid == 0) drain<S>(bars, j, ntiles, late_units(j, S));
            return;
        }
        // every thread is past tile j - 1, whose stage served the second exchange: it takes tile j - 1 + S
        if (tid == 0 && j > 0) {
            prc::tma::fence_proxy_async();
            issue(j - 1 + S);
        }
        Duo* sb = stages + st * DT::ELEMS;
        const TileAt a = tile_at(tile, tiles_per, ctiles, B);
        C va[8], vb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const Duo d = sb[(t + i * TL) * BP + q];
            va[i] = d.a, vb[i] = d.b;
        }
        fft_duo<N, DIR>(va, vb, t, xscr, xaddr, sb, addr, tw);
        const int c = a.c0 + 2 * q;
        C* g = data.p[a.bi] + (int64_t)a.o * s.os + c;
#pragma unroll
        for (int i = 0; i < 8; i++) store_duo(g + (int64_t)(t + i * TL) * s.ls, va[i], vb[i], c < s.ncols, c + 1 < s.ncols);
    }
}

// ---- inverse y pass of the local-line-of-sight iteration (y_hessian_tma on pairs) ----
template <int N, int BP, int S> struct HessDuoSmem {
    static constexpr size_t BYTES = StridedDuoSmem<N, BP, S>::BYTES + 2 * N * sizeof(float);
};

template <int N, int BP, int S, int MINB>
__global__ void __launch_bounds__(N / 8 * BP, MINB)
    y_hessian_duo(const __grid_constant__ prc::tma::Maps maps, Specs<float2> out, Strided s, HessGeom h) {
    typedef float2 C;
    typedef float T;
    typedef DuoTile<N, BP> DT;
    constexpr int TL = N / 8, B = 2 * BP;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Duo* stages = (Duo*)smem_raw;
    Duo* xscr = stages + S * DT::ELEMS;
    C* tw = (C*)(xscr + DT::PADDED);
    uint64_t* bars = (uint64_t*)(tw + N);
    T* x1tab = (T*)(bars + S);     // x1 and k_y of every y index
    T* kytab = x1tab + N;
    const int tid = threadIdx.x, qp = tid % BP, t = tid / BP;
    const PairAddr<BP> addr{qp};
    typedef typename std::conditional<(BP <= 4), PadPairAddr<BP>, PairAddr<BP>>::type XAddr;
    const XAddr xaddr{qp};
    if (tid == 0) {
        for (int i = 0; i < S; i++) prc::tma::barrier_init(&bars[i], 1);
        prc::tma::fence_barrier_init();
    }
    fill_pass_twiddles<C, N>(tw);
    for (int i = tid; i < N; i += blockDim.x) {
        x1tab[i] = (T)(h.x1_off + h.x1_cell * i);
        kytab[i] = kval<T>(i, h.ny, (T)h.fscale_y);
    }
    const int ctiles = (s.ncols + B - 1) / B;
    const int64_t ntiles = (int64_t)s.outer * ctiles;
    __syncthreads();
    if ((prc::tma::smem_addr(stages) & 127) != 0) {
        if (tid == 0) atomicOr(&prc::g_fault, prc::tma::FAULT_SMEM_ALIGN);
        return;
    }
    // unit u: tile blockIdx.x + (u / 6) gridDim.x, input spectrum F[2, 1, 0, 1, 0, 0][u % 6]
    auto input_of = [](int q) { return q == 0 ? 2 : (q == 1 || q == 3 ? 1 : 0); };
    auto issue = [&](int64_t u) {
        const int64_t tile = blockIdx.x + (u / 6) * gridDim.x;
        if (tile >= ntiles) return;
        const TileAt a = tile_at(tile, ntiles, ctiles, B);
        issue_tile<float, N, B>((C*)(stages + (u % S) * DT::ELEMS), &maps.m[input_of((int)(u % 6))], &bars[u % S], 1, a.o,
                                a.c0);
    };
    if (tid == 0)
        for (int u = 0; u < S; u++) issue(u);
    const int ynyq = h.ny % 2 == 0 ? h.ny / 2 : -1;
    const C* q01 = (const C*)h.q01;
    const C* l02 = (const C*)h.l02;
    int64_t u = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const TileAt a = tile_at(tile, ntiles, ctiles, B);
        const T x0 = (T)(h.x0_off + h.x0_cell * a.o);
        const int iz = a.c0 + 2 * qp;
        const T kza = kval<T>(iz, h.nz, (T)h.fscale_z), kzb = kval<T>(iz + 1, h.nz, (T)h.fscale_z);
        const bool nyqa = nyquist(iz, h.nz), nyqb = nyquist(iz + 1, h.nz);
        const T sza = nyqa ? (T)0 : kza, szb = nyqb ? (T)0 : kzb;
        const T xsign = (a.o & 1) ? (T)-1 : (T)1;     // (-1)^x
        const int64_t off = (int64_t)a.o * s.os + iz;
#pragma unroll 1
        for (int g = 0; g < 3; g++) {
            C aa[8], ab[8];
#pragma unroll
            for (int i = 0; i < 8; i++) aa[i] = ab[i] = cmake<C>(0, 0);
            const int nterm = g == 0 ? 3 : (g == 1 ? 2 : 1);
#pragma unroll 1
            for (int j = 0; j < nterm; j++, u++) {
                const int st = (int)(u % S);
                const bool ok = prc::tma::wait(&bars[st], (uint32_t)((u / S) & 1));
                const bool failed = __syncthreads_or(!ok);
                if (!failed && tid == 0 && u > 0) {
                    // every thread is past unit u - 1: its stage takes unit u - 1 + S
                    prc::tma::fence_proxy_async();
                    issue(u - 1 + S);
                }
                if (failed) {
                    if (tid == 0) {
                        atomicOr(&prc::g_fault, prc::tma::FAULT_WAIT_TIMEOUT);
                        for (int d = 0; d < late_units(u, S); d++) {
                            const int64_t uu = u + d;
                            if ((int64_t)blockIdx.x + (uu / 6) * gridDim.x >= ntiles) break;
                            prc::tma::wait(&bars[uu % S], (uint32_t)((uu / S) & 1));
                        }
                    }
                    return;
                }
                const int q = (int)(u % 6);
                Duo* sb = stages + st * DT::ELEMS;
                // D02 on the z-Nyquist column: the x-Nyquist mode of the line, (-1)^x l02
                const bool suba = q == 3 && nyqa && l02 != nullptr, subb = q == 3 && nyqb && l02 != nullptr;
                C va[8], vb[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const Duo d = sb[(t + i * TL) * BP + qp];
                    va[i] = d.a, vb[i] = d.b;
                }
                // y factor before the transform: k_y^2 (D11), s_y (D01, D12), k_y on the Nyquist index only (D12, z Nyquist)
                if (q == 2) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const T ky = kytab[t + i * TL];
                        va[i] = cscale(va[i], ky * ky), vb[i] = cscale(vb[i], ky * ky);
                    }
                } else if (q == 1 || q == 4) {
                    const bool on_a = q == 4 && nyqa, on_b = q == 4 && nyqb;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int iy = t + i * TL;
                        const T ky = kytab[iy];
                        va[i] = cscale(va[i], (on_a == (iy == ynyq)) ? ky : (T)0);
                        vb[i] = cscale(vb[i], (on_b == (iy == ynyq)) ? ky : (T)0);
                    }
                } else if (suba || subb) {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const C x = l02[t + i * TL];
                        const C y = cmake<C>(xsign * x.x, xsign * x.y);
                        if (suba) va[i] = y;
                        if (subb) vb[i] = y;
                    }
                }
                // scratch first: the stage is written only by the second exchange, behind the first exchange's barrier,
                // when every thread has read its points from it
                fft_duo<N, +1>(va, vb, t, xscr, xaddr, sb, addr, tw);
                if (q == 1 && q01 != nullptr) {
                    // D01 at the x and y Nyquist indices: q01[iz] (-1)^(x + y)
                    const C ca = iz < s.ncols ? q01[iz] : cmake<C>(0, 0), cb = iz + 1 < s.ncols ? q01[iz + 1] : cmake<C>(0, 0);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const T sg = ((t + i * TL) & 1) ? -xsign : xsign;
                        va[i] = cmake<C>(va[i].x + sg * ca.x, va[i].y + sg * ca.y);
                        vb[i] = cmake<C>(vb[i].x + sg * cb.x, vb[i].y + sg * cb.y);
                    }
                }
                // weight at this point: f00 x0^2 | f01 x0 x1 | f11 x1^2 | f02 x0 s_z (1 where substituted) |
                // f12 x1 k_z | f22 k_z^2
                if (q == 1 || q == 2 || q == 4) {
                    const T f = (T)(q == 1 ? h.f[1] : q == 2 ? h.f[3] : h.f[4]);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const T x1 = x1tab[t + i * TL];
                        const T wa = q == 1 ? f * (x0 * x1) : q == 2 ? f * (x1 * x1) : f * x1 * kza;
                        const T wb = q == 1 ? f * (x0 * x1) : q == 2 ? f * (x1 * x1) : f * x1 * kzb;
                        aa[i] = cmake<C>(aa[i].x + wa * va[i].x, aa[i].y + wa * va[i].y);
                        ab[i] = cmake<C>(ab[i].x + wb * vb[i].x, ab[i].y + wb * vb[i].y);
                    }
                } else {
                    const T f = (T)(q == 0 ? h.f[0] : q == 3 ? h.f[2] : h.f[5]);
                    const T wa = q == 0 ? f * (x0 * x0) : q == 3 ? f * x0 * (suba ? (T)1 : sza) : f * (kza * kza);
                    const T wb = q == 0 ? f * (x0 * x0) : q == 3 ? f * x0 * (subb ? (T)1 : szb) : f * (kzb * kzb);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        aa[i] = cmake<C>(aa[i].x + wa * va[i].x, aa[i].y + wa * va[i].y);
                        ab[i] = cmake<C>(ab[i].x + wb * vb[i].x, ab[i].y + wb * vb[i].y);
                    }
                }
            }
            C* o = (g == 0 ? out.p[0] : (g == 1 ? out.p[1] : out.p[2])) + off;
#pragma unroll
            for (int i = 0; i < 8; i++) store_duo(o + (int64_t)(t + i * TL) * s.ls, aa[i], ab[i], iz < s.ncols, iz + 1 < s.ncols);
        }
    }
}

}  // namespace fast
