// The V-cycle of the coarse levels as one kernel: a cluster of blocks per problem (included by multigrid.cu).
//
// Below some 10^4 cells a level costs more in launches than in work: a V-cycle visit of the levels from 16^3 down is ~40
// kernels of two to three microseconds each.  Whole solves, every level above 8^3 by launches -> from 16^3 (12^3, 20^3)
// down here: 64^3 FP64 1.84 -> 1.54 ms, 128^3 FP32 2.71 -> 2.38, 192^3 FP32 4.24 -> 3.93, 256^3 FP32 8.30 -> 7.90.  The
// planes of 32^3 on 8 blocks measured slower than launches (1.6 us a step), on 16 blocks no faster.  Here the planes of the larger levels are dealt to the blocks of a cluster
// (block r holds planes lo(r) .. lo(r + 1) - 1 of every such level, twice as many on each finer level), every level's v,
// scratch and f live in shared memory, a step (sweep, residual, restriction, prolongation) ends with a cluster barrier,
// and a block writes its outermost planes into its neighbours' halo planes as it computes them, so the sweeps read their
// own shared memory only.  The smallest levels run in block 0 alone.  A thread keeps its cells' coefficients, right-hand
// sides and neighbour positions over the sweeps of a level, so a step is little more than its loads, its arithmetic and
// a barrier.
// Dealt levels compute what the quad kernels do (op_terms), the ones of block 0 what the one-cell kernels do, in the same
// order of operations.
#pragma once

#include <cooperative_groups.h>

namespace prc {

constexpr int MG_COARSE_LEVELS = 8;
constexpr int MG_COARSE_THREADS = 512;
constexpr int MG_COARSE_SLOTS = 2;          // cells (block 0's levels) or pairs (dealt levels) a thread, at most
constexpr int MG_SINGLE_CELLS = 512;        // levels of at most this many cells run in block 0
constexpr size_t MG_COARSE_MAX_SMEM = 200 * 1024;
constexpr int MG_COARSE_CLUSTER = 8;        // blocks of a cluster, at most
constexpr int MG_COARSE_DEFAULT_CELLS = 13824;

template <typename T> struct CoarseCycle {
    int nl, ndist;                      // levels; the first ndist are dealt over the cluster
    Stencil<T> s[MG_COARSE_LEVELS];
    int at[MG_COARSE_LEVELS];           // level l: v and scratch (vsize values each), then f, from value at[l] on
    int vsize[MG_COARSE_LEVELS];
    int base;                           // planes of the coarsest dealt level
    T w;
    int jn;
    int zero_v;                         // the top level's v starts at zero (not read)
    int axis;                           // line of sight along this axis (-1: none), as residual_kernel4 orders it
};

// A pair of cells z, z + 1 of a dealt level (z and the row length even): where its rows begin, its coefficients.
template <typename T> struct PairSlot {
    int at, xm, xp, ym, yp, zm, zp;     // offset of the pair; of the same in planes x - 1, x + 1, rows y - 1, y + 1; of columns z - 1, z + 2
    int p;                              // plane of the block (1 .. np)
    int x, y, z;
    XYCoef<T> c;
    typename Pair<T>::T p2, s2, f;
};

// U, W, q, P of a pair from buffer v.
template <bool LOCAL, typename T, typename P2 = typename Pair<T>::T>
__device__ __forceinline__ void pair_terms(const T* v, const PairSlot<T>& n, const OpCoef<T>& k, P2& vc, P2& U, P2& W, P2& q, P2& PP) {
    typedef Pair<T> P;
    auto two = [&](int off) { return *(const P2*)(v + n.at + off); };
    vc = two(0);
    const P2 xp = two(n.xp), xm = two(n.xm), yp = two(n.yp), ym = two(n.ym);
    const P2 exy = P::sub(P::add(two(n.xp + n.yp), two(n.xm + n.ym)), P::add(two(n.xm + n.yp), two(n.xp + n.ym)));
    // cells z - 1 .. z + 2 of two rows a, b: (a[z + 1] + b[z - 1]) - (b[z + 1] + a[z - 1]) for both cells
    auto edge = [&](int oa, P2 a, int ob, P2 b) {
        const T *pa = v + n.at + oa, *pb = v + n.at + ob;
        return P::make(rn_sub(rn_add(a.y, pb[n.zm]), rn_add(b.y, pa[n.zm])), rn_sub(rn_add(pa[n.zp], b.x), rn_add(pb[n.zp], a.x)));
    };
    const P2 exz = edge(n.xp, xp, n.xm, xm), eyz = edge(n.yp, yp, n.ym, ym);
    const T* c0 = v + n.at;
    op_terms<LOCAL, P>(k, n.c, n.p2, n.s2, xp, xm, yp, ym, P::make(vc.y, c0[n.zp]), P::make(c0[n.zm], vc.x), exy, exz, eyz, U, W,
                       q, PP);
}

// A cell of a level whole in block 0's shared memory, with the one-cell kernels' coefficients (coeffs).
template <typename T> struct CellSlot {
    int at, xm, xp, ym, yp, zm, zp;     // offset of the cell; from it to its neighbours
    T p0, p1, p2, p01, p02, p12, g, gh, G0, G1, G2, den, f;
};
template <bool LOCAL, typename T> __device__ __forceinline__ void cell_slot(CellSlot<T>& c, const Stencil<T>& s, int i) {
    int x, y, z;
    const int *n = s.n, sx = n[1] * n[2];
    cell_xyz(i, n, x, y, z);
    c.at = i;
    c.xm = (wrap_dn(x, n[0]) - x) * sx, c.xp = (wrap_up(x, n[0]) - x) * sx;
    c.ym = (wrap_dn(y, n[1]) - y) * n[2], c.yp = (wrap_up(y, n[1]) - y) * n[2];
    c.zm = wrap_dn(z, n[2]) - z, c.zp = wrap_up(z, n[2]) - z;
    c.p0 = LOCAL ? rn_add((T)x, s.off[0]) : s.losh[0];
    c.p1 = LOCAL ? rn_add((T)y, s.off[1]) : s.losh[1];
    c.p2 = LOCAL ? rn_add((T)z, s.off[2]) : s.losh[2];
    const T q = fma_rn(rn_mul(s.h2[2], c.p2), c.p2, fma_rn(rn_mul(s.h2[0], c.p0), c.p0, rn_mul(rn_mul(s.h2[1], c.p1), c.p1)));
    c.g = rn_div(s.beta, q);
    c.gh = rn_mul(c.g, (T)0.5);
    c.G0 = fma_rn(rn_mul(c.g, c.p0), c.p0, s.ih2[0]);
    c.G1 = fma_rn(rn_mul(c.g, c.p1), c.p1, s.ih2[1]);
    c.G2 = fma_rn(rn_mul(c.g, c.p2), c.p2, s.ih2[2]);
    c.den = rn_mul((T)2, rn_add(rn_add(c.G0, c.G1), c.G2));
    c.p01 = rn_mul(c.p0, c.p1), c.p02 = rn_mul(c.p0, c.p2), c.p12 = rn_mul(c.p1, c.p2);
}
// S(v) at the cell (neighbour_sum).
template <bool LOCAL, typename T> __device__ __forceinline__ T cell_sum(const T* v, const CellSlot<T>& c) {
    const T* o = v + c.at;
    const T xp = o[c.xp], xm = o[c.xm], yp = o[c.yp], ym = o[c.ym], zp = o[c.zp], zm = o[c.zm];
    auto edge = [&](int ap, int am, int bp, int bm) { return rn_sub(rn_sub(rn_add(o[ap + bp], o[am + bm]), o[am + bp]), o[ap + bm]); };
    const T exy = edge(c.xp, c.xm, c.yp, c.ym), exz = edge(c.xp, c.xm, c.zp, c.zm), eyz = edge(c.yp, c.ym, c.zp, c.zm);
    T s = fma_rn(c.G0, rn_add(xp, xm), rn_mul(c.G1, rn_add(yp, ym)));
    s = fma_rn(c.G2, rn_add(zp, zm), s);
    const T e = fma_rn(c.p12, eyz, fma_rn(c.p01, exy, rn_mul(c.p02, exz)));
    s = fma_rn(c.gh, e, s);
    if (LOCAL) s = fma_rn(c.g, fma_rn(c.p2, rn_sub(zp, zm), fma_rn(c.p0, rn_sub(xp, xm), rn_mul(c.p1, rn_sub(yp, ym)))), s);
    return s;
}

// niter sweeps of a whole level, then (res) its residual into the buffer that does not hold v; v and tmp are swapped
// as the sweeps go.
template <bool LOCAL, typename T>
__device__ void whole_steps(const Stencil<T>& s, T*& v, const T* f, T*& tmp, T w, int niter, bool zero, bool res) {
    const int N = cells_of(s.n), tid = threadIdx.x;
    CellSlot<T> c[MG_COARSE_SLOTS];
#pragma unroll
    for (int j = 0; j < MG_COARSE_SLOTS; j++) {
        const int i = tid + j * MG_COARSE_THREADS;
        if (i < N) {
            cell_slot<LOCAL>(c[j], s, i);
            c[j].f = f[i];
            if (niter == 0 && zero) v[i] = (T)0;
        }
    }
    if (niter == 0 && zero) __syncthreads();
    for (int it = 0; it < niter; it++) {
#pragma unroll
        for (int j = 0; j < MG_COARSE_SLOTS; j++) {
            if (tid + j * MG_COARSE_THREADS < N) {
                T jac = c[j].f, vc = (T)0;
                if (!(zero && it == 0)) {
                    jac = rn_add(jac, cell_sum<LOCAL>(v, c[j]));
                    vc = v[c[j].at];
                }
                tmp[c[j].at] = fma_rn(rn_sub((T)1, w), vc, rn_mul(w, rn_div(jac, c[j].den)));
            }
        }
        T* t = v;
        v = tmp;
        tmp = t;
        __syncthreads();
    }
    if (res) {
#pragma unroll
        for (int j = 0; j < MG_COARSE_SLOTS; j++)
            if (tid + j * MG_COARSE_THREADS < N)
                tmp[c[j].at] = rn_sub(c[j].f, fma_rn(c[j].den, v[c[j].at], -cell_sum<LOCAL>(v, c[j])));
        __syncthreads();
    }
}

// f of the next level from this one's residual r (whole levels); the sum in reduce_kernel's order.
template <typename T> __device__ __forceinline__ T reduce_cell(const T* xm, const T* x0, const T* xp, const int nf[3], int y, int z) {
    const int Y[3] = {wrap_dn(2 * y, nf[1]) * nf[2], 2 * y * nf[2], wrap_up(2 * y, nf[1]) * nf[2]};
    const int Z[3] = {wrap_dn(2 * z, nf[2]), 2 * z, wrap_up(2 * z, nf[2])};
    T acc = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const T* p = a == 0 ? xm : (a == 1 ? x0 : xp);
#pragma unroll
        for (int b = 0; b < 3; b++)
#pragma unroll
            for (int c = 0; c < 3; c++) acc = fma_rn((T)(8 >> ((a != 1) + (b != 1) + (c != 1))), p[Y[b] + Z[c]], acc);
    }
    return acc / (T)64;
}

// The eight fine values of a coarse cell from the coarse planes x, x + 1, in prolong_kernel's order: e = 4 ex + 2 ey + ez.
template <typename T> __device__ __forceinline__ void prolong_cell(const T* p0, const T* p1, const int nc[3], int y, int z, T (&o)[8]) {
    const int ys[2] = {y * nc[2], wrap_up(y, nc[1]) * nc[2]}, zs[2] = {z, wrap_up(z, nc[2])};
    T c[2][2][2];
#pragma unroll
    for (int b = 0; b < 2; b++)
#pragma unroll
        for (int d = 0; d < 2; d++) c[0][b][d] = p0[ys[b] + zs[d]], c[1][b][d] = p1[ys[b] + zs[d]];
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const int ex = (e >> 2) & 1, ey = (e >> 1) & 1, ez = e & 1;
        T t = 0;
#pragma unroll
        for (int a = 0; a <= ex; a++)
#pragma unroll
            for (int b = 0; b <= ey; b++)
#pragma unroll
                for (int d = 0; d <= ez; d++) t = rn_add(t, c[a][b][d]);
        o[e] = rn_mul(t, (T)1 / (T)((1 + ex) * (1 + ey) * (1 + ez)));
    }
}

// ---- the cycle ----
template <typename T, bool LOCAL>
__global__ void __launch_bounds__(MG_COARSE_THREADS) vcycle_coarse(const T* __restrict__ fg, T* __restrict__ vg,
                                                                   const __grid_constant__ CoarseCycle<T> C) {
    namespace cg = cooperative_groups;
    typedef Pair<T> P;
    typedef typename P::T P2;
    pdl_trigger();
    cg::cluster_group cl = cg::this_cluster();
    const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank(), prob = blockIdx.x / CL;
    extern __shared__ __align__(16) unsigned char mg_smem[];
    T* sm = (T*)mg_smem;
    const int nd = C.ndist, tid = threadIdx.x;
    // planes of block r at dealt level l begin here (the split of the coarsest one, doubled)
    auto lo_of = [&](int r, int l) { return (r * C.base / CL) << (nd - 1 - l); };
    const int left = rank == 0 ? CL - 1 : rank - 1, right = rank == CL - 1 ? 0 : rank + 1;
    T *v[MG_COARSE_LEVELS], *t[MG_COARSE_LEVELS], *f[MG_COARSE_LEVELS];
    for (int l = 0; l < C.nl; l++) {
        v[l] = sm + C.at[l];
        t[l] = v[l] + C.vsize[l];
        f[l] = t[l] + C.vsize[l];
    }
    pdl_wait();
    {
        const int* n = C.s[0].n;
        const int pl = n[1] * n[2];
        fg += (int64_t)prob * n[0] * pl;
        vg += (int64_t)prob * n[0] * pl;
        const int lo = nd > 0 ? lo_of(rank, 0) : 0, np = nd > 0 ? lo_of(rank + 1, 0) - lo : n[0];
        if (nd > 0 || rank == 0) {
            for (int i = tid; i < np * pl; i += MG_COARSE_THREADS) f[0][i] = fg[(int64_t)lo * pl + i];
            if (!C.zero_v && nd > 0) {
                for (int i = tid; i < (np + 2) * pl; i += MG_COARSE_THREADS) {
                    int x = lo - 1 + i / pl;
                    x = x < 0 ? x + n[0] : (x >= n[0] ? x - n[0] : x);
                    v[0][i] = vg[(int64_t)x * pl + i % pl];
                }
            } else if (!C.zero_v) {
                for (int i = tid; i < np * pl; i += MG_COARSE_THREADS) v[0][i] = vg[i];
            }
        }
    }
    // every block's shared memory is in use from here on: no block writes to another's before
    cl.sync();

    // niter sweeps of dealt level l, then (res) its residual into the buffer that does not hold v.  A value goes to this
    // block's plane and, from its outermost planes, to the neighbours' halo planes.
    auto steps = [&](int l, int niter, bool zero, bool res) {
        const Stencil<T>& s = C.s[l];
        const int *n = s.n, pl = n[1] * n[2], h2 = n[2] / 2, per = n[1] * h2;
        const int lo = lo_of(rank, l), np = lo_of(rank + 1, l) - lo;
        const int to_left = (lo_of(left + 1, l) - lo_of(left, l) + 1) * pl;     // the left neighbour's upper halo plane
        const OpCoef<T> k = op_coef<LOCAL>(s);
        PairSlot<T> c[MG_COARSE_SLOTS];
        auto put = [&](T* b, const PairSlot<T>& a, P2 val) {
            *(P2*)(b + a.at) = val;
            if (a.p == 1) *(P2*)(cl.map_shared_rank(b, left) + to_left + a.at - pl) = val;
            if (a.p == np) *(P2*)(cl.map_shared_rank(b, right) + a.at - np * pl) = val;
        };
#pragma unroll
        for (int j = 0; j < MG_COARSE_SLOTS; j++) {
            const int i = tid + j * MG_COARSE_THREADS;
            if (i < np * per) {
                PairSlot<T>& a = c[j];
                const int p = i / per, r = i - p * per, y = r / h2, z = 2 * (r - y * h2);
                a.p = p + 1, a.x = lo + p, a.y = y, a.z = z;
                a.at = a.p * pl + y * n[2] + z;
                a.xm = -pl, a.xp = pl;
                a.ym = (wrap_dn(y, n[1]) - y) * n[2], a.yp = (wrap_up(y, n[1]) - y) * n[2];
                a.zm = z == 0 ? n[2] - 1 : -1, a.zp = z + 2 == n[2] ? -z : 2;
                a.c = xy_coef<LOCAL>(k, a.x, y);
                a.p2 = P::make(z_p2<LOCAL>(k, z), z_p2<LOCAL>(k, z + 1));
                a.s2 = P::mul(a.p2, a.p2);
                a.f = *(const P2*)(f[l] + a.at - pl);
            }
        }
        if (niter == 0 && zero) {
#pragma unroll
            for (int j = 0; j < MG_COARSE_SLOTS; j++)
                if (tid + j * MG_COARSE_THREADS < np * per) put(v[l], c[j], P::all((T)0));
            cl.sync();
        }
        for (int it = 0; it < niter; it++) {
#pragma unroll
            for (int j = 0; j < MG_COARSE_SLOTS; j++) {
                if (tid + j * MG_COARSE_THREADS < np * per) {
                    const PairSlot<T>& a = c[j];
                    P2 o;
                    if (zero && it == 0) {
                        T q4[4] = {a.f.x, a.f.y, (T)0, (T)0}, o4[4];
                        quad_zero<LOCAL>(k, C.w, a.x, a.y, a.z, q4, o4);
                        o = P::make(o4[0], o4[1]);
                    } else {
                        P2 vc, U, W, q, PP;
                        pair_terms<LOCAL>(v[l], a, k, vc, U, W, q, PP);
                        o = op_jacobi<P>(k, a.f, vc, U, W, q, PP, C.w);
                    }
                    put(t[l], a, o);
                }
            }
            T* x = v[l];
            v[l] = t[l];
            t[l] = x;
            cl.sync();
        }
        if (res) {
#pragma unroll
            for (int j = 0; j < MG_COARSE_SLOTS; j++) {
                if (tid + j * MG_COARSE_THREADS < np * per) {
                    P2 vc, U, W, q, PP;
                    pair_terms<LOCAL>(v[l], c[j], k, vc, U, W, q, PP);
                    P2 r;
                    if (!LOCAL && sizeof(T) == 4 && C.axis >= 0) {
                        const int ap = C.axis == 0 ? c[j].xp : c[j].yp, am = C.axis == 0 ? c[j].xm : c[j].ym;
                        const T* o = v[l] + c[j].at;
                        const P2 S = C.axis == 2 ? P::add(P::make(vc.y, o[c[j].zp]), P::make(o[c[j].zm], vc.x))
                                                 : P::add(*(const P2*)(o + ap), *(const P2*)(o + am));
                        const P2 wf = C.axis == 0 ? P::all(c[j].c.s0) : (C.axis == 1 ? P::all(c[j].c.s1) : c[j].s2);
                        r = op_residual_from<P>(k, c[j].f, vc, U, P::fma(wf, S, P::mul(P::mul(P::all((T)-2), PP), vc)), q);
                    } else {
                        r = op_residual<P>(k, c[j].f, vc, U, W, q, PP);
                    }
                    put(t[l], c[j], r);
                }
            }
            cl.sync();
        }
    };

    // down: pre-sweeps, the residual, its restriction to the next level's right-hand side
    for (int l = 0; l < nd; l++) {
        const bool more = l + 1 < C.nl;
        steps(l, C.jn, l > 0 || C.zero_v, more);
        if (!more) break;
        const int *nf = C.s[l].n, *nc = C.s[l + 1].n;
        // the coarse planes centred on this block's fine ones
        const int plc = nc[1] * nc[2], plf = nf[1] * nf[2], lo = lo_of(rank, l), loc = (lo + 1) / 2;
        const int npc = (lo_of(rank + 1, l) + 1) / 2 - loc;
        T* dst = l + 1 < nd ? f[l + 1] : cl.map_shared_rank(f[l + 1], 0) + loc * plc;
        for (int i = tid; i < npc * plc; i += MG_COARSE_THREADS) {
            const int p = i / plc, r = i - p * plc, y = r / nc[2], z = r - y * nc[2];
            const T* x0 = t[l] + (2 * (loc + p) - lo + 1) * plf;
            dst[i] = reduce_cell(x0 - plf, x0, x0 + plf, nf, y, z);
        }
        cl.sync();
    }
    // the smallest levels, in block 0
    if (nd < C.nl) {
        if (rank == 0) {
            for (int l = nd; l < C.nl; l++) {
                const bool more = l + 1 < C.nl;
                whole_steps<LOCAL>(C.s[l], v[l], f[l], t[l], C.w, C.jn, l > 0 || C.zero_v, more);
                if (!more) break;
                const int *nf = C.s[l].n, *nc = C.s[l + 1].n;
                const int pl = nf[1] * nf[2];
                for (int i = tid; i < cells_of(nc); i += MG_COARSE_THREADS) {
                    int x, y, z;
                    cell_xyz(i, nc, x, y, z);
                    f[l + 1][i] = reduce_cell(t[l] + wrap_dn(2 * x, nf[0]) * pl, t[l] + 2 * x * pl,
                                              t[l] + wrap_up(2 * x, nf[0]) * pl, nf, y, z);
                }
                __syncthreads();
            }
            for (int l = C.nl - 1; l >= nd; l--) {
                if (l + 1 < C.nl) {
                    const int* nc = C.s[l + 1].n;
                    const int plc = nc[1] * nc[2], nf1 = 2 * nc[1], nf2 = 2 * nc[2];
                    for (int i = tid; i < cells_of(nc); i += MG_COARSE_THREADS) {
                        int x, y, z;
                        cell_xyz(i, nc, x, y, z);
                        T o[8];
                        prolong_cell(v[l + 1] + x * plc, v[l + 1] + wrap_up(x, nc[0]) * plc, nc, y, z, o);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            T* d = v[l] + ((2 * x + (e >> 2)) * nf1 + 2 * y + ((e >> 1) & 1)) * nf2 + 2 * z + (e & 1);
                            *d = rn_add(*d, o[e]);
                        }
                    }
                    __syncthreads();
                }
                whole_steps<LOCAL>(C.s[l], v[l], f[l], t[l], C.w, C.jn, false, false);
            }
        }
        // block 0 swapped v[nd] 2 jn times, an even number: it is where the other blocks look for it
        cl.sync();
    }
    // up: the coarse correction prolonged and added, then post-sweeps
    for (int l = nd - 1; l >= 0; l--) {
        if (l + 1 < C.nl) {
            const int *nc = C.s[l + 1].n, *nf = C.s[l].n;
            const int plc = nc[1] * nc[2], plf = nf[1] * nf[2], lo = lo_of(rank, l), np = lo_of(rank + 1, l) - lo;
            const int to_left = (lo_of(left + 1, l) - lo_of(left, l) + 1) * plf;
            const bool dealt = l + 1 < nd;
            // coarse plane x at src + x plc (of a dealt level: this block's planes and the one after them)
            const T* src = dealt ? v[l + 1] + plc - lo / 2 * plc : (const T*)cl.map_shared_rank(v[l + 1], 0);
            for (int i = tid; i < np * plc; i += MG_COARSE_THREADS) {
                const int p = i / plc, r = i - p * plc, y = r / nc[2], z = r - y * nc[2];
                const int xf = lo + p, x = xf >> 1, xn = dealt ? x + 1 : wrap_up(x, nc[0]);
                T o[8];
                prolong_cell(src + x * plc, src + xn * plc, nc, y, z, o);
                const bool ex = xf & 1;
#pragma unroll
                for (int ey = 0; ey < 2; ey++) {
                    const int at = (2 * y + ey) * nf[2] + 2 * z;
                    P2* d = (P2*)(v[l] + (p + 1) * plf + at);
                    const P2 old = *d, val = P::make(rn_add(old.x, ex ? o[4 + 2 * ey] : o[2 * ey]),
                                                     rn_add(old.y, ex ? o[5 + 2 * ey] : o[1 + 2 * ey]));
                    *d = val;
                    if (p == 0) *(P2*)(cl.map_shared_rank(v[l], left) + to_left + at) = val;
                    if (p == np - 1) *(P2*)(cl.map_shared_rank(v[l], right) + at) = val;
                }
            }
            cl.sync();
        }
        steps(l, C.jn, false, false);
    }
    // (the last step's barrier has passed: no block writes to another's shared memory any more)
    {
        const int* n = C.s[0].n;
        const int pl = n[1] * n[2];
        if (nd > 0) {
            const int lo = lo_of(rank, 0), np = lo_of(rank + 1, 0) - lo;
            for (int i = tid; i < np * pl; i += MG_COARSE_THREADS) vg[(int64_t)lo * pl + i] = v[0][pl + i];
        } else if (rank == 0) {
            for (int i = tid; i < n[0] * pl; i += MG_COARSE_THREADS) vg[i] = v[0][i];
        }
    }
}

}  // namespace prc
