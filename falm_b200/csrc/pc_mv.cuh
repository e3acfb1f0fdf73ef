// Half a BiCGStab iteration in one pass: the vector update, the red-black SOR
// preconditioner (two sweeps from zero) and the operator application with its
// inner products.
//
//   P  v = r + beta (p - omega q)   z = pp ~ A^-1 v   y = q = A pp   rr.y          -> alpha
//   S  v = r - alpha q              z = ss ~ A^-1 v   y = t = A ss   y.v, y.y      -> omega
//
// The four half sweeps from zero and the product are five stages, each of which
// reads only the other colour's result of the stage before:
//   0  black  x = w v                      (w = omega_sor / ac: all neighbours are zero)
//   1  red    x = w (v - N x)              (N: the six off-diagonal terms)
//   2  black  x = x + w (v - ac x - N x)
//   3  red    s = N x;  x = x + w (v - ac x - s);  y = ac x + s
//   4  black  y = ac x + N x
// so the red half of the product costs one multiply-add: stage 3's off-diagonal
// sum is the product's.  (FP32
// keeps the order of the stand-alone kernels instead, PCTile::SEQ.)
//
// A thread owns a column of cell pairs (x0, x0+1) in two adjacent rows and
// marches along z; stage m works on plane q - m when plane q arrives.  The
// column's values of both colours on the planes in flight are kept in registers
// (z neighbours, the pair's other cell and the other row's cell), and only the
// outer x neighbour and the outer y neighbour of each row come from shared
// memory, where every stage leaves its plane for the next iteration: one block
// barrier per plane.  Colours are stored apart: at iteration parity S every
// stage works on the cells x0 + S of the first row and x0 + 1 - S of the second,
// so the march, unrolled over the parity, has no colour selection, and in FP32
// the two rows are one operation of the packed pipe.
//
// Cells outside the interior are zero (w = 0, v = 0): the guide cells of the
// solver's vectors.  The tile's outer four cells are recomputed by the
// neighbouring tiles: a tile of 64 x 32 (FP32) or 64 x 24 (FP64) cells owns
// 56 x 24 or 56 x 16 (and up to the walls where it touches them).  Operands are
// copied to shared memory NS planes ahead (four in FP32, three in FP64) by cp.async, each thread its own
// cells, so no alignment of the rows is needed: pairs of 8 or 16 bytes where the
// rows allow it, single cells elsewhere.
//
// What it replaces moved 10 (s half) and 11 (p half) values a cell in three
// kernels; this one moves 5 and 7.  Bound by instruction issue and the latency of
// a plane's iteration (FP32 16 warps an SM at 126 registers, FP64 12 at 168: a
// second CTA does not fit, a taller tile needs more registers), not by HBM.
// Measured, s half at 512 x 256 x 256 (cold, one kernel at a time): FP32 update
// 111 + sweeps 221 + product 107 -> 188 us, FP64 208 + 623 + 172 -> 348 us; FP64
// iteration at 128 x 64 x 64 85 -> 64 us, at 200 x 120 x 96 (general z
// coefficients) 260 -> 148 us.
#pragma once
#include "pair.cuh"
#include "pc_tile.cuh"
#include "poisson.cuh"
#include "sor_rb_tma.cuh"

namespace fb {

// The vectors of an iteration.  The new p and q may not overwrite the old ones,
// which neighbouring tiles still read, so {p, q} and {s, t} change places at
// every iteration: iteration n (SolverScalars::it) keeps p, q in pair n & 1 and
// s, t in the other; the first reads rr for p and r, the second rr for the old p.
template <typename T>
struct PCVec {
    const T *rr, *r;
    T *a0, *b0, *a1, *b1;   // pair 0 and 1: {p or s}, {q or t}
    T *z;             // pp or ss
};

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// MODE 0: P, 1: S.  ALN: rows, bases and tile origins allow pair accesses.
// [zr0, zr1): the longest run of planes with equal z coefficients.  GEN (FP64, no
// such run): a plane's weights, a division each, are computed when stages 0 and 1
// reach it and kept for stages 2 and 3 two iterations later, on the same cells
// (200 x 120 x 96 stretched: 168 -> 148 us an iteration).
template <typename T, int MODE, bool ALN, bool GEN>
__global__ void __launch_bounds__(PCTile<T>::NT, 1) k_pc_mv(Geom g, int kc, PoissonTables<T> tb, PCVec<T> vec, T omega, int zr0, int zr1,
                                                            RedWork rw, SolverScalars *sc) {
    using L = PCTile<T>;
    using V2 = P2<T>;
    constexpr int NT = L::NT, NS = L::NS, XP = L::XP, NF = MODE == 0 ? 3 : 2;
    if (sc->done) return;
    extern __shared__ __align__(128) unsigned char pc_smem[];
    V2 *ring = (V2 *)pc_smem;                              // [slot][field][row][thread]
    T *ex = (T *)(ring + NS * NF * 2 * NT);                // [parity][stage][row][pair]
    ZCoef<T> *ztab = (ZCoef<T> *)(ex + 8 * L::EPL);
    T *sdxy = (T *)(ztab + L::ZPL);                        // the thread's four in-plane diagonals
    V2 *scoef = (V2 *)(sdxy + 4 * NT);                     // CSM: acS[0], acS[1], wS[0], wS[1]
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const int gc = g.gc, it = sc->it;
    const bool first = it == 0;
    // vectors of this iteration
    const bool odd = it & 1;
    T *const a_cur = odd ? vec.a1 : vec.a0, *const a_oth = odd ? vec.a0 : vec.a1;
    T *const b_cur = odd ? vec.b1 : vec.b0, *const b_oth = odd ? vec.b0 : vec.b1;
    const T *rin = first ? vec.rr : vec.r;
    const T *f1 = MODE == 0 ? (it == 1 ? vec.rr : a_oth) : b_cur, *f2 = MODE == 0 ? b_oth : nullptr;
    T *const vout = MODE == 0 ? (first ? nullptr : a_cur) : a_oth, *const yout = MODE == 0 ? b_cur : b_oth;
    __shared__ T *sptr[4];   // CSM: f1, f2, vout, yout, read at each use
    if (L::CSM && threadIdx.x == 0) { sptr[0] = (T *)f1; sptr[1] = (T *)f2; sptr[2] = vout; sptr[3] = yout; }
    if (L::CSM) __syncthreads();
    const T c1 = MODE == 0 ? (T)sc->beta : -(T)sc->alpha, c2 = MODE == 0 ? -(T)sc->omega : T(0);

    // the thread's cells: x0, x0 + 1 in rows j0, j0 + 1
    const int xi = L::OX * blockIdx.x + 2 * lane, yi = L::OY * blockIdx.y + 2 * wp;   // from the interior's corner
    const int x0 = gc + xi, j0 = gc + yi;
    const bool inx[2] = {xi < g.nx, xi + 1 < g.nx}, iny[2] = {yi < g.ny, yi + 1 < g.ny};
    const int oxl = blockIdx.x == 0 ? 0 : L::OX * blockIdx.x + L::H, oyl = blockIdx.y == 0 ? 0 : L::OY * blockIdx.y + L::H;
    const int oxh = blockIdx.x == gridDim.x - 1 ? g.nx : L::OX * blockIdx.x + L::TX - L::H;
    const int oyh = blockIdx.y == gridDim.y - 1 ? g.ny : L::OY * blockIdx.y + L::TY - L::H;
    const bool ownx[2] = {xi >= oxl && xi < oxh, xi + 1 >= oxl && xi + 1 < oxh}, owny[2] = {yi >= oyl && yi < oyh, yi + 1 >= oyl && yi + 1 < oyh};
    const int k0 = gc + blockIdx.z * kc, k1 = min(k0 + kc, g.sz - gc);
    // first plane: the chunk's halo or the wall, at an even colour parity
    int qs = max(k0 - L::H, gc);
    qs -= (qs + g.koff) & 1;
    const int qe = k1 - 1 + L::H;
    const unsigned nown = k1 - k0;

    // omega / ac, or 1 / ac where the stages multiply by omega last (SEQ)
    auto weight = [&](T ac) -> T {
        if constexpr (L::SEQ) return rcp_approx(ac);
        else return omega / ac;
    };
    // in-plane coefficients of the parity-S cells (first row's cell x0 + S, second row's x0 + 1 - S):
    // towards the pair's other cell (in), the next pair (out), and y
    V2 cin[2], cou[2], acS[2], wS[2];
    V2 can, cas;
    const int xa = min(x0, g.sx - 1), xb = min(x0 + 1, g.sx - 1), ya = min(j0, g.sy - 1), yb = min(j0 + 1, g.sy - 1);
    const T ab_r = ldg(tb.cm[2] + zr0), at_r = ldg(tb.cp[2] + zr0);
    {
        const T aw0 = ldg(tb.cm[0] + xa), ae0 = ldg(tb.cp[0] + xa), aw1 = ldg(tb.cm[0] + xb), ae1 = ldg(tb.cp[0] + xb);
        // SEQ: towards x+ (in its place) and x-
        cin[0] = mk2(ae0, L::SEQ ? ae1 : aw1); cin[1] = mk2(L::SEQ ? ae1 : aw1, ae0);
        cou[0] = mk2(aw0, L::SEQ ? aw1 : ae1); cou[1] = mk2(L::SEQ ? aw1 : ae1, aw0);
        can = mk2(ldg(tb.cp[1] + ya), ldg(tb.cp[1] + yb));
        cas = mk2(ldg(tb.cm[1] + ya), ldg(tb.cm[1] + yb));
        const T d0 = ldg(tb.dx0 + xa), d1 = ldg(tb.dx0 + xb);
        const T up0 = ldg(tb.up[1] + ya), um0 = ldg(tb.um[1] + ya), up1 = ldg(tb.up[1] + yb), um1 = ldg(tb.um[1] + yb);
        const T d[2][2] = {{(d0 - up0) - um0, (d1 - up0) - um0}, {(d0 - up1) - um1, (d1 - up1) - um1}};   // [row][cell]
        const T zp = ldg(tb.up[2] + zr0), zm = ldg(tb.um[2] + zr0);
#pragma unroll
        for (int s = 0; s < 2; s++) {
            sdxy[(2 * s) * NT + tid] = d[0][s];
            sdxy[(2 * s + 1) * NT + tid] = d[1][1 - s];
            acS[s] = mk2(((d[0][s] - zp) - zm) * tb.scale, ((d[1][1 - s] - zp) - zm) * tb.scale);
            wS[s] = mk2(inx[s] && iny[0] ? weight(acS[s].x) : T(0), inx[1 - s] && iny[1] ? weight(acS[s].y) : T(0));
        }
    }
    if constexpr (L::CSM && !GEN) {
#pragma unroll
        for (int s = 0; s < 2; s++) { scoef[s * NT + tid] = acS[s]; scoef[(2 + s) * NT + tid] = wS[s]; }
    }
    // z coefficients of planes qs - 4 .. qe
    for (int n = tid; n < qe - qs + 5; n += NT) {
        const int kz = qs - 4 + n;
        const bool in = kz >= gc && kz < g.sz - gc;
        ztab[n] = in ? ZCoef<T>{ldg(tb.cm[2] + kz), ldg(tb.cp[2] + kz), -ldg(tb.up[2] + kz), -ldg(tb.um[2] + kz)} : ZCoef<T>{T(0), T(0), T(0), T(0)};
    }
    for (int n = tid; n < 8 * L::EPL; n += NT) ex[n] = T(0);

    // operand copies: each thread its own cells of plane q (row 0's cell x0 at offset o) into slot (q - qs) % NS
    const unsigned sxy = (unsigned)g.sx * g.sy, c00 = (unsigned)x0 + (unsigned)j0 * g.sx;
    const int qlast = min(qe, g.sz - gc - 1);
    const bool cp0 = inx[0] && iny[0], cp1 = inx[1] && iny[0], cp2 = inx[0] && iny[1], cp3 = inx[1] && iny[1];
    auto issue = [&](int q, int slot, unsigned o) {
        if (q >= gc && q <= qlast) {
            V2 *dst = ring + slot * (NF * 2 * NT) + tid;
            const unsigned o1 = o + g.sx;
#pragma unroll
            for (int f = 0; f < NF; f++) {
                if (MODE == 0 && f > 0 && first) break;
                const T *src = f == 0 ? rin : (L::CSM ? sptr[f - 1] : (f == 1 ? f1 : f2));
                V2 *d0 = dst + (2 * f) * NT, *d1 = d0 + NT;
                if (ALN) {
                    if (cp0) cp_async<2 * sizeof(T)>(d0, src + o);
                    if (cp2) cp_async<2 * sizeof(T)>(d1, src + o1);
                } else {
                    if (cp0) cp_async<sizeof(T)>((T *)d0, src + o);
                    if (cp1) cp_async<sizeof(T)>((T *)d0 + 1, src + o + 1);
                    if (cp2) cp_async<sizeof(T)>((T *)d1, src + o1);
                    if (cp3) cp_async<sizeof(T)>((T *)d1 + 1, src + o1 + 1);
                }
            }
        }
        cp_async_commit();
    };
    // cells outside the interior are never copied: their operands are zero
    if (!(cp0 && cp1 && cp2 && cp3))
        for (int n = 0; n < NS * NF * 2; n++) ring[n * NT + tid] = mk2(T(0), T(0));
#pragma unroll
    for (int n = 0; n < NS; n++) issue(qs + n, n, c00 + (unsigned)(qs + n) * sxy);

    // exchange planes: this thread's rows and the neighbours it reads
    const int e0 = (2 * wp + 1) * XP + lane + 1, e1 = e0 + XP;
    auto xch = [&](int par, int stage) { return ex + (par * 4 + stage) * L::EPL; };
    auto put = [&](T *e, V2 v) { e[e0] = v.x; e[e1] = v.y; };
    const V2 z2 = mk2(T(0), T(0));
    V2 X1[2] = {z2, z2}, X2[2] = {z2, z2}, X3[2] = {z2, z2}, X4[2] = {z2, z2};   // stage results by plane parity
    V2 vRa[2] = {z2, z2}, vRb[2] = {z2, z2}, vBa[2] = {z2, z2}, vBb[2] = {z2, z2};
    V2 tR = z2;
    V2 rr0 = z2, rr1 = z2;   // P: rr of plane q - 4, both rows
    constexpr int NV = MODE == 0 ? 1 : 2;
    double acc[NV];
#pragma unroll
    for (int d = 0; d < NV; d++) acc[d] = 0.0;
    const V2 mone = mk2(T(-1), T(-1)), ab_p = mk2(ab_r, ab_r), at_p = mk2(at_r, at_r), at_n = mk2(-at_r, -at_r);

    const bool st0 = ownx[0] && owny[0], st1 = ALN ? st0 : ownx[1] && owny[0];
    const bool st2_ = ownx[0] && owny[1], st3 = ALN ? st2_ : ownx[1] && owny[1];
    auto store = [&](T *base, unsigned c, V2 row0, V2 row1) {
        T *p = base + c, *p1 = p + g.sx;
        if (ALN) {
            if (st0) st2(p, row0);
            if (st2_) st2(p1, row1);
        } else {
            if (st0) p[0] = row0.x;
            if (st1) p[1] = row0.y;
            if (st2_) p1[0] = row1.x;
            if (st3) p1[1] = row1.y;
        }
    };

    if constexpr (GEN) {   // the weights of stages 2 and 3, none yet
#pragma unroll
        for (int s = 0; s < 4; s++) scoef[s * NT + tid] = z2;
    }
    // one iteration: plane q arrives (cell x0 of the first row at offset c); S its colour parity; REG: planes
    // q - 4 .. q have the regular z coefficients
    int slot = 0;   // of plane q
    auto iter = [&](auto SC, auto RC, int q, unsigned c) {
        constexpr int S = decltype(SC)::value, Q = 1 - S;
        constexpr bool REG = decltype(RC)::value;
        cp_async_wait<NS - 1>();
        const V2 *mine = ring + slot * (NF * 2 * NT) + tid;
        V2 v0 = mine[0], v1 = mine[NT];
        if (MODE == 0) {
            if (!first) {
                v0 = fma2(mk2(c1, c1), fma2(mk2(c2, c2), mine[4 * NT], mine[2 * NT]), v0);
                v1 = fma2(mk2(c1, c1), fma2(mk2(c2, c2), mine[5 * NT], mine[3 * NT]), v1);
            }
        } else {
            v0 = fma2(mk2(c1, c1), mine[2 * NT], v0);
            v1 = fma2(mk2(c1, c1), mine[3 * NT], v1);
        }
        if (!REG && (q < gc || q > qlast)) v0 = v1 = z2;   // a plane outside the interior: nothing was copied
        issue(q + NS, slot, c + NS * sxy);
        slot = slot + 1 == NS ? 0 : slot + 1;
        const bool in0 = (unsigned)(q - k0) < nown, in3 = (unsigned)(q - 3 - k0) < nown;   // planes q and q - 3 are the chunk's
        if (in0 && !(MODE == 0 && first)) store(L::CSM ? sptr[2] : vout, c, v0, v1);
        const V2 vB = S == 0 ? mk2(v0.x, v1.y) : mk2(v0.y, v1.x), vR = S == 0 ? mk2(v0.y, v1.x) : mk2(v0.x, v1.y);
        // z coefficients, diagonal and weight of the parity-S cells of planes q .. q - 4
        V2 ac[5], w[5], ab[5], at[5], nat[5];
        if constexpr (REG) {
            const V2 acr = L::CSM ? scoef[S * NT + tid] : acS[S], wr = L::CSM ? scoef[(2 + S) * NT + tid] : wS[S];
#pragma unroll
            for (int m = 0; m < 5; m++) { ac[m] = acr; w[m] = wr; ab[m] = ab_p; at[m] = at_p; nat[m] = at_n; }
        } else {
            const V2 dS = mk2(sdxy[(2 * S) * NT + tid], sdxy[(2 * S + 1) * NT + tid]);
#pragma unroll
            for (int m = 0; m < 5; m++) {
                const int pl = q - m;
                const ZCoef<T> zc = ztab[pl - (qs - 4)];
                ab[m] = mk2(zc.ab, zc.ab); at[m] = mk2(zc.at, zc.at); nat[m] = mk2(-zc.at, -zc.at);
                ac[m] = mul2(add2(add2(dS, mk2(zc.nup, zc.nup)), mk2(zc.num, zc.num)), mk2(tb.scale, tb.scale));
                const bool in = pl >= gc && pl < g.sz - gc;
                if (m < (GEN ? 2 : 4)) w[m] = mk2(in && inx[S] && iny[0] ? weight(ac[m].x) : T(0), in && inx[Q] && iny[1] ? weight(ac[m].y) : T(0));
            }
            if constexpr (GEN) {
                w[2] = scoef[S * NT + tid]; w[3] = scoef[(2 + S) * NT + tid];
                scoef[S * NT + tid] = w[0]; scoef[(2 + S) * NT + tid] = w[1];
            }
        }
        __syncthreads();   // the planes the stages left at the previous iteration
        const int oo0 = e0 + (S ? 1 : -1), oo1 = e1 + (S ? -1 : 1);
        V2 x1, x2, x3, x4, tRn, tB;
        // own: the pair's other cells, e: that stage's plane
        if constexpr (L::SEQ) {
            // ac xc + east + west + north + south, then above and below
            auto row = [&](V2 cc, V2 xc, V2 own, const T *e) {
                const T o0 = e[oo0], o1 = e[oo1];
                V2 s = mul2(cc, xc);
                s = fma2(cin[S], S == 0 ? mk2(own.x, o1) : mk2(o0, own.y), s);
                s = fma2(cou[S], S == 0 ? mk2(o0, own.y) : mk2(own.x, o1), s);
                s = fma2(can, mk2(own.y, e[e1 + XP]), s);
                return fma2(cas, mk2(e[e0 - XP], own.x), s);
            };
            const V2 om = mk2(omega, omega);
            const V2 s1 = row(z2, z2, X1[Q], xch(Q, 0)), s2 = row(ac[2], X1[S], X2[S], xch(Q, 1)), s3 = row(ac[3], X2[Q], X3[Q], xch(Q, 2));
            const V2 s4 = row(ac[4], X3[S], X4[S], xch(Q, 3));
            x1 = mul2(om, mul2(vB, w[0]));                                                                                    // 0: plane q, black
            x2 = mul2(om, mul2(fma2(fma2(ab[1], X1[S], fma2(at[1], x1, s1)), mone, vRa[Q]), w[1]));                           // 1: plane q - 1, red
            x3 = fma2(om, mul2(fma2(fma2(ab[2], X2[Q], fma2(at[2], x2, s2)), mone, vBa[S]), w[2]), X1[S]);                    // 2: plane q - 2, black
            x4 = fma2(om, mul2(fma2(fma2(ab[3], X3[S], fma2(at[3], x3, s3)), mone, vRb[Q]), w[3]), X2[Q]);                    // 3: plane q - 3, red
            tRn = fma2(ab[3], X3[S], fma2(at[3], x3, row(ac[3], x4, X3[Q], xch(Q, 2))));                                      // the product, red
            tB = fma2(ab[4], X4[Q], fma2(at[4], x4, s4));                                                                     // and black, plane q - 4
        } else {
            // the off-diagonal sum but for the plane above
            auto nbr = [&](V2 own, const T *e, V2 below, V2 abm) {
                V2 s = mul2(cin[S], own);
                s = fma2(abm, below, s);
                s = fma2(cou[S], mk2(e[oo0], e[oo1]), s);
                s = fma2(can, mk2(own.y, e[e1 + XP]), s);
                return fma2(cas, mk2(e[e0 - XP], own.x), s);
            };
            const V2 s1 = nbr(X1[Q], xch(Q, 0), X1[S], ab[1]), s2 = nbr(X2[S], xch(Q, 1), X2[Q], ab[2]);
            const V2 s3 = nbr(X3[Q], xch(Q, 2), X3[S], ab[3]), s4 = nbr(X4[S], xch(Q, 3), X4[Q], ab[4]);
            const V2 d1 = fma2(mone, s1, vRa[Q]), d2 = fma2(mone, fma2(ac[2], X1[S], s2), vBa[S]);
            const V2 d3 = fma2(mone, fma2(ac[3], X2[Q], s3), vRb[Q]), t4 = fma2(ac[4], X3[S], s4);
            x1 = mul2(w[0], vB);                             // 0: plane q, black
            x2 = mul2(w[1], fma2(nat[1], x1, d1));           // 1: plane q - 1, red
            x3 = fma2(w[2], fma2(nat[2], x2, d2), X1[S]);    // 2: plane q - 2, black
            x4 = fma2(w[3], fma2(nat[3], x3, d3), X2[Q]);    // 3: plane q - 3, red
            tRn = fma2(ac[3], x4, fma2(at[3], x3, s3));      // the product, red
            tB = fma2(at[4], x4, t4);                        // and black, plane q - 4
        }
        put(xch(S, 0), x1);
        put(xch(S, 1), x2);
        put(xch(S, 2), x3);
        put(xch(S, 3), x4);
        const V2 zB = X3[Q];   // plane q - 3, black
        X1[S] = x1; X2[Q] = x2; X3[S] = x3; X4[Q] = x4;
        if (in3) {
            store(vec.z, c - 3 * sxy, S == 0 ? mk2(x4.x, zB.x) : mk2(zB.x, x4.x), S == 0 ? mk2(zB.y, x4.y) : mk2(x4.y, zB.y));
            if (MODE == 1) {
                if (S == 0 ? st0 : st1) {
                    const double y = to_d(tRn.x);
                    acc[0] += y * to_d(vRb[Q].x); acc[NV - 1] += y * y;
                }
                if (S == 0 ? st3 : st2_) {
                    const double y = to_d(tRn.y);
                    acc[0] += y * to_d(vRb[Q].y); acc[NV - 1] += y * y;
                }
            }
        }
        if (q - 4 >= k0) {   // q - 4 < k1 always
            const V2 y0 = S == 0 ? mk2(tB.x, tR.x) : mk2(tR.x, tB.x), y1 = S == 0 ? mk2(tR.y, tB.y) : mk2(tB.y, tR.y);
            store(L::CSM ? sptr[3] : yout, c - 4 * sxy, y0, y1);
            if (MODE == 0) {
                if (st0) acc[0] += to_d(rr0.x) * to_d(y0.x);
                if (st1) acc[0] += to_d(rr0.y) * to_d(y0.y);
                if (st2_) acc[0] += to_d(rr1.x) * to_d(y1.x);
                if (st3) acc[0] += to_d(rr1.y) * to_d(y1.y);
            } else {
                if (S == 0 ? st0 : st1) {
                    const double y = to_d(tB.x);
                    acc[0] += y * to_d(vBb[S].x); acc[NV - 1] += y * y;
                }
                if (S == 0 ? st3 : st2_) {
                    const double y = to_d(tB.y);
                    acc[0] += y * to_d(vBb[S].y); acc[NV - 1] += y * y;
                }
            }
        }
        if (MODE == 0 && in3) {   // rr of the next iteration's product plane
            const T *a = vec.rr + (c - 3 * sxy), *b = a + g.sx;
            if (ALN) {
                if (st0) rr0 = ld2(a);
                if (st2_) rr1 = ld2(b);
            } else {
                if (st0) rr0.x = a[0];
                if (st1) rr0.y = a[1];
                if (st2_) rr1.x = b[0];
                if (st3) rr1.y = b[1];
            }
        }
        tR = tRn;
        vBb[S] = vBa[S]; vBa[S] = vB;
        vRb[S] = vRa[S]; vRa[S] = vR;
    };
    __syncthreads();   // ztab, the zeroed exchange planes
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    unsigned c = c00 + (unsigned)qs * sxy;
    for (int q = qs; q <= qe; q += 2, c += 2 * sxy) {
        if (!GEN && q - 4 >= zr0 && q + 1 < zr1) {
            if constexpr (!GEN) {
                iter(P0{}, std::true_type{}, q, c);
                if (q + 1 > qe) break;
                iter(P1{}, std::true_type{}, q + 1, c + sxy);
            }
        } else {
            iter(P0{}, std::false_type{}, q, c);
            if (q + 1 > qe) break;
            iter(P1{}, std::false_type{}, q + 1, c + sxy);
        }
    }
    cp_async_wait<0>();
    double tot[NV];
    if (grid_sum<NV, L::NW>(acc, rw, tot) && tid == 0) {
        if (MODE == 0) derive_alpha(sc, tot);
        else if constexpr (NV == 2) derive_omega(sc, tot);
    }
}

}  // namespace fb
