/*
 * Several linear-spherical time steps per launch, the tile held in registers,
 * for sm_100a.
 *
 * One launch advances every grid of its work by T outer steps: MASS_S
 * (mass.f90:61-100), the OPEN radiation boundary (boundaries.f90:22-202) and
 * MOMT_S (moment.f90:65-149), with the maximum-amplitude recorder
 * (GPUOutput.cu:46-53), the arrival record and the gauge samples (GET_TS,
 * output.f90:1078-1090) of every step.
 *
 * Work decomposition: a CTA of NW warps owns a window of 128 columns x
 * RW = R*NW rows.  A lane owns four adjacent columns of R rows and keeps
 * their Z, M, N and max-eta in registers from the first step of the launch
 * to the last; a warp's R rows lie under the next warp's.  Neighbours along
 * I are warp shuffles, neighbours along J are the lane's own registers, and
 * the one row above and the one row below a warp's block cross through
 * shared memory, once per step.  A step's result is exact where the previous
 * step was exact one cell further out, so after T steps a margin of T cells
 * at each side of the window is stale: windows overlap by it (by T rounded
 * up to a multiple of 4 along I, so that a lane lies in the margin or outside
 * it as a whole and its loads and stores stay 16-byte aligned) and only the
 * core is stored.  At the grid's own edges there is no margin: the perimeter
 * takes OPEN and the clamps, which read nothing beyond it.
 *
 * Arithmetic: the four columns of a lane are the halves of two packed
 * operations (add/sub/mul .rn.f32x2, each half rounded separately), except
 * where an operand is shifted by one column.  The order of operations is the
 * Fortran's, so the results are the bits of T launches of the one-step kernel.
 *
 * Three step bodies, chosen per warp and launch: `fast` where every cell the
 * warp computes is wet and inside the grid (no land tests; the EPS flush and
 * the land clamp are selects that can only act where a minimum over the
 * warp's values says so), `edge` where every cell is wet but the grid's
 * perimeter is among them, `gen` with the land tests from bit masks.  OPEN's
 * square roots and divisions are spread over the CTA's threads
 * (open_cells): evaluated by the perimeter's own lanes they made a corner
 * window last three times an inner one.  A warp whose water is still in every
 * reach of the step computes nothing for that step.
 *
 * What bounds it (ncu, 2401 x 2001, waves everywhere, 64-row windows, 8
 * steps): no unit is full.  46 % of the issue slots are busy with 15.5 warps
 * an SM (128 registers a thread), the FMA pipe 28 % and the ALU pipe 35 % of
 * the cycles, DRAM 9 % of its rate.  Per issued instruction a warp waits 1.4
 * cycles for a math pipe (a packed operation holds it for two cycles), 1.4 for
 * a fixed latency, 1.0 at the step's barrier and 0.7 for shared memory.  Its
 * 924 windows are 6.2 waves of one CTA an SM, so 14 % of the time is the last
 * wave.
 *
 * Time per step of eager launches, waves everywhere, against the two-step
 * kernel (kernels_pair.cu) on the same B200: 361 x 301 2.8 us against 8.3,
 * 961 x 801 4.5 against 9.8, 1201 x 1001 5.4 against 11.6, 2401 x 2001 19.0
 * against 22.1, eight grids of 1201 x 1001 39 against 47, 64 such grids 304
 * against 303.  Young forecasts, their waves in one corner: 2401 x 2001 10.8
 * against 21.4, 64 of 1201 x 1001 223 against 302.
 *
 * Tried and measured slower on 2401 x 2001 with 4 steps a launch: 64 columns a
 * window and two a lane (35 us a step, with twice the exchange and shuffles a
 * cell); a persistent form with the next window's fields fetched by tensor
 * copies into shared memory while this one steps, results out by tensor copies
 * (12 warps an SM, 24 us: the buffers cost the warps that hide latency); 1-D
 * copies issued by every lane (200 copies a window, 24 cycles each, 26 us).
 *
 * No copy engine and no waits on memory barriers of its own: plain loads, all
 * of a window's rows in flight at once, and CTA barriers.
 */
#include <math.h>

#include <algorithm>
#include <atomic>

#include "fused.h"
#include "packed.cuh"

namespace {

using namespace gcpacked;

constexpr int BW = 128; /* columns of a window */

/* the flush, and 0 on columns whose bit (row r of a mask of four bits a row)
 * is clear */
__device__ __forceinline__ float fkeep(float x, unsigned bit) { return (bit != 0 && !(fabsf(x) < CC_EPS)) ? x : 0.0f; }
__device__ __forceinline__ V4 fkeep4(const V4 &v, unsigned mask, int r) {
    return v4(fkeep(v.a.x, mask & (1u << (4 * r))), fkeep(v.a.y, mask & (2u << (4 * r))),
              fkeep(v.b.x, mask & (4u << (4 * r))), fkeep(v.b.y, mask & (8u << (4 * r))));
}

/* ---- layout ---- */
/* windows along one axis of n cells: width w, margin g at each side, stride
 * w - 2g */
__host__ __device__ __forceinline__ int block_count(int n, int w, int g) {
    return n <= w ? 1 : 1 + (n - w + (w - 2 * g) - 1) / (w - 2 * g);
}
/* margin columns for t steps: whole lanes */
__host__ __device__ __forceinline__ int block_hc(int t) { return (t + 3) & ~3; }

template <int R, int NW>
struct BlockSmem {
    static constexpr int RW = R * NW;
    float ex[2][NW][4][BW];   /* per step parity and warp: row 0's Z, M, N and row R-1's N */
    float r2[RW][BW];         /* R2 and R4 of the window's faces */
    float r4[RW][BW];
    float h[RW + 2][BW];      /* depth of rows -1 .. RW */
    float4 c1[RW + 2];        /* R1 R1 R11 R11 */
    float4 c2[RW + 2];        /* R6 R6 CX CY */
    float4 c3[RW + 2];        /* R3 R3 R5 R5 */
    float col[4][RW + 2];     /* perimeter columns of rows -1 .. RW: M, N (west), M, N (east) */
    /* OPEN on the perimeter cells of the window: rows (the grid's first, its
     * last) and columns (west, east; rows 0 .. RW): sqrt(g h) there, 0 where
     * dry, and a step's values; M of the last row and N of the one below it */
    float crow[2][BW], orow[2][BW], last[2][BW];
    float ccol[2][RW + 1], ocol[2][RW + 1];
    int ngl;                  /* gauges of the core */
    int gl[64];
};

enum { M_FAST = 0, M_EDGE = 1, M_GEN = 2 };

/* what a warp's step needs besides its state */
struct WarpCtx {
    int ib, jw, nx, ny;
    bool finite;           /* every coefficient and depth of the warp is (so still water stays still) */
    bool edge, west, east; /* the warp's rows touch or pass the perimeter; its first, its last column (warp-uniform) */
    int le, qe;            /* lane and column of the grid's last column */
    float hmin;            /* smallest depth of the warp's wet cells */
    unsigned wc, fx, fy;   /* wet cells (rows 0..R), wet x faces, wet y faces; four bits a row */
};

/* a window's perimeter, the same for all its threads */
struct Perimeter {
    int first, last; /* it holds the grid's first row (as its own), its last row: row index in the window or -1 */
    int west, east;  /* it holds the grid's first column, its last: column index in the window or -1 */
    __device__ __forceinline__ bool any() const { return first >= 0 || last >= 0 || west >= 0 || east >= 0; }
};

/* OPEN on all the window's perimeter cells, spread over the CTA's threads: a
 * square root and a division per cell, which one warp alone would run through
 * one after the other.  It needs the old level only: the rows' M and N from
 * the exchange buffer or `last`, the columns' from `col`. */
template <int R, int NW>
__device__ __forceinline__ void open_cells(BlockSmem<R, NW> &S, const float (*H)[BW], const Perimeter &p,
                                           const float (*ex)[4][BW], int sj, int ny) {
    constexpr int RW = R * NW;
    const int nrow = (p.first >= 0 ? BW : 0) + (p.last >= 0 ? BW : 0);
    const int n = nrow + (p.west >= 0 ? RW + 1 : 0) + (p.east >= 0 ? RW + 1 : 0);
#pragma unroll 1
    for (int k = threadIdx.x; k < n; k += 32 * NW) {
        float a, b, c, *out;
        bool neg;
        if (k < nrow) {
            const int i = k & (BW - 1), l = p.first >= 0 && k < BW ? 0 : 1;
            const float *m = l ? S.last[0] : ex[0][1], *across = l ? S.last[1] : ex[0][2];
            a = 0.5f * (m[i] + m[i > 0 ? i - 1 : 0]);
            b = across[i];
            neg = l ? b < 0.0f : b > 0.0f;
            c = S.crow[l][i];
            out = &S.orow[l][i];
        } else {
            const int side = p.west >= 0 && k - nrow <= RW ? 0 : 1;
            const int r = k - nrow - (side == 1 && p.west >= 0 ? RW + 1 : 0), j = sj + r;
            /* west: M, east: M one column west, as the owner left it */
            const float m = S.col[2 * side][r + 1], nc = S.col[2 * side + 1][r + 1], ns = S.col[2 * side + 1][r];
            const bool corner = j == 0 || j == ny - 1;
            /* the west side takes N alone where the cell below is dry */
            const float along = (side == 0 && !(H[r][p.west] > CC_GX)) ? nc : 0.5f * (nc + ns);
            a = corner ? m : along;
            b = corner ? (j == 0 ? nc : ns) : m;
            neg = side == 0 ? m > 0.0f : m < 0.0f;
            if (corner) neg = neg || (j == 0 ? b > 0.0f : b < 0.0f);
            c = S.ccol[side][r];
            out = &S.ocol[side][r];
        }
        *out = open_value(a, b, c > 0.0f ? c : 1.0f, neg, c > 0.0f);
    }
}

/* puts OPEN over the new surface of a warp's perimeter cells */
template <int R, int NW>
__device__ __forceinline__ void open_rows(BlockSmem<R, NW> &S, const WarpCtx &W, int w, int lane, V4 (&zn)[R + 1],
                                          const V4 (&m)[R], const V4 &mu, float (&mw)[R + 1]) {
#pragma unroll
    for (int r = 0; r <= R; r++) {
        if (W.jw + r == 0) zn[r] = lds4(&S.orow[0][4 * lane]);
        if (W.jw + r == W.ny - 1) zn[r] = lds4(&S.orow[1][4 * lane]);
    }
    if (W.west && lane == 0) {
#pragma unroll
        for (int r = 0; r <= R; r++) {
            zn[r].a.x = S.ocol[0][w * R + r];
            mw[r] = r < R ? m[r < R ? r : 0].a.x : mu.a.x; /* IM1 = max(I-1,1) */
        }
    }
    if (W.east && lane == W.le) {
#pragma unroll
        for (int r = 0; r <= R; r++) {
            const float o = S.ocol[1][w * R + r];
            zn[r].a.x = W.qe == 0 ? o : zn[r].a.x;
            zn[r].a.y = W.qe == 1 ? o : zn[r].a.y;
            zn[r].b.x = W.qe == 2 ? o : zn[r].b.x;
            zn[r].b.y = W.qe == 3 ? o : zn[r].b.y;
        }
    }
}

/* the CTA's barrier, from code that differs between its warps; and the one
 * that says OPEN's values are in shared memory, which warps without a
 * perimeter cell pass without waiting */
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 0;" ::: "memory"); }
template <int NT>
__device__ __forceinline__ void open_arrive() {
    __threadfence_block();
    asm volatile("bar.arrive 1, %0;" ::"n"(NT) : "memory");
}
template <int NT>
__device__ __forceinline__ void open_wait() {
    asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

template <int R, int NW, int MODE>
__device__ __forceinline__ bool block_step(BlockSmem<R, NW> &S, const float (*H)[BW], const WarpCtx &W, int w, int lane, V4 (&z)[R],
                                           V4 (&m)[R], V4 (&n)[R], const V4 &ns, const V4 &zu, const V4 &mu,
                                           const V4 &nu) {
    const int q0 = w * R + 1; /* shared row of the warp's row 0 */
    bool tiny = false;        /* some value was below the flush */
    V4 zn[R + 1];             /* the new surface of rows 0 .. R */
    float mw[R + 1];          /* M one column west of the lane's first */
    /* MASS_S (mass.f90:82-95) */
    {
        float amin = 3.0e38f, zmin = 3.0e38f;
        const float r6m = S.c2[q0 - 1].x;
        V4 nrs = make_float2(r6m, r6m) * ns; /* N * R6 of the row below */
#pragma unroll
        for (int r = 0; r <= R; r++) {
            const int rr = r < R ? r : 0;
            const V4 &zc = r < R ? z[rr] : zu, &mc = r < R ? m[rr] : mu, &nc = r < R ? n[rr] : nu;
            mw[r] = shw(mc.b.y);
            const float4 c1 = S.c1[q0 + r];
            const float2 r6 = *reinterpret_cast<const float2 *>(&S.c2[q0 + r]);
            const V4 nr = r6 * nc;
            const V4 d = v4(mc.a.x - mw[r], mc.a.y - mc.a.x, mc.b.x - mc.a.y, mc.b.y - mc.b.x);
            V4 zz = (zc - make_float2(c1.x, c1.y) * d) - make_float2(c1.z, c1.w) * (nr - nrs);
            nrs = nr;
            if (MODE != M_GEN) amin = minabs4(amin, zz);
            else zz = fkeep4(zz, W.wc, r);
            zmin = min4(zmin, zz);
            zn[r] = zz;
        }
        /* with every cell wet the flush is left to the minimum of |Z|; the
         * clamp Z+H <= EPS can act only where the smallest Z plus the smallest
         * wet H is at or below it (float addition is monotonic) */
        if (MODE != M_GEN) {
            tiny = __any_sync(FULL, amin < CC_EPS);
            if (tiny) {
#pragma unroll
                for (int r = 0; r <= R; r++) zn[r] = flush4(zn[r]);
            }
        }
        if (__any_sync(FULL, zmin + W.hmin <= CC_EPS)) {
#pragma unroll
            for (int r = 0; r <= R; r++) {
                const V4 c = clamp4(zn[r], lds4(&H[q0 + r][4 * lane]));
                zn[r] = MODE != M_GEN ? c
                                      : v4(W.wc & (1u << (4 * r)) ? c.a.x : 0.0f, W.wc & (2u << (4 * r)) ? c.a.y : 0.0f,
                                           W.wc & (4u << (4 * r)) ? c.b.x : 0.0f, W.wc & (8u << (4 * r)) ? c.b.y : 0.0f);
            }
        }
        if (MODE != M_FAST && W.edge) {
            open_wait<32 * NW>();
            open_rows<R, NW>(S, W, w, lane, zn, m, mu, mw);
        }
    }
    /* MOMT_S (moment.f90:86-145) */
    {
        float amin = 3.0e38f;
        V4 nsr = ns;            /* N of row r-1 */
        float nse = she(ns.a.x); /* and one column east of the lane's last */
#pragma unroll
        for (int r = 0; r < R; r++) {
            const float4 c3 = S.c3[q0 + r];
            const V4 r2 = lds4(&S.r2[q0 - 1 + r][4 * lane]), r4 = lds4(&S.r4[q0 - 1 + r][4 * lane]);
            const V4 mc = m[r], nc = n[r], ma = r + 1 < R ? m[r + 1 < R ? r + 1 : 0] : mu;
            const V4 &zc = zn[r];
            const float ze = she(zc.a.x), ne = she(nc.a.x);
            /* x faces: N of rows r and r-1 */
            V4 tot = v4(nc.a.x + nc.a.y, nc.a.y + nc.b.x, nc.b.x + nc.b.y, nc.b.y + ne) + nsr;
            tot = v4(tot.a.x + nsr.a.y, tot.a.y + nsr.b.x, tot.b.x + nsr.b.y, tot.b.y + nse);
            const V4 dz = v4(zc.a.y - zc.a.x, zc.b.x - zc.a.y, zc.b.y - zc.b.x, ze - zc.b.y);
            V4 vm = (mc - r2 * dz) + make_float2(c3.x, c3.y) * tot;
            /* y faces: M of rows r and r+1 */
            V4 tm = v4(mw[r] + mw[r + 1], mc.a.x + ma.a.x, mc.a.y + ma.a.y, mc.b.x + ma.b.x);
            tm = (tm + mc) + ma;
            V4 vn = (nc - r4 * (zn[r + 1] - zc)) - make_float2(c3.z, c3.w) * tm;
            if (MODE != M_GEN) {
                amin = minabs4(minabs4(amin, vm), vn);
            } else {
                vm = fkeep4(vm, W.fx, r);
                vn = fkeep4(vn, W.fy, r);
            }
            nsr = nc;
            nse = ne;
            m[r] = vm;
            n[r] = vn;
        }
        if (MODE != M_GEN) {
            if (__any_sync(FULL, amin < CC_EPS)) {
                tiny = true;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    m[r] = flush4(m[r]);
                    n[r] = flush4(n[r]);
                }
            }
            if (MODE == M_EDGE) { /* M to column NX-1, N to row NY-1 (the masks see to it elsewhere) */
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (W.east && lane == W.le) {
                        m[r].a.x = W.qe == 0 ? 0.0f : m[r].a.x;
                        m[r].a.y = W.qe == 1 ? 0.0f : m[r].a.y;
                        m[r].b.x = W.qe == 2 ? 0.0f : m[r].b.x;
                        m[r].b.y = W.qe == 3 ? 0.0f : m[r].b.y;
                    }
                    if (W.jw + r == W.ny - 1) n[r] = v4(0.f, 0.f, 0.f, 0.f);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) z[r] = zn[r];
    return MODE == M_GEN || tiny;
}

/* one gauge record of the stencil values l1..l4 at step index `k` */
template <class Desc>
__device__ __forceinline__ void gauge_record(const Desc &G, int k, int g, float l1, float l2, float l3, float l4) {
    if (G.flags & GC_F_STENCIL) {
        float *o = G.ts + ((size_t)k * G.ng + g) * 4;
        o[0] = l1; o[1] = l2; o[2] = l3; o[3] = l4;
    } else {
        const float cx = G.gw[2 * g], cy = G.gw[2 * g + 1];
        const float a = l1 * (1.0f - cx) * (1.0f - cy);
        const float b = l2 * (cx) * (1.0f - cy);
        const float d = l3 * (1.0f - cx) * (cy);
        const float e = l4 * (cx) * (cy);
        G.ts[(size_t)k * G.ng + g] = a + b + d + e;
    }
}

/* a window of one grid: where it lies and what it stores */
struct Window {
    int s, sj;            /* first column and row */
    int lo, hi, jlo, jhi; /* stored columns and rows */
};
/* window lt of a grid: the perimeter's windows first, since their OPEN makes
 * them dearer */
template <class Desc>
__device__ __forceinline__ Window block_window(const Desc &G, int rw, int lt) {
    int tx, ty;
    const int ntx = G.bntx, nty = G.bnty;
    if (ntx < 3 || nty < 3) {
        ty = ntx == 1 ? lt : (int)__umulhi((unsigned)lt, G.bmag);
        tx = lt - ty * ntx;
    } else if (lt < 2 * ntx) {
        tx = lt >> 1;
        ty = (lt & 1) ? nty - 1 : 0;
    } else if (lt < G.bper) {
        const int k = lt - 2 * ntx;
        tx = (k & 1) ? ntx - 1 : 0;
        ty = 1 + (k >> 1);
    } else {
        const int k = lt - G.bper, d = ntx - 2, y = d == 1 ? k : (int)__umulhi((unsigned)k, G.bmag);
        tx = 1 + k - y * d;
        ty = 1 + y;
    }
    const int hc = block_hc(G.bt);
    Window q;
    q.s = tx * (BW - 2 * hc);
    q.sj = ty * (rw - 2 * G.bt);
    q.lo = tx == 0 ? 0 : q.s + hc;
    q.hi = tx == ntx - 1 ? G.nx - 1 : q.s + BW - 1 - hc;
    q.jlo = ty == 0 ? 0 : q.sj + G.bt;
    q.jhi = ty == nty - 1 ? G.ny - 1 : q.sj + rw - 1 - G.bt;
    return q;
}
/* the buffers a launch of T steps reads and writes */
template <class Desc>
__device__ __forceinline__ void block_levels(const Desc &G, int local, int T, int &rd, int &wr) {
    if (G.nbuf == 3) {
        rd = local % 3;
        wr = (local + T) % 3;
    } else {
        rd = G.cur0 ^ (local & 1);
        wr = rd ^ 1;
    }
}

/* T steps of a warp's rows, from and to registers */
template <int R, int NW, int MODE, class Desc>
__device__ __forceinline__ void block_run(const Desc &G, BlockSmem<R, NW> &S, const float (*H)[BW], const WarpCtx &W,
                                          const Window &q, const Perimeter &per, int T, int local, int ngl,
                                          V4 (&z)[R], V4 (&m)[R], V4 (&n)[R],
                                          V4 (&x)[R]) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool do_max = (G.flags & GC_F_MAXAMP) != 0;
    const float thr = G.thr;
    /* a cell arrives when it is above the threshold and its maximum before was
     * not; where every maximum of the lane is above it none can any more */
    bool pend = false, first = true;
    bool tiny = W.finite; /* the last step met values below the flush: this warp's water may be still */
    for (int t = 0; t < T; t++) {
        float(*ex)[4][BW] = S.ex[t & 1];
        sts4(&ex[w][0][4 * lane], z[0]);
        sts4(&ex[w][1][4 * lane], m[0]);
        sts4(&ex[w][2][4 * lane], n[0]);
        sts4(&ex[w][3][4 * lane], n[R - 1]);
        if (MODE != M_FAST && W.west && lane == 0) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                S.col[0][w * R + 1 + r] = m[r].a.x;
                S.col[1][w * R + 1 + r] = n[r].a.x;
            }
        }
        if (MODE != M_FAST && W.east) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float mwr = shw(m[r].b.y);
                if (lane == W.le) {
                    S.col[2][w * R + 1 + r] = W.qe == 0 ? mwr : comp(m[r], W.qe - 1);
                    S.col[3][w * R + 1 + r] = comp(n[r], W.qe);
                }
            }
        }
        if (MODE != M_FAST && per.last >= 0) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                if (w * R + r == per.last) sts4(&S.last[0][4 * lane], m[r]);
                if (w * R + r == per.last - 1) sts4(&S.last[1][4 * lane], n[r]);
            }
        }
        cta_sync();
        if (MODE != M_FAST || per.any()) {
            open_cells<R, NW>(S, H, per, ex, q.sj, W.ny);
            if (per.any() && !(MODE != M_FAST && W.edge)) open_arrive<32 * NW>();
        }
        /* below the window's first row: its own N (JM1 = max(J-1,1) at the
         * grid's first row, a stale margin elsewhere); above its last row:
         * that row again (dry past the grid, a stale margin elsewhere) */
        const V4 ns = lds4(w > 0 ? &ex[w - 1][3][4 * lane] : &ex[0][2][4 * lane]);
        const int wu = w < NW - 1 ? w + 1 : w;
        const V4 zu = lds4(&ex[wu][0][4 * lane]), mu = lds4(&ex[wu][1][4 * lane]), nu = lds4(&ex[wu][2][4 * lane]);
        /* a warp whose rows lie beyond what later steps and the core need of
         * this one has nothing left to compute, nor has one whose water is
         * still: from +0 everywhere in reach each equation gives +0, the OPEN
         * boundary's included (most of an ocean until the wave gets there).
         * The test is made where the last step met values below the flush. */
        const int left = T - 1 - t;
        const bool work = (MODE != M_FAST && W.edge) || (W.jw + R - 1 >= q.jlo - left && W.jw <= q.jhi + left);
        bool still = false;
        if (work && tiny && W.finite) {
            unsigned b = bits4(ns) | bits4(zu) | bits4(mu) | bits4(nu);
#pragma unroll
            for (int r = 0; r < R; r++) b |= bits4(z[r]) | bits4(m[r]) | bits4(n[r]);
            still = __all_sync(FULL, b == 0);
            if (MODE != M_FAST && still && W.edge) open_arrive<32 * NW>();
        }
        if (work && !still) {
            tiny = block_step<R, NW, MODE>(S, H, W, w, lane, z, m, n, ns, zu, mu, nu);
            if (first && (G.flags & GC_F_ARRIVAL)) {
                float xt = 3.0e38f;
#pragma unroll
                for (int r = 0; r < R; r++) xt = min4(xt, x[r]);
                pend = __any_sync(FULL, xt <= thr);
            }
            first = false;
            if (pend) {
                float zt = -3.0e38f;
#pragma unroll
                for (int r = 0; r < R; r++) zt = max4(zt, z[r]);
                if (zt > thr) {
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        const int j = W.jw + r;
                        const float zv[4] = {z[r].a.x, z[r].a.y, z[r].b.x, z[r].b.y};
                        const float xv[4] = {x[r].a.x, x[r].a.y, x[r].b.x, x[r].b.y};
                        int *row = G.arrival + (size_t)j * G.pitch;
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int i = W.ib + k;
                            if (zv[k] > thr && xv[k] <= thr && (W.wc >> (4 * r + k) & 1) && j >= q.jlo && j <= q.jhi &&
                                i >= q.lo && i <= q.hi)
                                row[i] = local + t + 1;
                        }
                    }
                }
            }
        }
        /* max-eta: keeps the old value unless the new surface is above it */
        if (work && do_max) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                x[r].a.x = x[r].a.x >= z[r].a.x ? x[r].a.x : z[r].a.x;
                x[r].a.y = x[r].a.y >= z[r].a.y ? x[r].a.y : z[r].a.y;
                x[r].b.x = x[r].b.x >= z[r].b.x ? x[r].b.x : z[r].b.x;
                x[r].b.y = x[r].b.y >= z[r].b.y ? x[r].b.y : z[r].b.y;
            }
        }
        if (ngl > 0 && t < T - 1) {
            /* the surface goes through the exchange buffer of the other
             * parity, whose readers are past this step's barrier and whose
             * next writers wait for the second one here */
            static_assert(R <= 4, "a surface fits one parity of the exchange buffer");
            float(*zg)[BW] = reinterpret_cast<float(*)[BW]>(&S.ex[(t + 1) & 1][0][0][0]);
#pragma unroll
            for (int r = 0; r < R; r++) sts4(&zg[w * R + r][4 * lane], z[r]);
            cta_sync();
            for (int k = tid; k < ngl; k += 32 * NW) {
                const int g = S.gl[k];
                const int ki = G.gij[2 * g] - 1 - q.s, kj = G.gij[2 * g + 1] - 1 - q.sj;
                gauge_record(G, local + t, g, zg[kj][ki], zg[kj][ki + 1], zg[kj + 1][ki], zg[kj + 1][ki + 1]);
            }
            cta_sync();
        }
    }
}

/* one window: T steps from time level `local` of grid G */
template <int R, int NW, class Desc>
__device__ __forceinline__ void block_tile(const Desc &G, int lt, int step, int T, BlockSmem<R, NW> &S) {
    constexpr int RW = R * NW;
    const int local = step - G.step0;
    if (local < 0 || local > G.nsteps) return;
    const bool run = local + T <= G.nsteps; /* the launch after a grid's last step only samples its gauges */
    const int nx = G.nx, ny = G.ny;
    const unsigned P = (unsigned)G.pitch;
    int rd, wr;
    block_levels(G, local, T, rd, wr);
    const Window q = block_window(G, RW, lt);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool do_max = (G.flags & GC_F_MAXAMP) != 0;
    const int ng = G.ng;
    WarpCtx W;
    W.ib = q.s + 4 * lane;
    W.jw = q.sj + w * R;
    W.nx = nx;
    W.ny = ny;
    const float(*H)[BW] = S.h;
    V4 z[R], m[R], n[R], x[R];
    if (run) {
        /* all rows of a lane in flight together */
        float4 hq[R], hx = make_float4(1.0e4f, 1.0e4f, 1.0e4f, 1.0e4f);
        const char *zp = (const char *)G.z[rd], *mp = (const char *)G.m[rd], *np = (const char *)G.n[rd];
        const char *hp = (const char *)G.h, *xp = (const char *)G.zmax;
        const unsigned p4 = 4u * P, off = (unsigned)W.jw * p4 + 4u * (unsigned)W.ib;
        const int jx = w == 0 ? q.sj - 1 : q.sj + RW; /* the depth row beyond the window, for its first and last warp */
        const bool wx = w == 0 || w == NW - 1;
        if (q.s + BW <= nx && W.jw + R <= ny) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const unsigned o = off + (unsigned)r * p4;
                hq[r] = *(const float4 *)(hp + o);
                z[r] = v4(*(const float4 *)(zp + o));
                m[r] = v4(*(const float4 *)(mp + o));
                n[r] = v4(*(const float4 *)(np + o));
                if (do_max) x[r] = v4(*(const float4 *)(xp + o));
            }
            if (wx && jx >= 0 && jx < ny) hx = *(const float4 *)(hp + ((unsigned)jx * p4 + 4u * (unsigned)W.ib));
        } else {
            /* past the grid: the last row or the row's padding, over deep
             * water; what they become reaches no cell of the grid */
            const unsigned ic = 4u * min((unsigned)W.ib, P - 4u);
            auto deep = [&](float4 v, int j) {
                const bool row = j >= 0 && j < ny;
                const float d = 1.0e4f;
                return make_float4(row && W.ib < nx ? v.x : d, row && W.ib + 1 < nx ? v.y : d, row && W.ib + 2 < nx ? v.z : d,
                                   row && W.ib + 3 < nx ? v.w : d);
            };
#pragma unroll
            for (int r = 0; r < R; r++) {
                const unsigned o = (unsigned)min(W.jw + r, ny - 1) * p4 + ic;
                hq[r] = *(const float4 *)(hp + o);
                z[r] = v4(*(const float4 *)(zp + o));
                m[r] = v4(*(const float4 *)(mp + o));
                n[r] = v4(*(const float4 *)(np + o));
                if (do_max) x[r] = v4(*(const float4 *)(xp + o));
            }
            if (wx) hx = deep(*(const float4 *)(hp + ((unsigned)min(max(jx, 0), ny - 1) * p4 + ic)), jx);
#pragma unroll
            for (int r = 0; r < R; r++) hq[r] = deep(hq[r], W.jw + r);
        }
#pragma unroll
        for (int r = 0; r < R; r++) *(float4 *)&S.h[w * R + r + 1][4 * lane] = hq[r];
        if (wx) *(float4 *)&S.h[w == 0 ? 0 : RW + 1][4 * lane] = hx;
    }
    /* gauges whose base cell the core holds; the surface the previous launch
     * left is sampled here, the surfaces inside this launch below */
    if (ng > 0) {
        if (tid == 0) S.ngl = 0;
        __syncthreads();
        for (int g = tid; g < ng && g < 64; g += 32 * NW) {
            const int ki = G.gij[2 * g] - 1, kj = G.gij[2 * g + 1] - 1;
            if (ki >= q.lo && ki <= q.hi && kj >= q.jlo && kj <= q.jhi) {
                S.gl[atomicAdd(&S.ngl, 1)] = g;
                if (local > 0) {
                    const float *c = G.z[rd] + (size_t)kj * P + ki;
                    gauge_record(G, local - 1, g, c[0], c[1], c[P], c[P + 1]);
                }
            }
        }
    }
    if (!run) return;
    for (int k = tid; k < RW + 2; k += 32 * NW) {
        const int j = q.sj - 1 + k;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (j >= 0 && j < ny) {
            a = *reinterpret_cast<const float4 *>(G.rows + (size_t)j * GC_ROWW);
            b = *reinterpret_cast<const float4 *>(G.rows + (size_t)j * GC_ROWW + 4);
        }
        /* record: r1 r11 r6 r3 | r5 cx cy - */
        S.c1[k] = make_float4(a.x, a.x, a.y, a.y);
        S.c2[k] = make_float4(a.z, a.z, b.y, b.z);
        S.c3[k] = make_float4(a.w, a.w, b.x, b.x);
    }
    if (tid < 4) S.col[tid][0] = S.col[tid][RW + 1] = 0.0f;
    for (int k = tid; k < 2 * BW; k += 32 * NW) (&S.last[0][0])[k] = 0.0f;
    __syncthreads();
    const int ngl = ng > 0 ? S.ngl : 0;
    Perimeter per;
    per.first = q.sj == 0 ? 0 : -1;
    per.last = q.sj + RW >= ny - 1 ? ny - 1 - q.sj : -1; /* RW: the row above the window, which its last warp computes */
    per.west = q.s == 0 ? 0 : -1;
    per.east = q.s + BW - 1 >= nx - 1 ? nx - 1 - q.s : -1;
    if (per.any()) {
        auto speed = [](float h) { return h > CC_GX ? sqrtf(CC_GRAV * h) : 0.0f; };
        for (int i = tid; i < 2 * BW; i += 32 * NW) {
            const int l = i >= BW, r = l ? per.last : per.first;
            if (r >= 0) S.crow[l][i & (BW - 1)] = speed(H[r + 1][i & (BW - 1)]);
        }
        for (int i = tid; i < 2 * (RW + 1); i += 32 * NW) {
            const int e = i > RW, r = e ? i - RW - 1 : i, c = e ? per.east : per.west;
            if (c >= 0) S.ccol[e][r] = speed(H[r + 1][c]);
        }
    }
    int mode;
    {
        float hm = 3.0e38f, hx = 0.0f;
        V4 h = lds4(&H[w * R + 1][4 * lane]);
#pragma unroll
        for (int r = 0; r <= R; r++) {
            hm = min4nan(hm, h); /* NaN when a depth is */
            hx = max4(hx, h);
            if (r < R) {
                const float he = she(h.a.x);
                const V4 ha = lds4(&H[w * R + r + 2][4 * lane]);
                const float4 c2 = S.c2[w * R + r + 1];
                /* R2 = CX * (HP), HP the mean of the two cells (0.5f * sum, then the factor) */
                const float2 half = make_float2(0.5f, 0.5f);
                const V4 hs = v4(h.a.x + h.a.y, h.a.y + h.b.x, h.b.x + h.b.y, h.b.y + he);
                sts4(&S.r2[w * R + r][4 * lane], make_float2(c2.z, c2.z) * (half * hs));
                sts4(&S.r4[w * R + r][4 * lane], make_float2(c2.w, c2.w) * (half * (h + ha)));
                h = ha;
            }
        }
        {
            const int k = w * R + min(lane, R + 1); /* the warp's rows, the one below and the one above */
            const float4 c1 = S.c1[k], c2 = S.c2[k], c3 = S.c3[k];
            const float big = 1.0e30f;
            W.finite = __all_sync(FULL, hx < big && fabsf(c1.x) < big && fabsf(c1.z) < big && fabsf(c2.x) < big &&
                                            fabsf(c2.z) < big && fabsf(c2.w) < big && fabsf(c3.x) < big && fabsf(c3.z) < big);
        }
        const bool inside = q.s >= 1 && q.s + BW - 1 <= nx - 2 && W.jw >= 1 && W.jw + R <= ny - 2;
        const bool wet = __all_sync(FULL, hm > CC_GX);
        mode = !wet ? M_GEN : inside ? M_FAST : M_EDGE;
        W.edge = !inside;
        W.west = q.s == 0;
        W.east = q.s + BW - 1 >= nx - 1;
        W.le = (nx - 1 - q.s) >> 2;
        W.qe = (nx - 1 - q.s) & 3;
        W.wc = W.fx = W.fy = 0xffffffffu;
        if (mode == M_GEN) {
            W.wc = W.fx = W.fy = 0;
            hm = 3.0e38f;
            h = lds4(&H[w * R + 1][4 * lane]);
            const unsigned left = (unsigned)max(0, min(4, nx - W.ib)); /* columns inside the grid */
            const unsigned cin = (1u << left) - 1u;
#pragma unroll
            for (int r = 0; r <= R; r++) {
                const int j = W.jw + r;
                unsigned b = (h.a.x > CC_GX ? 1u : 0u) | (h.a.y > CC_GX ? 2u : 0u) | (h.b.x > CC_GX ? 4u : 0u)
                             | (h.b.y > CC_GX ? 8u : 0u);
                b &= j < ny ? cin : 0u;
                W.wc |= b << (4 * r);
                hm = min4(hm, v4(b & 1 ? h.a.x : hm, b & 2 ? h.a.y : hm, b & 4 ? h.b.x : hm, b & 8 ? h.b.y : hm));
                if (r < R) {
                    /* east of the window: a stale margin, or past the grid */
                    const float he = she(h.a.x);
                    const unsigned be = (b >> 1) | (W.ib + 4 < nx && he > CC_GX ? 8u : 0u);
                    const V4 ha = lds4(&H[w * R + r + 2][4 * lane]);
                    const unsigned ba = (ha.a.x > CC_GX ? 1u : 0u) | (ha.a.y > CC_GX ? 2u : 0u)
                                        | (ha.b.x > CC_GX ? 4u : 0u) | (ha.b.y > CC_GX ? 8u : 0u);
                    W.fx |= (b & be) << (4 * r);
                    W.fy |= (j + 1 < ny ? b & ba : 0u) << (4 * r);
                    h = ha;
                }
            }
        }
        /* the smallest wet depth; positive floats order as their bit patterns */
        W.hmin = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(hm)));
    }
    if (mode == M_FAST) block_run<R, NW, M_FAST>(G, S, H, W, q, per, T, local, ngl, z, m, n, x);
    else if (mode == M_EDGE) block_run<R, NW, M_EDGE>(G, S, H, W, q, per, T, local, ngl, z, m, n, x);
    else block_run<R, NW, M_GEN>(G, S, H, W, q, per, T, local, ngl, z, m, n, x);
    /* the core */
    const unsigned p4 = 4u * P;
    unsigned o = (unsigned)W.jw * p4 + 4u * (unsigned)W.ib;
    char *zo = (char *)G.z[wr], *mo = (char *)G.m[wr], *no = (char *)G.n[wr], *xo = (char *)G.zmax;
    const bool whole = W.ib >= q.lo && W.ib + 3 <= q.hi, part = !whole && W.ib + 3 >= q.lo && W.ib <= q.hi;
#pragma unroll
    for (int r = 0; r < R; r++, o += p4) {
        const int j = W.jw + r;
        if (j < q.jlo || j > q.jhi) continue;
        if (whole) {
            *(float4 *)(zo + o) = f4(z[r]);
            *(float4 *)(mo + o) = f4(m[r]);
            *(float4 *)(no + o) = f4(n[r]);
            if (do_max) *(float4 *)(xo + o) = f4(x[r]);
        }
        if (part) {
            const float4 zv = f4(z[r]), mv = f4(m[r]), nv = f4(n[r]), xv = f4(x[r]);
            const float zz[4] = {zv.x, zv.y, zv.z, zv.w}, mm[4] = {mv.x, mv.y, mv.z, mv.w};
            const float nn[4] = {nv.x, nv.y, nv.z, nv.w}, xx[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int i = W.ib + k;
                if (i < q.lo || i > q.hi) continue;
                *(float *)(zo + o + 4 * k) = zz[k];
                *(float *)(mo + o + 4 * k) = mm[k];
                *(float *)(no + o + 4 * k) = nn[k];
                if (do_max) *(float *)(xo + o + 4 * k) = xx[k];
            }
        }
    }
}

/* A class launch's view of one member: references into the parameter bank */
struct BlockClassDesc {
    const int &nx, &ny, &pitch, &bt, &bntx, &bnty, &bper;
    const unsigned &bmag;
    const int &nbuf, &cur0;
    const float *const &rows;
    float *const (&z)[3];
    float *const (&m)[3];
    float *const (&n)[3];
    float *const &zmax;
    int *const &arrival;
    const float *const &h;
    const int *const &gij;
    const float *const &gw;
    float *const &ts;
    const int &step0, &nsteps, &flags, &ng;
    const float &thr;
    __device__ __forceinline__ BlockClassDesc(const GcFusedGrid &p, const GcPairMember &q)
        : nx(p.nx), ny(p.ny), pitch(p.pitch), bt(p.bt), bntx(p.bntx), bnty(p.bnty), bper(p.bper), bmag(p.bmag),
          nbuf(p.nbuf), cur0(p.cur0), rows(p.rows), z(q.z), m(q.m), n(q.n), zmax(q.zmax), arrival(q.arrival), h(q.h),
          gij(q.gij), gw(q.gw), ts(q.ts), step0(q.step0), nsteps(q.nsteps), flags(q.flags), ng(q.ng), thr(q.thr) {}
};

/* one window per CTA: edge windows last longer, and the hardware hands the
 * next window to whichever CTA slot is free */
__device__ __forceinline__ void pdl_enter() {
    /* programmatic dependent launch: the previous kernel in the stream has
     * finished and its writes are visible past this point */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <int R, int NW>
__device__ __forceinline__ BlockSmem<R, NW> &block_smem() {
    extern __shared__ __align__(128) char smem[];
    return *reinterpret_cast<BlockSmem<R, NW> *>(smem);
}

/* one grid by value */
template <int R, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_block_one(const __grid_constant__ GcFusedGrid g,
                                                             const int *__restrict__ step_base, int step_off, int T) {
    pdl_enter();
    block_tile<R, NW>(g, blockIdx.x, step_off + (step_base ? *step_base : 0), T, block_smem<R, NW>());
}
/* a work list of {grid, window} over descriptors in memory */
template <int R, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_block_list(const GcFusedGrid *__restrict__ grids,
                                                              const int2 *__restrict__ tiles,
                                                              const int *__restrict__ step_base, int step_off, int T) {
    pdl_enter();
    const int2 t = tiles[blockIdx.x];
    block_tile<R, NW>(grids[t.x], t.y, step_off + (step_base ? *step_base : 0), T, block_smem<R, NW>());
}
/* the members of one class, their table in the parameter bank, windows
 * member-minor */
template <int R, int NW, int MINB>
__global__ void __launch_bounds__(32 * NW, MINB) k_block_class(const __grid_constant__ GcPairClass c,
                                                               const int *__restrict__ step_base, int step_off,
                                                               int T) {
    pdl_enter();
    const int lt = c.nm == 1 ? (int)blockIdx.x : (int)__umulhi(blockIdx.x, c.mag);
    const BlockClassDesc G(c.proto, c.m[blockIdx.x - lt * c.nm]);
    block_tile<R, NW>(G, lt, step_off + (step_base ? *step_base : 0), T, block_smem<R, NW>());
}

struct BlockVariant {
    int r, nw, smem;
    void (*one)(const GcFusedGrid, const int *, int, int);
    void (*list)(const GcFusedGrid *, const int2 *, const int *, int, int);
    void (*cls)(const GcPairClass, const int *, int, int);
};
#define GC_BVARIANT(R, NW, MINB)                                                                       \
    {R, NW, (int)sizeof(BlockSmem<R, NW>), k_block_one<R, NW, MINB>, k_block_list<R, NW, MINB>, k_block_class<R, NW, MINB>}
const BlockVariant kBlockVariants[] = {
    GC_BVARIANT(1, 16, 1), GC_BVARIANT(2, 8, 2), GC_BVARIANT(2, 12, 1), GC_BVARIANT(2, 16, 1),
    GC_BVARIANT(4, 8, 2), GC_BVARIANT(4, 12, 1), GC_BVARIANT(4, 16, 1),
};
#undef GC_BVARIANT
constexpr int kNumBlockVariants = sizeof(kBlockVariants) / sizeof(kBlockVariants[0]);

void prepare_block(const BlockVariant &v) {
    static bool done[64][kNumBlockVariants];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    const int idx = (int)(&v - kBlockVariants);
    if (done[dev][idx]) return;
    cudaFuncSetAttribute(v.one, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem);
    cudaFuncSetAttribute(v.list, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem);
    cudaFuncSetAttribute(v.cls, cudaFuncAttributeMaxDynamicSharedMemorySize, v.smem);
    done[dev][idx] = true;
}

template <typename... K, typename... A>
cudaError_t launch_block(void (*kern)(K...), const BlockVariant &v, int ctas, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)(32 * v.nw));
    cfg.dynamicSmemBytes = (size_t)v.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gc_pdl_on() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

} // namespace

static std::atomic<unsigned long long> g_field_limit{1ull << 32}; /* bytes of a field: its offsets have 32 bits */

void gc_block_set_field_limit(long long bytes) {
    g_field_limit = bytes > 0 ? std::min((unsigned long long)bytes, 1ull << 32) : 1ull << 32;
}

bool gc_block_fits(const GcFusedGrid &g, int members) {
    const unsigned long long lim = 1ull << 32, n = (unsigned long long)g.bntx * g.bnty;
    return 4ull * g.pitch * g.ny < g_field_limit && n * g.bntx < lim && n * members * members < lim;
}

/* ceil(2^32 / d): (k * that) >> 32 is k / d while k * d < 2^32 */
static unsigned block_magic(int d) { return d <= 1 ? 0u : (unsigned)(((1ull << 32) + (unsigned)d - 1) / (unsigned)d); }

int gc_block_plan(int variant, GcFusedGrid &g, int bt) {
    g.bt = bt;
    g.bntx = block_count(g.nx, BW, block_hc(bt));
    g.bnty = block_count(g.ny, kBlockVariants[variant].r * kBlockVariants[variant].nw, bt);
    const bool plain = g.bntx < 3 || g.bnty < 3;
    g.bper = plain ? g.bntx * g.bnty : 2 * g.bntx + 2 * (g.bnty - 2);
    g.bmag = block_magic(plain ? g.bntx : g.bntx - 2);
    return g.bntx * g.bnty;
}

/* The forms a launch can take, and a model of a launch's time in microseconds:
 * a + b * waves, a wave being the windows the device holds at once, and no less
 * than `lone`, what a launch of few windows takes (its corner window).  Fitted to
 * timed runs with waves everywhere on one grid of 361 x 301 to 2401 x 2001
 * cells and on 8 and 24 grids of 1201 x 1001 (within 15 % of most).  Small
 * grids want many small windows, large ones windows with little margin: per
 * step, 2.8 us (24 rows, 8 steps) against 5.2 us (64 rows) at 361 x 301, and
 * 46 us against 19.0 us at 2401 x 2001. */
struct BlockForm {
    int variant, steps, per_sm;
    float lone, a, b;
};
static const BlockForm kBlockForms[] = {
    {0, 4, 1, 10.2f, 4.0f, 6.1f},  {1, 4, 2, 14.0f, 4.5f, 7.1f},  {2, 8, 1, 20.0f, 9.0f, 10.2f},
    {3, 8, 1, 24.0f, 11.0f, 12.0f}, {5, 8, 1, 30.0f, 1.0f, 17.5f}, {5, 4, 1, 20.0f, 0.0f, 12.0f},
    {6, 8, 1, 36.0f, 1.0f, 23.4f},  {4, 4, 2, 22.0f, 0.0f, 14.0f},
};
constexpr int kNumBlockForms = sizeof(kBlockForms) / sizeof(kBlockForms[0]);

int gc_block_num_forms() { return kNumBlockForms; }
void gc_block_form(int form, int *variant, int *steps) {
    *variant = kBlockForms[form].variant;
    *steps = kBlockForms[form].steps;
}

int gc_block_pick_form(int ngrids, const int *nx, const int *ny) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int best = 0;
    float best_t = 0.0f;
    for (int f = 0; f < kNumBlockForms; f++) {
        const BlockForm &F = kBlockForms[f];
        const BlockVariant &v = kBlockVariants[F.variant];
        double windows = 0.0;
        for (int g = 0; g < ngrids; g++)
            windows += (double)block_count(nx[g], BW, block_hc(F.steps)) * block_count(ny[g], v.r * v.nw, F.steps);
        const double w = windows / (sms * F.per_sm), waves = w < 4.0 ? ceil(w) : w + 0.5;
        const float t = fmaxf(F.lone, F.a + F.b * (float)waves) / (float)F.steps;
        if (f == 0 || t < best_t) {
            best = f;
            best_t = t;
        }
    }
    return best;
}

cudaError_t gc_block_launch_one(int variant, const GcFusedGrid &g, int T, const int *d_step_base, int step_off,
                                cudaStream_t s) {
    const BlockVariant &v = kBlockVariants[variant];
    prepare_block(v);
    return launch_block(v.one, v, g.bntx * g.bnty, s, g, d_step_base, step_off, T);
}

cudaError_t gc_block_launch_list(int variant, const GcFusedGrid *d_grids, const int2 *d_tiles, int ntiles, int T,
                                 const int *d_step_base, int step_off, cudaStream_t s) {
    const BlockVariant &v = kBlockVariants[variant];
    if (ntiles <= 0) return cudaSuccess;
    prepare_block(v);
    return launch_block(v.list, v, ntiles, s, d_grids, d_tiles, d_step_base, step_off, T);
}

void gc_block_class_plan(GcPairClass &c) { c.mag = block_magic(c.nm); }

cudaError_t gc_block_launch_class(int variant, const GcPairClass &c, int T, const int *d_step_base, int step_off,
                                  cudaStream_t s) {
    const BlockVariant &v = kBlockVariants[variant];
    if (c.nm <= 0 || c.nm > GC_PAIR_CLASS_MAX) return cudaErrorInvalidValue;
    prepare_block(v);
    return launch_block(v.cls, v, c.nm * c.proto.bntx * c.proto.bnty, s, c, d_step_base, step_off, T);
}
