/*
 * One linear-spherical time step, a warp on its own, for sm_100a: MASS_S
 * (mass.f90:61-100), OPEN (boundaries.f90:22-202), MOMT_S (moment.f90:65-149)
 * and the maximum-amplitude and arrival records of one outer step, for the
 * callers that need every level: the reference ABI's per-step calls, the outer
 * grid of a nested member, the allocation-free step.
 *
 * A warp computes 128 columns x R rows (a lane four columns, as two packed
 * pairs), storing the inner 120: the flux of a cell reads the new surface one
 * row up and one column east, so the warp also computes the surface of the
 * row above its own from rows the next warp loads too (L1 or L2 serve the
 * second load).  Nothing crosses warps: no shared memory, no barrier, every
 * load of a warp in flight at once.
 *
 * Arithmetic order and results are those of kernels_fused.cu, bit for bit.
 *
 * Against the one-warp-per-tile march of kernels_fused.cu (warm, ncu): 361 x
 * 301 6.1 us against 20.3 (28 CTAs marching row by row), 481 x 401 6.7 against
 * 13.5, 1201 x 1001 11.9 against 17.2, six grids of 1201 x 1001 55.2 against
 * 69.3 (235 MB that the step cannot do without: 4.3 TB/s; with 20 resident
 * warps an SM the loads, not the pipes, are waited for).
 */
#include "fused.h"
#include "packed.cuh"

namespace {

using namespace gcpacked;

constexpr int SW = 128, SM = 4, SC = SW - 2 * SM; /* columns computed, margin, stored */
constexpr int SWARPS = 4;                         /* warps of a CTA, one above the other */

__device__ __forceinline__ float fkeep(float x, bool wet) { return (wet && !(fabsf(x) < CC_EPS)) ? x : 0.0f; }

struct Row {
    float r1, r11, r6, r3, r5, cx, cy;
};
__device__ __forceinline__ Row row_record(const float *rows, int j) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(rows + (size_t)j * GC_ROWW));
    const float4 b = __ldg(reinterpret_cast<const float4 *>(rows + (size_t)j * GC_ROWW + 4));
    return {a.x, a.y, a.z, a.w, b.x, b.y, b.z}; /* r1 r11 r6 r3 | r5 cx cy - */
}

/* warp `wt` of grid G at global step `step` */
template <int R>
__device__ __forceinline__ void step_rows(const GcFusedGrid &G, int tx, int jw, int step) {
    const int local = step - G.step0;
    if (local < 0 || local >= G.nsteps) return;
    const int nx = G.nx, ny = G.ny, lane = threadIdx.x & 31;
    if (jw >= ny) return;
    const size_t P = (size_t)G.pitch;
    int rd, wr;
    if (G.nbuf == 3) {
        rd = local % 3;
        wr = (local + 1) % 3;
    } else {
        rd = G.cur0 ^ (local & 1);
        wr = rd ^ 1;
    }
    const bool lone = nx <= SW;
    const int s = lone ? 0 : tx * SC;
    const int lo = tx == 0 ? 0 : s + SM, hi = (lone || s + SW >= nx) ? nx - 1 : s + SW - 1 - SM;
    const int ib = s + 4 * lane;
    const bool do_max = (G.flags & GC_F_MAXAMP) != 0;
    const float *zp = G.z[rd], *mp = G.m[rd], *np = G.n[rd], *hp = G.h, *xp = G.zmax;

    /* rows jw .. jw+R and N of the row below; past the grid, its last row and
     * the row's padding, which reach no cell of the grid */
    V4 z[R + 1], m[R + 1], n[R + 1], h[R + 1], x[R], ns;
    const size_t ic = (size_t)min(ib, G.pitch - 4);
    {
        auto ld = [&](const float *p, int j) {
            return v4(*reinterpret_cast<const float4 *>(p + (size_t)min(j, ny - 1) * P + ic));
        };
#pragma unroll
        for (int r = 0; r <= R; r++) {
            z[r] = ld(zp, jw + r);
            m[r] = ld(mp, jw + r);
            n[r] = ld(np, jw + r);
            h[r] = ld(hp, jw + r);
            if (do_max && r < R) x[r] = ld(xp, jw + r);
        }
        ns = ld(np, jw > 0 ? jw - 1 : 0); /* JM1 = max(J-1,1) */
    }
    Row rec[R + 1];
#pragma unroll
    for (int r = 0; r <= R; r++) rec[r] = row_record(G.rows, min(jw + r, ny - 1));
    const float r6m = jw > 0 ? row_record(G.rows, jw - 1).r6 : 0.0f;

    /* every cell wet and the perimeter out of reach */
    float hm = 3.0e38f;
#pragma unroll
    for (int r = 0; r <= R; r++) hm = min4nan(hm, h[r]);
    const bool inside = s >= 1 && s + SW - 1 <= nx - 2 && jw >= 1 && jw + R <= ny - 2;
    const bool fast = inside && __all_sync(FULL, hm > CC_GX);

    V4 zn[R + 1];
    float mw[R + 1];
    {
        float amin = 3.0e38f, cmin = 3.0e38f;
        V4 nrs = make_float2(r6m, r6m) * ns;
#pragma unroll
        for (int r = 0; r <= R; r++) {
            mw[r] = shw(m[r].b.y);
            const V4 nr = make_float2(rec[r].r6, rec[r].r6) * n[r];
            const V4 d = v4(m[r].a.x - mw[r], m[r].a.y - m[r].a.x, m[r].b.x - m[r].a.y, m[r].b.y - m[r].b.x);
            zn[r] = (z[r] - make_float2(rec[r].r1, rec[r].r1) * d) - make_float2(rec[r].r11, rec[r].r11) * (nr - nrs);
            nrs = nr;
            amin = minabs4(amin, zn[r]);
            cmin = min4(cmin, zn[r] + h[r]);
        }
        /* the flush and the clamp Z+H <= EPS, where some value calls for them */
        if (!fast || __any_sync(FULL, amin < CC_EPS || cmin <= CC_EPS)) {
#pragma unroll
            for (int r = 0; r <= R; r++) {
                zn[r] = clamp4(flush4(zn[r]), h[r]);
                zn[r] = v4(h[r].a.x > CC_GX ? zn[r].a.x : 0.0f, h[r].a.y > CC_GX ? zn[r].a.y : 0.0f,
                           h[r].b.x > CC_GX ? zn[r].b.x : 0.0f, h[r].b.y > CC_GX ? zn[r].b.y : 0.0f);
            }
        }
    }
    if (!inside) {
        /* OPEN on the perimeter: its rows (every lane its own four cells) and
         * its columns (the lane that holds them) */
        const int le = (nx - 1 - s) >> 2, qe = (nx - 1 - s) & 3;
        const bool west = s == 0 && lane == 0, east = s + SW - 1 >= nx - 1 && lane == le;
        float hb = west && jw > 0 ? hp[(size_t)(jw - 1) * P] : 0.0f; /* H below, read on the west column */
#pragma unroll
        for (int r = 0; r <= R; r++) {
            const int j = jw + r;
            if (j >= ny) break;
            const V4 nb = r == 0 ? ns : n[r > 0 ? r - 1 : 0];
            if (j == 0 || j == ny - 1) {
                const float hv[4] = {h[r].a.x, h[r].a.y, h[r].b.x, h[r].b.y};
                const float mv[5] = {mw[r], m[r].a.x, m[r].a.y, m[r].b.x, m[r].b.y};
                const V4 b = j == 0 ? n[r] : nb;
                const float bv[4] = {b.a.x, b.a.y, b.b.x, b.b.y};
                float o[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const bool wet = hv[q] > CC_GX;
                    o[q] = open_value(0.5f * (mv[q + 1] + mv[q]), bv[q], sqrtf(CC_GRAV * (wet ? hv[q] : 1.0f)),
                                      j == 0 ? bv[q] > 0.0f : bv[q] < 0.0f, wet);
                }
                zn[r] = v4(o[0], o[1], o[2], o[3]);
            }
            if (west) {
                zn[r].a.x = gcopen::open_cell(0, j, nx, ny, h[r].a.x, hb, m[r].a.x, m[r].a.x, n[r].a.x, nb.a.x);
                hb = h[r].a.x;
                mw[r] = m[r].a.x; /* IM1 = max(I-1,1) */
            }
            if (east) {
                const float o = gcopen::open_cell(nx - 1, j, nx, ny, comp(h[r], qe), 0.0f, comp(m[r], qe),
                                                  qe == 0 ? mw[r] : comp(m[r], qe - 1), comp(n[r], qe), comp(nb, qe));
                zn[r].a.x = qe == 0 ? o : zn[r].a.x;
                zn[r].a.y = qe == 1 ? o : zn[r].a.y;
                zn[r].b.x = qe == 2 ? o : zn[r].b.x;
                zn[r].b.y = qe == 3 ? o : zn[r].b.y;
            }
        }
        __syncwarp();
    }

    V4 mn[R], nn[R];
    {
        float amin = 3.0e38f;
        V4 nsr = ns;
        float nse = she(ns.a.x);
        const float2 half = make_float2(0.5f, 0.5f);
#pragma unroll
        for (int r = 0; r < R; r++) {
            const V4 hc = h[r], zc = zn[r], nc = n[r], mc = m[r], ma = m[r + 1];
            const float he = she(hc.a.x), ze = she(zc.a.x), ne = she(nc.a.x);
            V4 tot = v4(nc.a.x + nc.a.y, nc.a.y + nc.b.x, nc.b.x + nc.b.y, nc.b.y + ne) + nsr;
            tot = v4(tot.a.x + nsr.a.y, tot.a.y + nsr.b.x, tot.b.x + nsr.b.y, tot.b.y + nse);
            const V4 dz = v4(zc.a.y - zc.a.x, zc.b.x - zc.a.y, zc.b.y - zc.b.x, ze - zc.b.y);
            const V4 r2 = make_float2(rec[r].cx, rec[r].cx) *
                          (half * v4(hc.a.x + hc.a.y, hc.a.y + hc.b.x, hc.b.x + hc.b.y, hc.b.y + he));
            mn[r] = (mc - r2 * dz) + make_float2(rec[r].r3, rec[r].r3) * tot;
            V4 tm = v4(mw[r] + mw[r + 1], mc.a.x + ma.a.x, mc.a.y + ma.a.y, mc.b.x + ma.b.x);
            tm = (tm + mc) + ma;
            const V4 r4 = make_float2(rec[r].cy, rec[r].cy) * (half * (hc + h[r + 1]));
            nn[r] = (nc - r4 * (zn[r + 1] - zc)) - make_float2(rec[r].r5, rec[r].r5) * tm;
            nsr = nc;
            nse = ne;
            if (fast) {
                amin = minabs4(minabs4(amin, mn[r]), nn[r]);
            } else {
                const bool w0 = hc.a.x > CC_GX, w1 = hc.a.y > CC_GX, w2 = hc.b.x > CC_GX, w3 = hc.b.y > CC_GX;
                mn[r] = v4(fkeep(mn[r].a.x, w0 && w1 && ib < nx - 1), fkeep(mn[r].a.y, w1 && w2 && ib + 1 < nx - 1),
                           fkeep(mn[r].b.x, w2 && w3 && ib + 2 < nx - 1),
                           fkeep(mn[r].b.y, w3 && he > CC_GX && ib + 3 < nx - 1));
                const V4 ha = h[r + 1];
                const bool in = jw + r < ny - 1;
                nn[r] = v4(fkeep(nn[r].a.x, in && w0 && ha.a.x > CC_GX), fkeep(nn[r].a.y, in && w1 && ha.a.y > CC_GX),
                           fkeep(nn[r].b.x, in && w2 && ha.b.x > CC_GX), fkeep(nn[r].b.y, in && w3 && ha.b.y > CC_GX));
            }
        }
        if (fast && __any_sync(FULL, amin < CC_EPS)) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                mn[r] = flush4(mn[r]);
                nn[r] = flush4(nn[r]);
            }
        }
    }

    /* stores: whole lanes where the margin and the grid allow; max-eta and
     * arrival are left to a child's feedback inside its window */
    const bool whole = ib >= lo && ib + 3 <= hi, any = ib + 3 >= lo && ib <= hi;
    const bool inwin = G.has_win && s <= G.wi1 && s + SW > G.wi0 && jw <= G.wj1 && jw + R > G.wj0;
    const float thr = G.thr;
    const bool arr = (G.flags & GC_F_ARRIVAL) != 0;
    if (!any) return;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int j = jw + r;
        if (j >= ny) break;
        const size_t o = (size_t)j * P + ib;
        if (whole) {
            *reinterpret_cast<float4 *>(G.z[wr] + o) = f4(zn[r]);
            *reinterpret_cast<float4 *>(G.m[wr] + o) = f4(mn[r]);
            *reinterpret_cast<float4 *>(G.n[wr] + o) = f4(nn[r]);
        }
        const float zv[4] = {zn[r].a.x, zn[r].a.y, zn[r].b.x, zn[r].b.y};
        const float xv[4] = {x[r].a.x, x[r].a.y, x[r].b.x, x[r].b.y};
        if (whole && do_max && !inwin) {
            float4 xn;
            xn.x = xv[0] >= zv[0] ? xv[0] : zv[0];
            xn.y = xv[1] >= zv[1] ? xv[1] : zv[1];
            xn.z = xv[2] >= zv[2] ? xv[2] : zv[2];
            xn.w = xv[3] >= zv[3] ? xv[3] : zv[3];
            *reinterpret_cast<float4 *>(G.zmax + o) = xn;
        }
        const bool reach = arr && fmaxf(fmaxf(zv[0], zv[1]), fmaxf(zv[2], zv[3])) > thr;
        if (!whole || (do_max && inwin) || reach) {
            const float mv[4] = {mn[r].a.x, mn[r].a.y, mn[r].b.x, mn[r].b.y};
            const float nv[4] = {nn[r].a.x, nn[r].a.y, nn[r].b.x, nn[r].b.y};
            const float hv[4] = {h[r].a.x, h[r].a.y, h[r].b.x, h[r].b.y};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int i = ib + q;
                if (i < lo || i > hi) continue;
                if (!whole) {
                    G.z[wr][o + q] = zv[q];
                    G.m[wr][o + q] = mv[q];
                    G.n[wr][o + q] = nv[q];
                }
                if (G.has_win && i >= G.wi0 && i <= G.wi1 && j >= G.wj0 && j <= G.wj1) continue;
                if (do_max && (!whole || inwin)) G.zmax[o + q] = xv[q] >= zv[q] ? xv[q] : zv[q];
                /* a wet cell above the threshold whose maximum before was not */
                if (arr && zv[q] > thr && hv[q] > CC_GX && xv[q] <= thr) G.arrival[o + q] = local + 1;
            }
        }
    }
}

__host__ __device__ __forceinline__ int step_tx(int nx) { return nx <= SW ? 1 : 1 + (nx - SW + SC - 1) / SC; }

__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <int R>
__global__ void __launch_bounds__(32 * SWARPS) k_step_one(const __grid_constant__ GcFusedGrid g,
                                                          const int *__restrict__ step_base, int step_off, int ntx) {
    pdl_enter();
    const int ty = blockIdx.x / ntx;
    step_rows<R>(g, blockIdx.x - ty * ntx, (ty * SWARPS + (int)(threadIdx.x >> 5)) * R,
                 step_off + (step_base ? *step_base : 0));
}

/* a list of grids by value: grid g's CTAs are start[g] .. start[g + 1] - 1 */
template <int N>
struct StepGrids {
    int n, start[N + 1], tx[N];
    /* on a 16-byte boundary: at 8 bytes past one, one call on a 361 x 301 grid
     * took 15.8 us instead of 15.0 */
    alignas(16) GcFusedGrid g[N];
};
static_assert(sizeof(StepGrids<64>) <= 32000, "kernel parameters may take up to 32764 bytes");
template <int R, int N>
__global__ void __launch_bounds__(32 * SWARPS) k_step_grids(const __grid_constant__ StepGrids<N> p, int step) {
    pdl_enter();
    int lo = 0, hi = p.n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.start[mid] <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const int b = blockIdx.x - p.start[lo], ty = b / p.tx[lo];
    step_rows<R>(p.g[lo], b - ty * p.tx[lo], (ty * SWARPS + (int)(threadIdx.x >> 5)) * R, step);
}

template <typename... K, typename... A>
cudaError_t launch_step(void (*kern)(K...), long long ctas, cudaStream_t s, const A &...args) {
    cudaLaunchConfig_t cfg = {};
    if (ctas > 0x7fffffffll) return cudaErrorInvalidValue;
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(32 * SWARPS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = gc_pdl_on() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

/* One row a warp while that leaves the device idle warps to fill (361 x 301:
 * 6.1 us against 6.9 with two rows; 1201 x 1001: 11.9 against 12.5), two rows,
 * with less of the surface computed twice, beyond (six grids of 1201 x 1001:
 * 55.2 us against 56.1). */
int step_rows_for(long long cells) { return cells < 2000000 ? 1 : 2; }

template <int N>
cudaError_t launch_grids(int n, const GcFusedGrid *g, int step, cudaStream_t s) {
    StepGrids<N> p; /* on this thread's stack: the launch copies it */
    long long cells = 0;
    for (int k = 0; k < n; k++) cells += (long long)g[k].nx * g[k].ny;
    const int R = step_rows_for(cells);
    p.n = n;
    long long t = 0;
    for (int k = 0; k < n; k++) {
        p.g[k] = g[k];
        p.start[k] = (int)t;
        p.tx[k] = step_tx(g[k].nx);
        t += (long long)p.tx[k] * ((g[k].ny + R * SWARPS - 1) / (R * SWARPS));
        if (t > 0x7fffffffll) return cudaErrorInvalidValue; /* start[] holds it */
    }
    p.start[n] = (int)t;
    return R == 1 ? launch_step(k_step_grids<1, N>, t, s, p, step) : launch_step(k_step_grids<2, N>, t, s, p, step);
}

} // namespace

cudaError_t gc_step_launch_one(const GcFusedGrid &g, const int *d_step_base, int step_off, cudaStream_t s) {
    const int R = step_rows_for((long long)g.nx * g.ny);
    const int ntx = step_tx(g.nx);
    const long long ctas = (long long)ntx * ((g.ny + R * SWARPS - 1) / (R * SWARPS));
    return R == 1 ? launch_step(k_step_one<1>, ctas, s, g, d_step_base, step_off, ntx)
                  : launch_step(k_step_one<2>, ctas, s, g, d_step_base, step_off, ntx);
}

cudaError_t gc_step_launch_grids(int n, const GcFusedGrid *g, int step, cudaStream_t s) {
    if (n < 1 || n > 64) return cudaErrorInvalidValue;
    return n <= 4 ? launch_grids<4>(n, g, step, s) : launch_grids<64>(n, g, step, s);
}
