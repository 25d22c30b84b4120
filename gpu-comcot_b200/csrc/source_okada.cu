/*
 * On-device source generation: seafloor deformation of rectangular faults
 * (Okada 1985) applied to a layer, so a forecast request goes from fault
 * parameters to its initial state without a host upload of the surface.
 *
 * Follows the reference's GET_FLOOR_DEFORM / DEFORM_OKADA / STRIKE_SLIP /
 * DIP_SLIP / STEREO_PROJECTION (deform.f90:2-240, 494-586): per fault, the
 * vertical displacement US + UD of the free surface above a buried
 * dislocation (strike-slip and dip-slip parts, each a four-corner
 * combination F1 - F2 - F3 + F4), with cell positions mapped onto the fault
 * plane by an oblique stereographic projection on the WGS84 ellipsoid
 * (spherical layers) or from the layer origin and spacing (Cartesian
 * layers); non-finite values and |value| <= GX give 0; then Z += DEFORM and
 * H -= DEFORM in fault order.  The reference evaluates in single precision;
 * here every cell is evaluated in double (its float rounding jumps between
 * atan branches on the lines where a fault end is level with the cell) and
 * the per-fault result is rounded to float before it is applied, as the
 * reference's REAL DEFORM array is.
 *
 * The FP64 pipe bounds it: 961 x 801 cells and 24 faults take 0.97 ms against
 * 4.0 ms when every cell evaluated the
 * projection's sines and powers and each of the eight corner terms its own
 * divisions, logarithms and arc tangents.  The largest error against a 64-bit
 * evaluation is the same 1.6e-7 of the field's maximum, the float rounding of
 * 24 sums.
 */
#include <math.h>
#include <string.h>

#include "gc_internal.h"
#include "gcomcot.h"

namespace {

constexpr int MAX_FAULTS_PER_LAUNCH = 12;

/* per-fault constants, evaluated once on the host in double */
struct FaultDev {
    double hh, halfl, w, sn, cs, st, ct, ds, dd, del_x, del_y, xl, yl;
    /* projection (spherical layers): 2 rho k0, exponent, scale, origin */
    double big, n, c, sx0, cx0, ln0;
};
struct FaultPack {
    int n;
    FaultDev f[MAX_FAULTS_PER_LAUNCH];
};

constexpr double kE = 0.08181919092891, kF2 = 0.00669438000426;

__host__ __device__ double clip_lat(double lat) {
    const double pole = CC_PI / 2.0 - (double)CC_EPS;
    return lat > pole ? pole : (lat < -pole ? -pole : lat);
}

/* sine of the conformal latitude of the projection for a latitude (radians) */
__host__ __device__ double conformal(double lat, double n, double c) {
    const double sn = sin(lat);
    const double w = c * pow((1.0 + sn) / (1.0 - sn) * pow((1.0 - kE * sn) / (1.0 + kE * sn), kE), n);
    return (w - 1.0) / (w + 1.0);
}

/* the projection's constants for an origin (STEREO_PROJECTION, deform.f90) */
void stereo_origin(double lon0, double lat0, FaultDev &f) {
    const double lt0 = clip_lat(lat0 * CC_RAD_DEG), cs0 = cos(lt0), sn0 = sin(lt0);
    const double a = 6378137.0, k0 = 0.9996;
    const double tmp0 = sqrt(1.0 - kF2 * (sn0 * sn0));
    const double rho0 = a * (1.0 - kF2) / (tmp0 * tmp0 * tmp0);
    /* the reference's NU0 is an INTEGER by implicit typing: truncated */
    const double nu0 = (double)(int)(a / tmp0);
    f.big = 2.0 * sqrt(rho0 * nu0) * k0;
    f.n = sqrt(1.0 + kF2 * ((cs0 * cs0) * (cs0 * cs0)) / (1.0 - kF2));
    const double sx = conformal(lt0, f.n, 1.0);
    f.c = (f.n + sn0) * (1.0 - sx) / (f.n - sn0) / (1.0 + sx);
    f.sx0 = conformal(lt0, f.n, f.c);
    f.cx0 = sqrt((1.0 - f.sx0) * (1.0 + f.sx0));
    f.ln0 = lon0 * CC_RAD_DEG;
}

/* projected position from the sine and cosine of the conformal latitude and
 * of the longitude difference */
__host__ __device__ __forceinline__ void stereo_point(const FaultDev &f, double sx, double cx, double sl, double cl,
                                                      double &xo, double &yo) {
    const double g = f.big / (1.0 + sx * f.sx0 + cx * f.cx0 * cl);
    yo = g * (sx * f.cx0 - cx * f.sx0 * cl);
    xo = g * cx * sl;
}

/* multiplies the running unit of an angle sum, (pr, pi) with `wraps` turns, by
 * the complex number whose argument is s * atan(num / den): s = +-1, the
 * argument in [-pi/2, pi/2], so a change of sign of the imaginary part on the
 * far side is a turn past +-pi */
__device__ __forceinline__ void add_angle(double &pr, double &pi, int &wraps, double num, double den, double s) {
    const double ur = fabs(den), ui = s * copysign(1.0, den) * num;
    const double qr = pr * ur - pi * ui, qi = pr * ui + pi * ur + 0.0; /* + 0.0: never -0 */
    if (pi >= 0.0 && ui > 0.0 && qi < 0.0) wraps++;
    if (pi < 0.0 && ui < 0.0 && qi >= 0.0) wraps--;
    pr = qr;
    pi = qi;
}

/* US + UD of one fault at a cell of plane coordinates x1 (along strike), x2
 * (across), the four-corner combination F1 - F2 - F3 + F4 of STRIKE_SLIP and
 * DIP_SLIP (deform.f90) over (x1 +- L/2, p or p - W).  The corners are summed
 * before the costly operations: one division over a common denominator for
 * the algebraic terms of each, the logarithms as two logarithms of ratios,
 * and the eight arc tangents as one angle of a product of complex numbers. */
__device__ __forceinline__ float okada(const FaultDev &f, double x1, double x2) {
    const double sn = f.sn, cs = f.cs;
    const double q = x2 * sn - f.hh * cs, p = x2 * cs + f.hh * sn;
    double un = 0.0, ud = 1.0; /* sum of q (d + r sn) / (r (r + y2)), as a fraction */
    double dn = 0.0, dd = 1.0; /* sum of d q / (r (r + y1)) */
    double t1n = 1.0, t1d = 1.0, t2n = 1.0, t2d = 1.0;
    double pr = 1.0, pi = 0.0;
    int wraps = 0;
#pragma unroll
    for (int a = 0; a < 2; a++) {
        const double y1 = a == 0 ? x1 + f.halfl : x1 - f.halfl;
        const double xq = y1 * y1 + q * q, xx = sqrt(xq);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const double s = a == b ? 1.0 : -1.0;
            const double y2 = b == 0 ? p : p - f.w;
            const double d = y2 * sn - q * cs, r = sqrt(xq + y2 * y2), ry1 = r + y1, ry2 = r + y2;
            const double den = r * ry2, dem = r * ry1;
            un = un * den + s * (q * (d + r * sn)) * ud;
            ud = ud * den;
            dn = dn * dem + s * (d * q) * dd;
            dd = dd * dem;
            double t1 = r + d, t2 = ry2;
            if (t1 <= 1.0e-10) t1 = 1.0e-10;
            if (t2 <= 1.0e-10) t2 = 1.0e-10;
            if (a == b) { t1n *= t1; t2n *= t2; }
            else { t1d *= t1; t2d *= t2; }
            add_angle(pr, pi, wraps, y1 * y2, q * r, s);
            add_angle(pr, pi, wraps, y2 * (xx + q * cs) + xx * (r + xx) * sn, y1 * (r + xx) * cs, -s);
        }
        /* magnitudes up to 1e13 a factor: bring the product back to 1 */
        const double m = fabs(pr) > fabs(pi) ? fabs(pr) : fabs(pi), im = 1.0 / m;
        pr = pr * im;
        pi = pi * im;
    }
    const double k = 1.0 / 2.0 / 3.14159;
    double us = -(un / ud + 0.5 / cs * (log(t1n / t1d) - sn * log(t2n / t2d)) * sn) * k * f.ds;
    double dp = -(dn / dd + sn * (atan2(pi, pr) + 2.0 * CC_PI * (double)wraps)) * k * f.dd;
    if (!isfinite(us)) us = 0.0;
    if (!isfinite(dp)) dp = 0.0;
    if (fabs(us) <= (double)CC_GX) us = 0.0;
    if (fabs(dp) <= (double)CC_GX) dp = 0.0;
    return (float)(us + dp);
}

constexpr int OK_COLS = 128, OK_ROWS = 8; /* cells of a block: a column a thread, eight rows each */

/* The projection separates: its transcendental functions depend on the row
 * (sin, two powers) or on the column (sin and cos of the longitude difference)
 * alone, so a block evaluates them once per row and column of its cells and
 * fault, into shared memory. */
__global__ void __launch_bounds__(OK_COLS) k_okada(const __grid_constant__ FaultPack pk, int laycord, int nx, int ny,
                                                   int pitch, const float *x, const float *y, float dx, float dy,
                                                   float *z, float *h) {
    __shared__ double rowt[MAX_FAULTS_PER_LAUNCH][OK_ROWS][2];
    const int i = blockIdx.x * OK_COLS + threadIdx.x, j0 = blockIdx.y * OK_ROWS;
    if (laycord == 0) {
        static_assert(MAX_FAULTS_PER_LAUNCH * OK_ROWS <= OK_COLS, "one row entry a thread");
        const int t = threadIdx.x, k = t / OK_ROWS, r = t - k * OK_ROWS;
        if (k < pk.n && j0 + r < ny) {
            const double sx = conformal(clip_lat((double)y[j0 + r] * CC_RAD_DEG), pk.f[k].n, pk.f[k].c);
            rowt[k][r][0] = sx;
            rowt[k][r][1] = sqrt((1.0 - sx) * (1.0 + sx));
        }
        __syncthreads();
    }
    if (i >= nx) return;
    const int nr = min(OK_ROWS, ny - j0);
    float zc[OK_ROWS], hc[OK_ROWS];
#pragma unroll
    for (int r = 0; r < OK_ROWS; r++) {
        const size_t c = (size_t)(j0 + r) * pitch + i;
        zc[r] = z && r < nr ? z[c] : 0.0f;
        hc[r] = h && r < nr ? h[c] : 0.0f;
    }
    const double lon = laycord == 0 ? (double)x[i] * CC_RAD_DEG : 0.0;
#pragma unroll 1
    for (int k = 0; k < pk.n; k++) {
        const FaultDev &f = pk.f[k];
        double sl = 0.0, cl = 0.0;
        if (laycord == 0) sincos(f.n * (lon - f.ln0), &sl, &cl);
#pragma unroll 1
        for (int r = 0; r < OK_ROWS; r++) {
            float d = 0.0f;
            if (r < nr) {
                double xs, ys;
                if (laycord == 0) {
                    stereo_point(f, rowt[k][r][0], rowt[k][r][1], sl, cl, xs, ys);
                    xs = xs - f.del_x;
                    ys = ys + f.del_y;
                } else {
                    xs = (double)dx * (double)i - f.xl - f.del_x;
                    ys = (double)dy * (double)(j0 + r) - f.yl + f.del_y;
                }
                d = okada(f, xs * f.st + ys * f.ct, -(xs * f.ct - ys * f.st));
            }
#pragma unroll
            for (int u = 0; u < OK_ROWS; u++) {
                zc[u] = u == r ? zc[u] + d : zc[u];
                hc[u] = u == r ? hc[u] - d : hc[u];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < OK_ROWS; r++) {
        const size_t c = (size_t)(j0 + r) * pitch + i;
        if (z && r < nr) z[c] = zc[r];
        if (h && r < nr) h[c] = hc[r];
    }
}

FaultDev prepare_fault(const gc_fault &in, int laycord) {
    FaultDev f;
    const double rad = CC_RAD_DEG;
    const double ang_l = rad * in.dl, ang_r = rad * in.rd, ang_t = rad * in.th;
    f.halfl = 0.5 * in.l;
    f.w = in.w;
    if (in.sw == 9) {
        f.hh = in.hh + in.w * sin(ang_l);
        f.del_x = in.w * cos(ang_l) * cos(ang_t);
        f.del_y = in.w * cos(ang_l) * sin(ang_t);
    } else {
        f.hh = in.hh + 0.5 * in.w * sin(ang_l);
        f.del_x = 0.5 * in.w * cos(ang_l) * cos(ang_t);
        f.del_y = 0.5 * in.w * cos(ang_l) * sin(ang_t);
    }
    f.ds = in.d * cos(ang_r);
    f.dd = in.d * sin(ang_r);
    f.sn = sin(ang_l);
    f.cs = cos(ang_l);
    f.st = sin(ang_t);
    f.ct = cos(ang_t);
    f.xl = f.yl = 0.0;
    stereo_origin(in.x0, in.y0, f);
    if (laycord != 0) {
        const double sx = conformal(clip_lat(in.yo * rad), f.n, f.c), cx = sqrt((1.0 - sx) * (1.0 + sx));
        const double dl = f.n * (in.xo * rad - f.ln0);
        stereo_point(f, sx, cx, sin(dl), cos(dl), f.xl, f.yl);
    }
    return f;
}

} // namespace

extern "C" {

int gc_okada_apply(const gc_fault *faults, int nf, int laycord, int nx, int ny, int pitch, const float *d_x,
                   const float *d_y, float dx, float dy, float *d_z, float *d_h, void *stream) {
    if (!faults || nf < 0 || nx < 1 || ny < 1 || pitch < nx || (laycord != 0 && laycord != 1)) return GC_EINVAL;
    if (laycord == 0 && (!d_x || !d_y)) return GC_EINVAL;
    for (int k = 0; k < nf; k++)
        if (faults[k].sw != 0 && faults[k].sw != 9) return GC_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    for (int k0 = 0; k0 < nf; k0 += MAX_FAULTS_PER_LAUNCH) {
        FaultPack pk;
        memset(&pk, 0, sizeof pk);
        pk.n = nf - k0 < MAX_FAULTS_PER_LAUNCH ? nf - k0 : MAX_FAULTS_PER_LAUNCH;
        for (int k = 0; k < pk.n; k++) pk.f[k] = prepare_fault(faults[k0 + k], laycord);
        dim3 grid((unsigned)((nx + OK_COLS - 1) / OK_COLS), (unsigned)((ny + OK_ROWS - 1) / OK_ROWS), 1);
        k_okada<<<grid, OK_COLS, 0, s>>>(pk, laycord, nx, ny, pitch, d_x, d_y, dx, dy, d_z, d_h);
        GC_CUDA_OR_RET(cudaGetLastError());
    }
    return GC_OK;
}

} /* extern "C" */
