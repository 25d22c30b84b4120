/*
 * gcomcot_fused_step_noalloc: one linear-spherical time step over a
 * caller-supplied list of grids, for callers that cannot allocate device
 * memory.
 *
 * Who needs it: codes that own every byte of device memory themselves and
 * forbid library allocations (a Fortran model that sizes its arrays once at
 * start-up, an operational warning pipeline that reserves a fixed memory budget
 * before the first alert arrives), and time-critical loops in which an
 * allocation is not acceptable because it may synchronise the device or fail
 * under memory pressure.
 *
 * The grid descriptors travel to the GPU in the launch parameters of the step
 * kernel itself (kernels_step.cu: up to 64 descriptors in the parameter bank,
 * a short form for up to four), so a call is one launch, copies nothing from
 * host memory, holds no device memory of its own and returns as soon as the
 * kernel is queued; calls on different streams do not meet.  Before, a fill
 * kernel wrote the descriptors and a tile list into a device array for the
 * one-warp-per-tile step: three launches a call, and a 361 x 301 grid's 87
 * tiles kept 29 CTAs of 148 SMs busy for 20 us.
 *
 * The kernel has no waits, so it neither raises nor clears the flag that
 * gcomcot_sync() reports, and no call sets anything up: the first one may be
 * made inside a stream capture.
 */
#include <string.h>

#include "fused.h"
#include "gcomcot.h"

#define GC_NOALLOC_MAX_GRIDS 64
#define GC_NOALLOC_MAX_TILES 24576

namespace {

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

} // namespace

extern "C" int gcomcot_fused_step_noalloc(int ngrids, const gc_grid_step_io *grids, void *stream) {
    if (ngrids < 1 || !grids) {
        fprintf(stderr, "gcomcot_fused_step_noalloc: need at least one grid\n");
        return GC_EINVAL;
    }
    if (ngrids > GC_NOALLOC_MAX_GRIDS) {
        fprintf(stderr, "gcomcot_fused_step_noalloc: %d grids exceed the maximum of %d\n", ngrids,
                GC_NOALLOC_MAX_GRIDS);
        return GC_EINVAL;
    }
    for (int g = 0; g < ngrids; g++) {
        const gc_grid_step_io &q = grids[g];
        if (q.nx < 3 || q.ny < 3 || q.pitch < q.nx || (q.pitch % 32) != 0 || !q.z1 || !q.m1 || !q.n1 || !q.z2
            || !q.m2 || !q.n2 || !q.h || !q.rows) {
            fprintf(stderr, "gcomcot_fused_step_noalloc: grid %d: bad sizes or missing arrays "
                            "(nx,ny >= 3, pitch >= nx and a multiple of 32)\n", g);
            return GC_EINVAL;
        }
        if (!aligned16(q.z1) || !aligned16(q.m1) || !aligned16(q.n1) || !aligned16(q.z2) || !aligned16(q.m2)
            || !aligned16(q.n2) || !aligned16(q.h) || !aligned16(q.rows) || (q.zmax && !aligned16(q.zmax))) {
            fprintf(stderr, "gcomcot_fused_step_noalloc: grid %d: arrays must start on 16-byte boundaries\n", g);
            return GC_EINVAL;
        }
    }
    /* the documented limit: GC_NOALLOC_MAX_TILES tiles of 128 columns by at
     * most 4096 rows */
    long long least = 0;
    for (int g = 0; g < ngrids; g++) least += gc_fused_tiles(grids[g].nx, grids[g].ny, 4096, nullptr);
    if (least > GC_NOALLOC_MAX_TILES) {
        fprintf(stderr, "gcomcot_fused_step_noalloc: %lld tiles exceed the maximum of %d\n", least,
                GC_NOALLOC_MAX_TILES);
        return GC_EINVAL;
    }
    GcFusedGrid desc[GC_NOALLOC_MAX_GRIDS];
    for (int g = 0; g < ngrids; g++) {
        const gc_grid_step_io &q = grids[g];
        GcFusedGrid &d = desc[g];
        memset(&d, 0, sizeof d);
        d.nx = q.nx; d.ny = q.ny; d.pitch = q.pitch; d.root = 1;
        /* step 1 of a one-step window: buffers [0] are read, [1] written */
        d.step0 = 1; d.nsteps = 1;
        d.flags = q.zmax ? GC_F_MAXAMP : 0;
        d.z[0] = const_cast<float *>(q.z1); d.z[1] = q.z2;
        d.m[0] = const_cast<float *>(q.m1); d.m[1] = q.m2;
        d.n[0] = const_cast<float *>(q.n1); d.n[1] = q.n2;
        d.h = q.h; d.rows = q.rows; d.zmax = q.zmax;
    }
    GC_CUDA_OR_RET(gc_step_launch_grids(ngrids, desc, 1, (cudaStream_t)stream));
    return GC_OK;
}
