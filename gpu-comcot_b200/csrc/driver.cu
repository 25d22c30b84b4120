/*
 * The reference driver's per-step call sequence as a library entry point
 * (gauge stencils gathered on the device, read back once per chunk of
 * steps), the gauge snapshot that serves gcomcot_get_z_ after the first step
 * with one device round trip per step, and the DEBUG_CORE comparators.
 */
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "fused.h"
#include "gcomcot.h"
#include "runtime.h"

/* ------------------------------------------------------------------ */
/* gauge snapshot                                                      */
/* ------------------------------------------------------------------ */
struct GaugeReg {
    int lid, i, j;
};
static std::vector<GaugeReg> g_reg;
static bool g_snap_valid = false;
static bool g_ij_stale = true;    /* the device copy of the stencil indices needs an upload */
static int *g_d_ij = nullptr;     /* [2*cap] */
static float *g_h_out = nullptr;  /* mapped pinned [4*cap] */
static float *g_d_out = nullptr;  /* device alias of g_h_out */
static int g_cap = 0;

void gc_gauge_invalidate() { g_snap_valid = false; }

static int ensure_cap(int n) {
    if (n <= g_cap) return GC_OK;
    int cap = n < 64 ? 64 : 2 * n;
    if (g_d_ij) cudaFree(g_d_ij);
    if (g_h_out) cudaFreeHost(g_h_out);
    g_ij_stale = true;
    GC_CUDA_OR_RET(cudaMalloc(&g_d_ij, (size_t)2 * cap * sizeof(int)));
    GC_CUDA_OR_RET(cudaHostAlloc((void **)&g_h_out, (size_t)4 * cap * sizeof(float), cudaHostAllocMapped));
    GC_CUDA_OR_RET(cudaHostGetDevicePointer((void **)&g_d_out, g_h_out, 0));
    g_cap = cap;
    return GC_OK;
}

/* samples every registered gauge stencil of the current state, one launch
 * per layer that has gauges, then waits */
static int snapshot() {
    GcRuntime &rt = gc_rt();
    GcPdlScope pdl(true); /* the gauge kernel waits for the step on the device */
    int n = (int)g_reg.size();
    if (ensure_cap(n) != GC_OK) return GC_ECUDA;
    if (g_ij_stale) {
        /* only when the set of gauges changed: a copy from pageable memory
         * waits for the stream, which would cost a second round trip a step */
        std::vector<int> ij((size_t)2 * n);
        for (int g = 0; g < n; g++) { ij[2 * g] = g_reg[g].i; ij[2 * g + 1] = g_reg[g].j; }
        GC_CUDA_OR_RET(cudaMemcpy(g_d_ij, ij.data(), ij.size() * sizeof(int), cudaMemcpyHostToDevice));
        g_ij_stale = false;
    }
    /* gauges are registered grouped by first use; launch per run of equal lid */
    int g0 = 0;
    while (g0 < n) {
        int lid = g_reg[g0].lid, g1 = g0;
        while (g1 < n && g_reg[g1].lid == lid) g1++;
        GcLayer *L = gc_layer(lid);
        GcLayerDev d = L->view();
        if (!L->z2_valid) d.z2 = L->z[L->cur];
        gc_launch_gauges(d, g1 - g0, g_d_ij + 2 * g0, g_d_out + 4 * g0, rt.stream);
        rt.launches++;
        g0 = g1;
    }
    GC_CUDA_OR_RET(cudaStreamSynchronize(rt.stream));
    g_snap_valid = true;
    return GC_OK;
}

static int g_last = -1; /* registry slot of the previous lookup */

/* serves gcomcot_get_z_; returns false when the caller must fall back */
bool gc_gauge_lookup(int lid, int i, int j, float *out4) {
    int n = (int)g_reg.size();
    int found = -1;
    /* a driver asks for its gauges in the same order every step: try the
     * slot after the previous one first */
    const int guess = (g_last + 1 < n) ? g_last + 1 : 0;
    if (guess < n && g_reg[guess].lid == lid && g_reg[guess].i == i && g_reg[guess].j == j) found = guess;
    for (int g = 0; found < 0 && g < n; g++)
        if (g_reg[g].lid == lid && g_reg[g].i == i && g_reg[g].j == j) found = g;
    if (found < 0) {
        /* keep same-layer gauges contiguous */
        size_t pos = g_reg.size();
        for (size_t k = g_reg.size(); k > 0; k--)
            if (g_reg[k - 1].lid == lid) { pos = k; break; }
        g_reg.insert(g_reg.begin() + pos, GaugeReg{lid, i, j});
        found = (int)pos;
        g_snap_valid = false;
        g_ij_stale = true;
    }
    if (!g_snap_valid) {
        gc_flush();
        if (snapshot() != GC_OK) return false;
    }
    memcpy(out4, g_h_out + 4 * found, 4 * sizeof(float));
    g_last = found;
    return true;
}

void gc_gauge_release() {
    if (g_d_ij) cudaFree(g_d_ij);
    if (g_h_out) cudaFreeHost(g_h_out);
    g_d_ij = nullptr; g_h_out = nullptr; g_d_out = nullptr; g_cap = 0;
    g_reg.clear();
    g_last = -1;
    g_snap_valid = false;
    g_ij_stale = true;
}

extern "C" {

/* several outer steps per launch inside gcomcot_drive (kernels_block.cu): a lone
 * linear spherical outer layer with factored R2/R4, the fused path on,
 * max-eta recorded, no arrival tracking and every gauge on that layer (at
 * most 64).  GCOMCOT_DRIVE_PAIRS=0 keeps one step per launch. */
static bool drive_block_ok(const GcLayer &L, int maxamp, int ngauges, const int *g_layer) {
    const GcRuntime &rt = gc_rt();
    static const bool off = [] {
        const char *v = getenv("GCOMCOT_DRIVE_PAIRS");
        return v && v[0] == '0';
    }();
    if (off || !rt.fuse_enabled || !maxamp || gc_arrival_on() || ngauges > 64) return false;
    if (!L.children.empty() || L.parent != -1 || L.laycord != 0 || L.laygov != 0 || L.explicit_r24) return false;
    for (int g = 0; g < ngauges; g++)
        if (gc_layer(g_layer[g]) != &L) return false;
    return true;
}

int gcomcot_drive(int nsteps, int maxamp, int ngauges, const int *g_layer, const int *g_i,
                  const int *g_j, float *out4) {
    GcRuntime &rt = gc_rt();
    if (!rt.inited || rt.root < 0) return GC_ESTATE;
    if (nsteps < 0 || ngauges < 0 || (ngauges > 0 && (!g_layer || !g_i || !g_j || !out4))) return GC_EINVAL;
    int root = rt.root;
    GcLayer &R = rt.layers[root];
    bool nested = !R.children.empty();
    for (int g = 0; g < ngauges; g++) {
        GcLayer *L = gc_layer(g_layer[g]);
        if (!L || !L->used || g_i[g] < 1 || g_i[g] >= L->nx || g_j[g] < 1 || g_j[g] >= L->ny) return GC_EINVAL;
    }
    /* The caller of this entry point receives every step's stencils at the
     * end, so no step waits for the host: each step's stencils are gathered
     * on the device (by the kernel gcomcot_get_z_'s snapshot launches, at the
     * same point of the step, or inside a launch of several steps) into a history of
     * up to kChunk steps, which goes to out4 with one copy per chunk.  Same
     * values as the per-step calls. */
    constexpr int kChunk = 1024; /* a launch never straddles chunks */
    int *d_ij = nullptr;
    float *d_hist = nullptr;
    const int chunk = nsteps < kChunk ? (nsteps > 0 ? nsteps + (nsteps & 1) : 2) : kChunk;
    gc_flush();
    if (ngauges > 0) {
        std::vector<int> ij((size_t)2 * ngauges);
        for (int g = 0; g < ngauges; g++) { ij[2 * g] = g_i[g]; ij[2 * g + 1] = g_j[g]; }
        GC_CUDA_OR_RET(cudaMallocAsync((void **)&d_ij, ij.size() * sizeof(int), rt.stream));
        GC_CUDA_OR_RET(cudaMallocAsync((void **)&d_hist, (size_t)chunk * ngauges * 4 * sizeof(float), rt.stream));
        GC_CUDA_OR_RET(cudaMemcpyAsync(d_ij, ij.data(), ij.size() * sizeof(int), cudaMemcpyHostToDevice, rt.stream));
        GC_CUDA_OR_RET(cudaStreamSynchronize(rt.stream)); /* ij is a local vector */
    }
    int rc = GC_OK;
    /* the history holds steps [first, k]: copy it out when the chunk is full
     * or the run ends */
    auto flush_hist = [&](int k) {
        if (ngauges == 0 || rc != GC_OK) return;
        if ((k + 1) % chunk != 0 && k + 1 != nsteps) return;
        const int first = k - k % chunk, cnt = k - first + 1;
        if (cudaMemcpyAsync(out4 + (size_t)first * ngauges * 4, d_hist, (size_t)cnt * ngauges * 4 * sizeof(float),
                            cudaMemcpyDeviceToHost, rt.stream) != cudaSuccess ||
            cudaStreamSynchronize(rt.stream) != cudaSuccess)
            rc = GC_ECUDA;
    };
    /* the gauge stencils of the state after step k (the surface in z2 of
     * the current view, as gcomcot_get_z_'s snapshot reads it) */
    auto gauges_after = [&](int k, const float *z2) {
        GcPdlScope pdl(true);
        float *slot = d_hist + (size_t)(k % chunk) * ngauges * 4;
        int g0 = 0;
        while (g0 < ngauges) {
            int g1 = g0;
            while (g1 < ngauges && g_layer[g1] == g_layer[g0]) g1++;
            GcLayer *L = gc_layer(g_layer[g0]);
            GcLayerDev d = L->view();
            if (z2) d.z2 = (float *)z2;
            else if (!L->z2_valid) d.z2 = L->z[L->cur];
            gc_launch_gauges(d, g1 - g0, d_ij + 2 * g0, slot + 4 * g0, rt.stream);
            rt.launches++;
            g0 = g1;
        }
    };
    int k = 0;
    if (nsteps >= 1 && drive_block_ok(R, maxamp, ngauges, g_layer)) {
        /* each launch (kernels_block.cu; where the grid does not fit it, two
         * steps of kernels_pair.cu) reads the current level (buffer A) and
         * writes the level t steps on into the other buffer (B); the levels
         * between are never stored.  Their gauge stencils are recorded inside
         * the launch.  The last step's are taken by the next launch as it
         * starts (from the level it reads), or by the gauge kernel when no
         * launch of the same history chunk follows. */
        constexpr int kPairVariant = 7; /* 1 warp x 5 stages, the fastest single-grid form on B200 */
        int variant = 0, most = 1;
        gc_block_form(gc_block_pick_form(1, &R.nx, &R.ny), &variant, &most);
        GcFusedGrid g;
        gc_fill_fused_grid(R, g);
        gc_block_plan(variant, g, most);
        const bool block = gc_block_fits(g, 1);
        if (!block) {
            most = 2;
            g.pty = gc_pair_pick_ty(kPairVariant, 1, &R.nx, &R.ny, 2, false);
            g.pte = gc_pair_short_ty(2, g.pty);
            gc_pair_tiles(R.nx, R.ny, g.pty, g.pte, &g.ptiles_x);
        }
        const int least = block ? 1 : 2; /* a last step alone is left to the loop below */
        g.nbuf = 3;
        g.step0 = 0;
        g.nsteps = most + 1 + (block ? 1 : 0);
        g.flags = GC_F_MAXAMP | (ngauges > 0 ? GC_F_STENCIL : 0);
        g.ng = ngauges;
        g.gij = d_ij;
        g.gw = nullptr;
        while (nsteps - k >= least && rc == GC_OK) {
            const int A = R.cur, B = A ^ 1;
            /* local step 1 when the previous step's slot is in this history
             * chunk: the launch then also samples the level it reads into that
             * slot; local step 0 at a chunk's first slot.  Level L is in
             * buffer L % 3, so t is not a multiple of 3. */
            const int local = (ngauges > 0 && k % chunk > 0) ? 1 : 0;
            int t = std::min(most, nsteps - k);
            if (ngauges > 0) t = std::min(t, chunk - k % chunk); /* the chunk is even: so are pairs */
            if (t % 3 == 0) t--;
            for (int q = 0; q < 3; q++) { /* the buffer read is level `local`'s, every other one names B */
                g.z[q] = R.z[q == local ? A : B]; g.m[q] = R.m[q == local ? A : B];
                g.n[q] = R.n[q == local ? A : B];
            }
            g.ts = ngauges > 0 ? d_hist + (size_t)(k % chunk - local) * ngauges * 4 : nullptr;
            {
                GcPdlScope pdl(true);
                const cudaError_t e = block ? gc_block_launch_one(variant, g, t, nullptr, local, rt.stream)
                                            : gc_pair_launch_one_at(kPairVariant, g, nullptr, local, rt.stream);
                if (e != cudaSuccess) rc = GC_ECUDA;
            }
            rt.launches++;
            k += t;
            if (ngauges > 0) {
                /* the next launch samples this one's last step when it exists
                 * and that step's slot is not the last of its chunk */
                const bool next_samples = nsteps - k >= least && k % chunk != 0;
                if (!next_samples) gauges_after(k - 1, R.z[B]);
                flush_hist(k - 1);
            }
            gc_gauge_invalidate();
            gc_swap(R);
        }
    }
    for (; k < nsteps && rc == GC_OK; k++) {
        mass_launch_(nullptr, nullptr, nullptr, &root);
        openbd_launch_(nullptr);
        if (nested) all_grid_launch_();
        momt_launch_(nullptr, nullptr, nullptr, &root);
        if (maxamp) maxamp_launch_(&root);
        if (ngauges > 0) {
            gc_flush();
            gauges_after(k, nullptr);
            flush_hist(k);
        }
        cuda_update_layer_(&root);
    }
    if (d_ij) cudaFreeAsync(d_ij, rt.stream);
    if (d_hist) cudaFreeAsync(d_hist, rt.stream);
    const int rs = gcomcot_sync();
    return rc != GC_OK ? rc : rs;
}

/* GPUall_grids.cu:299-394: device JNQ/NEWQ for (idO, idA) at sub-step t,
 * then a cell-by-cell comparison of the child's boundary fluxes with the
 * caller's, printed like the reference (absolute tolerance 1e-4) */
void edgeinterp_dbglaunch_(float *mO, float *nO, int *idO, float *mA, float *nA, int *idA, int *t,
                           float *yflux, float *xflux) {
    (void)mO; (void)nO; (void)yflux; (void)xflux;
    GcLayer *P = gc_layer(*idO), *C = gc_layer(*idA);
    if (!P || !C || !P->used || !C->used) exit(EXIT_FAILURE);
    gc_flush();
    gc_launch_edges(P->view(), C->view(), C->rel_size, C->rel_time, C->corners, *t, gc_rt().stream);
    std::vector<float> m((size_t)C->nx * C->ny), n((size_t)C->nx * C->ny);
    if (gc_layer_download_field(*C, C->m[C->cur], m.data()) != GC_OK) exit(EXIT_FAILURE);
    if (gc_layer_download_field(*C, C->n[C->cur], n.data()) != GC_OK) exit(EXIT_FAILURE);
    for (int j = 0; j < C->ny; j++) {
        for (int side = 0; side < 2; side++) {
            size_t id = (size_t)j * C->nx + (side ? C->nx - 1 : 0);
            if (fabsf(m[id] - mA[id]) >= 1.0e-4f)
                printf("(%s) i = %d, %f, %f, diff=%f\n", side ? "right" : "left", j, m[id], mA[id],
                       fabsf(m[id] - mA[id]));
        }
    }
    for (int i = 0; i < C->nx; i++) {
        for (int side = 0; side < 2; side++) {
            size_t id = (size_t)(side ? C->ny - 1 : 0) * C->nx + i;
            if (fabsf(n[id] - nA[id]) >= 1.0e-4f)
                printf("(%s) i = %d, %f, %f, diff=%f\n", side ? "top" : "bottom", i, n[id], nA[id],
                       fabsf(n[id] - nA[id]));
        }
    }
}

/* GPUall_grids.cu:626-643: device JNZ, then compare the parent surface */
void jnz_dbglaunch_(float *Z_f, int *outid, int *inid) {
    GcLayer *P = gc_layer(*outid), *C = gc_layer(*inid);
    if (!P || !C || !P->used || !C->used) exit(EXIT_FAILURE);
    gc_flush();
    gc_launch_jnz(P->view(), C->view(), C->rel_size, C->rel_time, C->corners, gc_rt().stream);
    P->z2_valid = true;
    std::vector<float> z((size_t)P->nx * P->ny);
    if (gc_layer_download_field(*P, P->z[P->cur ^ 1], z.data()) != GC_OK) exit(EXIT_FAILURE);
    for (int j = 0; j < P->ny; j++)
        for (int i = 0; i < P->nx; i++) {
            size_t id = (size_t)j * P->nx + i;
            if (fabsf(z[id] - Z_f[id]) >= 1.0e-4f)
                printf("JNZ, layerid=%d(i,j)=(%d,%d), %f %f, diff=%lf\n", *inid, i, j, z[id], Z_f[id],
                       (double)fabsf(z[id] - Z_f[id]));
        }
}

} /* extern "C" */
