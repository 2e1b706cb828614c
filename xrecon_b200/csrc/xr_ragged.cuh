// Ragged batch of 2D reconstructions (projection then FBP) in one persistent
// cooperative launch.
//
// Every instance has its own geometry, image size, view count and detector.
// The kernel runs four phases over a list of tiles that spans all instances;
// each block takes tiles from a per-phase atomic counter, so instances of
// very different cost share the GPU without idle SMs.  Phases are separated
// by a grid barrier whose waits are bounded (a timeout sets the device error
// word and ends the kernel):
//   0  per-view DD tables of every instance (FP64) and the line tables of
//      every image (xr_dd2d.cuh);
//   1  projection A, cell-owned: a tile is CW pairs of columns of one view, the
//      256 / CW threads of a pair split its lines and reduce in shared
//      memory;
//   2  FBP pre-filter of every sinogram row: cosine weight x correlation with
//      the instance's filter taps (the same arithmetic as fbp_filter_kernel),
//      then the filtered row's table for the next phase (xr_dd2d.cuh);
//   3  weighted backprojection Bw of the filtered rows times the FBP scale,
//      pixel-owned: a tile is 8 / VS warps of 2 x 2 pixel blocks (xr_dd2d.cuh),
//      VS warps split a block's views and reduce in shared memory.
// CW and VS are launch parameters chosen by the autotuner of the Python
// wrapper.  No atomics touch data: the counters only hand out tiles.
#pragma once

#include "xr_dd2d.cuh"
#include "xr_tma.cuh"

namespace xr {

constexpr unsigned XR_DEVERR_BARRIER_TIMEOUT = 2u;
// polls of ~128 ns: about half a second by default (xr_set_wait_limits)
constexpr long long XR_BARRIER_LIMIT_DEFAULT = 1ll << 22;
__device__ long long g_barrier_limit = XR_BARRIER_LIMIT_DEFAULT;

// One instance, device side (pointers already resolved).
struct RaggedDev {
    Geom g;
    Geom2F f;
    ViewTables vt;
    int nview;
    float cw;       // backprojection column width
    float scale;    // FBP scale
    const float* img;
    LineTable lines;
    float* sino;
    float* filt_out;
    RowTable tab;   // row tables of filt_out and their error bounds (xr_dd2d.cuh; q null: no
                    // tables, every row is walked)
    float* eps;
    float* recon;
    const float* ang;
    const float* filt;
    const float* cosw;
    // first tile of this instance in each tile list: [0] tables and
    // line tables, [1] filter rows, [2 + i] projection with CW = 32 << i,
    // [6 + i] backprojection with VS = 1 << i
    int t0[10];
};

// Bounded grid barrier over nblocks co-resident blocks; bar[0] counts
// arrivals, bar[1] is the generation.  False when a wait gave up.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned nblocks) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned* vgen = bar + 1;
        const unsigned gen = *vgen;
        __threadfence();
        const unsigned arrived = atomicAdd(bar, 1u) + 1u;
        const long long limit = *(volatile long long*)&g_barrier_limit;
        // test hook: one block more than the grid is expected, nobody releases
        if (*(volatile unsigned*)&g_test_hooks & XR_HOOK_BARRIER_EXTRA) ++nblocks;
        int ok = 1;
        if (arrived == nblocks) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            long long i = 0;
            while (*vgen == gen) {
                if (++i > limit) {
                    atomicOr(&g_device_error, XR_DEVERR_BARRIER_TIMEOUT);
                    ok = 0;
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

// Instance owning global tile t of tile list p (t0[p] ascending).
__device__ __forceinline__ int find_instance(const RaggedDev* __restrict__ inst, int ninst, int p, int t) {
    int lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (inst[mid].t0[p] <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int next_tile(int* ctr) {
    __shared__ int t_s;
    __syncthreads();
    if (threadIdx.x == 0) t_s = atomicAdd(ctr, 1);
    __syncthreads();
    return t_s;
}

// Filtered rows of one view; written by this kernel, so not through __ldg.
struct FiltLanes {
    const float* p;
    __device__ __forceinline__ Lanes<1> operator()(int col) const {
        Lanes<1> r;
        r.v[0] = p[col];
        return r;
    }
};

__global__ void __launch_bounds__(256, 3)
ragged2d_fbp_kernel(const RaggedDev* __restrict__ inst, const int ninst, const int4 totals, const int4 lists,
                    const int project, const int CW, const int VS, unsigned* bar, int* ctr) {
    extern __shared__ float sm[];
    __shared__ double2 row_sums[8];
    const int tid = threadIdx.x;
    const unsigned nb = gridDim.x;

    // phase 0: view tables and transposes
    for (int t = next_tile(&ctr[0]); t < totals.x; t = next_tile(&ctr[0])) {
        const RaggedDev& I = inst[find_instance(inst, ninst, lists.x, t)];
        const int lt = t - I.t0[lists.x];
        const Geom& g = I.g;
        if (lt < I.nview) {
            for (int k = tid; k <= g.Nu; k += blockDim.x) setup_view_entry(g, 0, I.ang[lt], lt, k, I.vt, g.type == GEO_ARC);
        } else {
            const int l = (lt - I.nview) * 8 + (tid >> 5);
            if (l < g.W + g.H) {
                if (I.lines.q) build_line_table(I.img, I.lines, l, tid & 31);
                else I.lines.flags[l] = 1;
            }
        }
    }
    if (!grid_barrier(bar, nb)) return;

    // phase 1: projection
    if (project) {
        const int LS = blockDim.x / CW;
        for (int t = next_tile(&ctr[1]); t < totals.y; t = next_tile(&ctr[1])) {
            const RaggedDev& I = inst[find_instance(inst, ninst, lists.y, t)];
            const Geom& g = I.g;
            const int nbk = (g.Nu + 2 * CW - 1) / (2 * CW);
            const int lt = t - I.t0[lists.y];
            const int v = lt / nbk, kb = lt - v * nbk;
            const int c = tid % CW, s = tid / CW;
            const int k = 2 * (kb * CW + c);
            const ViewHdr& h = I.vt.hdr[v];
            float acc[2] = {0.0f, 0.0f};
            if (k < g.Nu) cell2t_walk<OP_A>(I.f, I.vt, h, v, k, 0.0f, s, LS, I.lines, I.img, acc);
            sm[tid] = acc[0];
            sm[256 + tid] = acc[1];
            __syncthreads();
            if (s == 0)
                for (int e = 0; e < 2 && k + e < g.Nu; ++e) {
                    float sum = 0.0f;
                    for (int j = 0; j < LS; ++j) sum += sm[e * 256 + j * CW + c];
                    sum *= I.vt.colE[(size_t)v * g.Nu + k + e];
                    const int col = h.keep ? k + e : g.Nu - 1 - (k + e);
                    I.sino[(size_t)v * g.Nu + col] = sum;
                }
        }
    }
    if (!grid_barrier(bar, nb)) return;

    // phase 2: cosine weight x filter correlation, one sinogram row per tile
    for (int t = next_tile(&ctr[2]); t < totals.z; t = next_tile(&ctr[2])) {
        const RaggedDev& I = inst[find_instance(inst, ninst, lists.z, t)];
        const int Nu = I.g.Nu;
        const int v = t - I.t0[lists.z];
        float* x = sm;             // Nu
        float* f = sm + Nu;        // 2 Nu - 1
        for (int j = tid; j < Nu; j += blockDim.x) x[j] = I.sino[(size_t)v * Nu + j] * I.cosw[j];
        for (int j = tid; j < 2 * Nu - 1; j += blockDim.x) f[j] = I.filt[j];
        __syncthreads();
        for (int i = tid; i < Nu; i += blockDim.x) {
            // out[i] = sum_j x[j] f[j - i + Nu - 1]
            const float* fi = f + (Nu - 1 - i);
            float a0 = 0.0f, a1 = 0.0f;
            int j = 0;
            for (; j + 1 < Nu; j += 2) {
                a0 = fmaf(x[j], fi[j], a0);
                a1 = fmaf(x[j + 1], fi[j + 1], a1);
            }
            if (j < Nu) a0 = fmaf(x[j], fi[j], a0);
            I.filt_out[(size_t)v * Nu + i] = a0 + a1;
        }
        if (!I.tab.q) {  // uniform over the CTA
            if (tid == 0) I.eps[v] = ROW_WALK;
            continue;
        }
        __syncthreads();  // the whole row is in filt_out
        const float* y = I.filt_out + (size_t)v * Nu;
        const int keep = I.vt.hdr[v].keep;
        const float e = build_row_table(I.f, I.vt, v, I.tab.at(v, Nu), row_sums,
                                        [&](int j) -> float { return y[keep ? j : Nu - 1 - j]; });
        if (tid == 0) I.eps[v] = e;
    }
    if (!grid_barrier(bar, nb)) return;

    // phase 3: weighted backprojection x FBP scale
    {
        const int ntile = 8 / VS, lane = tid & 31, wp = tid >> 5, slice = wp / ntile;
        for (int t = next_tile(&ctr[3]); t < totals.w; t = next_tile(&ctr[3])) {
            const RaggedDev& I = inst[find_instance(inst, ninst, lists.w, t)];
            const int W = I.f.W, H = I.f.H;
            int ix0, iy0;
            pix2t_origin(I.f, VS, t - I.t0[lists.w], wp % ntile, lane, ix0, iy0);
            const bool active = ix0 < W && iy0 < H;
            float acc[P2][P2] = {};
            auto row = [&](int v) { return FiltLanes{I.filt_out + (size_t)v * I.f.Nu}; };
            if (active && I.vt.arc) pix2t_views<OP_BW, true>(I.f, I.vt, I.tab, I.eps, ix0, iy0, I.cw, slice, I.nview, VS, row, acc);
            else if (active) pix2t_views<OP_BW, false>(I.f, I.vt, I.tab, I.eps, ix0, iy0, I.cw, slice, I.nview, VS, row, acc);
            float* a = &acc[0][0];
#pragma unroll
            for (int e = 0; e < P2 * P2; ++e) sm[e * 256 + tid] = a[e];
            __syncthreads();
            if (!slice && active) {
                for (int s = 1; s < VS; ++s)
#pragma unroll
                    for (int e = 0; e < P2 * P2; ++e) a[e] += sm[e * 256 + s * ntile * 32 + tid];
#pragma unroll
                for (int r = 0; r < P2; ++r)
#pragma unroll
                    for (int c = 0; c < P2; ++c)
                        if (ix0 + c < W && iy0 + r < H) I.recon[(iy0 + r) * W + ix0 + c] = acc[r][c] * I.scale;
            }
        }
    }
    // leave the tile counters at zero for the next launch
    if (!grid_barrier(bar, nb)) return;
    if (blockIdx.x == 0 && tid < 4) ctr[tid] = 0;
}

}  // namespace xr
