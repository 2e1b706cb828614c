// 2D distance-driven gathers.
//
// Cell gather (A, B^T, Bw^T): a thread owns one detector cell and a slice of
// the image lines.  Pixel gather (A^T, B, Bw): a thread owns one pixel and a
// slice of the views.  2D images and sinograms are small (they stay in L2,
// most of them in L1), so what costs is the geometry per (cell, line) or
// (pixel, view) and, when few cells or pixels are asked for, the length of
// one thread's serial loop.  Hence:
//   - the loop is split over up to 8 warps of the CTA, summed in a fixed order
//     through shared memory;
//   - a batch of images shares the geometry: the input is first interleaved in
//     groups of NB = 2, 4 or 8 images, and a thread carries NB sums, so each
//     (pixel, column) pair costs one or two 16-byte loads and NB FMAs once its
//     weight is known;
//   - a pixel-gather thread owns a 2 x 2 block of pixels, whose edges on a
//     line are shared;
//   - single images are projected through tables of their lines' integrals
//     (cell2t_kernel), and up to PT_MAX_BATCH images are gathered through per-view tables of the
//     detector row's integral (pix2t_kernel: one table entry per pixel edge,
//     no column loop); larger batches walk the columns once for NB images
//     (pix2d_kernel).
// No atomics: every output has one owner.
//
// Measured on a B200, before (one thread per output, no split, no tables) and
// now, us: FBP of 256 x 256 pixels from 720 fan-flat views 1055 -> 223; a batch of
// eight 512 x 512 arc slices, A + A^T over 360 views, 10855 -> 1546; A + FBP of 16
// ragged fan-arc instances 20344 -> 12300.  The pixel gathers
// are held by the latency of their table entries in L1 and by conversions, the
// batched walks by L1 wavefronts and lanes in different columns.
//
// Which of these a call takes goes by the batch, the scratch given and the values
// (a row of too wide a spread is walked), so the same image may differ by float32
// rounding between them.
#pragma once

#include <cmath>

#include <cooperative_groups.h>

#include "xr_kernels.cuh"

namespace xr {

// Column width, in pixels, up to which a boundary may be its neighbour plus an
// FP32 width (error below 2.4e-7 pixel).
constexpr float XR_WIDE2D = 4.0f;

// FP32 constants of a 2D geometry (column guesses; exactness comes from the
// FP64 tables).
struct Geom2F {
    float x0, y0, xc0, yc0;  // left / bottom image edge, centre of column 0 / row 0
    float dx, dy, inv_dx, inv_dy;
    float sod, shu, du, inv_du, half_nu;
    // error bound of pix2t_view's FP32 column position, in columns: eps0 + eps1
    // / distance from the source (flat: along the central ray) of any point of the
    // 2 x 2 block, at most epsw
    float eps0, eps1, epsw;
    float guess;  // error bound of pix2d_axis's column guess, in columns
    int W, H, Nu, type;
};

__host__ __device__ inline Geom2F make_geom2f(const Geom& g) {
    Geom2F f;
    f.x0 = (float)(-0.5 * g.W * g.dx + g.shx);
    f.y0 = (float)(-0.5 * g.H * g.dy + g.shy);
    f.xc0 = (float)((0.5 - 0.5 * g.W) * g.dx + g.shx);
    f.yc0 = (float)((0.5 * g.H - 0.5) * g.dy + g.shy);
    f.dx = (float)g.dx; f.dy = (float)g.dy;
    f.inv_dx = (float)(1.0 / g.dx); f.inv_dy = (float)(1.0 / g.dy);
    f.sod = (float)g.sod; f.shu = (float)g.shu; f.du = (float)g.du;
    f.inv_du = (float)(1.0 / g.du);
    f.half_nu = 0.5f * (float)g.Nu;
    // First-order sums of the roundings, u = 2^-24 each.  r bounds |x| and |y| together (its square root of
    // two is in the factors), U the detector's half-width.
    const double u = std::ldexp(1.0, -24);
    const double hx = 0.5 * g.W * g.dx + std::fabs(g.shx), hy = 0.5 * g.H * g.dy + std::fabs(g.shy);
    const double r = std::sqrt(hx * hx + hy * hy), U = 0.5 * g.Nu * g.du + std::fabs(g.shu);
    double e0 = u * 2.0 * g.Nu, e1 = 0.0, near = 1.0;
    if (g.type == GEO_FLAT) {
        // u = sod (x cos + y sin) / (sod + x sin - y cos)
        e0 += u * 3.0 * U / g.du;
        e1 = u * (4.3 * g.sod * r + U * (2.0 * g.sod + 4.3 * r)) / g.du;
        near = g.sod - r;
    } else if (g.type == GEO_ARC) {
        // atan2 of the point seen from the source, and the float32 axis
        // positions of the boundaries (arc_axis_f; within 1.7e-7 rad)
        e0 += (u * 1.5 + 1.3e-7 + 1.7e-7) / g.du;
        e1 = u * 1.5 * (r + g.sod) / g.du;
        near = (g.sod - r) * 0.7;  // the larger component of a vector of that length
    } else {
        e0 += u * 4.3 * r / g.du;
    }
    // (half as much again: the block is three pixels across, a third of `near`)
    e1 *= 1.5;
    if (near < 9.0 * std::max(g.dx, g.dy)) e0 += e1 / near, e1 = 0.0;
    f.eps0 = (float)e0;
    f.eps1 = (float)e1;
    f.epsw = (float)(e0 + e1 / near);
    f.guess = f.epsw + (g.type == GEO_ARC ? XR_GUESS_ATAN_ERR * f.inv_du : 0.0f);
    f.W = g.W; f.H = g.H; f.Nu = g.Nu; f.type = g.type;
    return f;
}

// fbp_weight at FP32 pixel centre (px, py) from the header's FP32 source.
__device__ __forceinline__ float fbp_weight2d(const Geom2F& f, float sx, float sy, float px, float py) {
    if (f.type == GEO_FLAT) {
        const float R = f.sod;
        const float den = R - __fdividef(sx * px + sy * py, R);
        return __fdividef(R * R, den * den);
    }
    if (f.type == GEO_ARC) {
        const float ex = sx - px, ey = sy - py;
        return __fdividef(1.0f, ex * ex + ey * ey);
    }
    return 1.0f;
}

// NB images' values of one element i of an interleaved group: planes of up
// to four images, [plane][n][4] (NB = 2: [n][2]), so that a warp's 16-byte
// loads of neighbouring elements are contiguous.
template <int NB> struct Lanes { float v[NB]; };
template <int NB>
__device__ __forceinline__ Lanes<NB> ld_lanes(const float* p, size_t n, size_t i) {
    Lanes<NB> r;
    if constexpr (NB == 2) {
        const float2 a = reinterpret_cast<const float2*>(p)[i];
        r.v[0] = a.x; r.v[1] = a.y;
    } else {
#pragma unroll
        for (int e = 0; e < NB; e += 4) {
            const float4 a = reinterpret_cast<const float4*>(p)[(size_t)(e / 4) * n + i];
            r.v[e] = a.x; r.v[e + 1] = a.y; r.v[e + 2] = a.z; r.v[e + 3] = a.w;
        }
    }
    return r;
}

// ------------------------------------------------------------ preparation

// Per-view tables and the input's second form in one launch (both small):
// blocks [0, nset) fill the tables, one view and 256 boundaries each; the
// rest prepare the input, NB = 1: the flipped transpose of every image, 32 x
// 32 pixels a block (out_cols; nothing for a sinogram); NB > 1: the
// interleaved copy of each group of NB (the planes of ld_lanes), 256 elements a
// block, for images also in the flipped transpose's order.
template <typename T, int NB>
__global__ void __launch_bounds__(256)
prep2d_kernel(const Geom g, const float* __restrict__ ang, const int nview, const ViewTables vt, const int nset,
              const T* __restrict__ in, void* __restrict__ out_rows, void* __restrict__ out_cols, const int nbatch,
              const long long n, const int per_img) {
    const int tid = threadIdx.x;
    if ((int)blockIdx.x < nset) {
        const int bpv = (g.Nu + 1 + 255) / 256;
        const int v = blockIdx.x / bpv, k = (blockIdx.x % bpv) * 256 + tid;
        if (v < nview && k <= g.Nu) setup_view_entry(g, 0, ang[v], v, k, vt, g.type == GEO_ARC);
        return;
    }
    const int id = blockIdx.x - nset, b = id / per_img, t = id % per_img;
    if constexpr (NB == 1) {
        __shared__ T tile[32][33];
        const int tx = (g.W + 31) / 32, x0 = (t % tx) * 32, y0 = (t / tx) * 32;
        const T* src = in + (size_t)b * g.H * g.W;
        T* dst = static_cast<T*>(out_cols) + (size_t)b * g.H * g.W;
        for (int dy = tid / 32; dy < 32; dy += 8) {
            const int y = y0 + dy, x = x0 + tid % 32;
            if (y < g.H && x < g.W) tile[dy][tid % 32] = src[(size_t)y * g.W + x];
        }
        __syncthreads();
        for (int dx = tid / 32; dx < 32; dx += 8) {
            const int x = x0 + dx, y = y0 + tid % 32;
            if (y < g.H && x < g.W) dst[(size_t)x * g.H + (g.H - 1 - y)] = tile[tid % 32][dx];
        }
    } else {
        const int i = t * 256 + tid;  // a group is at most 1 GiB
        if (i >= n) return;
        float x[NB];
#pragma unroll
        for (int e = 0; e < NB; ++e) {
            const int bb = b * NB + e;
            x[e] = bb < nbatch ? ld(in + (size_t)bb * n + i) : 0.0f;
        }
        auto put = [&](void* o, size_t j) {
            float* ob = static_cast<float*>(o) + (size_t)b * n * NB;
            if constexpr (NB == 2) reinterpret_cast<float2*>(ob)[j] = make_float2(x[0], x[1]);
            else
#pragma unroll
                for (int e = 0; e < NB; e += 4)
                    reinterpret_cast<float4*>(ob)[(size_t)(e / 4) * n + j] = make_float4(x[e], x[e + 1], x[e + 2], x[e + 3]);
        };
        put(out_rows, i);
        if (out_cols) {
            const int y = i / g.W, xx = i - y * g.W;
            put(out_cols, (size_t)xx * g.H + (g.H - 1 - y));
        }
    }
}

// ------------------------------------------------------------ cell gather

// Cell k of view v (traversal order), lines L = l0, l0 + ls, ...: calls
// add(L, p, w) for every pixel p of line L the column overlaps, w the overlap
// in pixels times the line factor (A; the cell scale colE is the caller's) or
// the column width (B^T, Bw^T; times the FBP weight).  Pixels come from one
// FP64 boundary per line: its floor is an add of 1.5 * 2^52 rounded down,
// whose low word is the pixel, and the column's width on the line is FP32
// (dA + dB L).  Columns wider than XR_WIDE2D pixels (an FP32 sum would lose
// more of the far boundary than FP64 does), cells whose boundaries leave
// +-2^30 pixels, lines entered left of the image and the chained arc
// transposes take both boundaries in FP64.
template <int MODE, typename Add>
__device__ __forceinline__ void cell2d_walk(const Geom& g, const Geom2F& f, const ViewTables& vt, const ViewHdr& h,
                                            const int v, const int k, const float cw, const int l0, const int ls,
                                            Add&& add) {
    const int Nu = f.Nu;
    const size_t ob = (size_t)v * (Nu + 1) + k;
    const double bA0 = vt.bA[ob], bB0 = vt.bB[ob], bA1 = vt.bA[ob + 1], bB1 = vt.bB[ob + 1];
    const int nlines = h.nlines, npix = h.npix;
    const float dpixf = (float)h.dpix;
    // arc detector, B^T / Bw^T: the column's upper boundary on the chained
    // walk of a pixel whose first edge lies in this column (every pixel but
    // the band's first); the same on every line
    const bool chain = (MODE == OP_BT || MODE == OP_BWT) && vt.arc;
    const float4* ea = chain ? vt.arc + 2 * (size_t)v * (Nu + 1) : nullptr;
    float d1 = 0.0f;
    if (chain) {
        ArcChain ch;
        ch.start(ea, k, h.keep, f.du);
        d1 = ch.next_exact(h, ea, k + 1);
        if (k + 1 == Nu) d1 = fminf(d1, 0.0f);
    }
    const double lim = 1073741824.0, nl = (double)(nlines - 1);
    auto in_lim = [&](double x) { return x > -lim && x < lim; };
    const float dA = (float)(bA1 - bA0), dB = (float)(bB1 - bB0);
    const double q0 = h.q0, q1 = h.q1;
    const bool behind = !(q0 > 0.0 && fma(q1, nl, q0) > 0.0);  // some lines lie behind the source's plane
    const bool exact = chain || behind || !(in_lim(bA0) && in_lim(fma(bB0, nl, bA0)) && in_lim(bA1) && in_lim(fma(bB1, nl, bA1))) ||
                       !(fmaxf(fabsf(dA), fabsf(fmaf(dB, (float)nl, dA))) < XR_WIDE2D);
    for (int L = l0; L < nlines; L += ls) {
        const double dL = (double)L;
        const double pk = fma(bB0, dL, bA0);
        int pa, pb = npix - 1;
        float u0, u1, u1b;
        if (!exact) {
            const double tr = __dadd_rd(pk, 6755399441055744.0);  // 1.5 * 2^52: floor in the low word
            const int ip = __double2loint(tr);
            pa = max(ip, 0);
            if (ip >= 0) {
                u0 = (float)(pk - (tr - 6755399441055744.0));
                u1 = u0 + fmaf(dB, (float)L, dA);
            } else {
                u0 = (float)pk;
                u1 = (float)fma(bB1, dL, bA1);
            }
            u1b = u1;
            if (pa > pb || !(u1 > 0.0f)) continue;
        } else {
            const double pk1 = fma(bB1, dL, bA1);
            if (behind && !(fma(q1, dL, q0) > 0.0)) continue;
            pa = max((int)floor(pk), 0);
            pb = min(max((int)ceil(pk1), 0) - 1, pb);
            if (pa > pb) continue;
            u0 = (float)(pk - (double)pa);
            u1 = (float)(pk1 - (double)pa);
            u1b = u1;  // upper boundary for the band's later pixels
            if (chain) {
                const float qd = (float)(fma(q1, dL, q0) / h.dpix);
                u1b = fmaf(d1, qd, u1);
                u1 = u1b;
                if (k > 0 && pk > (double)pa)
                    arc_first_pixel_bounds(g, vt, h, ea, v, k, L, pa, pk, pk1, qd, u0, u1);
            }
        }
        float lf;
        if (MODE == OP_A) lf = __fdividef(dpixf, (float)fma(q1, dL, q0));
        else lf = cw;
        for (int pp = pa; pp <= pb; ++pp) {
            const float o = (float)(pp - pa);
            if (!exact && !(o < u1)) break;
            float w = (fminf(o + 1.0f, pp == pa ? u1 : u1b) - fmaxf(o, u0)) * lf;
            if (MODE == OP_BWT) {
                const int ix = h.use_x ? pp : L, iy = h.use_x ? L : f.H - 1 - pp;
                w *= fbp_weight2d(f, h.sxr, h.syr, fmaf((float)ix, f.dx, f.xc0), fmaf(-(float)iy, f.dy, f.yc0));
            }
            add(L, XR_BOUND(pp, 0, npix - 1), w);
        }
    }
}

// A CTA's 8 warps are 8 / LS blocks of 32 columns times LS line slices.
// NB = 1: rows and cols are the images [batch][line][pixel] of type TI;
// NB > 1: their interleaved FP32 copies, blockIdx.z the group.
template <typename TI, int NB, int MODE>
__global__ void __launch_bounds__(256)
cell2d_kernel(const Geom g, const Geom2F f, const ViewTables vt, const TI* __restrict__ rows,
              const TI* __restrict__ cols, void* __restrict__ sino, const int dto, const int nview, const int b0,
              const int nbatch, const float cw, const int LS) {
    __shared__ float red[8][NB][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nblk = 8 / LS, slice = wp / nblk;
    const int k = (blockIdx.x * nblk + wp % nblk) * 32 + lane;
    const int v = blockIdx.y;
    const ViewHdr& h = vt.hdr[v];
    const size_t plane = (size_t)f.W * f.H;
    const TI* __restrict__ img = (h.use_x ? rows : cols) + blockIdx.z * plane * NB;
    const int npix = h.npix;
    float acc[NB];
#pragma unroll
    for (int e = 0; e < NB; ++e) acc[e] = 0.0f;
    if (k < f.Nu)
        cell2d_walk<MODE>(g, f, vt, h, v, k, cw, slice, LS, [&](int L, int p, float w) {
            const size_t q = (size_t)L * npix + p;
            if constexpr (NB == 1) {
                acc[0] = fmaf(w, ld(img + q), acc[0]);
            } else {
                const Lanes<NB> x = ld_lanes<NB>(img, plane, q);
#pragma unroll
                for (int e = 0; e < NB; ++e) acc[e] = fmaf(w, x.v[e], acc[e]);
            }
        });
    if (LS > 1) {
#pragma unroll
        for (int e = 0; e < NB; ++e) red[wp][e][lane] = acc[e];
        __syncthreads();
        if (slice) return;
        for (int s = 1; s < LS; ++s)
#pragma unroll
            for (int e = 0; e < NB; ++e) acc[e] += red[s * nblk + wp][e][lane];
    }
    if (k >= f.Nu) return;
    const float scale = MODE == OP_A ? vt.colE[(size_t)v * f.Nu + k] : 1.0f;
    const int col = h.keep ? k : f.Nu - 1 - k;
#pragma unroll
    for (int e = 0; e < NB; ++e) {
        const int b = b0 + blockIdx.z * NB + e;
        if (b < nbatch) st_dt(sino, dto, ((size_t)b * nview + v) * f.Nu + col, acc[e] * scale);
    }
}

// ------------------------------------------ cell gather through line tables
//
// With x in pixel p of line L, the line integrated up to x is S(x) = Q_p + v_p x,
// Q_p = sum_{j < p} v_j - v_p p, so a cell's sum over the line is S(upper
// boundary) - S(lower boundary): one 16-byte entry and one FP64 FMA per boundary
// (shared by two neighbouring cells), whatever the number of pixels.  S is FP64,
// of up to n |v|max in magnitude (n pixels), so a difference is off by a few
// 2^-53 n |v|max: less than FP32 loses on pixels near the largest, but all of a
// pixel that is 2^-40 of it.  Lines whose smallest value would lose 2^-18 of itself
// (Spread::too_wide: one dead pixel of 1e20, a mask of the lowest float), and those
// holding an infinity or a NaN, are flagged and walked pixel by pixel.  S is
// continuous, so the pixel may be taken from the FP32 position (one off for the
// few positions within its rounding of an integer, by at most that rounding times
// the pixels' difference).  Lines of both orientations are tabulated, entries -1 ..
// npix (the outer ones continue S as a constant).

// Magnitudes of a table's values, as the bits of |v|: the largest (an infinity or
// a NaN is above every finite one) and the smallest but zero.
struct Spread {
    unsigned most = 0u, least = 0xffffffffu;
    __device__ __forceinline__ void add(float v) {
        const unsigned b = (unsigned)__float_as_int(v) & 0x7fffffffu;
        most = max(most, b);
        if (b) least = min(least, b);
    }
    __device__ __forceinline__ void warp() {
        most = __reduce_max_sync(0xffffffffu, most);
        least = __reduce_min_sync(0xffffffffu, least);
    }
    // whether sums over positions of up to `reach` pixels are no good for these
    // values: 2^-53 reach |v|max, a few times, is to stay below 2^-18 |v|min
    __device__ __forceinline__ bool too_wide(float reach) const {
        if (most == 0u) return false;
        return most >= 0x7f800000u || !((double)__int_as_float((int)most) * (double)reach <=
                                        8589934592.0 * (double)__int_as_float((int)least));
    }
};

struct LineTable {
    double2* q;  // H lines of W + 2, then W lines of H + 2; null: no table, every line is flagged
    int* flags;  // H, then W
    int W, H;
    __host__ __device__ __forceinline__ size_t start(bool rows, int L) const {
        return rows ? (size_t)L * (W + 2) : (size_t)H * (W + 2) + (size_t)L * (H + 2);
    }
};
__host__ __device__ inline size_t line_table_entries(int W, int H) { return (size_t)H * (W + 2) + (size_t)W * (H + 2); }

// One line's table, by one warp: line l < H is image row l, the others the
// columns from the bottom up.
template <typename T>
__device__ __forceinline__ void build_line_table(const T* img, const LineTable& t, int l, int lane) {
    const bool rows = l < t.H;
    const int L = rows ? l : l - t.H, n = rows ? t.W : t.H;
    double2* q = t.q + t.start(rows, L);
    double carry = 0.0;
    Spread spread;
    if (lane == 0) q[0] = make_double2(0.0, 0.0);
    for (int base = 0; base <= n; base += 32) {
        const int p = base + lane;
        double v = 0.0;
        if (p < n) {
            const float x = ld(rows ? img + (size_t)L * t.W + p : img + (size_t)(t.H - 1 - p) * t.W + L);
            spread.add(x);
            if (isfinite(x)) v = (double)x;
        }
        double s = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double u = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += u;
        }
        if (p <= n) q[p + 1] = make_double2(carry + (s - v) - v * (double)p, v);
        carry += __shfl_sync(0xffffffffu, s, 31);
    }
    spread.warp();
    if (lane == 0) t.flags[l] = spread.too_wide((float)n);
}

// Blocks [0, nset): view tables; the rest: eight lines each of an image's table.
template <typename T>
__global__ void __launch_bounds__(256)
linetab2d_kernel(const Geom g, const float* __restrict__ ang, const int nview, const ViewTables vt, const int nset,
                 const T* __restrict__ in, LineTable tab) {
    if ((int)blockIdx.x < nset) {
        const int bpv = (g.Nu + 1 + 255) / 256;
        const int v = blockIdx.x / bpv, k = (blockIdx.x % bpv) * 256 + threadIdx.x;
        if (v < nview && k <= g.Nu) setup_view_entry(g, 0, ang[v], v, k, vt, g.type == GEO_ARC);
        return;
    }
    const int per = (g.W + g.H + 7) / 8, id = blockIdx.x - nset, b = id / per;
    const int l = (id % per) * 8 + (threadIdx.x >> 5);
    if (l >= g.W + g.H) return;
    tab.q += b * line_table_entries(g.W, g.H);
    tab.flags += (size_t)b * (g.W + g.H);
    build_line_table(in + (size_t)b * g.W * g.H, tab, l, threadIdx.x & 31);
}

// One cell's sum over line L, pixel by pixel: columns from pk to pk1, weight lf per
// pixel.
template <typename T>
__device__ __noinline__ float line_walk(const LineTable& tab, const T* img, bool rows, int L, int npix, double pk, double pk1,
                                        float lf) {
    const int pa = max((int)floor(pk), 0), pb = min(max((int)ceil(pk1), 0), npix) - 1;
    float s = 0.0f;
    for (int p = pa; p <= pb; ++p) {
        const float w = (float)(fmin((double)(p + 1), pk1) - fmax((double)p, pk)) * lf;
        s = fmaf(w, ld(rows ? img + (size_t)L * tab.W + p : img + (size_t)(tab.H - 1 - p) * tab.W + L), s);
    }
    return s;
}

// Cells k and k + 1 (k + 1 < Nu or dropped by the caller) of view v over lines
// l0, l0 + ls, ...; img is the image itself (flagged lines).
template <int MODE, typename T>
__device__ __forceinline__ void cell2t_walk(const Geom2F& f, const ViewTables& vt, const ViewHdr& h, const int v,
                                            const int k, const float cw, const int l0, const int ls,
                                            const LineTable& tab, const T* img, float (&acc)[2]) {
    const int Nu = f.Nu, nlines = h.nlines, npix = h.npix;
    const bool rows = h.use_x;
    const size_t ob = (size_t)v * (Nu + 1);
    double A[3], B[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int kk = min(k + e, Nu);
        A[e] = vt.bA[ob + kk];
        B[e] = vt.bB[ob + kk];
    }
    const double q0 = h.q0, q1 = h.q1;
    const float dpixf = (float)h.dpix;
    const int* flags = tab.flags + (rows ? 0 : tab.H);
    // columns whose boundaries are not in order on every line are walked: a ray
    // past 90 degrees from the axis, or an image with lines behind the source's
    // plane, which a column overlaps nowhere
    const double nl = (double)(nlines - 1);
    bool ordered = true;
#pragma unroll
    for (int c = 0; c < 2; ++c)
        ordered = ordered && (k + c >= Nu || (A[c + 1] > A[c] && A[c + 1] - A[c] < 1.0e300 &&
                                              fma(B[c + 1], nl, A[c + 1]) > fma(B[c], nl, A[c])));
    auto factor = [&](double dL) { return MODE == OP_A ? dpixf * rcp_fast((float)fma(q1, dL, q0)) : cw; };
    bool rest = !ordered;  // lines left to the walk
    for (int L = ordered ? l0 : nlines; L < nlines; L += ls) {
        const double dL = (double)L;
        if (flags[L]) {
            rest = true;
            continue;
        }
        const float lf = factor(dL);
        const double2* q = tab.q + tab.start(rows, L);
        double S[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            const double pos = fma(B[e], dL, A[e]);
            const float pf = fminf(fmaxf((float)pos, -1.0f), (float)npix);
            const double2 t = q[XR_BOUND((__float_as_int(__fadd_rd(pf, 12582912.0f)) - 0x4B400000) + 1, 0, npix + 1)];
            S[e] = fma(t.y, pos, t.x);
        }
        acc[0] = fmaf(lf, (float)(S[1] - S[0]), acc[0]);
        acc[1] = fmaf(lf, (float)(S[2] - S[1]), acc[1]);
    }
    // after the others, so that the loop above keeps its registers
    for (int L = rest ? l0 : nlines; L < nlines; L += ls) {
        const double dL = (double)L;
        if ((ordered && !flags[L]) || !(fma(q1, dL, q0) > 0.0)) continue;
        const double p0 = fma(B[0], dL, A[0]), p1 = fma(B[1], dL, A[1]), p2 = fma(B[2], dL, A[2]);
        const float lf = factor(dL);
        acc[0] += line_walk(tab, img, rows, L, npix, p0, p1, lf);
        acc[1] += line_walk(tab, img, rows, L, npix, p1, p2, lf);
    }
}

// A CTA's 8 warps are 8 / LS blocks of 64 columns times LS line slices;
// blockIdx.z is the image.
template <typename TI, int MODE>
__global__ void __launch_bounds__(256, 4)
cell2t_kernel(const Geom2F f, const ViewTables vt, LineTable tab, const TI* __restrict__ img, void* __restrict__ sino,
              const int dto, const int nview, const float cw, const int LS) {
    __shared__ float red[8][2][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int nblk = 8 / LS, slice = wp / nblk;
    const int k = ((blockIdx.x * nblk + wp % nblk) * 32 + lane) * 2;
    const int v = blockIdx.y, b = blockIdx.z;
    const ViewHdr& h = vt.hdr[v];
    tab.q += b * line_table_entries(f.W, f.H);
    tab.flags += (size_t)b * (f.W + f.H);
    float acc[2] = {0.0f, 0.0f};
    if (k < f.Nu) cell2t_walk<MODE>(f, vt, h, v, k, cw, slice, LS, tab, img + (size_t)b * f.W * f.H, acc);
    if (LS > 1) {
        red[wp][0][lane] = acc[0];
        red[wp][1][lane] = acc[1];
        __syncthreads();
        if (slice) return;
        for (int s = 1; s < LS; ++s) {
            acc[0] += red[s * nblk + wp][0][lane];
            acc[1] += red[s * nblk + wp][1][lane];
        }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
        if (k + c < f.Nu) {
            const float scale = MODE == OP_A ? vt.colE[(size_t)v * f.Nu + k + c] : 1.0f;
            const int col = h.keep ? k + c : f.Nu - 1 - (k + c);
            st_dt(sino, dto, ((size_t)b * nview + v) * f.Nu + col, acc[c] * scale);
        }
}

// ----------------------------------------------------------- pixel gather

constexpr int P2 = 2;                  // pixels per side of a thread's block

// NB images' sinogram values of one column of one view.
template <typename TI, int NB>
struct SinoLanes {
    const TI* p;   // element 0 of the view (its first plane)
    size_t n;      // elements of a plane
    __device__ __forceinline__ Lanes<NB> operator()(int col) const {
        if constexpr (NB == 1) {
            Lanes<1> r;
            r.v[0] = ld(p + col);
            return r;
        } else {
            return ld_lanes<NB>(p, n, col);
        }
    }
};

// View v's contribution to the P2 x P2 pixels from (ix0, iy0), acc[row][column]
// (pixels past the image's edge are evaluated like the others; the caller
// drops them).  For every line of the block, the columns are merged with the
// run of P2 pixels in the line's pixel coordinates, relative to the run's
// start: each overlap is weighted with the line factor and cell scale (A^T) or
// the column width (B; times the FBP weight for Bw).  The run's first column is
// guessed in FP32 at its lower edge, low by the guess's error bound, and corrected
// against the tables, so the guess decides no result.  Its lower boundary is
// FP64; the next ones add the columns' FP32 widths on the line (columns wider
// than XR_WIDE2D: FP64 as well).
template <int MODE, int NB, bool USE_X, typename Src>
__device__ __forceinline__ void pix2d_axis(const Geom2F& f, const ViewTables& vt, const ViewHdr* h, const int keep,
                                           const int v, const int ix0, const int iy0, const float cw, const Src& src,
                                           float (&acc)[P2][P2][NB]) {
    const int Nu = f.Nu;
    const float4 hs = *reinterpret_cast<const float4*>(&h->sf);  // sin, cos, source
    const double q0 = h->q0, q1 = h->q1;
    const float dcx = h->dcx, dcy = h->dcy;
    const bool chain = MODE != OP_AT && vt.arc;
    const double* bA = vt.bA + (size_t)v * (Nu + 1);
    const double* bB = vt.bB + (size_t)v * (Nu + 1);
    const float4* wr = vt.colWR + (size_t)v * Nu;
    auto guess = [&](float x, float y) -> float {
        float u;
        if (f.type == GEO_FLAT) {
            u = (__fdividef(f.sod * (x * hs.y + y * hs.x), f.sod + x * hs.x - y * hs.y) - f.shu) * f.inv_du;
        } else if (f.type == GEO_ARC) {
            const float ex = x - hs.z, ey = y - hs.w;
            u = guess_atan2f(dcx * ey - dcy * ex, dcx * ex + dcy * ey) * f.inv_du;
        } else {
            u = (x * hs.y + y * hs.x - f.shu) * f.inv_du;
        }
        return keep ? f.half_nu + u : f.half_nu - u;
    };
    // (float32 boundary angles: half a unit of the view's own)
    const float margin = f.type == GEO_ARC ? fmaf(fabsf((float)h->beta) * 5.9604645e-8f, f.inv_du, f.guess) : f.guess;
    const int p0 = USE_X ? ix0 : f.H - P2 - iy0;  // first pixel of the runs
    const double dp = (double)p0;
#pragma unroll
    for (int j = 0; j < P2; ++j) {
        const int L = (USE_X ? iy0 : ix0) + j;
        const float Lf = (float)L;
        const double dL = (double)L;
        const float xa = USE_X ? fmaf((float)p0, f.dx, f.x0) : fmaf(Lf, f.dx, f.xc0);
        const float ya = USE_X ? fmaf(-Lf, f.dy, f.yc0) : fmaf((float)p0, f.dy, f.y0);
        float lf = cw, q = 1.0f;
        if (MODE == OP_AT || chain) q = (float)fma(q1, dL, q0);
        if (!(fma(q1, dL, q0) > 0.0)) continue;  // behind the source's plane
        if (MODE == OP_AT) lf = __fdividef(USE_X ? f.dx : f.dy, q);
        const float kf = guess(xa, ya) - margin;
        if (kf >= (float)Nu) continue;
        if (kf < 0.0f &&
            guess(USE_X ? fmaf((float)P2, f.dx, xa) : xa, USE_X ? ya : fmaf((float)P2, f.dy, ya)) + margin < 0.0f)
            continue;
        int k = (int)fminf(fmaxf(kf, 0.0f), (float)(Nu - 1));
        float pk0 = (float)(fma(bB[k], dL, bA[k]) - dp);
        while (pk0 > 0.0f && k > 0) {
            --k;
            pk0 = (float)(fma(bB[k], dL, bA[k]) - dp);
        }
        // pixel i of the run gains s: the block's pixel (row, column)
        auto gain = [&](int i, const Lanes<NB>& s) {
            const int r = USE_X ? j : P2 - 1 - i, c = USE_X ? i : j;
            float w = lf;
            if (MODE == OP_BW)
                w *= fbp_weight2d(f, hs.z, hs.w, fmaf((float)(ix0 + c), f.dx, f.xc0),
                                  fmaf(-(float)(iy0 + r), f.dy, f.yc0));
#pragma unroll
            for (int e = 0; e < NB; ++e) acc[r][c][e] = fmaf(w, s.v[e], acc[r][c][e]);
        };
        auto col_of = [&](int kk) { return XR_BOUND(keep ? kk : Nu - 1 - kk, 0, Nu - 1); };
        if (chain) {
            // arc detector: every pixel's columns walked with chained angles
            // from the column that holds its lower edge; pk0, pd are the
            // direct boundaries of column k, the widths those of the walk's
            // entries
            const float4* ea = vt.arc + 2 * (size_t)v * (Nu + 1);
            const float qd = q * (USE_X ? f.inv_dx : f.inv_dy);  // pixels per axis unit
            auto width = [&](int b) { const float4 a = ea[2 * b]; return fmaf(a.w, Lf, a.z); };
            float pd = pk0 + width(k + 1);
#pragma unroll
            for (int i = 0; i < P2; ++i) {
                const float e0 = (float)i, e1 = (float)(i + 1);
                while (!(pd > e0) && k < Nu - 1) {
                    ++k;
                    pk0 = pd;
                    pd += width(k + 1);
                }
                Lanes<NB> s = {};
                ArcChain ch;
                ch.start(ea, k, keep, f.du);
                float lo = fmaxf(e0, pk0), pj = pd, d = ch.next_linear(ea, k + 1);
                for (int kk = k;;) {
                    if (kk + 1 == Nu) d = fminf(d, 0.0f);  // the detector's end
                    const float pk1 = fmaf(d, qd, pj);
                    const float w = fminf(e1, pk1) - lo;
                    if (w > 0.0f) {
                        const Lanes<NB> y = src(col_of(kk));
#pragma unroll
                        for (int e = 0; e < NB; ++e) s.v[e] = fmaf(w, y.v[e], s.v[e]);
                    }
                    if (++kk >= Nu || pk1 >= e1) break;
                    lo = fmaxf(e0, pk1);
                    float wk;
                    d = ch.next_linear(ea, kk + 1, Lf, wk);
                    pj += wk;
                }
                gain(i, s);
            }
            continue;
        }
        float4 W;
        auto upper = [&](float lower) -> float {  // boundary k + 1 from boundary k
            W = wr[k];
            const float w = fmaf(W.y, Lf, W.x);
            return fabsf(w) < XR_WIDE2D ? lower + w : (float)(fma(bB[k + 1], dL, bA[k + 1]) - dp);
        };
        auto value = [&]() -> Lanes<NB> {
            Lanes<NB> y = src(col_of(k));
            if (MODE == OP_AT)
#pragma unroll
                for (int e = 0; e < NB; ++e) y.v[e] *= W.z;
            return y;
        };
        float pk1 = upper(pk0);
        while (!(pk1 > 0.0f) && k < Nu - 1) {
            ++k;
            pk0 = pk1;
            pk1 = upper(pk0);
        }
        Lanes<NB> y = value();
        float lo = fmaxf(0.0f, pk0);
#pragma unroll
        for (int i = 0; i < P2; ++i) {
            const float e1 = (float)(i + 1);
            Lanes<NB> s = {};
            while (pk1 < e1) {  // column k ends inside pixel i
                const float w = pk1 - lo;
                if (w > 0.0f)
#pragma unroll
                    for (int e = 0; e < NB; ++e) s.v[e] = fmaf(w, y.v[e], s.v[e]);
                lo = fmaxf(lo, pk1);
                if (++k < Nu) {
                    pk1 = upper(pk1);
                    y = value();
                } else {  // past the detector
                    pk1 = 3.0e38f;
                    y = {};
                }
            }
            const float w = e1 - lo;
            if (w > 0.0f)
#pragma unroll
                for (int e = 0; e < NB; ++e) s.v[e] = fmaf(w, y.v[e], s.v[e]);
            lo = fmaxf(lo, e1);
            gain(i, s);
        }
    }
}

template <int MODE, int NB, typename Src>
__device__ __forceinline__ void pix2d_view(const Geom2F& f, const ViewTables& vt, const int v, const int ix0,
                                           const int iy0, const float cw, const Src& src, float (&acc)[P2][P2][NB]) {
    const ViewHdr* h = vt.hdr + v;
    const int use_x = h->use_x, keep = h->keep;
    if (use_x) pix2d_axis<MODE, NB, true>(f, vt, h, keep, v, ix0, iy0, cw, src, acc);
    else pix2d_axis<MODE, NB, false>(f, vt, h, keep, v, ix0, iy0, cw, src, acc);
}

// A warp's 8 x 4 threads own a tile of 8 P2 x 4 P2 pixels.
__host__ __device__ inline int pix2d_tiles(int W, int H) {
    return ((W + 8 * P2 - 1) / (8 * P2)) * ((H + 4 * P2 - 1) / (4 * P2));
}

// A CTA's 8 warps are 8 / VS tiles times VS view slices.  NB = 1: the
// sinograms [batch][view][column] of type TI; NB > 1: their interleaved FP32
// copy.  blockIdx.y is the group of NB images.
// A^T of eight images held at 80 registers (three CTAs per SM; 126 unbound, 32
// bytes of spills): a batch of eight 512 x 512 slices, A + A^T, 1732 -> 1628 us
// when it came; B and Bw got slower that way (167 -> 190, 1235 -> 1266 us) and stay
// unbound.
template <typename TI, int NB, int MODE>
__global__ void __launch_bounds__(256, MODE == OP_AT && NB == 8 ? 3 : 1)
pix2d_kernel(const Geom2F f, const ViewTables vt, const TI* __restrict__ sino, void* __restrict__ img,
             const int dto, const int nview, const int b0, const int nbatch, const float cw, const float oscale,
             const int VS) {
    constexpr int NA = P2 * P2 * NB;
    __shared__ float red[8][NA][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int ntile = 8 / VS, slice = wp / ntile;
    const int tile = blockIdx.x * ntile + wp % ntile, tx = (f.W + 8 * P2 - 1) / (8 * P2);
    const int ix0 = ((tile % tx) * 8 + (lane & 7)) * P2, iy0 = ((tile / tx) * 4 + (lane >> 3)) * P2;
    const bool active = ix0 < f.W && iy0 < f.H;
    const size_t n = (size_t)nview * f.Nu;
    const TI* __restrict__ sb = sino + (size_t)blockIdx.y * n * NB;
    float acc[P2][P2][NB] = {};
    if (active)
        for (int v = slice; v < nview; v += VS) {
            const SinoLanes<TI, NB> src{sb + (size_t)v * f.Nu * (NB < 4 ? NB : 4), n};
            pix2d_view<MODE, NB>(f, vt, v, ix0, iy0, cw, src, acc);
        }
    float* a = &acc[0][0][0];
    if (VS > 1) {
#pragma unroll
        for (int e = 0; e < NA; ++e) red[wp][e][lane] = a[e];
        __syncthreads();
        if (slice) return;
        for (int s = 1; s < VS; ++s)
#pragma unroll
            for (int e = 0; e < NA; ++e) a[e] += red[s * ntile + wp][e][lane];
    }
    if (!active) return;
#pragma unroll
    for (int r = 0; r < P2; ++r)
#pragma unroll
        for (int c = 0; c < P2; ++c)
#pragma unroll
            for (int e = 0; e < NB; ++e) {
                const int b = b0 + blockIdx.y * NB + e, x = ix0 + c, y = iy0 + r;
                if (b < nbatch && x < f.W && y < f.H)
                    st_dt(img, dto, ((size_t)b * f.H + y) * f.W + x, acc[r][c][e] * oscale);
            }
}

// ------------------------------------------- pixel gather through row tables
//
// On line L of view v, the detector row integrated along the line up to pixel
// position x is, with x in column k,
//     S(x) = sum_{j < k} y_j (pos_{j+1} - pos_j) + y_k (x - pos_k),
// and pos_j = bA_j + bB_j L, so S(x) = QA_k + QB_k L + y_k x with
//     QA_k = sum_{j < k} y_j (bA_{j+1} - bA_j) - y_k bA_k,   QB_k likewise.
// A pixel's backprojection from the view is S(upper edge) - S(lower edge): one
// table entry and two FP64 FMAs per edge, whatever the number of columns, with
// no loop and no divergence.  S is FP64, of up to |y|max times the boundaries'
// positions in magnitude; rows whose smallest value a difference would lose 2^-18
// of (Spread::too_wide), and those holding an infinity or a NaN, are walked
// column by column instead (pix2d_view).  The column of an edge
// comes from an FP32 position; within that position's error bound of a boundary
// (row_eps, about 1e-4 to 1e-3 columns) the FP64 boundary decides.
//
// On the arc detector B and Bw walk each pixel's columns with float32 angles
// chained from its first column (ArcChain): boundary j inside the pixel lies
// delta_j = (t_j - angle_j) dD/dangle_j off its direct position, which adds
// delta_j (y_{j-1} - y_j) to the pixel; entry j carries angle_j and that
// factor.  A pixel with an edge so close to a boundary that its column is uncertain,
// or that the boundary may cross the edge by its offset, is walked (pixel_walk).
//
// Views whose column positions FP32 leaves uncertain by a quarter of a column
// are walked as well.
//
// Entries -1 .. Nu of a row are at [0 .. Nu + 1], in three arrays (a lane's
// neighbours then load neighbouring words): {QA, QB}, y, and on the arc
// detector {angle, dD/dangle (y_{j-1} - y_j)}.
struct RowTable {
    double2* q;
    float* y;
    float2* c;
    __host__ __device__ __forceinline__ RowTable at(size_t row, int Nu) const {
        const size_t o = row * (Nu + 2);
        return RowTable{q + o, y + o, c + o};
    }
};
constexpr size_t ROW_ENTRY_BYTES = sizeof(double2) + sizeof(float) + sizeof(float2);
constexpr int PT_MAX_BATCH = 4;

// Of a row: error bound of its view's column positions without the distance
// term (columns; ROW_WALK: the row is walked).  `steps` bounds the columns of a
// pixel where chained angles are walked (0: none): a boundary is then up to steps +
// 3 roundings off its direct angle.
constexpr float ROW_WALK = 2.0f;
__device__ __forceinline__ float row_eps(const Geom2F& f, const ViewHdr& h, float steps) {
    float q = 0.0f;
    if (f.type == GEO_ARC) {
        // half a unit of the largest angle: 2^-24 of its power of two
        const float a = fabsf((float)h.beta) + fabsf(f.shu) + f.half_nu * f.du;
        q = __int_as_float((__float_as_int(fmaxf(a, 1.0e-6f)) & 0x7f800000) - (24 << 23)) * f.inv_du;
        q *= 1.1f + (steps > 0.0f ? steps + 3.0f : 0.0f);
    }
    return f.epsw + q < 0.25f ? f.eps0 + q : ROW_WALK;
}

// The table of one detector row (the outer entries continue S as a
// constant), by a whole CTA of 256 threads; val(j)
// is the value of traversal column j.  Returns (to all threads) the row's error
// bound (row_eps).
template <typename Val>
__device__ __forceinline__ float build_row_table(const Geom2F& f, const ViewTables& vt, const int v, const RowTable e,
                                                 double2* sums, Val&& val) {
    const int Nu = f.Nu;
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    const double* bA = vt.bA + (size_t)v * (Nu + 1);
    const double* bB = vt.bB + (size_t)v * (Nu + 1);
    const float4* ea = vt.arc ? vt.arc + 2 * (size_t)v * (Nu + 1) : nullptr;
    const double nl = (double)(vt.hdr[v].nlines - 1);
    double ca = 0.0, cb = 0.0;  // sums over the columns before this round
    Spread spread;
    float reach = (float)(nl + 1.0);  // positions of pixels and boundaries, on the first and the last line
    float width = 3.0e38f;            // narrowest column there
    if (tid == 0) {
        e.q[0] = make_double2(0.0, 0.0);
        e.y[0] = 0.0f;
    }
    for (int base = 0; base <= Nu; base += 256) {
        const int j = base + tid;  // j == Nu: the entry past the end
        float y = 0.0f;
        double a = 0.0, b = 0.0, A = 0.0, B = 0.0;
        if (j <= Nu) {
            A = bA[j];
            B = bB[j];
            reach = fmaxf(reach, fmaxf(fabsf((float)A), fabsf((float)fma(B, nl, A))));
        }
        if (j < Nu) {
            y = val(j);
            spread.add(y);
            const double dA = bA[j + 1] - A, dB = bB[j + 1] - B;
            if (isfinite(y)) {
                a = (double)y * dA;
                b = (double)y * dB;
            }
            const double d1 = fma(dB, nl, dA);
            width = dA > 0.0 && d1 > 0.0 ? fminf(width, (float)fmin(dA, d1)) : 0.0f;
        }
        const double a0 = a, b0 = b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double ta = __shfl_up_sync(0xffffffffu, a, o), tb = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) { a += ta; b += tb; }
        }
        __syncthreads();  // the previous round's sums are read
        if (lane == 31) sums[wp] = make_double2(a, b);
        __syncthreads();
        double wa = ca, wb = cb;
        for (int w = 0; w < 8; ++w) {
            const double2 s = sums[w];
            if (w < wp) { wa += s.x; wb += s.y; }
            ca += s.x;
            cb += s.y;
        }
        if (j <= Nu) {
            e.q[j + 1] = make_double2(wa + (a - a0) - (double)y * A, wb + (b - b0) - (double)y * B);
            e.y[j + 1] = y;
            if (ea) {
                const float4 c = ea[2 * j];
                e.c[j + 1] = make_float2(c.x, c.y * ((j > 0 ? val(j - 1) : 0.0f) - y));
            }
        }
    }
    spread.warp();
    // boundaries out of order on a line (a ray past 90 degrees from the axis; lines
    // behind the source's plane): S would run back there
    if (!(width > 0.0f)) reach = __int_as_float(0x7f800000);
    const unsigned far = __reduce_max_sync(0xffffffffu, (unsigned)__float_as_int(reach));
    const unsigned thin = __reduce_min_sync(0xffffffffu, (unsigned)__float_as_int(fmaxf(width, 0.0f)));
    uint4* part = reinterpret_cast<uint4*>(sums);
    __syncthreads();  // the last round's sums are read
    if (lane == 0) part[wp] = make_uint4(spread.most, spread.least, far, thin);
    __syncthreads();
    unsigned r = 0u, t = 0xffffffffu;
    for (int w = 0; w < 8; ++w) {
        const uint4 p = part[w];
        spread.most = max(spread.most, p.x);
        spread.least = min(spread.least, p.y);
        r = max(r, p.z);
        t = min(t, p.w);
    }
    if (r >= 0x7f800000u || spread.too_wide(__int_as_float((int)r))) return ROW_WALK;
    return row_eps(f, vt.hdr[v], vt.arc ? 2.0f + 1.0f / __int_as_float((int)t) : 0.0f);
}

// View tables and row tables of one view per CTA, for all images of the batch.
template <typename TI, bool SCALE>
__global__ void __launch_bounds__(256)
table2d_kernel(const Geom g, const Geom2F f, const float* __restrict__ ang, const int nview, const ViewTables vt,
               const TI* __restrict__ sino, const int nbatch, const RowTable tab, float* __restrict__ eps) {
    __shared__ double2 sums[8];
    const int v = blockIdx.x, Nu = g.Nu;
    for (int k = threadIdx.x; k <= Nu; k += 256) setup_view_entry(g, 0, ang[v], v, k, vt, g.type == GEO_ARC);
    __syncthreads();
    const int keep = vt.hdr[v].keep;
    for (int b = 0; b < nbatch; ++b) {
        const size_t row = (size_t)b * nview + v;
        const TI* y = sino + row * Nu;
        const float e = build_row_table(f, vt, v, tab.at(row, Nu), sums, [&](int j) -> float {
            const float x = ld(y + (keep ? j : Nu - 1 - j));
            return SCALE ? x * vt.colE[(size_t)v * Nu + j] : x;
        });
        if (threadIdx.x == 0) eps[row] = e;
    }
}

// pix2d_view of one image, out of line: the rare path of pix2t_view.
template <int MODE, typename Src>
__device__ __noinline__ float4 pix2d_view_walk(const Geom2F& f, const ViewTables& vt, int v, int ix0, int iy0, float cw,
                                               const Src src) {
    float acc[P2][P2][1] = {};
    pix2d_view<MODE, 1>(f, vt, v, ix0, iy0, cw, src, acc);
    return make_float4(acc[0][0][0], acc[0][1][0], acc[1][0][0], acc[1][1][0]);
}

// View v's contribution to pixel (ix, iy) on the arc detector (B, Bw), its columns
// walked with chained angles as pix2d_axis walks them but with every direct
// boundary in FP64; y is the row's values, entry j + 1 that of column j.
template <int MODE>
__device__ __noinline__ float pixel_walk(const Geom2F& f, const ViewTables& vt, int v, int ix, int iy, float cw,
                                         const float* y) {
    const ViewHdr& h = vt.hdr[v];
    const int Nu = f.Nu, keep = h.keep, p = h.use_x ? ix : f.H - 1 - iy;
    const size_t ob = (size_t)v * (Nu + 1);
    const double dL = (double)(h.use_x ? iy : ix), dp = (double)p;
    auto pos = [&](int b) { return fma(vt.bB[ob + b], dL, vt.bA[ob + b]); };
    const float px = fmaf((float)ix, f.dx, f.xc0), py = fmaf(-(float)iy, f.dy, f.yc0);
    const float rx = px - h.sxr, ry = py - h.syr;
    const float u = guess_atan2f(h.dcx * ry - h.dcy * rx, h.dcx * rx + h.dcy * ry) * f.inv_du;
    int k = (int)fminf(fmaxf(f.half_nu + (keep ? u : -u), 0.0f), (float)(Nu - 1));
    while (k > 0 && pos(k) > dp) --k;
    while (k < Nu - 1 && pos(k + 1) <= dp) ++k;
    const float q = (float)fma(h.q1, dL, h.q0), qd = q * (h.use_x ? f.inv_dx : f.inv_dy);  // pixels per axis unit
    const float4* ea = vt.arc + 2 * ob;
    float s = 0.0f, lo = fmaxf(0.0f, (float)(pos(k) - dp));
    ArcChain ch;
    ch.start(ea, k, keep, f.du);
    for (; k < Nu && lo < 1.0f; ++k) {
        float d = ch.next_linear(ea, k + 1);
        if (k + 1 == Nu) d = fminf(d, 0.0f);  // the detector's end
        const float hi = fmaf(d, qd, (float)(pos(k + 1) - dp)), c = fminf(1.0f, hi) - lo;
        if (c > 0.0f) s = fmaf(c, y[k + 1], s);
        lo = fmaxf(lo, hi);
    }
    return s * (MODE == OP_BW ? cw * fbp_weight2d(f, h.sxr, h.syr, px, py) : cw);
}

// View v's contribution to a P2 x P2 block through its row table.  Both axes
// run the same code (line j, pixel i of its run), the sums are placed at the
// end.  CHAIN: chained boundary angles (B and Bw on the arc detector); returns the
// pixels left out (bit row P2 + column), which the caller walks: those with an edge
// within its position's error bound of a boundary, and those whose chained offsets
// may cross an edge.
template <int MODE, bool CHAIN>
__device__ __forceinline__ unsigned pix2t_view(const Geom2F& f, const ViewTables& vt, const int v, const int ix0,
                                           const int iy0, const float cw, const RowTable tab, const float eps,
                                           float (&acc)[P2][P2]) {
    const ViewHdr* h = vt.hdr + v;
    const int4 hi = *reinterpret_cast<const int4*>(&h->use_x);
    const float4 hs = *reinterpret_cast<const float4*>(&h->sf);  // sin, cos, source
    const bool use_x = hi.x != 0, keep = hi.y != 0;
    const int Nu = f.Nu;
    const int p0 = use_x ? ix0 : f.H - P2 - iy0, L0 = use_x ? iy0 : ix0;  // first pixel of the runs, first line
    // the runs' first edge, the step along a run and from line to line
    const float x0 = use_x ? fmaf((float)p0, f.dx, f.x0) : fmaf((float)L0, f.dx, f.xc0);
    const float y0 = use_x ? fmaf(-(float)L0, f.dy, f.yc0) : fmaf((float)p0, f.dy, f.y0);
    const float ex = use_x ? f.dx : 0.0f, ey = use_x ? 0.0f : f.dy;
    const float lx = use_x ? 0.0f : f.dx, ly = use_x ? -f.dy : 0.0f;
    // column coordinate, less a half = u sg + k0f
    const float sg = keep ? f.inv_du : -f.inv_du;
    const float k0f = f.half_nu - 0.5f - (f.type == GEO_ARC ? 0.0f : f.shu * sg);
    float t[P2][P2];
    unsigned walk = 0;  // pixels to walk, bit j P2 + i
#pragma unroll
    for (int j = 0; j < P2; ++j) {
        const double dL = (double)(L0 + j);
        const float xa = fmaf((float)j, lx, x0), ya = fmaf((float)j, ly, y0);
        double S[P2 + 1];
        int ki[P2 + 1];  // entry of each edge's column (0: before the first)
        float off[P2 + 1], lim = 0.5f;  // offset of each edge from its column's middle; above lim its column is uncertain
#pragma unroll
        for (int i = 0; i <= P2; ++i) {
            const float x = fmaf((float)i, ex, xa), y = fmaf((float)i, ey, ya);
            float u, inv = 0.0f;
            if (f.type == GEO_FLAT) {
                inv = rcp_fast(f.sod + x * hs.x - y * hs.y);
                u = f.sod * (x * hs.y + y * hs.x) * inv;
            } else if (f.type == GEO_ARC) {
                const float rx = x - hs.z, ry = y - hs.w;
                u = fine_atan2f(h->dcx * ry - h->dcy * rx, h->dcx * rx + h->dcy * ry, inv);
            } else {
                u = x * hs.y + y * hs.x;
            }
            if (i == 0) lim -= fmaf(f.eps1, inv, eps);
            // (a place outside the detector is as good as any there)
            const float kf = fminf(fmaxf(fmaf(u, sg, k0f), -1.0f), (float)Nu);
            // rounded by an add of 1.5 * 2^23: the column in the low bits
            const float tr = kf + 12582912.0f;
            ki[i] = XR_BOUND((__float_as_int(tr) - 0x4B400000) + 1, 0, Nu + 1);
            off[i] = kf - (tr - 12582912.0f);
        }
        bool near[P2 + 1];
#pragma unroll
        for (int i = 0; i <= P2; ++i) near[i] = fabsf(off[i]) > lim;
        if (!CHAIN && (near[0] || near[1] || near[2])) {
#pragma unroll
            for (int i = 0; i <= P2; ++i)
                if (near[i]) {  // boundary b decides
                    const int b = XR_BOUND(ki[i] - 1 + (off[i] > 0.0f), 0, Nu);
                    const size_t ob = (size_t)v * (Nu + 1) + b;
                    ki[i] = b + (fma(vt.bB[ob], dL, vt.bA[ob]) <= (double)(p0 + i));
                }
        }
#pragma unroll
        for (int i = 0; i <= P2; ++i) {
            const double2 q = tab.q[ki[i]];
            S[i] = fma((double)tab.y[ki[i]], (double)(p0 + i), fma(q.y, dL, q.x));
        }
        float lf = 1.0f;
        if (MODE == OP_AT || CHAIN) {
            const float q = (float)fma(h->q1, dL, h->q0);
            lf = MODE == OP_AT ? (use_x ? f.dx : f.dy) * rcp_fast(q) : q * (use_x ? f.inv_dx : f.inv_dy);
        }
#pragma unroll
        for (int i = 0; i < P2; ++i) {
            float s = (float)(S[i + 1] - S[i]);
            if (MODE == OP_AT) s *= lf;
            if (CHAIN) {
                // boundaries ka + 1 .. kb (entries ka + 2 ..) lie in the pixel;
                // the walk starts at column ka
                const int ka = max(ki[i] - 1, 0), kb = min(ki[i + 1] - 1, Nu);
                if (near[i] || near[i + 1]) {
                    s = 0.0f;
                    walk |= 1u << (use_x ? j * P2 + i : (P2 - 1 - i) * P2 + j);
                } else if (kb > ka) {
                    const float step = keep ? f.du : -f.du;
                    float a = keep ? tab.c[ka + 1].x : __fadd_rn(tab.c[ka + 2].x, f.du), corr = 0.0f;
                    for (int b = ka + 1; b <= kb; ++b) {
                        const float2 cb = tab.c[b + 1];
                        a = __fadd_rn(a, step);
                        float d = __fsub_rn(a, cb.x);
                        if (b == Nu) d = keep ? fminf(d, 0.0f) : fmaxf(d, 0.0f);  // the detector's end
                        corr = fmaf(d, cb.y, corr);
                    }
                    s = fmaf(corr, lf, s);
                }
            }
            t[j][i] = s;
        }
    }
#pragma unroll
    for (int r = 0; r < P2; ++r)
#pragma unroll
        for (int c = 0; c < P2; ++c) {
            const float s = use_x ? t[r][c] : t[c][P2 - 1 - r];
            float w = cw;
            if (MODE == OP_BW) {
                const float px = fmaf((float)(ix0 + c), f.dx, f.xc0), py = fmaf(-(float)(iy0 + r), f.dy, f.yc0);
                if (f.type == GEO_FLAT) {  // (R / (R - (s . p) / R))^2, s . p / R = -px sin + py cos
                    const float m = f.sod * rcp_fast(fmaf(px, hs.x, fmaf(-py, hs.y, f.sod)));
                    w *= m * m;
                } else if (f.type == GEO_ARC) {
                    const float wx = hs.z - px, wy = hs.w - py;
                    w *= rcp_fast(fmaf(wx, wx, wy * wy));
                }
            }
            acc[r][c] = MODE == OP_AT ? acc[r][c] + s : fmaf(w, s, acc[r][c]);
        }
    return walk;
}

// Views v0, v0 + vs, ... < nview of one block: row v's table and error bound at
// tab.at(v) and eps[v], its values as src(v) gives them.  The few pixels that a
// view leaves out are listed and walked together, every lane its own (walked at
// once, a warp would wait for one of them in most views of an arc scan: a ragged
// batch of 16 arc scans 14488 -> 12028 us).
template <int MODE, bool CHAIN, typename Src>
__device__ __forceinline__ void pix2t_views(const Geom2F& f, const ViewTables& vt, const RowTable tab, const float* eps,
                                            const int ix0, const int iy0, const float cw, const int v0, const int nview,
                                            const int vs, Src&& src, float (&acc)[P2][P2]) {
    constexpr int CAP = 16;
    unsigned list[CAP];
    int n = 0;
    auto flush = [&]() {
        for (int i = 0; i < n; ++i) {
            const int v = list[i] >> 2, r = (list[i] >> 1) & 1, c = list[i] & 1;
            const float s = pixel_walk<MODE>(f, vt, v, ix0 + c, iy0 + r, cw, tab.at(v, f.Nu).y);
#pragma unroll
            for (int e = 0; e < P2 * P2; ++e)
                if (e == (int)(list[i] & 3)) acc[e / P2][e % P2] += s;
        }
        n = 0;
    };
    for (int v = v0; v < nview; v += vs) {
        const float e = eps[v];
        if (e >= 1.0f) {
            const float4 s = pix2d_view_walk<MODE>(f, vt, v, ix0, iy0, cw, src(v));
            acc[0][0] += s.x; acc[0][1] += s.y; acc[1][0] += s.z; acc[1][1] += s.w;
            continue;
        }
        const unsigned left = pix2t_view<MODE, CHAIN>(f, vt, v, ix0, iy0, cw, tab.at(v, f.Nu), e, acc);
        if (CHAIN) {
            for (unsigned m = left; m; m &= m - 1) list[n++] = (unsigned)v << 2 | (unsigned)(__ffs(m) - 1);
            if (__any_sync(__activemask(), n > CAP - P2 * P2)) flush();
        }
    }
    if (CHAIN) flush();
}

// Tiles of a CTA: 2 x 4 warp tiles when its 8 warps share the views, else 8 /
// VS tiles side by side.
__host__ __device__ inline int pix2t_cta_x(int VS) { return VS == 1 ? 2 : 8 / VS; }
__host__ __device__ inline int pix2t_cta_y(int VS) { return VS == 1 ? 4 : 1; }
__host__ __device__ inline int pix2t_ctas(int W, int H, int VS) {
    const int tx = (W + 8 * P2 - 1) / (8 * P2), ty = (H + 4 * P2 - 1) / (4 * P2);
    return ((tx + pix2t_cta_x(VS) - 1) / pix2t_cta_x(VS)) * ((ty + pix2t_cta_y(VS) - 1) / pix2t_cta_y(VS));
}
// First pixel of this thread's block: warp tile wt of CTA tile `cta`.
__device__ __forceinline__ void pix2t_origin(const Geom2F& f, int VS, int cta, int wt, int lane, int& ix0, int& iy0) {
    const int cx = pix2t_cta_x(VS), cy = pix2t_cta_y(VS);
    const int tx = (f.W + 8 * P2 - 1) / (8 * P2), nx = (tx + cx - 1) / cx;
    ix0 = (((cta % nx) * cx + wt % cx) * 8 + (lane & 7)) * P2;
    iy0 = (((cta / nx) * cy + wt / cx) * 4 + (lane >> 3)) * P2;
}

// Slices of the views: VS warps of a CTA times the CTAs of a cluster along z.
// Warps of one CTA that share a view (VS = 1) also share its header and table
// in L1; the cluster's sums meet through distributed shared memory, in rank
// order.  blockIdx.y is the image.
template <typename TI, int MODE, bool CHAIN>
__global__ void __launch_bounds__(256, 4)
pix2t_kernel(const __grid_constant__ Geom2F f, const __grid_constant__ ViewTables vt, const RowTable tab,
             const float* __restrict__ eps, const TI* __restrict__ sino, void* __restrict__ img, const int dto,
             const int nview, const float cw, const float oscale, const int VS) {
    namespace cg = cooperative_groups;
    __shared__ float red[8][P2 * P2][32];
    cg::cluster_group cluster = cg::this_cluster();
    const int CS = gridDim.z, rank = blockIdx.z;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int ntile = 8 / VS, slice = wp / ntile + VS * rank;
    int ix0, iy0;
    pix2t_origin(f, VS, blockIdx.x, wp % ntile, lane, ix0, iy0);
    const size_t row0 = (size_t)blockIdx.y * nview;
    float acc[P2][P2] = {};
    if (ix0 < f.W && iy0 < f.H)
        pix2t_views<MODE, CHAIN>(f, vt, tab.at(row0, f.Nu), eps + row0, ix0, iy0, cw, slice, nview, VS * CS,
                                 [&](int v) { return SinoLanes<TI, 1>{sino + (row0 + v) * f.Nu, 0}; }, acc);
    float* a = &acc[0][0];
    auto store = [&](int wt, const float* sum) {
        int x0, y0;
        pix2t_origin(f, VS, blockIdx.x, wt, lane, x0, y0);
#pragma unroll
        for (int e = 0; e < P2 * P2; ++e) {
            const int x = x0 + e % P2, y = y0 + e / P2;
            if (x < f.W && y < f.H) st_dt(img, dto, ((size_t)blockIdx.y * f.H + y) * f.W + x, sum[e] * oscale);
        }
    };
    if (VS * CS == 1) {
        store(wp, a);
        return;
    }
#pragma unroll
    for (int e = 0; e < P2 * P2; ++e) red[wp][e][lane] = a[e];
    if (CS > 1) cluster.sync();
    else __syncthreads();
    // tile wt is finished by warp wt / CS of the CTA of rank wt % CS
    for (int wt = wp * CS + rank; wt < ntile; wt += 8 * CS) {
        float sum[P2 * P2] = {};
        for (int r = 0; r < CS; ++r) {
            const float* p = CS > 1 ? cluster.map_shared_rank(&red[0][0][0], r) : &red[0][0][0];
            for (int s = 0; s < VS; ++s)
#pragma unroll
                for (int e = 0; e < P2 * P2; ++e) sum[e] += p[((s * ntile + wt) * P2 * P2 + e) * 32 + lane];
        }
        store(wt, sum);
    }
    if (CS > 1) cluster.sync();  // the others still read this CTA's sums
}

}  // namespace xr
