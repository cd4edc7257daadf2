// spr_diff.cu -- differentiable rendering: a float per-sample composite of
// the draw list (forward) and its adjoint (backward).
//
// The coverage pipeline (fragments, sort, winding scan, merged sample masks,
// draw list) is the bit-exact one of spr_kernels.cu.  On top of it every
// sample is composited in linear float RGBA over a white background in
// painter's order, c' = f.rgb * a + c.rgb * (1 - a), c'.a = a * a + c.a *
// (1 - a) (the same blend as the multisample resolve, without the 8-bit
// sRGB storage), and a pixel is the mean of its samples.
//
// Spans cover every sample of a cell, so the spans between two fragments of a
// cell are one affine map: a first pass composes them, a lane per cell, and the
// passes over samples go through the cells' fragments only.
//
// Backward, per sample: a tape of the state before every fragment of the
// sample's cell is recorded in draw order and swept in reverse with the adjoint
// lambda of the state (lambda *= 1 - a through every covering item), giving the
// exact fill gradients (the spans' in a last pass, from two sums per run of
// them).  A path has up to millions of fragments and spans, whose shares of its fill
// gradient are added to memory one by one: in 64 bits, where their order and number
// do not show (in 32 bits the gradient of a path of 1,500 curves was off by 3e-6, ten
// times its shares' own rounding).  Geometry is
// differentiated by edge sampling: a pixel is taken as the mean over its S
// sample rows of the row integral of the composite, so moving the crossing
// x_c of a chord with sample row y_r by dx changes the pixel by
// (c_left - c_right) dx / S.  c_left - c_right is the jump of path k's
// coverage (from the exact winding on both sides of the crossing, the same
// chords, left masks and scanline winding the forward masks use) times
// lambda . (blend_k(c) - c) at the sample of that row.  The crossing moves
// with the chord's end points, which lie on cell lines (x = 2m or y = 2n,
// moving along the line as the curve moves) or at fixed curve parameters
// (curve ends and monotone split points), and so with the curve's control
// points.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "spr_device.cuh"
#include "spr_internal.h"

namespace spr {

namespace {

constexpr int kDiffThreads = 256;    // 8 warps, each working on its own cells
constexpr int kTileW = kBinW;  // columns of a resolve bin
// Items that a warp takes of a bin, at most, in the passes with a lane per cell.
// Forward and backward of 2,000 paths over 256 x 256, of 4,096 paths in one bin of
// 1024 x 1024 and of a batch of 16 scenes, us: a warp to a bin 8793, 3784 and 4514;
// 256 items 3902, 1634 and 4560; 128 items 3954, 1604 and 4507.
constexpr uint32_t kPartItems = 128;

__device__ __forceinline__ uint32_t pixel_mask(const uint4 &mm, int S, int k) {
    if (S == 32) return k == 0 ? mm.x : (k == 1 ? mm.y : (k == 2 ? mm.z : mm.w));
    if (S == 16) return ((k < 2 ? mm.x : mm.y) >> (16 * (k & 1))) & 0xFFFFu;
    return (mm.x >> (8 * k)) & 0xFFu;
}

// Words of a vertical row mask (vertical_mask / vertical_mask2) that hold the 2S
// stacked sample rows of a cell: the masks repeat them for both pixel columns.
template <int S>
constexpr int kRowWords = S == 32 ? 2 : 1;

// Bit r of the rows.  The word is picked by a select: r varies by lane, and a
// lane-dependent array index would put the masks in local memory.
template <int S>
__device__ __forceinline__ uint32_t row_bit(const uint32_t (&m)[kRowWords<S>], int r) {
    if constexpr (S == 32) return ((r < 32 ? m[0] : m[1]) >> (r & 31)) & 1u;
    else return (m[0] >> r) & 1u;
}

// Curve basis at t: P(t) = sum_j B[j] P_j, and P'(t).
__device__ __forceinline__ void curve_basis(const CurveGeom &g, float t, float *B, float &dx, float &dy) {
    const float u = 1.f - t;
    B[0] = B[1] = B[2] = B[3] = 0.f;
    if (g.type == kLinear) {
        B[0] = u;
        B[1] = t;
        dx = g.px[1] - g.px[0];
        dy = g.py[1] - g.py[0];
    } else if (g.type == kQuad) {
        B[0] = u * u;
        B[1] = 2.f * t * u;
        B[2] = t * t;
        dx = 2.f * (u * (g.px[1] - g.px[0]) + t * (g.px[2] - g.px[1]));
        dy = 2.f * (u * (g.py[1] - g.py[0]) + t * (g.py[2] - g.py[1]));
    } else if (g.type == kCubic) {
        B[0] = u * u * u;
        B[1] = 3.f * t * u * u;
        B[2] = 3.f * t * t * u;
        B[3] = t * t * t;
        dx = 3.f * (u * u * (g.px[1] - g.px[0]) + 2.f * t * u * (g.px[2] - g.px[1]) + t * t * (g.px[3] - g.px[2]));
        dy = 3.f * (u * u * (g.py[1] - g.py[0]) + 2.f * t * u * (g.py[2] - g.py[1]) + t * t * (g.py[3] - g.py[2]));
    } else {  // rational quadratic, weights (1, w, 1)
        const float w = g.w;
        const float b0 = u * u, b1 = 2.f * t * u * w, b2 = t * t;
        const float W = b0 + b1 + b2;
        const float iW = W != 0.f ? 1.f / W : 0.f;
        B[0] = b0 * iW;
        B[1] = b1 * iW;
        B[2] = b2 * iW;
        const float nx = b0 * g.px[0] + b1 * g.px[1] + b2 * g.px[2];
        const float ny = b0 * g.py[0] + b1 * g.py[1] + b2 * g.py[2];
        const float dnx = 2.f * (u * (w * g.px[1] - g.px[0]) + t * (g.px[2] - w * g.px[1]));
        const float dny = 2.f * (u * (w * g.py[1] - g.py[0]) + t * (g.py[2] - w * g.py[1]));
        const float dW = 2.f * (u * (w - 1.f) + t * (1.f - w));
        dx = (dnx - nx * iW * dW) * iW;
        dy = (dny - ny * iW * dW) * iW;
    }
}

// d(end point)/d(control point j) of a chord end at entry value ev (t bits
// | flags) as a 2x2 block per control point: dC[j] = (dCx/dPx, dCx/dPy,
// dCy/dPx, dCy/dPy).
__device__ __forceinline__ void end_point_jacobian(const CurveGeom &g, float t, uint32_t flags, bool fixed,
                                                   float4 *dC) {
    float B[4], dx, dy;
    curve_basis(g, t, B, dx, dy);
    int kind = 0;  // 0: fixed parameter, 1: on a vertical cell line, 2: on a horizontal one
    if (!fixed && !(flags & 2u)) kind = (flags & 1u) ? 2 : 1;
    if (kind == 1 && fabsf(dx) < 1e-12f) kind = 0;
    if (kind == 2 && fabsf(dy) < 1e-12f) kind = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float b = B[j];
        if (kind == 0) dC[j] = make_float4(b, 0.f, 0.f, b);
        else if (kind == 1) dC[j] = make_float4(0.f, 0.f, -(dy / dx) * b, b);
        else dC[j] = make_float4(b, -(dx / dy) * b, 0.f, 0.f);
    }
}

__device__ __forceinline__ bool filled(int w, int rule) { return rule == 0 ? (w & 0x7f) != 0 : (w & 1) != 0; }


__device__ __forceinline__ void load_curve(const CurveDesc &d, const float2 *__restrict__ tv, CurveGeom &g) {
    g.type = (int)(d.type & 0xFFu);
    g.w = g.type == kRational ? d.w : 0.f;
    const int n = g.type & 7;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 v = j < n ? tv[d.vpos + j] : make_float2(0.f, 0.f);
        g.px[j] = v.x;
        g.py[j] = v.y;
    }
}

// Warp sums of N values (a power of two): a reduce-scatter in which a lane
// keeps, at the exchange across lane bit O, the half of its partial sums that
// its side owns (M values), then plain butterflies over the remaining lane
// bits; value i ends in lane i * 32 / N, which stores it: there is no
// broadcast.  N + 4 - log2(N) shuffles instead of 5N.
template <int M, int O, int N>
__device__ __forceinline__ void reduce_scatter(float (&t)[N], int lane) {
    if constexpr (M >= 1) {
        const bool hi = (lane & O) != 0;
#pragma unroll
        for (int i = 0; i < M; ++i) {
            const float keep = hi ? t[M + i] : t[i];
            const float send = hi ? t[i] : t[M + i];
            t[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
        }
        reduce_scatter<M / 2, O / 2, N>(t, lane);
    } else {
#pragma unroll
        for (int o = O; o >= 1; o >>= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
    }
}

// Sum i of v over the warp, in the N lanes i * 32 / N (other lanes: no meaning).
template <int N>
__device__ __forceinline__ float scattered_sums(float (&v)[N], int lane) {
    reduce_scatter<N / 2, 16, N>(v, lane);
    return v[0];
}

// One fragment of a merged group, held by one lane of the cell's warp.
template <int S>
struct GroupFrag {
    float4 q;                    // chord in cell units: x0, y0, slope dx/dy (0 when horizontal), y1
    uint32_t vm[kRowWords<S>];   // rows between the chord's end points
    uint32_t lm[kRowWords<S>];   // left mask
    int chg;                     // winding change (0: no contribution)
    uint32_t raw;
};

template <int S>
__device__ __forceinline__ void load_group_frag(const DiffArgs &d, uint32_t raw, GroupFrag<S> &f) {
    constexpr int WORDS = S / 8;
    f.raw = raw;
    f.chg = (int32_t)d.pidw[raw] >> 30;
    const float4 c = d.chord[raw];
#pragma unroll
    for (int w = 0; w < kRowWords<S>; ++w) {
        f.vm[w] = d.vmask[(size_t)raw * WORDS + w];
        f.lm[w] = d.lmask[(size_t)raw * WORDS + w];
    }
    f.q = make_float4(c.x, c.y, c.w != c.y ? (c.z - c.x) / (c.w - c.y) : 0.f, c.w);
}

// What a warp reads of a merged group before its fragments: the winding before it,
// and lane l's entry and key of sorted position h + l.
struct GroupHead {
    int w0;
    uint32_t raw;
    uint64_t key;  // (no key past the last position)
};
__device__ __forceinline__ GroupHead group_head(const DiffArgs &d, int64_t h, int lane) {
    const bool in = h + lane < d.nf;
    return GroupHead{(int)__ldg(&d.wn_scan[h]), in ? __ldg(&d.perm[h + lane]) : 0u,
                     in ? __ldg(&d.skey[h + lane]) & kKeyMask : ~0ull};
}

// Chain of one fragment's crossings to its curve's control points: the
// crossings contribute sum dL/dx * ((1 - lam) dC0 + lam dC1) projected on x
// at fixed y, i.e. A * (dC0x - s dC0y) + B * (dC1x - s dC1y).
__device__ void fragment_chain(const FrameArgs &a, const DiffArgs &d, uint32_t raw, float slope, float A, float B) {
    const int2 e0 = d.entries[raw];
    const int2 e1 = (int64_t)raw + 1 < d.nf ? d.entries[raw + 1] : make_int2(-1, 0x3f800000);
    float t0 = ffrom((uint32_t)e0.y & 0xFFFFFFFCu), t1 = ffrom((uint32_t)e1.y & 0xFFFFFFFCu);
    if (t0 < 0.f) t0 = 0.f;
    if (t1 < 0.f) t1 = 0.f;
    const bool end1 = e0.x != e1.x;
    if (end1) t1 = 1.f;
    const CurveDesc cd = a.curves[e0.x];
    CurveGeom g;
    load_curve(cd, d.tvert, g);
    float4 dC0[4], dC1[4];
    end_point_jacobian(g, t0, (uint32_t)e0.y & 3u, t0 == 0.f || t0 == 1.f, dC0);
    end_point_jacobian(g, t1, end1 ? 0u : ((uint32_t)e1.y & 3u), end1 || t1 == 0.f || t1 == 1.f, dC1);
    const int n = g.type & 7;
    for (int k = 0; k < n; ++k) {
        const float gx = A * (dC0[k].x - slope * dC0[k].z) + B * (dC1[k].x - slope * dC1[k].z);
        const float gy = A * (dC0[k].y - slope * dC0[k].w) + B * (dC1[k].y - slope * dC1[k].w);
        atomicAdd(&d.grad_tvert[cd.vpos + k].x, gx);
        atomicAdd(&d.grad_tvert[cd.vpos + k].y, gy);
    }
}

// Edge-sampling adjoint of one merged group (a path's chords in one cell,
// sorted positions from h) for the cell's warp.  Lane l holds samples sub + 8k
// of cell pixel k4 = l >> 3 and J[k] = lambda . (blend(c) - c) of the path at
// those samples.  A chord crosses a sample row in one of the cell's two pixel
// columns, so lane l works on rows l (and l + 32 at 32 samples) of the cell and
// takes J at the crossing's pixel from the lane that holds it.  Groups are
// loaded 32 fragments at a time, one per lane, and broadcast by shuffles; every
// shuffle is executed by the whole warp.  Every fragment is in one group, so
// its sums have a place of their own (d.chain).
template <int S>
__device__ __forceinline__ void group_adjoint(const FrameArgs &a, const DiffArgs &d, int64_t h, const GroupHead &head,
                                              int rule, const float *J, int lane) {
    constexpr int SPT = S / 8, ROWS = 2 * S, RPL = (ROWS + 31) / 32;
    const int w0 = head.w0;
    uint32_t raw = head.raw;
    // the group's size: the run of equal keys from h
    const uint64_t kh = __shfl_sync(0xffffffffu, head.key, 0);
    uint64_t key = head.key;
    int gs = 0;
    for (;;) {
        const uint32_t ends = __ballot_sync(0xffffffffu, key != kh);
        if (ends) {
            gs += __ffs(ends) - 1;
            break;
        }
        gs += 32;
        key = h + gs + lane < d.nf ? d.skey[h + gs + lane] & kKeyMask : ~0ull;
    }
    float yr[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) yr[i] = ((float)(lane + 32 * i) + 0.5f) / (float)ROWS;
    for (int base = 0; base < gs; base += 32) {
        const int nw = min(32, gs - base);
        GroupFrag<S> mine{};
        if (lane < nw) {
            if (base > 0) raw = d.perm[h + base + lane];
            load_group_frag<S>(d, raw, mine);
        }
        for (int j = 0; j < nw; ++j) {
            const int chg = __shfl_sync(0xffffffffu, mine.chg, j);
            const float y0 = __shfl_sync(0xffffffffu, mine.q.y, j), y1 = __shfl_sync(0xffffffffu, mine.q.w, j);
            if (chg == 0 || y0 == y1) continue;  // uniform
            const float x0 = __shfl_sync(0xffffffffu, mine.q.x, j), slope = __shfl_sync(0xffffffffu, mine.q.z, j);
            uint32_t vm[kRowWords<S>];
#pragma unroll
            for (int w = 0; w < kRowWords<S>; ++w) vm[w] = __shfl_sync(0xffffffffu, mine.vm[w], j);
            float xc[RPL], Jr[RPL];
            int W[RPL];
            bool any = false;
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const int r = lane + 32 * i, py = r / S, s = r % S;  // row s of pixel row py
                xc[i] = x0 + (yr[i] - y0) * slope;
                const int pc = xc[i] * 2.f >= 1.f ? 1 : 0;  // the crossing's pixel column
                const int src = ((pc * 2 + py) & 3) * 8 + (s & 7);
                float v = 0.f;
#pragma unroll
                for (int k = 0; k < SPT; ++k) {
                    const float t = __shfl_sync(0xffffffffu, J[k], src);
                    v = (s >> 3) == k ? t : v;
                }
                Jr[i] = r < ROWS && row_bit<S>(vm, r & (ROWS - 1)) ? v : 0.f;
                W[i] = w0;
                any |= Jr[i] != 0.f;
            }
            if (!__any_sync(0xffffffffu, any)) continue;
            // winding just left of each crossing: this window by shuffles ...
            for (int j2 = 0; j2 < nw; ++j2) {
                const int chg2 = nw == 1 ? chg : __shfl_sync(0xffffffffu, mine.chg, j2);
                if (chg2 == 0) continue;  // uniform
                uint32_t vm2[kRowWords<S>], lm2[kRowWords<S>];
#pragma unroll
                for (int w = 0; w < kRowWords<S>; ++w) lm2[w] = __shfl_sync(0xffffffffu, mine.lm[w], j2);
                float x2 = 0.f, y2 = 0.f, s2 = 0.f;
                if (j2 != j) {  // uniform
                    x2 = __shfl_sync(0xffffffffu, mine.q.x, j2);
                    y2 = __shfl_sync(0xffffffffu, mine.q.y, j2);
                    s2 = __shfl_sync(0xffffffffu, mine.q.z, j2);
#pragma unroll
                    for (int w = 0; w < kRowWords<S>; ++w) vm2[w] = __shfl_sync(0xffffffffu, mine.vm[w], j2);
                }
#pragma unroll
                for (int i = 0; i < RPL; ++i) {
                    const int r = (lane + 32 * i) & (ROWS - 1);
                    uint32_t bit = row_bit<S>(lm2, r);
                    if (j2 != j && row_bit<S>(vm2, r)) bit ^= xc[i] > x2 + (yr[i] - y2) * s2 ? 1u : 0u;
                    W[i] += chg2 * (int)bit;
                }
            }
            // ... and the other windows of a group of more than 32 fragments from memory
            if (gs > 32 && any) {
                for (int j2 = 0; j2 < gs; ++j2) {
                    if (j2 >= base && j2 < base + nw) continue;
                    GroupFrag<S> f2;
                    load_group_frag<S>(d, d.perm[h + j2], f2);
                    if (f2.chg == 0) continue;
#pragma unroll
                    for (int i = 0; i < RPL; ++i) {
                        const int r = (lane + 32 * i) & (ROWS - 1);
                        uint32_t bit = row_bit<S>(f2.lm, r);
                        if (row_bit<S>(f2.vm, r)) bit ^= xc[i] > f2.q.x + (yr[i] - f2.q.y) * f2.q.z ? 1u : 0u;
                        W[i] += f2.chg * (int)bit;
                    }
                }
            }
            float sAB[2] = {0.f, 0.f};
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const bool cl = filled(W[i], rule), cr = filled(W[i] + chg, rule);
                if (Jr[i] == 0.f || cl == cr) continue;
                const float g = cl ? Jr[i] : -Jr[i];
                const float lam = (yr[i] - y0) / (y1 - y0);
                sAB[0] += g * (1.f - lam);
                sAB[1] += g * lam;
            }
            const float sum = scattered_sums<2>(sAB, lane);
            const uint32_t to = __shfl_sync(0xffffffffu, mine.raw, j);
            if ((lane & 15) == 0) reinterpret_cast<float *>(d.chain + to)[lane >> 4] = sum;
        }
    }
}

__device__ __forceinline__ uint4 load_merged(const uint32_t *merged, int words, uint32_t g) {
    if (words == 4) return reinterpret_cast<const uint4 *>(merged)[g];
    if (words == 2) {
        const uint2 v = reinterpret_cast<const uint2 *>(merged)[g];
        return make_uint4(v.x, v.y, 0u, 0u);
    }
    return make_uint4(merged[g], 0u, 0u, 0u);
}

// c -> a * c + b per channel.
struct Affine {
    float a;
    float4 b;
};

// The scene of resolve bin b: viewport, the bin index within the scene and
// the scene's first pixel (batch frames; a single scene otherwise).
struct BinScene {
    int W, H;
    uint32_t lb;
    int64_t image_off;
};
__device__ __forceinline__ BinScene bin_scene(const FrameArgs &a, uint32_t b) {
    BinScene r{a.W, a.H, b, 0};
    if (a.scenes != nullptr) {
        int lo = 0, hi = a.n_scenes - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.scenes[mid].bin_off <= b) lo = mid;
            else hi = mid - 1;
        }
        const SceneInfo *sc = a.scenes + lo;
        r.W = sc->W;
        r.H = sc->H;
        r.lb = b - sc->bin_off;
        r.image_off = sc->image_off;
    }
    return r;
}

// The items of the resolve pairs in bin order, one contiguous record each, and the
// parts of the bins that have more than kPartItems.
__global__ void k_diff_gather(DiffArgs d, int words, int64_t n_bins) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n_bins) {
        const uint32_t n = d.bend[p] - d.bstart[p];
        if (n > kPartItems) {
            const uint32_t parts = (n + kPartItems - 1) / kPartItems, at = atomicAdd(d.n_parts, parts);
            d.part_done[p] = 0u;
            for (uint32_t k = 0; k < parts; ++k) d.part[at + k] = make_uint2((uint32_t)p, k);
        }
    }
    if (p >= d.npairs) return;
    const uint32_t idx = d.pval[p];
    const int4 it = d.draw[idx];
    const uint32_t path = d.item_path[idx];
    // (a fragment is one cell wide: its length's place holds its group's first sorted position)
    d.bitem[p] = make_uint4((uint32_t)it.x, it.w != 0 ? d.heads[it.w - 1] : (uint32_t)it.y, (uint32_t)it.w, path);
    d.bfill[p] = d.fill[path];
    d.bmm[p] = it.w != 0 ? load_merged(d.merged, words, (uint32_t)it.w - 1u) : make_uint4(0u, 0u, 0u, 0u);
}

// The crossing sums of every fragment chained to its curve's control points, and
// the fill gradients from their sums.
__global__ void k_diff_chain(FrameArgs a, DiffArgs d) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 4 * (int64_t)a.P) reinterpret_cast<float *>(d.grad_fill)[i] = (float)d.fill_sum[i];
    if (i >= d.nf) return;
    const float2 r = d.chain[i];
    if (r.x == 0.f && r.y == 0.f) return;
    const float4 c = d.chord[i];
    fragment_chain(a, d, (uint32_t)i, (c.z - c.x) / (c.w - c.y), r.x, r.y);
}

// A bin of the passes with a lane per cell, or kPartItems items of a bin that has
// more, taken by a warp from a queue (the parts first).  Such a bin's parts are
// worked on by different warps: 2,000 paths over 256 x 256 have 3,300 items a bin
// and 512 bins, and a warp to each of them left most of the chip idle.
struct Unit {
    BinScene bs;
    uint32_t bin, part, parts;  // part of parts (one: the whole bin)
    uint32_t place;     // ... its place in the list of parts
    uint32_t beg, fin;  // its items
    uint32_t cell0;     // the first cell's number (bin * cells of a bin + column)
    int x0, y0, cells;  // its pixel; cells within the viewport
};
__device__ __forceinline__ bool next_unit(const FrameArgs &a, const DiffArgs &d, uint32_t n_parts, int lane, Unit &u) {
    uint32_t b, n;
    for (;;) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(d.queue, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        u.place = k;
        u.part = 0u;
        if (k < n_parts) {
            const uint2 e = __ldg(&d.part[k]);
            b = e.x;
            u.part = e.y;
        } else {
            if ((int64_t)(k - n_parts) >= a.n_bins) return false;
            b = k - n_parts;
        }
        u.beg = d.bstart[b];
        n = d.bend[b] - u.beg;
        if (k < n_parts || n <= kPartItems) break;
    }
    u.bin = b;
    u.parts = max((n + kPartItems - 1) / kPartItems, 1u);
    u.beg += u.part * kPartItems;
    u.fin = u.beg + min(n - u.part * kPartItems, kPartItems);
    u.bs = bin_scene(a, b);
    const int ntx = (u.bs.W + kTileW - 1) / kTileW, tile = (int)(u.bs.lb % ntx);
    u.cell0 = b * (kTileW / 2);
    u.x0 = tile * kTileW;
    u.y0 = (int)(u.bs.lb / ntx) * 2;
    u.cells = min(kTileW / 2, (u.bs.W - u.x0 + 1) / 2);
    return true;
}

// (The gathered items are read with __ldg: an earlier kernel wrote them, and the
// stores to the runs' maps and factors between the loads would otherwise keep
// them one after the other.)

// 32 of a bin's items, one per lane, for the passes with a lane per cell, which
// take them one by one through shuffles (a load at a time would leave a memory
// latency between them).  Column | length << 16 (a fragment: 0).
__device__ __forceinline__ uint32_t item_cols(const uint4 &it) {
    return (it.x & 0xFFFFu) | (it.z != 0u ? 0u : min(it.y, 0xFFFFu) << 16);
}
__device__ __forceinline__ float4 shfl_fill(const float4 &f, int q) {
    return make_float4(__shfl_sync(0xffffffffu, f.x, q), __shfl_sync(0xffffffffu, f.y, q),
                       __shfl_sync(0xffffffffu, f.z, q), __shfl_sync(0xffffffffu, f.w, q));
}
// An item of columns `cols` touches the cell at column x.
__device__ __forceinline__ bool touches(uint32_t cols, int x) {
    const int ix = (int)(cols & 0xFFFFu), len = (int)(cols >> 16);
    return len == 0 ? ix == x : (x >= ix && x < ix + len);
}

// A span: c -> fill * alpha + c * (1 - alpha), after the map `run`.
__device__ __forceinline__ void add_span(Affine &run, const float4 &f) {
    const float om = 1.f - f.w;
    run.b = make_float4(f.x * f.w + run.b.x * om, f.y * f.w + run.b.y * om, f.z * f.w + run.b.z * om,
                        f.w * f.w + run.b.w * om);
    run.a *= om;
}
// In place of a run's factor: the run holds no span.  Any value can be a factor
// (alpha has no range: the product of 1 - alpha goes below zero past alpha 1), so
// the mark is a NaN that no operation returns (theirs is 0x7FFFFFFF), told by its bits.
constexpr uint32_t kNoSpans = 0xFFFFFFFFu;
__device__ __forceinline__ bool no_spans(float ra) { return __float_as_uint(ra) == kNoSpans; }
__device__ __forceinline__ Affine empty_run() {
    return Affine{__uint_as_float(kNoSpans), make_float4(0.f, 0.f, 0.f, 0.f)};
}
// The run f, then the run g.
__device__ __forceinline__ Affine run_then(const Affine &f, const Affine &g) {
    if (no_spans(f.a)) return g;
    if (no_spans(g.a)) return f;
    return Affine{f.a * g.a, make_float4(g.a * f.b.x + g.b.x, g.a * f.b.y + g.b.y, g.a * f.b.z + g.b.z,
                                         g.a * f.b.w + g.b.w)};
}
constexpr uint32_t kNoFragment = 0xFFFFFFFFu;  // in place of a fragment's place: there is none ...
constexpr uint32_t kLaterFragment = 0xFFFFFFFEu;  // ... before, but the cell has some

// Fragment p follows fragment prev in their cell.
__device__ __forceinline__ void link(const DiffArgs &d, uint32_t prev, uint32_t p) {
    d.run_next[prev] = p;
    if (d.run_prev != nullptr) d.run_prev[p] = prev;
}

// First pass over a unit's items, a lane per cell (at column x).  A span covers
// every sample of a cell, so the spans between two fragments of a cell are one
// affine map of its samples' state: the map before each fragment goes to
// d.run_b / d.run_a at the fragment's place (a fragment is in one cell), with
// the places of the cell's next and (backward) previous fragments, the map after
// the last one is returned (no_spans(a): none).  ends: the cell's first and
// last fragment, if it has any (kNoFragment otherwise).
__device__ __forceinline__ Affine cell_runs(const DiffArgs &d, const Unit &u, bool active, int x, uint2 &ends) {
    const int lane = threadIdx.x & 31;
    Affine run = empty_run();
    ends = make_uint2(kNoFragment, kNoFragment);
    for (uint32_t base = u.beg; base < u.fin; base += 32) {
        const uint32_t mine = min(base + lane, u.fin - 1);
        const uint32_t my_cols = item_cols(__ldg(&d.bitem[mine]));
        const float4 my_fill = __ldg(&d.bfill[mine]);
        const int n = (int)min(u.fin - base, 32u);
        for (int q = 0; q < n; ++q) {
            const uint32_t cols = __shfl_sync(0xffffffffu, my_cols, q);
            const bool touch = active && touches(cols, x);
            if (cols >> 16) {  // (uniform) a span
                const float4 f = shfl_fill(my_fill, q);
                if (touch) {
                    if (no_spans(run.a)) run.a = 1.f;
                    add_span(run, f);
                }
            } else if (touch) {
                const uint32_t p = base + q;
                d.run_b[p] = run.b;
                d.run_a[p] = run.a;
                if (ends.x == kNoFragment) ends.x = p;
                else link(d, ends.y, p);
                ends.y = p;
                run = empty_run();
            }
        }
    }
    return run;
}

// A part of a bin is done: its cells' runs after their last fragments (of the whole
// part, where they have none) and their first and last fragments are left for the
// warp that finishes the bin's last part, which joins the parts' runs and links
// (true: as if it had gone through the whole bin; last, ends: the bin's).  For the
// adjoint's third pass it leaves each part the state that it starts from: the run
// and the last fragment before it, and the factor of the spans after it.
__device__ __forceinline__ bool join_parts(const DiffArgs &d, const Unit &u, int lane, Affine &last, uint2 &ends) {
    const size_t mine = (size_t)u.place * 32 + lane;
    d.part_b[mine] = last.b;
    d.part_a[mine] = last.a;
    d.part_ends[mine] = ends;
    __threadfence();
    __syncwarp();
    uint32_t done = 0;
    if (lane == 0) done = atomicAdd(&d.part_done[u.bin], 1u);
    if (__shfl_sync(0xffffffffu, done, 0) + 1u != u.parts) return false;
    __threadfence();
    // (written by other warps of this launch: read from L2)
    const size_t first = (size_t)(u.place - u.part) * 32 + lane;
    bool frags = false;
    if (d.part_pi != nullptr) {
        float pi = 1.f;
        for (uint32_t k = u.parts; k-- > 0;) {
            const size_t at = first + (size_t)k * 32;
            const uint2 e = __ldcg(&d.part_ends[at]);
            d.part_pi[at] = pi;
            if (e.x != kNoFragment) pi = 1.f, frags = true;
            const float f = e.x != kNoFragment ? __ldcg(&d.run_a[e.x]) : __ldcg(&d.part_a[at]);
            if (!no_spans(f)) pi *= f;
        }
    }
    last = empty_run();
    ends = make_uint2(kNoFragment, kNoFragment);
    for (uint32_t k = 0; k < u.parts; ++k) {
        const size_t at = first + (size_t)k * 32;
        const uint2 e = __ldcg(&d.part_ends[at]);
        const Affine run{__ldcg(&d.part_a[at]), __ldcg(&d.part_b[at])};
        if (d.part_pi != nullptr) {
            d.part_b[at] = last.b;
            d.part_a[at] = last.a;
            d.part_ends[at].x = ends.y != kNoFragment ? ends.y : (frags ? kLaterFragment : kNoFragment);
        }
        if (e.x == kNoFragment) {
            last = run_then(last, run);
            continue;
        }
        if (!no_spans(last.a)) {
            const Affine lead = run_then(last, Affine{__ldcg(&d.run_a[e.x]), __ldcg(&d.run_b[e.x])});
            d.run_b[e.x] = lead.b;
            d.run_a[e.x] = lead.a;
        }
        if (ends.x == kNoFragment) ends.x = e.x;
        else link(d, ends.y, e.x);
        ends.y = e.y;
        last = run;
    }
    return true;
}

template <int SPT>
__device__ __forceinline__ void apply_run(float4 (&c)[SPT], float ra, const float4 &rb) {
    if (no_spans(ra)) return;  // (uniform)
#pragma unroll
    for (int k = 0; k < SPT; ++k)
        c[k] = make_float4(ra * c[k].x + rb.x, ra * c[k].y + rb.y, ra * c[k].z + rb.z, ra * c[k].w + rb.w);
}

template <int S, int SPT>
__device__ __forceinline__ void apply_fragment(float4 (&c)[SPT], const float4 &f, uint32_t m, int sub) {
    const float om = 1.f - f.w;
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        if ((m >> (sub + 8 * k)) & 1u) {
            c[k].x = f.x * f.w + c[k].x * om;
            c[k].y = f.y * f.w + c[k].y * om;
            c[k].z = f.z * f.w + c[k].z * om;
            c[k].w = f.w * f.w + c[k].w * om;
        }
    }
}

__device__ __forceinline__ void store_pixel(const DiffArgs &d, int64_t pix, float4 v) {
    if (d.accumulate) {
        const float4 o = d.image[pix];
        v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
    }
    d.image[pix] = v;
}

// First pass of the composite and of its adjoint: the spans of every cell, a
// lane per cell (cell_runs).  Cells without fragments have one colour, which
// the forward writes at once; the others are listed for the second pass, with
// the map of their last run.
template <bool FORWARD>
__global__ void __launch_bounds__(kDiffThreads) k_diff_runs(FrameArgs a, DiffArgs d) {
    const int lane = threadIdx.x & 31;
    const uint32_t n_parts = *d.n_parts;
    Unit u;
    while (next_unit(a, d, n_parts, lane, u)) {
        const bool active = lane < u.cells;
        const int x = u.x0 + 2 * lane;
        uint2 ends;
        Affine last = cell_runs(d, u, active, x, ends);
        if (u.parts > 1u && !join_parts(d, u, lane, last, ends)) continue;
        const bool frags = ends.x != kNoFragment;
        if (FORWARD && active && !frags) {
            float4 c[1] = {make_float4(1.f, 1.f, 1.f, 1.f)};
            apply_run(c, last.a, last.b);
            const float s = d.out_scale;
            const float4 v = make_float4(c[0].x * s, c[0].y * s, c[0].z * s, c[0].w * s);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int X = x + (k >> 1), Y = u.y0 + (k & 1);
                if (X < u.bs.W && Y < u.bs.H) store_pixel(d, u.bs.image_off + (int64_t)Y * u.bs.W + X, v);
            }
        }
        const uint32_t cells = __ballot_sync(0xffffffffu, frags);
        uint32_t base = 0;
        if (lane == 0 && cells) base = atomicAdd(d.n_cells, (uint32_t)__popc(cells));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (frags) {
            d.cell[base + __popc(cells & ((1u << lane) - 1u))] = u.cell0 + lane;
            d.cell_ends[u.cell0 + lane] = ends;
            d.cell_b[u.cell0 + lane] = last.b;
            d.cell_a[u.cell0 + lane] = last.a;
        }
    }
}

// A cell of the second pass: warp = cell, lane l = pixel k4 = l >> 3 of the cell
// (k4 = px * 2 + py), samples (l & 7) + 8k.  Warps take a lot of cells at a time
// from the list: up to kCellBatch, fewer if every warp would get less than two such
// lots, and no more than hold kLotItems items on average (neighbouring cells are
// deep together: with lots of 8 cells the last warps of a scene of 29 items a cell
// worked on alone).  Forward and backward, us, at 8 cells / 2 cells / by the items:
// 5,000 paths over 700 x 700 at 8 samples 6174 / 5238 / 5086, 15,000 small paths
// over 700 x 700 3545 / 3399 / 3354, a batch of 16 scenes of few items a cell
// 4495 / 4780 / 4520.
constexpr uint32_t kCellBatch = 8;
constexpr uint32_t kLotItems = 32;
__device__ __forceinline__ uint32_t cell_lot(const DiffArgs &d, uint32_t n_cells) {
    const uint64_t by_items = (uint64_t)kLotItems * n_cells / (uint64_t)max(d.npairs, (int64_t)1);
    const uint32_t share = n_cells / (2u * gridDim.x * (kDiffThreads / 32));
    return max(min(min(share, kCellBatch), (uint32_t)min(by_items, (uint64_t)kCellBatch)), 1u);
}
struct Cell {
    uint32_t id, first, last;  // number, first and last fragment
    int64_t pix;  // this lane's pixel in the image
    bool valid;   // ... is inside the viewport
    uint32_t next, end;  // the warp's listed cells
    BinScene bs;         // of its bin
};
__device__ __forceinline__ bool next_cell(const FrameArgs &a, const DiffArgs &d, uint32_t n_cells, uint32_t lot, int lane,
                                          Cell &c) {
    if (c.next == c.end) {
        uint32_t k = 0;
        if (lane == 0) k = atomicAdd(d.cell_queue, lot);
        c.next = __shfl_sync(0xffffffffu, k, 0);
        if (c.next >= n_cells) return false;
        c.end = min(c.next + lot, n_cells);
    }
    const uint32_t id = d.cell[c.next++], b = id / (kTileW / 2);
    const uint2 ends = __ldg(&d.cell_ends[id]);
    if (c.id / (kTileW / 2) != b) c.bs = bin_scene(a, b);  // (a bin's cells are listed together)
    c.id = id;
    c.first = ends.x;
    c.last = ends.y;
    const int ntx = (c.bs.W + kTileW - 1) / kTileW;
    const int x = (int)(c.bs.lb % ntx) * kTileW + 2 * (int)(id % (kTileW / 2));  // its column
    const int X = x + (lane >> 4), Y = (int)(c.bs.lb / ntx) * 2 + ((lane >> 3) & 1);
    c.pix = c.bs.image_off + (int64_t)Y * c.bs.W + X;
    c.valid = X < c.bs.W && Y < c.bs.H;
    return true;
}

// The composite of the cells with fragments, through their fragments only.  With
// every cell walking all items of its bin, the spans composed over the lanes
// that held them, the composite of a 1024 x 1024 scene of 256 paths took 151 us
// and that of a batch of 16 scenes 1435; in these two passes 93 and 818, and with
// the cell's fragments linked instead of searched among its bin's items 633 on the
// batch.
template <int S>
__global__ void __launch_bounds__(kDiffThreads, 5) k_diff_forward(FrameArgs a, DiffArgs d) {
    constexpr int SPT = S / 8;
    const int lane = threadIdx.x & 31;
    const int k4 = lane >> 3, sub = lane & 7;
    const uint32_t n_cells = *d.n_cells, lot = cell_lot(d, n_cells);
    Cell cell{};
    cell.id = 0xFFFFFFFFu;
    while (next_cell(a, d, n_cells, lot, lane, cell)) {
        float4 c[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) c[k] = make_float4(1.f, 1.f, 1.f, 1.f);
        for (uint32_t p = cell.first;;) {
            const uint32_t next = p != cell.last ? __ldg(&d.run_next[p]) : p;
            apply_run(c, __ldg(&d.run_a[p]), __ldg(&d.run_b[p]));
            apply_fragment<S>(c, __ldg(&d.bfill[p]), pixel_mask(__ldg(&d.bmm[p]), S, k4), sub);
            if (p == cell.last) break;
            p = next;
        }
        apply_run(c, d.cell_a[cell.id], d.cell_b[cell.id]);
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            sum.x += c[k].x;
            sum.y += c[k].y;
            sum.z += c[k].z;
            sum.w += c[k].w;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
            sum.z += __shfl_xor_sync(0xffffffffu, sum.z, o);
            sum.w += __shfl_xor_sync(0xffffffffu, sum.w, o);
        }
        if (sub == 0 && cell.valid) {
            const float inv = d.out_scale / (float)S;
            store_pixel(d, cell.pix, make_float4(sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv));
        }
    }
}

// The adjoint of the cells with fragments: forward through the fragments, the
// samples' states before each to the tape, and in reverse with the samples'
// adjoints lambda, which gives the fragments' gradients and for every run of
// spans Lsum = sum lambda and Ksum = sum lambda * c_run (c_run the state where
// the run starts; of the first run, white, Lsum alone).  Bound by dependent
// loads and arithmetic at 6 warps a scheduler.  The adjoint with every cell
// walking all items of its bin twice took 505 us on a 1024 x 1024 scene of 256
// paths and 5120 on a batch of 16 scenes; in three passes 350 and 3240, and with
// the fragments linked and the sums stored by the lanes they end in 3010 on the
// batch (this kernel 2573 -> 2282).
template <int S>
__global__ void __launch_bounds__(kDiffThreads, 3) k_diff_backward(FrameArgs a, DiffArgs d) {
    constexpr int SPT = S / 8;
    const int lane = threadIdx.x & 31;
    const int k4 = lane >> 3, sub = lane & 7;
    const size_t wslot = (size_t)blockIdx.x * (kDiffThreads / 32) + (threadIdx.x >> 5);
    float4 *const tape = d.tape + wslot * (size_t)d.tape_depth * SPT * 32 + lane;  // slot e, k: [(e * SPT + k) * 32]
    const float inv = d.out_scale / (float)S;
    const uint32_t n_cells = *d.n_cells, lot = cell_lot(d, n_cells);
    Cell cell{};
    cell.id = 0xFFFFFFFFu;
    while (next_cell(a, d, n_cells, lot, lane, cell)) {
        float4 c[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) c[k] = make_float4(1.f, 1.f, 1.f, 1.f);
        int slot = 0;
        for (uint32_t p = cell.first;;) {
            const uint32_t next = p != cell.last ? __ldg(&d.run_next[p]) : p;
            apply_run(c, __ldg(&d.run_a[p]), __ldg(&d.run_b[p]));
            if (slot < d.tape_depth) {
#pragma unroll
                for (int k = 0; k < SPT; ++k) tape[((size_t)slot * SPT + k) * 32] = c[k];
            }
            ++slot;
            apply_fragment<S>(c, __ldg(&d.bfill[p]), pixel_mask(__ldg(&d.bmm[p]), S, k4), sub);
            if (p == cell.last) break;
            p = next;
        }
        if (slot > d.tape_depth) {
            if (lane == 0) atomicOr(d.status, 1u);
            continue;
        }
        const float4 G = cell.valid ? d.grad_image[cell.pix] : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 lam[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) lam[k] = make_float4(G.x * inv, G.y * inv, G.z * inv, G.w * inv);
        float ra = d.cell_a[cell.id];  // the run after the current fragment
        for (uint32_t p = cell.last;;) {
            const uint4 it = __ldg(&d.bitem[p]);
            const float4 f = __ldg(&d.bfill[p]);
            const float next_ra = __ldg(&d.run_a[p]);
            const uint32_t prev = p != cell.first ? __ldg(&d.run_prev[p]) : p;
            const uint32_t m = pixel_mask(__ldg(&d.bmm[p]), S, k4);
            // (the group's, on their way while the samples are worked on)
            const GroupHead head = group_head(d, (int64_t)it.y, lane);
            const float av = f.w, om = 1.f - av;
            --slot;
            float4 cb[SPT];
#pragma unroll
            for (int k = 0; k < SPT; ++k) cb[k] = tape[((size_t)slot * SPT + k) * 32];
            if (!no_spans(ra)) {  // (uniform) the run of spans that follows starts where the fragment ends
#pragma unroll
                for (int k = 0; k < SPT; ++k) c[k] = cb[k];
                apply_fragment<S>(c, f, m, sub);
                float lk[8] = {};
#pragma unroll
                for (int k = 0; k < SPT; ++k) {
                    lk[0] += lam[k].x;
                    lk[1] += lam[k].y;
                    lk[2] += lam[k].z;
                    lk[3] += lam[k].w;
                    lk[4] += lam[k].x * c[k].x;
                    lk[5] += lam[k].y * c[k].y;
                    lk[6] += lam[k].z * c[k].z;
                    lk[7] += lam[k].w * c[k].w;
                    lam[k] = make_float4(lam[k].x * ra, lam[k].y * ra, lam[k].z * ra, lam[k].w * ra);
                }
                const float sum = scattered_sums<8>(lk, lane);
                if ((lane & 3) == 0) reinterpret_cast<float *>(d.run_sum + 2 * (size_t)p)[lane >> 2] = sum;
            }
            float gf[4] = {0.f, 0.f, 0.f, 0.f};
            float J[SPT];
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                const float4 l = lam[k];
                J[k] = l.x * av * (f.x - cb[k].x) + l.y * av * (f.y - cb[k].y) + l.z * av * (f.z - cb[k].z) +
                       l.w * av * (av - cb[k].w);
                if ((m >> (sub + 8 * k)) & 1u) {
                    gf[0] += l.x * av;
                    gf[1] += l.y * av;
                    gf[2] += l.z * av;
                    gf[3] += l.x * (f.x - cb[k].x) + l.y * (f.y - cb[k].y) + l.z * (f.z - cb[k].z) +
                            l.w * (2.f * av - cb[k].w);
                    lam[k] = make_float4(l.x * om, l.y * om, l.z * om, l.w * om);
                }
            }
            group_adjoint<S>(a, d, (int64_t)it.y, head, a.fill_rule[it.w], J, lane);
            const float sum = scattered_sums<4>(gf, lane);
            if ((lane & 7) == 0 && sum != 0.f)
                atomicAdd(d.fill_sum + 4 * (size_t)it.w + (lane >> 3), (double)sum);
            ra = next_ra;
            if (p == cell.first) break;
            p = prev;
        }
        if (!no_spans(ra)) {  // the first run
            float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                s[0] += lam[k].x;
                s[1] += lam[k].y;
                s[2] += lam[k].z;
                s[3] += lam[k].w;
            }
            const float sum = scattered_sums<4>(s, lane);
            if ((lane & 7) == 0) reinterpret_cast<float *>(d.cell_sum + cell.id)[lane >> 3] = sum;
        }
    }
}

// Third pass of the adjoint: the spans' fill gradients, a lane per cell again.
// The adjoint inside a run is its end's times pi, the product of 1 - alpha of
// the run's later spans (found first, in reverse), so a span's gradient needs
// only its run's sums (c before the span = ra * c_run + rb); it is summed over
// the unit's cells before it goes to memory.
// The factors pi of 32 items and 32 cells are held in shared memory, and the first
// sweep, from the unit's end, leaves pi at the end of every 32 items there too: the
// forward sweep finds those of its 32 items again from it.  (A factor for every item
// and cell of the deepest bin, for every warp, took 2.5 GB for a bin of 4,096.)
__global__ void __launch_bounds__(kDiffThreads) k_diff_spans(FrameArgs a, DiffArgs d) {
    const int lane = threadIdx.x & 31;
    __shared__ float s_pi[kDiffThreads / 32][32][32];                // item, cell
    __shared__ float s_ends[kDiffThreads / 32][kPartItems / 32][32];  // 32 items, cell
    float(*const pis)[32] = s_pi[threadIdx.x >> 5], (*const pi_ends)[32] = s_ends[threadIdx.x >> 5];
    const uint32_t n_parts = *d.n_parts;
    Unit u;
    while (next_unit(a, d, n_parts, lane, u)) {
        if (u.fin == u.beg) continue;
        const bool active = lane < u.cells;
        const int x = u.x0 + 2 * lane;
        // the state that a part of a bin starts from
        uint32_t before = kNoFragment;  // the last fragment before it
        Affine run = empty_run();       // the spans since
        float pi = 1.f;
        if (u.parts > 1u) {
            const size_t at = (size_t)u.place * 32 + lane;
            before = d.part_ends[at].x;
            run = Affine{d.part_a[at], d.part_b[at]};
            pi = d.part_pi[at];
        }
        bool frags = before != kNoFragment;
        // pi before each of the 32 items from base on, given that after them
        auto sweep = [&](uint32_t base, float pi) {
            const uint32_t mine = min(base + lane, u.fin - 1);
            const uint32_t my_cols = item_cols(__ldg(&d.bitem[mine]));
            const float my_a = __ldg(&d.bfill[mine].w);
            for (int q = (int)min(u.fin - base, 32u) - 1; q >= 0; --q) {
                const uint32_t cols = __shfl_sync(0xffffffffu, my_cols, q);
                const float om = 1.f - __shfl_sync(0xffffffffu, my_a, q);
                if (!active || !touches(cols, x)) continue;
                if ((cols >> 16) == 0u) {
                    pi = 1.f;
                    frags = true;
                } else {
                    pis[q][lane] = pi;
                    pi *= om;
                }
            }
            return pi;
        };
        for (uint32_t base = u.beg + ((u.fin - u.beg - 1) & ~31u); base != u.beg; base -= 32) {
            pi_ends[(base - u.beg) / 32][lane] = pi;
            pi = sweep(base, pi);
        }
        sweep(u.beg, pi);
        // the sums of the cell's first run, whose samples start white (not
        // used if that run is empty); of a cell without fragments: the pixels'
        // adjoints
        float4 Ls = make_float4(0.f, 0.f, 0.f, 0.f), Ks;
        const bool inside = before < kLaterFragment;  // past a fragment: its run's sums
        if (inside) {
            Ls = d.run_sum[2 * (size_t)before];
            Ks = d.run_sum[2 * (size_t)before + 1];
        } else if (frags) {
            Ls = d.cell_sum[u.cell0 + lane];
        } else if (active) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int X = x + (k >> 1), Y = u.y0 + (k & 1);
                if (X < u.bs.W && Y < u.bs.H) {
                    const float4 G = d.grad_image[u.bs.image_off + (int64_t)Y * u.bs.W + X];
                    Ls = make_float4(Ls.x + G.x * d.out_scale, Ls.y + G.y * d.out_scale, Ls.z + G.z * d.out_scale,
                                     Ls.w + G.w * d.out_scale);
                }
            }
        }
        if (!inside) Ks = Ls;
        if (no_spans(run.a)) run.a = 1.f;
        for (uint32_t base = u.beg; base < u.fin; base += 32) {
            if (base != u.beg) sweep(base, pi_ends[(base - u.beg) / 32][lane]);
            const uint32_t mine = min(base + lane, u.fin - 1);
            const uint4 my_it = __ldg(&d.bitem[mine]);
            const uint32_t my_cols = item_cols(my_it);
            const float4 my_fill = __ldg(&d.bfill[mine]);
            const int n = (int)min(u.fin - base, 32u);
            for (int q0 = 0; q0 < n; q0 += 8) {  // 8 items' gradients of this cell, then summed over the cells together
                float v[32];
                bool any = false;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int q = q0 + j;
                    const uint32_t cols = __shfl_sync(0xffffffffu, my_cols, q);
                    const bool touch = active && q < n && touches(cols, x);
                    const size_t p = base + q;
                    v[4 * j] = v[4 * j + 1] = v[4 * j + 2] = v[4 * j + 3] = 0.f;
                    if ((cols >> 16) == 0u) {  // (uniform) a fragment
                        if (touch) {           // (its sums are not used where no span follows)
                            Ls = d.run_sum[2 * p];
                            Ks = d.run_sum[2 * p + 1];
                            run = Affine{1.f, make_float4(0.f, 0.f, 0.f, 0.f)};
                        }
                        continue;
                    }
                    const float4 f = shfl_fill(my_fill, q);
                    if (touch) {
                        any = true;
                        const float pl = pis[q][lane], av = f.w;
                        const float cx = run.a * Ks.x + run.b.x * Ls.x, cy = run.a * Ks.y + run.b.y * Ls.y;
                        const float cz = run.a * Ks.z + run.b.z * Ls.z, cw = run.a * Ks.w + run.b.w * Ls.w;
                        v[4 * j] = pl * av * Ls.x;
                        v[4 * j + 1] = pl * av * Ls.y;
                        v[4 * j + 2] = pl * av * Ls.z;
                        v[4 * j + 3] = pl * (Ls.x * f.x - cx + Ls.y * f.y - cy + Ls.z * f.z - cz + 2.f * av * Ls.w - cw);
                        add_span(run, f);
                    }
                }
                if (!__any_sync(0xffffffffu, any)) continue;
                reduce_scatter<16, 16, 32>(v, lane);  // lane i: the sum of value i
                const uint32_t path = __shfl_sync(0xffffffffu, my_it.w, min(q0 + (lane >> 2), 31));
                if (v[0] != 0.f) atomicAdd(d.fill_sum + 4 * (size_t)path + (lane & 3), (double)v[0]);
            }
        }
    }
}

// dL/d(transformed vertex) -> dL/d(input vertex) and dL/d(path affine),
// through k_transform's map (affine, 4x4 with the projective divide, the
// depth fold; the integer-x nudge has unit derivative).
__global__ void k_diff_vertex(FrameArgs a, const float2 *__restrict__ gt, const uint32_t *__restrict__ vmap,
                              float2 *__restrict__ gv, float *__restrict__ ga) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.V) return;
    const float2 g = gt[i];
    const float2 p = a.vertex[i];
    const uint32_t pid = a.vertex_pid[i];
    float xa = p.x, ya = p.y;
    float A[6] = {1.f, 0.f, 0.f, 1.f, 0.f, 0.f};
    if (a.affine) {
#pragma unroll
        for (int k = 0; k < 6; ++k) A[k] = a.affine[6 * (size_t)pid + k];
        xa = A[0] * p.x + A[2] * p.y + A[4];
        ya = A[1] * p.x + A[3] * p.y + A[5];
    }
    float m[16];
    int Wv = a.W, Hv = a.H;
    if (a.path_scene != nullptr) {
        const SceneInfo *sc = a.scenes + a.path_scene[pid];
#pragma unroll
        for (int k = 0; k < 16; ++k) m[k] = sc->m[k];
        Wv = sc->W;
        Hv = sc->H;
    } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) m[k] = a.m[k];
    }
    float ov[4], dox[4], doy[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        ov[r] = m[4 * r] * xa + m[4 * r + 1] * ya + m[4 * r + 3];
        dox[r] = m[4 * r];
        doy[r] = m[4 * r + 1];
    }
    float q[3], qx[3], qy[3];
    const float i3 = 1.f / ov[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        q[r] = ov[r] * i3;
        qx[r] = (dox[r] - q[r] * dox[3]) * i3;
        qy[r] = (doy[r] - q[r] * doy[3]) * i3;
    }
    const float w = (float)Wv, h = (float)Hv, z = (float)min(Wv, Hv);
    const float cutoff = -z * 0.5f;
    if (q[2] < cutoff) {
        q[2] = cutoff;
        qx[2] = qy[2] = 0.f;
    }
    const float den = q[2] + z, f = z / den;
    // d(out)/d(xa, ya): out.x = (q0 - w/2) f + w/2, out.y = (q1 - h/2) f + h/2
    const float fx = -f / den * qx[2], fy = -f / den * qy[2];
    const float Jxx = qx[0] * f + (q[0] - w * .5f) * fx, Jxy = qy[0] * f + (q[0] - w * .5f) * fy;
    const float Jyx = qx[1] * f + (q[1] - h * .5f) * fx, Jyy = qy[1] * f + (q[1] - h * .5f) * fy;
    const float gxa = Jxx * g.x + Jyx * g.y, gya = Jxy * g.x + Jyy * g.y;
    gv[vmap[i]] = make_float2(A[0] * gxa + A[1] * gya, A[2] * gxa + A[3] * gya);
    if (a.affine && ga && (gxa != 0.f || gya != 0.f)) {
        float *G = ga + 6 * (size_t)pid;
        atomicAdd(G + 0, gxa * p.x);
        atomicAdd(G + 1, gya * p.x);
        atomicAdd(G + 2, gxa * p.y);
        atomicAdd(G + 3, gya * p.y);
        atomicAdd(G + 4, gxa);
        atomicAdd(G + 5, gya);
    }
}

int diff_sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    }
    return n;
}

template <bool BWD>
int launch_diff(const FrameArgs &a, const DiffArgs &d, cudaStream_t s) {
    if (a.n_bins <= 0) return 0;
    cudaMemsetAsync(d.queue, 0, 4 * sizeof(uint32_t), s);  // (and the lists' lengths and the cells' queue after it)
    const unsigned grid = (unsigned)diff_blocks(a);
    int n = 2;
    if (d.npairs > 0) {
        k_diff_gather<<<(unsigned)((std::max(d.npairs, a.n_bins) + 255) / 256), 256, 0, s>>>(d, a.S / 8, a.n_bins);
        ++n;
    }
    // (a warp per bin, or part of one, as far as they are resident)
    const int64_t units = a.n_bins + diff_parts(d.npairs);
    const unsigned bin_grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((units + 7) / 8, 8 * (int64_t)diff_sm_count()));
    k_diff_runs<!BWD><<<bin_grid, kDiffThreads, 0, s>>>(a, d);
    // (the forward has no tape of its own per warp: as many blocks as are resident)
    const unsigned fwd_grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(a.n_bins * 4, 5 * (int64_t)diff_sm_count()));
    auto run = [&](auto fwd, auto bwd) {
        if (BWD) bwd<<<grid, kDiffThreads, 0, s>>>(a, d);
        else fwd<<<fwd_grid, kDiffThreads, 0, s>>>(a, d);
    };
    if (a.S == 8) run(k_diff_forward<8>, k_diff_backward<8>);
    else if (a.S == 16) run(k_diff_forward<16>, k_diff_backward<16>);
    else run(k_diff_forward<32>, k_diff_backward<32>);
    if (BWD) {
        cudaMemsetAsync(d.queue, 0, sizeof(uint32_t), s);
        k_diff_spans<<<bin_grid, kDiffThreads, 0, s>>>(a, d);
        ++n;
    }
    const int64_t chain = std::max<int64_t>(d.nf, 4 * (int64_t)a.P);
    if (BWD && chain > 0) {
        k_diff_chain<<<(unsigned)((chain + 255) / 256), 256, 0, s>>>(a, d);
        ++n;
    }
    return n;
}

}  // namespace

int64_t diff_blocks(const FrameArgs &a) {
    const int64_t units = a.n_bins * (kTileW / 2);
    const int64_t per_block = kDiffThreads / 32;
    return std::max<int64_t>(1, std::min<int64_t>((units + per_block - 1) / per_block, (int64_t)diff_sm_count() * 4));
}

int64_t diff_tape_words(const FrameArgs &a, int depth) {
    return diff_blocks(a) * (int64_t)depth * (a.S / 8) * kDiffThreads;
}

// (a bin of n > kPartItems items has fewer than 2 n / kPartItems parts)
int64_t diff_parts(int64_t npairs) { return npairs > kPartItems ? 2 * npairs / kPartItems : 0; }

__global__ void k_accumulate(float *__restrict__ dst, const float *__restrict__ src, int64_t n, int first) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = first ? src[i] : dst[i] + src[i];
}

int launch_accumulate(float *dst, const float *src, int64_t n, int first, cudaStream_t s) {
    if (n <= 0) return 0;
    k_accumulate<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dst, src, n, first);
    return 1;
}

int launch_diff_forward(const FrameArgs &a, const DiffArgs &d, cudaStream_t s) { return launch_diff<false>(a, d, s); }

int launch_diff_backward(const FrameArgs &a, const DiffArgs &d, cudaStream_t s) { return launch_diff<true>(a, d, s); }

int launch_diff_vertex(const FrameArgs &a, const float2 *grad_tvert, const uint32_t *vmap, float2 *grad_vertex,
                       float *grad_affine, cudaStream_t s) {
    if (a.V <= 0) return 0;
    k_diff_vertex<<<(unsigned)((a.V + 255) / 256), 256, 0, s>>>(a, grad_tvert, vmap, grad_vertex, grad_affine);
    return 1;
}

}  // namespace spr
