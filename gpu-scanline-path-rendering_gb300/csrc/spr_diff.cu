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
// Backward, per sample: a tape of the state before every draw item that
// touches the sample's cell is recorded in draw order and swept in reverse
// with the adjoint lambda of the state (lambda *= 1 - a through every
// covering item), giving the exact fill gradients.  Geometry is
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
constexpr int kDiffItemAcc = 128;    // items of a bin whose fill gradients a warp gathers in shared memory (backward)
constexpr int kTileW = kBinW;  // columns of a resolve bin

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

// Warp sums of N values (N = 2, 4, 8), returned to every lane: a
// reduce-scatter in which a lane keeps, at the exchange across lane bit O, the
// half of its partial sums that its side owns (M values), then plain
// butterflies over the remaining lane bits and one broadcast per value; value
// i ends in lane i * 32 / N.  2N + 4 - log2(N) shuffles instead of 5N.
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

template <int N>
__device__ __forceinline__ void warp_sums(float (&v)[N], int lane) {
    float t[N];
#pragma unroll
    for (int i = 0; i < N; ++i) t[i] = v[i];
    reduce_scatter<N / 2, 16, N>(t, lane);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __shfl_sync(0xffffffffu, t[0], i * (32 / N));
}

__device__ __forceinline__ float4 warp_sum4(float4 x, int lane) {
    float v[4] = {x.x, x.y, x.z, x.w};
    warp_sums<4>(v, lane);
    return make_float4(v[0], v[1], v[2], v[3]);
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
__device__ __forceinline__ void group_adjoint(const FrameArgs &a, const DiffArgs &d, int64_t h, int rule, const float *J, int lane) {
    constexpr int SPT = S / 8, ROWS = 2 * S, RPL = (ROWS + 31) / 32;
    const int w0 = (int)d.wn_scan[h];
    // the first 32 fragments, and the group's size: the run of equal keys from h
    const uint64_t kh = d.skey[h] & kKeyMask;
    uint32_t raw = h + lane < d.nf ? d.perm[h + lane] : 0u;
    int gs = 0;
    for (;;) {
        const int64_t j = h + gs + lane;
        const uint32_t ends = __ballot_sync(0xffffffffu, j >= d.nf || (d.skey[j] & kKeyMask) != kh);
        if (ends) {
            gs += __ffs(ends) - 1;
            break;
        }
        gs += 32;
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
            warp_sums<2>(sAB, lane);
            if (lane == j) d.chain[mine.raw] = make_float2(sAB[0], sAB[1]);
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

__device__ __forceinline__ void global_fill_grad(const DiffArgs &d, uint32_t path, float4 g) {
    atomicAdd(&d.grad_fill[path].x, g.x);
    atomicAdd(&d.grad_fill[path].y, g.y);
    atomicAdd(&d.grad_fill[path].z, g.z);
    atomicAdd(&d.grad_fill[path].w, g.w);
}

// c -> a * c + b per channel, and maps composed: `first`, then `t`.
struct Affine {
    float a;
    float4 b;
};
__device__ __forceinline__ Affine after(const Affine &first, const Affine &t) {
    return Affine{t.a * first.a, make_float4(t.a * first.b.x + t.b.x, t.a * first.b.y + t.b.y, t.a * first.b.z + t.b.z,
                                             t.a * first.b.w + t.b.w)};
}
// From `o` lanes below (UP), or from lane o.
template <bool UP>
__device__ __forceinline__ Affine shfl_affine(const Affine &t, int o) {
    auto get = [&](float v) { return UP ? __shfl_up_sync(0xffffffffu, v, o) : __shfl_sync(0xffffffffu, v, o); };
    return Affine{get(t.a), make_float4(get(t.b.x), get(t.b.y), get(t.b.z), get(t.b.w))};
}

// A fill gradient of item `idx` of the warp's bin (lanes that call it together
// have different items): into the item's accumulator, or, past those, straight
// to the global gradient.
__device__ __forceinline__ void add_fill_grad(const DiffArgs &d, float4 *acc, uint32_t idx, uint32_t path, float4 g) {
    if (idx < (uint32_t)kDiffItemAcc) {
        float4 v = acc[idx];
        v.x += g.x;
        v.y += g.y;
        v.z += g.z;
        v.w += g.w;
        acc[idx] = v;
    } else {
        global_fill_grad(d, path, g);
    }
}

// The accumulators of a bin's items [beg, fin) added to their paths' gradients
// and cleared.
__device__ __forceinline__ void flush_fill_grads(const DiffArgs &d, float4 *acc, uint32_t beg, uint32_t fin, int lane) {
    __syncwarp();
    for (uint32_t i = lane; i < min(fin - beg, (uint32_t)kDiffItemAcc); i += 32) {
        const float4 v = acc[i];
        if (v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f) {
            global_fill_grad(d, d.bitem[beg + i].w, v);
            acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __syncwarp();
}

// Tape slot (at most 65,536) and item of a record in one word; items past the
// accumulators need no number of their own.
__device__ __forceinline__ float slot_and_item(int slot, uint32_t item) {
    return __uint_as_float((uint32_t)slot | (min(item, 0xFFFFu) << 16));
}

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

// The items of the resolve pairs in bin order, one contiguous record each.
__global__ void k_diff_gather(DiffArgs d, int words) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= d.npairs) return;
    const uint32_t idx = d.pval[p];
    const int4 it = d.draw[idx];
    const uint32_t path = d.item_path[idx];
    // (a fragment is one cell wide: its length's place holds its group's first sorted position)
    d.bitem[p] = make_uint4((uint32_t)it.x, it.w != 0 ? d.heads[it.w - 1] : (uint32_t)it.y, (uint32_t)it.w, path);
    d.bfill[p] = d.fill[path];
    d.bmm[p] = it.w != 0 ? load_merged(d.merged, words, (uint32_t)it.w - 1u) : make_uint4(0u, 0u, 0u, 0u);
}

// The crossing sums of every fragment chained to its curve's control points.
__global__ void k_diff_chain(FrameArgs a, DiffArgs d) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.nf) return;
    const float2 r = d.chain[i];
    if (r.x == 0.f && r.y == 0.f) return;
    const float4 c = d.chord[i];
    fragment_chain(a, d, (uint32_t)i, (c.z - c.x) / (c.w - c.y), r.x, r.y);
}

// Persistent warps over units from a queue, 1 << unit_shift consecutive cells of
// a bin each: warp = one cell of a bin at a time, lane l = pixel k4 = l >> 3 of the cell (k4 = px * 2 + py), samples
// (l & 7) + 8k.  Every item touching a cell touches all its pixels, so the
// walk over the bin's items is warp-uniform; the items are read 32 at a time
// (one per lane), the touching ones found by a ballot and broadcast.  Warps
// never wait for one another.
template <int S, bool BWD>
__global__ void __launch_bounds__(kDiffThreads, 3) k_diff(FrameArgs a, DiffArgs d, int unit_shift) {
    constexpr int SPT = S / 8;
    constexpr int WORDS = S / 8;
    // fill-gradient accumulators of the warp's bin items: a warp's cells of one
    // bin share them, so a path costs one set of global atomics a unit
    __shared__ float4 s_acc[BWD ? kDiffThreads / 32 : 1][BWD ? kDiffItemAcc : 1];
    // the reverse sweep's next 32 records of each warp (held in registers they
    // would spill others)
    __shared__ float4 s_rec[BWD ? kDiffThreads / 32 : 1][BWD ? 3 : 1][BWD ? 32 : 1];
    const int lane = threadIdx.x & 31;
    const int k4 = lane >> 3, sub = lane & 7;
    const int px_in = k4 >> 1, py_in = k4 & 1;
    const size_t wslot = (size_t)blockIdx.x * (kDiffThreads / 32) + (threadIdx.x >> 5);
    float4 *const acc = s_acc[BWD ? threadIdx.x >> 5 : 0];
    if (BWD) {
        for (int i = lane; i < kDiffItemAcc; i += 32) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();
    }
    const int64_t n_units = a.n_bins * (kTileW / 2) >> unit_shift;
    // the unit's bin and the next cell of it
    BinScene bs{};
    int tile = 0, crow = 0, cw = 0, end = 0;
    uint32_t beg = 0, fin = 0;
    // the bin's items, 32 at a time (lane l holds item base + l); in the forward
    // a bin of one such chunk keeps it from cell to cell (the backward's reverse
    // sweep needs the registers)
    uint4 it = make_uint4(0u, 0u, 0u, 0u), my_mm = it;
    float4 my_fill = make_float4(0.f, 0.f, 0.f, 0.f);
    for (;;) {
        bool load = BWD || fin - beg > 32;
        if (cw == end) {
            if (BWD) flush_fill_grads(d, acc, beg, fin, lane);
            uint32_t u = 0;
            if (lane == 0) u = atomicAdd(d.queue, 1u);
            u = __shfl_sync(0xffffffffu, u, 0);
            if ((int64_t)u >= n_units) break;
            const uint32_t b = (u << unit_shift) / (kTileW / 2);
            bs = bin_scene(a, b);
            const int ntx = (bs.W + kTileW - 1) / kTileW;
            tile = (int)(bs.lb % ntx), crow = (int)(bs.lb / ntx);
            cw = (int)((u << unit_shift) % (kTileW / 2));
            end = min(cw + (1 << unit_shift), (bs.W - tile * kTileW + 1) / 2);  // (cells within the viewport)
            beg = fin = 0;
            if (cw >= end) {
                cw = end;
                continue;
            }
            beg = d.bstart[b], fin = d.bend[b];
            load = true;
        }
        const int cellx = tile * kTileW + 2 * cw++;
        const int X = cellx + px_in, Y = crow * 2 + py_in;
        const bool valid = X < bs.W && Y < bs.H;
        const int64_t pix = bs.image_off + (int64_t)Y * bs.W + X;
        float4 c[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) c[k] = make_float4(1.f, 1.f, 1.f, 1.f);
        // backward tape: ne item records; nsl sample-state slots (the state
        // before every fragment and at the start of every run of spans)
        int ne = 0, nsl = 0, run_slot = -1;
        float ralpha = 1.f;
        float4 rbeta = make_float4(0.f, 0.f, 0.f, 0.f);
        const size_t rbase = wslot * (size_t)d.tape_depth;
        for (uint32_t base = beg; base < fin; base += 32) {
            if ((load || base != beg) && base + lane < fin) {
                it = d.bitem[base + lane];
                my_fill = d.bfill[base + lane];
                my_mm = d.bmm[base + lane];
            }
            bool touch = false;
            if (base + lane < fin) {
                const int x = (int)(it.x & 0xFFFFu);
                touch = it.z != 0u ? x == cellx : (cellx >= x && cellx < x + (int)it.y);
            }
            uint32_t tm = __ballot_sync(0xffffffffu, touch);
            const uint32_t frags = __ballot_sync(0xffffffffu, touch && it.z != 0u);
            while (tm) {
                const int q = __ffs(tm) - 1;
                const uint32_t later = frags & tm;  // the touching fragments ahead
                if (!((frags >> q) & 1u)) {
                    // The spans up to the next fragment.  A span covers every
                    // sample of the cell, so a run of them is an affine map c =
                    // ralpha * c_run + rbeta of the samples' state c_run where
                    // the run starts; the maps are composed over the lanes that
                    // hold the spans, each lane getting the map before its own.
                    const uint32_t run = later ? tm & ((later & (0u - later)) - 1u) : tm;
                    tm &= ~run;
                    if (run_slot < 0) {
                        run_slot = nsl++;
                        ralpha = 1.f;
                        rbeta = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (BWD && run_slot < d.tape_depth) {
                            const size_t e = rbase + run_slot;
#pragma unroll
                            for (int k = 0; k < SPT; ++k) d.tape[(e * SPT + k) * 32 + lane] = c[k];
                        }
                    }
                    const bool mine = (run >> lane) & 1u;
                    Affine t = mine ? Affine{1.f - my_fill.w, make_float4(my_fill.x * my_fill.w, my_fill.y * my_fill.w,
                                                                         my_fill.z * my_fill.w, my_fill.w * my_fill.w)}
                                    : Affine{1.f, make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const Affine up = shfl_affine<true>(t, o);
                        if (lane >= o) t = after(up, t);
                    }
                    if (BWD) {
                        Affine ex = shfl_affine<true>(t, 1);
                        if (lane == 0) ex = Affine{1.f, make_float4(0.f, 0.f, 0.f, 0.f)};
                        ex = after(Affine{ralpha, rbeta}, ex);
                        const int e = ne + __popc(run & ((1u << lane) - 1u));
                        if (mine && e < d.tape_depth) {
                            float4 *rec = d.tape_rec + (rbase + e) * 3;
                            rec[0] = my_fill;
                            rec[1] = ex.b;
                            rec[2] = make_float4(ex.a, __uint_as_float(it.w), __uint_as_float(0u),
                                                 slot_and_item(run_slot, base - beg + lane));
                        } else if (mine) {
                            atomicOr(d.status, 1u);
                        }
                        ne += __popc(run);
                    }
                    const Affine all = after(Affine{ralpha, rbeta}, shfl_affine<false>(t, 31));
                    ralpha = all.a;
                    rbeta = all.b;
                    continue;
                }
                tm &= tm - 1u;
                float4 f;
                f.x = __shfl_sync(0xffffffffu, my_fill.x, q);
                f.y = __shfl_sync(0xffffffffu, my_fill.y, q);
                f.z = __shfl_sync(0xffffffffu, my_fill.z, q);
                f.w = __shfl_sync(0xffffffffu, my_fill.w, q);
                uint4 mm;
                mm.x = __shfl_sync(0xffffffffu, my_mm.x, q);
                mm.y = WORDS > 1 ? __shfl_sync(0xffffffffu, my_mm.y, q) : 0u;
                mm.z = WORDS > 2 ? __shfl_sync(0xffffffffu, my_mm.z, q) : 0u;
                mm.w = WORDS > 2 ? __shfl_sync(0xffffffffu, my_mm.w, q) : 0u;
                const uint32_t m = pixel_mask(mm, S, k4);
                const float om = 1.f - f.w;
                // the samples' states are materialized at fragments and at the end
                if (run_slot >= 0) {
#pragma unroll
                    for (int k = 0; k < SPT; ++k)
                        c[k] = make_float4(ralpha * c[k].x + rbeta.x, ralpha * c[k].y + rbeta.y,
                                           ralpha * c[k].z + rbeta.z, ralpha * c[k].w + rbeta.w);
                    run_slot = -1;
                }
                if (BWD) {
                    const int sidx = nsl++;
                    if (sidx < d.tape_depth) {
                        const size_t e = rbase + sidx;
#pragma unroll
                        for (int k = 0; k < SPT; ++k) d.tape[(e * SPT + k) * 32 + lane] = c[k];
                    }
                    if (lane == q) {  // (the lane that holds the item)
                        if (ne < d.tape_depth) {
                            // (a fragment needs no run state: its mask and its group's place)
                            float4 *rec = d.tape_rec + (rbase + ne) * 3;
                            rec[0] = my_fill;
                            rec[1] = make_float4(__uint_as_float(my_mm.x), __uint_as_float(my_mm.y),
                                                 __uint_as_float(my_mm.z), __uint_as_float(my_mm.w));
                            rec[2] = make_float4(__uint_as_float(it.y), __uint_as_float(it.w), __uint_as_float(it.z),
                                                 slot_and_item(sidx, base - beg + lane));
                        } else {
                            atomicOr(d.status, 1u);
                        }
                    }
                    ++ne;
                }
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
        }
        if (run_slot >= 0) {
#pragma unroll
            for (int k = 0; k < SPT; ++k)
                c[k] = make_float4(ralpha * c[k].x + rbeta.x, ralpha * c[k].y + rbeta.y, ralpha * c[k].z + rbeta.z,
                                   ralpha * c[k].w + rbeta.w);
        }
        if (!BWD) {
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
            if (valid && sub == 0) {
                const float inv = d.out_scale / (float)S;
                float4 v = make_float4(sum.x * inv, sum.y * inv, sum.z * inv, sum.w * inv);
                if (d.accumulate) {
                    const float4 o = d.image[pix];
                    v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
                }
                d.image[pix] = v;
            }
            continue;
        }
        // ---- reverse sweep (warp-uniform)
        if (ne > d.tape_depth || nsl > d.tape_depth) continue;
        const float inv = d.out_scale / (float)S;
        const float4 G = valid ? d.grad_image[pix] : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 lam[SPT];
#pragma unroll
        for (int k = 0; k < SPT; ++k) lam[k] = make_float4(G.x * inv, G.y * inv, G.z * inv, G.w * inv);
        int cur_slot = -1;  // run being swept (its start slot), -1 outside runs
        float pi = 1.f;
        float4 Lsum = make_float4(0.f, 0.f, 0.f, 0.f), Ksum = Lsum;
        float4(*const rec_s)[BWD ? 32 : 1] = s_rec[BWD ? threadIdx.x >> 5 : 0];  // record e_hi - l at l
        __syncwarp();  // (records written by their items' lanes)
        for (int e0 = ne - 1, e_hi = ne + 31; e0 >= 0;) {
            if (e_hi - e0 >= 32) {  // the next 32 records
                __syncwarp();
                e_hi = e0;
                if (e0 - lane >= 0) {
                    const float4 *rec = d.tape_rec + (rbase + e0 - lane) * 3;
#pragma unroll
                    for (int i = 0; i < 3; ++i) rec_s[i][lane] = rec[i];
                }
                __syncwarp();
            }
            const int jl = e_hi - e0;
            const float4 r2 = rec_s[2][jl];
            const uint32_t w = __float_as_uint(r2.z), si = __float_as_uint(r2.w);
            const int sidx = (int)(si & 0xFFFFu);
            if (w == 0u) {
                // A run of spans, in the lanes that hold them: every sample is
                // covered, so inside the run the samples' adjoints are the run
                // end's times the scalar pi (the product of 1 - a of the later
                // spans), and the fill gradients need only the run's sums Lsum =
                // sum lambda and Ksum = sum lambda * c_run (c before the span =
                // ra * c_run + rb).
                if (sidx != cur_slot) {
                    if (cur_slot >= 0) {
#pragma unroll
                        for (int k = 0; k < SPT; ++k)
                            lam[k] = make_float4(lam[k].x * pi, lam[k].y * pi, lam[k].z * pi, lam[k].w * pi);
                    }
                    const size_t es = rbase + sidx;
                    float4 ls = make_float4(0.f, 0.f, 0.f, 0.f), ks = ls;
#pragma unroll
                    for (int k = 0; k < SPT; ++k) {
                        const float4 cr = d.tape[(es * SPT + k) * 32 + lane];
                        ls.x += lam[k].x;
                        ls.y += lam[k].y;
                        ls.z += lam[k].z;
                        ls.w += lam[k].w;
                        ks.x += lam[k].x * cr.x;
                        ks.y += lam[k].y * cr.y;
                        ks.z += lam[k].z * cr.z;
                        ks.w += lam[k].w * cr.w;
                    }
                    float lk[8] = {ls.x, ls.y, ls.z, ls.w, ks.x, ks.y, ks.z, ks.w};
                    warp_sums<8>(lk, lane);
                    Lsum = make_float4(lk[0], lk[1], lk[2], lk[3]);
                    Ksum = make_float4(lk[4], lk[5], lk[6], lk[7]);
                    cur_slot = sidx;
                    pi = 1.f;
                }
                // the run's records among the loaded ones: lanes [jl, jl + R)
                const float4 rf = rec_s[0][lane], rbb = rec_s[1][lane], rr2 = rec_s[2][lane];
                const uint32_t of_run = __ballot_sync(0xffffffffu, e_hi - lane >= 0 && __float_as_uint(rr2.z) == 0u &&
                                                                       (int)(__float_as_uint(rr2.w) & 0xFFFFu) == sidx) >>
                                         jl;
                const int R = of_run == 0xFFFFFFFFu ? 32 : __ffs((int)~of_run) - 1;
                const bool mine = lane >= jl && lane < jl + R;
                float p = mine ? 1.f - rf.w : 1.f;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float up = __shfl_up_sync(0xffffffffu, p, o);
                    if (lane >= o) p *= up;
                }
                float pl = __shfl_up_sync(0xffffffffu, p, 1);
                pl = lane == 0 ? pi : pi * pl;
                const float av = rf.w, ra = rr2.x;
                const float cx = ra * Ksum.x + rbb.x * Lsum.x, cy = ra * Ksum.y + rbb.y * Lsum.y;
                const float cz = ra * Ksum.z + rbb.z * Lsum.z, cw = ra * Ksum.w + rbb.w * Lsum.w;
                const float4 gf = make_float4(
                    pl * av * Lsum.x, pl * av * Lsum.y, pl * av * Lsum.z,
                    pl * (Lsum.x * rf.x - cx + Lsum.y * rf.y - cy + Lsum.z * rf.z - cz + 2.f * av * Lsum.w - cw));
                if (mine && (gf.x != 0.f || gf.y != 0.f || gf.z != 0.f || gf.w != 0.f))
                    add_fill_grad(d, acc, __float_as_uint(rr2.w) >> 16, __float_as_uint(rr2.y), gf);
                __syncwarp();
                pi *= __shfl_sync(0xffffffffu, p, 31);
                e0 -= R;
                continue;
            }
            --e0;
            const float4 f = rec_s[0][jl], rb = rec_s[1][jl];
            const uint32_t head = __float_as_uint(r2.x), path = __float_as_uint(r2.y);
            const float av = f.w, om = 1.f - av;
            // fragment: per-sample coverage; first close a pending run
            if (cur_slot >= 0) {
#pragma unroll
                for (int k = 0; k < SPT; ++k)
                    lam[k] = make_float4(lam[k].x * pi, lam[k].y * pi, lam[k].z * pi, lam[k].w * pi);
                cur_slot = -1;
            }
            Lsum = Ksum = make_float4(0.f, 0.f, 0.f, 0.f);  // (of the closed run: not kept)
            const uint32_t m = pixel_mask(make_uint4(__float_as_uint(rb.x), __float_as_uint(rb.y), __float_as_uint(rb.z),
                                                     __float_as_uint(rb.w)),
                                          S, k4);
            const size_t es = rbase + sidx;
            float4 gf = make_float4(0.f, 0.f, 0.f, 0.f);
            float J[SPT];
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                const float4 cb = d.tape[(es * SPT + k) * 32 + lane];
                const float4 l = lam[k];
                J[k] = l.x * av * (f.x - cb.x) + l.y * av * (f.y - cb.y) + l.z * av * (f.z - cb.z) +
                       l.w * av * (av - cb.w);
                if ((m >> (sub + 8 * k)) & 1u) {
                    gf.x += l.x * av;
                    gf.y += l.y * av;
                    gf.z += l.z * av;
                    gf.w += l.x * (f.x - cb.x) + l.y * (f.y - cb.y) + l.z * (f.z - cb.z) + l.w * (2.f * av - cb.w);
                    lam[k] = make_float4(l.x * om, l.y * om, l.z * om, l.w * om);
                }
            }
            group_adjoint<S>(a, d, (int64_t)head, a.fill_rule[path], J, lane);
            gf = warp_sum4(gf, lane);
            if (lane == 0 && (gf.x != 0.f || gf.y != 0.f || gf.z != 0.f || gf.w != 0.f))
                add_fill_grad(d, acc, si >> 16, path, gf);
            __syncwarp();
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

template <int S, bool BWD>
void run_diff(const FrameArgs &a, const DiffArgs &d, unsigned grid, cudaStream_t s) {
    // units of up to a bin's 32 cells, at least 4 for every warp
    int shift = 5;
    while (shift > 0 && (a.n_bins * (kTileW / 2) >> shift) < 4 * (int64_t)grid * (kDiffThreads / 32)) --shift;
    k_diff<S, BWD><<<grid, kDiffThreads, 0, s>>>(a, d, shift);
}

template <bool BWD>
int launch_diff(const FrameArgs &a, const DiffArgs &d, cudaStream_t s) {
    if (a.n_bins <= 0) return 0;
    cudaMemsetAsync(d.queue, 0, sizeof(uint32_t), s);
    const unsigned grid = (unsigned)diff_blocks(a);
    int n = 1;
    if (d.npairs > 0) {
        k_diff_gather<<<(unsigned)((d.npairs + 255) / 256), 256, 0, s>>>(d, a.S / 8);
        ++n;
    }
    if (a.S == 8) run_diff<8, BWD>(a, d, grid, s);
    else if (a.S == 16) run_diff<16, BWD>(a, d, grid, s);
    else run_diff<32, BWD>(a, d, grid, s);
    if (BWD && d.nf > 0) {
        k_diff_chain<<<(unsigned)((d.nf + 255) / 256), 256, 0, s>>>(a, d);
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

int64_t diff_tape_rec_words(const FrameArgs &a, int depth) {
    return diff_blocks(a) * (int64_t)(kDiffThreads / 32) * depth * 3;
}

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
