// spr_kernels.cu -- the scanline fill pipeline on sm_103a.
//
// Stage map (reference function -> kernel here):
//   k_transformVertex (cu:36-105)                    -> k_transform
//   k_make_intersection_0 + escan (ras_cut.h:1254)   -> k_curve_count + scan
//   k_make_intersection_1 (ras_cut.h:1484)           -> k_curve_emit
//   k_gen_fragment_and_stencil_mask (cu:112-441)     -> k_fragment
//   cuda_seg_sort_int_by_int (cuda_sort.cu:12)       -> k_segment_sort(_small), radix_sort
//                                                       (spr_sort.cu)
//   k_shuffleFragments + int8 scan (cu:444, 1099),
//   k_mark_merged_fragment_and_span + scans,
//   k_gen_gl_merged_fragment_and_span (cu:444-868)   -> k_scan_mark (one look-back pass)
//   k_gen_stencil_cuda_sm + block boundary (cu:554)  -> k_stencil
//   OpenGL draw + multisample resolve (cu:1312-1433) -> bin counts (k_scan_mark),
//                                                       k_scan_lb, k_bin_scatter,
//                                                       k_bin_sort, k_resolve
// ("cu" = gpu-scanline/src/rasterizer/R_cut_A_mask_comb_scanline/ras_cut_mask_comb_scanline.cu)

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "spr_device.cuh"
#include "spr_internal.h"
#include "spr_lookback.cuh"

namespace spr {

namespace {

constexpr int kThreads = 256;

inline uint32_t cap32(int64_t cap) { return (uint32_t)std::min<int64_t>(cap, INT32_MAX); }
inline unsigned grid_for(int64_t n, int t = kThreads) { return (unsigned)((n + t - 1) / t); }

// Viewport of the scene that path pid belongs to.
struct Dim {
    int W, H;
};
__device__ __forceinline__ Dim dim_of(const FrameArgs &a, uint32_t pid) {
    if (a.path_scene == nullptr) return Dim{a.W, a.H};
    const SceneInfo *sc = a.scenes + __ldg(a.path_scene + pid);
    return Dim{sc->W, sc->H};
}

// Admission of a size by the first kernel that uses it: *admitted = *need if
// it fits cap and no scan gave up before, else 0 and kStatusOverflow.  Every
// block takes the same decision (the timeout bit was set by earlier kernels
// only) and block 0 records it.
__device__ __forceinline__ bool admit(const uint32_t *need, uint32_t *admitted, uint32_t cap, uint32_t *status) {
    const uint32_t n = *need, st = *status & kStatusTimeout;
    const bool ok = n <= cap && st == 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *admitted = ok ? n : 0u;
        if (!ok) atomicOr(status, kStatusOverflow);
    }
    return ok;
}

__device__ __forceinline__ void load_geom(const CurveDesc &d, const float2 *__restrict__ tv, CurveGeom &g) {
    g.type = (int)(d.type & 0xFFu);
    g.w = g.type == kRational ? d.w : 0.f;
    const int n = g.type & 7;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j < n) {
            float2 v = tv[d.vpos + j];
            g.px[j] = v.x;
            g.py[j] = v.y;
        } else {
            g.px[j] = 0.f;
            g.py[j] = 0.f;
        }
    }
}

// ---------------------------------------------------------- transform --
__global__ void k_transform(FrameArgs a, float2 *__restrict__ tvert, uint32_t *__restrict__ flags) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < a.V;
    uint32_t pid = 0, bit = 0;
    if (valid) {
        float2 p = a.vertex[i];
        pid = a.vertex_pid[i];
        if (a.affine) {
            const float *A = a.affine + 6 * (size_t)pid;
            float x = A[0] * p.x + A[2] * p.y + A[4];
            float y = A[1] * p.x + A[3] * p.y + A[5];
            p = make_float2(x, y);
        }
        const float iv0 = p.x, iv1 = p.y, iv2 = 0.f, iv3 = 1.f;
        float m[16];
        int W = a.W, H = a.H;
        if (a.path_scene != nullptr) {
            const SceneInfo *sc = a.scenes + a.path_scene[pid];
#pragma unroll
            for (int k = 0; k < 16; ++k) m[k] = sc->m[k];
            W = sc->W;
            H = sc->H;
        } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) m[k] = a.m[k];
        }
        float ov[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
            ov[r] = m[4 * r] * iv0 + m[4 * r + 1] * iv1 + m[4 * r + 2] * iv2 + m[4 * r + 3] * iv3;
        ov[0] /= ov[3];
        ov[1] /= ov[3];
        ov[2] /= ov[3];
        const float w = (float)W, h = (float)H;
        const float z = (float)min(W, H);
        const float cutoff = -z * 0.5f;
        if (ov[2] < cutoff) ov[2] = cutoff;
        const float w2 = w * .5f, h2 = h * .5f;
        ov[0] = (ov[0] - w2) * z / (ov[2] + z) + w2;
        ov[1] = (ov[1] - h2) * z / (ov[2] + z) + h2;
        if (a.pass_dy != 0.f) ov[1] = ov[1] - a.pass_dy;
        const int xf = ov[0] < 0 ? 0 : (ov[0] <= w ? 1 : 2);
        const int yf = ov[1] < 0 ? 0 : (ov[1] <= h ? 1 : 2);
        switch ((yf << 4) | xf) {
        case 0x00: bit = 1u << 0; break;
        case 0x01: bit = 1u << 1; break;
        case 0x02: bit = 1u << 2; break;
        case 0x10: bit = 1u << 3; break;
        case 0x11: bit = (1u << 0) | (1u << 7); break;
        case 0x12: bit = 1u << 4; break;
        case 0x20: bit = 1u << 5; break;
        case 0x21: bit = 1u << 6; break;
        default: bit = 1u << 7; break;
        }
        if (floorf(ov[0]) == ov[0]) ov[0] = ov[0] - 1.f / 256.f;
        tvert[i] = make_float2(ov[0], ov[1]);
    }
    // One atomic per distinct path per warp.
    const uint32_t key = valid ? pid : 0xFFFFFFFFu;
    const uint32_t peers = __match_any_sync(0xffffffffu, key);
    const uint32_t agg = __reduce_or_sync(peers, bit);
    if (valid && (threadIdx.x & 31) == (unsigned)(__ffs(peers) - 1)) atomicOr(&flags[pid], agg);
}

// PATH_VISIBLE (ras_define.h:113-127): not entirely on one side of the viewport.
__device__ __forceinline__ bool path_visible(uint32_t f) {
    return (f & 0xF8u) && (f & 0x6Bu) && (f & 0x1Fu) && (f & 0xD6u);
}

// ------------------------------------------------------ intersections --
// Thread i: path i's visibility, for the later stages, and curve i's entries.
__global__ void k_curve_count(FrameArgs a, const float2 *__restrict__ tv, const uint32_t *__restrict__ flags,
                              uint8_t *__restrict__ vis, uint32_t *__restrict__ counts) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < a.P) vis[c] = path_visible(flags[c]) ? 1 : 0;
    if (c >= a.C) return;
    const CurveDesc d = a.curves[c];
    CurveGeom g;
    load_geom(d, tv, g);
    float q[5];
    const int np = monotonize_r(g, path_visible(flags[d.pid]), q);
    const Dim dm = dim_of(a, d.pid);
    float v0x = g.px[0], v0y = g.py[0];
    uint32_t p = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        if (i >= np) break;
        const float t1 = q[i];
        const float v1x = curve_coord(g.type, g.w, g.px, t1), v1y = curve_coord(g.type, g.w, g.py, t1);
        const CutRange cr = cut_range(v0x, v0y, v1x, v1y, dm.W, dm.H);
        p += 1 + cr.nx + cr.ny;
        v0x = v1x;
        v0y = v1y;
    }
    counts[c] = p;
}

// Entries of one curve in t order: each monotone piece emits its start and
// every crossing with a vertical (x = even) or horizontal (y = even) cell
// line, the two crossing chains merged by t; equal t values OR their flags.
// Emission order (a tuning choice, off by default): curves grouped by type
// (cubics, whose crossings are bisections, first) and within a type by
// decreasing entry count.  16-bit key, ascending.
__global__ void k_emit_keys(FrameArgs a, const uint32_t *__restrict__ counts, uint32_t *__restrict__ key,
                            uint32_t *__restrict__ val) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= a.C) return;
    const uint32_t type = a.curves[c].type & 0xFFu;
    const uint32_t rank = type == (uint32_t)kCubic ? 0u : (type == (uint32_t)kRational ? 1u : (type == (uint32_t)kQuad ? 2u : 3u));
    key[c] = (rank << 13) | (0x1FFFu - min(counts[c], 0x1FFFu));
    val[c] = (uint32_t)c;
}

// Entries of one monotone piece (k_make_intersection_impl_1,
// ras_cut.h:837-1241): its start and its crossings with vertical and
// horizontal cell lines.  The reference solves the crossings one by one in
// merged t order, each from the parameter of the previous crossing with a
// line of the same direction: the two directions are independent chains, and
// the merge takes the nearer of their current crossings, the vertical one on
// ties (CurveChain below solves a chain, merge_piece merges two).
constexpr int kEmitThreads = 256;
constexpr int kEmitCurves = 128;   // curves of a block, at most
constexpr int kEmitLocal = 4096;   // crossings of a block's curves held in shared memory (else in global scratch)
constexpr int kMergeSerial = 24;   // entries of a piece merged by one lane (longer pieces: by a warp)
constexpr int kChainClasses = 24;  // solver (cubic, quadratic, line) x length octave
constexpr uint32_t kNoChain = 0xFFFFu;

// A block's curves, their monotone pieces' end parameters (flags in the low
// bits), the pieces' first entries within the curve, and per piece and
// direction the crossings: first line (13 bits) | falling << 13 | count << 14.
struct EmitBlock {
    float px[4][kEmitCurves], py[4][kEmitCurves], w[kEmitCurves], tq[5][kEmitCurves];
    uint32_t chain[2][5][kEmitCurves];
    uint32_t rel[5][kEmitCurves];
    uint32_t type[kEmitCurves], cid[kEmitCurves];
    uint32_t off[kEmitCurves];  // the curve's first entry
    uint32_t tof[kEmitCurves];  // its first solved parameter
    uint32_t cls[32], warp_pieces[8], warp_entries[8], next_chain;
    uint16_t item[2 * 5 * kEmitCurves + 64];  // chains in the order they are solved: curve | piece << 7 | direction << 10
    uint16_t piece[5 * kEmitCurves];     // the pieces: curve | piece << 7
    float t[kEmitLocal];
};

__device__ __forceinline__ float piece_t0(const EmitBlock &S, int L, int ms) { return ms > 0 ? S.tq[ms - 1][L] : 0.f; }

// Class of a chain: solver, then length octaves from the longest.
__device__ __forceinline__ uint32_t chain_class(int type, uint32_t n) {
    return (type == kCubic ? 0u : (type == kLinear ? 16u : 8u)) + 7u - (uint32_t)min(31 - __clz((int)n), 7);
}

// Entries of a piece from its solved chains, X[nx] and Y[ny], by one lane:
// the heads of the two chains compared as the reference does.  Coincident
// parameters: both entries get both flags.
__device__ __forceinline__ void merge_piece(const float *X, int nx, const float *Y, int ny, float t0, int cid,
                                            int2 *__restrict__ out) {
    const float none0 = 2.f, none1 = ffrom(fbits(2.f) | 1u);
    int ix = 0, iy = 0;
    float h0, h1;
    if (nx == 0) {
        h0 = none0;
        h1 = t0;
    } else if (ny == 0) {
        h0 = t0;
        h1 = none1;
    } else {
        h0 = X[ix++];
        h1 = t0;
    }
    uint32_t last = fbits(-1.f);
    const int n = nx + ny + 1;
    for (int p = 0; p < n; ++p) {
        uint32_t ob;
        if (h0 <= h1) {
            ob = fbits(h0);
            h0 = ix < nx ? X[ix++] : none0;
        } else {
            ob = fbits(h1);
            h1 = iy < ny ? Y[iy++] : none1;
        }
        if ((ob & 0xFFFFFFFCu) == (last & 0xFFFFFFFCu)) {
            ob |= last;
            out[p - 1] = make_int2(cid, (int)ob);
        }
        out[p] = make_int2(cid, (int)ob);
        last = ob;
    }
}

// The same by the whole warp, 32 entries at a time: entry p's split between
// the chains by a binary search on the merge diagonal.  X ascends; Y, with
// the piece start before it, ascends but for crossings whose flag bits order
// them just before the start: the search compares the running maximum, which
// gives the head comparison's order.  A run of coincident parameters
// accumulates its flags in order (an entry gets those up to its successor).
__device__ __forceinline__ void merge_piece_warp(const float *X, int nx, const float *Y, int ny, float t0, int cid,
                                                 int2 *__restrict__ out, int lane) {
    const int n = nx + ny + 1;
    uint32_t carry_t = 0xFFFFFFFFu, carry_f = 0u;
    for (int base = 0; base < n; base += 32) {
        const int p = base + lane;
        const bool live = p < n;
        float e = 0.f;
        if (live) {
            if (nx == 0 || ny == 0) {
                e = p == 0 ? t0 : (nx == 0 ? Y[p - 1] : X[p - 1]);
            } else {
                const int b = ny + 1;  // the start, then Y
                int lo = max(0, p - b), hi = min(p, nx);
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1, j = p - 1 - mid;
                    const float y = j == 0 ? t0 : fmaxf(t0, Y[j - 1]);
                    if (X[mid] <= y) lo = mid + 1;
                    else hi = mid;
                }
                const int j = p - lo;
                const float y = j == 0 ? t0 : (j < b ? Y[j - 1] : 2.f);
                e = lo < nx && (j >= b || X[lo] <= fmaxf(t0, y)) ? X[lo] : y;
            }
        }
        const uint32_t tb = live ? fbits(e) & 0xFFFFFFFCu : 0xFFFFFFF8u, f = live ? fbits(e) & 3u : 0u;
        uint32_t prev = __shfl_up_sync(0xffffffffu, tb, 1);
        if (lane == 0) prev = carry_t;
        const uint32_t eq = __ballot_sync(0xffffffffu, live && tb == prev);
        const uint32_t b0 = __ballot_sync(0xffffffffu, f & 1u), b1 = __ballot_sync(0xffffffffu, f & 2u);
        const uint32_t le = 0xFFFFFFFFu >> (31 - lane);
        const uint32_t heads = ~eq & le;  // this lane's run: from its last head (or from the previous window)
        const uint32_t run = heads ? le & ~((1u << (31 - __clz(heads))) - 1u) : le;
        const uint32_t nx1 = lane < 31 ? (eq >> (lane + 1)) & 1u : 0u;  // the next entry is in the run
        const uint32_t upto = run | (nx1 << (lane < 31 ? lane + 1 : 0));
        const uint32_t in = heads ? 0u : carry_f;
        const uint32_t own = in | ((b0 & run) ? 1u : 0u) | ((b1 & run) ? 2u : 0u);
        const uint32_t full = in | ((b0 & upto) ? 1u : 0u) | ((b1 & upto) ? 2u : 0u);
        if (live) out[p] = make_int2(cid, (int)(tb | full));
        if (lane == 0 && (eq & 1u)) out[p - 1] = make_int2(cid, (int)(tb | own));  // (written by the last window)
        carry_t = __shfl_sync(0xffffffffu, tb, 31);
        carry_f = __shfl_sync(0xffffffffu, own, 31);
        __syncwarp();
    }
}

// One block per `per_block` curves.  Each thread expands one curve into its
// monotone pieces; the crossings of a piece are two independent chains (see
// above), and every chain is one work item of a lane: the longest serial
// sequence is the crossings of one curve with the lines of one direction.
// The block's chains are solved grouped by solver (cubics, whose crossings are
// bisections, first; each solver from a multiple of 32 on, so that the first
// chains of a warp are of one solver) and by decreasing length, a lane whose
// chain is done taking the block's next one, so that the lanes of a warp run the
// same solver and stay busy until the list runs out.  Then the pieces are merged,
// short ones one per lane and long ones by a warp.  Bound by the latency of a
// chain's bisections (about 0.7 us a crossing) where curves are few and by
// issue (400 thread instructions an entry, 19 lanes active) where they are
// many.  Emission + fragments of 64 paths over 512 x 512, 2,500 paths over
// 1917 x 1079, 20,000 paths over 2048 x 2048 and a batch of 48 scenes, us:
//   620  533  787  2510  one lane per piece, 32 curves to a warp, ordered by
//                        type and length over the whole frame
//   304  282  783  2550  a lane per chain, solvers one after the other
//   253  280  777  2580  each solver's chains in warps of their own
//   234  280  759  2450  one comparison instead of a difference's sign
//   216  272  760  2450  AHEAD for few curves
template <bool AHEAD>
__global__ void __launch_bounds__(kEmitThreads)
    k_curve_emit(FrameArgs a, int per_block, const float2 *__restrict__ tv, const uint8_t *__restrict__ vis,
                 const uint32_t *__restrict__ offsets, const uint32_t *__restrict__ order, float *scratch,
                 int2 *__restrict__ entries, uint32_t cap_nf, FrameCounters *ctr) {
    __shared__ EmitBlock S;
    // the entries admitted for the rest of the frame; too many for the buffers,
    // or the offsets not to be trusted (a scan gave up waiting): none, and
    // nothing is written
    if (!admit(&ctr->need_nf, &ctr->nf, cap_nf, &ctr->status)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t i = (int64_t)blockIdx.x * per_block + tid;
    int np = 0, type = 0;
    uint32_t n_ent = 0;
    if (tid < 32) S.cls[tid] = 0u;
    if (tid == 0) S.next_chain = 0u;
    __syncthreads();
    if (tid < per_block && i < a.C) {
        const int cid = order != nullptr ? (int)order[i] : (int)i;
        const CurveDesc d = a.curves[cid];
        CurveGeom g;
        load_geom(d, tv, g);
        type = g.type;
        float q[5];
        np = monotonize_r(g, vis[d.pid] != 0, q);
        const Dim dm = dim_of(a, d.pid);
#pragma unroll
        for (int k = 0; k < 4; ++k) S.px[k][tid] = g.px[k], S.py[k][tid] = g.py[k];
        S.w[tid] = g.w;
        S.type[tid] = (uint32_t)type;
        S.cid[tid] = (uint32_t)cid;
        S.off[tid] = offsets[cid];
        float v0x = g.px[0], v0y = g.py[0];
#pragma unroll
        for (int ms = 0; ms < 5; ++ms) {
            if (ms < np) {
                const float v1x = curve_coord(g.type, g.w, g.px, q[ms]), v1y = curve_coord(g.type, g.w, g.py, q[ms]);
                const CutRange cr = cut_range(v0x, v0y, v1x, v1y, dm.W, dm.H);
                const uint32_t tb = fbits(q[ms]) & 0xFFFFFFFCu;
                S.tq[ms][tid] = (floorf(v1x) == v1x) ? ffrom(tb | 2u) : ffrom(tb | 3u);
                S.rel[ms][tid] = n_ent;
                const int bx = cr.dx < 0.f ? cr.xe : cr.xb, by = cr.dy < 0.f ? cr.ye : cr.yb;
                S.chain[0][ms][tid] = ((uint32_t)bx & 0x1FFFu) | (cr.dx < 0.f ? 0x2000u : 0u) | ((uint32_t)cr.nx << 14);
                S.chain[1][ms][tid] = ((uint32_t)by & 0x1FFFu) | (cr.dy < 0.f ? 0x2000u : 0u) | ((uint32_t)cr.ny << 14);
                if (cr.nx) atomicAdd(&S.cls[chain_class(type, (uint32_t)cr.nx)], 1u);
                if (cr.ny) atomicAdd(&S.cls[chain_class(type, (uint32_t)cr.ny)], 1u);
                n_ent += 1 + cr.nx + cr.ny;
                v0x = v1x;
                v0y = v1y;
            }
        }
    }
    // the block's pieces and entries; the chains placed by class
    uint32_t pre = (uint32_t)np, lpre = n_ent;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, pre, o), u = __shfl_up_sync(0xffffffffu, lpre, o);
        if (lane >= o) pre += v, lpre += u;
    }
    if (lane == 31) S.warp_pieces[warp] = pre, S.warp_entries[warp] = lpre;
    __syncthreads();
    uint32_t n_pieces = 0, n_total = 0, wp = 0, we = 0;
#pragma unroll
    for (int k = 0; k < kEmitThreads / 32; ++k) {
        if (k == warp) wp = n_pieces, we = n_total;
        n_pieces += S.warp_pieces[k];
        n_total += S.warp_entries[k];
    }
    pre += wp - (uint32_t)np;
    lpre += we - n_ent;
    const bool local = n_total <= (uint32_t)kEmitLocal;
    // every warp scans the class counts (the same values); one keeps them as cursors
    uint32_t cls = lane < kChainClasses ? S.cls[lane] : 0u;
    const uint32_t cls_n = cls;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, cls, o);
        if (lane >= o) cls += v;
    }
    // each solver's chains from a multiple of 32 on, with places left empty
    const uint32_t n_cubic = __shfl_sync(0xffffffffu, cls, 7), n_quad = __shfl_sync(0xffffffffu, cls, 15) - n_cubic;
    const uint32_t quad0 = (n_cubic + 31u) & ~31u, line0 = (quad0 + n_quad + 31u) & ~31u;
    const uint32_t n_chains = line0 + __shfl_sync(0xffffffffu, cls, 31) - n_cubic - n_quad;
    __syncthreads();
    if (warp == 0) {
        S.cls[lane] = cls - cls_n + (lane < 8 ? 0u : (lane < 16 ? quad0 - n_cubic : line0 - n_cubic - n_quad));
        if (n_cubic + lane < quad0) S.item[n_cubic + lane] = kNoChain;
        if (quad0 + n_quad + lane < line0) S.item[quad0 + n_quad + lane] = kNoChain;
    }
    __syncthreads();
    if (np > 0) {
        S.tof[tid] = local ? lpre : S.off[tid];
        for (int ms = 0; ms < np; ++ms) {
            S.piece[pre + ms] = (uint16_t)(tid | (ms << 7));
            for (int ax = 0; ax < 2; ++ax) {
                const uint32_t n = S.chain[ax][ms][tid] >> 14;
                if (n) S.item[atomicAdd(&S.cls[chain_class(type, n)], 1u)] = (uint16_t)(tid | (ms << 7) | (ax << 10));
            }
        }
    }
    __syncthreads();
    float *const tbuf = local ? S.t : scratch;
    // chains: crossing k of a piece's vertical lines at t[1 + k] of the piece,
    // of its horizontal ones past them
    {
        int ctype = 0, rem = 0, ax = 0;
        float P[4] = {0.f, 0.f, 0.f, 0.f}, w = 0.f, c = 0.f, dc = 0.f, t = 0.f, t1 = 0.f;
        float *out = nullptr;
        bool more = true;
        for (;;) {
            const uint32_t want = __ballot_sync(0xffffffffu, rem == 0);
            if (more && want) {
                uint32_t next = 0;
                if (lane == 0) next = atomicAdd(&S.next_chain, (uint32_t)__popc(want));
                next = __shfl_sync(0xffffffffu, next, 0);
                more = next + __popc(want) < n_chains;
                const uint32_t k = next + __popc(want & ((1u << lane) - 1u));
                const uint32_t it = rem == 0 && k < n_chains ? S.item[k] : kNoChain;
                if (it != kNoChain) {
                    const int L = (int)(it & 127u), ms = (int)(it >> 7) & 7;
                    ax = (int)(it >> 10);
                    ctype = (int)S.type[L];
                    w = S.w[L];
#pragma unroll
                    for (int j = 0; j < 4; ++j) P[j] = ax ? S.py[j][L] : S.px[j][L];
                    const uint32_t ch = S.chain[ax][ms][L];
                    rem = (int)(ch >> 14);
                    c = (float)(ch & 0x1FFFu);
                    dc = (ch & 0x2000u) ? -2.f : 2.f;
                    t = piece_t0(S, L, ms);
                    t1 = S.tq[ms][L];
                    out = tbuf + S.tof[L] + S.rel[ms][L] + 1 + (ax ? S.chain[0][ms][L] >> 14 : 0u);
                }
            }
            if (!__any_sync(0xffffffffu, rem > 0)) break;
            if (rem > 0) {
                t = ffrom((fbits(solve_crossing<AHEAD>(ctype, w, P, c, t, t1)) & 0xFFFFFFFCu) | (uint32_t)ax);
                *out++ = t;
                c += dc;
                --rem;
            }
        }
    }
    __syncthreads();
    for (uint32_t base = warp * 32; base < n_pieces; base += kEmitThreads) {
        const uint32_t k = base + lane;
        int L = 0, ms = 0, nx = 0, ny = 0;
        if (k < n_pieces) {
            L = S.piece[k] & 127;
            ms = S.piece[k] >> 7;
            nx = (int)(S.chain[0][ms][L] >> 14);
            ny = (int)(S.chain[1][ms][L] >> 14);
        }
        const bool lng = nx + ny + 1 > kMergeSerial;
        if (k < n_pieces && !lng) {
            const float *X = tbuf + S.tof[L] + S.rel[ms][L] + 1;
            merge_piece(X, nx, X + nx, ny, piece_t0(S, L, ms), (int)S.cid[L], entries + S.off[L] + S.rel[ms][L]);
        }
        for (uint32_t m = __ballot_sync(0xffffffffu, lng); m; m &= m - 1u) {
            const int src = __ffs(m) - 1;
            const int qL = __shfl_sync(0xffffffffu, L, src), qm = __shfl_sync(0xffffffffu, ms, src);
            const int qx = __shfl_sync(0xffffffffu, nx, src), qy = __shfl_sync(0xffffffffu, ny, src);
            const float *X = tbuf + S.tof[qL] + S.rel[qm][qL] + 1;
            merge_piece_warp(X, qx, X + qx, qy, piece_t0(S, qL, qm), (int)S.cid[qL], entries + S.off[qL] + S.rel[qm][qL],
                             lane);
        }
    }
}

// ---------------------------------------------------------- fragments --
template <int S>
__global__ void __launch_bounds__(kThreads, 8) k_fragment(FrameArgs a, const float2 *__restrict__ tv,
                                                       const int2 *__restrict__ entries,
                                                       const FrameCounters *__restrict__ ctr,
                                                       int32_t *__restrict__ key_out, uint32_t *__restrict__ pid_out,
                                                       int8_t *__restrict__ wn_out, uint32_t *__restrict__ mask_out,
                                                       uint64_t *__restrict__ sort_key, uint32_t *__restrict__ sort_val,
                                                       uint64_t *__restrict__ mark_words, int64_t n_mark) {
    constexpr int WORDS = S / 8;
    const int64_t nf = ctr->nf;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_mark) mark_words[i] = 0ull;  // the scan-mark pass's look-back words, cleared on the way
    if (i >= nf) return;
    const int2 e0 = entries[i];
    const int2 e1 = (i + 1) != nf ? entries[i + 1] : make_int2(-1, 0x3f800000);
    int f0 = e0.y & 1, f1 = e1.y & 1;
    float t0 = ffrom((uint32_t)e0.y & 0xFFFFFFFCu);
    float t1 = ffrom((uint32_t)e1.y & 0xFFFFFFFCu);
    if (t0 < 0) t0 = 0.f;
    if (t1 < 0) t1 = 0.f;
    if (t0 == 0.f || t0 == 1.f) f0 = 1;
    if (t1 == 0.f || t1 == 1.f) f1 = 1;
    const int cid = e0.x;
    const CurveDesc d = a.curves[cid];
    const uint32_t pathid = d.pid;
    const Dim dm = dim_of(a, pathid);
    int32_t yx = kInvalidKey;
    if (e0.x != e1.x) t1 = 1.f;
    int wnchg = 0, swn = 0;
    uint32_t mask[4] = {0u, 0u, 0u, 0u};
    float4 chord = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t lmk[4] = {0u, 0u, 0u, 0u};
    if (t0 < t1) {
        CurveGeom g;
        load_geom(d, tv, g);
        const float fi0 = 0 / 1.f, fi1 = 1 / 1.f;
        const float ta = (1 - fi0) * t0 + fi0 * t1;
        const float tb = (1 - fi1) * t0 + fi1 * t1;
        const float c0x = curve_coord(g.type, g.w, g.px, ta), c0y = curve_coord(g.type, g.w, g.py, ta);
        const float c1x = curve_coord(g.type, g.w, g.px, tb), c1y = curve_coord(g.type, g.w, g.py, tb);
        const bool rev = ((d.type >> 8) & 1u) != 0;
        const float vfx = rev ? c1x : c0x, vfy = rev ? c1y : c0y;
        const float vlx = rev ? c0x : c1x, vly = rev ? c0y : c1y;
        const int sf = rev ? f1 : f0;
        const int sl = rev ? f0 : f1;
        const int rx = floor2((vfx + vlx) * 0.5f);
        const int ry = floor2((vfy + vly) * 0.5f);
        const int px = min(max(rx, -2), (int)(((uint32_t)dm.W & 0xFFFFFFFEu) + 2));
        const int py = min(max(ry, -2), (int)(((uint32_t)dm.H & 0xFFFFFFFEu) + 2));
        const uint32_t ys = (uint32_t)(py + 0x7FFF) << 16;
        const uint32_t xs = (uint32_t)(px + 0x7FFF) & 0xFFFFu;
        if ((uint32_t)ry < (uint32_t)dm.H) yx = (int32_t)(ys | xs);
        const int wy = py + 1;
        if (vfy == vly) {
            swn = 0;
        } else if (vfy <= wy && wy < vly) {
            swn = -1;
        } else if (vly <= wy && wy < vfy) {
            swn = 1;
        }
        if (vfy < vly) {
            wnchg = -1;
        } else if (vfy > vly) {
            wnchg = 1;
        } else {
            wnchg = (vfx < vlx) ? 1 : -1;
        }
        float lx = 0.f, ly = 0.f, rgt_y = 0.f;
        int left_flag = 1;
        if (vfx < vlx) {
            lx = vfx;
            ly = vfy;
            rgt_y = vly;
            left_flag = sf;
        } else if (vfx > vlx) {
            lx = vlx;
            ly = vly;
            rgt_y = vfy;
            left_flag = sl;
        } else if (vfx < px + 1) {
            if (sf == 0) {
                lx = vfx;
                ly = vfy;
                rgt_y = vly;
                left_flag = 0;
            } else if (sl == 0) {
                lx = vlx;
                ly = vly;
                rgt_y = vfy;
                left_flag = 0;
            }
        }
        (void)lx;
        uint32_t lm[4] = {0u, 0u, 0u, 0u};
        if (left_flag == 0) {
            vertical_mask<S>((ly - py) * .5f, lm);
            if (ly <= py + 1) {
                if (ly >= rgt_y) wnchg = -wnchg;
            } else {
                if (ly < rgt_y) wnchg = -wnchg;
#pragma unroll
                for (int w = 0; w < 4; ++w) lm[w] = ~lm[w];
            }
        }
        const float bx = (float)px, by = (float)py;
        const float q0x = (c0x - bx) * .5f, q0y = (c0y - by) * .5f;
        const float q1x = (c1x - bx) * .5f, q1y = (c1y - by) * .5f;
        chord = make_float4(q0x, q0y, q1x, q1y);
#pragma unroll
        for (int w = 0; w < 4; ++w) lmk[w] = lm[w];
        uint32_t vm[4];
        vertical_mask2<S>(q0y, q1y, vm);
        const int texel = table_texel(q0x, q0y, q1x, q1y);
        if (S == 8) {
            const uint32_t tm = __ldg(a.mask_table + texel);
            mask[0] = (tm & vm[0]) ^ lm[0];
        } else if (S == 16) {
            const uint2 tm = __ldg(reinterpret_cast<const uint2 *>(a.mask_table) + texel);
            mask[0] = (tm.x & vm[0]) ^ lm[0];
            mask[1] = (tm.y & vm[1]) ^ lm[1];
        } else {
            const uint4 tm = __ldg(reinterpret_cast<const uint4 *>(a.mask_table) + texel);
            mask[0] = (tm.x & vm[0]) ^ lm[0];
            mask[1] = (tm.y & vm[1]) ^ lm[1];
            mask[2] = (tm.z & vm[2]) ^ lm[2];
            mask[3] = (tm.w & vm[3]) ^ lm[3];
        }
    }
    if (a.chord != nullptr) {
        a.chord[i] = chord;
        uint32_t vmk[4] = {0u, 0u, 0u, 0u};
        if (chord.y != chord.w) vertical_mask2<S>(chord.y, chord.w, vmk);
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
            a.lmask[i * WORDS + w] = lmk[w];
            a.vmask[i * WORDS + w] = vmk[w];
        }
    }
    key_out[i] = yx;
    pid_out[i] = pathid | ((uint32_t)wnchg << 30);
    wn_out[i] = (int8_t)swn;
    if (WORDS == 1) {
        mask_out[i] = mask[0];
    } else if (WORDS == 2) {
        reinterpret_cast<uint2 *>(mask_out)[i] = make_uint2(mask[0], mask[1]);
    } else {
        reinterpret_cast<uint4 *>(mask_out)[i] = make_uint4(mask[0], mask[1], mask[2], mask[3]);
    }
    const int nrows = (dm.H + 1) / 2;
    sort_key[i] = ((uint64_t)pathid << 24) | (uint64_t)local_sort_key(yx, nrows) |
                  ((uint64_t)pack_fw(swn, wnchg) << kFwShift);
    sort_val[i] = (uint32_t)i;
}

// --------------------------------------------- winding scan + marks --
constexpr int kMarkThreads = 512;
constexpr int kMarkItems = 8;
constexpr int kMarkTile = kMarkThreads * kMarkItems;
constexpr uint64_t kSegBit = 1ull << 32;  // winding look-back: a scene starts in the tile (batches)

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}
// Exclusive scan over the block, one barrier: every warp scans the warps' totals
// itself.  sw (one word per warp) is not used for anything else.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *sw, uint32_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kMarkThreads / 32;
    const uint32_t inc = warp_incl_scan(v);
    if (lane == 31) sw[warp] = inc;
    __syncthreads();
    uint32_t t = lane < W ? sw[lane] : 0u;
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, t, o);
        if (lane >= o) t += n;
    }
    *total = __shfl_sync(0xffffffffu, t, W - 1);
    return __shfl_sync(0xffffffffu, t, (warp + 31) & 31) * (warp ? 1u : 0u) + inc - v;
}

// Segmented sums: (s, f) where f = a segment starts inside; a then b.
struct SegSum {
    uint32_t s, f;
};
__device__ __forceinline__ SegSum seg_then(SegSum a, SegSum b) { return SegSum{b.f ? b.s : a.s + b.s, a.f | b.f}; }

__device__ __forceinline__ SegSum block_excl_segscan(SegSum v, uint32_t *ss, uint32_t *sf, SegSum *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int W = kMarkThreads / 32;
    SegSum inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const SegSum up{__shfl_up_sync(0xffffffffu, inc.s, o), __shfl_up_sync(0xffffffffu, inc.f, o)};
        if (lane >= o) inc = seg_then(up, inc);
    }
    SegSum prev{__shfl_up_sync(0xffffffffu, inc.s, 1), __shfl_up_sync(0xffffffffu, inc.f, 1)};
    if (lane == 0) prev = SegSum{0u, 0u};
    if (lane == 31) ss[warp] = inc.s, sf[warp] = inc.f;
    __syncthreads();
    SegSum t = lane < W ? SegSum{ss[lane], sf[lane]} : SegSum{0u, 0u};
#pragma unroll
    for (int o = 1; o < W; o <<= 1) {
        const SegSum up{__shfl_up_sync(0xffffffffu, t.s, o), __shfl_up_sync(0xffffffffu, t.f, o)};
        if (lane >= o) t = seg_then(up, t);
    }
    *total = SegSum{__shfl_sync(0xffffffffu, t.s, W - 1), __shfl_sync(0xffffffffu, t.f, W - 1)};
    const SegSum before{__shfl_sync(0xffffffffu, t.s, (warp + 31) & 31), __shfl_sync(0xffffffffu, t.f, (warp + 31) & 31)};
    return warp ? seg_then(before, prev) : prev;
}

struct Mark {
    uint32_t ff, sf;
};

// Columns [x0, x1) of draw item `it` in a viewport W wide (its first column
// read as unsigned 16 bits: cells at x = -2 cover nothing).
__device__ __forceinline__ void item_cols(const int4 &it, int W, int &x0, int &x1) {
    const int x = (int)((uint32_t)it.x & 0xFFFFu);
    x0 = max(x, 0);
    x1 = min(x + it.y, W);
}

// Resolve bins of draw item `it` (the tiles of 1 << shift columns of the
// band of 64 >> shift cell rows holding its row) in a viewport W x H whose
// bins are numbered from bin0: *first and the count (consecutive bins).
__device__ __forceinline__ int item_bins(const int4 &it, int W, int H, int shift, uint32_t bin0, uint32_t *first) {
    int x0, x1;
    item_cols(it, W, x0, x1);
    const int row = (it.x >> 16) / 2;
    if (x1 <= x0 || row < 0 || row >= (H + 1) / 2) return 0;
    const int ntx = bin_cols(W, shift);
    *first = bin0 + (uint32_t)((row >> (kBinShift - shift)) * ntx + (x0 >> shift));
    return ((x1 - 1) >> shift) - (x0 >> shift) + 1;
}

// Counts item `it`'s pairs in its bins; returns its pairs in the other
// built-in tile (0 if there is none).
__device__ __forceinline__ uint32_t count_bins(const FrameArgs &a, const int4 &it, const Dim &dp, uint32_t p,
                                               uint32_t *__restrict__ bin_count) {
    const uint32_t bin0 = a.scenes != nullptr ? a.scenes[a.path_scene[p]].bin_off : 0u;
    uint32_t b0 = 0;
    const int nb = item_bins(it, dp.W, dp.H, a.bin_shift, bin0, &b0);
    for (int t = 0; t < nb; ++t) atomicAdd(bin_count + b0 + t, 1u);
    return a.alt_shift >= 0 ? (uint32_t)item_bins(it, dp.W, dp.H, a.alt_shift, 0u, &b0) : 0u;
}

// Column and row of a cell from its key within the path (the inverse of
// local_sort_key; the out-of-range sentinel's row is far outside).
__device__ __forceinline__ int local_x(uint64_t k) { return 2 * (int)((uint32_t)k & 0xFFFu) - 2; }
__device__ __forceinline__ int local_y(uint64_t k, int nrows) {
    const int rr = (int)(((uint32_t)k >> 12) & 0xFFFu);
    return rr == nrows ? 0 : (rr == nrows - 1 ? 0x7FFF : 2 * (rr + 1));
}

// k_mark_merged_fragment_and_span (cu:462-535) on sorted position i with
// keys k0 (position i - 1) and k1 (position i) and scanned winding w.  Keys of
// one path order and compare as its cells do, so the marks need the cell's
// column and row only for the viewport test.
__device__ __forceinline__ Mark mark_of(int64_t i, uint64_t k0, uint64_t k1, int8_t w, const FrameArgs &a) {
    const uint32_t p1 = (uint32_t)(k1 >> 24);
    const Dim dm = dim_of(a, p1);
    const int x1 = local_x(k1), y1 = local_y(k1, (dm.H + 1) / 2);
    const bool in = x1 >= 0 && x1 < dm.W && y1 < dm.H;
    if (i == 0) return Mark{in ? 1u : 0u, 0u};
    Mark m{in && k0 != k1 ? 1u : 0u, 0u};
    // a span: the same row of the same path, with columns left out between
    // (equal for two sentinels: none)
    if ((k0 >> 12) == (k1 >> 12) && ((uint32_t)k0 & 0xFFFu) + 1u < ((uint32_t)k1 & 0xFFFu)) {
        const uint8_t fr = a.fill_rule[p1];
        m.sf = (fr == 0 && w != 0) || (fr == 1 && (w & 1)) ? 1u : 0u;
    }
    return m;
}

// Stages 9-12 and 14 in one pass over the sorted entries (thrust's int8
// scan of the shuffled windings, cu:1099-1101; the marks, cu:462-535; their
// inclusive scans, cu:1139-1157; the draw list, cu:789-868).  Per tile:
// the windings gathered through the sort permutation and scanned (int8
// arithmetic: only the low 8 bits are kept), with the tile's prefix from a
// decoupled look-back (restarting at every scene of a batch, so that each
// scene sees the scan a single-scene render gives it); then the merged and
// span marks, scanned with a second look-back, and the draw items written.
// The last tile writes the item counts.  Sorted keys are read 128 bits at a
// time; each carries its fragment's scan winding in bits 60-63.  Bound by the
// wait for the two look-backs (40% of the stalls) and by issue: an entry makes
// up to two draw items, so a warp lists its items and writes them 32 at a time.
// With the two kinds written entry by entry (20 lanes active), 2048 entries to
// a tile and three barriers to a scan, this took 373 us on 20,000 paths over
// 2048 x 2048, 1230 on a batch of 48 scenes and 88 on 2,500 paths over 1917 x
// 1079; here 307, 941 and 72 (tiles of 2048 entries: 321, 972, 78).
__global__ void __launch_bounds__(kMarkThreads) k_scan_mark(FrameArgs a, const uint64_t *__restrict__ skey,
                                                            int8_t *__restrict__ wn_scan,
                                                            int4 *__restrict__ draw, uint32_t *__restrict__ heads,
                                                            uint32_t *__restrict__ item_scene,
                                                            uint32_t *__restrict__ bin_count,
                                                            FrameCounters *__restrict__ ctr,
                                                            uint64_t *__restrict__ st_wn, uint64_t *__restrict__ st_fl,
                                                            uint32_t spin_cap) {
    __shared__ uint32_t ss[kMarkThreads / 32], sf[kMarkThreads / 32], sm[kMarkThreads / 32];
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_pre, s_pre2;
    __shared__ uint16_t s_item[kMarkThreads / 32][2 * 32 * kMarkItems];
    const int64_t nf = ctr->nf;
    const int64_t ntiles = (nf + kMarkTile - 1) / kMarkTile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&ctr->tiles[1], 1u);
    __syncthreads();
    const int64_t t = s_tile;
    if (t >= ntiles) {
        if (t == 0 && threadIdx.x == 0) ctr->n_merged = ctr->n_span = ctr->n_items = 0u;
        return;
    }
    const int64_t base = t * kMarkTile + (int64_t)threadIdx.x * kMarkItems;
    const int64_t left = nf - base;
    const int cnt = left <= 0 ? 0 : (left >= kMarkItems ? kMarkItems : (int)left);
    uint64_t k[kMarkItems + 1];  // sorted keys at base - 1 .. base + 7
    if (cnt == kMarkItems) {
        const uint4 *kp = reinterpret_cast<const uint4 *>(skey + base);
#pragma unroll
        for (int q = 0; q < kMarkItems / 2; ++q) {
            const uint4 v = kp[q];
            k[1 + 2 * q] = (uint64_t)v.x | ((uint64_t)v.y << 32);
            k[2 + 2 * q] = (uint64_t)v.z | ((uint64_t)v.w << 32);
        }
    } else {
#pragma unroll
        for (int j = 0; j < kMarkItems; ++j) k[1 + j] = j < cnt ? skey[base + j] : 0ull;
    }
    k[0] = (cnt > 0 && base > 0) ? skey[base - 1] : 0ull;
    uint32_t fb[kMarkItems];  // the windings, and the keys without them
#pragma unroll
    for (int j = 0; j < kMarkItems; ++j) fb[j] = (uint32_t)(k[1 + j] >> kFwShift);
#pragma unroll
    for (int j = 0; j <= kMarkItems; ++j) k[j] &= kKeyMask;
    // windings in sorted order, and the scene starts of a batch
    const bool batch = a.scenes != nullptr && a.n_scenes > 1;
    int32_t v[kMarkItems];
    uint32_t seg = 0u;  // bit j: a scene starts at base + j
    SegSum agg{0u, 0u};
#pragma unroll
    for (int j = 0; j < kMarkItems; ++j) {
        v[j] = j < cnt ? fw_swn(fb[j]) : 0;
        if (batch && j < cnt &&
            (base + j == 0 || a.path_scene[(uint32_t)(k[j + 1] >> 24)] != a.path_scene[(uint32_t)(k[j] >> 24)]))
            seg |= 1u << j;
        agg = seg_then(agg, SegSum{(uint32_t)v[j], (seg >> j) & 1u});
    }
    SegSum tot;
    const SegSum tpre = block_excl_segscan(agg, ss, sf, &tot);
    if (threadIdx.x < 32) {
        uint64_t pre = 0;
        if (t > 0) {
            if (threadIdx.x == 0) lb_store(st_wn + t, kLbAggregate | (tot.f ? kSegBit : 0ull) | tot.s);
            pre = lb_walk(st_wn, t, kSegBit, spin_cap, &ctr->status);
        }
        if (threadIdx.x == 0) {
            lb_store(st_wn + t, kLbInclusive | (uint32_t)(tot.f ? tot.s : (uint32_t)pre + tot.s));
            s_pre = pre;
        }
    }
    __syncthreads();
    // scanned windings (exclusive, restarting at scene starts)
    SegSum run = seg_then(SegSum{(uint32_t)s_pre, 0u}, tpre);
    int8_t ws[kMarkItems];
#pragma unroll
    for (int j = 0; j < kMarkItems; ++j) {
        if ((seg >> j) & 1u) run.s = 0u;
        ws[j] = (int8_t)(uint8_t)run.s;
        run.s += (uint32_t)v[j];
    }
    if (cnt == kMarkItems) {
        uint32_t packed[kMarkItems / 4] = {};
#pragma unroll
        for (int j = 0; j < kMarkItems; ++j) packed[j / 4] |= (uint32_t)(uint8_t)ws[j] << (8 * (j % 4));
#pragma unroll
        for (int j = 0; j < kMarkItems / 4; ++j) reinterpret_cast<uint32_t *>(wn_scan + base)[j] = packed[j];
    } else {
#pragma unroll
        for (int j = 0; j < kMarkItems; ++j)
            if (j < cnt) wn_scan[base + j] = ws[j];
    }
    // marks and their scans
    Mark mk[kMarkItems];
    uint32_t fs = 0;
#pragma unroll
    for (int j = 0; j < kMarkItems; ++j) {
        mk[j] = j < cnt ? mark_of(base + j, k[j], k[j + 1], ws[j], a) : Mark{0u, 0u};
        fs += mk[j].ff | (mk[j].sf << 16);
    }
    uint32_t ftot;
    const uint32_t fpre = block_excl_scan(fs, sm, &ftot);
    const uint64_t ftot_w = ((uint64_t)(ftot & 0xFFFFu) << 31) | (uint64_t)(ftot >> 16);
    if (threadIdx.x < 32) {
        uint64_t pre = 0;
        if (t > 0) {
            if (threadIdx.x == 0) lb_store(st_fl + t, kLbAggregate | ftot_w);
            pre = lb_walk(st_fl, t, 0ull, spin_cap, &ctr->status);
        }
        if (threadIdx.x == 0) {
            lb_store(st_fl + t, kLbInclusive | ((pre + ftot_w) & kLbPayload));
            s_pre2 = pre;
            if (t == ntiles - 1) {  // the frame's item counts
                const uint64_t all = pre + ftot_w;
                const uint32_t nm = (uint32_t)(all >> 31) & 0x7FFFFFFFu, ns = (uint32_t)all & 0x7FFFFFFFu;
                ctr->n_merged = nm;
                ctr->n_span = ns;
                ctr->n_items = nm + ns;
            }
        }
    }
    __syncthreads();
    // the warp's items listed (entry within the warp, a span's with bit 15 set),
    // then written 32 at a time, whichever lane's entry they come from
    const int lane = threadIdx.x & 31;
    uint16_t *const item = s_item[threadIdx.x >> 5];
    uint32_t nfb = (uint32_t)(s_pre2 >> 31) + (fpre & 0xFFFFu);
    const uint32_t nsb = (uint32_t)(s_pre2 & 0x7FFFFFFFu) + (fpre >> 16);
    const uint32_t first = __shfl_sync(0xffffffffu, nfb + nsb, 0);
    uint32_t at = nfb + nsb - first;
#pragma unroll
    for (int j = 0; j < kMarkItems; ++j) {
        if (mk[j].ff) item[at++] = (uint16_t)(lane * kMarkItems + j);
        if (mk[j].sf) item[at++] = (uint16_t)(0x8000 | (lane * kMarkItems + j));
    }
    const uint32_t n = __shfl_sync(0xffffffffu, at, 31);
    nfb = __shfl_sync(0xffffffffu, nfb, 0);
    __syncwarp();
    const int64_t warp_base = base - lane * kMarkItems;
    uint32_t span_px = 0, pairs_alt = 0;  // this thread's span pixels and pairs in the other tile
    for (uint32_t q0 = 0; q0 < n; q0 += 32) {
        const uint32_t q = q0 + lane;
        const bool live = q < n;
        const uint32_t code = live ? item[q] : 0x8000u;
        const bool span = (code & 0x8000u) != 0u;
        const uint32_t frags = __ballot_sync(0xffffffffu, !span);
        if (live) {
            const int64_t i = warp_base + (code & 0x7FFFu);
            const uint64_t k1 = skey[i] & kKeyMask;
            const uint32_t p = (uint32_t)(k1 >> 24);
            const Dim dp = dim_of(a, p);
            const int x1 = local_x(k1), y = local_y(k1, (dp.H + 1) / 2);
            int4 it = make_int4((int32_t)(((uint32_t)y << 16) | (uint32_t)x1), 2, (int32_t)a.fill_rgba[p], 0);
            if (span) {
                const int x0 = local_x(skey[i - 1]) + 2;  // (columns start at -2)
                it.x = (int32_t)(((uint32_t)y << 16) | (uint32_t)x0);
                it.y = x1 - x0;
                span_px += (uint32_t)(x1 - x0);
            } else {
                const uint32_t g = nfb + __popc(frags & ((1u << lane) - 1u));
                it.w = (int)(g + 1);
                heads[g] = (uint32_t)i;
            }
            draw[first + q] = it;
            if (item_scene != nullptr) item_scene[first + q] = a.path_scene[p];
            if (a.item_path != nullptr) a.item_path[first + q] = p;
            pairs_alt += count_bins(a, it, dp, p, bin_count);
        }
        nfb += __popc(frags);
    }
    const uint32_t wpx = __reduce_add_sync(0xffffffffu, span_px);
    const uint32_t wpa = __reduce_add_sync(0xffffffffu, pairs_alt);
    if ((threadIdx.x & 31) == 0 && wpx) atomicAdd(&ctr->span_px, (unsigned long long)wpx);
    if ((threadIdx.x & 31) == 0 && wpa) atomicAdd(&ctr->pairs_alt, wpa);
}

// ------------------------------------------------------- merged masks --
// Per merged fragment: the scanned winding number plus the signed boundary
// masks of every fragment of the (path, cell) group, in 8-bit lanes per
// mask bit (the reference's packed counters), reduced to the 7-bit winding
// number and tested against the fill rule.
//
// A thread per group: the group's head, then its first key, index and winding
// together, then mask by mask with the next key and index on the way.  Bound by
// the latency of these loads, one after the other.  With 256 groups' keys and
// indices staged in shared memory by bulk copies, which every thread of the block
// waited for, the stage took 346 us on 20,000 paths over 2048 x 2048, 846 on a
// batch of 48 scenes and 57 on 2,500 paths over 1917 x 1079; here 293, 678 and 41
// (with two threads a group at 32 samples 344 and 772; with 4 blocks to an SM at
// 32 samples and 6 at fewer 303, 705 and 41).
template <int S>
__global__ void __launch_bounds__(kThreads, S == 32 ? 5 : 8) k_stencil(FrameArgs a, const FrameCounters *__restrict__ ctr,
                                                      const uint64_t *__restrict__ skey,
                                                      const uint32_t *__restrict__ perm,
                                                      const uint32_t *__restrict__ mask,
                                                      const int8_t *__restrict__ wn_scan,
                                                      const uint32_t *__restrict__ heads,
                                                      uint32_t *__restrict__ merged) {
    constexpr int WORDS = S / 8;
    const uint32_t nf = ctr->nf, g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ctr->n_merged) return;
    const uint32_t h = heads[g];
    const int32_t w0 = (int32_t)__ldg(wn_scan + h);
    const uint64_t k0 = __ldg(skey + h);
    const uint32_t raw0 = __ldg(perm + h);
    const uint64_t kh = k0 & kKeyMask;
    // the group's fragments with a winding change: fn(change sign, mask)
    auto walk = [&](auto &&fn) {
        uint64_t kj = k0;
        uint32_t raw = raw0;
        for (uint32_t j = h;;) {
            // (the next position, asked for with this one's mask)
            const uint32_t jn = j + 1;
            const uint64_t kn = jn < nf ? __ldg(skey + jn) : ~0ull;
            const uint32_t rn = jn < nf ? __ldg(perm + jn) : 0u;
            const int32_t chg = fw_chg((uint32_t)(kj >> kFwShift));
            if (chg != 0) {
                uint32_t m[WORDS];
                if constexpr (WORDS == 1) {
                    m[0] = __ldg(mask + raw);
                } else if constexpr (WORDS == 2) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(mask) + raw);
                    m[0] = v.x;
                    m[1] = v.y;
                } else {
                    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(mask) + raw);
                    m[0] = v.x;
                    m[1] = v.y;
                    m[2] = v.z;
                    m[3] = v.w;
                }
                fn(chg, m);
            }
            if (jn >= nf || (kn & kKeyMask) != kh) break;
            j = jn;
            kj = kn;
            raw = rn;
        }
    };
    const int fr = a.fill_rule[(uint32_t)(kh >> 24)];
    // Every sample's winding w0 + (sum of the changes of the fragments covering
    // it) as a 7-bit counter, bit-sliced: plane p holds bit p of the counters of
    // all samples, and adding a fragment is a ripple carry (or borrow) over the
    // planes.  The packed counters below (four 8-bit counters per word, the
    // reference's form) give each sample its winding modulo 128 as long as no
    // winding leaves [-128, 127], where a byte's carry would reach its
    // neighbour; with |w0| + (fragments) <= 127 that cannot happen, and the
    // planes give the same bits.
    uint32_t pl[7][WORDS];
#pragma unroll
    for (int q = 0; q < 7; ++q)
#pragma unroll
        for (int w = 0; w < WORDS; ++w) pl[q][w] = (((uint32_t)w0 >> q) & 1u) ? 0xFFFFFFFFu : 0u;
    int k = 0;
    walk([&](int32_t chg, const uint32_t (&m)[WORDS]) {
        ++k;
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
            uint32_t c = m[w];
            if (chg > 0) {
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    const uint32_t t = pl[q][w] & c;
                    pl[q][w] ^= c;
                    c = t;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 7; ++q) {
                    const uint32_t t = ~pl[q][w] & c;
                    pl[q][w] ^= c;
                    c = t;
                }
            }
        }
    });
    if ((w0 < 0 ? -w0 : w0) + k <= 127) {
#pragma unroll
        for (int w = 0; w < WORDS; ++w) {
            // nonzero: any bit of the 7-bit winding; even-odd: its lowest bit
            const uint32_t ret = fr == 0 ? (pl[0][w] | pl[1][w] | pl[2][w] | pl[3][w] | pl[4][w] | pl[5][w] | pl[6][w])
                                         : pl[0][w];
            merged[(size_t)g * WORDS + w] = ret;
        }
        return;
    }
    // packed 8-bit counters per mask bit, reduced to the 7-bit winding number
    const uint32_t init = 0x01010101u * (uint32_t)w0;
    uint32_t acc[WORDS][8];
#pragma unroll
    for (int w = 0; w < WORDS; ++w)
#pragma unroll
        for (int b = 0; b < 8; ++b) acc[w][b] = init;
    walk([&](int32_t chg, const uint32_t (&m)[WORDS]) {
#pragma unroll
        for (int w = 0; w < WORDS; ++w)
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint32_t bits = (m[w] >> b) & 0x01010101u;
                acc[w][b] = chg > 0 ? acc[w][b] + bits : acc[w][b] - bits;
            }
    });
#pragma unroll
    for (int w = 0; w < WORDS; ++w) {
        uint32_t ret = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            uint32_t wv = (0x80808080u + acc[w][b]) & 0x7f7f7f7fu;
            if (fr == 0) {
                wv |= wv >> 4;
                wv |= wv >> 2;
                wv |= wv >> 1;
            }
            ret |= (wv & 0x01010101u) << b;
        }
        merged[(size_t)g * WORDS + w] = ret;
    }
}

// ------------------------------------------------------------ resolve --
constexpr int kResolveWarps = 8;
constexpr int kResolveMaxBlocksPerSM = 4;

// The draw items of every resolve bin, in draw order: each item's index is
// placed in its bins' ranges (bin offsets from the scan of the counts that
// k_scan_mark took) by warp-aggregated atomic slots, and every bin's range
// is then sorted (item indices are the draw order).
__global__ void k_bin_scatter(FrameArgs a, const int4 *__restrict__ draw, const uint32_t *__restrict__ item_scene,
                              FrameCounters *ctr, const uint32_t *__restrict__ bin_off,
                              uint32_t *__restrict__ bin_fill, uint32_t *__restrict__ pval, uint32_t cap_pairs) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    // (not admitted: the pair buffer is too small, or a scan gave up; entries
    // not admitted: there are no items)
    const bool ok = admit(&ctr->need_pairs, &ctr->n_pairs, cap_pairs, &ctr->status);
    int nb = 0;
    uint32_t b0 = 0;
    if (ok && i < (int64_t)ctr->n_items) {
        const int4 it = draw[i];
        int W = a.W, H = a.H;
        uint32_t bin0 = 0;
        if (item_scene != nullptr) {
            const SceneInfo *sc = a.scenes + item_scene[i];
            W = sc->W;
            H = sc->H;
            bin0 = sc->bin_off;
        }
        nb = item_bins(it, W, H, a.bin_shift, bin0, &b0);
    }
    const int most = __reduce_max_sync(0xffffffffu, nb);
    for (int t = 0; t < most; ++t) {
        const bool act = t < nb;
        const uint32_t bin = act ? b0 + (uint32_t)t : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xffffffffu, bin);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (act && lane == leader) base = atomicAdd(bin_fill + bin, (uint32_t)__popc(peers));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (act) pval[bin_off[bin] + base + __popc(peers & ((1u << lane) - 1u))] = (uint32_t)i;
    }
}

// Pairs of every bin counted again from the draw list (a sized frame that
// changes its resolve tile after the scan-mark pass counted them).
__global__ void k_bin_count(FrameArgs a, const int4 *__restrict__ draw, const uint32_t *__restrict__ item_scene,
                            const FrameCounters *__restrict__ ctr, uint32_t *__restrict__ bin_count) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ctr->status != 0u || i >= (int64_t)ctr->n_items) return;
    const int4 it = draw[i];
    int W = a.W, H = a.H;
    uint32_t bin0 = 0;
    if (item_scene != nullptr) {
        const SceneInfo *sc = a.scenes + item_scene[i];
        W = sc->W;
        H = sc->H;
        bin0 = sc->bin_off;
    }
    uint32_t b0 = 0;
    const int nb = item_bins(it, W, H, a.bin_shift, bin0, &b0);
    for (int t = 0; t < nb; ++t) atomicAdd(bin_count + b0 + t, 1u);
}

// One warp per bin: its item indices sorted ascending by a bitonic network
// that compares in one direction only (stage k compares each element with
// its mirror in the k-block, then the half-cleaners), so that the missing
// elements past n behave as +infinity.  Bins of up to kBinSortRegs items are
// sorted in registers, K to a lane (element lane * K + r in register r:
// strides below K stay inside a lane, the others are shuffles), larger ones in
// place.  With rec_a set, the bin's resolve records are written in the same
// order: the item's colour, its columns and cell row within the bin's band
// (first | width << 16 | row << 29) and its merged sample mask (every sample
// for a span), so that the resolve reads each bin's items and masks as one
// contiguous run instead of gathering them.  (Widths stay below 2^13:
// viewports are at most 4096 pixels wide.)  Bound by the
// records' gathers.  On the 20,000-path 2048 x 2048 scene this kernel took 522 us
// with the network in shared memory (about 12,000 warp instructions for a bin of
// 528 items against 2,700), 264 with it in registers, 228 with the records
// gathered 4 x 32 at a time and 185 with one rolled body for the strides across
// lanes (the unrolled bodies of the six list lengths did not fit the instruction
// cache); all of the binning 695 -> 438 -> 398 -> 358, on a batch of 48 scenes
// 2180 -> 1498 -> 1356 -> 1318.  (2 and 8 x 32 at a time: 410 and 399, 1396 and
// 1383.)
constexpr int kBinSortWarps = 4;
constexpr int kBinSortRegs = 1024;
constexpr int kBinGather = 4;

template <int K>
__device__ __forceinline__ void warp_sort(uint32_t (&k)[K], int lane) {
    auto order = [](uint32_t &x, uint32_t &y) {
        const uint32_t lo = min(x, y), hi = max(x, y);
        x = lo;
        y = hi;
    };
    // within the lane
#pragma unroll
    for (int size = 2; size <= K; size *= 2) {
#pragma unroll
        for (int r = 0; r < K; ++r)
            if ((r ^ (size - 1)) > r) order(k[r], k[r ^ (size - 1)]);
#pragma unroll
        for (int j = size / 4; j > 0; j /= 2)
#pragma unroll
            for (int r = 0; r < K; ++r)
                if ((r ^ j) > r) order(k[r], k[r ^ j]);
    }
    // across 2, 4, .. 32 lanes (one body for all, which the instruction cache holds
    // beside the other list lengths')
#pragma unroll 1
    for (int lanes = 2; lanes <= 32; lanes *= 2) {
        const bool lo = (lane & (lanes / 2)) == 0;  // with register K - 1 - r of the mirrored lane
#pragma unroll
        for (int r = 0; r < (K + 1) / 2; ++r) {
            const uint32_t u = __shfl_xor_sync(0xffffffffu, k[K - 1 - r], lanes - 1);
            const uint32_t v = __shfl_xor_sync(0xffffffffu, k[r], lanes - 1);
            k[r] = (k[r] < u) == lo ? k[r] : u;
            if (K - 1 - r != r) k[K - 1 - r] = (k[K - 1 - r] < v) == lo ? k[K - 1 - r] : v;
        }
#pragma unroll 1
        for (int j = lanes / 4; j > 0; j /= 2) {
            const bool jlo = (lane & j) == 0;
#pragma unroll
            for (int r = 0; r < K; ++r) {
                const uint32_t u = __shfl_xor_sync(0xffffffffu, k[r], j);
                k[r] = (k[r] < u) == jlo ? k[r] : u;
            }
        }
#pragma unroll
        for (int j = K / 2; j > 0; j /= 2)
#pragma unroll
            for (int r = 0; r < K; ++r)
                if ((r ^ j) > r) order(k[r], k[r ^ j]);
    }
}

// Sorts the n <= 32 K items at src into dst (a padded place: bin_sort_at).
__device__ __forceinline__ uint32_t bin_sort_at(uint32_t e) { return e + (e >> 5); }
template <int K>
__device__ __forceinline__ void sort_in_registers(const uint32_t *__restrict__ src, uint32_t n, uint32_t *dst,
                                                  int lane) {
    uint32_t k[K];
#pragma unroll
    for (int r = 0; r < K; ++r) k[r] = r * 32 + lane < n ? src[r * 32 + lane] : 0xFFFFFFFFu;
    warp_sort<K>(k, lane);
#pragma unroll
    for (int r = 0; r < K; ++r) dst[bin_sort_at(lane * K + r)] = k[r];
    __syncwarp();
}
template <int MW>
struct MaskVec;
template <>
struct MaskVec<1> {
    using T = uint32_t;
    static __device__ __forceinline__ T all() { return 0xFFFFFFFFu; }
};
template <>
struct MaskVec<2> {
    using T = uint2;
    static __device__ __forceinline__ T all() { return make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu); }
};
template <>
struct MaskVec<4> {
    using T = uint4;
    static __device__ __forceinline__ T all() { return make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu); }
};

template <int MW>
__global__ void __launch_bounds__(kBinSortWarps * 32)
    k_bin_sort(const uint32_t *__restrict__ bin_off, int64_t nbins, uint32_t *__restrict__ pval,
               const FrameCounters *__restrict__ ctr, const int4 *__restrict__ draw,
               const uint32_t *__restrict__ merged, uint2 *__restrict__ rec_a,
               typename MaskVec<MW>::T *__restrict__ rec_m, int band_mask) {
    using MV = typename MaskVec<MW>::T;
    __shared__ uint32_t sk[kBinSortWarps][kBinSortRegs + kBinSortRegs / 32];
    if (ctr->status != 0u || ctr->n_pairs != ctr->need_pairs) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b = (int64_t)blockIdx.x * kBinSortWarps + warp;
    if (b >= nbins) return;
    const uint32_t beg = bin_off[b], n = bin_off[b + 1] - beg;
    if (n == 0u) return;
    uint32_t *const run = pval + beg, *const st = sk[warp];
    const bool regs = n <= (uint32_t)kBinSortRegs;
    if (n <= 32u) sort_in_registers<1>(run, n, st, lane);
    else if (n <= 64u) sort_in_registers<2>(run, n, st, lane);
    else if (n <= 128u) sort_in_registers<4>(run, n, st, lane);
    else if (n <= 256u) sort_in_registers<8>(run, n, st, lane);
    else if (n <= 512u) sort_in_registers<16>(run, n, st, lane);
    else if (regs) sort_in_registers<32>(run, n, st, lane);
    if (!regs) {
        int lp = 1;
        while ((1u << lp) < n) ++lp;  // 2^lp >= n
        const uint32_t half = 1u << (lp - 1);
        for (int lk = 1; lk <= lp; ++lk) {
            for (int lj = lk - 1; lj >= 0; --lj) {
                const uint32_t j = 1u << lj;
                for (uint32_t i = lane; i < half; i += 32) {
                    uint32_t x, y;
                    if (lj == lk - 1) {  // mirror within the 2j-block
                        const uint32_t blk = (i >> lj) << lk, off = i & (j - 1u);
                        x = blk + off;
                        y = blk + (2u * j - 1u) - off;
                    } else {
                        x = ((i >> lj) << (lj + 1)) + (i & (j - 1u));
                        y = x + j;
                    }
                    if (y < n) {
                        const uint32_t u = run[x], v = run[y];
                        if (u > v) {
                            run[x] = v;
                            run[y] = u;
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
    if (regs)
        for (uint32_t i = lane; i < n; i += 32) run[i] = st[bin_sort_at(i)];
    if (rec_a == nullptr) return;
    // the records of kBinGather x 32 items at a time: all their items' loads, then
    // all their masks', before the first is used
    for (uint32_t i0 = lane; i0 < n + lane; i0 += 32 * kBinGather) {
        int4 it[kBinGather];
        MV m[kBinGather];
#pragma unroll
        for (int r = 0; r < kBinGather; ++r) {
            const uint32_t i = min(i0 + 32 * r, n - 1);
            it[r] = __ldg(draw + (regs ? st[bin_sort_at(i)] : run[i]));
        }
#pragma unroll
        for (int r = 0; r < kBinGather; ++r) {
            m[r] = MaskVec<MW>::all();
            if (it[r].w != 0) m[r] = __ldg(reinterpret_cast<const MV *>(merged) + (it[r].w - 1));
        }
#pragma unroll
        for (int r = 0; r < kBinGather; ++r) {
            const uint32_t i = i0 + 32 * r;
            if (i >= n) break;
            const uint32_t ro = (uint32_t)(((it[r].x >> 16) / 2) & band_mask);  // the item's cell row within the band
            rec_a[beg + i] = make_uint2((uint32_t)it[r].z,
                                        ((uint32_t)it[r].x & 0xFFFFu) | ((uint32_t)it[r].y << 16) | (ro << 29));
            rec_m[beg + i] = m[r];
        }
    }
}

// Under sRGB blending the resolve carries linear colour values times 4096: a
// power of two changes no rounding, and the encode's bin is then the value's
// integer part.
constexpr float kLinScale = 4096.f;

// Shared-memory tables of the resolve.  The sRGB decode table is replicated
// twice (entry k of lane l at k * 2 + l % 2), which measures as fast as more
// replicas and leaves the room for 4 resolve blocks per SM.
struct SmemTables {
    float dec8r[256 * 2];  // x kLinScale
    float th[256];         // x kLinScale; th[255] is infinite
    uint8_t bin[4112];     // number of thresholds <= b / 4096; 255 at b = 4096
};

template <bool DECODE>
__device__ __forceinline__ void load_tables(SmemTables &T, const ResolveTables *rt) {
    if constexpr (DECODE)
        for (int i = threadIdx.x; i < 256 * 2; i += blockDim.x) T.dec8r[i] = rt->srgb_dec[i >> 1] * kLinScale;
    for (int i = threadIdx.x; i < 256; i += blockDim.x)
        T.th[i] = i < 255 ? rt->threshold[i] * kLinScale : __uint_as_float(0x7F800000u);
    for (int i = threadIdx.x; i < 1028; i += blockDim.x)
        reinterpret_cast<uint32_t *>(T.bin)[i] =
            i < 1024 ? reinterpret_cast<const uint32_t *>(rt->bin)[i] : 0xFFFFFFFFu;
}

// Float of an 8-bit value (the exponent trick: one add instead of a conversion).
__device__ __forceinline__ float u8f(uint32_t k) { return ffrom(0x4B000000u | k) - 8388608.f; }
__device__ __forceinline__ float lin8(uint32_t k) { return u8f(k) * (1.f / 255.f); }
// Integer part of v in [0, 8191].
__device__ __forceinline__ uint32_t floor_u13(float v) { return fbits(__fadd_rd(v, 8388608.f)) & 0x1FFFu; }

// 8-bit code of a linear value in [0, 1] (a hair above 1 allowed).
__device__ __forceinline__ uint32_t enc_lin(float v) { return floor_u13(v * 255.f + 0.5f); }

// sRGB encode of v = value x kLinScale, value in [0, 1] (a hair above 1
// allowed): the number of thresholds t[k] (the linear value at which the
// 8-bit code steps from k to k+1) that are <= the value.  The thresholds are
// at least 3.0e-4 apart, wider than the 1/4096 bins of `bin`, so a bin holds
// at most one of them: the count is the bin's base plus one comparison.
__device__ __forceinline__ uint32_t enc_srgb(const SmemTables &t, float v) {
    const uint32_t k = t.bin[floor_u13(v)];
    return k + (v >= t.th[k] ? 1u : 0u);
}

template <bool SRGB>
__device__ __forceinline__ float dec8(const SmemTables &t, uint32_t k, int lane) {
    if constexpr (SRGB) return t.dec8r[k * 2 + (lane & 1)];
    else return lin8(k);
}

template <bool SRGB>
__device__ __forceinline__ uint32_t enc8(const SmemTables &t, float v) {
    if constexpr (SRGB) return enc_srgb(t, v);
    else return enc_lin(v);
}

// An item's colour as its blends use it: premultiplied by alpha (linear,
// x kLinScale under sRGB), alpha squared and 1 - alpha.
struct Source {
    float r, g, b, aa, om;
};
__device__ __forceinline__ Source make_source(float r, float g, float b, float a) {
    return Source{r * a, g * a, b * a, a * a, 1.f - a};
}
template <bool SRGB>
__device__ __forceinline__ Source solid_source(const SmemTables &T, int lane, uint32_t c) {
    return make_source(dec8<SRGB>(T, c & 0xFF, lane), dec8<SRGB>(T, (c >> 8) & 0xFF, lane),
                       dec8<SRGB>(T, (c >> 16) & 0xFF, lane), lin8(c >> 24));
}

// Blend results are finite, never negative and at most a rounding above 1
// (sums of products of values in [0, 1] with weights a and 1 - a), except of
// paints whose map is not finite: CLAMP takes those to [0, 1], NaN to 0.
template <bool SRGB, bool CLAMP>
__device__ __forceinline__ uint32_t blend_sample(const SmemTables &t, int lane, uint32_t dv, const Source &s) {
    const float dr = dec8<SRGB>(t, dv & 0xFF, lane), dg = dec8<SRGB>(t, (dv >> 8) & 0xFF, lane),
                db = dec8<SRGB>(t, (dv >> 16) & 0xFF, lane);
    const float da = lin8(dv >> 24);
    float orr = s.r + dr * s.om;
    float og = s.g + dg * s.om;
    float ob = s.b + db * s.om;
    float oa = s.aa + da * s.om;
    if constexpr (CLAMP) {
        constexpr float one = SRGB ? kLinScale : 1.f;
        orr = fminf(fmaxf(orr, 0.f), one);
        og = fminf(fmaxf(og, 0.f), one);
        ob = fminf(fmaxf(ob, 0.f), one);
        oa = fminf(fmaxf(oa, 0.f), 1.f);
    }
    return enc8<SRGB>(t, orr) | (enc8<SRGB>(t, og) << 8) | (enc8<SRGB>(t, ob) << 16) | (enc_lin(oa) << 24);
}

// ---- gradient paints -----------------------------------------------------
// Gradient coordinate of pixel position (x, y): back to the scene through
// the reverse transform, then the entry's 2x3 map (ms_output_32.vert.glsl
// calc_color).
__device__ __forceinline__ float2 grad_coord(const FrameArgs &a, const float4 &w0, const float4 &w1, float x, float y) {
    const float rdx = (a.rev[0] * x + a.rev[3] * y) + a.rev[6];
    const float rdy = (a.rev[1] * x + a.rev[4] * y) + a.rev[7];
    const float rdz = (a.rev[2] * x + a.rev[5] * y) + a.rev[8];
    const float k = a.rev[12] / rdz;
    const float ox = a.rev[9] + k * rdx, oy = a.rev[10] + k * rdy;
    return make_float2((ox * w0.x + oy * w0.y) + w0.z, (ox * w0.w + oy * w1.x) + w1.y);
}

// Colour of gradient entry e at the centre of pixel (X, Y) for a draw item
// starting at column x0, w pixels wide: the coordinate interpolated along
// the item's row between its ends (the GL line primitive), the focal-point
// ratio c, and the ramp sampled at c (n - 1) texels past the first with
// linear filtering (ms_output_32.frag.glsl).  Texels are decoded from sRGB
// first under sRGB blending.
template <bool SRGB>
__device__ __forceinline__ float4 gradient_colour(const FrameArgs &a, const SmemTables &T, uint32_t e, int x0, int w,
                                                  int X, int Y, int lane) {
    const float4 w0 = a.grad_table[3 * e], w1 = a.grad_table[3 * e + 1], w2 = a.grad_table[3 * e + 2];
    const float yr = (float)Y + 0.5f;
    const float2 g0 = grad_coord(a, w0, w1, (float)x0, yr), g1 = grad_coord(a, w0, w1, (float)(x0 + w), yr);
    const float t = ((float)X + 0.5f - (float)x0) / (float)w;
    const float gx = g0.x * (1.f - t) + g1.x * t, gy = g0.y * (1.f - t) + g1.y * t;
    const float dx = gx - w2.x, dy = gy - w2.y;
    const float A = dx * dx + dy * dy, B = dx * w2.x + dy * w2.y;
    const float den = sqrtf(B * B + A * w2.z) - B;
    const float c = fminf(A * (den > 1e-6f ? 1.f / den : 0.f), 1.f);
    const int p = __float_as_int(w1.z);
    const float pos = c * (w1.w * 1024.f);
    const int i0 = (int)floorf(pos);
    const float f = pos - (float)i0;
    const int row = p >> 10, col = min((p & 1023) + i0, 1023), col1 = min(col + 1, 1023);
    const uint32_t t0 = a.grad_ramp[row * 1024 + col], t1 = a.grad_ramp[row * 1024 + col1];
    const float u = 1.f - f;
    return make_float4(dec8<SRGB>(T, t0 & 0xFF, lane) * u + dec8<SRGB>(T, t1 & 0xFF, lane) * f,
                       dec8<SRGB>(T, (t0 >> 8) & 0xFF, lane) * u + dec8<SRGB>(T, (t1 >> 8) & 0xFF, lane) * f,
                       dec8<SRGB>(T, (t0 >> 16) & 0xFF, lane) * u + dec8<SRGB>(T, (t1 >> 16) & 0xFF, lane) * f,
                       lin8(t0 >> 24) * u + lin8(t1 >> 24) * f);
}

// ---- resolve state -------------------------------------------------------
// A bin is a tile of 32 cells of 2x2 pixels; lane l of the warp resolving the
// bin owns cell l.  Every draw item covers whole cells, and the 4 pixels of a
// cell see the same items in the same order, so a cell keeps its 4 x S samples
// (pixel k = px.x * 2 + px.y, the merged masks' layout: bits [k S, (k + 1) S)
// of the cell's mask words) as a short list of (sample mask, RGBA8 colour)
// entries whose masks partition the samples.  An item blends each entry it
// touches once, splitting the entries it covers in part, and covered parts of
// equal colour become one entry: a cell typically holds 1-4 entries, and an
// entry often spans several pixels, so one blend serves many samples.  Entries
// 0..kCellCap-1 live in shared memory; a cell that needs more (rare: up to
// one per sample) keeps the rest in a global area owned by its warp and
// lane.  Every sample gets exactly the value the per-sample rule gives.
constexpr int kCellCap = 8;

// Draw items per window: kWin batches of 32.  (Resolve of the three scenes
// measured above: 2 batches 1807 / 209 / 5143, 4 batches 1832 / 209 / 5190, 8
// batches 1895 / 223 / 5433 us; on 64 paths 133, 121 and 127.)
constexpr int kWin = 4;

template <int MW, int CAP>
struct CellState {
    using MV = typename MaskVec<MW>::T;
    // entry j of lane l's cell, in column (l + j) % 32 (which puts the entries
    // of one cell into different banks)
    MV mask[CAP][32];
    uint32_t colour[CAP][32];
    uint32_t mine[kWin][32];  // per batch, the window's items covering lane l's cell
    uint32_t owner[32];       // a round's runs: the lane whose cell the run at a start belongs to
};

// Mask and colour of entry j of lane `lane`'s cell.  gx: the warp's global area
// of the entries past CAP (S the samples per pixel: up to 4 S entries); with
// LOCAL the entry is known to be among the first CAP.
template <int S, bool LOCAL, int CAP>
__device__ __forceinline__ typename MaskVec<S / 8>::T *entry_mask(CellState<S / 8, CAP> &w, uint32_t *gx, int j,
                                                                 int lane) {
    using MV = typename MaskVec<S / 8>::T;
    return LOCAL || j < CAP ? &w.mask[j][(lane + j) & 31] : reinterpret_cast<MV *>(gx) + (j - CAP) * 32 + lane;
}
template <int S, bool LOCAL, int CAP>
__device__ __forceinline__ uint32_t *entry_colour(CellState<S / 8, CAP> &w, uint32_t *gx, int j, int lane) {
    return LOCAL || j < CAP ? &w.colour[j][(lane + j) & 31]
                            : gx + ((4 * S - CAP) * (S / 8) + (j - CAP)) * 32 + lane;
}
__device__ __forceinline__ void get_mask(const uint32_t *p, uint32_t (&m)[1]) { m[0] = *p; }
__device__ __forceinline__ void get_mask(const uint2 *p, uint32_t (&m)[2]) {
    const uint2 v = *p;
    m[0] = v.x, m[1] = v.y;
}
__device__ __forceinline__ void get_mask(const uint4 *p, uint32_t (&m)[4]) {
    const uint4 v = *p;
    m[0] = v.x, m[1] = v.y, m[2] = v.z, m[3] = v.w;
}
__device__ __forceinline__ void put_mask(uint32_t *p, const uint32_t (&m)[1]) { *p = m[0]; }
__device__ __forceinline__ void put_mask(uint2 *p, const uint32_t (&m)[2]) { *p = make_uint2(m[0], m[1]); }
__device__ __forceinline__ void put_mask(uint4 *p, const uint32_t (&m)[4]) { *p = make_uint4(m[0], m[1], m[2], m[3]); }

// Cells [c0, c1) of cell row `ro` of a bin whose rows hold cpr cells (lane
// ro * cpr + c holds cell c of row ro) as a lane mask.
__device__ __forceinline__ uint32_t cell_bits(int c0, int c1, int cpr, int ro) {
    c0 = max(c0, 0);
    c1 = min(c1, cpr);
    if (c1 <= c0) return 0u;
    const uint32_t hi = c1 >= 32 ? 0xFFFFFFFFu : ((1u << c1) - 1u);
    return (hi & ~((1u << c0) - 1u)) << (ro * cpr);
}

// Bits of pixel k within mask word `wd` (cell masks of S samples per pixel).
template <int S>
__device__ __forceinline__ uint32_t pixel_word_bits(int wd, int k) {
    if constexpr (S == 32) return wd == k ? 0xFFFFFFFFu : 0u;
    else if constexpr (S == 16) return wd == (k >> 1) ? (0xFFFFu << (16 * (k & 1))) : 0u;
    else return 0xFFu << (8 * k);
}

// One item per lane (source src over the samples of mask m of the lane's
// cell; none if !have) in the multisample modes, called by the whole warp.
// The cells' entries differ in number (2.9 on average, 6 to 7 in the longest
// cell of a warp), so they are listed over the warp and blended in rounds of
// 32, one pair (cell, entry) per lane whoever owns the cell.  An entry keeps
// what the item does not cover and gives the covered samples, blended, to an
// entry of their colour: the covered parts of one cell that come out equal are
// found by a match over the round and become one entry.  The cell's entries
// are written back without gaps.  A cell whose pairs fall into two rounds is
// not merged this time: covered parts of split entries go past its last one.
//
// Bound by issue (73% of the schedulers' slots, 25 of 32 lanes active).  With
// a lane blending its own cell's entries one after the other and comparing all
// pairs of them for merges (10 lanes active), the resolve took 3430 us on the
// 20,000-path 2048 x 2048 scene, 390 us on a 3,300-path 1024 x 1024 page and
// 8350 us on a batch of 48 scenes; here 1832, 209 and 5190.  Sharing only the
// entries past the first took 2833, 287 and 6710; lanes as independent state
// machines 4340, 479 and 8966.
template <int S, bool SRGB, bool CLAMP, int CAP>
__device__ __forceinline__ void warp_apply(CellState<S / 8, CAP> &w, uint32_t *gx, int lane, int &n, bool have,
                                           const uint32_t (&m)[S / 8], const SmemTables &T, const Source &src) {
    constexpr int MW = S / 8;
    const int cnt = have ? n : 0;
    if (!__any_sync(0xffffffffu, cnt > 1)) {
        // every cell has one entry (open background, flat areas): its own lane
        // blends it, with nothing to merge but a colour that stays the same
        if (cnt == 1) {
            uint32_t em[MW], in[MW], rest[MW], any = 0u, part = 0u;
            get_mask(&w.mask[0][lane], em);
            const uint32_t old = w.colour[0][lane];
#pragma unroll
            for (int k = 0; k < MW; ++k) {
                in[k] = em[k] & m[k];
                rest[k] = em[k] & ~m[k];
                any |= in[k];
                part |= rest[k];
            }
            const uint32_t r = blend_sample<SRGB, CLAMP>(T, lane, old, src);
            if (any && !part) {
                w.colour[0][lane] = r;
            } else if (any && r != old) {
                put_mask(&w.mask[0][lane], rest);
                put_mask(entry_mask<S, (CAP > 1)>(w, gx, 1, lane), in);
                *entry_colour<S, (CAP > 1)>(w, gx, 1, lane) = r;
                n = 2;
            }
        }
        __syncwarp();
        return;
    }
    const int incl = (int)warp_incl_scan((uint32_t)cnt), first = incl - cnt;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int base = 0; base < total; base += 32) {
        // this cell's pairs of the round: lanes [lo, hi)
        const int lo = min(max(first - base, 0), 32), hi = min(max(incl - base, 0), 32);
        const bool mine = hi > lo, whole = mine && hi - lo == cnt;
        if (mine) w.owner[lo] = (uint32_t)lane;
        const uint32_t starts = __reduce_or_sync(0xffffffffu, mine ? 1u << lo : 0u);
        __syncwarp();
        const bool act = base + lane < total;
        const uint32_t lt = (1u << lane) - 1u;
        const int run = 31 - __clz((int)(starts & (lt | (1u << lane))));
        const int L = (int)w.owner[run];
        // the owner's first pair, entries and whether it is whole
        const uint32_t info = __shfl_sync(0xffffffffu, (uint32_t)first | ((uint32_t)n << 16) | (whole ? 1u << 31 : 0u), L);
        uint32_t mL[MW];
#pragma unroll
        for (int k = 0; k < MW; ++k) mL[k] = __shfl_sync(0xffffffffu, m[k], L);
        Source sL;
        sL.r = __shfl_sync(0xffffffffu, src.r, L);
        sL.g = __shfl_sync(0xffffffffu, src.g, L);
        sL.b = __shfl_sync(0xffffffffu, src.b, L);
        sL.aa = __shfl_sync(0xffffffffu, src.aa, L);
        sL.om = __shfl_sync(0xffffffffu, src.om, L);
        const int j = act ? base + lane - (int)(info & 0xFFFFu) : 0;
        const bool merge = (info >> 31) != 0u;
        uint32_t em[MW], rest = 0u, any = 0u;
        uint32_t old;
        if (!__any_sync(0xffffffffu, j >= CAP)) {
            get_mask(entry_mask<S, true>(w, gx, j, L), em);
            old = *entry_colour<S, true>(w, gx, j, L);
        } else {
            get_mask(entry_mask<S, false>(w, gx, j, L), em);
            old = *entry_colour<S, false>(w, gx, j, L);
        }
#pragma unroll
        for (int k = 0; k < MW; ++k) {
            any |= em[k] & mL[k];
            rest |= em[k] & ~mL[k];
        }
        const bool hit = act && any, keep = act && rest;
        const uint32_t r = blend_sample<SRGB, CLAMP>(T, lane, old, sL);
        // lanes of this cell, and among those before this one
        const uint32_t hits = __ballot_sync(0xffffffffu, hit);
        const uint32_t later = starts & ~(lt | (1u << lane));
        const uint32_t seg = (later ? (later & (0u - later)) - 1u : 0xFFFFFFFFu) & ~((1u << run) - 1u);
        const uint32_t same = __match_any_sync(0xffffffffu, r) & seg & hits;
        const int lead = merge ? __ffs(same) - 1 : lane;
        const bool put = hit && lead == lane;
        const uint32_t keeps = __ballot_sync(0xffffffffu, keep), puts = __ballot_sync(0xffffffffu, put);
        const uint32_t before = seg & lt;
        // the rest's and the covered part's places
        const int at = merge ? __popc(keeps & before) + __popc(puts & before) : j;
        const int slot = merge ? at + (keep ? 1 : 0)
                               : (keep ? (int)((info >> 16) & 0x7FFFu) + __popc(keeps & hits & before) : j);
        const bool move = keep && (hit || merge);
        uint32_t rm[MW], cm[MW];
#pragma unroll
        for (int k = 0; k < MW; ++k) {
            rm[k] = em[k] & ~mL[k];
            cm[k] = em[k] & mL[k];
        }
        const int to = __shfl_sync(0xffffffffu, slot, lead & 31);
        __syncwarp();  // (every pair is read: the cells' entries may be overwritten)
        auto write = [&](auto local) {
            constexpr bool LOCAL = decltype(local)::value;
            if (move) {
                put_mask(entry_mask<S, LOCAL>(w, gx, at, L), rm);
                *entry_colour<S, LOCAL>(w, gx, at, L) = old;
            }
            if (put) {
                put_mask(entry_mask<S, LOCAL>(w, gx, slot, L), cm);
                *entry_colour<S, LOCAL>(w, gx, slot, L) = r;
            }
            __syncwarp();
            if (hit && !put) {
                uint32_t *const d = reinterpret_cast<uint32_t *>(entry_mask<S, LOCAL>(w, gx, to, L));
#pragma unroll
                for (int k = 0; k < MW; ++k) atomicOr(d + k, cm[k]);
            }
        };
        if (!__any_sync(0xffffffffu, max(at, slot) >= CAP)) write(std::true_type{});
        else write(std::false_type{});
        if (mine) {
            const uint32_t range = (hi < 32 ? (1u << hi) - 1u : 0xFFFFFFFFu) & ~((1u << lo) - 1u);
            n = whole ? __popc(keeps & range) + __popc(puts & range) : n + __popc(keeps & hits & range);
        }
        __syncwarp();
    }
}

// Sample mask m (MW words) of resolve record p.
template <int MW>
__device__ __forceinline__ void load_mask(const uint32_t *__restrict__ rec_m, uint32_t p, uint32_t (&m)[MW]) {
    if constexpr (MW == 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(rec_m) + p);
        m[0] = v.x, m[1] = v.y, m[2] = v.z, m[3] = v.w;
    } else if constexpr (MW == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(rec_m) + p);
        m[0] = v.x, m[1] = v.y;
    } else {
        m[0] = __ldg(rec_m + p);
    }
}

// Exact mean of a pixel's samples: every decoded value x 2^36 is an integer,
// the 64-bit sums are exact, one rounding to float at the end.
struct PixelSum {
    long long r = 0, g = 0, b = 0, a = 0;
};
template <bool SRGB>
__device__ __forceinline__ void add_sample(PixelSum &p, const SmemTables &T, int lane, uint32_t v, int weight) {
    constexpr float unit = SRGB ? 68719476736.0f / kLinScale : 68719476736.0f;
    p.r += (long long)weight * (long long)(dec8<SRGB>(T, v & 0xFF, lane) * unit);
    p.g += (long long)weight * (long long)(dec8<SRGB>(T, (v >> 8) & 0xFF, lane) * unit);
    p.b += (long long)weight * (long long)(dec8<SRGB>(T, (v >> 16) & 0xFF, lane) * unit);
    p.a += (long long)weight * (long long)(lin8(v >> 24) * 68719476736.0f);
}

template <bool SRGB>
__device__ __forceinline__ uint32_t encode_mean(const SmemTables &T, const PixelSum &p, double scale) {
    constexpr float k = SRGB ? kLinScale : 1.f;
    const float ar = (float)((double)p.r * scale) * k, ag = (float)((double)p.g * scale) * k;
    const float ab = (float)((double)p.b * scale) * k, aa = (float)((double)p.a * scale);
    return enc8<SRGB>(T, ar) | (enc8<SRGB>(T, ag) << 8) | (enc8<SRGB>(T, ab) << 16) | (enc_lin(aa) << 24);
}

// Applies the window's items to the warp's cells, every lane its own cell's
// items in order, in the multisample modes.
template <int S, bool SRGB, int CAP, bool GRAD, class NextItem>
__device__ __forceinline__ void apply_items(const FrameArgs &a, CellState<S / 8, CAP> &w, uint32_t *gx, int lane,
                                            int &n_io, const SmemTables &T, const uint2 *__restrict__ rec_a,
                                            const uint32_t *__restrict__ rec_m, uint32_t base, int X0, int y0,
                                            NextItem &&next_item) {
    constexpr int MW = S / 8;
    int n = n_io;
    int q = next_item();
    uint32_t m[MW];
    uint2 r = make_uint2(0u, 0u);
    if (q >= 0) {
        r = __ldg(rec_a + base + q);
        load_mask<MW>(rec_m, base + q, m);
    }
    while (__any_sync(0xffffffffu, q >= 0)) {
        const int qn = next_item();  // the next item, loaded while the current one is applied
        uint32_t mn[MW];
        uint2 rn = make_uint2(0u, 0u);
        if (qn >= 0) {
            rn = __ldg(rec_a + base + qn);
            load_mask<MW>(rec_m, base + qn, mn);
        }
        bool have = q >= 0;
        const bool paint = GRAD && have && r.x - 1u < a.n_grad;
        Source src{};
        if (have && !paint) {
            uint32_t full = 0xFFFFFFFFu;
#pragma unroll
            for (int k = 0; k < MW; ++k) full &= m[k];
            if ((r.x >> 24) == 255u && full == 0xFFFFFFFFu) {
                // opaque over every sample: src * 1 + dst * 0 is the source
                // whatever dst holds, and its code is the source's own, so one
                // entry stands for all (the per-sample blends and the merge
                // give the same)
                w.mask[0][lane] = MaskVec<MW>::all();
                w.colour[0][lane] = r.x;
                n = 1;
                have = false;
            } else {
                src = solid_source<SRGB>(T, lane, r.x);
            }
        }
        if constexpr (!GRAD) {
            warp_apply<S, SRGB, false, CAP>(w, gx, lane, n, have, m, T, src);
        } else {
            // a paint has a colour per pixel: one application per pixel
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                uint32_t mk[MW], any = 0u;
#pragma unroll
                for (int wd = 0; wd < MW; ++wd) {
                    mk[wd] = paint ? m[wd] & pixel_word_bits<S>(wd, k) : m[wd];
                    any |= mk[wd];
                }
                const bool hk = have && any && (paint || k == 0);
                if (!__any_sync(0xffffffffu, hk)) continue;
                if (hk && paint) {
                    const float4 gc = gradient_colour<SRGB>(a, T, r.x - 1u, (int)(int16_t)(r.y & 0xFFFFu),
                                                            (int)((r.y >> 16) & 0x1FFFu), X0 + (k >> 1), y0 + (k & 1),
                                                            lane);
                    src = make_source(gc.x, gc.y, gc.z, gc.w);
                }
                warp_apply<S, SRGB, true, CAP>(w, gx, lane, n, hk, mk, T, src);
            }
        }
        q = qn;
        r = rn;
#pragma unroll
        for (int k = 0; k < MW; ++k) m[k] = mn[k];
    }
    n_io = n;
}

// One warp per bin.  The bin's resolve records (merged fragments and spans
// in draw-list order: colour, columns, sample mask) are taken kWin x 32 at a
// time; a 32 x 32 ballot transpose of each batch's cell sets gives every
// lane the window's items covering its cell, which are applied in order, the
// k-th of every lane together (a warp's steps are the most items over one of
// its cells in the window, not in each batch).
// The record of the lane's next item is loaded while it applies the current
// one.  Then every pixel is averaged over its samples.
template <int S, bool MS, bool SRGB, int CAP, bool GRAD>
__device__ __forceinline__ void resolve_bin(const FrameArgs &a, const uint2 *__restrict__ rec_a,
                                            const uint32_t *__restrict__ rec_m,
                                            const uint32_t *__restrict__ bstart, const uint32_t *__restrict__ bend,
                                            uint32_t *__restrict__ image, uint32_t *__restrict__ gx,
                                            const SmemTables &T, CellState<S / 8, CAP> &w, const int lane,
                                            const uint32_t b) {
    constexpr int MW = S / 8;
    // the bin's scene: viewport, first bin, image
    int W = a.W, H = a.H;
    uint32_t lb = b;
    int64_t image_off = 0;
    if (a.scenes != nullptr) {
        int lo = 0, hi = a.n_scenes - 1;  // last scene whose bin_off <= b
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.scenes[mid].bin_off <= b) lo = mid;
            else hi = mid - 1;
        }
        const SceneInfo *sc = a.scenes + lo;
        W = sc->W;
        H = sc->H;
        lb = b - sc->bin_off;
        image_off = sc->image_off;
        image += image_off;
    }
    // the bin: band `brow` of 64 >> sh cell rows, tile `tile` of 1 << sh
    // columns; lane l: cell l % cpr of the band's row l / cpr
    const int sh = a.bin_shift, cs = sh - 1, cpr = 1 << cs;  // cells per row: 1 << cs
    const int ntx = bin_cols(W, sh);
    const int brow = (int)(lb / ntx), tile = (int)(lb % ntx);
    const int tx0 = tile << sh;
    const int y0 = ((brow << (kBinShift - sh)) + (lane >> cs)) * 2;
    const int X0 = tx0 + 2 * (lane & (cpr - 1));  // this lane's cell: columns X0, X0 + 1, rows y0, y0 + 1
    // state: one white entry over every sample (multisample), or one colour
    // per pixel (single-sample output)
    int n = 1;
    uint32_t pc[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
    if constexpr (MS) {
        w.mask[0][lane] = MaskVec<MW>::all();
        w.colour[0][lane] = 0xFFFFFFFFu;
    }
    const uint32_t beg = bstart[b], fin = bend[b];
    for (uint32_t base = beg; base < fin; base += kWin * 32) {
        __syncwarp();
        const int nb = (int)min((uint32_t)kWin, (fin - base + 31) / 32);  // batches in this window
        // the columns of the window's items (lane l: item 32 c + l of batch
        // c), all loads issued before the first is used
        uint32_t xws[kWin];
#pragma unroll
        for (int c = 0; c < kWin; ++c) {
            const uint32_t p = base + c * 32 + lane;
            xws[c] = c < nb && p < fin ? __ldg(&rec_a[p].y) : 0u;
        }
#pragma unroll
        for (int c = 0; c < kWin; ++c) {
            if (c >= nb) break;
            uint32_t cm = 0u;  // cells of this lane's item (a fragment: one cell of 2 columns)
            {
                const int x = (int)(xws[c] & 0xFFFFu);
                const int xb = min(x + (int)((xws[c] >> 16) & 0x1FFFu), W);
                cm = xb > x ? cell_bits((x - tx0) >> 1, (xb - tx0 + 1) >> 1, cpr, (int)(xws[c] >> 29)) : 0u;
            }
            // bit q of lane L's word: staged item q covers cell L (a transpose
            // of the 32 x 32 bit matrix of cell sets)
            uint32_t mine = 0u;
#pragma unroll
            for (int L = 0; L < 32; ++L) {
                const uint32_t bm = __ballot_sync(0xffffffffu, (cm >> L) & 1u);
                if (lane == L) mine = bm;
            }
            w.mine[c][lane] = mine;
        }
        __syncwarp();
        // this lane's items in draw order: batch cw, remaining bits
        int cw = 0;
        uint32_t bits = w.mine[0][lane];
        auto next_item = [&]() -> int {
            while (bits == 0u && ++cw < nb) bits = w.mine[cw][lane];
            if (bits == 0u) return -1;
            const int q = cw * 32 + __ffs(bits) - 1;
            bits &= bits - 1u;
            return q;
        };
        if constexpr (MS) {
            apply_items<S, SRGB, CAP, GRAD>(a, w, gx, lane, n, T, rec_a, rec_m, base, X0, y0, next_item);
        } else {
            // single-sample output: alpha x coverage per pixel, the next
            // item's record loaded while the current one is applied
            int q = next_item();
            uint32_t m[MW];
            uint2 r = make_uint2(0u, 0u);
            if (q >= 0) {
                r = __ldg(rec_a + base + q);
                load_mask<MW>(rec_m, base + q, m);
            }
            while (q >= 0) {
                const int qn = next_item();
                uint32_t mn[MW];
                uint2 rn = make_uint2(0u, 0u);
                if (qn >= 0) {
                    rn = __ldg(rec_a + base + qn);
                    load_mask<MW>(rec_m, base + qn, mn);
                }
                const uint32_t c = r.x;
                const bool paint = GRAD && c - 1u < a.n_grad;
                float4 col = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!paint)
                    col = make_float4(dec8<SRGB>(T, c & 0xFF, lane), dec8<SRGB>(T, (c >> 8) & 0xFF, lane),
                                      dec8<SRGB>(T, (c >> 16) & 0xFF, lane), lin8(c >> 24));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int cov = 0;
#pragma unroll
                    for (int wd = 0; wd < MW; ++wd) cov += __popc(m[wd] & pixel_word_bits<S>(wd, k));
                    if (cov == 0) continue;
                    if constexpr (GRAD) {
                        if (paint)
                            col = gradient_colour<SRGB>(a, T, c - 1u, (int)(int16_t)(r.y & 0xFFFFu),
                                                        (int)((r.y >> 16) & 0x1FFFu), X0 + (k >> 1), y0 + (k & 1), lane);
                    }
                    const float ak = col.w * ((float)cov / (float)S);
                    pc[k] = blend_sample<SRGB, GRAD>(T, lane, pc[k], make_source(col.x, col.y, col.z, ak));
                }
                q = qn;
                r = rn;
#pragma unroll
                for (int k = 0; k < MW; ++k) m[k] = mn[k];
            }
        }
    }
    __syncwarp();
    // per-pixel means: pixel k = px * 2 + py of the cell, at column X0 + px,
    // row y0 + py
    const double scale = 1.0 / (68719476736.0 * (double)(MS ? S : 1));
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        PixelSum p;
        if constexpr (MS) {
            if (n == 1 && a.sums == nullptr) {  // one colour: its mean encodes to its own code
                out[k] = w.colour[0][lane];
                continue;
            }
            for (int j = 0; j < n; ++j) {
                uint32_t em[MW];
                get_mask(entry_mask<S, false>(w, gx, j, lane), em);
                int cov = 0;
#pragma unroll
                for (int wd = 0; wd < MW; ++wd) cov += __popc(em[wd] & pixel_word_bits<S>(wd, k));
                if (cov) add_sample<SRGB>(p, T, lane, *entry_colour<S, false>(w, gx, j, lane), cov);
            }
        } else {
            add_sample<SRGB>(p, T, lane, pc[k], 1);
        }
        const int X = X0 + (k >> 1), Y = y0 + (k & 1);
        if (a.sums != nullptr) {  // a pass of a 256-sample frame: exact sums, encoded after the last pass
            if (X < W && Y < H) {
                longlong2 *q = reinterpret_cast<longlong2 *>(a.sums) + 2 * (image_off + (int64_t)Y * W + X);
                const longlong2 q0 = q[0], q1 = q[1];
                q[0] = make_longlong2(q0.x + p.r, q0.y + p.g);
                q[1] = make_longlong2(q1.x + p.b, q1.y + p.a);
            }
            continue;
        }
        out[k] = encode_mean<SRGB>(T, p, scale);
    }
    if (a.sums != nullptr) return;
#pragma unroll
    for (int py = 0; py < 2; ++py) {
        const int Y = y0 + py;
        if (Y >= H) continue;
        const int64_t pix = (int64_t)Y * W + X0;
        if (X0 + 1 < W && (reinterpret_cast<uintptr_t>(image + pix) & 7u) == 0) {
            *reinterpret_cast<uint2 *>(image + pix) = make_uint2(out[py], out[2 + py]);
        } else {
            if (X0 < W) image[pix] = out[py];
            if (X0 + 1 < W) image[pix + 1] = out[2 + py];
        }
    }
}

// Persistent resolve: each warp takes bins from the frame's bin queue until
// it is empty; a warp's overflow entry area is reused from bin to bin.
template <int S, bool MS, bool SRGB, bool GRAD>
__device__ __forceinline__ void resolve_persistent(const FrameArgs &a, const uint2 *__restrict__ rec_a,
                                                   const uint32_t *__restrict__ rec_m,
                                                   const uint32_t *__restrict__ bstart,
                                                   const uint32_t *__restrict__ bend, uint32_t *__restrict__ image,
                                                   uint32_t *__restrict__ overflow, FrameCounters *__restrict__ ctr) {
    constexpr int CAP = MS ? kCellCap : 1;
    // sizes not admitted or a scan that gave up: the bin offsets run past the
    // records, and the frame is rendered again or reported
    if (ctr->status != 0u) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemTables &T = *reinterpret_cast<SmemTables *>(smem_raw);
    load_tables<SRGB>(T, a.rtables);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    CellState<S / 8, CAP> &w = reinterpret_cast<CellState<S / 8, CAP> *>(smem_raw + sizeof(SmemTables))[warp];
    const int64_t slot = (int64_t)blockIdx.x * kResolveWarps + warp;
    // entries past CAP: up to one per sample of the cell
    uint32_t *gx = MS ? overflow + slot * (int64_t)(4 * S - CAP) * (S / 8 + 1) * 32 : nullptr;
    for (;;) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(&ctr->bin_queue, 1u);
        b = __shfl_sync(0xffffffffu, b, 0);
        if ((int64_t)b >= a.n_bins) break;
        resolve_bin<S, MS, SRGB, CAP, GRAD>(a, rec_a, rec_m, bstart, bend, image, gx, T, w, lane, b);
        __syncwarp();
    }
}

// 3 blocks per SM where cells keep entries (76 registers; 4 blocks spill: 2080
// against 1832 us), 4 where they keep a colour per pixel.
template <int S, bool MS, bool SRGB>
__global__ void __launch_bounds__(kResolveWarps * 32, MS ? 3 : 4) k_resolve(FrameArgs a, const uint2 *__restrict__ rec_a,
                                                                 const uint32_t *__restrict__ rec_m,
                                                                 const uint32_t *__restrict__ bstart,
                                                                 const uint32_t *__restrict__ bend,
                                                                 uint32_t *__restrict__ image,
                                                                 uint32_t *__restrict__ overflow,
                                                                 FrameCounters *__restrict__ ctr) {
    resolve_persistent<S, MS, SRGB, false>(a, rec_a, rec_m, bstart, bend, image, overflow, ctr);
}

// With gradient paints: registers capped so that two blocks stay resident
// (the per-pixel paint would otherwise take more).
template <int S, bool MS, bool SRGB>
__global__ void __launch_bounds__(kResolveWarps * 32, 2)
    k_resolve_grad(FrameArgs a, const uint2 *__restrict__ rec_a, const uint32_t *__restrict__ rec_m,
                   const uint32_t *__restrict__ bstart,
                   const uint32_t *__restrict__ bend, uint32_t *__restrict__ image, uint32_t *__restrict__ overflow,
                   FrameCounters *__restrict__ ctr) {
    resolve_persistent<S, MS, SRGB, true>(a, rec_a, rec_m, bstart, bend, image, overflow, ctr);
}

// The image of a 256-sample frame from its passes' fixed-point sample sums
// (the same averaging and encoding as the resolve's last step).
template <bool SRGB>
__global__ void k_encode_sums(FrameArgs a, const long long *__restrict__ sums, uint32_t *__restrict__ image,
                              int64_t npix) {
    __shared__ SmemTables T;
    load_tables<false>(T, a.rtables);
    __syncthreads();
    const double scale = 1.0 / (68719476736.0 * 256.0);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += (int64_t)gridDim.x * blockDim.x) {
        const longlong2 q0 = reinterpret_cast<const longlong2 *>(sums)[2 * i];
        const longlong2 q1 = reinterpret_cast<const longlong2 *>(sums)[2 * i + 1];
        PixelSum p;
        p.r = q0.x, p.g = q0.y, p.b = q1.x, p.a = q1.y;
        image[i] = encode_mean<SRGB>(T, p, scale);
    }
}

// Exhaustive check of enc_srgb against the definition (the number of
// thresholds <= the clamped value, by binary search) over every float bit
// pattern in [lo, hi).
__global__ void k_selftest_encode(const ResolveTables *__restrict__ rt, uint32_t lo, uint32_t hi,
                                  unsigned long long *__restrict__ bad) {
    __shared__ SmemTables T;
    load_tables<false>(T, rt);
    __syncthreads();
    unsigned long long local = 0;
    for (uint64_t u = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < hi;
         u += (uint64_t)gridDim.x * blockDim.x) {
        const float v = fmax_r(__uint_as_float((uint32_t)u), 0.f);
        const float c = fmin_r(v, 1.f);
        int a = 0, b = 255;  // thresholds th[0..254] ascending: count those <= c
        while (a < b) {
            const int m = (a + b) >> 1;
            if (rt->threshold[m] <= c) a = m + 1;
            else b = m;
        }
        if (enc_srgb(T, v * kLinScale) != (uint32_t)a) ++local;
    }
    if (local) atomicAdd(bad, local);
}

// ---------------------------------------------------- scene upload --
// Checks of spr_validate_scene and unifyCurveVertexOrder (ras_base.cpp:523-569)
// on the device.  flags: bit 0 = invalid scene, bit 1 = vertex ranges of
// consecutive curves not disjoint and ascending (the in-place reversal would
// depend on the curve order: the host path handles such scenes).
__global__ void k_scene_vertices(const uint32_t *__restrict__ vpid, uint32_t V, uint32_t P,
                                 uint32_t *__restrict__ vmap, uint32_t *__restrict__ flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    vmap[i] = i;
    if (vpid[i] >= P) atomicOr(flags, 1u);
}

__global__ void k_scene_curves(const uint32_t *__restrict__ cvp, const uint8_t *__restrict__ ctype,
                               const uint32_t *__restrict__ cpid, const float *__restrict__ arcw, uint32_t C,
                               uint32_t V, uint32_t P, float2 *__restrict__ vert, uint32_t *__restrict__ vmap,
                               CurveDesc *__restrict__ cd, uint32_t *__restrict__ flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C) return;
    const int type = ctype[i];
    const bool known = type == kLinear || type == kQuad || type == kCubic || type == kRational;
    const int vn = type & 7;
    const uint32_t p = cvp[i], pid = cpid[i];
    bool bad = !known || (type == kRational && arcw == nullptr) || (uint64_t)p + (uint64_t)vn > V || pid >= P ||
               (i > 0 && pid < cpid[i - 1]);
    if (bad) {
        atomicOr(flags, 1u);
        return;
    }
    if (i + 1 < C && (uint64_t)p + (uint64_t)vn > (uint64_t)cvp[i + 1]) atomicOr(flags, 2u);
    // reverse unless (y_first, x_first) < (y_last, x_last) as float bit patterns
    const float2 vf = vert[p], vl = vert[p + vn - 1];
    const uint32_t bxf = __float_as_uint(vf.x), byf = __float_as_uint(vf.y);
    const uint32_t bxl = __float_as_uint(vl.x), byl = __float_as_uint(vl.y);
    const uint32_t rev = (byf < byl || (byf == byl && bxf < bxl)) ? 0u : 1u;
    CurveDesc d;
    d.vpos = p;
    d.pid = pid;
    d.w = type == kRational ? arcw[i] : 0.f;
    d.type = (uint32_t)type | (rev << 8);
    cd[i] = d;
    if (rev) {
        for (int k = 0; k < vn / 2; ++k) {
            const float2 t = vert[p + k];
            vert[p + k] = vert[p + vn - 1 - k];
            vert[p + vn - 1 - k] = t;
        }
        for (int k = 0; k < vn; ++k) vmap[p + k] = p + vn - 1 - k;
    }
}

__global__ void k_fill(uint32_t *image, int64_t n, uint32_t v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) image[i] = v;
}

__global__ void k_decode_keys(const uint64_t *__restrict__ skey, int64_t n, int nrows, int32_t *__restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = key_from_local((uint32_t)(skey[i] & 0xFFFFFFu), nrows);
}


int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 152;
    }
    return n;
}

// Shared memory of a resolve block: the tables and one cell state per warp.
template <int S>
size_t resolve_smem(bool ms) {
    return sizeof(SmemTables) + (size_t)kResolveWarps * (ms ? sizeof(CellState<S / 8, kCellCap>) : sizeof(CellState<S / 8, 1>));
}
size_t resolve_smem(int S, bool ms) {
    return S == 8 ? resolve_smem<8>(ms) : (S == 16 ? resolve_smem<16>(ms) : resolve_smem<32>(ms));
}

// Resolve blocks per SM: as many as fit in shared memory (at most 4), or
// the tuned count if lower.
int resolve_bps(const FrameArgs &a) {
    const int fit = std::max(1, std::min<int>(kResolveMaxBlocksPerSM, (int)((227u << 10) / resolve_smem(a.S, a.ms_output))));
    return a.resolve_bps >= 1 && a.resolve_bps < fit ? a.resolve_bps : fit;
}

int64_t resolve_blocks(const FrameArgs &a) {
    const int64_t need = (a.n_bins + kResolveWarps - 1) / kResolveWarps;
    return std::max<int64_t>(1, std::min<int64_t>(need, (int64_t)sm_count() * resolve_bps(a)));
}

// The frame's resolve kernel.  Gradient paints get their own instantiations: the
// per-pixel paint costs registers that plain frames should not pay for.
using ResolveKernel = void (*)(FrameArgs, const uint2 *, const uint32_t *, const uint32_t *, const uint32_t *,
                               uint32_t *, uint32_t *, FrameCounters *);
template <int S, bool MS, bool SRGB>
ResolveKernel resolve_kernel(bool paints) {
    return paints ? k_resolve_grad<S, MS, SRGB> : k_resolve<S, MS, SRGB>;
}
template <int S>
ResolveKernel resolve_kernel(bool ms, bool srgb, bool paints) {
    if (ms) return srgb ? resolve_kernel<S, true, true>(paints) : resolve_kernel<S, true, false>(paints);
    return srgb ? resolve_kernel<S, false, true>(paints) : resolve_kernel<S, false, false>(paints);
}
ResolveKernel resolve_kernel(const FrameArgs &a) {
    const bool ms = a.ms_output != 0, srgb = a.srgb != 0, paints = a.grad_table != nullptr;
    if (a.S == 8) return resolve_kernel<8>(ms, srgb, paints);
    if (a.S == 16) return resolve_kernel<16>(ms, srgb, paints);
    return resolve_kernel<32>(ms, srgb, paints);
}

}  // namespace

int launch_transform(const FrameArgs &a, float2 *tvert, uint32_t *path_flags, cudaStream_t s) {
    if (a.V <= 0) return 0;
    k_transform<<<grid_for(a.V), kThreads, 0, s>>>(a, tvert, path_flags);
    return 1;
}

// Curves a block of k_curve_emit takes: about 5 blocks per SM, so that few
// curves still reach every SM, up to the 128 that a block holds, which pack
// their chains best.  Emission + fragments of the measured scenes, us at
// 8 / 32 / 128 curves (solvers still in one list): 1,378 curves 304 / 309 / 395, 24 k 288 / 167 / 169,
// 158 k 386 / 167 / 118, 1.74 M 3972 / 1488 / 783.
static int emit_curves(int C) {
    int n = 8;
    while (n < kEmitCurves && n * 768 < C) n *= 2;
    return n;
}

int launch_curve_count(const FrameArgs &a, const float2 *tvert, const uint32_t *path_flags, uint8_t *vis,
                       uint32_t *counts, cudaStream_t s) {
    if (a.C <= 0 && a.P <= 0) return 0;
    k_curve_count<<<grid_for(std::max(a.C, a.P)), kThreads, 0, s>>>(a, tvert, path_flags, vis, counts);
    return 1;
}

int launch_emit_keys(const FrameArgs &a, const uint32_t *counts, uint32_t *key, uint32_t *val, cudaStream_t s) {
    if (a.C <= 0) return 0;
    k_emit_keys<<<grid_for(a.C), kThreads, 0, s>>>(a, counts, key, val);
    return 1;
}

int launch_curve_emit(const FrameArgs &a, const float2 *tvert, const uint8_t *vis, const uint32_t *offsets,
                       const uint32_t *order, float *scratch, int2 *entries, int64_t cap_nf, FrameCounters *ctr,
                       cudaStream_t s) {
    if (a.C <= 0) return 0;
    const int per_block = emit_curves(a.C);
    // few curves leave issue slots idle, which two bisection steps at a time use;
    // with more of them they only cost (1,378 curves 234 -> 216 us, but 24 k
    // 280 -> 288 and 1.74 M 759 -> 859)
    const auto kernel = per_block <= 8 ? k_curve_emit<true> : k_curve_emit<false>;
    kernel<<<grid_for(a.C, per_block), kEmitThreads, 0, s>>>(a, per_block, tvert, vis, offsets, order, scratch, entries,
                                                             cap32(cap_nf), ctr);
    return 1;
}

int launch_fragment(const FrameArgs &a, const float2 *tvert, const int2 *entries, int64_t cap_nf,
                    const FrameCounters *ctr, int32_t *key, uint32_t *pidw, int8_t *wn, uint32_t *mask,
                    uint64_t *sort_key, uint32_t *sort_val, uint64_t *mark_words, cudaStream_t s) {
    const int64_t n_mark = scan_mark_status_words(cap_nf);
    const unsigned g = grid_for(std::max(cap_nf, n_mark));
    if (a.S == 8)
        k_fragment<8><<<g, kThreads, 0, s>>>(a, tvert, entries, ctr, key, pidw, wn, mask, sort_key, sort_val,
                                            mark_words, n_mark);
    else if (a.S == 16)
        k_fragment<16><<<g, kThreads, 0, s>>>(a, tvert, entries, ctr, key, pidw, wn, mask, sort_key, sort_val,
                                            mark_words, n_mark);
    else
        k_fragment<32><<<g, kThreads, 0, s>>>(a, tvert, entries, ctr, key, pidw, wn, mask, sort_key, sort_val,
                                            mark_words, n_mark);
    return 1;
}

int64_t scan_mark_status_words(int64_t cap_nf) { return 2 * std::max<int64_t>(1, (cap_nf + kMarkTile - 1) / kMarkTile); }

int launch_scan_mark(const FrameArgs &a, int64_t cap_nf, const uint64_t *skey, int8_t *wn_scan, int4 *draw, uint32_t *heads, uint32_t *item_scene, uint32_t *bin_count,
                     FrameCounters *counters, uint64_t *tile_status, uint32_t spin_cap, cudaStream_t s) {
    const int64_t words = scan_mark_status_words(cap_nf);
    k_scan_mark<<<(unsigned)(words / 2), kMarkThreads, 0, s>>>(a, skey, wn_scan, draw, heads, item_scene,
                                                               bin_count, counters, tile_status, tile_status + words / 2,
                                                               spin_cap);
    return 1;
}

int launch_stencil(const FrameArgs &a, int64_t cap_nf, const FrameCounters *ctr, const uint64_t *skey,
                   const uint32_t *perm, const uint32_t *mask, const int8_t *wn_scan, const uint32_t *heads,
                   uint32_t *merged, cudaStream_t s) {
    if (cap_nf <= 0) return 0;
    const unsigned g = grid_for(cap_nf);
    if (a.S == 8)
        k_stencil<8><<<g, kThreads, 0, s>>>(a, ctr, skey, perm, mask, wn_scan, heads, merged);
    else if (a.S == 16)
        k_stencil<16><<<g, kThreads, 0, s>>>(a, ctr, skey, perm, mask, wn_scan, heads, merged);
    else
        k_stencil<32><<<g, kThreads, 0, s>>>(a, ctr, skey, perm, mask, wn_scan, heads, merged);
    return 1;
}

int launch_bin_scatter(const FrameArgs &a, const int4 *draw, const uint32_t *item_scene, int64_t cap_items,
                       int64_t cap_pairs, FrameCounters *ctr, const uint32_t *bin_off, uint32_t *bin_fill, uint32_t *pval,
                       cudaStream_t s) {
    if (cap_items <= 0) return 0;
    k_bin_scatter<<<grid_for(cap_items), kThreads, 0, s>>>(a, draw, item_scene, ctr, bin_off, bin_fill, pval,
                                                         cap32(cap_pairs));
    return 1;
}

int launch_bin_count(const FrameArgs &a, const int4 *draw, const uint32_t *item_scene, int64_t cap_items,
                     const FrameCounters *ctr, uint32_t *bin_count, cudaStream_t s) {
    if (cap_items <= 0) return 0;
    k_bin_count<<<grid_for(cap_items), kThreads, 0, s>>>(a, draw, item_scene, ctr, bin_count);
    return 1;
}

int launch_bin_sort(const uint32_t *bin_off, int64_t nbins, uint32_t *pval, const FrameCounters *ctr, int S,
                    int bin_shift, const int4 *draw, const uint32_t *merged, uint2 *rec_a, uint32_t *rec_m,
                    cudaStream_t s) {
    const int band_mask = (1 << (kBinShift - bin_shift)) - 1;  // cell rows per band - 1
    if (nbins <= 0) return 0;
    const unsigned g = (unsigned)((nbins + kBinSortWarps - 1) / kBinSortWarps);
    if (S == 8)
        k_bin_sort<1><<<g, kBinSortWarps * 32, 0, s>>>(bin_off, nbins, pval, ctr, draw, merged, rec_a, rec_m, band_mask);
    else if (S == 16)
        k_bin_sort<2><<<g, kBinSortWarps * 32, 0, s>>>(bin_off, nbins, pval, ctr, draw, merged, rec_a,
                                                        reinterpret_cast<uint2 *>(rec_m), band_mask);
    else
        k_bin_sort<4><<<g, kBinSortWarps * 32, 0, s>>>(bin_off, nbins, pval, ctr, draw, merged, rec_a,
                                                        reinterpret_cast<uint4 *>(rec_m), band_mask);
    return 1;
}


// Resident resolve blocks per SM (registers or shared memory).
int resolve_resident(const FrameArgs &a) {
    const ResolveKernel kern = resolve_kernel(a);
    const size_t smem = resolve_smem(a.S, a.ms_output != 0);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int fit = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, kResolveWarps * 32, smem) != cudaSuccess || fit < 1)
        fit = 1;
    return fit;
}

int launch_resolve(const FrameArgs &a, const uint2 *rec_a, const uint32_t *rec_m, const uint32_t *bstart, const uint32_t *bend, uint32_t *image, uint32_t *overflow,
                    FrameCounters *counters, cudaStream_t s) {
    if (a.n_bins <= 0) return 0;
    // every launched block runs at once; never more than resolve_blocks(a),
    // which sized the overflow entry area
    const int64_t blocks = std::min<int64_t>(resolve_blocks(a), (int64_t)sm_count() * resolve_resident(a));
    resolve_kernel(a)<<<(unsigned)blocks, kResolveWarps * 32, resolve_smem(a.S, a.ms_output != 0), s>>>(
        a, rec_a, rec_m, bstart, bend, image, overflow, counters);
    return 1;
}

int launch_encode_sums(const FrameArgs &a, const long long *sums, uint32_t *image, int64_t npix, cudaStream_t s) {
    if (npix <= 0) return 0;
    const unsigned grid = (unsigned)std::min<int64_t>((npix + 255) / 256, 152 * 8);
    if (a.srgb) k_encode_sums<true><<<grid, 256, 0, s>>>(a, sums, image, npix);
    else k_encode_sums<false><<<grid, 256, 0, s>>>(a, sums, image, npix);
    return 1;
}

// The output view (drawOutputResize with output_scale.{vert,frag}.glsl,
// ras_base.cpp:760-803): pixel (x, y) shows the image texel nearest to
// inv * (x + 0.5, y + 0.5, 0, 1) after the divide by w, clamped to the edge
// (the scale texture's GL_NEAREST / GL_CLAMP_TO_EDGE).  inv holds the
// inverse transform's rows 0, 1 and 3, columns 0, 1 and 3.
__global__ void k_output_view(const uint32_t *__restrict__ image, uint32_t *__restrict__ out, int W, int H,
                              OutputInverse inv) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)W * H) return;
    const int x = (int)(i % W), y = (int)(i / W);
    const float px = (float)x + 0.5f, py = (float)y + 0.5f;
    const float qx = inv.m[0] * px + inv.m[1] * py + inv.m[2];
    const float qy = inv.m[3] * px + inv.m[4] * py + inv.m[5];
    const float qw = inv.m[6] * px + inv.m[7] * py + inv.m[8];
    float u = qx / qw, v = qy / qw;
    u = fminf(fmaxf(floorf(u), 0.f), (float)(W - 1));  // fmaxf takes 0 for a NaN
    v = fminf(fmaxf(floorf(v), 0.f), (float)(H - 1));
    out[i] = image[(int64_t)(int)v * W + (int)u];
}

int launch_output_view(const uint32_t *image, uint32_t *out, int W, int H, const OutputInverse &inv, cudaStream_t s) {
    const int64_t n = (int64_t)W * H;
    if (n <= 0) return 0;
    k_output_view<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(image, out, W, H, inv);
    return 1;
}

int launch_selftest_encode(const ResolveTables *rt, unsigned long long *bad, cudaStream_t s) {
    // non-negative floats up to and a little beyond 1.0, plus the negative zero
    k_selftest_encode<<<4 * 152, 256, 0, s>>>(rt, 0u, 0x3F800100u, bad);
    k_selftest_encode<<<1, 256, 0, s>>>(rt, 0x80000000u, 0x80000100u, bad);
    return 2;
}

int64_t resolve_warps(const FrameArgs &a) { return resolve_blocks(a) * kResolveWarps; }

int64_t resolve_overflow_words(const FrameArgs &a) {
    if (!a.ms_output) return 0;
    const int S = a.S == 256 ? 32 : a.S;
    return resolve_warps(a) * (int64_t)(4 * S - kCellCap) * (S / 8 + 1) * 32;
}

int launch_scene_prepare(const uint32_t *cvp, const uint8_t *ctype, const uint32_t *cpid, const float *arcw,
                         uint32_t C, uint32_t V, uint32_t P, float2 *vert, const uint32_t *vpid, uint32_t *vmap,
                         CurveDesc *cd, uint32_t *flags, cudaStream_t s) {
    int n = 0;
    if (V > 0) k_scene_vertices<<<grid_for(V), kThreads, 0, s>>>(vpid, V, P, vmap, flags), ++n;
    if (C > 0) k_scene_curves<<<grid_for(C), kThreads, 0, s>>>(cvp, ctype, cpid, arcw, C, V, P, vert, vmap, cd, flags), ++n;
    return n;
}

int launch_fill(uint32_t *image, int64_t n, uint32_t value, cudaStream_t s) {
    if (n <= 0) return 0;
    k_fill<<<grid_for(n), kThreads, 0, s>>>(image, n, value);
    return 1;
}

int launch_decode_keys(const uint64_t *skey, int64_t n, int nrows, int32_t *out, cudaStream_t s) {
    if (n <= 0) return 0;
    k_decode_keys<<<grid_for(n), kThreads, 0, s>>>(skey, n, nrows, out);
    return 1;
}

}  // namespace spr
