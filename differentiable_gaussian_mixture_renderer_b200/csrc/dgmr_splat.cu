// Tile-based EWA splat renderer: forward (src/dgmr/splat_forward.cu:30-338)
// and a reverse-order backward (no reference kernel), behind the C ABI of
// include/dgmr_b200.h.
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <cuda_runtime.h>

#include "../../include/dgmr_b200.h"
#include "dgmr_abi_common.h"
#include "dgmr_batch.cuh"
#include "dgmr_binning.cuh"
#include "dgmr_device_grad.cuh"
#include "dgmr_f32x2.cuh"

namespace dgmr {

// Frame workspace: everything sized by the Gaussian count, tiles and pixels.
// Pair workspace: the (tile, Gaussian) pair buffers and sort scratch.
struct SplatLayout {
    int32_t* rects;
    float* rgb;
    uint8_t* clamped;
    float* depths;
    float* xy;
    float* conic_opacity;
    uint32_t* tiles_touched;
    uint2* tile_rect;
    uint32_t* point_offsets;
    int32_t* ranges;
    float* final_T;
    int32_t* n_contrib;
    double* grad_acc; // [N,9]: xy(2) conic(3) opacity rgb(3), summed over pixels in double
    float4* blend_rec; // [N,2]: (x, y, a, c), (2b, opacity, q_cut, 0) -- the blend's 32-byte record
    uint32_t* tile_order; // [tiles] launch order of the per-tile kernels, heaviest first
    uint32_t* tile_cost; // [tiles] predicted blend cost of each tile as a bucket, 0 = heaviest
    uint32_t* stats; // [4] used when the caller passes none
    BinningBuffers bin;
    size_t bytes; // frame workspace
    size_t pair_bytes; // pair workspace
};

// N Gaussians (or view-Gaussians of a batch), n_tiles tiles and n_px pixels
inline SplatLayout splat_layout_n(uint32_t N, uint32_t n_tiles, size_t n_px, uint32_t cap, void* base, void* pair_base)
{
    SplatLayout L;
    Carver c;
    c.base = static_cast<char*>(base);
    L.rects = c.take<int32_t>(size_t(N) * 2);
    L.rgb = c.take<float>(size_t(N) * 3);
    L.clamped = c.take<uint8_t>(size_t(N) * 3);
    L.depths = c.take<float>(N);
    L.xy = c.take<float>(size_t(N) * 2);
    L.conic_opacity = c.take<float>(size_t(N) * 4);
    L.tiles_touched = c.take<uint32_t>(N);
    L.point_offsets = c.take<uint32_t>(N);
    L.ranges = c.take<int32_t>(size_t(n_tiles) * 2);
    L.final_T = c.take<float>(n_px);
    L.n_contrib = c.take<int32_t>(n_px);
    L.grad_acc = c.take<double>(size_t(N) * 9);
    // from the preprocess to the binning only; the backward, which follows both, zeroes grad_acc first
    L.tile_rect = reinterpret_cast<uint2*>(L.grad_acc);
    L.blend_rec = c.take<float4>(size_t(N) * 2);
    L.tile_order = c.take<uint32_t>(n_tiles);
    L.tile_cost = c.take<uint32_t>(n_tiles);
    L.stats = c.take<uint32_t>(4);
    carve_binning_gaussians(c, L.bin, N, n_tiles);
    L.bytes = c.off;
    Carver cp;
    cp.base = static_cast<char*>(pair_base);
    carve_binning_pairs(cp, L.bin, N, cap);
    L.pair_bytes = cp.off;
    return L;
}

inline SplatLayout splat_layout(uint32_t N, uint32_t W, uint32_t H, uint32_t cap, void* base, void* pair_base)
{
    const uint32_t gx = (W + kTile - 1) / kTile, gy = (H + kTile - 1) / kTile;
    return splat_layout_n(N, gx * gy, size_t(W) * H, cap, base, pair_base);
}

struct SplatPre {
    uint32_t N;
    const float* centroids;
    const float* sh;
    int sh_stride, sh_degree;
    const float* weights;
    const float* scales;
    const float* rotations;
    int32_t* rects;
    float* rgb;
    uint8_t* clamped;
    float* depths;
    float* xy;
    float* conic_opacity;
    uint32_t* tiles_touched;
    uint2* tile_rect; // (x0 | y0 << 16, x1 | y1 << 16)
    uint32_t* depth_key;
    uint32_t* perm;
    float4* blend_rec;
    Formulation form;
};

// splat_forward.cu:70-118 for Gaussian i of the scene, written to output
// slot o (o = i for one frame; o = the view's offset + i in a batch).
// Bound by memory: 56 bytes in and 103 out per Gaussian at SH degree 0.  Every
// output is stored once, from the values of a Gaussian on no tile unless it
// reaches one (stored first and overwritten: 40.7 us at 1M, now 37.6; 48
// registers, 39.6 with 62 and 41 with 40).
__device__ __forceinline__ void preprocess_one(const SplatPre& p, const CameraT<float>& cam, uint32_t i, uint32_t o)
{
    int ex = 0, ey = 0;
    uint2 tile_rect = make_uint2(0u, 0u);
    float depth = 0.f;
    V2<float> xy = { 0.f, 0.f };
    V3<float> col = { 0.f, 0.f, 0.f };
    uint8_t mask[3] = { 0, 0, 0 };
    float4 conic = make_float4(0.f, 0.f, 0.f, 0.f), r0 = conic, r1 = conic;
    const V3<float> mu = { p.centroids[3 * i], p.centroids[3 * i + 1], p.centroids[3 * i + 2] };
    if (!(view_z(cam.view, mu) < 0.2f)) {
        const float w = p.weights[i];
        const V3<float> sc = mul3(V3<float> { p.scales[3 * i], p.scales[3 * i + 1], p.scales[3 * i + 2] }, cam.cov_scale_multiplier);
        const float* q = p.rotations + 4 * size_t(i);
        const M3<float> R = quat_to_mat3(q[0], q[1], q[2], q[3]);
        const Gaussian2d<float> g = splat_project(p.form, w, mu, sc, R, cam, 0.3f);
        ex = dgmr_fm::to_int_rz(dgmr_fm::ceil_f(3.f * dgmr_fm::sqrt_f(g.cov.v[0])));
        ey = dgmr_fm::to_int_rz(dgmr_fm::ceil_f(3.f * dgmr_fm::sqrt_f(g.cov.v[2])));
        const TileRect r = get_rect(g.centroid.x, g.centroid.y, ex, ey, cam.gx, cam.gy);
        if ((r.x1 - r.x0) * (r.y1 - r.y0) != 0) {
            tile_rect = make_uint2(r.x0 | (r.y0 << 16), r.x1 | (r.y1 << 16));
            xy = g.centroid;
            const V3<float> campos = { cam.campos[0], cam.campos[1], cam.campos[2] };
            depth = len3(sub3(campos, mu));
            const V3<float> v = sub3(mu, campos);
            const V3<float> dir = mul3(v, 1.f / dgmr_fm::sqrt_f(dot3(v, v)));
            col = sh_to_colour(p.sh, i, p.sh_stride, p.sh_degree, dir, mask);
            const S2<float> con = inverse2(g.cov);
            conic = make_float4(con.v[0], con.v[1], con.v[2], g.weight);
            // q_cut: any pixel with d'Qd > q_cut has opacity * exp(-d'Qd/2) < exp(-1e-3) / 255, i.e. alpha < 1/255
            // with a margin far above the rounding of the exponential, so the blend may skip it without changing
            // a single result
            const float q_cut = 2.f * (dgmr_fm::log_f(255.f * g.weight) + 1e-3f);
            r0 = make_float4(g.centroid.x, g.centroid.y, con.v[0], con.v[2]);
            r1 = make_float4(2.f * con.v[1], g.weight, q_cut, 0.f);
        }
    }
    p.tiles_touched[o] = ((tile_rect.y & 0xffffu) - (tile_rect.x & 0xffffu)) * ((tile_rect.y >> 16) - (tile_rect.x >> 16));
    p.tile_rect[o] = tile_rect;
    p.perm[o] = o;
    p.depth_key[o] = __float_as_uint(depth);
    reinterpret_cast<int2*>(p.rects)[o] = make_int2(ex, ey);
    reinterpret_cast<float2*>(p.xy)[o] = make_float2(xy.x, xy.y);
    p.depths[o] = depth;
    p.rgb[3 * o] = col.x;
    p.rgb[3 * o + 1] = col.y;
    p.rgb[3 * o + 2] = col.z;
#pragma unroll
    for (int c = 0; c < 3; ++c)
        p.clamped[3 * o + c] = mask[c];
    reinterpret_cast<float4*>(p.conic_opacity)[o] = conic;
    p.blend_rec[2 * o] = r0;
    p.blend_rec[2 * o + 1] = r1;
}

__global__ void __launch_bounds__(256, 5) k_splat_preprocess(SplatPre p, CameraT<float> cam)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < p.N)
        preprocess_one(p, cam, i, i);
}

// d'Qd of one (pixel, splat) pair (splat_forward.cu:302), evaluated as
// dx * (a dx + 2b dy) + (c dy) dy with two fused multiply-adds; r0 = (x, y, a, c), b2 = 2b
__device__ __forceinline__ float splat_q(float4 r0, float b2, float px, float py, float* dx_o, float* dy_o)
{
    const float dx = px - r0.x;
    const float dy = py - r0.y;
    *dx_o = dx;
    *dy_o = dy;
    return __fmaf_rn(__fmaf_rn(r0.z, dx, b2 * dy), dx, (r0.w * dy) * dy);
}

// Per-pixel blend state of the pixel a thread owns (splat_forward.cu:299-321).
struct PixelState {
    float T, c0, c1, c2;
    int32_t last;
    bool done;
};

// One blend step after the cutoff test, given exp(-q/2)
// (splat_forward.cu:303-321): alpha = min(0.99, opacity * exp), skipped below
// 1/255; the pixel saturates (and keeps its state) once T * (1 - alpha) would
// drop below 1e-4.  Written as selects so that a warp can run it for every
// lane, whether or not the lane uses the record (`use`): the arithmetic and
// its order are the reference's, applied only where `use` holds.
__device__ __forceinline__ void blend_alpha_select(PixelState& ps, bool use, float ex, float opacity, float r, float g, float b, int32_t idx)
{
    const float alpha = min_f(0.99f, opacity * ex);
    const float test_T = ps.T * (1.f - alpha);
    const bool live = use && !ps.done && !(alpha < 1.0f / 255.0f);
    const bool stop = live && test_T < 0.0001f;
    const bool take = live && !stop;
    const float w = alpha * ps.T;
    ps.c0 = take ? __fmaf_rn(r, w, ps.c0) : ps.c0;
    ps.c1 = take ? __fmaf_rn(g, w, ps.c1) : ps.c1;
    ps.c2 = take ? __fmaf_rn(b, w, ps.c2) : ps.c2;
    ps.T = take ? test_T : ps.T;
    ps.last = take ? idx : ps.last;
    ps.done = ps.done || stop;
}

// Minimum of d'Qd over the tile's pixel rectangle [x0,x1] x [y0,y1] for a
// splat at (cx, cy) with conic (a, b, c): 0 if the centre is inside, else the
// minimum over the four edges (each a clamped 1-D quadratic).  Returns 0 (keep)
// for a conic that is not positive definite.  Only used to drop splats with a
// wide margin, so approximate division is fine here.
__device__ __forceinline__ float rect_min_q(float cx, float cy, float a, float b, float c, float x0, float x1, float y0, float y1)
{
    if (!(a > 0.f && c > 0.f && a * c - b * b > 0.f))
        return 0.f;
    if (cx >= x0 && cx <= x1 && cy >= y0 && cy <= y1)
        return 0.f;
    const auto q = [&](float dx, float dy) { return a * dx * dx + 2.f * b * dx * dy + c * dy * dy; };
    float m = 3.0e38f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float dx = (e == 0 ? x0 : x1) - cx;
        const float dy = fminf(fmaxf(cy - __fdividef(b * dx, c), y0), y1) - cy;
        m = fminf(m, q(dx, dy));
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float dy = (e == 0 ? y0 : y1) - cy;
        const float dx = fminf(fmaxf(cx - __fdividef(b * dy, a), x0), x1) - cx;
        m = fminf(m, q(dx, dy));
    }
    return m;
}

// The packed walks (two pixels per lane, the halves of packed floats) take
// records and pixels of ordinary magnitude: the half that does not use a record is
// multiplied by an exact zero, which needs finite operands, and its exp is
// evaluated without the tests for special cases.  The largest operand is the
// backward's product of four: transmittance (kPlainT), the distance of a colour
// from the one behind (3 x 2 kPlain over the channels), the image gradient
// (kPlain) and the opacity (at most e^50 / 255 = 2.1e19 by kPlainCut), together
// below 3e36.  The conic has to be positive definite, and close enough to the
// 8x8 quarter for the rounding of the quadratic form (4 ulp of its terms) to stay
// far above the -170 where exp(-q/2) overflows, and q_cut (NaN for a negative
// opacity) to keep it off the range where the exp is subnormal.  Other records take
// the guarded walk.
constexpr float kPlain = 1.0e8f, kPlainT = 2.f, kPlainForm = 1.0e8f, kPlainCut = 100.f;
__device__ __forceinline__ bool plain_value(float x) { return fabsf(x) <= kPlain; } // false for NaN
__device__ __forceinline__ bool plain_record(float4 r0, float4 r1, float4 rgb, float x0, float y0)
{
    const float dx = fabsf(r0.x - x0) + 8.f, dy = fabsf(r0.y - y0) + 8.f;
    const float b = 0.5f * r1.x;
    return r0.z > 0.f && r0.w > 0.f && r0.z * r0.w - b * b > 0.f && (r0.z + r0.w) * (dx * dx + dy * dy) <= kPlainForm && r1.z <= kPlainCut
        && plain_value((fabsf(rgb.x) + fabsf(rgb.y)) + fabsf(rgb.z));
}

// One 16x16 tile per block of 256 threads, one pixel per thread.  Each batch
// of up to 256 list entries is loaded one per thread; splats whose cutoff
// ellipse cannot reach the tile are dropped (an exact rectangle minimum with a
// margin, so no pixel that could pass its own cutoff test loses a splat); the
// rest are compacted in list order into shared memory as 32-byte records and
// evaluated by every pixel.  The block stops when every pixel is saturated.
// The kernel's duration is set by its slowest tile (a few tiles with ~2-3k
// unsaturated entries run from the first wave to the end), so a tile's
// pixels are spread over as many threads as it has pixels: two pixels per
// thread, evaluated one after the other, made that critical path, and the launch,
// 12 % longer.  (The quarters below take two per thread in packed instructions.)

// A single frame: every tile is one of its tiles.
struct SingleFrame {
    unsigned W, H, gx;
    float bg0, bg1, bg2;
    float* fb;
    float* final_T;
    int32_t* n_contrib;
    const float* grad_fb;
    __device__ __forceinline__ FrameRef frame(uint32_t tile) const { return FrameRef { W, H, gx, tile, bg0, bg1, bg2, fb, final_T, n_contrib, grad_fb }; }
};

// Blocks of either blend kernel on an SM; a block is a tile.
constexpr int kBlendBlocks = 5;
inline bool blend_fits_chip(uint32_t n_tiles) { return n_tiles <= uint32_t(num_sms()) * kBlendBlocks; }

// The blend with a 16x16 tile per block of 256 threads, a pixel each (batches may
// choose it, dgmr_batch_view.blend_block; the same bits as the quarters below).
// __launch_bounds__ keeps it at 48 registers, five blocks per SM instead of four at
// the 52 the compiler picks unbounded: 3 % shorter launches over 8 cameras at
// 1080p/1M.
template <class Frames>
__global__ void __launch_bounds__(kTilePixels, kBlendBlocks) k_splat_blend_tiles(const int32_t* __restrict__ ranges, const uint32_t* __restrict__ list,
    const float4* __restrict__ rec, const float* __restrict__ rgb, uint32_t N, uint32_t cap, uint32_t* __restrict__ stats,
    const uint32_t* __restrict__ tile_order, const __grid_constant__ Frames frames)
{
    chain_start();
    constexpr int kThreads = kTilePixels;
    constexpr int kBatch = kThreads;
    constexpr int kWarps = kThreads / 32;
    constexpr int kGroup = 4;
    static_assert(kBatch % kGroup == 0, "a group never reads past the batch");
    __shared__ float4 s_r0[kBatch];
    __shared__ float4 s_r1[kBatch]; // (2b, opacity, q_cut, 1-based list index as int bits)
    __shared__ float4 s_rgb[kBatch]; // (r, g, b, .): one 16-byte load per record that a warp blends
    __shared__ int s_warp_tot[kWarps];
    const unsigned tile = tile_order ? tile_order[blockIdx.x] : blockIdx.x;
    const FrameRef f = frames.frame(tile);
    const unsigned W = f.W, H = f.H;
    const unsigned tx = f.tile % f.gx, ty = f.tile / f.gx;
    // warp w covers the 8x4 pixel block (8 (w % 2), 4 (w / 2)) of the tile: a
    // compact footprint, so fewer records pass some lane's cutoff than over a 16x2
    // strip (a record no lane needs costs one vote)
    const unsigned wb = threadIdx.x >> 5;
    const unsigned px = tx * kTile + 8u * (wb & 1u) + (threadIdx.x & 7u);
    const unsigned py = ty * kTile + 4u * (wb >> 1) + ((threadIdx.x >> 3) & 3u);
    PixelState p0 { 1.f, 0.f, 0.f, 0.f, 0, !(px < W && py < H) };
    const bool in0 = !p0.done;
    int32_t b = ranges[2 * tile], e = ranges[2 * tile + 1];
    if (b < 0 || e < b || uint32_t(e) > cap) {
        if (threadIdx.x == 0)
            flag_bounds(stats, 0x31u);
        b = e = 0;
    }
    const float fx0 = float(tx * kTile), fx1 = fx0 + float(kTile - 1), fy0 = float(ty * kTile), fy1 = fy0 + float(kTile - 1);
    const float fpx = float(px), fpy = float(py);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int32_t base = b; base < e; base += kBatch) {
        if (__syncthreads_count(p0.done) == kThreads)
            break;
        float4 r0, r1;
        uint32_t id = 0xffffffffu;
        int keep = 0;
        {
            const int32_t k = base + int(threadIdx.x);
            if (k < e) {
                uint32_t g = list[k];
                if (g >= N) {
                    flag_bounds(stats, 0x32u);
                    g = 0;
                }
                r0 = rec[2 * size_t(g)];
                r1 = rec[2 * size_t(g) + 1];
                const float qmin = rect_min_q(r0.x, r0.y, r0.z, 0.5f * r1.x, r0.w, fx0, fx1, fy0, fy1);
                if (!(qmin > r1.z * 1.001f + 0.01f)) {
                    id = g;
                    r1.w = __int_as_float(k - b + 1);
                    keep = 1;
                }
            }
        }
        // order-preserving compaction: warp ballot, then the warps' totals in order
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0)
            s_warp_tot[warp] = __popc(m);
        __syncthreads();
        int slot = __popc(m & ((1u << lane) - 1u));
        int n = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const int t = s_warp_tot[w];
            slot += (w < warp) ? t : 0;
            n += t;
        }
        if (keep) {
            s_r0[slot] = r0;
            s_r1[slot] = r1;
            s_rgb[slot] = make_float4(rgb[3 * size_t(id)], rgb[3 * size_t(id) + 1], rgb[3 * size_t(id) + 2], 0.f);
        }
        // the slots after the last record up to the group boundary: a cutoff below
        // every quadratic form (q = 0 here), so no lane ever uses them
        if (int(threadIdx.x) < kGroup - 1 && n + int(threadIdx.x) < kBatch) {
            s_r0[n + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
            s_r1[n + threadIdx.x] = make_float4(0.f, 0.f, -1.f, 0.f);
        }
        __syncthreads();
        if (!__all_sync(0xffffffffu, p0.done)) {
            // kGroup records at a time, with control flow that is uniform over
            // the warp: the group's quadratic forms (independent, so their
            // shared-memory loads and multiply-adds overlap), then, in list
            // order, the exp and the blend step (as selects) of each record
            // that some lane's cutoff admits; a record no lane needs costs a
            // vote, and the warp leaves once all its pixels are saturated.
            for (int j = 0; j < n; j += kGroup) {
                float q[kGroup];
                bool u[kGroup];
#pragma unroll
                for (int i = 0; i < kGroup; ++i) {
                    const float4 a0 = s_r0[j + i], a1 = s_r1[j + i]; // j + i < kBatch (kBatch % kGroup == 0)
                    float dx, dy;
                    q[i] = splat_q(a0, a1.x, fpx, fpy, &dx, &dy);
                    u[i] = !(q[i] > a1.z) && !p0.done;
                }
#pragma unroll
                for (int i = 0; i < kGroup; ++i) {
                    if (!__any_sync(0xffffffffu, u[i]))
                        continue;
                    const float ex = u[i] ? dgmr_fm::exp_f_nonpos(-0.5f * q[i]) : 0.f;
                    const float4 a1 = s_r1[j + i];
                    const float4 c = s_rgb[j + i];
                    blend_alpha_select(p0, u[i], ex, a1.y, c.x, c.y, c.z, __float_as_int(a1.w));
                }
                if (__all_sync(0xffffffffu, p0.done))
                    break;
            }
        }
        __syncthreads();
    }
    const size_t plane = size_t(W) * H;
    if (in0) {
        const size_t pix = size_t(py) * W + px;
        f.fb[pix] = p0.c0 + p0.T * f.bg0;
        f.fb[plane + pix] = p0.c1 + p0.T * f.bg1;
        f.fb[2 * plane + pix] = p0.c2 + p0.T * f.bg2;
        f.final_T[pix] = p0.T;
        f.n_contrib[pix] = p0.last;
    }
}

// The blend with a warp per 8x8 quarter of a tile and two pixels per lane, (x, y)
// and (x, y + 4), as the halves of packed floats: one packed operation evaluates
// a record for both, bit for bit what a pixel per thread gives.  The quarters of
// a tile are independent warps -- each culls the tile's list against its own
// pixels, 32 entries at a time, and stops when they are saturated -- so there is
// no block barrier.  A launch ends with its slowest warp's serial walk (some 2000
// records), so the walk's latencies are overlapped rather than its instructions
// saved: the next batch is requested ahead (ListWalk: 226 -> 177 us at 1M, 1080p
// for a camera with a few slow tiles), a group's four exps are evaluated together,
// needed or not, and 92 registers without spills beat more warps (177 -> 133).
constexpr int kQuarterWarps = 4;
// A warp's walk of a tile's list, 32 entries at a time: the next batch's records
// and the ids of the one after are requested before the current batch is
// worked on.  (Loaded when their batch began, list, record and colour were three
// latencies in a row, 94 times for the 3000 entries of a slow tile, and the
// launch waits for its slowest tile.)  A walk of an empty list requests nothing; in
// any other, N > 0, and a lane without an entry reads Gaussian 0's record.
struct ListWalk {
    float4 r0, r1; // of the lane's entry in the next batch
    float c0, c1, c2;
    uint32_t id, later; // its Gaussian, and that of the batch after
    __device__ __forceinline__ static uint32_t entry(const uint32_t* __restrict__ list, int32_t k, int32_t first, int32_t end)
    {
        return k >= first && k < end ? list[k] : 0xffffffffu;
    }
    __device__ __forceinline__ void request(const float4* __restrict__ rec, const float* __restrict__ rgb, uint32_t N)
    {
        const size_t g = id < N ? id : 0u;
        r0 = rec[2 * g];
        r1 = rec[2 * g + 1];
        c0 = rgb[3 * g];
        c1 = rgb[3 * g + 1];
        c2 = rgb[3 * g + 2];
    }
};

struct QuarterPixels {
    F2 T, c0, c1, c2;
    int32_t last0, last1;
    bool done0, done1;
};

template <bool kGuarded>
__device__ __forceinline__ void blend_record2(QuarterPixels& p, F2 q, F2 ex, bool use0, bool use1, float4 r1, float4 c)
{
    float e0, e1;
    split2(ex, &e0, &e1);
    if (kGuarded) {
        float q0, q1;
        split2(q, &q0, &q1);
        if (use0 && !(q0 >= -170.f && q0 <= 170.f))
            e0 = dgmr_fm::exp_f_nonpos(-0.5f * q0);
        if (use1 && !(q1 >= -170.f && q1 <= 170.f))
            e1 = dgmr_fm::exp_f_nonpos(-0.5f * q1);
    }
    const float a0 = min_f(0.99f, r1.y * e0), a1 = min_f(0.99f, r1.y * e1);
    const F2 alpha = f2(a0, a1);
    const F2 test = mul2(p.T, fma2(alpha, f2(-1.f), f2(1.f)));
    float t0, t1, T0, T1, w0, w1;
    split2(test, &t0, &t1);
    split2(p.T, &T0, &T1);
    split2(mul2(alpha, p.T), &w0, &w1);
    const bool live0 = use0 && !(a0 < 1.0f / 255.0f), live1 = use1 && !(a1 < 1.0f / 255.0f);
    const bool stop0 = live0 && t0 < 0.0001f, stop1 = live1 && t1 < 0.0001f;
    const bool take0 = live0 && !stop0, take1 = live1 && !stop1;
    if (kGuarded) {
        const auto add = [&](F2& to, float col) {
            float lo, hi;
            split2(to, &lo, &hi);
            to = f2(take0 ? __fmaf_rn(col, w0, lo) : lo, take1 ? __fmaf_rn(col, w1, hi) : hi);
        };
        add(p.c0, c.x);
        add(p.c1, c.y);
        add(p.c2, c.z);
    } else {
        const F2 w = f2(take0 ? w0 : 0.f, take1 ? w1 : 0.f);
        p.c0 = fma2(f2(c.x), w, p.c0);
        p.c1 = fma2(f2(c.y), w, p.c1);
        p.c2 = fma2(f2(c.z), w, p.c2);
    }
    p.T = f2(take0 ? t0 : T0, take1 ? t1 : T1);
    const int32_t idx = __float_as_int(r1.w);
    p.last0 = take0 ? idx : p.last0;
    p.last1 = take1 ? idx : p.last1;
    p.done0 = p.done0 || stop0;
    p.done1 = p.done1 || stop1;
}

template <class Frames>
__global__ void __launch_bounds__(kQuarterWarps * 32, kBlendBlocks) k_splat_blend_quarters(const int32_t* __restrict__ ranges, const uint32_t* __restrict__ list,
    const float4* __restrict__ rec, const float* __restrict__ rgb, uint32_t N, uint32_t cap, uint32_t* __restrict__ stats,
    const uint32_t* __restrict__ tile_order, const __grid_constant__ Frames frames)
{
    chain_start();
    constexpr int kGroup = 4;
    __shared__ float4 s_r0[kQuarterWarps][32];
    __shared__ float4 s_r1[kQuarterWarps][32]; // (2b, opacity, q_cut, 1-based list index as int bits)
    __shared__ float4 s_rgb[kQuarterWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned tile = tile_order ? tile_order[blockIdx.x] : blockIdx.x;
    const FrameRef f = frames.frame(tile);
    const unsigned W = f.W, H = f.H;
    const unsigned x0 = (f.tile % f.gx) * kTile + 8u * (unsigned(warp) & 1u), y0 = (f.tile / f.gx) * kTile + 8u * (unsigned(warp) >> 1);
    const unsigned px = x0 + (unsigned(lane) & 7u), py = y0 + (unsigned(lane) >> 3);
    const bool in0 = px < W && py < H, in1 = px < W && py + 4u < H;
    QuarterPixels p { f2(1.f), f2(0.f), f2(0.f), f2(0.f), 0, 0, !in0, !in1 };
    int32_t b = ranges[2 * tile], e = ranges[2 * tile + 1];
    if (b < 0 || e < b || uint32_t(e) > cap) {
        if (threadIdx.x == 0)
            flag_bounds(stats, 0x31u);
        b = e = 0;
    }
    const float fpx = float(px), fx0 = float(x0), fx1 = fx0 + 7.f, fy0 = float(y0), fy1 = fy0 + 7.f;
    const F2 fpy = f2(float(py), float(py + 4u));
    using Walk = ListWalk;
    Walk next;
    next.id = Walk::entry(list, b + lane, b, e);
    next.later = Walk::entry(list, b + 32 + lane, b, e);
    if (b < e)
        next.request(rec, rgb, N);
    for (int32_t base = b; base < e; base += 32) {
        if (__all_sync(0xffffffffu, p.done0 && p.done1))
            break;
        const int32_t k = base + lane;
        bool keep = false, fine = true;
        const float4 r0 = next.r0;
        float4 r1 = next.r1;
        const float4 c = make_float4(next.c0, next.c1, next.c2, 0.f);
        const uint32_t g = next.id;
        next.id = next.later;
        next.later = Walk::entry(list, k + 64, b, e);
        next.request(rec, rgb, N);
        if (k < e) {
            if (g >= N)
                flag_bounds(stats, 0x32u);
            const float qmin = rect_min_q(r0.x, r0.y, r0.z, 0.5f * r1.x, r0.w, fx0, fx1, fy0, fy1);
            keep = !(qmin > r1.z * 1.001f + 0.01f);
            if (keep) {
                r1.w = __int_as_float(k - b + 1);
                fine = plain_record(r0, r1, c, fx0, fy0);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        const bool guarded = !__all_sync(0xffffffffu, fine);
        const int n = __popc(m);
        __syncwarp(); // the last batch is read
        if (keep) {
            const int pos = __popc(m & ((1u << lane) - 1u));
            s_r0[warp][pos] = r0;
            s_r1[warp][pos] = r1;
            s_rgb[warp][pos] = c;
        }
        // up to the group boundary: a cutoff below every quadratic form (q = 0
        // here), so no lane ever uses them
        if (lane < kGroup - 1 && n + lane < 32) {
            s_r0[warp][n + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            s_r1[warp][n + lane] = make_float4(0.f, 0.f, -1.f, 0.f);
            s_rgb[warp][n + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncwarp();
        // kGroup records at a time: their quadratic forms (independent), then, in
        // list order, the exp and the blend step of each record that some
        // lane's cutoff admits
        for (int j = 0; j < n; j += kGroup) {
            F2 q[kGroup];
            bool u0[kGroup], u1[kGroup];
#pragma unroll
            for (int i = 0; i < kGroup; ++i) {
                const float4 s0 = s_r0[warp][j + i], s1 = s_r1[warp][j + i]; // j + i < 32
                const float dx = fpx - s0.x;
                const F2 dy = add2(fpy, f2(-s0.y));
                q[i] = fma2(fma2(f2(s0.z), f2(dx), mul2(f2(s1.x), dy)), f2(dx), mul2(mul2(f2(s0.w), dy), dy));
                float qa, qb;
                split2(q[i], &qa, &qb);
                u0[i] = !(qa > s1.z);
                u1[i] = !(qb > s1.z);
            }
            bool any = false;
#pragma unroll
            for (int i = 0; i < kGroup; ++i) {
                u0[i] = u0[i] && !p.done0;
                u1[i] = u1[i] && !p.done1;
                any = any || u0[i] || u1[i];
            }
            if (!__any_sync(0xffffffffu, any))
                continue;
            F2 ex[kGroup];
#pragma unroll
            for (int i = 0; i < kGroup; ++i)
                ex[i] = exp2_nonpos(mul2(q[i], f2(-0.5f)));
            if (guarded) {
#pragma unroll
                for (int i = 0; i < kGroup; ++i)
                    blend_record2<true>(p, q[i], ex[i], u0[i] && !p.done0, u1[i] && !p.done1, s_r1[warp][j + i], s_rgb[warp][j + i]);
            } else {
#pragma unroll
                for (int i = 0; i < kGroup; ++i)
                    blend_record2<false>(p, q[i], ex[i], u0[i] && !p.done0, u1[i] && !p.done1, s_r1[warp][j + i], s_rgb[warp][j + i]);
            }
            if (__all_sync(0xffffffffu, p.done0 && p.done1))
                break;
        }
    }
    const size_t plane = size_t(W) * H;
    float T[2], col[3][2];
    split2(p.T, &T[0], &T[1]);
    split2(p.c0, &col[0][0], &col[0][1]);
    split2(p.c1, &col[1][0], &col[1][1]);
    split2(p.c2, &col[2][0], &col[2][1]);
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (h ? in1 : in0) {
            const size_t pix = size_t(py + 4u * unsigned(h)) * W + px;
            f.fb[pix] = col[0][h] + T[h] * f.bg0;
            f.fb[plane + pix] = col[1][h] + T[h] * f.bg1;
            f.fb[2 * plane + pix] = col[2][h] + T[h] * f.bg2;
            f.final_T[pix] = T[h];
            f.n_contrib[pix] = h ? p.last1 : p.last0;
        }
}

// The blend over n_tiles tiles: a warp per 8x8 quarter (side 8), or a block per
// tile (16).  Single frames use quarters, 157 -> 133 us at 1M, 1080p and 148 -> 135
// at 200k, 1024^2 against a pixel per thread; batches take the side from their
// views (dgmr_batch_view.blend_block).
constexpr int kBlendSide = 8;
template <class Frames>
void launch_blend(int side, uint32_t n_tiles, const int32_t* ranges, const uint32_t* list, const float4* rec, const float* rgb, uint32_t N, uint32_t cap,
    uint32_t* stats, const uint32_t* tile_order, const Frames& frames, cudaStream_t s)
{
    if (n_tiles == 0)
        return;
    if (side == 8)
        launch_chained(k_splat_blend_quarters<Frames>, n_tiles, kQuarterWarps * 32, 0, ChainStream(s, blend_fits_chip(n_tiles)), ranges, list, rec, rgb, N, cap, stats, tile_order, frames);
    else
        launch_chained(k_splat_blend_tiles<Frames>, n_tiles, kTilePixels, 0, ChainStream(s, blend_fits_chip(n_tiles)), ranges, list, rec, rgb, N, cap, stats, tile_order, frames);
    note_launch();
}

// Sums of 12 per-lane values over a warp, scattered: halve the slots each lane
// holds at every butterfly level (12 -> 6 -> 3, the upper half kept by the lanes
// whose level bit is set), exchange one pair of the three and sum the third,
// then halve the two that are left.  Every sum is the tree over lane distances 16,
// 8, 4, 2.  Lane l returns slot reduce_slot(l)'s sum over the 16 lanes of its own
// parity.
__device__ __forceinline__ int reduce_slot(int lane)
{
    const int base = 6 * ((lane >> 4) & 1) + 3 * ((lane >> 3) & 1);
    return base + ((lane & 2) ? 2 : ((lane >> 2) & 1));
}
__device__ __forceinline__ float warp_reduce_scatter12(const float (&v)[12], int lane)
{
    float a[6], b[3];
    const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0, b2 = (lane & 4) != 0, b1 = (lane & 2) != 0;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        a[q] = (b4 ? v[q + 6] : v[q]) + __shfl_xor_sync(0xffffffffu, b4 ? v[q] : v[q + 6], 16);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        b[q] = (b3 ? a[q + 3] : a[q]) + __shfl_xor_sync(0xffffffffu, b3 ? a[q] : a[q + 3], 8);
    // slots 0 and 1 of the three between the lanes of bit 2; slot 2 on both
    const float c = (b2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, b2 ? b[0] : b[1], 4);
    const float d = b[2] + __shfl_xor_sync(0xffffffffu, b[2], 4);
    return (b1 ? d : c) + __shfl_xor_sync(0xffffffffu, b1 ? c : d, 2);
}

// Reverse-order blend adjoint.  A warp owns an 8x8 quarter of a tile and a lane
// two of its pixels, (x, y) and (x, y + 4), as the halves of packed floats: the
// quadratic form, the exp, the inverse blend step and the partials are one
// packed operation for both, and a record's partials are summed over 64 pixels
// by one warp reduction.  Each pixel walks its contributors back to front,
// recovering T_i = T_{i+1} / (1 - alpha_i).  Per record the warp sums the
// gradients of the centre, the conic, the opacity and the colour over its pixels,
// and eighteen lanes add one value each.  A float sum covers 32 pixels, which meet in
// double: for the conic the upper or the lower half of the quarter, for the others
// its even or its odd columns.  The chain from the conic to a long thin splat's
// scales cancels by 10^5; with float sums over 64 pixels single elements moved by
// 1e-3, and grouped as the others (16 pixels at a time then) they are closer to the
// exact sums but move by up to 2e-2 on splats 30 to 1000 times as long as wide.  The
// totals over warps are double too: in float, the order in which the atomics of
// many cancelling terms land moved single elements by ~1e-3 relative from run to
// run at 200k Gaussians, 1024^2.
// Distance from per-pixel double sums, mean of 32 frames in the 2-norm: colours
// 5.8e-8, opacities 6.3e-8, centres 8.4e-8; with float sums over 64 pixels 6.5e-8
// and 7.0e-8, in the time of the columns; over 32 pixels as 8x4 blocks 6.0e-8 and
// 6.5e-8, in a tenth more.  The centre's gradient from the moments g_q dx and g_q
// dy, multiplied by the conic once per Gaussian, is 1.3e-7 off (the products
// cancel after the sums are rounded), in 2.5 % less time.
// Tiles run in the forward's launch order (heaviest predicted walk first); a
// warp walks its tile's list only up to its own pixels' last contributor.
//
// Bound by instruction issue, and at the end of a launch by the longest warp's
// serial walk: so a record's reduction is issued with the next record's body, and
// 89 registers without spills beat 64 with them, and the next batch is requested
// ahead (ListWalk: 299 -> 273 us at 1M, 1080p, 284 -> 288 at 200k, 1024^2).  Against a
// pixel per lane, a reduction per 32 pixels of all nine values and 48 registers:
// 401 -> 282 us at 1M, 1080p; 430 -> 304 us at 200k, 1024^2.
constexpr int kBwdWarps = 4; // the quarters of a tile
static_assert(kTile == 16, "four 8x8 quarters per tile");

struct BwdPixels {
    F2 Tr; // transmittance in front of the records walked so far
    F2 a0, a1, a2; // colour behind the current record
    F2 g0, g1, g2; // image gradient
    F2 bg; // final T times the gradient's product with the background
    int32_t n0, n1; // contributors
};

// A record's quadratic form on the lane's two pixels, q = x dx + y dy, in splat_q's operations.
struct BwdForm {
    F2 x; // a dx + 2b dy
    F2 y; // c dy
    F2 q;
};

// Whether the packed walk's products with an unused record are exact zeros for
// what the lane's pixels have collected so far.
__device__ __forceinline__ bool plain_state(const BwdPixels& p)
{
    const auto both = [](F2 t, float most) {
        float lo, hi;
        split2(t, &lo, &hi);
        return fabsf(lo) <= most && fabsf(hi) <= most; // false for NaN
    };
    return both(p.Tr, kPlainT) && both(p.a0, kPlain) && both(p.a1, kPlain) && both(p.a2, kPlain);
}

// One record on the lane's two pixels: `use` says which of them it reaches.
// Returns whether any partial is nonzero.  kGuarded: values may be huge or not
// finite, and a pixel that does not use the record must not see them.
template <bool kGuarded>
__device__ __forceinline__ bool bwd_record(BwdPixels& p, float4 r0, float4 r1, float4 c, const BwdForm& f, float dx, F2 dy, bool use0, bool use1, float (&v)[12])
{
    const float op = r1.y;
    float e0, e1;
    split2(exp2_nonpos(mul2(f.q, f2(-0.5f))), &e0, &e1);
    if (kGuarded) {
        float q0, q1;
        split2(f.q, &q0, &q1);
        if (use0 && !(q0 >= -170.f && q0 <= 170.f))
            e0 = dgmr_fm::exp_f_nonpos(-0.5f * q0);
        if (use1 && !(q1 >= -170.f && q1 <= 170.f))
            e1 = dgmr_fm::exp_f_nonpos(-0.5f * q1);
    }
    const float og0 = op * e0, og1 = op * e1;
    float al0 = min_f(0.99f, og0), al1 = min_f(0.99f, og1);
    use0 = use0 && !(al0 < 1.0f / 255.0f);
    use1 = use1 && !(al1 < 1.0f / 255.0f);
    al0 = use0 ? al0 : 0.f;
    al1 = use1 ? al1 : 0.f;
    const F2 g = f2(use0 ? e0 : 0.f, use1 ? e1 : 0.f), alpha = f2(al0, al1);
    const float x0 = 1.f - al0, x1 = 1.f - al1; // in [0.01, 1]
    const F2 keep = f2(x0, x1), inv = recip2(keep);
    const F2 Tr = mul2(p.Tr, inv);
    const F2 aT = mul2(alpha, Tr);
    const F2 w0 = mul2(aT, p.g0), w1 = mul2(aT, p.g1), w2 = mul2(aT, p.g2);
    const F2 neg = f2(-1.f);
    const F2 d0 = fma2(p.a0, neg, f2(c.x)), d1 = fma2(p.a1, neg, f2(c.y)), d2 = fma2(p.a2, neg, f2(c.z));
    const F2 dot = add2(add2(mul2_rounded(d0, p.g0), mul2_rounded(d1, p.g1)), mul2_rounded(d2, p.g2));
    const F2 ga = add2(mul2_rounded(Tr, dot), mul2_rounded(mul2(p.bg, neg), inv));
    float ga0, ga1;
    split2(ga, &ga0, &ga1);
    ga0 = og0 < 0.99f ? ga0 : 0.f; // alpha = 0.99 there, whatever the opacity
    ga1 = og1 < 0.99f ? ga1 : 0.f;
    const F2 go = mul2(f2(ga0, ga1), g); // d/dopacity
    const F2 gq = mul2(mul2(g, f2(-0.5f)), mul2(f2(ga0, ga1), f2(op)));
    const F2 gx = mul2(gq, f2(dx)), gy = mul2(gq, dy);
    // d/dcentre = -g_q (2a dx + 2b dy, 2c dy + 2b dx)
    const F2 ux = fma2(f2(-r0.z), f2(dx), mul2(f.x, neg)), uy = fma2(f.y, f2(-2.f), f2(-r1.x * dx));
    const F2 gxx = mul2(gx, f2(dx)), gxy = mul2(mul2(gx, f2(2.f)), dy), gyy = mul2(gy, dy);
    const F2 na0 = add2(mul2_rounded(alpha, f2(c.x)), mul2_rounded(keep, p.a0));
    const F2 na1 = add2(mul2_rounded(alpha, f2(c.y)), mul2_rounded(keep, p.a1));
    const F2 na2 = add2(mul2_rounded(alpha, f2(c.z)), mul2_rounded(keep, p.a2));
    // a saturated pixel has no gradient but the colour's, whatever the opacity (it may be infinite) or the exponent
    const bool live0 = use0 && og0 < 0.99f, live1 = use1 && og1 < 0.99f;
    const auto halves = [&](F2 t, bool take0, bool take1, float* lo, float* hi) {
        split2(t, lo, hi);
        if (kGuarded) {
            *lo = take0 ? *lo : 0.f;
            *hi = take1 ? *hi : 0.f;
        }
    };
    const auto sum = [&](F2 t, bool take0, bool take1) {
        float lo, hi;
        halves(t, take0, take1, &lo, &hi);
        return lo + hi;
    };
    // in the order of k_splat_bwd_pixels' accumulators
    v[0] = sum(mul2(gq, ux), live0, live1);
    v[1] = sum(mul2(gq, uy), live0, live1);
    halves(gxx, live0, live1, &v[2], &v[3]);
    halves(gxy, live0, live1, &v[4], &v[5]);
    halves(gyy, live0, live1, &v[6], &v[7]);
    v[8] = sum(go, live0, live1);
    v[9] = sum(w0, use0, use1);
    v[10] = sum(w1, use0, use1);
    v[11] = sum(w2, use0, use1);
    if (kGuarded) {
        const auto pick = [&](F2& to, F2 from) {
            float a, b, x, y;
            split2(to, &a, &b);
            split2(from, &x, &y);
            to = f2(use0 ? x : a, use1 ? y : b);
        };
        pick(p.Tr, Tr);
        pick(p.a0, na0);
        pick(p.a1, na1);
        pick(p.a2, na2);
    } else {
        p.Tr = Tr;
        p.a0 = na0;
        p.a1 = na1;
        p.a2 = na2;
    }
    return use0 || use1;
}

template <class Frames>
__global__ void __launch_bounds__(kBwdWarps * 32, 5) k_splat_bwd_pixels(const int32_t* __restrict__ ranges, const uint32_t* __restrict__ list,
    const float4* __restrict__ rec, const float* __restrict__ rgb, uint32_t N, double* __restrict__ acc, const uint32_t* __restrict__ tile_order,
    const __grid_constant__ Frames frames)
{
    __shared__ float4 s_r0[kBwdWarps][32]; // the blend records: (x, y, a, c), (2b, opacity, q_cut, list index as int bits)
    __shared__ float4 s_r1[kBwdWarps][32];
    __shared__ float4 s_rgb[kBwdWarps][32]; // colour, Gaussian as int bits
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned ordered = tile_order ? tile_order[blockIdx.x] : blockIdx.x;
    const unsigned tile = ordered < gridDim.x ? ordered : blockIdx.x; // the order is a permutation of the tiles
    const FrameRef f = frames.frame(tile);
    if (!f.grad_fb) // a view without an image gradient (batched renders that only asked for the image)
        return;
    const unsigned W = f.W, H = f.H;
    const unsigned x0 = (f.tile % f.gx) * kTile + 8u * (unsigned(warp) & 1u), y0 = (f.tile / f.gx) * kTile + 8u * (unsigned(warp) >> 1);
    const unsigned px = x0 + (unsigned(lane) & 7u), py = y0 + (unsigned(lane) >> 3);
    const size_t plane = size_t(W) * H;
    BwdPixels p;
    float g[2][3], T[2], bg[2];
    int32_t n[2];
    bool plain = true;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const unsigned y = py + 4u * unsigned(h);
        const bool inside = px < W && y < H;
        const size_t pix = size_t(y) * W + px;
        n[h] = inside ? f.n_contrib[pix] : 0;
        T[h] = inside ? f.final_T[pix] : 1.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            g[h][c] = inside ? f.grad_fb[c * plane + pix] : 0.f;
            plain = plain && plain_value(g[h][c]);
        }
        bg[h] = T[h] * ((f.bg0 * g[h][0] + f.bg1 * g[h][1]) + f.bg2 * g[h][2]);
        plain = plain && plain_value(bg[h]);
    }
    p.Tr = f2(T[0], T[1]);
    p.a0 = p.a1 = p.a2 = f2(0.f);
    p.g0 = f2(g[0][0], g[1][0]);
    p.g1 = f2(g[0][1], g[1][1]);
    p.g2 = f2(g[0][2], g[1][2]);
    p.bg = f2(bg[0], bg[1]);
    p.n0 = n[0];
    p.n1 = n[1];
    plain = __all_sync(0xffffffffu, plain && plain_state(p));
    const int32_t b = ranges[2 * tile];
    const int32_t end = __reduce_max_sync(0xffffffffu, max(n[0], n[1]));
    const float fpx = float(px);
    const F2 fpy = f2(float(py), float(py + 4u));
    const float fx0 = float(x0), fx1 = fx0 + 7.f, fy0 = float(y0), fy1 = fy0 + 7.f;
    float held[12] = {};
    uint32_t held_id = 0xffffffffu;
    // the accumulator of each reduced slot: 0, 1, then the conic's three from both halves, then opacity and colour
    const int slot = reduce_slot(lane);
    const int my_slot = slot < 2 ? slot : slot < 8 ? 1 + slot / 2 : slot - 3;
    const bool conic = slot >= 2 && slot < 8; // its lanes of both parities add up in float, and the even one adds the sum
    const bool adds = ((lane & 1) == 0 || !conic) && ((lane & 2) == 0 || (lane & 4) == 0); // slot 2 of three is on both lanes of bit 2
    const auto add = [&](float part) {
        const float other = __shfl_xor_sync(0xffffffffu, part, 1);
        const float sum = conic ? part + other : part;
        if (adds && held_id != 0xffffffffu && sum != 0.f)
            atomicAdd(acc + size_t(held_id) * 9 + my_slot, double(sum));
    };
    ListWalk next;
    next.id = ListWalk::entry(list + b, end - 32 + lane, 0, end);
    next.later = ListWalk::entry(list + b, end - 64 + lane, 0, end);
    if (end > 0)
        next.request(rec, rgb, N);
    for (int32_t hi = end; hi > 0; hi -= 32) {
        // the batch's records that can reach a pixel of this quarter (the
        // forward's exact rectangle cull), compacted in list order with their
        // list positions; the others add nothing to any pixel here
        const int32_t k = hi - 32 + lane;
        bool keep = false, fine = true;
        const float4 r0 = next.r0;
        float4 r1 = next.r1;
        const uint32_t id = next.id;
        const float4 c = make_float4(next.c0, next.c1, next.c2, __uint_as_float(id));
        next.id = next.later;
        next.later = ListWalk::entry(list + b, k - 64, 0, end);
        next.request(rec, rgb, N);
        if (id < N) {
            const float qmin = rect_min_q(r0.x, r0.y, r0.z, 0.5f * r1.x, r0.w, fx0, fx1, fy0, fy1);
            keep = !(qmin > r1.z * 1.001f + 0.01f);
            if (keep) {
                r1.w = __int_as_float(k);
                fine = plain_record(r0, r1, c, fx0, fy0);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        const bool guarded = !plain || !__all_sync(0xffffffffu, fine);
        __syncwarp(); // the last batch is read
        if (keep) {
            const int pos = __popc(m & ((1u << lane) - 1u));
            s_r0[warp][pos] = r0;
            s_r1[warp][pos] = r1;
            s_rgb[warp][pos] = c;
        }
        __syncwarp();
        for (int j = __popc(m) - 1; j >= 0; --j) {
            const float4 q0 = s_r0[warp][j], q1 = s_r1[warp][j];
            const int32_t kk = __float_as_int(q1.w);
            // splat_q on both pixels
            const float dx = fpx - q0.x;
            const F2 dy = add2(fpy, f2(-q0.y));
            BwdForm form;
            form.x = fma2(f2(q0.z), f2(dx), mul2(f2(q1.x), dy));
            form.y = mul2(f2(q0.w), dy);
            form.q = fma2(form.x, f2(dx), mul2(form.y, dy));
            float qa, qb;
            split2(form.q, &qa, &qb);
            // the forward's cutoff: past q_cut alpha < 1/255, so exp is not
            // needed; a record no lane of the warp needs costs one vote
            const bool u0 = kk < p.n0 && !(qa > q1.z), u1 = kk < p.n1 && !(qb > q1.z);
            if (!__any_sync(0xffffffffu, u0 || u1))
                continue;
            const float4 col = s_rgb[warp][j];
            // the last record's reduction is issued with this record's body: they
            // are independent, and each is a long dependent chain
            float v[12], w;
            bool any;
            if (guarded) {
                any = bwd_record<true>(p, q0, q1, col, form, dx, dy, u0, u1, v);
                w = warp_reduce_scatter12(held, lane);
            } else {
                any = bwd_record<false>(p, q0, q1, col, form, dx, dy, u0, u1, v);
                w = warp_reduce_scatter12(held, lane);
            }
            add(w);
            any = __any_sync(0xffffffffu, any);
            held_id = any ? __float_as_uint(col.w) : 0xffffffffu;
#pragma unroll
            for (int k = 0; k < 12; ++k)
                held[k] = v[k];
        }
        // a record of the guarded walk may leave a state that is not plain, which
        // the records in front meet: the rest of the walk is then guarded too
        if (guarded && plain)
            plain = __all_sync(0xffffffffu, plain_state(p));
    }
    add(warp_reduce_scatter12(held, lane));
}

// The per-pixel adjoint over n_tiles tiles.
template <class Frames>
void launch_blend_bwd(uint32_t n_tiles, const int32_t* ranges, const uint32_t* list, const float4* rec, const float* rgb, uint32_t N, double* acc,
    const uint32_t* tile_order, const Frames& frames, cudaStream_t s)
{
    if (n_tiles == 0)
        return;
    k_splat_bwd_pixels<Frames><<<n_tiles, kBwdWarps * 32, 0, s>>>(ranges, list, rec, rgb, N, acc, tile_order, frames);
}

struct SplatBwdGauss {
    uint32_t N;
    const float* centroids;
    const float* sh;
    int sh_stride, sh_degree;
    const float* weights;
    const float* scales;
    const float* rotations;
    const uint8_t* clamped;
    const uint32_t* tiles_touched;
    const double* acc;
    float* g_sh;
    float* g_weights;
    float* g_centroids;
    float* g_scales;
    float* g_rotations;
    Formulation form;
};

// The gradients of one Gaussian besides its SH coefficients.
struct GaussianGrads {
    float weight = 0.f;
    V3<float> mu = { 0.f, 0.f, 0.f }, s = { 0.f, 0.f, 0.f };
    float q[4] = { 0.f, 0.f, 0.f, 0.f };
};

__device__ __forceinline__ void store_gaussian_grads(const SplatBwdGauss& p, uint32_t i, const GaussianGrads& g)
{
    p.g_weights[i] = g.weight;
    p.g_centroids[3 * i] = g.mu.x;
    p.g_centroids[3 * i + 1] = g.mu.y;
    p.g_centroids[3 * i + 2] = g.mu.z;
    p.g_scales[3 * i] = g.s.x;
    p.g_scales[3 * i + 1] = g.s.y;
    p.g_scales[3 * i + 2] = g.s.z;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        p.g_rotations[4 * size_t(i) + k] = g.q[k];
}

// A block's SH gradient rows in shared memory, one per thread, an odd number of
// words apart (no bank conflicts); each warp copies its 32 rows out together.
// Stored by each thread, a row of 16 coefficients is 48 stores that touch 32
// sectors each, twice with the zeros that go first.  The kernel at 1M with 1, 4, 9
// and 16 coefficients: 80, 126, 295, 632 us direct; 88, 103, 134, 319 through rows.
// So rows of one coefficient (kShDirect) are stored directly; a batch, which adds
// up several views' rows, always goes through shared memory.
constexpr int kBwdGaussThreads = 128;
constexpr int kShDirect = 1;
__host__ __device__ constexpr int sh_row_words(int sh_stride) { return 3 * sh_stride | 1; }

__device__ __forceinline__ void store_sh_rows(const SplatBwdGauss& p, const float* rows, uint32_t i0, uint32_t n_rows, int lane, int step)
{
    const int width = 3 * p.sh_stride;
    float* out = p.g_sh + size_t(i0) * width;
    int r = 0, c = lane;
    __syncwarp();
    for (uint32_t t = uint32_t(lane); t < n_rows * uint32_t(width); t += 32) {
        while (c >= width) {
            c -= width;
            ++r;
        }
        out[t] = rows[r * step + c];
        c += 32;
    }
}

// per-Gaussian chain rule: conic -> 2-D covariance -> projection adjoint, SH.
// Gaussian i of the scene, per-view state at slot o, on a tile of its view; the
// result is added to `sum` and, for the SH coefficients, written to the Gaussian's
// `row` (kAddSh: added to it), so several views of one scene sum up.
// Rows and sums are stored once per Gaussian (zeroed first and added to in
// memory, with the same arithmetic: 106.6 us at 1M, SH degree 0, now 85.9, and 78
// with 80 registers instead of 96; bound by its ~1900 instructions per warp, 29
// us of memory traffic).
template <bool kAddSh>
__device__ __forceinline__ void bwd_gaussian_one(const SplatBwdGauss& p, const CameraT<float>& cam, uint32_t i, uint32_t o, GaussianGrads& sum, float* row)
{
    float a[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
        a[k] = float(p.acc[size_t(o) * 9 + k]);
    const V3<float> mu = { p.centroids[3 * i], p.centroids[3 * i + 1], p.centroids[3 * i + 2] };
    const V3<float> sc = mul3(V3<float> { p.scales[3 * i], p.scales[3 * i + 1], p.scales[3 * i + 2] }, cam.cov_scale_multiplier);
    const float* q = p.rotations + 4 * size_t(i);
    const M3<float> R = quat_to_mat3(q[0], q[1], q[2], q[3]);
    const Gaussian2d<float> g2 = splat_project(p.form, p.weights[i], mu, sc, R, cam, 0.3f);
    const S2<float> M = inverse2(g2.cov);
    const float G00 = a[2], G01 = a[3] * 0.5f, G11 = a[4];
    // H = -M G M (2x2 symmetric)
    const float MG00 = M.v[0] * G00 + M.v[1] * G01, MG01 = M.v[0] * G01 + M.v[1] * G11;
    const float MG10 = M.v[1] * G00 + M.v[2] * G01, MG11 = M.v[1] * G01 + M.v[2] * G11;
    const float H00 = -(MG00 * M.v[0] + MG01 * M.v[1]);
    const float H01 = -(MG00 * M.v[1] + MG01 * M.v[2]);
    const float H11 = -(MG10 * M.v[1] + MG11 * M.v[2]);
    const S2<float> g_cov = { { H00, 2.f * H01, H11 } };
    float g_weight = 0.f;
    V3<float> g_mu = { 0.f, 0.f, 0.f }, g_s = { 0.f, 0.f, 0.f };
    float g_q[4] = { 0.f, 0.f, 0.f, 0.f };
    grad_splat(p.form, p.weights[i], mu, sc, q[0], q[1], q[2], q[3], cam, 0.3f, a[5], V2<float> { a[0], a[1] }, g_cov, &g_weight, &g_mu, &g_s, g_q);
    const V3<float> campos = { cam.campos[0], cam.campos[1], cam.campos[2] };
    const V3<float> v = sub3(mu, campos);
    const float vl = dgmr_fm::sqrt_f(dot3(v, v));
    const V3<float> dir = mul3(v, 1.f / vl);
    const V3<float> g_dir
        = grad_sh_to_colour(p.sh, i, p.sh_stride, p.sh_degree, dir, V3<float> { a[6], a[7], a[8] }, p.clamped + 3 * size_t(o), 0.f, row, kAddSh);
    const float gd = dot3(g_dir, dir);
    g_mu = add3(g_mu, mul3(sub3(g_dir, mul3(dir, gd)), 1.f / vl));
    sum.weight += g_weight;
    sum.mu = add3(sum.mu, g_mu);
    sum.s.x += g_s.x * cam.cov_scale_multiplier;
    sum.s.y += g_s.y * cam.cov_scale_multiplier;
    sum.s.z += g_s.z * cam.cov_scale_multiplier;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        sum.q[k] += g_q[k];
}

// kRows: through shared memory (store_sh_rows), else each thread stores its row.
template <bool kRows>
__global__ void __launch_bounds__(kBwdGaussThreads, 6) k_splat_bwd_gaussians(SplatBwdGauss p, CameraT<float> cam)
{
    extern __shared__ float sh_rows[];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int spacing = sh_row_words(p.sh_stride);
    if (i < p.N) {
        float* row = kRows ? sh_rows + threadIdx.x * spacing : p.g_sh + size_t(i) * 3 * p.sh_stride;
        GaussianGrads g;
        if (p.tiles_touched[i] != 0) {
            bwd_gaussian_one<false>(p, cam, i, i, g, row);
        } else {
            for (int k = 0; k < 3 * p.sh_stride; ++k)
                row[k] = 0.f;
        }
        store_gaussian_grads(p, i, g);
    }
    const uint32_t i0 = i & ~31u;
    if (kRows && i0 < p.N)
        store_sh_rows(p, sh_rows + (threadIdx.x & ~31u) * spacing, i0, min(32u, p.N - i0), int(threadIdx.x & 31u), spacing);
}

} // namespace dgmr

using namespace dgmr;

namespace {

bool bad_sizes(int32_t n, int32_t w, int32_t h, int64_t cap)
{
    return n < 0 || w <= 0 || h <= 0 || w > 65536 || h > 65536 || cap < 0 || cap > int64_t(0x7fffffff);
}

SplatPre make_pre(const dgmr_scene* scene, const SplatLayout& L)
{
    return SplatPre { uint32_t(scene->n_gaussians), static_cast<const float*>(scene->centroids), static_cast<const float*>(scene->sh), scene->sh_stride,
        scene->sh_degree, static_cast<const float*>(scene->weights), static_cast<const float*>(scene->scales), static_cast<const float*>(scene->rotations),
        L.rects, L.rgb, L.clamped, L.depths, L.xy, L.conic_opacity, L.tiles_touched, L.tile_rect, L.bin.depth_key, L.bin.perm, L.blend_rec,
        scene_formulation(scene, Formulation::Ots) };
}

SingleFrame single_frame(const CameraT<float>& cam, float* fb, const SplatLayout& L, const float* grad_fb = nullptr)
{
    return SingleFrame { cam.W, cam.H, cam.gx, cam.bg[0], cam.bg[1], cam.bg[2], fb, L.final_T, L.n_contrib, grad_fb };
}

// per-Gaussian preprocess and the inclusive scan (splat_forward.cu:70-139)
void launch_preprocess(const dgmr_scene* scene, const CameraT<float>& cam, const SplatLayout& L, uint32_t* st_dev, cudaStream_t s)
{
    const uint32_t N = uint32_t(scene->n_gaussians);
    cudaMemsetAsync(st_dev, 0, 16, s);
    if (N == 0)
        return;
    k_splat_preprocess<<<(N + 255) / 256, 256, 0, s>>>(make_pre(scene, L), cam);
    note_launch();
    inclusive_scan_u32(L.tiles_touched, L.point_offsets, N, L.bin.scan_tmp, ChainStream(s, kChainAlways));
}

// Launch order of the blend's tiles, heaviest first, from a predicted cost
// (scheduling only: results never depend on it).  A tile's block walks its
// list until every pixel is saturated, so the cost is the list length L for a
// tile that some pixel never saturates, and far less for one that is densely
// covered: the longest lists belong to dense tiles that saturate within a few
// hundred entries, and ordering by length alone starts the truly slow tiles
// late.  From the first 128 entries of its list, one warp per tile estimates
// the coverage of each 8x8 quadrant (summed opacity of the splats whose cutoff
// ellipse holds the quadrant's centre pixel, per entry); the least covered
// quadrant inside the frame sets the walk: cost = min(L, 100 / density), kept
// as a bucket of a quarter octave (0 = heaviest).  The last block to finish
// (counter n_sort[6], zeroed by the binning) counting-sorts the tiles by bucket
// with warp-aggregated shared atomics (most tiles share the "empty" bucket)
// and resets the counter.  On 1080p frames of 1M Gaussians this order ends
// the blend 5-26 % sooner than ordering by list length.
constexpr int kCostBuckets = 128;
constexpr uint32_t kOrderWarps = 8;
constexpr uint32_t kOrderPerThread = 16; // buckets a thread of the last block loads at once

template <class Frames>
__global__ void __launch_bounds__(kOrderWarps * 32) k_blend_tile_order(const int32_t* __restrict__ ranges, const uint32_t* __restrict__ list,
    const float4* __restrict__ rec, uint32_t N, uint32_t cap, uint32_t n_tiles, uint32_t* __restrict__ bucket, uint32_t* __restrict__ blocks_done,
    uint32_t* __restrict__ order, const __grid_constant__ Frames frames)
{
    chain_start();
    constexpr int kSample = 128;
    __shared__ uint32_t count[kCostBuckets];
    __shared__ uint32_t cursor[kCostBuckets];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x * kOrderWarps + (threadIdx.x >> 5);
    if (tile < n_tiles) {
        const FrameRef f = frames.frame(tile);
        const int32_t b = ranges[2 * tile], e = ranges[2 * tile + 1];
        uint32_t bk = kCostBuckets - 1; // empty (or flagged by the blend): lightest
        if (b >= 0 && e > b && uint32_t(e) <= cap) {
            const unsigned tx = f.tile % f.gx, ty = f.tile / f.gx;
            const float x0 = float(tx * kTile), y0 = float(ty * kTile);
            const int n = min(e - b, kSample);
            float hit[4] = { 0.f, 0.f, 0.f, 0.f };
            // the sample's list entries, then their records, all requested
            // before the first is used (kSample / 32 entries per lane)
            constexpr int kPerLane = kSample / 32;
            uint32_t gs[kPerLane];
#pragma unroll
            for (int i = 0; i < kPerLane; ++i) {
                const int k = lane + 32 * i;
                gs[i] = k < n ? list[b + k] : 0xffffffffu;
            }
            float4 r0s[kPerLane], r1s[kPerLane];
#pragma unroll
            for (int i = 0; i < kPerLane; ++i) {
                const size_t g = gs[i] < N ? gs[i] : 0u;
                r0s[i] = rec[2 * g];
                r1s[i] = rec[2 * g + 1];
            }
#pragma unroll
            for (int i = 0; i < kPerLane; ++i) {
                if (gs[i] >= N)
                    continue;
                const float4 r0 = r0s[i], r1 = r1s[i];
#pragma unroll
                for (int qd = 0; qd < 4; ++qd) {
                    const float dx = x0 + ((qd & 1) ? 12.f : 4.f) - r0.x;
                    const float dy = y0 + ((qd & 2) ? 12.f : 4.f) - r0.y;
                    const float q = r0.z * dx * dx + r1.x * dx * dy + r0.w * dy * dy;
                    hit[qd] += q <= r1.z ? r1.y : 0.f;
                }
            }
#pragma unroll
            for (int qd = 0; qd < 4; ++qd)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    hit[qd] += __shfl_xor_sync(0xffffffffu, hit[qd], o);
            float dmin = 3.0e38f;
#pragma unroll
            for (int qd = 0; qd < 4; ++qd)
                if (tx * kTile + ((qd & 1) ? 12u : 4u) < f.W && ty * kTile + ((qd & 2) ? 12u : 4u) < f.H)
                    dmin = fminf(dmin, hit[qd] / float(n));
            const float cost = dmin > 1.0e37f ? 0.f : fminf(float(e - b), 100.f / fmaxf(dmin, 1.0e-4f));
            const int level = int(4.f * __log2f(cost + 1.f));
            bk = uint32_t(kCostBuckets - 1 - min(max(level, 0), kCostBuckets - 1));
        }
        if (lane == 0)
            bucket[tile] = bk;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        is_last = atomicAdd(blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last)
        return;
    __threadfence();
    // counting sort by bucket: count every tile, an exclusive prefix over the
    // buckets, then scatter; each sweep loads kOrderPerThread buckets per
    // thread at once so that their latencies overlap
    const unsigned below = (1u << lane) - 1u;
    const uint32_t sweep = kOrderPerThread * blockDim.x;
    const auto load = [&](uint32_t s0, uint32_t (&bk)[kOrderPerThread]) {
#pragma unroll
        for (uint32_t i = 0; i < kOrderPerThread; ++i) {
            const uint32_t t = s0 + i * blockDim.x + threadIdx.x;
            bk[i] = t < n_tiles ? min(__ldcg(bucket + t), uint32_t(kCostBuckets - 1)) : 0xffffffffu;
        }
    };
    if (threadIdx.x < kCostBuckets)
        count[threadIdx.x] = 0;
    __syncthreads();
    for (uint32_t s0 = 0; s0 < n_tiles; s0 += sweep) {
        uint32_t bk[kOrderPerThread];
        load(s0, bk);
#pragma unroll
        for (uint32_t i = 0; i < kOrderPerThread; ++i) {
            const unsigned peers = __match_any_sync(0xffffffffu, bk[i]);
            if (bk[i] != 0xffffffffu && lane == __ffs(peers) - 1)
                atomicAdd(&count[bk[i]], uint32_t(__popc(peers)));
        }
    }
    __syncthreads();
    if (threadIdx.x < 32) { // exclusive prefix of the counts, kCostBuckets / 32 per lane
        constexpr int kPer = kCostBuckets / 32;
        uint32_t v[kPer];
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            v[k] = count[lane * kPer + k];
            sum += v[k];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += up;
        }
        uint32_t run = incl - sum;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            cursor[lane * kPer + k] = run;
            run += v[k];
        }
    }
    __syncthreads();
    for (uint32_t s0 = 0; s0 < n_tiles; s0 += sweep) {
        uint32_t bk[kOrderPerThread];
        load(s0, bk);
#pragma unroll
        for (uint32_t i = 0; i < kOrderPerThread; ++i) {
            const unsigned peers = __match_any_sync(0xffffffffu, bk[i]);
            const int leader = __ffs(peers) - 1;
            uint32_t base = 0;
            if (bk[i] != 0xffffffffu && lane == leader)
                base = atomicAdd(&cursor[bk[i]], uint32_t(__popc(peers)));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (bk[i] != 0xffffffffu)
                order[base + uint32_t(__popc(peers & below))] = s0 + i * blockDim.x + threadIdx.x;
        }
    }
    if (threadIdx.x == 0)
        *blocks_done = 0u;
}

template <class Frames>
void launch_tile_order(const SplatLayout& L, int par, uint32_t N, uint32_t cap, uint32_t n_tiles, const Frames& frames, cudaStream_t s)
{
    if (n_tiles == 0)
        return;
    launch_chained(k_blend_tile_order<Frames>, (n_tiles + kOrderWarps - 1) / kOrderWarps, kOrderWarps * 32, 0,
        ChainStream(s, blend_fits_chip(n_tiles)), L.ranges, L.bin.pair_val[par], L.blend_rec, N, cap,
        n_tiles, L.tile_cost, L.bin.n_sort + 6, L.tile_order, frames);
    note_launch();
}

// binning (after the preprocess) and the blend
void launch_render(const dgmr_scene* scene, const CameraT<float>& cam, float* fb, SplatLayout& L, uint32_t cap, uint32_t* st_dev, cudaStream_t s)
{
    const uint32_t N = uint32_t(scene->n_gaussians);
    const int par
        = run_binning<float>(N, cam.gx, cam.gy, L.tiles_touched, L.point_offsets, L.rects, L.xy, cap, L.bin, L.ranges, st_dev, num_sms(), s, true, true, L.tile_rect);
    launch_tile_order(L, par, N, cap, cam.gx * cam.gy, single_frame(cam, fb, L), s);
    launch_blend(kBlendSide, cam.gx * cam.gy, L.ranges, L.bin.pair_val[par], L.blend_rec, L.rgb, N, cap, st_dev, L.tile_order, single_frame(cam, fb, L), s);
}

} // namespace

extern "C" {

size_t dgmr_splat_frame_workspace_size(int32_t n_gaussians, int32_t width, int32_t height)
{
    if (bad_sizes(n_gaussians, width, height, 0))
        return 0;
    return splat_layout(uint32_t(n_gaussians), uint32_t(width), uint32_t(height), 0, nullptr, nullptr).bytes;
}

size_t dgmr_splat_pair_workspace_size(int32_t n_gaussians, int64_t pair_capacity)
{
    if (bad_sizes(n_gaussians, 1, 1, pair_capacity))
        return 0;
    return splat_layout(uint32_t(n_gaussians), 1, 1, uint32_t(pair_capacity), nullptr, nullptr).pair_bytes;
}

dgmr_status dgmr_splat_workspace_views(int32_t n_gaussians, int32_t width, int32_t height, int64_t pair_capacity, void* frame_workspace,
    size_t frame_workspace_bytes, void* pair_workspace, size_t pair_workspace_bytes, dgmr_splat_views* views)
{
    if (!views || !frame_workspace || bad_sizes(n_gaussians, width, height, pair_capacity) || (pair_capacity > 0 && !pair_workspace))
        return DGMR_ERR_BAD_ARG;
    const uint32_t W = uint32_t(width), H = uint32_t(height);
    const SplatLayout L = splat_layout(uint32_t(n_gaussians), W, H, uint32_t(pair_capacity), frame_workspace, pair_workspace);
    if (frame_workspace_bytes < L.bytes || pair_workspace_bytes < L.pair_bytes)
        return DGMR_ERR_WORKSPACE;
    const uint32_t gx = (W + kTile - 1) / kTile, gy = (H + kTile - 1) / kTile;
    const int par = tile_sort_parity(super_count(gx, gy));
    views->rects = L.rects;
    views->rgb = L.rgb;
    views->rgb_sh_clamped = L.clamped;
    views->depths = L.depths;
    views->points_xy_image = L.xy;
    views->conic_opacity = L.conic_opacity;
    views->tiles_touched = reinterpret_cast<int32_t*>(L.tiles_touched);
    views->point_offsets = reinterpret_cast<int32_t*>(L.point_offsets);
    views->i_ranges = L.ranges;
    views->point_list = pair_workspace ? reinterpret_cast<int32_t*>(L.bin.pair_val[par]) : nullptr;
    views->point_list_tiles = pair_workspace ? L.bin.pair_tile[par] : nullptr;
    views->final_transmittance = L.final_T;
    views->n_contrib = L.n_contrib;
    return DGMR_OK;
}

dgmr_status dgmr_splat_preprocess(const dgmr_scene* scene, const dgmr_camera* camera, void* frame_workspace, size_t frame_workspace_bytes,
    dgmr_frame_stats* stats, dgmr_stream stream)
{
    dgmr_status st = check_scene(scene, camera, DGMR_F32);
    if (st != DGMR_OK)
        return st;
    if (!frame_workspace)
        return DGMR_ERR_BAD_ARG;
    const SplatLayout L = splat_layout(uint32_t(scene->n_gaussians), uint32_t(camera->width), uint32_t(camera->height), 0, frame_workspace, nullptr);
    if (frame_workspace_bytes < L.bytes)
        return DGMR_ERR_WORKSPACE;
    const CameraT<float> cam = make_camera<float>(*camera);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : L.stats;
    launch_preprocess(scene, cam, L, st_dev, s);
    if (scene->n_gaussians > 0) {
        launch_chained(k_pair_count, 1, 1, 0, ChainStream(s, kChainAlways), L.point_offsets, uint32_t(scene->n_gaussians), 0xffffffffu, st_dev, L.bin.n_sort);
        note_launch();
    }
    return launch_status();
}

dgmr_status dgmr_splat_render(const dgmr_scene* scene, const dgmr_camera* camera, float* framebuffer, void* frame_workspace, size_t frame_workspace_bytes,
    void* pair_workspace, size_t pair_workspace_bytes, int64_t pair_capacity, dgmr_frame_stats* stats, dgmr_stream stream)
{
    dgmr_status st = check_scene(scene, camera, DGMR_F32);
    if (st != DGMR_OK)
        return st;
    if (!framebuffer || !frame_workspace || pair_capacity < 0 || pair_capacity > int64_t(0x7fffffff) || (pair_capacity > 0 && !pair_workspace))
        return DGMR_ERR_BAD_ARG;
    SplatLayout L = splat_layout(uint32_t(scene->n_gaussians), uint32_t(camera->width), uint32_t(camera->height), uint32_t(pair_capacity), frame_workspace,
        pair_workspace);
    if (frame_workspace_bytes < L.bytes || pair_workspace_bytes < L.pair_bytes)
        return DGMR_ERR_WORKSPACE;
    const CameraT<float> cam = make_camera<float>(*camera);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : L.stats;
    launch_render(scene, cam, framebuffer, L, uint32_t(pair_capacity), st_dev, s);
    return launch_status();
}

dgmr_status dgmr_splat_forward(const dgmr_scene* scene, const dgmr_camera* camera, float* framebuffer, void* frame_workspace, size_t frame_workspace_bytes,
    void* pair_workspace, size_t pair_workspace_bytes, int64_t pair_capacity, dgmr_frame_stats* stats, dgmr_stream stream)
{
    dgmr_status st = check_scene(scene, camera, DGMR_F32);
    if (st != DGMR_OK)
        return st;
    if (!framebuffer || !frame_workspace || pair_capacity < 0 || pair_capacity > int64_t(0x7fffffff) || (pair_capacity > 0 && !pair_workspace))
        return DGMR_ERR_BAD_ARG;
    SplatLayout L = splat_layout(uint32_t(scene->n_gaussians), uint32_t(camera->width), uint32_t(camera->height), uint32_t(pair_capacity), frame_workspace,
        pair_workspace);
    if (frame_workspace_bytes < L.bytes || pair_workspace_bytes < L.pair_bytes)
        return DGMR_ERR_WORKSPACE;
    const CameraT<float> cam = make_camera<float>(*camera);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : L.stats;
    launch_preprocess(scene, cam, L, st_dev, s);
    launch_render(scene, cam, framebuffer, L, uint32_t(pair_capacity), st_dev, s);
    return launch_status();
}

dgmr_status dgmr_splat_blend(const dgmr_camera* camera, int32_t n_gaussians, float* framebuffer, void* frame_workspace, size_t frame_workspace_bytes,
    void* pair_workspace, size_t pair_workspace_bytes, int64_t pair_capacity, dgmr_stream stream)
{
    if (!camera || !framebuffer || !frame_workspace || bad_sizes(n_gaussians, camera->width, camera->height, pair_capacity)
        || (pair_capacity > 0 && !pair_workspace))
        return DGMR_ERR_BAD_ARG;
    const SplatLayout L = splat_layout(uint32_t(n_gaussians), uint32_t(camera->width), uint32_t(camera->height), uint32_t(pair_capacity), frame_workspace,
        pair_workspace);
    if (frame_workspace_bytes < L.bytes || pair_workspace_bytes < L.pair_bytes)
        return DGMR_ERR_WORKSPACE;
    const CameraT<float> cam = make_camera<float>(*camera);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int par = tile_sort_parity(super_count(cam.gx, cam.gy));
    launch_blend(kBlendSide, cam.gx * cam.gy, L.ranges, L.bin.pair_val[par], L.blend_rec, L.rgb, uint32_t(n_gaussians), uint32_t(pair_capacity), L.stats,
        L.tile_order, single_frame(cam, framebuffer, L), s);
    return launch_status();
}

dgmr_status dgmr_splat_backward(const dgmr_scene* scene, const dgmr_camera* camera, const float* grad_framebuffer, float* grad_sh, float* grad_weights,
    float* grad_centroids, float* grad_scales, float* grad_rotations, void* frame_workspace, size_t frame_workspace_bytes, void* pair_workspace,
    size_t pair_workspace_bytes, int64_t pair_capacity, dgmr_stream stream)
{
    dgmr_status st = check_scene(scene, camera, DGMR_F32);
    if (st != DGMR_OK)
        return st;
    // per-Gaussian outputs may have no address when there are no Gaussians
    const bool grads_ok = scene->n_gaussians == 0 || (grad_sh && grad_weights && grad_centroids && grad_scales && grad_rotations);
    if (!grad_framebuffer || !grads_ok || !frame_workspace || pair_capacity < 0 || pair_capacity > int64_t(0x7fffffff)
        || (pair_capacity > 0 && !pair_workspace))
        return DGMR_ERR_BAD_ARG;
    const uint32_t N = uint32_t(scene->n_gaussians);
    const SplatLayout L = splat_layout(N, uint32_t(camera->width), uint32_t(camera->height), uint32_t(pair_capacity), frame_workspace, pair_workspace);
    if (frame_workspace_bytes < L.bytes || pair_workspace_bytes < L.pair_bytes)
        return DGMR_ERR_WORKSPACE;
    if (N == 0)
        return DGMR_OK;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const CameraT<float> cam = make_camera<float>(*camera);
    const int par = tile_sort_parity(super_count(cam.gx, cam.gy));
    cudaMemsetAsync(L.grad_acc, 0, size_t(N) * 9 * sizeof(double), s);
    launch_blend_bwd(cam.gx * cam.gy, L.ranges, L.bin.pair_val[par], L.blend_rec, L.rgb, N, L.grad_acc, L.tile_order,
        single_frame(cam, nullptr, L, grad_framebuffer), s);
    SplatBwdGauss p { N, static_cast<const float*>(scene->centroids), static_cast<const float*>(scene->sh), scene->sh_stride, scene->sh_degree,
        static_cast<const float*>(scene->weights), static_cast<const float*>(scene->scales), static_cast<const float*>(scene->rotations), L.clamped,
        L.tiles_touched, L.grad_acc, grad_sh, grad_weights, grad_centroids, grad_scales, grad_rotations, scene_formulation(scene, Formulation::Ots) };
    const uint32_t blocks = (N + kBwdGaussThreads - 1) / kBwdGaussThreads;
    if (p.sh_stride > kShDirect)
        k_splat_bwd_gaussians<true><<<blocks, kBwdGaussThreads, size_t(kBwdGaussThreads) * sh_row_words(p.sh_stride) * sizeof(float), s>>>(p, cam);
    else
        k_splat_bwd_gaussians<false><<<blocks, kBwdGaussThreads, 0, s>>>(p, cam);
    note_launch(2);
    return launch_status();
}

} // extern "C"

// ---------------------------------------------------------------------------
// Batched multi-view rendering over the view table of dgmr_batch.cuh.

namespace dgmr {

__global__ void __launch_bounds__(256) k_batch_preprocess(SplatPre out, const __grid_constant__ BatchTable tab)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= tab.G)
        return;
    const uint32_t v = BatchTable::owner(tab.g_off, tab.n_views, g);
    const BatchView& bv = tab.views[v];
    const BatchScene& sc = tab.scenes[bv.scene];
    SplatPre p = out;
    p.N = sc.n;
    p.centroids = sc.centroids;
    p.sh = sc.sh;
    p.sh_stride = sc.sh_stride;
    p.sh_degree = sc.sh_degree;
    p.weights = sc.weights;
    p.scales = sc.scales;
    p.rotations = sc.rotations;
    p.form = sc.form;
    preprocess_one(p, bv.cam, g - tab.g_off[v], g);
}

// per scene Gaussian: the chain rule of every view of its scene, added in view
// order (deterministic, no atomics)
__global__ void __launch_bounds__(kBwdGaussThreads, 6) k_batch_bwd_gaussians(SplatBwdGauss state, const __grid_constant__ BatchTable tab)
{
    extern __shared__ float sh_rows[];
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t total = tab.scene_off[tab.n_scenes];
    const bool in = k < total;
    const uint32_t s = BatchTable::owner(tab.scene_off, tab.n_scenes, in ? k : total - 1u);
    const BatchScene& sc = tab.scenes[s];
    const uint32_t i = k - tab.scene_off[s];
    SplatBwdGauss p = state;
    p.N = sc.n;
    p.centroids = sc.centroids;
    p.sh = sc.sh;
    p.sh_stride = sc.sh_stride;
    p.sh_degree = sc.sh_degree;
    p.weights = sc.weights;
    p.scales = sc.scales;
    p.rotations = sc.rotations;
    p.g_sh = sc.g_sh;
    p.g_weights = sc.g_weights;
    p.g_centroids = sc.g_centroids;
    p.g_scales = sc.g_scales;
    p.g_rotations = sc.g_rotations;
    p.form = sc.form;
    // state.sh_stride: the largest of the scenes, by which the threads' rows are spaced
    const int spacing = sh_row_words(state.sh_stride);
    float* row = sh_rows + threadIdx.x * spacing;
    const bool wanted = in && sc.g_sh; // a scene entry may have no gradient outputs
    if (wanted) {
        for (int c = 0; c < 3 * p.sh_stride; ++c)
            row[c] = 0.f;
        GaussianGrads g;
        for (uint32_t q = sc.view_begin; q < sc.view_end; ++q) {
            const uint32_t v = tab.view_by_scene[q];
            const uint32_t o = tab.g_off[v] + i;
            if (tab.views[v].grad_fb && p.tiles_touched[o] != 0)
                bwd_gaussian_one<true>(p, tab.views[v].cam, i, o, g, row);
        }
        store_gaussian_grads(p, i, g);
    }
    // a warp of one scene copies its rows out together; where two scenes meet, every lane its own
    const uint32_t there = __ballot_sync(0xffffffffu, in), want = __ballot_sync(0xffffffffu, wanted);
    const uint32_t first_scene = __shfl_sync(0xffffffffu, s, 0), first_row = __shfl_sync(0xffffffffu, i, 0);
    if (__all_sync(0xffffffffu, !in || s == first_scene)) {
        if (want)
            store_sh_rows(p, sh_rows + (threadIdx.x & ~31u) * spacing, first_row, uint32_t(__popc(there)), int(threadIdx.x & 31u), spacing);
    } else if (wanted) {
        for (int c = 0; c < 3 * p.sh_stride; ++c)
            p.g_sh[size_t(i) * 3 * p.sh_stride + c] = row[c];
    }
}

} // namespace dgmr

namespace {

struct BatchPlan {
    BatchTable tab;
    SplatLayout L;
    size_t px_total;
    int blend_side; // the blend's block side (dgmr_batch_view.blend_block)
};

// Validates the batch and builds its table and workspace layout.  grads may be
// null (forward).  Bases may be null (size query).
dgmr_status make_batch(const dgmr_scene* scenes, int32_t n_scenes, const dgmr_batch_view* views, int32_t n_views, const dgmr_scene_grads* grads,
    int64_t pair_capacity, void* frame_ws, void* pair_ws, BatchPlan& plan)
{
    if (pair_capacity < 0 || pair_capacity > int64_t(0x7fffffff))
        return DGMR_ERR_BAD_ARG;
    BatchTable& t = plan.tab;
    const dgmr_status st = build_batch_table(scenes, n_scenes, views, n_views, grads, Formulation::Ots, t);
    if (st != DGMR_OK)
        return st;
    const int side = views[0].blend_block;
    if (side != 0 && side != 8 && side != 16)
        return DGMR_ERR_BAD_ARG;
    for (int v = 1; v < n_views; ++v)
        if (views[v].blend_block != 0 && views[v].blend_block != side)
            return DGMR_ERR_BAD_ARG;
    plan.blend_side = side ? side : kBlendSide;
    plan.px_total = t.px_total;
    plan.L = splat_layout_n(t.G, t.n_tiles, plan.px_total, uint32_t(pair_capacity), frame_ws, pair_ws);
    t.final_T = plan.L.final_T;
    t.n_contrib = plan.L.n_contrib;
    return DGMR_OK;
}

SplatPre batch_pre(const SplatLayout& L, uint32_t G)
{
    return SplatPre { G, nullptr, nullptr, 1, 0, nullptr, nullptr, nullptr, L.rects, L.rgb, L.clamped, L.depths, L.xy, L.conic_opacity, L.tiles_touched, L.tile_rect,
        L.bin.depth_key, L.bin.perm, L.blend_rec, Formulation::Ots };
}

// need_pairs = false for the preprocess alone, which touches no pair buffer
dgmr_status batch_check_ws(const BatchPlan& plan, void* frame_ws, size_t frame_bytes, void* pair_ws, size_t pair_bytes, int64_t pair_capacity,
    bool need_pairs = true)
{
    if (!frame_ws || (need_pairs && pair_capacity > 0 && !pair_ws))
        return DGMR_ERR_BAD_ARG;
    if (frame_bytes < plan.L.bytes || (need_pairs && pair_bytes < plan.L.pair_bytes))
        return DGMR_ERR_WORKSPACE;
    return DGMR_OK;
}

void batch_preprocess(const BatchPlan& plan, uint32_t* st_dev, cudaStream_t s)
{
    const SplatLayout& L = plan.L;
    const uint32_t G = plan.tab.G;
    cudaMemsetAsync(st_dev, 0, 16, s);
    if (G == 0)
        return;
    k_batch_preprocess<<<(G + 255) / 256, 256, 0, s>>>(batch_pre(L, G), plan.tab);
    note_launch();
    inclusive_scan_u32(L.tiles_touched, L.point_offsets, G, L.bin.scan_tmp, ChainStream(s, G <= kChainMost));
}

} // namespace

extern "C" {

dgmr_status dgmr_splat_batch_workspace_size(const dgmr_scene* scenes, int32_t n_scenes, const dgmr_batch_view* views, int32_t n_views, int64_t pair_capacity,
    size_t* frame_workspace_bytes, size_t* pair_workspace_bytes)
{
    if (!frame_workspace_bytes || !pair_workspace_bytes)
        return DGMR_ERR_BAD_ARG;
    static thread_local BatchPlan plan;
    const dgmr_status st = make_batch(scenes, n_scenes, views, n_views, nullptr, pair_capacity, nullptr, nullptr, plan);
    if (st != DGMR_OK)
        return st;
    *frame_workspace_bytes = plan.L.bytes;
    *pair_workspace_bytes = plan.L.pair_bytes;
    return DGMR_OK;
}

dgmr_status dgmr_splat_batch_preprocess(const dgmr_scene* scenes, int32_t n_scenes, const dgmr_batch_view* views, int32_t n_views, void* frame_workspace,
    size_t frame_workspace_bytes, dgmr_frame_stats* stats, dgmr_stream stream)
{
    static thread_local BatchPlan plan;
    dgmr_status st = make_batch(scenes, n_scenes, views, n_views, nullptr, 0, frame_workspace, nullptr, plan);
    if (st != DGMR_OK)
        return st;
    st = batch_check_ws(plan, frame_workspace, frame_workspace_bytes, nullptr, 0, 0, false);
    if (st != DGMR_OK)
        return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : plan.L.stats;
    batch_preprocess(plan, st_dev, s);
    if (plan.tab.G > 0) {
        launch_chained(k_pair_count, 1, 1, 0, ChainStream(s, kChainAlways), plan.L.point_offsets, plan.tab.G, 0xffffffffu, st_dev, plan.L.bin.n_sort);
        note_launch();
    }
    return launch_status();
}

dgmr_status dgmr_splat_batch_forward(const dgmr_scene* scenes, int32_t n_scenes, const dgmr_batch_view* views, int32_t n_views, void* frame_workspace,
    size_t frame_workspace_bytes, void* pair_workspace, size_t pair_workspace_bytes, int64_t pair_capacity, dgmr_frame_stats* stats, dgmr_stream stream)
{
    static thread_local BatchPlan plan;
    dgmr_status st = make_batch(scenes, n_scenes, views, n_views, nullptr, pair_capacity, frame_workspace, pair_workspace, plan);
    if (st != DGMR_OK)
        return st;
    st = batch_check_ws(plan, frame_workspace, frame_workspace_bytes, pair_workspace, pair_workspace_bytes, pair_capacity);
    if (st != DGMR_OK)
        return st;
    for (int v = 0; v < n_views; ++v)
        if (!views[v].framebuffer)
            return DGMR_ERR_BAD_ARG;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    SplatLayout& L = plan.L;
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : L.stats;
    const uint32_t G = plan.tab.G, cap = uint32_t(pair_capacity);
    batch_preprocess(plan, st_dev, s);
    const int par = run_binning_grids<float>(G, plan.tab.n_tiles, plan.tab.n_stiles, plan.tab, L.tiles_touched, L.point_offsets, L.rects, L.xy, cap, L.bin, L.ranges, st_dev,
        num_sms(), s, true, false, L.tile_rect);
    launch_tile_order(L, par, G, cap, plan.tab.n_tiles, plan.tab, s);
    launch_blend(plan.blend_side, plan.tab.n_tiles, L.ranges, L.bin.pair_val[par], L.blend_rec, L.rgb, G, cap, st_dev, L.tile_order, plan.tab, s);
    note_launch();
    return launch_status();
}

dgmr_status dgmr_splat_batch_backward(const dgmr_scene* scenes, int32_t n_scenes, const dgmr_batch_view* views, int32_t n_views,
    const dgmr_scene_grads* grads, void* frame_workspace, size_t frame_workspace_bytes, void* pair_workspace, size_t pair_workspace_bytes,
    int64_t pair_capacity, dgmr_stream stream)
{
    if (!grads)
        return DGMR_ERR_BAD_ARG;
    static thread_local BatchPlan plan;
    dgmr_status st = make_batch(scenes, n_scenes, views, n_views, grads, pair_capacity, frame_workspace, pair_workspace, plan);
    if (st != DGMR_OK)
        return st;
    st = batch_check_ws(plan, frame_workspace, frame_workspace_bytes, pair_workspace, pair_workspace_bytes, pair_capacity);
    if (st != DGMR_OK)
        return st;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const SplatLayout& L = plan.L;
    const uint32_t G = plan.tab.G;
    const uint32_t n_scene_gaussians = plan.tab.scene_off[n_scenes];
    if (n_scene_gaussians == 0)
        return DGMR_OK;
    const int par = tile_sort_parity(plan.tab.n_stiles);
    cudaMemsetAsync(L.grad_acc, 0, size_t(G) * 9 * sizeof(double), s);
    launch_blend_bwd(plan.tab.n_tiles, L.ranges, L.bin.pair_val[par], L.blend_rec, L.rgb, G, L.grad_acc, L.tile_order, plan.tab, s);
    int sh_stride = 1;
    for (int32_t k = 0; k < n_scenes; ++k)
        sh_stride = scenes[k].sh_stride > sh_stride ? scenes[k].sh_stride : sh_stride;
    SplatBwdGauss state { 0, nullptr, nullptr, sh_stride, 0, nullptr, nullptr, nullptr, L.clamped, L.tiles_touched, L.grad_acc, nullptr, nullptr, nullptr, nullptr,
        nullptr, Formulation::Ots };
    k_batch_bwd_gaussians<<<(n_scene_gaussians + kBwdGaussThreads - 1) / kBwdGaussThreads, kBwdGaussThreads,
        size_t(kBwdGaussThreads) * sh_row_words(sh_stride) * sizeof(float), s>>>(state, plan.tab);
    note_launch(2);
    return launch_status();
}

} // extern "C"

// ---------------------------------------------------------------------------
// Splat forward without any device allocation.
//
// Some callers cannot hand this library a workspace: a plugin inside a host
// application that owns every byte of GPU memory through its own pool, or
// code running in a per-frame callback where a cudaMalloc would synchronise
// the whole device and stall everything else in flight.  For them the frame
// and pair workspaces live in one fixed-size array in device memory, defined
// below, which every GPU that loads this library keeps until the process
// exits.  A call whose two workspaces do not fit is rejected with
// DGMR_ERR_STATIC_SCRATCH; nothing else is allocated.
//
// The array is shared by every call on a device and keeps whatever the last
// call left in it.  The forward writes everything it later reads (the frame
// statistics and tile ranges are cleared on the stream at the start of each
// frame), so consecutive calls are independent -- but two calls that overlap
// on the GPU (different streams, no ordering between them) race on the array
// and corrupt each other's frame.

namespace {

constexpr size_t kStaticScratchBytes = size_t(64) << 20; // 64 MiB per device

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
void* g_static_ptr[kMaxDevices] = {};

// Device address of the scratch array on the current device.  Host code must
// not pass g_static_scratch itself to a kernel: on the host that name is only
// a stand-in for the device symbol.  Looked up once per device, on the first
// call made with that device current.
dgmr_status static_scratch(void** out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return DGMR_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || !p)
            return DGMR_ERR_CUDA;
        g_static_ptr[dev] = p;
    }
    *out = g_static_ptr[dev];
    return DGMR_OK;
}

} // namespace

extern "C" dgmr_status dgmr_splat_forward_noalloc(const dgmr_scene* scene, const dgmr_camera* camera, float* framebuffer, int64_t pair_capacity,
    dgmr_frame_stats* stats, dgmr_stream stream)
{
    dgmr_status st = check_scene(scene, camera, DGMR_F32);
    if (st != DGMR_OK)
        return st;
    if (!framebuffer || pair_capacity < 0 || pair_capacity > int64_t(0x7fffffff))
        return DGMR_ERR_BAD_ARG;
    const uint32_t N = uint32_t(scene->n_gaussians), W = uint32_t(camera->width), H = uint32_t(camera->height), cap = uint32_t(pair_capacity);
    const SplatLayout sizes = splat_layout(N, W, H, cap, nullptr, nullptr);
    const size_t frame_bytes = align_up(sizes.bytes);
    if (frame_bytes + sizes.pair_bytes > kStaticScratchBytes)
        return DGMR_ERR_STATIC_SCRATCH;
    void* base = nullptr;
    st = static_scratch(&base);
    if (st != DGMR_OK)
        return st;
    char* frame_ws = static_cast<char*>(base);
    char* pair_ws = frame_ws + frame_bytes;
    SplatLayout L = splat_layout(N, W, H, cap, frame_ws, pair_ws);
    const CameraT<float> cam = make_camera<float>(*camera);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    uint32_t* st_dev = stats ? reinterpret_cast<uint32_t*>(stats) : L.stats;
    launch_preprocess(scene, cam, L, st_dev, s);
    launch_render(scene, cam, framebuffer, L, cap, st_dev, s);
    st = launch_status();
    if (st != DGMR_OK || stats)
        return st;
    // No caller-visible statistics: the overflow flag sits in the static
    // array, so wait for the frame and report it as the call's status.
    uint32_t flags = 0;
    if (cudaMemcpyAsync(&flags, L.stats + 1, sizeof(flags), cudaMemcpyDeviceToHost, s) != cudaSuccess
        || cudaStreamSynchronize(s) != cudaSuccess)
        return DGMR_ERR_CUDA;
    return (flags & DGMR_FLAG_PAIR_OVERFLOW) ? DGMR_ERR_PAIR_OVERFLOW : DGMR_OK;
}

// ---------------------------------------------------------------------------
// A camera on the device, read by the host.

namespace {

constexpr int kCameraValues = 16 + 16 + 3 + 3;
static_assert(offsetof(dgmr_camera, proj) == offsetof(dgmr_camera, view) + 16 * sizeof(double)
        && offsetof(dgmr_camera, campos) == offsetof(dgmr_camera, proj) + 16 * sizeof(double)
        && offsetof(dgmr_camera, background) == offsetof(dgmr_camera, campos) + 3 * sizeof(double),
    "the four arrays follow one another");

// While it lives, this thread's allocations are no part of a capture that another thread has under way.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// pinned host memory that the kernel writes: one block per thread, kept until the thread ends
struct CameraStaging {
    double* host = nullptr;
    cudaError_t allocate(size_t bytes)
    {
        const RelaxedCapture relaxed;
        const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&host), bytes, cudaHostAllocPortable | cudaHostAllocMapped);
        if (e != cudaSuccess)
            host = nullptr;
        return e;
    }
    ~CameraStaging()
    {
        if (!host)
            return;
        const RelaxedCapture relaxed;
        cudaFreeHost(host);
    }
};

template <class T>
__global__ void k_camera_read(const T* __restrict__ view, const T* __restrict__ proj, const T* __restrict__ campos, const T* __restrict__ background,
    double* __restrict__ out)
{
    const int i = threadIdx.x;
    if (i < kCameraValues)
        out[i] = double(i < 16 ? view[i] : i < 32 ? proj[i - 16] : i < 35 ? campos[i - 32] : background[i - 35]);
}

} // namespace

extern "C" dgmr_status dgmr_camera_read(const void* view, const void* proj, const void* campos, const void* background, int32_t dtype, dgmr_camera* camera,
    dgmr_stream stream)
{
    if (!view || !proj || !campos || !background || !camera || (dtype != DGMR_F32 && dtype != DGMR_F64))
        return DGMR_ERR_BAD_ARG;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    // refused inside a capture, before anything touches the stream: the wait below would end the capture
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return DGMR_ERR_CUDA;
    }
    static thread_local CameraStaging staging;
    if (!staging.host && staging.allocate(kCameraValues * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        return DGMR_ERR_CUDA;
    }
    if (dtype == DGMR_F32)
        k_camera_read<<<1, 64, 0, s>>>(static_cast<const float*>(view), static_cast<const float*>(proj), static_cast<const float*>(campos),
            static_cast<const float*>(background), staging.host);
    else
        k_camera_read<<<1, 64, 0, s>>>(static_cast<const double*>(view), static_cast<const double*>(proj), static_cast<const double*>(campos),
            static_cast<const double*>(background), staging.host);
    note_launch();
    if (launch_status() != DGMR_OK || cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError(); // reported here, not by the next call
        return DGMR_ERR_CUDA;
    }
    std::memcpy(camera->view, staging.host, kCameraValues * sizeof(double));
    return DGMR_OK;
}
