// Volume march with one warp per ray (included by dgmr_marcher.cu).
//
// A ray's work is mostly its pass 2: for every Gaussian it can use, 127
// CDF differences -- and the heaviest rays of a frame set its duration.  With
// one thread per ray that work is a long dependent chain on one lane (with
// the 127 bins in local memory), so the kernel ends up waiting on a few
// rays while the SMs idle.  Here the 32 lanes of a warp share one ray:
//  * the tile's list is cut down to the entries the ray can use, once (RayList);
//    every pass walks those 32 at a time, one entry per lane (intersection with
//    the ray, gates), results exchanged by shuffles;
//  * lane l owns bins l, l+32, l+64, l+96 (four register bins); for each
//    Gaussian, in list order, every lane evaluates the CDF at its own
//    borders and takes the next border's value from its neighbour;
//  * a section is inserted by the whole warp, lane i holding section i (pass 1),
//    and the sample positions are written a section per lane;
//  * the sequential parts -- the blend and its adjoint peel -- run on every
//    lane in lockstep from shared values;
//  * in the backward every lane runs one Gaussian's adjoint over its bins.
// Per bin, Gaussian order and every arithmetic operation are those of the
// one-thread loops (vol_marcher_forward.cu:295-501, math.h:412-468), so the
// image is the same bits.  Warps are independent (no block barrier); blocks
// of kRayWarps rays are launched heaviest tile first.
#pragma once

#include "dgmr_f32x2.cuh"
#include "dgmr_section_warp.cuh"

namespace dgmr {

constexpr unsigned kRayWarps = 4; // rays per block
constexpr unsigned kRayRounds = 4; // 4 x 32 lanes = 128 borders
template <class T>
constexpr unsigned kRayList = sizeof(T) == 4 ? 1024 : 512; // list entries a ray can use that its warp keeps (RayList; 48 KB per block)

// A ray's section set lives in shared memory, once per warp: the warp inserts,
// every lane reads it after a __syncwarp (kept per lane, the 32 identical
// copies and the insertion's scratch went to local memory).
template <class T>
struct RayWarpShared {
    T borders[kSmallSteps];
    Bin<T> bins[kSmallSteps]; // (r, g, b, exp(-mass))
    SectionSet<kLargeSteps, T> sec;
    Section<T> pieces[2 * kLargeSteps + 1]; // warp_put_pieces: the merged sections of one insertion
    uint16_t use[kRayList<T>]; // RayList
};

template <class T>
struct RayWarpSharedBwd {
    T borders[kSmallSteps];
    Bin<T> bins[kSmallSteps];
    Bin<T> gbins[kSmallSteps]; // bin adjoints
    int32_t queue[64]; // pass 3: list entries waiting for a lane
    SectionSet<kLargeSteps, T> sec;
    union {
        Section<T> pieces[2 * kLargeSteps + 1]; // pass 1
        T inv_t[kSmallSteps]; // warp_peel: 1 / exp(-mass) of each bin
    };
    uint16_t use[kRayList<T>]; // RayList
};

// The entries of the tile's list that the ray can use (ray_can_use), as offsets
// into the list, packed in list order: `use` holds the first n of them, found
// in the list's first `raw` entries; entries from `raw` on are not packed (the
// list has more than kRayList usable entries, or offsets past 16 bits) and
// every pass tests them.  A warp reads the packed entries 32 at a time, one per
// lane, then the rest of the list.
// The passes of a large step intersect every usable entry again, and a ray can
// use few of its tile's entries: 175 of 545 at 100k Gaussians, 512^2, spread
// over 23 of the list's 23.6 batches of 32; 282 of 9500 in 151 of 298 batches at
// 64^2.  Packed, they fill 6 and 9 batches.  Against a bit mask per batch of 32
// (one sparse batch after the other): forward + backward 53.7 -> 40.4 ms at
// 100k, 512^2 (with the step store), 81.2 -> 38.8 ms for 16 batched 64^2 views,
// forward 2.43 -> 1.88 ms at 10k, 256^2.
struct RayList {
    const uint16_t* use;
    uint32_t n, raw;
};

// One list entry as seen by its lane.
template <class T>
struct RayEntry {
    uint32_t id;
    V3<T> mu;
    S3<T> Q;
    T mass, depth;
};

template <class T>
__device__ __forceinline__ RayEntry<T> load_entry(const VmMarch<T>& a, int32_t k)
{
    RayEntry<T> en;
    en.id = uint32_t(a.list[k]);
    const size_t id = en.id;
    en.mu = { a.centroids[3 * id], a.centroids[3 * id + 1], a.centroids[3 * id + 2] };
#pragma unroll
    for (int c = 0; c < 6; ++c)
        en.Q.v[c] = a.inv_cov[6 * id + c];
    en.mass = a.masses[id];
    en.depth = a.depths[id];
    return en;
}
// in float from the Gaussian's record: three 16-byte loads instead of eleven of 4
template <>
__device__ __forceinline__ RayEntry<float> load_entry<float>(const VmMarch<float>& a, int32_t k)
{
    RayEntry<float> en;
    en.id = uint32_t(a.list[k]);
    const float4* r = a.rec + size_t(kMarchRec) * en.id;
    const float4 q0 = r[0], q1 = r[1], m = r[2];
    en.Q = { { q0.x, q0.y, q0.z, q0.w, q1.x, q1.y } };
    en.mass = q1.z;
    en.depth = q1.w;
    en.mu = { m.x, m.y, m.z };
    return en;
}

// The frames a march launch covers.  A single frame: one camera (a kernel
// parameter) and the image planes of VmMarch.  A batch (VmBatchFrames, float)
// looks each tile's view up in its view table; its tiles are numbered across
// views and its rays index one array of all views' pixels.
template <class T>
struct VmSingleFrame {
    CameraT<T> cam0;
    __device__ __forceinline__ unsigned view(unsigned) const { return 0u; }
    __device__ __forceinline__ const CameraT<T>& cam(unsigned) const { return cam0; }
    __device__ __forceinline__ unsigned tile_base(unsigned) const { return 0u; }
    __device__ __forceinline__ size_t px_base(unsigned) const { return 0; }
    __device__ __forceinline__ size_t rays() const { return size_t(cam0.W) * cam0.H; }
    __device__ __forceinline__ T* fb(unsigned, const VmMarch<T>& a) const { return a.fb; }
    __device__ __forceinline__ T* remaining_T(unsigned, const VmMarch<T>& a) const { return a.remaining_T; }
    __device__ __forceinline__ const T* grad_fb(unsigned, const VmMarch<T>& a) const { return a.grad_fb; }
};

// Tile work order for the march: heaviest tile first (k_tile_order), so the
// longest rays start at the head of the grid.  tile = the launch-wide tile
// (it indexes the ranges), view = its frame, (px, py) = the ray's pixel there.
template <class T, class Frames>
__device__ __forceinline__ bool ray_pixel(const Frames& frames, const uint32_t* order, unsigned* tile, unsigned* view, unsigned* px, unsigned* py)
{
    const unsigned groups = kTilePixels / kRayWarps;
    const unsigned item = blockIdx.x / groups, group = blockIdx.x % groups;
    *tile = order ? order[item] : item;
    *view = frames.view(*tile);
    const CameraT<T>& cam = frames.cam(*view);
    const unsigned lt = *tile - frames.tile_base(*view);
    const unsigned p = group * kRayWarps + (threadIdx.x >> 5);
    *px = (lt % cam.gx) * kTile + (p % kTile);
    *py = (lt / cam.gx) * kTile + (p / kTile);
    return *px < cam.W && *py < cam.H;
}

// Tests the packed entries [from, to) exactly and packs the usable ones behind
// `from`; returns their end.
template <class T>
__device__ __forceinline__ uint32_t warp_refine_list(uint16_t* use, uint32_t from, uint32_t to, const VmMarch<T>& a, int32_t b, V3<T> o, V3<T> d, unsigned lane)
{
    uint32_t n = from;
    __syncwarp();
    for (uint32_t j = from; j < to; j += 32) {
        uint16_t k = 0;
        bool can = false;
        if (j + lane < to) {
            k = use[j + lane];
            const RayEntry<T> en = load_entry(a, b + int32_t(k));
            can = ray_can_use(intersect_with_ray_inv_C(en.mu, en.Q, o, d), en.mass);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, can); // every lane has read its entry
        if (can)
            use[n + uint32_t(__popc(m & lanes_below(int(lane))))] = k;
        n += uint32_t(__popc(m));
        __syncwarp();
    }
    return n;
}

// Whether the ray's mass on a Gaussian can reach 1/255, from the Gaussian's
// record (k_vm_records): its logarithm by approximate instructions, against the
// gate with a margin for the rounding of both this and the exact evaluation.
// With c = centre - origin: a = d'Qd, b = d'Qc, k = c'Qc; the exponent e = k -
// b^2 / a.  Each dot product is off by at most 6 ulp of the sum of its terms'
// magnitudes, which Q's positive definiteness bounds by tr Q |d|^2, tr Q |c| and t =
// tr Q |c|^2; together e is off by less than 28 ulp t (1 + tr Q / a) either way,
// e / 2 in base 2 by 2.4e-6 of that: 4e-6 and 1 on the whole are allowed.
struct RayQuick {
    float xx, yy, zz, xy, xz, yz; // products of the direction
    V3<float> d;
};
__device__ __forceinline__ bool ray_may_use(const RayQuick& r, float4 q0, float4 q1, float4 qc, float4 lt)
{
    const float a = __fmaf_rn(q0.x, r.xx, __fmaf_rn(q0.w, r.yy, __fmaf_rn(q1.y, r.zz, __fmaf_rn(q0.y, r.xy, __fmaf_rn(q0.z, r.xz, q1.x * r.yz)))));
    const float b = __fmaf_rn(qc.x, r.d.x, __fmaf_rn(qc.y, r.d.y, qc.z * r.d.z));
    const float inv = __fdividef(1.f, a);
    const float e = __fmaf_rn(-b * b, inv, qc.w);
    const float log_mass = lt.x - 0.5f * __log2f(a) - 0.72134752f * e;
    const float margin = __fmaf_rn(4.0e-6f * (lt.y + 1.f), __fmaf_rn((q0.x + q0.w) + q1.y, inv, 1.f), 1.f);
    return !(log_mass < -7.9943534f - margin); // log2(1/255); NaN: the exact test decides
}

// pass 0: the ray's usable entries, lane-parallel.  In float most of the list
// is turned away by ray_may_use, whose 30 instructions stand against 120 for the
// exact test; the candidates are packed, then tested exactly in full batches.
// (Every entry tested exactly, the list was 58 % of a ray's time at 64^2, where it
// has 9500 entries: 16 batched views forward + backward 35.5 -> 26.1 ms; at 100k,
// 512^2, with the records' wider loads, 34.8 -> 33.4.)
template <class T>
__device__ __forceinline__ RayList warp_ray_list(uint16_t* use, const VmMarch<T>& a, int32_t b, int32_t e, V3<T> o, V3<T> d, unsigned lane)
{
    uint32_t n = 0, raw = 0, exact = 0; // packed, list entries behind them, tested exactly
    const uint32_t len = e > b ? uint32_t(e - b) : 0u;
    RayQuick quick;
    if constexpr (sizeof(T) == 4)
        quick = RayQuick { d.x * d.x, d.y * d.y, d.z * d.z, 2.f * d.x * d.y, 2.f * d.x * d.z, 2.f * d.y * d.z, d };
    for (; raw < len && raw + 32u <= 0x10000u; raw += 32) {
        const uint32_t k = raw + lane;
        bool can = false;
        if (k < len) {
            if constexpr (sizeof(T) == 4) {
                const float4* r = a.rec + size_t(kMarchRec) * uint32_t(a.list[b + int32_t(k)]);
                can = ray_may_use(quick, r[0], r[1], r[3], r[4]);
            } else {
                const RayEntry<T> en = load_entry(a, b + int32_t(k));
                can = ray_can_use(intersect_with_ray_inv_C(en.mu, en.Q, o, d), en.mass);
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, can);
        if (sizeof(T) == 4 && n + uint32_t(__popc(m)) > kRayList<T> && exact < n)
            exact = n = warp_refine_list(use, exact, n, a, b, o, d, lane);
        if (n + uint32_t(__popc(m)) > kRayList<T>)
            break;
        if (can)
            use[n + uint32_t(__popc(m & lanes_below(int(lane))))] = uint16_t(k);
        n += uint32_t(__popc(m));
    }
    if (sizeof(T) == 4)
        n = warp_refine_list(use, exact, n, a, b, o, d, lane);
    __syncwarp();
    return RayList { use, n, min(raw, len) };
}

// The list entry of the lane in batch t of a pass (-1: none), and how many batches a pass has.
__device__ __forceinline__ uint32_t ray_batches(const RayList& rl, int32_t b, int32_t e) { return (rl.n + 31u) / 32u + (uint32_t(e - b) - rl.raw + 31u) / 32u; }
__device__ __forceinline__ int32_t ray_entry(const RayList& rl, int32_t b, int32_t e, uint32_t t, unsigned lane)
{
    const uint32_t packed = (rl.n + 31u) / 32u;
    if (t < packed) {
        const uint32_t j = 32u * t + lane;
        return j < rl.n ? b + int32_t(rl.use[j]) : -1;
    }
    const int32_t k = b + int32_t(rl.raw + 32u * (t - packed) + lane);
    return k < e ? k : -1;
}

} // namespace dgmr

namespace dgmr {

// warp_put as a call: the backward march, whose loop is sensitive to its code
// size (instruction fetch), is faster with the insertion out of line; the forward
// inlines it.
template <class T>
__device__ __noinline__ void warp_put_call(SectionSet<kLargeSteps, T>& sec, Section<T>* pieces, Section<T> s, unsigned lane)
{
    warp_put(sec, pieces, s, lane);
}

enum class PutMode { Inline, Call };

// sample_positions (marching_steps.h:202-220) by the warp, in the form of
// sample_positions_by_sections (dgmr_sections.h): lane j < n runs section j's
// chain -- counting its samples, then, after a prefix over the counts, writing
// them behind the samples of the sections before it -- and the lanes fill the
// rest with the last section's end.  The same positions, bit for bit, with the
// longest section's chain as the critical path instead of all 128 samples.
template <class T>
__device__ __forceinline__ void warp_sample_positions(const SectionSet<kLargeSteps, T>& d, T* out, unsigned lane)
{
    const unsigned n = d.n;
    if (n == 0) {
        for (unsigned k = lane; k < kSmallSteps; k += 32)
            out[k] = T(0);
        __syncwarp();
        return;
    }
    const unsigned len = lane < n ? section_samples<kSmallSteps>(d, lane) : 0u;
    unsigned incl = len;
#pragma unroll
    for (unsigned o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += t;
    }
    const unsigned off = 1u + incl - len; // out[0] is the first section's start
    const unsigned filled = 1u + __shfl_sync(0xffffffffu, incl, 31);
    if (lane == 0)
        out[0] = d.e[0].start;
    if (lane < n) {
        const T end = d.e[lane].end, dt = d.e[lane].delta_t;
        T v = lane == 0 ? d.e[0].start : d.e[lane - 1].end;
        for (unsigned k = 0; k < len && off + k < kSmallSteps; ++k) {
            v = min_f(end, v + dt);
            out[off + k] = v;
        }
    }
    const T last = d.e[n - 1].end;
    for (unsigned k = filled + lane; k < kSmallSteps; k += 32)
        out[k] = last;
    __syncwarp();
}

// Pass 1 (vol_marcher_forward.cu:351-403): a batch of the ray's entries is
// intersected lane-parallel, then walked in list order and inserted into the
// warp's section set (in shared memory, warp_put), which every lane reads.
template <PutMode kPut = PutMode::Inline, class T>
__device__ __forceinline__ void warp_collect(SectionSet<kLargeSteps, T>& sec, Section<T>* pieces, const VmMarch<T>& a, int32_t b, int32_t e, V3<T> o,
    V3<T> d, const RayList& rl, unsigned lane)
{
    if (a.cs.n > 0) {
        if (lane == 0)
            for (int i = 0; i < a.cs.n; ++i)
                sec.put(Section<T> { a.cs.s[i][0], a.cs.s[i][1], a.cs.s[i][2] });
        __syncwarp();
        return;
    }
    const uint32_t batches = ray_batches(rl, b, e);
    const T from = sec.lo; // the same for the whole step
    for (uint32_t t = 0; t < batches; ++t) {
        const int32_t entry = ray_entry(rl, b, e, t, lane);
        T depth = T(0), s0 = T(0), s1 = T(0), dt = T(0);
        bool ok = false;
        if (entry >= 0) {
            const RayEntry<T> en = load_entry(a, entry);
            const Gauss1d<T> g = intersect_with_ray_inv_C(en.mu, en.Q, o, d);
            const T sd = dgmr_fm::sqrt_f(g.C);
            depth = en.depth;
            const T mor = g.weight * en.mass;
            s0 = g.centre - sd * T(kRelevanceSigma);
            s1 = g.centre + sd * T(kRelevanceSigma);
            dt = ((sd * T(kRelevanceSigma)) * T(2)) / T(float(kStepsPerGaussian - 1));
            ok = !(mor <= T(1.0f / 255.f) || mor > T(1000)) && !(g.C <= T(0)) && !dgmr_fm::isnan_f(g.centre);
            // put() returns at once for a section outside [lo, hi): never walked
            ok = ok && !(s1 <= from);
        }
        uint32_t m = __ballot_sync(0xffffffffu, ok);
        // the walk ends before the first entry deeper than the set reaches at that
        // point (`reach`, which only insertions change), so only entries to insert are
        // walked: 1.684 -> 1.647 ms at 10k, 256^2, forward, 1.18 -> 1.155 ms in float64 at 4k,
        // 97x65, with the backward; even with walking every entry at 100k, 512^2
        T reach = sec.hi;
        uint32_t deep = __ballot_sync(0xffffffffu, entry >= 0 && reach < depth);
        bool stop = false;
        while (m) {
            const int j = __ffs(int(m)) - 1;
            m &= m - 1u;
            if (deep & lanes_below(j + 1)) {
                stop = true;
                break;
            }
            const Section<T> sj = { __shfl_sync(0xffffffffu, s0, j), __shfl_sync(0xffffffffu, s1, j), __shfl_sync(0xffffffffu, dt, j) };
            // (hi may have come in; put() leaves the set unchanged for a covered section)
            if (sj.start >= sec.hi || warp_section_covered(sec, sj, lane))
                continue;
            if (kPut == PutMode::Inline)
                warp_put(sec, pieces, sj, lane);
            else
                warp_put_call(sec, pieces, sj, lane);
            const T hi = sec.hi;
            if (hi < reach) {
                deep = __ballot_sync(0xffffffffu, entry >= 0 && hi < depth) & ~lanes_below(j + 1);
                reach = hi;
            }
        }
        if (stop || deep)
            break;
    }
}

// CDF differences of one Gaussian into the lane's bins 32 r + lane
// (math.h:461-467).  Every lane evaluates the CDF at its own borders, x[r] =
// border 32 r + lane; the right border of a bin is the next lane's left one.
// In float the four CDFs are two packed evaluations (dgmr_f32x2.cuh) instead of
// four calls; the same bits (forward 1.88 -> 1.80 ms at 10k, 256^2; 16 batched
// 64^2 views forward + backward 38.8 -> 37.4 ms).
template <class T>
__device__ __forceinline__ void lane_cdfs(T (&cs)[kRayRounds], const T (&x)[kRayRounds], T centre, T inv_sd)
{
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r)
        cs[r] = cdf_inv_SD(centre, inv_sd, x[r]);
}
template <>
__device__ __forceinline__ void lane_cdfs<float>(float (&cs)[kRayRounds], const float (&x)[kRayRounds], float centre, float inv_sd)
{
    static_assert(kRayRounds % 2 == 0, "rounds are evaluated in pairs");
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; r += 2)
        split2(cdf2_inv_SD(f2(-centre), f2(inv_sd), f2(x[r], x[r + 1])), &cs[r], &cs[r + 1]);
}

template <class T>
__device__ __forceinline__ void warp_bins(Bin<T> (&acc)[kRayRounds], const T (&x)[kRayRounds], T centre, T inv_sd, T mor, V3<T> rgb, unsigned lane)
{
    T cs[kRayRounds];
    lane_cdfs<T>(cs, x, centre, inv_sd);
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r) {
        T ce = __shfl_down_sync(0xffffffffu, cs[r], 1);
        const T next = (r + 1 < kRayRounds) ? __shfl_sync(0xffffffffu, cs[(r + 1 < kRayRounds) ? r + 1 : r], 0) : T(0);
        if (lane == 31)
            ce = next;
        const unsigned k = 32 * r + lane;
        if (k < kBins) {
            const T m = max_f(T(0), (ce - cs[r]) * mor);
            if (!(m < T(0.00001f))) {
                acc[r].r = acc[r].r + rgb.x * m;
                acc[r].g = acc[r].g + rgb.y * m;
                acc[r].b = acc[r].b + rgb.z * m;
                acc[r].m = acc[r].m + m;
            }
        }
    }
}

// cdf(b) - cdf(a); one packed evaluation in the float forward, the same bits.
// (1.725 -> 1.677 ms at 10k, 256^2; in the backward, whose registers it takes, the
// batched 64^2 views went from 23.3 to 23.7 ms.)
enum class FillPass { Forward, Backward };
template <FillPass kPass, class T>
__device__ __forceinline__ T cdf_span(T centre, T inv_sd, T b, T a)
{
    if constexpr (kPass == FillPass::Forward && sizeof(T) == 4) {
        float cb, ca;
        split2(cdf2_inv_SD(f2(-centre), f2(inv_sd), f2(b, a)), &cb, &ca);
        return cb - ca;
    } else {
        return cdf_inv_SD(centre, inv_sd, b) - cdf_inv_SD(centre, inv_sd, a);
    }
}

// The 1-D Gaussian of a usable entry if it reaches the bins (the early-outs of
// math.h:442-459); the same test in the forward and backward.
template <FillPass kPass, class T>
__device__ __forceinline__ bool warp_entry_on_bins(const RayEntry<T>& en, V3<T> o, V3<T> d, const T* borders, Gauss1d<T>* g_out, T* sd_out, T* inv_sd_out,
    T* mor_out)
{
    const Gauss1d<T> g = intersect_with_ray_inv_C(en.mu, en.Q, o, d);
    T sd, mor;
    if (!gaussian_on_ray(g, en.mass, &sd, &mor))
        return false;
    const T inv_sd = T(1) / sd;
    const T mib = mor * cdf_span<kPass>(g.centre, inv_sd, borders[kBins], borders[0]);
    if (mib < T(0.0001f))
        return false;
    *g_out = g;
    *sd_out = sd;
    *inv_sd_out = inv_sd;
    *mor_out = mor;
    return true;
}

// Pass 2 (vol_marcher_forward.cu:405-437): Gaussians in list order, bins spread
// over the lanes; returns how many Gaussians filled the bins (the same on every
// lane).  on_bins: lane t keeps which of batch t's entries these are (the first
// 32 batches), for pass 3.
template <FillPass kPass, class T>
__device__ __forceinline__ unsigned warp_fill(Bin<T> (&acc)[kRayRounds], const T* borders, const VmMarch<T>& a, int32_t b, int32_t e, V3<T> o, V3<T> d,
    const RayList& rl, unsigned lane, uint32_t* on_bins)
{
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r)
        acc[r] = Bin<T> { T(0), T(0), T(0), T(0) };
    T x[kRayRounds]; // the lane's borders
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r)
        x[r] = borders[32 * r + lane];
    unsigned fills = 0;
    const uint32_t batches = ray_batches(rl, b, e);
    for (uint32_t t = 0; t < batches; ++t) {
        const int32_t entry = ray_entry(rl, b, e, t, lane);
        T centre = T(0), inv_sd = T(0), mor = T(0);
        V3<T> rgb = { T(0), T(0), T(0) };
        bool ok = false;
        if (entry >= 0) {
            const RayEntry<T> en = load_entry(a, entry);
            Gauss1d<T> g;
            T sd;
            ok = warp_entry_on_bins<kPass>(en, o, d, borders, &g, &sd, &inv_sd, &mor);
            if (ok) {
                centre = g.centre;
                rgb = { a.rgb[3 * size_t(en.id)], a.rgb[3 * size_t(en.id) + 1], a.rgb[3 * size_t(en.id) + 2] };
            }
        }
        uint32_t okm = __ballot_sync(0xffffffffu, ok);
        fills += unsigned(__popc(okm));
        if (kPass == FillPass::Backward && lane == t)
            *on_bins = okm;
        while (okm) {
            const int j = __ffs(int(okm)) - 1;
            okm &= okm - 1u;
            const V3<T> c = { __shfl_sync(0xffffffffu, rgb.x, j), __shfl_sync(0xffffffffu, rgb.y, j), __shfl_sync(0xffffffffu, rgb.z, j) };
            warp_bins(acc, x, __shfl_sync(0xffffffffu, centre, j), __shfl_sync(0xffffffffu, inv_sd, j), __shfl_sync(0xffffffffu, mor, j), c, lane);
        }
    }
    return fills;
}

// bins to shared memory in order (.m = exp(-mass), or the mass itself for the Bins mode)
template <class T>
__device__ __forceinline__ void warp_store_bins(Bin<T>* bins, const Bin<T> (&acc)[kRayRounds], unsigned lane, bool transmittance)
{
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r) {
        const unsigned k = 32 * r + lane;
        if (k < kBins)
            bins[k] = Bin<T> { acc[r].r, acc[r].g, acc[r].b, transmittance ? dgmr_fm::exp_f(-acc[r].m) : acc[r].m };
    }
    __syncwarp();
}

template <class T, class Frames>
__global__ void __launch_bounds__(kRayWarps * 32, sizeof(T) == 4 ? 8 : 2) k_vm_march_warp(VmMarch<T> a, const __grid_constant__ Frames frames,
    const uint32_t* __restrict__ order)
{
    __shared__ RayWarpShared<T> shared_rays[kRayWarps];
    RayWarpShared<T>& sm = shared_rays[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    unsigned tile, view, px, py;
    if (!ray_pixel<T>(frames, order, &tile, &view, &px, &py))
        return; // the whole warp: no block-level barrier below
    const CameraT<T>& cam = frames.cam(view);
    const V3<T> o = { cam.campos[0], cam.campos[1], cam.campos[2] };
    const V3<T> d = pixel_dir(cam, px, py);
    const int32_t b = a.ranges[2 * tile], e = a.ranges[2 * tile + 1];
    const RayList rl = warp_ray_list(sm.use, a, b, e, o, d, lane);
    V3<T> colour = { T(0), T(0), T(0) };
    T tr = T(1);
    T start = T(0);
    T distance = T(0); // Depth mode
    SectionSet<kLargeSteps, T>& sec = sm.sec;
    unsigned long long fills = 0;
    for (unsigned step = 0;; ++step) {
        if (step >= kMaxLargeSteps) {
            if (lane == 0)
                atomicOr(&a.stats[1], DGMR_FLAG_STEP_LIMIT);
            break;
        }
        if (lane == 0)
            sec.reset(start);
        __syncwarp();
        warp_collect(sec, sm.pieces, a, b, e, o, d, rl, lane);
        warp_sample_positions(sec, sm.borders, lane);
        if (step < a.store_steps) {
            // keep this step's samples for the backward (coalesced: 32 lanes x 4 rounds)
            const size_t ray = frames.px_base(view) + size_t(py) * cam.W + px, rays = frames.rays();
            T* dst = a.store_borders + (size_t(step) * rays + ray) * kSmallSteps;
#pragma unroll
            for (unsigned r = 0; r < kRayRounds; ++r)
                dst[32 * r + lane] = sm.borders[32 * r + lane];
            if (lane == 0)
                a.store_sections[size_t(step) * rays + ray] = int32_t(sec.n);
        }
        Bin<T> acc[kRayRounds];
        fills += warp_fill<FillPass::Forward>(acc, sm.borders, a, b, e, o, d, rl, lane, nullptr);
        warp_store_bins(sm.bins, acc, lane, a.mode != DGMR_RENDER_BINS);
        if (a.mode == DGMR_RENDER_FULL) {
            // math.h:412-428, identical on every lane
            for (unsigned k = 0; k < kBins; ++k) {
                const Bin<T> bk = sm.bins[k];
                colour.x = colour.x + bk.r * tr;
                colour.y = colour.y + bk.g * tr;
                colour.z = colour.z + bk.b * tr;
                tr = tr * bk.m;
                if (tr < T(1. / 255.))
                    break;
            }
        } else if (a.mode == DGMR_RENDER_BINS) {
            // vol_marcher_forward.cu:453-465: the sum of one bin's four channels
            const Bin<T> bk = sm.bins[min(unsigned(a.debug_bin), kBins - 1)];
            const T mass = ((bk.r + bk.g) + bk.b) + bk.m;
            colour = { mass * a.max_depth, mass * a.max_depth, mass * a.max_depth };
            if (mass == T(0))
                colour = { T(0), T(1), T(0) };
            if (dgmr_fm::isnan_f(mass))
                colour = { T(1), T(0), T(0.5) };
            if (mass < T(0))
                colour = { T(1), T(0), T(0) };
            tr = T(0);
        } else {
            // vol_marcher_forward.cu:466-481: the distance marched so far
            for (unsigned k = 0; k < kBins; ++k)
                tr = tr * sm.bins[k].m;
            distance = max_f(sec.hi, distance);
            const T dd = distance / a.max_depth;
            colour = { dd, dd, dd };
        }
        const bool done = sec.n == 0 || tr < T(1.f / 255.f);
        start = sm.borders[kSmallSteps - 1];
        __syncwarp();
        if (done)
            break;
    }
    if (lane == 0) {
        if (a.work)
            atomicAdd(a.work, fills);
        const size_t pix = size_t(py) * cam.W + px;
        const size_t plane = size_t(cam.W) * cam.H;
        T* fb = frames.fb(view, a);
        fb[pix] = colour.x + tr * cam.bg[0];
        fb[plane + pix] = colour.y + tr * cam.bg[1];
        fb[2 * plane + pix] = colour.z + tr * cam.bg[2];
        frames.remaining_T(view, a)[pix] = tr;
    }
}

} // namespace dgmr

namespace dgmr {

// Adjoint of one Gaussian's bin masses (grad/math.h:559-620), run by one lane
// over the bins in shared memory -- in bin order, so its sums round exactly
// as the one-thread loop does -- then added to the per-Gaussian accumulators.
// Inlined at its one call: out of line it cost 5 % (31.0 ms instead of 29.1, forward +
// backward at 100k, 512^2; 24.7 instead of 23.3 for 16 batched 64^2 views).
template <class T>
__device__ __forceinline__ void lane_grad_entry(const VmMarch<T>& a, int32_t k, const Bin<T>* gbins, const T* borders, V3<T> o, V3<T> d, int live_end)
{
    const RayEntry<T> en = load_entry(a, k);
    const V3<T> rgb = { a.rgb[3 * size_t(en.id)], a.rgb[3 * size_t(en.id) + 1], a.rgb[3 * size_t(en.id) + 2] };
    T g_mass = T(0);
    V3<T> grgb = { T(0), T(0), T(0) }, gmu = { T(0), T(0), T(0) };
    S3<T> gQ = { { T(0), T(0), T(0), T(0), T(0), T(0) } };
    grad_sample_gaussian(en.mu, en.Q, o, d, en.mass, rgb, borders, gbins, &g_mass, &grgb, &gmu, &gQ, live_end);
    // summed in double: a Gaussian's 13 totals collect terms from every ray and
    // large step that reaches it, in no fixed order, and many cancel; float
    // sums of that kind drift by far more than the gradients' 1e-3 tolerance
    double* dst = a.acc + size_t(en.id) * kVmAcc;
    const T v[kVmAcc] = { g_mass, grgb.x, grgb.y, grgb.z, gQ.v[0], gQ.v[1], gQ.v[2], gQ.v[3], gQ.v[4], gQ.v[5], gmu.x, gmu.y, gmu.z };
#pragma unroll
    for (int q = 0; q < int(kVmAcc); ++q)
        if (v[q] != T(0))
            atomicAdd(dst + q, double(v[q]));
}

// Pass 3: the ray's Gaussians that reach the bins are gathered, in list
// order, into a queue and run 32 at a time, one per lane, so the lanes stay busy
// however sparse the ray's entries are in the tile list.  (Each Gaussian's
// adjoint is independent of the others'; only the atomic additions of
// different pixels meet, in no fixed order, as in the one-thread kernel.)
// on_bins: lane t holds which of batch t's entries pass 2 found on the bins;
// batches past the 32nd are tested again.  Testing every
// batch again cost 1.5 ms of 33.1, forward + backward at 100k, 512^2, and 1.0 of
// 26.1 for 16 batched 64^2 views.
// live_end: the bins from there on have zero adjoints (the ray stopped before
// them), so a Gaussian whose live bins all lie there adds nothing.
template <class T>
__device__ __forceinline__ void warp_grad(const Bin<T>* gbins, const T* borders, int32_t* queue, const VmMarch<T>& a, int32_t b, int32_t e, V3<T> o, V3<T> d,
    const RayList& rl, uint32_t on_bins, unsigned lane, int live_end)
{
    unsigned fill = 0;
    const uint32_t batches = ray_batches(rl, b, e);
    for (uint32_t t = 0; t <= batches; ++t) {
        if (t < batches) {
            uint32_t okm = t < 32 ? __shfl_sync(0xffffffffu, on_bins, int(t)) : 0u;
            const int32_t entry = ray_entry(rl, b, e, t, lane);
            if (t >= 32) {
                bool ok = false;
                if (entry >= 0) {
                    Gauss1d<T> g;
                    T sd, inv_sd, mor;
                    ok = warp_entry_on_bins<FillPass::Backward>(load_entry(a, entry), o, d, borders, &g, &sd, &inv_sd, &mor);
                }
                okm = __ballot_sync(0xffffffffu, ok);
            }
            if ((okm >> lane) & 1u)
                queue[fill + unsigned(__popc(okm & lanes_below(int(lane))))] = entry;
            fill += unsigned(__popc(okm));
            __syncwarp();
        }
        if (fill >= 32 || (t == batches && fill > 0)) {
            if (lane < fill)
                lane_grad_entry(a, queue[lane], gbins, borders, o, d, live_end);
            __syncwarp();
            // the entries that did not fit go to the front of the emptied queue
            if (lane + 32 < fill)
                queue[lane] = queue[lane + 32];
            __syncwarp();
            fill = fill > 32 ? fill - 32 : 0;
        }
    }
}

// The colour peel of one large step and the bin adjoints (grad/math.h:529-557),
// from the lane's bins 32 r + lane; returns one past the bin where the ray
// stopped.  exp(-mass) and its reciprocal are computed by the bin's own lane,
// and so are the adjoints, from the colour and transmittance that the lane
// takes out of the walk at its bin.  Only the walk itself (the two products and
// the subtraction that chain the bins) runs on every lane, and only over the
// bins that hold any mass: an empty bin changes neither the colour nor the
// transmittance, and its adjoint is never read (no Gaussian reached it with
// the mass that pass 3 asks for).  The same operations, in the same order.
// Against the walk over every bin with the exp and the division on every lane:
// forward + backward 45.1 -> 41.3 ms at 100k, 512^2 (mean of four cameras), 1.86
// -> 1.63 ms in float64 at 4k, 97x65.
template <class T>
__device__ __forceinline__ int warp_peel(Bin<T>* gbins, Bin<T>* bins, T* inv_t, const Bin<T> (&acc)[kRayRounds], V3<T> gc, T gt, T final_T, V3<T>& colour,
    T& tr, unsigned lane)
{
    T tks[kRayRounds], invs[kRayRounds];
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r) {
        tks[r] = dgmr_fm::exp_f(-acc[r].m);
        invs[r] = min_f(T(255), T(1) / tks[r]);
        bins[32 * r + lane] = Bin<T> { acc[r].r, acc[r].g, acc[r].b, tks[r] };
        inv_t[32 * r + lane] = invs[r];
    }
    __syncwarp();
    int live_end = int(kBins);
#pragma unroll
    for (unsigned r = 0; r < kRayRounds; ++r) {
        Bin<T> gb = { T(0), T(0), T(0), T(0) };
        uint32_t held = __ballot_sync(0xffffffffu, acc[r].m != T(0));
        if (live_end == int(kBins) && held) {
            T my_tr = T(0);
            V3<T> my_colour = { T(0), T(0), T(0) };
            while (held) {
                const int j = __ffs(int(held)) - 1;
                held &= held - 1u;
                const Bin<T> bk = bins[32 * r + j];
                const T inv_tk = inv_t[32 * r + j];
                colour.x = (colour.x - bk.r) * inv_tk;
                colour.y = (colour.y - bk.g) * inv_tk;
                colour.z = (colour.z - bk.b) * inv_tk;
                if (int(lane) == j) {
                    my_tr = tr;
                    my_colour = colour;
                }
                tr = tr * bk.m;
                if (tr < T(1. / 255.)) {
                    live_end = int(32 * r) + j + 1;
                    break;
                }
            }
            if (my_tr != T(0)) {
                gb.r = my_tr * gc.x;
                gb.g = my_tr * gc.y;
                gb.b = my_tr * gc.z;
                const T g_tk = (final_T * invs[r]) * gt + dot3(gc, my_colour) * my_tr;
                gb.m = T(0) - g_tk * tks[r];
            }
        }
        gbins[32 * r + lane] = gb;
    }
    __syncwarp();
    return live_end;
}

// vol_marcher_backward.cu:115-319 with one warp per ray
template <class T, class Frames>
__global__ void __launch_bounds__(kRayWarps * 32, sizeof(T) == 4 ? 6 : 2) k_vm_march_warp_bwd(VmMarch<T> a, const __grid_constant__ Frames frames,
    const uint32_t* __restrict__ order)
{
    __shared__ RayWarpSharedBwd<T> shared_rays[kRayWarps];
    RayWarpSharedBwd<T>& sm = shared_rays[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    unsigned tile, view, px, py;
    if (!ray_pixel<T>(frames, order, &tile, &view, &px, &py))
        return;
    const T* grad_fb = frames.grad_fb(view, a);
    if (!grad_fb) // a view of a batch without an image gradient
        return;
    const CameraT<T>& cam = frames.cam(view);
    const V3<T> o = { cam.campos[0], cam.campos[1], cam.campos[2] };
    const V3<T> d = pixel_dir(cam, px, py);
    const int32_t b = a.ranges[2 * tile], e = a.ranges[2 * tile + 1];
    const RayList rl = warp_ray_list(sm.use, a, b, e, o, d, lane);
    const size_t pix = size_t(py) * cam.W + px;
    const size_t plane = size_t(cam.W) * cam.H;
    const T* fb = frames.fb(view, a);
    const T final_T = frames.remaining_T(view, a)[pix];
    V3<T> colour = { fb[pix] - final_T * cam.bg[0], fb[plane + pix] - final_T * cam.bg[1], fb[2 * plane + pix] - final_T * cam.bg[2] };
    const V3<T> gc = { grad_fb[pix], grad_fb[plane + pix], grad_fb[2 * plane + pix] };
    const T gt = (gc.x * cam.bg[0] + gc.y * cam.bg[1]) + gc.z * cam.bg[2];
    T tr = T(1);
    T start = T(0);
    SectionSet<kLargeSteps, T>& sec = sm.sec;
    for (unsigned step = 0;; ++step) {
        if (step >= kMaxLargeSteps) {
            if (lane == 0)
                atomicOr(&a.stats[1], DGMR_FLAG_STEP_LIMIT);
            break;
        }
        int n_sections;
        if (step < a.store_steps) {
            // the forward kept this step's samples: no section set, no sampling
            const size_t ray = frames.px_base(view) + size_t(py) * cam.W + px, rays = frames.rays();
            const T* src = a.store_borders + (size_t(step) * rays + ray) * kSmallSteps;
#pragma unroll
            for (unsigned r = 0; r < kRayRounds; ++r)
                sm.borders[32 * r + lane] = src[32 * r + lane];
            n_sections = a.store_sections[size_t(step) * rays + ray];
            __syncwarp();
        } else {
            if (lane == 0)
                sec.reset(start);
            __syncwarp();
            warp_collect<PutMode::Call>(sec, sm.pieces, a, b, e, o, d, rl, lane);
            warp_sample_positions(sec, sm.borders, lane);
            n_sections = int(sec.n);
        }
        Bin<T> acc[kRayRounds];
        uint32_t on_bins = 0;
        warp_fill<FillPass::Backward>(acc, sm.borders, a, b, e, o, d, rl, lane, &on_bins);
        const int live_end = warp_peel(sm.gbins, sm.bins, sm.inv_t, acc, gc, gt, final_T, colour, tr, lane);
        warp_grad(sm.gbins, sm.borders, sm.queue, a, b, e, o, d, rl, on_bins, lane, live_end);
        const bool done = n_sections == 0 || tr < T(1.f / 255.f);
        start = sm.borders[kSmallSteps - 1];
        __syncwarp();
        if (done)
            break;
    }
}

} // namespace dgmr
