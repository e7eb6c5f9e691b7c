// Volume rasteriser with one warp per ray (included by dgmr_raster.cu).
//
// A ray has 32 depth bins and a warp has 32 lanes: lane q owns bin q.
//  * Pass A: the bin sizer's 32 slots live one per lane (mass, border, sd).
//    The tile list is walked 32 entries at a time (ray intersection, gates
//    and the added mass computed lane-parallel), then the qualifying entries
//    are added in list order: the insertion position is one ballot (the
//    first slot from the right whose border is not greater), the shift one
//    shuffle; once every slot holds mass, lane j prices merging slots j and
//    j+1 and a warp minimum picks the cheapest (the first of equals).
//    The transmittance in front of each slot is the same left-to-right
//    product as the one-thread sizer's, so every merge decision matches it.
//  * Pass B: the tile's Gaussians that reach the bins are packed into shared
//    memory, what depends on the Gaussian alone (its CDF at 0, its value at the
//    far end) computed by the lane that loaded it; then, two Gaussians at a time
//    as the halves of packed floats, lane q evaluates the CDF at its bin's right
//    border (the left one is its neighbour's) and accumulates its bin's four
//    masses and border values in registers -- per bin the same Gaussian order and
//    operations as the one-thread loop.
//  * Blend: lane q fits its bin and integrates its 256 steps from T = 1; the
//    bins' colours and transmittances are then chained in bin order.
// The one-thread-per-pixel kernel this replaces kept ~1 KB of bins and the
// sizer per thread (local memory) and ran 32 x 256 integration steps on one
// lane.  Warps are independent (no block barrier); rays outside the frame
// leave at once.
#pragma once

#include "dgmr_f32x2.cuh"

namespace dgmr {

constexpr unsigned kVrRayWarps = 4; // rays per block

// eval_exponential_1d of two Gaussians at one position; nc = -centre
__device__ __forceinline__ F2 eval2_exponential_1d(F2 nc, float var0, float var1, float x)
{
    const F2 dx = add2(f2(x), nc);
    float a0, a1;
    split2(mul2(f2(-0.5f), mul2(dx, dx)), &a0, &a1);
    const float x0 = a0 / var0, x1 = a1 / var1;
    float e0, e1;
    split2(exp2_nonpos(f2(x0, x1)), &e0, &e1);
    // past the packed exp's range: zero, or (NaN, the subnormal results) the scalar one
    if (!(x0 >= -87.f && x0 <= 0.f))
        e0 = x0 < -104.f ? 0.f : dgmr_fm::exp_f(x0);
    if (!(x1 >= -87.f && x1 <= 0.f))
        e1 = x1 < -104.f ? 0.f : dgmr_fm::exp_f(x1);
    return f2(e0, e1);
}

// A Gaussian of pass B as every lane reads it.
struct alignas(16) VrStaged {
    float centre, inv_sd, var, weight;
    float cdf0, last; // CDF at 0; weight times the value at the far end
    float r, g;
    float b, one, pad0, pad1;
};

struct RayEntryVr {
    uint32_t id;
    V3<float> mu;
    S3<float> Q;
    float mass;
};

// the sizer's slot held by this lane, and the ray-wide totals; front: the
// transmittance in front of the slot, up to date for slots 0 to front_ok
struct WarpBinSizer {
    float mass, border, sd, front;
    float total, far, full_mass, sigma;
    unsigned front_ok;
};

__device__ __forceinline__ void wbs_init(WarpBinSizer& s, float sigma, float transmission_threshold)
{
    s.mass = 0.f;
    s.border = 1.f / 0.f;
    s.sd = 0.f;
    s.front = 1.f;
    s.front_ok = 0u;
    s.total = 0.f;
    s.far = 0.f;
    s.sigma = sigma;
    s.full_mass = -dgmr_fm::log_f(transmission_threshold);
}

__device__ __forceinline__ float wbs_kl(float c1, float sd1, float c2, float sd2)
{
    return ((c1 - c2) * (c1 - c2) + sd1 * sd1 - sd2 * sd2) / (2.f * sd2 * sd2) + dgmr_fm::log_f(sd2 / sd1);
}

// RasterBinSizer::add_gaussian with the slots spread over the lanes; the
// arguments are the same on every lane (on_ray and reach precomputed by the
// entry's lane with RasterBinSizer's own cdf)
__device__ __forceinline__ void wbs_add(WarpBinSizer& s, unsigned lane, float mass, float centre, float sd, float on_ray, float reach)
{
    constexpr unsigned kFull = 0xffffffffu;
    if (mass < 0.0001f)
        return;
    s.far = max_f(reach, s.far);
    s.total = s.total + on_ray;
    // the new lobe enters the spare last slot and moves left past every border
    // strictly greater than its centre: it stops after the first slot (from
    // the right) that is not greater
    const unsigned not_greater = __ballot_sync(kFull, lane < kVrBins - 1 && !(s.border > centre));
    const unsigned p = not_greater ? 32u - unsigned(__clz(int(not_greater))) : 0u;
    const float um = __shfl_up_sync(kFull, s.mass, 1), ub = __shfl_up_sync(kFull, s.border, 1), us = __shfl_up_sync(kFull, s.sd, 1);
    if (lane > p) {
        s.mass = um;
        s.border = ub;
        s.sd = us;
    } else if (lane == p) {
        s.mass = on_ray;
        s.border = centre;
        s.sd = sd;
    }
    s.front_ok = min(s.front_ok, p);
    if (!(__shfl_sync(kFull, s.mass, kVrBins - 1) > 0.f))
        return;
    // transmittance in front of each slot: the one-thread sizer's left-to-right
    // product, continued from the last slot that it holds for
    const float ex = dgmr_fm::exp_f(-s.mass);
    float run = __shfl_sync(kFull, s.front, int(s.front_ok));
#pragma unroll 1
    for (unsigned i = s.front_ok; i + 1 < kVrBins; ++i) {
        run = run * __shfl_sync(kFull, ex, int(i));
        if (lane == i + 1)
            s.front = run;
    }
    s.front_ok = kVrBins - 1;
    const float front = s.front;
    // lane j < 31: the merge of slots j and j + 1 and its cost
    const float nm = __shfl_down_sync(kFull, s.mass, 1), nb = __shfl_down_sync(kFull, s.border, 1), nsd = __shfl_down_sync(kFull, s.sd, 1);
    const float nfront = __shfl_down_sync(kFull, front, 1);
    const float sa = front * s.mass, sb = nfront * nm;
    const float pa = (sa + sb >= 0.0000001f) ? min_f(sa / (sa + sb), 0.999999f) : 0.5f;
    const float pb = 1.f - pa;
    const float c = pa * s.border + pb * nb;
    const float va = s.sd * s.sd, vb = nsd * nsd;
    const float v = pa * (va + (s.border - c) * (s.border - c)) + pb * (vb + (nb - c) * (nb - c));
    const float m_mass = s.mass + nm, m_sd = dgmr_fm::sqrt_f(v);
    const float cost = nfront * (wbs_kl(s.border, s.sd, c, m_sd) + wbs_kl(nb, nsd, c, m_sd));
    // the one-thread loop keeps the first index of the smallest cost below +inf
    const float key = (lane < kVrBins - 1 && cost < 1.f / 0.f) ? cost : 1.f / 0.f;
    float lo = key;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
        lo = fminf(lo, __shfl_xor_sync(kFull, lo, o));
    if (!(lo < 1.f / 0.f))
        return;
    const unsigned pick = unsigned(__ffs(int(__ballot_sync(kFull, key == lo))) - 1);
    s.front_ok = pick;
    // the merged lobe takes slot pick, the slots behind it move one left, the last stays
    if (lane == pick) {
        s.mass = m_mass;
        s.border = c;
        s.sd = m_sd;
    } else if (lane > pick && lane + 1 < kVrBins) {
        s.mass = nm;
        s.border = nb;
        s.sd = nsd;
    }
}

// RasterBinSizer::finalise: monotone borders, empty slots spread to the far end
__device__ __forceinline__ void wbs_finalise(WarpBinSizer& s, unsigned lane)
{
    float prev = 0.f;
#pragma unroll 1
    for (unsigned i = 0; i < kVrBins; ++i) {
        float b = __shfl_sync(0xffffffffu, s.border, int(i));
        const bool empty = b == 1.f / 0.f;
        if (!empty)
            b = max_f(b, prev + 0.00001f);
        else
            b = prev + (s.far - prev) / float(kVrBins - i);
        prev = b;
        if (lane == i) {
            s.border = b;
            if (empty)
                s.mass = 0.f;
        }
    }
}

__device__ __forceinline__ RayEntryVr load_vr_entry(const VrRender& a, int32_t k)
{
    RayEntryVr en;
    uint32_t id = a.list[k];
    if (id >= a.N) {
        flag_bounds(a.stats, 0x41u);
        id = 0;
    }
    en.id = id;
    en.mu = { a.centroids[3 * size_t(id)], a.centroids[3 * size_t(id) + 1], a.centroids[3 * size_t(id) + 2] };
#pragma unroll
    for (int c = 0; c < 6; ++c)
        en.Q.v[c] = a.inv_cov[6 * size_t(id) + c];
    en.mass = a.masses[id];
    return en;
}

// vol_raster_forward.cu:253-517, one warp per ray.  Bound by instruction issue
// (30,000 warp instructions per ray at 100k, 512^2, a third of them the 256
// integration steps).  Against a Gaussian at a time in pass B (its CDF at 0 and
// its far value evaluated by one lane while 31 waited), a scalar integration and
// the whole product of transmittances per added Gaussian: 10.40 -> 8.48 ms, mean
// of four cameras; 56 registers and nine blocks per SM instead of 70: 8.29.
__global__ void __launch_bounds__(kVrRayWarps * 32, 9) k_vr_render_warp(VrRender a, CameraT<float> cam)
{
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ VrStaged staged[kVrRayWarps][32];
    const unsigned lane = threadIdx.x & 31u;
    const unsigned per_tile = kTilePixels / kVrRayWarps;
    const unsigned tile = blockIdx.x / per_tile;
    const unsigned pix_in_tile = (blockIdx.x % per_tile) * kVrRayWarps + (threadIdx.x >> 5);
    const unsigned tx = tile % cam.gx, ty = tile / cam.gx;
    const unsigned px = tx * kTile + (pix_in_tile % kTile), py = ty * kTile + (pix_in_tile / kTile);
    if (px >= cam.W || py >= cam.H)
        return; // the whole warp
    const V3<float> o = { cam.campos[0], cam.campos[1], cam.campos[2] };
    const V3<float> d = vr_pixel_dir(cam, px, py);
    int32_t b = a.ranges[2 * tile], e = a.ranges[2 * tile + 1];
    if (b < 0 || e < b || uint32_t(e) > a.cap) {
        if (lane == 0)
            flag_bounds(a.stats, 0x42u);
        b = e = 0;
    }
    // pass A: bin sizes, until the ray's mass is used up
    WarpBinSizer sz;
    wbs_init(sz, kVrRelevanceSigma, kVrTransmission);
    bool full = false;
    for (int32_t base = b; base < e && !full; base += 32) {
        float mor = 0.f, centre = 0.f, sd = 0.f, on_ray = 0.f, reach = 0.f;
        bool ok = false;
        if (base + int32_t(lane) < e) {
            const RayEntryVr en = load_vr_entry(a, base + int32_t(lane));
            const Gauss1d<float> g = intersect_with_ray_inv_C(en.mu, en.Q, o, d);
            mor = g.weight * en.mass;
            ok = !(mor < 0.001f || mor > 1000.f) && !(g.C + 0.f <= 0.f);
            if (ok) {
                centre = g.centre;
                sd = dgmr_fm::sqrt_f(g.C + 0.f);
                reach = centre + sd * kVrRelevanceSigma;
                // RasterBinSizer::cdf at both ends
                const float scale = sd * 1.41421356237309505f;
                float at_reach, at_zero;
                split2(mul2(f2(0.5f), add2(f2(1.f), erf2(f2((reach - centre) / scale, (0.f - centre) / scale)))), &at_reach, &at_zero);
                on_ray = mor * (at_reach - at_zero);
            }
        }
        uint32_t m = __ballot_sync(kFull, ok);
        while (m) {
            const int j = __ffs(int(m)) - 1;
            m &= m - 1u;
            wbs_add(sz, lane, __shfl_sync(kFull, mor, j), __shfl_sync(kFull, centre, j), __shfl_sync(kFull, sd, j), __shfl_sync(kFull, on_ray, j),
                __shfl_sync(kFull, reach, j));
            if (sz.total >= sz.full_mass) {
                full = true;
                break;
            }
        }
    }
    wbs_finalise(sz, lane);
    // this lane's bin: [begin, end)
    const float end = lane == kVrBins - 1 ? sz.far : sz.border;
    const float begin_up = __shfl_up_sync(kFull, end, 1);
    const float begin = lane == 0 ? 0.f : begin_up;
    float res0 = 0.f, res1 = 0.f, res2 = 0.f, transparency = 1.f; // the final colour adds T = 1 x background in Full and Bins mode
    if (a.mode == DGMR_RENDER_FULL) {
        // pass B: bin masses and border values of every Gaussian of the tile
        VrStaged* row = staged[threadIdx.x >> 5];
        F2 bm_rg = f2(0.f), bm_bm = f2(0.f), be_rg = f2(0.f), be_bm = f2(0.f), last_rg = f2(0.f), last_bm = f2(0.f); // (r, g), (b, mass)
        const float max_distance = sz.far;
        const F2 ends = f2(end);
        for (int32_t base = b; base < e; base += 32) {
            VrStaged st;
            bool ok = false;
            if (base + int32_t(lane) < e) {
                const RayEntryVr en = load_vr_entry(a, base + int32_t(lane));
                const Gauss1d<float> g = intersect_with_ray_inv_C(en.mu, en.Q, o, d);
                st.centre = g.centre;
                st.var = g.C + 0.f;
                const float sd = dgmr_fm::sqrt_f(st.var);
                st.inv_sd = 1.f / sd;
                st.weight = g.weight * en.mass;
                ok = !(st.var <= 0.f || dgmr_fm::isnan_f(st.var) || dgmr_fm::isnan_f(st.weight) || st.weight > 100000.f);
                if (ok) {
                    float far;
                    split2(cdf2_inv_SD(f2(-st.centre), f2(st.inv_sd), f2(max_distance, 0.f)), &far, &st.cdf0);
                    ok = !(st.weight * (far - st.cdf0) <= 0.001f);
                }
                if (ok) {
                    st.last = st.weight * eval_exponential_1d(st.centre, st.var, max_distance);
                    st.r = a.rgb[3 * size_t(en.id)];
                    st.g = a.rgb[3 * size_t(en.id) + 1];
                    st.b = a.rgb[3 * size_t(en.id) + 2];
                    st.one = 1.f;
                }
            }
            const uint32_t m = __ballot_sync(kFull, ok);
            if (!m)
                continue;
            const int n = __popc(m);
            __syncwarp(); // the last batch is read
            if (ok)
                row[__popc(m & ((1u << lane) - 1u))] = st;
            if ((n & 1) && lane == 0) // an odd one's partner: no weight, no mass
                row[n] = VrStaged { 0.f, 1.f, 1.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f };
            __syncwarp();
            for (int j = 0; j < n; j += 2) {
                const VrStaged &g0 = row[j], &g1 = row[j + 1];
                const F2 nc = f2(-g0.centre, -g1.centre);
                const F2 cdf_end = cdf2_inv_SD(nc, f2(g0.inv_sd, g1.inv_sd), ends);
                float end0, end1;
                split2(cdf_end, &end0, &end1);
                const float left0 = __shfl_up_sync(kFull, end0, 1), left1 = __shfl_up_sync(kFull, end1, 1);
                const float mass0 = (end0 - (lane == 0 ? g0.cdf0 : left0)) * g0.weight, mass1 = (end1 - (lane == 0 ? g1.cdf0 : left1)) * g1.weight;
                const bool has0 = !(mass0 < 0.0001f), has1 = !(mass1 < 0.0001f);
                const F2 rg0 = f2(g0.r, g0.g), rg1 = f2(g1.r, g1.g), bm0 = f2(g0.b, g0.one), bm1 = f2(g1.b, g1.one);
                if (has0 || has1) {
                    float ev0, ev1;
                    split2(mul2(f2(g0.weight, g1.weight), eval2_exponential_1d(nc, g0.var, g1.var, begin)), &ev0, &ev1);
                    if (has0) {
                        bm_rg = add2(bm_rg, mul2_rounded(rg0, f2(mass0)));
                        bm_bm = add2(bm_bm, mul2_rounded(bm0, f2(mass0)));
                        be_rg = add2(be_rg, mul2_rounded(rg0, f2(ev0)));
                        be_bm = add2(be_bm, mul2_rounded(bm0, f2(ev0)));
                    }
                    if (has1) {
                        bm_rg = add2(bm_rg, mul2_rounded(rg1, f2(mass1)));
                        bm_bm = add2(bm_bm, mul2_rounded(bm1, f2(mass1)));
                        be_rg = add2(be_rg, mul2_rounded(rg1, f2(ev1)));
                        be_bm = add2(be_bm, mul2_rounded(bm1, f2(ev1)));
                    }
                }
                // the values at the far end (read by the last bin's lane)
                last_rg = add2(last_rg, mul2_rounded(rg0, f2(g0.last)));
                last_bm = add2(last_bm, mul2_rounded(bm0, f2(g0.last)));
                last_rg = add2(last_rg, mul2_rounded(rg1, f2(g1.last)));
                last_bm = add2(last_bm, mul2_rounded(bm1, f2(g1.last)));
            }
        }
        float bm[4], be[4], be_last[4];
        split2(bm_rg, &bm[0], &bm[1]);
        split2(bm_bm, &bm[2], &bm[3]);
        split2(be_rg, &be[0], &be[1]);
        split2(be_bm, &be[2], &be[3]);
        split2(last_rg, &be_last[0], &be_last[1]);
        split2(last_bm, &be_last[2], &be_last[3]);
        // blend: lane q fits bin q (the split of a bin's mass between its halves is
        // 0.5 for every bin and channel, vol_raster_forward.cu:473) and integrates
        // it from T = 1; then the bins are chained in order
        float right[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float nxt = __shfl_down_sync(kFull, be[c], 1);
            right[c] = lane == kVrBins - 1 ? be_last[c] : nxt;
        }
        const float t_right = end - begin;
        float l0 = 0.f, l1 = 0.f, l2 = 0.f, cur = 1.f;
        if (t_right > 0.f) {
            const float half[4] = { 0.5f, 0.5f, 0.5f, 0.5f };
            const FunctionGroup<float> f = create_approximation(half, bm, be, right, t_right);
            const float dt = f.t_right / float(kVrStepsPerBin);
            float t = dt / 2.f;
            // FunctionGroup::sample of channels (r, g) and (b, mass) as packed halves
            const F2 d01 = f2(f.d0[0], f.d0[1]), d23 = f2(f.d0[2], f.d0[3]), k01 = f2(f.k0[0], f.k0[1]), k23 = f2(f.k0[2], f.k0[3]);
            const F2 b01 = add2(d01, mul2_rounded(f2(f.t1[0], f.t1[1]), k01)), b23 = add2(d23, mul2_rounded(f2(f.t1[2], f.t1[3]), k23));
            const F2 n01 = f2(-f.t2[0], -f.t2[1]), n23 = f2(-f.t2[2], -f.t2[3]), r01 = f2(f.k2[0], f.k2[1]), r23 = f2(f.k2[2], f.k2[3]);
            F2 l01 = f2(0.f);
            for (unsigned s = 0; s < kVrStepsPerBin; ++s) {
                const F2 tt = f2(t);
                float lo[4], hi[4], ev[4];
                split2(add2(d01, mul2_rounded(k01, tt)), &lo[0], &lo[1]);
                split2(add2(d23, mul2_rounded(k23, tt)), &lo[2], &lo[3]);
                split2(add2(b01, mul2_rounded(add2(tt, n01), r01)), &hi[0], &hi[1]);
                split2(add2(b23, mul2_rounded(add2(tt, n23), r23)), &hi[2], &hi[3]);
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    ev[c] = t <= f.t1[c] ? lo[c] : t <= f.t2[c] ? 0.f : hi[c];
                l01 = add2(l01, mul2_rounded(mul2(f2(ev[0], ev[1]), f2(cur)), f2(dt)));
                l2 = l2 + (ev[2] * cur) * dt;
                cur = cur * max_f(0.f, 1.f - ev[3] * dt);
                t = t + dt;
            }
            split2(l01, &l0, &l1);
        }
        float tr = 1.f;
#pragma unroll 1
        for (unsigned q = 0; q < kVrBins; ++q) {
            res0 = res0 + tr * __shfl_sync(kFull, l0, int(q));
            res1 = res1 + tr * __shfl_sync(kFull, l1, int(q));
            res2 = res2 + tr * __shfl_sync(kFull, l2, int(q));
            tr = tr * __shfl_sync(kFull, cur, int(q));
        }
    } else if (a.mode == DGMR_RENDER_DEPTH) {
        // vol_raster_forward.cu:495-507
        const unsigned bin = min(unsigned(a.debug_bin), kVrBins - 1);
        const float distance = __shfl_sync(kFull, end, int(bin));
        float c0 = distance / a.max_depth, c1 = c0, c2 = c0;
        if (distance == 0.f) {
            c0 = 0.f;
            c1 = 1.f;
            c2 = 0.f;
        }
        if (dgmr_fm::isnan_f(distance)) {
            c0 = 1.f;
            c1 = 0.f;
            c2 = 0.5f;
        }
        if (distance < 0.f) {
            c0 = 1.f;
            c1 = 0.5f;
            c2 = 0.f;
        }
        res0 = c0;
        res1 = c1;
        res2 = c2;
        transparency = 0.f;
    }
    if (lane == 0) {
        const size_t pix = size_t(py) * cam.W + px;
        const size_t plane = size_t(cam.W) * cam.H;
        a.fb[pix] = res0 + transparency * cam.bg[0];
        a.fb[plane + pix] = res1 + transparency * cam.bg[1];
        a.fb[2 * plane + pix] = res2 + transparency * cam.bg[2];
    }
}

} // namespace dgmr
