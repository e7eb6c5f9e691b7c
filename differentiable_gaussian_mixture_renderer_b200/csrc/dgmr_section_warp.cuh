// Section insertion by a whole warp: SectionSet (dgmr_sections.h) in shared memory,
// lane i holding section i.  All functions are for full warps.
#pragma once

#include "dgmr_marching.cuh"

namespace dgmr {

static_assert(kLargeSteps <= 16, "warp_put keeps a section per lane on lanes 0-15 and writes others from lanes 16-31");

__device__ __forceinline__ uint32_t lanes_below(int n) { return n >= 32 ? 0xffffffffu : ((1u << n) - 1u); }

// SectionSet::put_leaves_unchanged (dgmr_sections.h) with lane i (< kLargeSteps)
// testing section i: whether inserting s would leave the warp's set exactly as
// it is, so that the insertion (and lane 0's serial walk) can be skipped.
template <class T>
__device__ __forceinline__ bool warp_section_covered(const SectionSet<kLargeSteps, T>& sec, const Section<T>& s, unsigned lane)
{
    const T cs = max_f(sec.lo, s.start), ce = min_f(sec.hi, s.end);
    const unsigned n = sec.n;
    if (n == kLargeSteps && sec.e[kLargeSteps - 1].end < sec.hi)
        return false;
    Section<T> my = { T(0), T(0), T(0) };
    if (lane < n)
        my = sec.e[lane];
    const bool ov = lane < n && my.end > cs && my.start < ce;
    const uint32_t ovm = __ballot_sync(0xffffffffu, ov);
    const T next_start = __shfl_down_sync(0xffffffffu, my.start, 1);
    const T next_dt = __shfl_down_sync(0xffffffffu, my.delta_t, 1);
    if (!ovm)
        return false;
    const unsigned f = unsigned(__ffs(int(ovm)) - 1), l = 31u - unsigned(__clz(int(ovm)));
    bool bad = ov && my.delta_t > s.delta_t;
    if (ov && lane < l && (my.end != next_start || (my.delta_t == s.delta_t && next_dt == s.delta_t)))
        bad = true; // a gap, or two neighbours that the insertion would merge
    if (lane == f && my.start > cs)
        bad = true;
    if (lane == l && my.end < ce)
        bad = true;
    return __ballot_sync(0xffffffffu, bad) == 0u;
}

// The insertion of warp_put where an overlapped section or s is empty or has a NaN
// step: lane 0 merges the run (SectionSet::merge_pieces, into the warp's
// scratch), then the kept tail is moved (lanes 0-15) and the pieces written (lanes
// 16-31) in one step -- put()'s set, bit for bit (put_by_pieces, the serial form
// of this split, is tested against put() on random insertion sequences).
template <class T>
__device__ __noinline__ void warp_put_pieces(SectionSet<kLargeSteps, T>& sec, Section<T>* pieces, Section<T> s, unsigned first, unsigned last, unsigned lane)
{
    const unsigned n = sec.n;
    Section<T> my = { T(0), T(0), T(0) };
    if (lane < n)
        my = sec.e[lane];
    unsigned np = 0, end = last;
    if (lane == 0)
        np = sec.merge_pieces(s, first, last, pieces, &end);
    np = __shfl_sync(0xffffffffu, np, 0);
    end = __shfl_sync(0xffffffffu, end, 0);
    __syncwarp();
    const unsigned k = lane - 16u;
    const bool move = lane >= end && lane < n && first + np + (lane - end) < kLargeSteps;
    const bool write = lane >= 16u && k < np && first + k < kLargeSteps;
    Section<T> pv = { T(0), T(0), T(0) };
    if (write)
        pv = pieces[k];
    __syncwarp();
    if (move)
        sec.e[first + np + (lane - end)] = my;
    if (write)
        sec.e[first + k] = pv;
    __syncwarp();
    if (lane == 0) {
        const unsigned nn = min(kLargeSteps, first + np + (n - end));
        sec.n = nn;
        if (nn == kLargeSteps)
            sec.hi = min_f(sec.hi, sec.e[kLargeSteps - 1].end);
    }
    __syncwarp();
}

// SectionSet::put (dgmr_sections.h) by the whole warp, for an s that reaches
// into [lo, hi): lane i holds section i; the overlapped run [first, last) is found
// by ballots.  put()'s walk over the run leaves
//  * every section of the run with a smaller step than s as it is;
//  * s in the gaps between those, from s.start (or the start of a first section
//    with s's own step) to s.end (or the end of such a last one): the sections
//    with steps not smaller than s's are absorbed;
//  * what sticks out of s of an absorbed first or last section with a larger step;
// so each lane finds the places of its section and of the gap before it from
// ballots, and all write at once.  The same set, bit for bit (a GPU test builds
// random sequences both ways); empty sections and NaN steps take
// warp_put_pieces.  Insertions are most of pass 1 (85 per ray at 100k, 512^2, 3.7
// sections overlapped).  Against the pieces merged by lane 0 for every insertion:
// forward + backward 36.7 -> 34.8 ms at 100k, 512^2 (with the step store), 36.9 ->
// 35.5 ms for 16 batched 64^2 views, 1.38 -> 1.34 ms in float64 at 4k, 97x65.
template <class T>
__device__ __forceinline__ void warp_put(SectionSet<kLargeSteps, T>& sec, Section<T>* pieces, Section<T> s, unsigned lane)
{
    constexpr unsigned kFull = 0xffffffffu;
    s.start = max_f(sec.lo, s.start);
    s.end = min_f(sec.hi, s.end);
    const unsigned n = sec.n;
    Section<T> my = { T(0), T(0), T(0) };
    if (lane < n)
        my = sec.e[lane];
    const uint32_t after = __ballot_sync(kFull, lane < n && my.end > s.start);
    const unsigned first = after ? unsigned(__ffs(int(after)) - 1) : n;
    if (first >= n) {
        if (lane == 0) {
            if (first < kLargeSteps) {
                sec.e[n] = s;
                sec.n = n + 1;
            } else {
                sec.hi = s.start;
            }
        }
        __syncwarp();
        return;
    }
    const uint32_t beyond = __ballot_sync(kFull, lane >= first && lane < n && my.end > s.end);
    unsigned last = beyond ? unsigned(__ffs(int(beyond)) - 1) : n;
    const T last_start = __shfl_sync(kFull, my.start, int(last < n ? last : 0u));
    if (last < n && last_start < s.end)
        ++last;
    const bool in_run = lane >= first && lane < last;
    if (!(s.end > s.start) || s.delta_t != s.delta_t || __any_sync(kFull, in_run && (!(my.end > my.start) || my.delta_t != my.delta_t))) {
        warp_put_pieces(sec, pieces, s, first, last, lane);
        return;
    }
    const bool keep = in_run && my.delta_t < s.delta_t;
    const uint32_t kept = __ballot_sync(kFull, keep);
    // the ends of the run; an empty one (s lies in a gap) has neither
    const bool run = last > first;
    const unsigned tail = run ? last - 1u : first;
    const T f_start = __shfl_sync(kFull, my.start, int(first)), f_step = __shfl_sync(kFull, my.delta_t, int(first));
    const T l_end = __shfl_sync(kFull, my.end, int(tail)), l_step = __shfl_sync(kFull, my.delta_t, int(tail));
    const bool left = run && !((kept >> first) & 1u) && f_start < s.start, right = run && !((kept >> tail) & 1u) && s.end < l_end;
    const T from = left && f_step == s.delta_t ? f_start : s.start, to = right && l_step == s.delta_t ? l_end : s.end;
    const unsigned n_left = left && f_step != s.delta_t, n_right = right && l_step != s.delta_t;
    // the gap before the lane's kept section starts at the end of the one before
    const uint32_t before = kept & lanes_below(int(lane));
    const T gap = __shfl_sync(kFull, my.end, before ? 31 - __clz(int(before)) : 0), last_gap = __shfl_sync(kFull, my.end, kept ? 31 - __clz(int(kept)) : 0);
    const T gap_start = before ? gap : from, end_start = kept ? last_gap : from;
    const uint32_t gaps = __ballot_sync(kFull, keep && my.start - gap_start > T(0));
    const unsigned n_end = to - end_start > T(0);
    const unsigned base = first + n_left;
    const unsigned place = base + unsigned(__popc(gaps & lanes_below(int(lane) + 1))) + unsigned(__popc(before));
    const unsigned end_place = base + unsigned(__popc(gaps)) + unsigned(__popc(kept));
    const unsigned tail_place = end_place + n_end + n_right; // of section `last`
    __syncwarp(); // every lane has its section
    if (keep && place < kLargeSteps)
        sec.e[place] = my;
    if (((gaps >> lane) & 1u) && place - 1u < kLargeSteps)
        sec.e[place - 1u] = Section<T> { gap_start, my.start, s.delta_t };
    if (lane >= last && lane < n && tail_place + (lane - last) < kLargeSteps)
        sec.e[tail_place + (lane - last)] = my;
    if (lane == 29u && n_left) // lanes past the sections write what no section stands for
        sec.e[first] = Section<T> { f_start, s.start, f_step };
    if (lane == 30u && n_right && end_place + n_end < kLargeSteps)
        sec.e[end_place + n_end] = Section<T> { s.end, l_end, l_step };
    if (lane == 31u && n_end && end_place < kLargeSteps)
        sec.e[end_place] = Section<T> { end_start, to, s.delta_t };
    __syncwarp();
    if (lane == 0) {
        const unsigned nn = min(kLargeSteps, tail_place + (n - last));
        sec.n = nn;
        if (nn == kLargeSteps)
            sec.hi = min_f(sec.hi, sec.e[kLargeSteps - 1].end);
    }
    __syncwarp();
}

} // namespace dgmr
