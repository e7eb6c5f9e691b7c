// warp_put and warp_section_covered on random insertion sequences, compared after
// every insertion with SectionSet::put, for tests/test_gpu_warp_sections.py.  A warp
// builds one set both ways: its own in shared memory, and lane 0 a second by put().
#include <cuda_runtime.h>

#include "dgmr_section_warp.cuh"

namespace {

constexpr int kWarps = 4;
using dgmr::kLargeSteps;

struct Counts {
    unsigned long long puts, covered, pieces, full, bad;
};

__device__ uint32_t next_random(uint32_t& state)
{
    state = state * 1664525u + 1013904223u;
    uint32_t x = state;
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return x ^ (x >> 16);
}

template <class T>
__device__ T unit(uint32_t& state) { return T(next_random(state) >> 8) * T(1.0 / 16777216.0); }

template <class T>
__device__ bool same(T a, T b) { return a == b || (a != a && b != b); }

template <class T>
__global__ void __launch_bounds__(kWarps * 32) check(uint32_t seed, int trials, int odd, Counts* total)
{
    __shared__ dgmr::SectionSet<kLargeSteps, T> warp_set[kWarps], lane_set[kWarps];
    __shared__ dgmr::Section<T> scratch[kWarps][2 * kLargeSteps + 1];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    dgmr::SectionSet<kLargeSteps, T>&a = warp_set[warp], &b = lane_set[warp];
    Counts c {};
    for (int trial = blockIdx.x * kWarps + int(warp); trial < trials; trial += int(gridDim.x) * kWarps) {
        uint32_t state = seed + 7919u * uint32_t(trial); // the same on every lane
        const T start = T(next_random(state) % 3) * T(0.5);
        if (lane == 0) {
            a.reset(start);
            b.reset(start);
        }
        __syncwarp();
        const int n_put = 5 + int(next_random(state) % 80);
        for (int k = 0; k < n_put; ++k) {
            T centre = T(10) * unit<T>(state), half = T(0.02) + T(2) * unit<T>(state);
            if (next_random(state) % 2) { // equal ends
                centre = T(int(centre * T(4))) / T(4);
                half = T(1 + next_random(state) % 8) / T(4);
            }
            dgmr::Section<T> s { centre - half, centre + half, next_random(state) % 3 == 0 ? T(1 + next_random(state) % 4) / T(32) : half / T(31) };
            if (odd && next_random(state) % 16 == 0)
                s.end = T(1) / T(0);
            if (odd && next_random(state) % 16 == 0)
                s.end = s.start;
            if (odd && next_random(state) % 32 == 0)
                s.delta_t = T(0) / T(0);
            ++c.puts;
            // as the march calls them; it has no NaN steps, which the test for covered sections does not see
            if (!(s.end <= a.lo || s.start >= a.hi)) {
                if (!odd && dgmr::warp_section_covered(a, s, lane)) {
                    ++c.covered;
                } else {
                    bool piece = s.delta_t != s.delta_t || !(s.end > s.start);
                    for (unsigned i = 0; i < a.n; ++i)
                        piece = piece || a.e[i].delta_t != a.e[i].delta_t || !(a.e[i].end > a.e[i].start);
                    c.pieces += piece;
                    __syncwarp();
                    dgmr::warp_put(a, scratch[warp], s, lane);
                }
            }
            if (lane == 0)
                b.put(s);
            __syncwarp();
            c.full += a.n == kLargeSteps;
            bool fine = a.n == b.n && same(a.lo, b.lo) && same(a.hi, b.hi);
            if (lane < a.n && lane < kLargeSteps)
                fine = fine && same(a.e[lane].start, b.e[lane].start) && same(a.e[lane].end, b.e[lane].end) && same(a.e[lane].delta_t, b.e[lane].delta_t);
            fine = __all_sync(0xffffffffu, fine);
            if (!fine) {
                ++c.bad;
                break;
            }
            __syncwarp();
        }
        __syncwarp();
    }
    if (lane == 0) {
        atomicAdd(&total->puts, c.puts);
        atomicAdd(&total->covered, c.covered);
        atomicAdd(&total->pieces, c.pieces);
        atomicAdd(&total->full, c.full);
        atomicAdd(&total->bad, c.bad);
    }
}

} // namespace

// counts: insertions, skipped as covered, with an empty section or a NaN step about, sets that were full, sets that differ
extern "C" int warp_sections(int is_double, int odd, uint32_t seed, int trials, unsigned long long* counts)
{
    Counts* total = nullptr;
    if (cudaMalloc(&total, sizeof(Counts)) != cudaSuccess)
        return 1;
    cudaMemset(total, 0, sizeof(Counts));
    if (is_double)
        check<double><<<296, kWarps * 32>>>(seed, trials, odd, total);
    else
        check<float><<<296, kWarps * 32>>>(seed, trials, odd, total);
    const bool fine = cudaGetLastError() == cudaSuccess && cudaMemcpy(counts, total, sizeof(Counts), cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(total);
    return fine ? 0 : 1;
}
