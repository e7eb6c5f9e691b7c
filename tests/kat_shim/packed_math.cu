// The packed float functions against their scalar forms, every float of a range,
// for tests/test_gpu_packed_math.py.  The halves of a pair walk the range from its
// two ends, so both are checked and take different branches.
#include <cuda_runtime.h>

#include "dgmr_f32x2.cuh"

namespace {

enum Function { kRecip, kExp, kErf };

template <int kFunction>
__global__ void sweep(uint32_t lo, uint32_t hi, unsigned long long* bad, uint32_t* one_bad)
{
    const uint64_t n = uint64_t(hi) - lo + 1u, step = uint64_t(gridDim.x) * blockDim.x;
    unsigned long long mine = 0;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) {
        const float x[2] = { __uint_as_float(lo + uint32_t(i)), __uint_as_float(hi - uint32_t(i)) };
        const dgmr::F2 v = dgmr::f2(x[0], x[1]);
        float got[2];
        dgmr::split2(kFunction == kRecip ? dgmr::recip2(v) : kFunction == kExp ? dgmr::exp2_nonpos(v) : dgmr::erf2(v), &got[0], &got[1]);
        for (int h = 0; h < 2; ++h) {
            const float want = kFunction == kRecip ? 1.f / x[h] : kFunction == kExp ? dgmr_fm::exp_f(x[h]) : dgmr_fm::erf_f(x[h]);
            if (__float_as_uint(got[h]) != __float_as_uint(want) && !(got[h] != got[h] && want != want)) {
                ++mine;
                *one_bad = __float_as_uint(x[h]);
            }
        }
    }
    if (mine)
        atomicAdd(bad, mine);
}

} // namespace

// Values with the bit patterns lo to hi for which a half differs (-1: a CUDA error), and one of them.
extern "C" long long packed_math_mismatches(int function, uint32_t lo, uint32_t hi, uint32_t* one)
{
    unsigned long long* buffer = nullptr;
    if (cudaMalloc(&buffer, 16) != cudaSuccess)
        return -1;
    cudaMemset(buffer, 0, 16);
    uint32_t* one_bad = reinterpret_cast<uint32_t*>(buffer + 1);
    switch (function) {
    case kRecip: sweep<kRecip><<<1184, 256>>>(lo, hi, buffer, one_bad); break;
    case kExp: sweep<kExp><<<1184, 256>>>(lo, hi, buffer, one_bad); break;
    default: sweep<kErf><<<1184, 256>>>(lo, hi, buffer, one_bad); break;
    }
    unsigned long long got[2] = { 0, 0 };
    const bool fine = cudaGetLastError() == cudaSuccess && cudaMemcpy(got, buffer, 16, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(buffer);
    *one = uint32_t(got[1]);
    return fine ? static_cast<long long>(got[0]) : -1;
}
