// Launches of short kernels that follow one another on a stream, without the
// gap between one's end and the next one's start: the next grid is launched when
// every block of the current one runs (programmatic dependent launch), and waits
// on the device for the current one to finish.
//
// A kernel launched this way calls chain_start() before it reads or writes
// anything; a kernel that such a launch may follow only has to end.  The waiting
// blocks hold their place on the SMs while the current kernel ends, so a kernel
// that follows a long one with a thin tail (the blend, the march, the per-pixel
// backward) is launched plainly.
//
// Forward at 10k, 256^2: 0.219 -> 0.173 ms; at 1M, 1080p: 0.577 -> 0.528; forward +
// backward at 200k, 1024^2: 0.669 -> 0.620 (means of four cameras).  Above
// kChainMost Gaussian slots the kernels over them are long enough for the places
// they hold to cost more than the gaps (12 batched views of 7.4M slots: 5.228 ms
// plain, 5.241 chained).  At any size chained (kChainAlways): kernels of one block,
// which hold one place, and the scan behind a single frame's preprocess (2.5M
// Gaussians, 1080p: 0.835 ms, plain 0.845; 4M, 1024^2: 0.929, 0.933).  A blend that
// does not fit the chip at once is launched plainly, and so is its order kernel (1M,
// 1080p, 8160 tiles: chained 0.540 ms instead of 0.528; at 256 tiles 0.173 instead of
// 0.180).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <utility>

namespace dgmr {

__device__ __forceinline__ void chain_start()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr uint32_t kChainMost = 2u << 20;
constexpr bool kChainAlways = true;

// A stream, and whether a kernel launched on it is chained.
struct ChainStream {
    cudaStream_t s;
    bool chained;
    ChainStream(cudaStream_t stream, bool chain)
        : s(stream)
        , chained(chain)
    {
    }
    operator cudaStream_t() const { return s; }
};

template <class... Params, class... Args>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, const ChainStream& stream, Args&&... args)
{
    cudaLaunchAttribute chained {};
    chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chained.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config {};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream.s;
    config.attrs = &chained;
    config.numAttrs = stream.chained ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

} // namespace dgmr
