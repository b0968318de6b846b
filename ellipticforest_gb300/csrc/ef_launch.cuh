// Launches of kernel chains with programmatic stream serialisation: a kernel may start while the one before it in
// the stream drains, so that its launch, its block scheduling and what it does before pdl_wait() overlap.  Every
// thread of such a kernel calls pdl_wait() before its first access to global memory: it returns when the kernels
// before have completed and their writes are visible.  pdl_trigger() lets the next kernel start early; it still
// waits for this one's completion in its own pdl_wait().  A chain of short kernels (the merges' digits and
// products, the levels of a small solve) saves 1 to 2 us per kernel.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace efgb {
namespace {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
    pdl_wait();
    pdl_trigger();
}

// the largest grid that is chained inside a graph
constexpr unsigned kChainedBlocks = 76;

inline bool being_captured(cudaStream_t st) {
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &c) == cudaSuccess && c != cudaStreamCaptureStatusNone;
}

// few: grids that leave SMs free only; all: for chains that are launched kernel by kernel
enum class Chain { none, few, all };

// a build's merges: a chain when they are launched one by one, plain edges when they are captured (there even small
// grids lose: level-7 build 28.6 -> 28.9 ms)
inline Chain merge_chain(cudaStream_t st) { return being_captured(st) ? Chain::none : Chain::all; }

template <class... P, class... A>
inline void launch_chained(Chain chain, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                           A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chain == Chain::all || (chain == Chain::few && grid.x * grid.y * grid.z <= kChainedBlocks) ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace
}  // namespace efgb
