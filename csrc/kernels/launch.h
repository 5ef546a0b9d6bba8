// Launches whose start may overlap the end of the previous kernel of the stream (programmatic stream serialization).
//
// A short kernel spends a few microseconds on its launch, on barriers, TMEM and descriptors before it touches memory, and
// the SMs sit idle meanwhile.  A kernel launched through launchOverlapped() may be placed on SMs while its predecessor's
// last CTAs are still running; it calls pdl_wait() before its first access to global memory, which returns when the
// predecessor has completed and its writes are visible, and pdl_launch(), which lets its own successor do the same: a short
// kernel once it holds its resources, a GEMM with its last operand load.  Both are no-ops in a kernel that was launched the
// ordinary way, and an ordinary launch behind such a kernel waits for its end as usual.
//
// What a kernel reads after pdl_wait() may have been written after the kernel started.  So its pointers are not `__restrict__`
// (a `const` one would promise data that nobody writes during the kernel: the compiler could read it through the non-coherent
// path, or above the wait, which orders nothing that cannot alias) and it uses neither __ldg nor __ldcg, whose place in the
// program is not fixed either (prims.cuh: ld_f32 and the like).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace pccl {

template <class... KArgs, class... Args>
inline cudaError_t launchOverlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

#ifdef __CUDACC__
namespace dev {
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
}  // namespace dev
#endif

}  // namespace pccl
