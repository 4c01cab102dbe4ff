// Programmatic dependent launch (PDL): a kernel launched with the stream-serialisation attribute may start while its
// predecessor in the stream is still running; it must call pdl_wait() before it touches anything the predecessor
// (or any earlier kernel) wrote or still reads, and pdl_trigger() lets its own successor start early in turn.
// A decode step is several hundred short kernels in one stream: without this every boundary costs the full
// drain -> launch -> ramp sequence; with it the successor's CTAs are resident with their set-up done (barriers,
// TMEM, descriptor prefetch) when the predecessor's last CTA retires. Inside a CUDA graph the attribute becomes a
// programmatic dependency edge.
//
// Rules used in this library:
//   * pdl_trigger() as early as possible; pdl_wait() before the first global-memory access that is not a read of
//     weights / constants that no work in flight writes. The caller vouches for a GEMM's weight operand (`fixed_w`): loaded weights
//     are never written while the engine runs; a matrix that a step makes (4-bit weights expanded into scratch) is not one of them, and
//     its GEMM takes an ordinary launch;
//   * a kernel launched through launch_pdl() that lacks pdl_wait() would race: only kernels that call it are launched
//     with the attribute;
//   * both calls are no-ops in a kernel launched without the attribute.
// The attribute is on for the kernels launched through launch_early(): those of decode steps, most of which leave room on the SM for a
// neighbour, so that a GEMM's first weight tiles are on their way while the norm or the attention before it ends. (Not all do: decode
// attention with heads of 192 and 256 columns and e4m3 GEMMs with K in the tens of thousands take more than half of the shared memory;
// what follows them starts as their CTAs end.) 8 layers of 4096, one sequence: 1070 -> 976 us per step, 64 sequences: 1575 -> 1544 us. The others take it with
// KSANA_PDL=1 only: kernels that need a whole SM gained nothing (graphs of 800 kernels, within noise), and the 4-bit stream, whose CTAs
// fill the register file, made its step slower (1130 -> 1386 us). KSANA_PDL=0 switches it off everywhere.
#pragma once
#include <cuda_runtime.h>
#include <cstdlib>
#include <utility>

namespace ksana {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool pdl_enabled() {
  static const bool on = []() {
    const char* e = std::getenv("KSANA_PDL");
    return e && e[0] == '1';
  }();
  return on;
}

inline bool pdl_early_enabled() {
  static const bool on = []() {
    const char* e = std::getenv("KSANA_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

// kernel<<<grid, block, smem, st>>>(args...) in clusters of `cluster` blocks along x, with the programmatic stream-serialisation
// attribute where `early`.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_cluster(bool early, void (*kernel)(KArgs...), dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t st,
                                  Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (early) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                              Args&&... args) {
  return launch_cluster(pdl_enabled(), kernel, grid, block, 1, smem, st, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_early(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  return launch_cluster(pdl_early_enabled(), kernel, grid, block, 1, smem, st, std::forward<Args>(args)...);
}

}  // namespace ksana
