// Kernel launches of the library, direct or gathered into CUDA graphs.
//
// A launch into a stream costs the host 4 to 6 us here, more than most of the
// kernels of one operation take, and the GPU 2 us from one kernel to the next.
// The launches an entry point makes are therefore gathered and submitted
// together before it returns, as one CUDA graph (a chain in launch order): 1.1 us
// per graph plus 0.25 us per node whose parameters changed, and 0.7 us from node
// to node on the GPU.  (An entry point with 12 launches: 48 us of host time
// launched one by one, 4 us as a graph.)  The executable graph is kept and found
// again by the sequence of kernels and grid shapes; only parameters are renewed,
// so what is computed never depends on what an earlier call computed.
//
// Launches go straight to the stream outside such a scope, while a program run
// is captured (capture_dag.cu orders those), while per-kernel timing is on, and
// with FHERT_LAUNCH_GRAPHS=0.  Anything else that is put on the stream, or that
// gives memory back to the driver, first submits what was gathered.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <tuple>
#include <utility>

namespace fhert {

// Around the body of an entry point; nested scopes submit when the outermost ends.
struct LaunchScope {
  LaunchScope();
  ~LaunchScope();
  LaunchScope(const LaunchScope&)            = delete;
  LaunchScope& operator=(const LaunchScope&) = delete;
};

void launch_flush();    // submits what was gathered so far
// A device-to-device copy (or, without a source, a clear) as one of the gathered
// launches; false when nothing is being gathered or the ranges are not made of
// 16-byte words: the caller then uses the stream.
bool launch_copy(void* dst, const void* src, size_t bytes, cudaStream_t stream);
void launch_release();  // drops the kept graphs (context teardown)
void launch_raw(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                void** params, const size_t* sizes, int count);

namespace launch_detail {
template <typename Tuple, size_t... I>
inline void go(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
               Tuple& bound, std::index_sequence<I...>) {
  void*        params[] = {(void*)&std::get<I>(bound)...};
  const size_t sizes[]  = {sizeof(std::tuple_element_t<I, Tuple>)...};
  launch_raw(func, grid, block, smem, stream, params, sizes, (int)sizeof...(I));
}
}  // namespace launch_detail

template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                   const A&... args) {
  std::tuple<P...> bound(static_cast<P>(args)...);
  launch_detail::go((const void*)kernel, grid, block, smem, stream, bound,
                    std::index_sequence_for<P...>());
}

}  // namespace fhert
