// Gathering of kernel launches into CUDA graphs (see launch.h).
#include <algorithm>
#include <cstring>
#include <list>
#include <unordered_map>
#include <vector>

#include "runtime.h"

namespace fhert {

namespace {

// Longer sequences are submitted in pieces, so that the GPU starts while the
// host is still preparing the rest (a bootstrap makes about 1500 launches).
constexpr size_t kMaxNodes = 48;
// Kept graphs; the one used longest ago goes first.
constexpr size_t kMaxGraphs = 1024;

struct Item {
  const void* func;
  dim3        grid, block;
  size_t      smem;
  size_t      first, bytes;  // parameters in the arena
  int         count, first_param;
};

struct Shape {  // what a kept graph is found by
  const void* func;
  dim3        grid, block;
  size_t      smem;
  bool operator==(const Shape& o) const {
    return func == o.func && smem == o.smem && grid.x == o.grid.x && grid.y == o.grid.y &&
           grid.z == o.grid.z && block.x == o.block.x && block.y == o.block.y && block.z == o.block.z;
  }
};

struct Kept {
  uint64_t                     hash;
  std::vector<Shape>           shapes;
  cudaGraph_t                  graph = nullptr;
  cudaGraphExec_t              exec  = nullptr;
  std::vector<cudaGraphNode_t> nodes;
  std::vector<unsigned char>   bytes;  // parameters the executable graph holds now
};

struct Batch {
  int                        depth = 0;
  std::vector<Item>          items;
  std::vector<unsigned char> arena;    // parameter bytes of all items
  std::vector<size_t>        offsets;  // of every parameter in the arena
  std::list<Kept>            kept;     // most recently used first
  std::unordered_multimap<uint64_t, std::list<Kept>::iterator> by_hash;
};
Batch g_batch;

bool graphs_on() {
  static const bool on = [] {
    const char* e = std::getenv("FHERT_LAUNCH_GRAPHS");
    return !(e != nullptr && e[0] == '0');
  }();
  return on;
}

uint64_t mix(uint64_t h, uint64_t v) { return (h ^ v) * 0x9E3779B97F4A7C15ull + (h >> 29); }

Shape shape_of(const Item& it) { return Shape{it.func, it.grid, it.block, it.smem}; }

uint64_t hash_items(const std::vector<Item>& items) {
  uint64_t h = items.size();
  for (const Item& it : items) {
    h = mix(h, (uint64_t)(uintptr_t)it.func);
    h = mix(h, ((uint64_t)it.grid.x << 32) | (it.grid.y << 16) | it.grid.z);
    h = mix(h, ((uint64_t)it.block.x << 32) | it.smem);
  }
  return h;
}

cudaKernelNodeParams node_params(Batch& b, const Item& it, std::vector<void*>& ptrs) {
  ptrs.resize(it.count);
  for (int i = 0; i < it.count; i++) ptrs[i] = b.arena.data() + b.offsets[it.first_param + i];
  cudaKernelNodeParams p{};
  p.func           = const_cast<void*>(it.func);
  p.gridDim        = it.grid;
  p.blockDim       = it.block;
  p.sharedMemBytes = (unsigned)it.smem;
  p.kernelParams   = ptrs.data();
  return p;
}

void drop(Kept& k) {
  if (k.exec) cudaGraphExecDestroy(k.exec);
  if (k.graph) cudaGraphDestroy(k.graph);
}

std::list<Kept>::iterator find_kept(Batch& b, uint64_t h) {
  auto range = b.by_hash.equal_range(h);
  for (auto it = range.first; it != range.second; ++it) {
    const Kept& k = *it->second;
    if (k.shapes.size() != b.items.size()) continue;
    bool same = true;
    for (size_t i = 0; i < b.items.size() && same; i++) same = k.shapes[i] == shape_of(b.items[i]);
    if (same) return it->second;
  }
  return b.kept.end();
}

std::list<Kept>::iterator build(Batch& b, uint64_t h) {
  if (b.kept.size() >= kMaxGraphs) {
    auto last  = std::prev(b.kept.end());
    auto range = b.by_hash.equal_range(last->hash);
    for (auto it = range.first; it != range.second; ++it)
      if (it->second == last) {
        b.by_hash.erase(it);
        break;
      }
    drop(*last);
    b.kept.erase(last);
  }
  b.kept.emplace_front();
  auto  pos = b.kept.begin();
  Kept& k   = *pos;
  k.hash    = h;
  CUDA_CHECK(cudaGraphCreate(&k.graph, 0));
  std::vector<void*> ptrs;
  for (const Item& it : b.items) {
    k.shapes.push_back(shape_of(it));
    cudaKernelNodeParams p = node_params(b, it, ptrs);
    cudaGraphNode_t      node;
    CUDA_CHECK(cudaGraphAddKernelNode(&node, k.graph, k.nodes.empty() ? nullptr : &k.nodes.back(),
                                      k.nodes.empty() ? 0 : 1, &p));
    k.nodes.push_back(node);
  }
  CUDA_CHECK(cudaGraphInstantiate(&k.exec, k.graph, 0));
  k.bytes = b.arena;
  b.by_hash.emplace(h, pos);
  return pos;
}

// res = src, or 0: one 16-byte word per thread and step
template <bool CLEAR>
__global__ void __launch_bounds__(256) copy_words_kernel(uint4* res, const uint4* src, size_t words) {
  const size_t step = (size_t)gridDim.x * 256;
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < words; i += step)
    res[i] = CLEAR ? make_uint4(0, 0, 0, 0) : src[i];
}

bool gathering() {
  return g_batch.depth > 0 && graphs_on() && !image_capturing() && !prof_running();
}

}  // namespace

LaunchScope::LaunchScope() { g_batch.depth++; }
LaunchScope::~LaunchScope() {
  if (--g_batch.depth == 0) launch_flush();
}

void launch_flush() {
  Batch& b = g_batch;
  if (b.items.empty()) return;
  const uint64_t h   = hash_items(b.items);
  auto           pos = find_kept(b, h);
  if (pos == b.kept.end()) {
    pos = build(b, h);
  } else {
    if (pos != b.kept.begin()) b.kept.splice(b.kept.begin(), b.kept, pos);
    std::vector<void*> ptrs;
    for (size_t i = 0; i < b.items.size(); i++) {
      const Item& it = b.items[i];
      // same kernels, same parameter layout: same offsets
      if (std::memcmp(pos->bytes.data() + it.first, b.arena.data() + it.first, it.bytes) == 0) continue;
      cudaKernelNodeParams p = node_params(b, it, ptrs);
      CUDA_CHECK(cudaGraphExecKernelNodeSetParams(pos->exec, pos->nodes[i], &p));
      std::memcpy(pos->bytes.data() + it.first, b.arena.data() + it.first, it.bytes);
    }
  }
  b.items.clear();
  b.offsets.clear();
  b.arena.clear();
  CUDA_CHECK(cudaGraphLaunch(pos->exec, ctx_noflush()->stream));
}

void launch_release() {
  for (Kept& k : g_batch.kept) drop(k);
  g_batch.kept.clear();
  g_batch.by_hash.clear();
}

bool launch_copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
  if (!gathering() || bytes == 0 || (((uintptr_t)dst | (uintptr_t)src | bytes) & 15) != 0) {
    launch_flush();  // the caller's copy comes after what was gathered
    return false;
  }
  const size_t   words = bytes / 16;
  const unsigned grid  = (unsigned)std::min<size_t>((words + 1023) / 1024, 148 * 16);
  uint4*         d     = static_cast<uint4*>(dst);
  const uint4*   s     = static_cast<const uint4*>(src);
  if (src == nullptr) launch(copy_words_kernel<true>, grid, 256, 0, stream, d, s, words);
  else launch(copy_words_kernel<false>, grid, 256, 0, stream, d, s, words);
  return true;
}

void launch_raw(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                void** params, const size_t* sizes, int count) {
  Batch& b = g_batch;
  if (!gathering()) {
    CUDA_CHECK(cudaLaunchKernel(func, grid, block, params, smem, stream));
    return;
  }
  Item it{func, grid, block, smem, b.arena.size(), 0, count, (int)b.offsets.size()};
  for (int i = 0; i < count; i++) {
    const size_t at = (b.arena.size() + 15) & ~(size_t)15;
    b.arena.resize(at + sizes[i]);
    std::memcpy(b.arena.data() + at, params[i], sizes[i]);
    b.offsets.push_back(at);
  }
  it.bytes = b.arena.size() - it.first;
  b.items.push_back(it);
  if (b.items.size() >= kMaxNodes) launch_flush();
}

}  // namespace fhert
