// dsem_blocks.cu -- the device blocks that contexts keep between dsem_adjoint calls: one per context
// of at most BLOCK_MAX bytes, all together at most BLOCK_KEEP.  A block goes back to the device with its context, when
// its context needs a larger one, and when an allocation of the library fails (dev_malloc).
#include <cuda_runtime.h>

#include <map>
#include <mutex>

#include "dsem_ctx.h"

namespace {

constexpr size_t BLOCK_MAX = (size_t)4 << 30, BLOCK_KEEP = (size_t)16 << 30;

struct Kept {
  void *p;
  size_t size;
};
std::mutex g_mutex;
std::map<const dsem_ctx *, Kept> g_kept;  // blocks not in use
size_t g_total = 0;

void free_kept(std::map<const dsem_ctx *, Kept>::iterator it) {
  cudaFree(it->second.p);
  g_total -= it->second.size;
  g_kept.erase(it);
}

}  // namespace

namespace dsem_int {

void *block_take(const dsem_ctx *c, size_t bytes, size_t *size) {
  std::lock_guard<std::mutex> lock(g_mutex);
  const auto it = g_kept.find(c);
  if (it == g_kept.end()) return nullptr;
  if (it->second.size < bytes) {
    free_kept(it);
    return nullptr;
  }
  void *p = it->second.p;
  *size = it->second.size;
  g_total -= it->second.size;
  g_kept.erase(it);
  return p;
}

void block_give(const dsem_ctx *c, void *p, size_t size) {
  if (!p) return;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (size > BLOCK_MAX || size > BLOCK_KEEP - g_total || g_kept.count(c)) {
    cudaFree(p);
    return;
  }
  g_kept[c] = Kept{p, size};
  g_total += size;
}

bool block_drop(const dsem_ctx *c) {
  std::lock_guard<std::mutex> lock(g_mutex);
  const bool any = c ? g_kept.count(c) != 0 : !g_kept.empty();
  if (c && any) free_kept(g_kept.find(c));
  while (!c && !g_kept.empty()) free_kept(g_kept.begin());
  return any;
}

}  // namespace dsem_int
