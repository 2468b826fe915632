// DevArena (afmm_internal.cuh) over a device of a given size that only counts:
// slabs, a slab that does not fit, and the spare piece.  Needs no GPU.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <map>

static size_t g_free = 0, g_live = 0;
static std::map<void*, size_t> g_size;
static cudaError_t counted_malloc(void** p, size_t n) {
  if (n > g_free) return cudaErrorMemoryAllocation;
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  g_free -= n;
  g_size[*p] = n;
  ++g_live;
  return cudaSuccess;
}
static cudaError_t counted_free(void* p) {
  g_free += g_size.at(p);
  g_size.erase(p);
  std::free(p);
  --g_live;
  return cudaSuccess;
}
#define cudaMalloc counted_malloc
#define cudaFree counted_free
#define cudaGetLastError() cudaSuccess
#include "../../afmm2d_b200/csrc/afmm_internal.cuh"

std::atomic<int64_t>& afmm::device_alloc_counter() {
  static std::atomic<int64_t> n{0};
  return n;
}

#define CHECK(c)                                        \
  do {                                                  \
    if (!(c)) {                                         \
      std::printf("line %d: %s\n", __LINE__, #c);       \
      return 1;                                         \
    }                                                   \
  } while (0)

template <class F>
static bool out_of_memory(F&& f) {
  try {
    f();
  } catch (const afmm::Error& e) {
    return e.status == AFMM_OOM;
  }
  return false;
}

int main() {
  const size_t MB = 1 << 20;
  {  // pieces are carved from slabs on 256-byte boundaries and do not overlap
    g_free = 64 * MB;
    afmm::DevArena a;
    unsigned char* last = nullptr;
    for (int i = 0; i < 1000; ++i) {
      unsigned char* p = a.alloc<unsigned char>(1 + i % 700);
      CHECK((uintptr_t)p % 256 == 0);
      for (int t = 0; t < 1 + i % 700; ++t) p[t] = 1;
      CHECK(p != last);
      last = p;
    }
    CHECK(g_live == 1);
    a.alloc<double>(3 * MB);  // above kPiece: its own
    CHECK(g_live == 2);
  }
  CHECK(g_live == 0 && g_free == 64 * MB);
  {  // no room for a whole slab: the piece alone
    g_free = 100 * 1024;
    afmm::DevArena a;
    CHECK(a.alloc<double>(1000) != nullptr);
    CHECK(a.bytes == 8192);
    CHECK(a.alloc<double>(1000) != nullptr && a.bytes == 16384);
    CHECK(out_of_memory([&] { a.alloc<double>(20000); }));
    CHECK(a.alloc<double>(1000) != nullptr);  // the arena goes on after a refusal
  }
  {  // the spare piece goes when nothing else fits, once
    g_free = 40 * MB;
    afmm::DevArena a;
    double* spare = a.alloc_own<double>(2 * MB);  // 16 MB
    a.spare = &spare;
    double* kept = a.alloc_own<double>(MB);       // 8 MB
    CHECK(spare && kept);
    double* big = a.alloc<double>(3 * MB);        // 24 MB: 16 are free
    CHECK(big && !spare && g_free == 8 * MB);
    CHECK(out_of_memory([&] { a.alloc<double>(3 * MB); }));
    CHECK(kept && g_live == 2);
  }
  {  // another arena's request, and a slab of its own, take it too
    g_free = 20 * MB;
    afmm::DevArena a, tmp;
    tmp.lender = &a;
    double* spare = a.alloc_own<double>(2 * MB);
    a.spare = &spare;
    CHECK(tmp.alloc<double>(100) && spare);  // a small slab still fits
    CHECK(tmp.alloc<double>(MB) && !spare);
    CHECK(out_of_memory([&] { tmp.alloc<double>(4 * MB); }));
  }
  CHECK(g_live == 0);
  std::printf("ok\n");
  return 0;
}
