// Page-locked host memory for the operands of the host entry points.
//
// On GB300 hosts (Arm, 64 KB base pages) a 2 GiB page-locked buffer from
// cudaHostAlloc copies at 10 ms when it was just used, but its first copy
// after a pause grows with the buffer's age (to 200+ ms for 2 GiB after a
// minute of alternating compute and copies), while a buffer backed by
// transparent huge pages copies at the same 10 ms throughout.  This
// allocator maps anonymous memory aligned to the huge-page size, asks for
// huge pages (MADV_HUGEPAGE), touches it and page-locks it with
// cudaHostRegister.  Where the kernel offers no huge pages the memory is
// still page-locked and usable.
//
// The host entry points copy operands in such memory directly.  Other host
// buffers (malloc'd, as the reference's, or page-locked elsewhere) of up to a
// staging chunk are moved by a kernel that reads or writes them where they
// lie: the GPU shares the host's page tables over NVLink-C2C and moves 200
// GB/s in and 170 GB/s out (8 MB: 52 us), where one CPU core packs 10 GB/s.
// Every page of them is touched on the host first (host_touch.h).  Larger ones
// are packed into two staging buffers of the above kind by several CPU threads,
// each chunk's DMA overlapping the packing of the next (host_copy2d).  (Just
// above the default chunk the packing is the slower of the two, whole calls of
// m = n = 5800, 257 MiB: 11.2 against 6.9 ms; 8192: 21.6 / 14.7, warm.  A larger
// UVATRMM_OPT_HOST_STAGE_KB moves the line.)
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "api_internal.h"
#include "host_touch.h"

namespace uvt {
namespace {

std::mutex g_host_mu;
std::map<void *, size_t> g_host_maps;  // base -> mapped length

// The transparent-huge-page size the kernel reports, else 2 MiB.
size_t huge_page_bytes() {
  static size_t hp = [] {
    size_t v = 0;
    if (FILE *f = fopen("/sys/kernel/mm/transparent_hugepage/hpage_pmd_size", "r")) {
      unsigned long long x = 0;
      if (fscanf(f, "%llu", &x) == 1) v = (size_t)x;
      fclose(f);
    }
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    if (v < page || (v & (v - 1))) v = (size_t)2 << 20;
    return v;
  }();
  return hp;
}

// True when [p, p + bytes) lies inside one uvatrmm_host_alloc region.
bool in_host_alloc(const void *p, size_t bytes) {
  std::lock_guard<std::mutex> g(g_host_mu);
  auto it = g_host_maps.upper_bound(const_cast<void *>(p));
  if (it == g_host_maps.begin()) return false;
  --it;
  const uintptr_t base = reinterpret_cast<uintptr_t>(it->first), a = reinterpret_cast<uintptr_t>(p);
  return a >= base && a + bytes <= base + it->second;
}

int map_region(size_t bytes, void **out, size_t *len_out) {
  const size_t hp = huge_page_bytes();
  const size_t len = ((bytes ? bytes : 1) + hp - 1) / hp * hp;
  if (len < bytes) return fail(UVATRMM_EINVAL, "size overflows");
  // Over-map by one huge page and trim, so the region starts on a huge-page boundary.
  void *raw = mmap(nullptr, len + hp, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (raw == MAP_FAILED) return fail(UVATRMM_ENOMEM, "mmap of " + std::to_string(len + hp) + " bytes failed");
  const uintptr_t a = reinterpret_cast<uintptr_t>(raw), b = (a + hp - 1) / hp * hp;
  if (b > a) munmap(raw, b - a);
  munmap(reinterpret_cast<void *>(b + len), a + hp - b);
  void *p = reinterpret_cast<void *>(b);
  madvise(p, len, MADV_HUGEPAGE);  // advisory: ignored where huge pages are off
  memset(p, 0, len);               // fault the pages in (as huge pages where granted)
  cudaError_t e = cudaHostRegister(p, len, cudaHostRegisterDefault);
  if (e != cudaSuccess) {
    munmap(p, len);
    return cuda_fail(e, "cudaHostRegister");
  }
  {
    std::lock_guard<std::mutex> g(g_host_mu);
    g_host_maps[p] = len;
  }
  *out = p;
  *len_out = len;
  return UVATRMM_OK;
}

// dst[l][i] = src[l][i] for lines of `width` doubles, either side in host
// memory.  tri: 0 all; 1 only i >= l; 2 only i <= l.  Four elements in flight
// per thread; under 2^32 elements.
__global__ void __launch_bounds__(256) host_move_kernel(double *dst, int64_t dpitch, const double *src,
                                                        int64_t spitch, uint32_t width, uint32_t total, int tri) {
  const uint32_t step = gridDim.x * 256;
  for (uint64_t i0 = blockIdx.x * 256 + threadIdx.x; i0 < total; i0 += 4ull * step) {
    double v[4];
    int64_t to[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint64_t i = i0 + (uint64_t)q * step;
      to[q] = -1;
      if (i < total) {
        const uint32_t l = (uint32_t)i / width, c = (uint32_t)i - l * width;
        if (tri == 0 || (tri == 1 ? c >= l : c <= l)) {
          to[q] = c + l * dpitch;
          v[q] = src[c + l * spitch];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (to[q] >= 0) dst[to[q]] = v[q];
  }
}

// Touches every page of the host lines (of the triangle, see line_part), so
// that a bad pointer or a hole in the operand faults here and not on the GPU,
// and, with `write`, so that the GPU does not wait for the kernel to map a new
// buffer's pages one by one.
void touch_lines(const void *host, size_t pitch, size_t width, size_t lines, int tri, bool write) {
  for_each_page(reinterpret_cast<uintptr_t>(host), pitch, width, lines, tri, (size_t)sysconf(_SC_PAGESIZE),
                [&](uintptr_t a) {
                  volatile char *b = reinterpret_cast<volatile char *>(a);
                  const char c = *b;
                  if (write) *b = c;
                });
}

// Moves the lines by a kernel, where it can: sizes in bytes.
bool move_by_kernel(uvatrmm_handle_t h, void *dst, size_t dpitch, const void *src, size_t spitch, size_t width,
                    size_t lines, bool h2d, int tri, cudaError_t *e) {
  const size_t bits = reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src) | dpitch | spitch | width;
  if (!h->host_direct || bits % 8 != 0 || width * lines > h->hstage_bytes || width * lines / 8 > UINT32_MAX / 2)
    return false;
  if (dpitch == width && spitch == width && !tri) {  // one long line
    width *= lines;
    dpitch = spitch = width;
    lines = 1;
  }
  touch_lines(h2d ? src : dst, h2d ? spitch : dpitch, width, lines, tri, !h2d);
  const uint32_t total = (uint32_t)(width / 8 * lines);
  const unsigned grid = std::min<unsigned>((total + 1023) / 1024, (unsigned)h->num_sms * 8);
  host_move_kernel<<<grid, 256, 0, h->stream>>>(static_cast<double *>(dst), (int64_t)(dpitch / 8),
                                                static_cast<const double *>(src), (int64_t)(spitch / 8),
                                                (uint32_t)(width / 8), total, tri);
  *e = cudaGetLastError();
  return true;
}

// Copies `lines` lines of `width` bytes with up to 16 threads.
void par_copy(void *dst, size_t dpitch, const void *src, size_t spitch, size_t width, size_t lines) {
  char *d = static_cast<char *>(dst);
  const char *s = static_cast<const char *>(src);
  const size_t total = width * lines;
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  const size_t nt = std::min<size_t>({16, hw, std::max<size_t>(1, total >> 22)});  // >= 4 MiB per thread
  auto part = [&](size_t i) {
    if (dpitch == width && spitch == width) {
      const size_t b0 = total * i / nt, b1 = total * (i + 1) / nt;
      memcpy(d + b0, s + b0, b1 - b0);
    } else {
      for (size_t l = lines * i / nt, l1 = lines * (i + 1) / nt; l < l1; ++l)
        memcpy(d + l * dpitch, s + l * spitch, width);
    }
  };
  std::vector<std::thread> th;
  size_t started = 1;
  try {
    for (; started < nt; ++started) th.emplace_back(part, started);
  } catch (...) {  // no thread available: the caller copies the remaining parts
  }
  part(0);
  for (size_t i = started; i < nt; ++i) part(i);
  for (auto &t : th) t.join();
}

}  // namespace

bool host_alloc_contains(const void *p, size_t bytes) { return in_host_alloc(p, bytes); }

cudaError_t copy_triangle_h2d(uvatrmm_handle_t h, double *dA, int64_t la, const double *A, int64_t lda, int64_t ka,
                              bool lower) {
  cudaError_t moved = cudaSuccess;
  if (!in_host_alloc(A, (size_t)(lda * (ka - 1) + ka) * 8) &&
      move_by_kernel(h, dA, (size_t)la * 8, A, (size_t)lda * 8, (size_t)ka * 8, (size_t)ka, true, lower ? 1 : 2, &moved))
    return moved;
  for (int64_t j0 = 0; j0 < ka; j0 += kTriCopyCols) {
    const int64_t w = std::min<int64_t>(kTriCopyCols, ka - j0);
    const int64_t r0 = lower ? j0 : 0, r1 = lower ? ka : j0 + w;
    const cudaError_t e = host_copy2d(h, dA + r0 + j0 * la, (size_t)la * 8, A + r0 + j0 * lda, (size_t)lda * 8,
                                      (size_t)(r1 - r0) * 8, (size_t)w, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t host_copy2d(uvatrmm_handle_t h, void *dst, size_t dpitch, const void *src, size_t spitch, size_t width,
                        size_t height, cudaMemcpyKind kind) {
  if (width == 0 || height == 0) return cudaSuccess;
  const bool h2d = kind == cudaMemcpyHostToDevice;
  const void *host = h2d ? src : dst;
  const size_t hpitch = h2d ? spitch : dpitch;
  const size_t extent = hpitch * (height - 1) + width;
  const bool flat = dpitch == width && spitch == width;
  // Direct DMA: operands in uvatrmm_host_alloc memory, small copies, or lines
  // longer than a staging chunk.
  const bool own = in_host_alloc(host, extent);
  cudaError_t moved = cudaSuccess;
  if (!own && move_by_kernel(h, dst, dpitch, src, spitch, width, height, h2d, 0, &moved)) {
    if (moved == cudaSuccess && !h2d) moved = cudaStreamSynchronize(h->stream);  // landed on return
    return moved;
  }
  if (own || width * height < ((size_t)1 << 20) || (!flat && width > h->hstage_bytes)) {
    if (flat) return cudaMemcpyAsync(dst, src, width * height, kind, h->stream);
    return cudaMemcpy2DAsync(dst, dpitch, src, spitch, width, height, kind, h->stream);
  }
  if (h->hstage_cap < h->hstage_bytes) {
    release_host_staging(h);
    size_t len = 0;
    for (int b = 0; b < 2; ++b) {
      if (map_region(h->hstage_bytes, &h->hstage[b], &len) != UVATRMM_OK) return cudaErrorMemoryAllocation;
      cudaError_t e = cudaEventCreateWithFlags(&h->hstage_ev[b], cudaEventDisableTiming);
      if (e != cudaSuccess) return e;
    }
    h->hstage_cap = h->hstage_bytes;
  }
  // A chunk is `lpc` lines (or, for a flat copy, `lpc` bytes of one line).
  const size_t unit = flat ? 1 : width, count = flat ? width * height : height;
  const size_t lpc = std::max<size_t>(1, h->hstage_bytes / unit);
  const size_t nchunk = (count + lpc - 1) / lpc;
  auto rows = [&](size_t k) { return std::min(lpc, count - k * lpc); };
  cudaError_t e = cudaSuccess;
  if (h2d) {
    const char *s = static_cast<const char *>(src);
    char *d = static_cast<char *>(dst);
    for (size_t k = 0; k < nchunk && e == cudaSuccess; ++k) {
      const int b = (int)(k & 1);
      e = cudaEventSynchronize(h->hstage_ev[b]);  // the DMA that last read this buffer
      if (e != cudaSuccess) break;
      const size_t n = rows(k);
      if (flat) {
        par_copy(h->hstage[b], n, s + k * lpc, n, n, 1);
        e = cudaMemcpyAsync(d + k * lpc, h->hstage[b], n, kind, h->stream);
      } else {
        par_copy(h->hstage[b], width, s + k * lpc * spitch, spitch, width, n);
        e = cudaMemcpy2DAsync(d + k * lpc * dpitch, dpitch, h->hstage[b], width, width, n, kind, h->stream);
      }
      if (e == cudaSuccess) e = cudaEventRecord(h->hstage_ev[b], h->stream);
    }
    return e;
  }
  const char *s = static_cast<const char *>(src);
  char *d = static_cast<char *>(dst);
  auto issue = [&](size_t k) {
    const int b = (int)(k & 1);
    const size_t n = rows(k);
    cudaError_t r = flat ? cudaMemcpyAsync(h->hstage[b], s + k * lpc, n, kind, h->stream)
                         : cudaMemcpy2DAsync(h->hstage[b], width, s + k * lpc * spitch, spitch, width, n, kind,
                                             h->stream);
    return r == cudaSuccess ? cudaEventRecord(h->hstage_ev[b], h->stream) : r;
  };
  e = issue(0);
  for (size_t k = 0; k < nchunk && e == cudaSuccess; ++k) {
    if (k + 1 < nchunk) e = issue(k + 1);  // into the buffer unpacked at step k - 1
    if (e == cudaSuccess) e = cudaEventSynchronize(h->hstage_ev[k & 1]);
    if (e != cudaSuccess) break;
    const size_t n = rows(k);
    if (flat) par_copy(d + k * lpc, n, h->hstage[k & 1], n, n, 1);
    else par_copy(d + k * lpc * dpitch, dpitch, h->hstage[k & 1], width, width, n);
  }
  return e;
}

void release_host_staging(uvatrmm_handle_t h) {
  for (int b = 0; b < 2; ++b) {
    if (h->hstage_ev[b]) {
      cudaEventSynchronize(h->hstage_ev[b]);
      cudaEventDestroy(h->hstage_ev[b]);
      h->hstage_ev[b] = nullptr;
    }
    if (h->hstage[b]) {
      uvatrmm_host_free(h->hstage[b]);
      h->hstage[b] = nullptr;
    }
  }
  h->hstage_cap = 0;
}

}  // namespace uvt

using namespace uvt;

extern "C" {

UVATRMM_API int uvatrmm_host_alloc(size_t bytes, void **ptr) {
  if (!ptr) return fail(UVATRMM_EINVAL, "ptr is NULL");
  *ptr = nullptr;
  size_t len = 0;
  const int rc = map_region(bytes, ptr, &len);
  return rc == UVATRMM_OK ? ok() : rc;
}

UVATRMM_API int uvatrmm_host_free(void *ptr) {
  if (!ptr) return ok();
  size_t len = 0;
  {
    std::lock_guard<std::mutex> g(g_host_mu);
    auto it = g_host_maps.find(ptr);
    if (it == g_host_maps.end()) return fail(UVATRMM_EINVAL, "pointer was not returned by uvatrmm_host_alloc");
    len = it->second;
    g_host_maps.erase(it);
  }
  cudaError_t e = cudaHostUnregister(ptr);
  munmap(ptr, len);
  return e == cudaSuccess ? ok() : cuda_fail(e, "cudaHostUnregister");
}

}  // extern "C"
