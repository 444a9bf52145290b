// staging.cu -- host <-> device transfers of large user arrays.
//
// The C ABI takes ordinary (pageable) host arrays.  Large ones are copied by
// several host threads into the context's pinned staging buffer (kept between
// calls, grown on demand) in chunks, each moved by its own DMA as soon as it is
// filled (downloads the same way in reverse, through a few chunks of it), instead
// of the driver's single-threaded pageable path; connectivity is narrowed to int32 and
// coefficients are checked on the way.  Small arrays go directly.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

#include "objects.hpp"

namespace tptfem {

namespace {

constexpr size_t STAGE_MIN_BYTES = 1u << 20;  // below this the direct copy is as fast
constexpr size_t STAGE_CHUNK = 8u << 20;      // pipelined transfers move chunks of this size
// Chunks of a download in flight.  to_csr with 3.8M entries (46 MB), the first of a
// context and later ones: a slot for every chunk 20-27 and 2.4 ms, three slots 17-20 and
// 2.5 (of 4 MB 12 and 2.7, of 2 MB 8 and 3.6: the threads' slices get short), pageable
// copies 22 and 18.  With 99.8M entries: 530-1000 and 58 ms (1.2 GB of pinned memory),
// 80-110 and 54, 570 and 484.
constexpr size_t STAGE_RING = 3;

unsigned stage_threads(size_t bytes) {
  const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
  return (unsigned)std::max<size_t>(1, std::min<size_t>(std::min(16u, hw), bytes / (1u << 18)));
}

// The pinned buffer, of at least `bytes`.
void* stage(tptfem_context* ctx, size_t bytes) {
  if (ctx->h_stage_bytes < bytes) {
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    ctx->h_stage = nullptr;
    ctx->h_stage_bytes = 0;
    TPT_CUDA(cudaHostAlloc(&ctx->h_stage, bytes, cudaHostAllocDefault));
    ctx->h_stage_bytes = bytes;
  }
  return ctx->h_stage;
}

// The same, null where there is none to be had.
void* try_stage(tptfem_context* ctx, size_t bytes) {
  try {
    return stage(ctx, bytes);
  } catch (const Error&) {
    ctx->h_stage = nullptr;  // (what a failed call leaves is not defined)
    cudaGetLastError();
    return nullptr;
  }
}

// Host -> device through the pinned buffer, pipelined: n staged elements of
// `elem` bytes in chunks; host thread t fills its slice of every chunk in turn
// (fill(i0, i1) writes staged elements [i0, i1) and returns false if the
// input there is invalid), and this thread issues each chunk's DMA as soon as
// every slice of it is in, so the copies overlap the host work on the next
// chunks.  Returns false if any fill did.
template <typename Fill>
bool staged_in(tptfem_context* ctx, void* dst, size_t n, size_t elem, Fill fill) {
  const size_t bytes = n * elem;
  char* p = static_cast<char*>(stage(ctx, bytes));
  const size_t cel = std::max<size_t>(1, STAGE_CHUNK / elem), nchunk = (n + cel - 1) / cel;
  const unsigned nt = stage_threads(bytes);
  std::vector<std::atomic<unsigned>> done(nchunk);
  for (auto& d : done) d.store(0);
  std::atomic<bool> ok(true);
  auto work = [&](unsigned t) {
    for (size_t c = 0; c < nchunk; ++c) {
      const size_t c0 = c * cel, c1 = std::min(n, c0 + cel), len = c1 - c0;
      const size_t b = c0 + len * t / nt, e = c0 + len * (t + 1) / nt;
      if (b < e && !fill(b, e)) ok = false;
      done[c].fetch_add(1, std::memory_order_release);
    }
  };
  std::vector<std::thread> th;
  for (unsigned t = 1; t < nt; ++t) th.emplace_back(work, t);
  // this thread fills slice 0 of each chunk, then issues the chunk once all
  // slices are in (a copy error is raised only after the workers have finished)
  cudaError_t err = cudaSuccess;
  for (size_t c = 0; c < nchunk; ++c) {
    const size_t c0 = c * cel, c1 = std::min(n, c0 + cel), len = c1 - c0;
    const size_t e = c0 + len / nt;
    if (c0 < e && !fill(c0, e)) ok = false;
    done[c].fetch_add(1, std::memory_order_release);
    while (done[c].load(std::memory_order_acquire) < nt) std::this_thread::yield();
    if (err == cudaSuccess)
      err = cudaMemcpyAsync(static_cast<char*>(dst) + c0 * elem, p + c0 * elem, len * elem, cudaMemcpyHostToDevice,
                            ctx->stream);
  }
  for (auto& x : th) x.join();
  TPT_CUDA(err);
  TPT_CUDA(cudaStreamSynchronize(ctx->stream));  // the staging buffer is reused by the next call
  return ok;
}

}  // namespace

void host_to_device(tptfem_context* ctx, void* dst, const void* src, size_t bytes) {
  if (!bytes) return;
  if (bytes < STAGE_MIN_BYTES) {
    TPT_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return;
  }
  char* p = static_cast<char*>(stage(ctx, bytes));
  const char* s = static_cast<const char*>(src);
  staged_in(ctx, dst, bytes, 1, [&](size_t b, size_t e) {
    std::memcpy(p + b, s + b, e - b);
    return true;
  });
}

// Device -> host through the pinned buffer, pipelined: chunk k's DMA is followed by
// an event; host thread t copies its slice of each chunk out once that chunk's event
// has completed (int32 indices widened to int64 on the way), while the next chunks
// are still moving.  The chunks go round a ring of STAGE_RING slots, so the pinned
// memory stays small whatever is downloaded: chunk k is issued when every thread has
// copied chunk k - STAGE_RING out.  All arrays of a call share one pipeline and one
// team of threads.  Small arrays, and all where no pinned memory is to be had, go as
// pageable copies with a widening loop.
void device_to_host(tptfem_context* ctx, const HostCopy* copies, int ncopies) {
  struct Chunk {
    const HostCopy* c;
    size_t first, count;  // elements of the array
  };
  size_t bytes = 0, slot = 0;  // of all arrays, of a ring slot
  std::vector<Chunk> chunks;
  for (int k = 0; k < ncopies; ++k) {
    const HostCopy& c = copies[k];
    const size_t cel = STAGE_CHUNK / c.elem;
    for (size_t i = 0; i < c.count; i += cel) {
      chunks.push_back({&c, i, std::min(cel, c.count - i)});
      slot = std::max(slot, chunks.back().count * c.elem);
    }
    bytes += c.count * c.elem;
  }
  if (!bytes) return;
  slot = (slot + 255) & ~(size_t)255;
  const size_t n = chunks.size(), ring = std::min(n, STAGE_RING);
  char* p = bytes < STAGE_MIN_BYTES ? nullptr : static_cast<char*>(try_stage(ctx, ring * slot));
  if (!p) {
    std::vector<int> narrow;
    for (int k = 0; k < ncopies; ++k) {
      const HostCopy& c = copies[k];
      if (!c.count) continue;
      if (c.widen) narrow.resize(c.count);
      TPT_CUDA(cudaMemcpyAsync(c.widen ? narrow.data() : c.dst, c.src, c.count * c.elem, cudaMemcpyDeviceToHost,
                               ctx->stream));
      TPT_CUDA(cudaStreamSynchronize(ctx->stream));
      if (c.widen) std::copy(narrow.begin(), narrow.end(), static_cast<int64_t*>(c.dst));
    }
    return;
  }
  const unsigned nt = stage_threads(bytes);
  std::vector<cudaEvent_t> ev(ring, nullptr);
  std::vector<std::atomic<unsigned>> out(n);  // slices of a chunk that have been copied out
  for (auto& o : out) o.store(0);
  std::atomic<size_t> issued(0);
  std::atomic<bool> failed(false);
  cudaError_t err = cudaSuccess;
  auto issue = [&](size_t k) {
    const Chunk& c = chunks[k];
    cudaEvent_t& e = ev[k % ring];
    if (!e) err = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (err == cudaSuccess)
      err = cudaMemcpyAsync(p + k % ring * slot, static_cast<const char*>(c.c->src) + c.first * c.c->elem,
                            c.count * c.c->elem, cudaMemcpyDeviceToHost, ctx->stream);
    if (err == cudaSuccess) err = cudaEventRecord(e, ctx->stream);
    if (err == cudaSuccess) issued.store(k + 1, std::memory_order_release);
    else failed = true;
  };
  auto copy_out = [&](size_t k, unsigned t) {
    const Chunk& c = chunks[k];
    const char* from = p + k % ring * slot;
    const size_t b = c.count * t / nt, e = c.count * (t + 1) / nt;
    if (c.c->widen) {
      const int* v = reinterpret_cast<const int*>(from);
      int64_t* to = static_cast<int64_t*>(c.c->dst) + c.first;
      for (size_t i = b; i < e; ++i) to[i] = v[i];
    } else {
      std::memcpy(static_cast<char*>(c.c->dst) + (c.first + b) * c.c->elem, from + b * c.c->elem, (e - b) * c.c->elem);
    }
    out[k].fetch_add(1, std::memory_order_release);
  };
  auto work = [&](unsigned t) {
    for (size_t k = 0; k < n; ++k) {
      while (issued.load(std::memory_order_acquire) <= k) {
        if (failed) return;
        std::this_thread::yield();
      }
      if (cudaEventSynchronize(ev[k % ring]) != cudaSuccess) { failed = true; return; }
      copy_out(k, t);
    }
  };
  size_t next = 0;
  while (next < ring && !failed) issue(next++);  // (before there are threads that wait on events)
  std::vector<std::thread> th;
  th.reserve(nt);
  try {
    for (unsigned t = 1; t < nt; ++t) th.emplace_back(work, t);
  } catch (const std::system_error&) {  // no more threads: this one copies the slices that are left
  }
  const unsigned alone = 1 + (unsigned)th.size();
  for (size_t k = 0; k < n && !failed; ++k) {
    // every chunk whose slot is free goes out; chunk k itself is waited for
    while (next < n && next < k + ring && !failed) {
      if (out[next - ring].load(std::memory_order_acquire) < nt) {
        if (next > k) break;
        std::this_thread::yield();
        continue;
      }
      issue(next++);
    }
    if (failed) break;
    if (cudaEventSynchronize(ev[k % ring]) != cudaSuccess) { failed = true; break; }
    copy_out(k, 0);
    for (unsigned t = alone; t < nt; ++t) copy_out(k, t);
  }
  for (auto& x : th) x.join();
  if (failed) cudaStreamSynchronize(ctx->stream);  // nothing moves into the buffer any more
  for (auto e : ev)
    if (e) cudaEventDestroy(e);
  TPT_CUDA(err);
  TPT_REQUIRE(!failed, TPTFEM_ERR_DEVICE, "device-to-host copy failed");
}

void device_to_host(tptfem_context* ctx, void* dst, const void* src, size_t bytes) {
  const HostCopy c{dst, src, bytes, 1, false};
  device_to_host(ctx, &c, 1);
}

bool host_to_device_ids(tptfem_context* ctx, int* dst, const int64_t* src, size_t count, int64_t limit) {
  if (!count) return true;
  int* p = static_cast<int*>(stage(ctx, count * sizeof(int)));
  return staged_in(ctx, dst, count, sizeof(int), [&](size_t b, size_t e) {
    bool good = true;
    for (size_t i = b; i < e; ++i) {
      const int64_t v = src[i];
      good &= v >= 0 && v < limit;
      p[i] = (int)v;
    }
    return good;
  });
}

bool host_to_device_finite(tptfem_context* ctx, double* dst, const double* src, size_t count) {
  if (!count) return true;
  double* p = static_cast<double*>(stage(ctx, count * sizeof(double)));
  return staged_in(ctx, dst, count, sizeof(double), [&](size_t b, size_t e) {
    bool good = true;
    for (size_t i = b; i < e; ++i) {
      good &= std::isfinite(src[i]);
      p[i] = src[i];
    }
    return good;
  });
}

}  // namespace tptfem
