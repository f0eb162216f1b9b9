// transfer.cpp -- host <-> device copies of bulk data (transfer.h).
//
// The CUDA driver copies pageable host memory through its own staging, one
// host thread at a time: 86 MB go up in 8.1 ms (10.6 GB/s), where the DMA from
// page-locked memory takes 1.63 (55 GB/s).  Callers hand the library ordinary
// arrays and byte strings, so bulk pageable copies go through a pinned ring of
// the context: pool threads copy 2 MB pieces into (or out of) ring slots and
// the DMA engine moves each slot as soon as it is filled, 2.0 ms for the same
// 86 MB.  The pieces are stored past the caches (streaming stores): an ordinary
// memcpy first reads every line it is about to overwrite, and the ring's lines
// would push the source out of the caches; with it the pipeline takes 2.8 ms,
// and 16 MB slots, each copied whole before its DMA starts, took 4.0.
#include "transfer.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace cpsz {

namespace {

inline void relax() {
#ifdef __SSE2__
  _mm_pause();
#endif
}

// memcpy with streaming stores (complete when it returns).
void stream_copy(char* d, const char* s, size_t n) {
#ifdef __SSE2__
  const size_t head = std::min(n, (size_t)(-(uintptr_t)d & 15));
  memcpy(d, s, head);
  size_t i = head;
  for (; i + 64 <= n; i += 64) {
    const __m128i a = _mm_loadu_si128((const __m128i*)(s + i)), b = _mm_loadu_si128((const __m128i*)(s + i + 16)),
                  c = _mm_loadu_si128((const __m128i*)(s + i + 32)), e = _mm_loadu_si128((const __m128i*)(s + i + 48));
    _mm_stream_si128((__m128i*)(d + i), a);
    _mm_stream_si128((__m128i*)(d + i + 16), b);
    _mm_stream_si128((__m128i*)(d + i + 32), c);
    _mm_stream_si128((__m128i*)(d + i + 48), e);
  }
  memcpy(d + i, s + i, n - i);
  _mm_sfence();
#else
  memcpy(d, s, n);
#endif
}

// Process-wide copy threads.  One job at a time (contexts on several threads
// take turns): run(pieces, work, drive) has the workers take pieces 0, 1, ...
// and call work(k) for each once `open` exceeds k, while the calling thread
// runs drive(open, done), which opens pieces and waits for done[k].
class CopyPool {
 public:
  static CopyPool& get() {
    static CopyPool p;
    return p;
  }
  bool parallel() const { return !workers_.empty(); }

  template <class Work, class Drive>
  int run(int pieces, const Work& work, const Drive& drive) {
    std::lock_guard<std::mutex> turn(turn_);
    std::vector<std::atomic<int>> done(pieces);
    for (auto& d : done) d.store(0, std::memory_order_relaxed);
    std::atomic<int> open{0}, next{0};
    std::atomic<bool> stop{false};
    auto body = [&] {
      for (int k; (k = next.fetch_add(1)) < pieces;) {
        while (open.load(std::memory_order_acquire) <= k) {
          if (stop.load(std::memory_order_relaxed)) return;
          relax();
        }
        work(k);
        done[k].store(1, std::memory_order_release);
      }
    };
    const std::function<void()> f = body;
    {
      std::lock_guard<std::mutex> lk(m_);
      f_ = &f;
      active_ = (int)workers_.size();
      gen_++;
    }
    cv_.notify_all();
    const int rc = drive(open, done);
    if (rc != CPSZ_OK) stop.store(true);  // pieces that were never opened
    std::unique_lock<std::mutex> lk(m_);
    done_.wait(lk, [&] { return active_ == 0; });
    f_ = nullptr;
    return rc;
  }

  void copy(void* dst, const void* src, size_t n) {
    constexpr size_t P = (size_t)256 << 10;
    if (n < 2 * P || !parallel()) {
      memcpy(dst, src, n);
      return;
    }
    const int pieces = (int)((n + P - 1) / P);
    run(
        pieces,
        [&](int k) { stream_copy((char*)dst + k * P, (const char*)src + k * P, std::min(P, n - k * P)); },
        [&](std::atomic<int>& open, std::vector<std::atomic<int>>&) {
          open.store(pieces, std::memory_order_release);
          return CPSZ_OK;
        });
  }

 private:
  CopyPool() {
    const unsigned hw = std::thread::hardware_concurrency();
    const int nw = (int)std::min(8u, hw > 1 ? hw - 1 : 0u);
    for (int w = 0; w < nw; w++) workers_.emplace_back([this] { loop(); });
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(m_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : workers_) t.join();
  }
  void loop() {
    unsigned long long seen = 0;
    for (;;) {
      const std::function<void()>* f;
      {
        std::unique_lock<std::mutex> lk(m_);
        cv_.wait(lk, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
        f = f_;
      }
      (*f)();
      std::lock_guard<std::mutex> lk(m_);
      if (--active_ == 0) done_.notify_one();
    }
  }
  std::vector<std::thread> workers_;
  std::mutex turn_, m_;
  std::condition_variable cv_, done_;
  const std::function<void()>* f_ = nullptr;
  int active_ = 0;
  unsigned long long gen_ = 0;
  bool stop_ = false;
};

// copies at least this large from or to pageable memory go through the ring
constexpr size_t kStageMin = (size_t)1 << 20;

int stage_reserve(cpsz_b200_ctx* ctx) {
  if (ctx->stage) return CPSZ_OK;
  cudaError_t e = cudaMallocHost(&ctx->stage, (size_t)cpsz_b200_ctx::kStageSlots * cpsz_b200_ctx::kStageBytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    ctx->stage = nullptr;
    return set_error(CPSZ_ERR_NOMEM, "pinned transfer ring: %s", cudaGetErrorString(e));
  }
  return CPSZ_OK;
}

// Bytes of a ring piece of a copy of n: a slot, or less so that a smaller copy
// still has a piece for every worker and a first transfer that starts soon.
size_t piece_bytes(size_t n) {
  const size_t step = (size_t)64 << 10, least = (size_t)256 << 10;
  return std::min(cpsz_b200_ctx::kStageBytes, std::max(least, align_up(n / 16, step)));
}

inline void wait_for(const std::atomic<int>& d) {
  while (!d.load(std::memory_order_acquire)) relax();
}

}  // namespace

HostKind host_kind(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return HOST_PAGEABLE;
  }
  if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) return HOST_DEVICE;
  if (a.type == cudaMemoryTypeHost) return HOST_PINNED;
  return HOST_PAGEABLE;
}

int h2d(cpsz_b200_ctx* ctx, void* dst, const void* src, size_t n, cudaStream_t st) {
  if (!n) return CPSZ_OK;
  const HostKind k = host_kind(src);
  if (k != HOST_PAGEABLE || n < kStageMin) {
    CPSZ_CUDA_TRY(cudaMemcpyAsync(dst, src, n, k == HOST_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                                  st));
    return CPSZ_OK;
  }
  CPSZ_TRY(stage_reserve(ctx));
  CopyPool& pool = CopyPool::get();
  const size_t C = piece_bytes(n), W = cpsz_b200_ctx::kStageBytes;
  const int S = cpsz_b200_ctx::kStageSlots;
  char* ring = (char*)ctx->stage;
  const int pieces = (int)((n + C - 1) / C), pos = ctx->stage_pos;
  ctx->stage_pos = (pos + pieces) % S;
  auto slot = [&](int k) { return (pos + k) % S; };
  auto bytes = [&](int k) { return std::min(C, n - (size_t)k * C); };
  auto work = [&](int k) { stream_copy(ring + slot(k) * W, (const char*)src + (size_t)k * C, bytes(k)); };
  // piece k's slot is free once its last transfer is done: that of piece k - S
  // here, or of an earlier call's (its event may still be pending)
  auto drive = [&](std::atomic<int>& open, std::vector<std::atomic<int>>& done) -> int {
    int opened = 0;
    for (int k = 0; k < pieces; k++) {
      while (opened < pieces && opened < k + S) {
        const cudaError_t e = cudaEventQuery(ctx->stage_ev[slot(opened)]);
        if (e == cudaErrorNotReady) {
          if (opened > k) break;  // enough to go on with
          CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(opened)]));
        } else {
          CPSZ_CUDA_TRY(e);
        }
        open.store(++opened, std::memory_order_release);
      }
      wait_for(done[k]);
      CPSZ_CUDA_TRY(cudaMemcpyAsync((char*)dst + (size_t)k * C, ring + slot(k) * W, bytes(k), cudaMemcpyHostToDevice,
                                    st));
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->stage_ev[slot(k)], st));
    }
    return CPSZ_OK;
  };
  if (pool.parallel()) return pool.run(pieces, work, drive);
  for (int k = 0; k < pieces; k++) {
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(k)]));
    work(k);
    CPSZ_CUDA_TRY(cudaMemcpyAsync((char*)dst + (size_t)k * C, ring + slot(k) * W, bytes(k), cudaMemcpyHostToDevice, st));
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->stage_ev[slot(k)], st));
  }
  return CPSZ_OK;
}

int d2h(cpsz_b200_ctx* ctx, void* dst, const void* src, size_t n, cudaStream_t st) {
  if (!n) return CPSZ_OK;
  const HostKind k = host_kind(dst);
  if (k != HOST_PAGEABLE || n < kStageMin) {
    CPSZ_CUDA_TRY(cudaMemcpyAsync(dst, src, n, k == HOST_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                  st));
    return CPSZ_OK;
  }
  CPSZ_TRY(stage_reserve(ctx));
  CopyPool& pool = CopyPool::get();
  const size_t C = piece_bytes(n), W = cpsz_b200_ctx::kStageBytes;
  const int S = cpsz_b200_ctx::kStageSlots;
  char* ring = (char*)ctx->stage;
  const int pieces = (int)((n + C - 1) / C), pos = ctx->stage_pos;
  ctx->stage_pos = (pos + pieces) % S;
  auto slot = [&](int k) { return (pos + k) % S; };
  auto bytes = [&](int k) { return std::min(C, n - (size_t)k * C); };
  auto work = [&](int k) { stream_copy((char*)dst + (size_t)k * C, ring + slot(k) * W, bytes(k)); };
  auto issue = [&](int k) -> int {
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(k)]));  // no other transfer still uses the slot
    CPSZ_CUDA_TRY(cudaMemcpyAsync(ring + slot(k) * W, (const char*)src + (size_t)k * C, bytes(k),
                                  cudaMemcpyDeviceToHost, st));
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->stage_ev[slot(k)], st));
    return CPSZ_OK;
  };
  const int ahead = S / 2;  // transfers in flight; the other slots are being copied out
  auto drive = [&](std::atomic<int>& open, std::vector<std::atomic<int>>& done) -> int {
    for (int k = 0; k < pieces && k < ahead; k++) CPSZ_TRY(issue(k));
    for (int k = 0; k < pieces; k++) {
      CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(k)]));
      open.store(k + 1, std::memory_order_release);
      const int q = k + ahead;
      if (q < pieces) {
        if (q >= S) wait_for(done[q - S]);
        CPSZ_TRY(issue(q));
      }
    }
    return CPSZ_OK;
  };
  if (pool.parallel()) return pool.run(pieces, work, drive);
  for (int k = 0; k < pieces; k++) {
    CPSZ_TRY(issue(k));
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(k)]));
    work(k);
  }
  return CPSZ_OK;
}

int Upload::send_whole(cpsz_b200_ctx* ctx, uint8_t* dst, cudaStream_t st) const {
  if (!bytes_) return CPSZ_OK;
  CPSZ_TRY(upload_reserve(ctx, bytes_));
  char* h = (char*)ctx->up_pinned;
  for (const Piece& p : pieces_) {
    CopyPool::get().copy(h + p.at, p.src, p.n);
    memset(h + p.at + p.n, 0, p.pad);
  }
  CPSZ_CUDA_TRY(cudaMemcpyAsync(dst, h, bytes_, cudaMemcpyHostToDevice, st));
  return CPSZ_OK;
}

int Upload::send_part(cpsz_b200_ctx* ctx, uint8_t* dst, int part, cudaStream_t st) const {
  for (const Piece& p : pieces_) {
    if (p.part != part) continue;
    if (p.pad) CPSZ_CUDA_TRY(cudaMemsetAsync(dst + p.at + p.n, 0, p.pad, st));
    CPSZ_TRY(h2d(ctx, dst + p.at, p.src, p.n, st));
  }
  return CPSZ_OK;
}

}  // namespace cpsz
