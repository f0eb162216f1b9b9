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
#include <cstring>

#include "copy_pool.h"

namespace cpsz {

namespace {

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

// dst[0, n) = src[0, n), by the calling thread and the copy threads.
void parallel_copy(void* dst, const void* src, size_t n) {
  constexpr size_t P = (size_t)256 << 10;
  if (n < 2 * P || !CopyPool::get().parallel()) {
    memcpy(dst, src, n);
    return;
  }
  CopyPool& pool = CopyPool::get();
  auto work = [&](int k) { stream_copy((char*)dst + k * P, (const char*)src + k * P, std::min(P, n - k * P)); };
  CopyPool::Job job(pool, work);
  job.open((int)((n + P - 1) / P));
  job.help();
}

// copies at least this large from or to pageable memory go through the ring
constexpr size_t kStageMin = (size_t)1 << 20;
// page-locked pieces of an image at least this large go up by themselves
// instead of through its staging
constexpr size_t kDirectMin = (size_t)256 << 10;

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

int transfer_reserve(cpsz_b200_ctx* ctx, const void* host, size_t n) {
  return n >= kStageMin && host_kind(host) == HOST_PAGEABLE ? stage_reserve(ctx) : CPSZ_OK;
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
  static_assert(cpsz_b200_ctx::kStageSlots <= CopyPool::kWindow, "a slot's piece is waited for before its next one");
  char* ring = (char*)ctx->stage;
  const int pieces = (int)((n + C - 1) / C), pos = ctx->stage_pos;
  ctx->stage_pos = (pos + pieces) % S;
  auto slot = [&](int k) { return (pos + k) % S; };
  auto bytes = [&](int k) { return std::min(C, n - (size_t)k * C); };
  auto work = [&](int k) { stream_copy(ring + slot(k) * W, (const char*)src + (size_t)k * C, bytes(k)); };
  // piece k's slot is free once its last transfer is done: that of piece k - S
  // here, or of an earlier call's (its event may still be pending)
  if (pool.parallel()) {
    CopyPool::Job job(pool, work);
    int opened = 0;
    for (int k = 0; k < pieces; k++) {
      int free = opened;
      while (free < pieces && free < k + S) {
        const cudaError_t e = cudaEventQuery(ctx->stage_ev[slot(free)]);
        if (e == cudaErrorNotReady) {
          if (free > k) break;  // enough to go on with
          CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(free)]));
        } else {
          CPSZ_CUDA_TRY(e);
        }
        if (++free == opened + 4) job.open(opened = free);  // copied while the other slots are looked at
      }
      job.open(opened = free);
      job.wait(k);
      CPSZ_CUDA_TRY(cudaMemcpyAsync((char*)dst + (size_t)k * C, ring + slot(k) * W, bytes(k), cudaMemcpyHostToDevice,
                                    st));
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->stage_ev[slot(k)], st));
    }
    return CPSZ_OK;
  }
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
  static_assert(cpsz_b200_ctx::kStageSlots <= CopyPool::kWindow, "a slot's piece is waited for before its next one");
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
  if (pool.parallel()) {
    CopyPool::Job job(pool, work);
    job.arm();
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->stage_arm, st));
    for (int k = 0; k < pieces && k < ahead; k++) CPSZ_TRY(issue(k));
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_arm));  // the kernels before the copy are done
    job.arm();  // (again: those that had nothing to do for a millisecond sleep)
    for (int k = 0; k < pieces; k++) {
      CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->stage_ev[slot(k)]));
      job.open(k + 1);
      const int q = k + ahead;
      if (q < pieces) {
        if (q >= S) job.wait(q - S);
        CPSZ_TRY(issue(q));
      }
    }
    job.help();
    return CPSZ_OK;
  }
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
  size_t from = 0, to = 0;  // staged and not yet sent
  auto flush = [&]() -> int {
    if (to > from) CPSZ_CUDA_TRY(cudaMemcpyAsync(dst + from, h + from, to - from, cudaMemcpyHostToDevice, st));
    from = to;
    return CPSZ_OK;
  };
  for (const Piece& p : pieces_) {
    if (p.n >= kDirectMin && host_kind(p.src) == HOST_PINNED) {
      CPSZ_TRY(flush());
      CPSZ_CUDA_TRY(cudaMemcpyAsync(dst + p.at, p.src, p.n, cudaMemcpyHostToDevice, st));
      if (p.pad) CPSZ_CUDA_TRY(cudaMemsetAsync(dst + p.at + p.n, 0, p.pad, st));
      from = to = p.at + p.n + p.pad;
      continue;
    }
    parallel_copy(h + p.at, p.src, p.n);
    memset(h + p.at + p.n, 0, p.pad);
    to = p.at + p.n + p.pad;
  }
  return flush();
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
