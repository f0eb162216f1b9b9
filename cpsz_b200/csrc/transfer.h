// transfer.h -- host <-> device copies of bulk data.
//
// Device and page-locked host memory are copied directly (enqueued on `st`).
// Pageable host memory of 1 MiB or more moves through the context's pinned
// ring (kStageSlots slots of kStageBytes) with the host copies spread over a
// small thread pool (copy_pool.h), piece by piece, the pieces' DMA overlapping
// the others' host copies.  Transfers of several contexts share the pool's
// threads and wait for one another nowhere.  For pageable memory both calls return once the host
// side is complete: after h2d the source may be reused, after d2h the
// destination holds the data.  Device-side ordering is that of `st`.
#pragma once

#include <vector>

#include "runtime.h"

namespace cpsz {

enum HostKind { HOST_PAGEABLE = 0, HOST_PINNED = 1, HOST_DEVICE = 2 };
HostKind host_kind(const void* p);

int h2d(cpsz_b200_ctx* ctx, void* dst, const void* src, size_t n, cudaStream_t st);
int d2h(cpsz_b200_ctx* ctx, void* dst, const void* src, size_t n, cudaStream_t st);
// Whatever a copy of n bytes between the device and `host` allocates the first
// time (the ring: 64 MB, some 25 ms), before work that must not wait for it.
int transfer_reserve(cpsz_b200_ctx* ctx, const void* host, size_t n);

// Several host pieces that go up to one device buffer: add() places a piece
// (256-byte aligned, `pad` zero bytes behind it) and returns its offset there;
// cut() ends a part.  Either the whole image goes up in one copy from the
// context's page-locked staging (send_whole: no other copy from it may be in
// flight; large pieces that are page-locked themselves go up from where they
// are, in their own copies, and are read until these have run), or part by
// part (send_part, h2d's rules).  Sources are read when they are sent.
class Upload {
 public:
  size_t add(const void* src, size_t n, size_t pad = 0) {
    const size_t at = align_up(bytes_, 256);
    pieces_.push_back(Piece{src, n, pad, at, part_});
    bytes_ = at + n + pad;
    return at;
  }
  void cut() { part_++; }
  size_t bytes() const { return bytes_; }
  int send_whole(cpsz_b200_ctx* ctx, uint8_t* dst, cudaStream_t st) const;
  int send_part(cpsz_b200_ctx* ctx, uint8_t* dst, int part, cudaStream_t st) const;

 private:
  struct Piece {
    const void* src;
    size_t n, pad, at;
    int part;
  };
  std::vector<Piece> pieces_;
  size_t bytes_ = 0;
  int part_ = 0;
};
// Images up to this size go up whole: one upload, one decoder launch for all
// streams and no gap between them; above it the staging copy takes longer than
// decoding a stream while the next one travels.  Whole against in parts, 2D
// decompression from a host blob: 3.1 MB 0.56 and 0.75 ms, 6.2 MB 0.80 and 0.95,
// 11.7 MB 1.15 and 1.26, 23.8 MB 1.86 and 1.82.
constexpr size_t UPLOAD_WHOLE = (size_t)12 << 20;

}  // namespace cpsz
