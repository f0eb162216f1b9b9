// pack_group.h -- the host side of packing once the code trees are known:
// uploads built in page-locked staging, and streams packed in one launch.
#pragma once

#include <algorithm>
#include <cstring>
#include <vector>

#include "huffman_host.h"
#include "kernels.h"

namespace cpsz {

// An upload built piece by piece in page-locked staging, each piece at the
// place it has on the device, and sent in one copy (send may be called again
// after further pieces).
struct UpImage {
  uint8_t* h = nullptr;
  uint8_t* d = nullptr;
  size_t cap = 0, at = 0, sent = 0;
  // room for n bytes; the device address in *dev (null: no room)
  uint8_t* take(size_t n, uint8_t** dev) {
    const size_t o = align_up(at, 16);
    if (o + n > cap) return nullptr;
    at = o + n;
    *dev = d + o;
    return h + o;
  }
  int send(cudaStream_t st) {
    if (at > sent) CPSZ_CUDA_TRY(cudaMemcpyAsync(d + sent, h + sent, at - sent, cudaMemcpyHostToDevice, st));
    sent = at = align_up(at, 256);
    return CPSZ_OK;
  }
};
inline int up_overrun() { return set_error(CPSZ_ERR_INVALID, "internal: upload staging overrun"); }

// Streams packed together (at most three per field of a pass).
struct PackGroup {
  std::vector<PackPrep> prep;
  std::vector<PackJob> jobs;
  std::vector<const HuffCodebook*> cbs;
  PackPrep* d_prep = nullptr;
  PackJob* d_jobs = nullptr;
  size_t max_entries = 0, max_zero = 0;
  unsigned ctas = 0;

  // A stream of n symbols with codebook cb, `bytes` bytes of bits to dst
  // (device, any alignment, `room` bytes from there on); code / len: device
  // tables of the symbols' range; scratch: huff_encode_tmp_bytes(n), zeroed.
  void add(const HuffCodebook& cb, const void* sym, int sym_bytes, bool map_id_zero, size_t n, uint8_t* dst,
           size_t bytes, size_t room, unsigned long long* code, uint8_t* len, unsigned long long* scratch) {
    const size_t mis = (uintptr_t)dst & 3;
    PackPrep r;
    r.n = cb.entries.size();
    r.code = code;
    r.len = len;
    r.zero = dst;
    r.zero_bytes = bytes;
    PackJob p;
    p.sym = sym;
    p.sym_bytes = sym_bytes;
    p.map_id_zero = map_id_zero ? 1 : 0;
    p.n = n;
    p.tab = HuffEncTable{code, len, sym_bytes == 2 ? 65536 : 256};
    p.out = (uint32_t*)(dst - mis);
    p.cap_words = (room + mis) / 4;
    p.scratch = scratch;
    p.bit0 = (int)(8 * mis);
    prep.push_back(r);
    jobs.push_back(p);
    cbs.push_back(&cb);
  }
  size_t up_bytes() const {
    size_t b = align_up(jobs.size() * sizeof(PackPrep), 16) + align_up(jobs.size() * sizeof(PackJob), 16) + 64;
    for (const HuffCodebook* cb : cbs) b += align_up(cb->entries.size() * sizeof(HuffEntry), 16) + 16;
    return b;
  }
  // The jobs and entries into `up` (not sent).
  int stage(UpImage& up, int num_sms) {
    const size_t n = jobs.size();
    ctas = pack_assign_ctas(num_sms, jobs.data(), (int)n);
    uint8_t *dp, *dj, *de;
    uint8_t* hp = up.take(n * sizeof(PackPrep), &dp);
    if (!hp) return up_overrun();
    uint8_t* hj = up.take(n * sizeof(PackJob), &dj);
    if (!hj) return up_overrun();
    for (size_t q = 0; q < n; q++) {
      const std::vector<HuffEntry>& e = cbs[q]->entries;
      uint8_t* he = up.take(e.size() * sizeof(HuffEntry), &de);
      if (!he) return up_overrun();
      memcpy(he, e.data(), e.size() * sizeof(HuffEntry));
      prep[q].entries = (const HuffEntry*)de;
      max_entries = std::max(max_entries, prep[q].n);
      max_zero = std::max(max_zero, prep[q].zero_bytes);
    }
    memcpy(hp, prep.data(), n * sizeof(PackPrep));
    memcpy(hj, jobs.data(), n * sizeof(PackJob));
    d_prep = (PackPrep*)dp;
    d_jobs = (PackJob*)dj;
    return CPSZ_OK;
  }
  int launch(cpsz_b200_ctx* ctx) const {
    CPSZ_TRY(launch_pack_prep(ctx, d_prep, (int)jobs.size(), max_entries, max_zero));
    CPSZ_TRY(launch_pack(ctx->stream, jobs.data(), d_jobs, (int)jobs.size(), ctas, ctx->d_flag));
    count_launch(ctx);
    return CPSZ_OK;
  }
};

}  // namespace cpsz
