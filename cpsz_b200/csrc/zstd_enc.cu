// zstd_enc.cu -- the GPU lossless stage: Zstandard frames of device data.
//
// The reference applies ZSTD_compress(level 3) to every blob on the host
// (src/sz_lossless.cpp:11-26); here the same kind of frame is written on the
// GPU (format: zstd_format.h), readable by any Zstandard decoder and so by the
// reference's sz_lossless_decompress.  The input is cut into 8 KB blocks that
// are encoded independently, one warp each (16 warps an SM):
//   0. the warp stages its block in shared memory with 16-byte loads, so the
//      match loop below (a dependent chain: one step per match on the
//      Huffman bit streams of a blob, a match every few bytes) waits on
//      shared memory, not on global loads (32 KB blocks read from global
//      memory: 9.6 ms for a 89 MB blob; staged, with four warps an SM for
//      lack of shared memory: 17.7 ms);
//   1. greedy matching: the warp looks at 32 consecutive positions at a time,
//      each lane hashing the 4 bytes at its position into the warp's table of
//      last positions (shared memory, 2048 16-bit entries) and checking the
//      candidate; the first matching lane starts a match, which the warp
//      extends 32 bytes per step; positions before it enter the table.  With
//      no match the window advances 32 positions.  The literals (the bytes no
//      match covers) go to the block's slot as they are passed over;
//   2. the sequences, with the predefined FSE tables (every offset a real
//      offset, so blocks share no state), 32 at a time: the three state chains
//      on three lanes, the rest on all (code_sequences).
// An all-equal block becomes an RLE block, a block that does not shrink a raw
// block.  Block sizes are scanned and a gather kernel places the blocks after
// the frame header.  Matches stay inside their block.
//
// Bound: the two serial chains of the densest block: a match takes about 560
// cycles (three dependent rounds of shared loads, two votes, a shuffle and the
// instructions between them, one warp at a time), its coding 180.  Step 2 on one
// lane, with a global load and byte stores per sequence, and a second pass over
// the sequences for the literals took three times as long as both do now: a 9.1
// MB blob (2048 x 3001, eb 0.01; up to 1500 sequences in an 8 KB block) 1.58 ms,
// now 0.56.  Measured and not kept: match lengths up to 12 bytes on every lane
// (0.61 ms), the windows' bytes and hashes kept in registers (0.55 ms, and the
// table's updates then need two stores): fewer loads, but not fewer instructions.
#include <cstring>

#include "kernels.h"
#include "zstd_format.h"

namespace cpsz {

namespace {

constexpr int ZBLK = 8 * 1024;
constexpr int ZHT_BITS = 11;
constexpr int ZWARPS = 8;  // blocks per CTA
constexpr int ZMAXSEQ = ZBLK / zstd::kMinMatch + 1;
constexpr int ZSEQW = ZBLK / 4 + 8;         // words of a block's sequence stream that are kept (a longer one loses to raw)
constexpr int ZSLOT = ZBLK + 4 * ZSEQW;     // per-block slot: literals, then the sequence stream
constexpr unsigned FULLMASK = 0xffffffffu;

__constant__ zstd::Tables c_tables;

__device__ __forceinline__ uint32_t zhash(uint32_t v) { return (v * 2654435761u) >> (32 - ZHT_BITS); }

// Bytes of the literals section's header and of the sequences section's count and modes.
__device__ __forceinline__ int lit_header_bytes(int nlit) { return nlit < 32 ? 1 : nlit < 4096 ? 2 : 3; }
__device__ __forceinline__ int seq_header_bytes(int nseq) { return nseq < 128 ? 2 : 3; }

// A sequence as the matcher leaves it: literals (14 bits), match length (14), offset (14).
__device__ __forceinline__ unsigned long long seq_pack(unsigned lit, unsigned ml, unsigned off) {
  return (unsigned long long)lit | (unsigned long long)ml << 14 | (unsigned long long)off << 28;
}

// What the gather needs of a block: its bytes in the frame, type and literals.
struct ZBlock {
  unsigned size;   // header included
  unsigned type;   // 0 raw, 1 RLE, 2 compressed
  unsigned nlit;
};

// Work memory of the sequence coder (it takes the hash table's place).
struct ZCoder {
  uint8_t code[3][32];   // offset, match length, literals length codes of 32 sequences
  uint16_t fse[3][32];   // their state bits: value | count << 8
  uint32_t word[64 + 4]; // bits of 32 sequences (at most 62 each), from the last unstored word on
};
// Shared memory of one warp: its block's bytes and its hash table of
// block-local positions + 1 (0 = empty), whose place the coder takes over.
struct ZWarpSmem {
  uint32_t data[ZBLK / 4];
  union {
    uint16_t ht[1 << ZHT_BITS];
    ZCoder c;
  };
  __device__ __forceinline__ uint8_t byte(int i) const { return reinterpret_cast<const uint8_t*>(data)[i]; }
  // 4 bytes at any position (a word past the end is the hash table's: in place, its bytes not used)
  __device__ __forceinline__ uint32_t load4(int i) const {
    return __funnelshift_r(data[i >> 2], data[(i >> 2) + 1], 8 * (i & 3));
  }
};
// The format's tables in shared memory (lanes look up different entries, which
// constant memory would serve one by one): the FSE tables (offset, match
// length, literals length) and the codes and extra bits of lengths.
struct ZFse {
  uint16_t state[3][64];
  zstd::FseSym sym[3][64];
  uint8_t ll_code[64], ml_code[128], ll_bits[64], ml_bits[64];
};
constexpr size_t ZSMEM = sizeof(ZWarpSmem) * ZWARPS + sizeof(ZFse);

// The sequence stream of a block (zstd::write_sequences' bit stream) into
// `out` (words); returns its bytes, which may exceed what `out` holds (then
// only the first ZSEQW words are stored).  The stream is written from the
// last sequence to the first, 32 at a time:
//   1. a lane per sequence looks its three codes up;
//   2. the state chains, which are the stream's only serial part, run on
//      three lanes, one per table, and leave every sequence's state bits;
//   3. a lane per sequence puts its bits together (state bits and extra bits,
//      at most 62), a scan of their counts places them in a shared word
//      buffer, and whole words are stored.
__device__ __forceinline__ int code_sequences(const unsigned long long* __restrict__ seqs, int nseq, const ZFse& T,
                                              ZCoder& C, uint32_t* __restrict__ out, int lane) {
  unsigned state = 0;  // lanes 0-2: of, ml, ll
  int stored = 0;      // whole words stored
  unsigned fill = 0;   // bits in C.word from its first word on
  for (int k = lane; k < 64 + 4; k += 32) C.word[k] = 0;
  for (int n0 = 0; n0 < nseq; n0 += 32) {
    const int m = min(32, nseq - n0);
    unsigned lit = 0, ml3 = 0, ofv = 0, llc = 0, mlc = 0, ofc = 0;
    if (lane < m) {
      const unsigned long long q = seqs[nseq - 1 - n0 - lane];
      lit = (unsigned)q & 0x3fffu;
      const unsigned ml = (unsigned)(q >> 14) & 0x3fffu;
      ofv = (unsigned)(q >> 28) + 3;
      ml3 = ml - 3;
      llc = lit < 64 ? T.ll_code[lit] : (unsigned)zstd::highbit32(lit) + 19;
      mlc = ml3 < 128 ? T.ml_code[ml3] : (unsigned)zstd::highbit32(ml3) + 36;
      ofc = (unsigned)zstd::highbit32(ofv);
      C.code[0][lane] = (uint8_t)ofc;
      C.code[1][lane] = (uint8_t)mlc;
      C.code[2][lane] = (uint8_t)llc;
    }
    __syncwarp();
    if (lane < 3) {
      int k = 0;
      if (n0 == 0) {  // the first symbol sets the state and emits nothing
        const zstd::FseSym t = T.sym[lane][C.code[lane][0]];
        const unsigned nb = (t.delta_nb_bits + (1u << 15)) >> 16;
        state = T.state[lane][(int)(((nb << 16) - t.delta_nb_bits) >> nb) + t.delta_find_state];
        C.fse[lane][0] = 0;
        k = 1;
      }
#pragma unroll 4
      for (; k < m; k++) {
        const zstd::FseSym t = T.sym[lane][C.code[lane][k]];
        const unsigned nb = (state + t.delta_nb_bits) >> 16;
        C.fse[lane][k] = (uint16_t)((state & ((1u << nb) - 1u)) | nb << 8);
        state = T.state[lane][(int)(state >> nb) + t.delta_find_state];
      }
    }
    __syncwarp();
    unsigned long long v = 0;
    unsigned nb = 0;
    if (lane < m) {
      auto put = [&](unsigned x, unsigned b) {
        v |= (unsigned long long)(x & ((1u << b) - 1u)) << nb;
        nb += b;
      };
#pragma unroll
      for (int t = 0; t < 3; t++) put(C.fse[t][lane] & 255u, C.fse[t][lane] >> 8);
      put(lit, T.ll_bits[llc]);
      put(ml3, T.ml_bits[mlc]);
      put(ofv, ofc);
    }
    unsigned x = nb;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned y = __shfl_up_sync(FULLMASK, x, d);
      if (lane >= d) x += y;
    }
    const unsigned at = fill + x - nb;
    if (nb) {
      const unsigned w = at >> 5, s = at & 31;
      atomicOr(&C.word[w], (uint32_t)(v << s));
      const unsigned long long hi = s ? v >> (32 - s) : v >> 32;
      if (hi) atomicOr(&C.word[w + 1], (uint32_t)hi);
      if (hi >> 32) atomicOr(&C.word[w + 2], (uint32_t)(hi >> 32));
    }
    fill += __shfl_sync(FULLMASK, x, 31);
    __syncwarp();
    const int whole = (int)(fill >> 5);
    for (int k = lane; k < whole; k += 32)
      if (stored + k < ZSEQW) out[stored + k] = C.word[k];
    const uint32_t part = C.word[whole];
    __syncwarp();
    for (int k = lane; k < 64 + 4; k += 32) C.word[k] = k ? 0u : part;
    stored += whole;
    fill &= 31;
    __syncwarp();
  }
  // the final states (match length, offset, literals length), the end bit
  const unsigned s_of = __shfl_sync(FULLMASK, state, 0), s_ml = __shfl_sync(FULLMASK, state, 1),
                 s_ll = __shfl_sync(FULLMASK, state, 2);
  if (lane == 0) {
    unsigned long long v = C.word[0];
    v |= (unsigned long long)((s_ml & 63u) | (s_of & 31u) << 6 | (s_ll & 63u) << 11 | 1u << 17) << fill;
    if (stored < ZSEQW) out[stored] = (uint32_t)v;
    if (stored + 1 < ZSEQW) out[stored + 1] = (uint32_t)(v >> 32);
  }
  return 4 * stored + (int)((fill + 18 + 7) >> 3);
}
static_assert(zstd::kMLLog == 6 && zstd::kOFLog == 5 && zstd::kLLLog == 6, "state bits of the sequence coder");

// One warp per block: the block staged in shared memory (16-byte loads), so
// the match loop's reads are shared-memory reads; matches (the literals go to
// the block's slot as they are passed over), then the sequence stream behind
// them.  Blocks that do not shrink are copied from the source by the gather.
__global__ void __launch_bounds__(32 * ZWARPS) zstd_block_kernel(const uint8_t* __restrict__ src, size_t n,
                                                                 long long nblocks,
                                                                 unsigned long long* __restrict__ seq_all,
                                                                 uint8_t* __restrict__ slots,
                                                                 ZBlock* __restrict__ blocks,
                                                                 unsigned int* __restrict__ sizes) {
  extern __shared__ __align__(16) uint8_t zsm[];
  ZFse& fse = *reinterpret_cast<ZFse*>(zsm + sizeof(ZWarpSmem) * ZWARPS);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = threadIdx.x; k < 3 * 64; k += 32 * ZWARPS) {
    const zstd::FseCTable& t = k < 64 ? c_tables.of : k < 128 ? c_tables.ml : c_tables.ll;
    fse.state[k >> 6][k & 63] = t.state[k & 63];
    fse.sym[k >> 6][k & 63] = t.sym[k & 63];
  }
  for (int k = threadIdx.x; k < 128; k += 32 * ZWARPS) {
    fse.ml_code[k] = c_tables.ml_code[k];
    if (k < 64) fse.ll_code[k] = c_tables.ll_code[k];
    if (k < 36) fse.ll_bits[k] = c_tables.ll_bits[k];
    if (k < 53) fse.ml_bits[k] = c_tables.ml_bits[k];
  }
  __syncthreads();
  const long long b = (long long)blockIdx.x * ZWARPS + warp;
  if (b >= nblocks) return;  // warp-uniform; only __syncwarp below
  ZWarpSmem& W = reinterpret_cast<ZWarpSmem*>(zsm)[warp];
  const size_t s0 = (size_t)b * ZBLK;
  const int len = (int)((n - s0) < (size_t)ZBLK ? (n - s0) : (size_t)ZBLK);
  {
    const uint8_t* g = src + s0;
    uint8_t* d = reinterpret_cast<uint8_t*>(W.data);
    int k0 = 0;
    if (((uintptr_t)g & 15) == 0) {
      const int nv = len >> 4;
      for (int q = lane; q < nv; q += 32)
        reinterpret_cast<uint4*>(W.data)[q] = __ldcs(reinterpret_cast<const uint4*>(g) + q);
      k0 = nv << 4;
    }
    for (int i = k0 + lane; i < len; i += 32) d[i] = g[i];
    __syncwarp();
  }
  uint8_t* slot = slots + (size_t)b * ZSLOT;

  // ---- RLE block: every byte equal ----
  {
    const uint8_t first = len > 0 ? W.byte(0) : 0;
    bool same = true;
    for (int i = lane; i < len && same; i += 32) same = W.byte(i) == first;
    if (__all_sync(FULLMASK, same) && len > 1) {
      if (lane == 0) {
        blocks[b] = ZBlock{4, 1, 0};
        sizes[b] = 4;
      }
      return;
    }
  }

  // ---- greedy matching ----
  for (int i = lane; i < (1 << ZHT_BITS); i += 32) W.ht[i] = 0;
  __syncwarp();
  unsigned long long* seqs = seq_all + (size_t)b * ZMAXSEQ;
  int nseq = 0, anchor = 0, p = 0, nlit = 0;
  while (p + zstd::kMinMatch <= len) {
    const int pos = p + lane;
    const bool ok = pos + zstd::kMinMatch <= len;
    const uint32_t v = W.load4(ok ? pos : 0);
    const uint32_t h = zhash(v);
    const uint32_t at = W.ht[h], cand = ok ? at : 0u;  // position + 1 in the block, 0 = none
    const bool m = cand != 0u && W.load4((int)cand - 1) == v;
    const unsigned bal = __ballot_sync(FULLMASK, m);
    const int f = bal ? __ffs(bal) - 1 : 32;
    __syncwarp();
    if (ok && lane <= f) W.ht[h] = (uint16_t)(pos + 1);
    __syncwarp();
    if (!bal) {
      p += 32;
      continue;
    }
    const int mpos = p + f;
    const int mref = (int)__shfl_sync(FULLMASK, cand, f) - 1;
    int L = zstd::kMinMatch;
    for (;;) {
      const int i = mpos + L + lane;
      const bool eq = i < len && W.byte(mref + L + lane) == W.byte(i);
      const unsigned ne = __ballot_sync(FULLMASK, !eq);
      if (ne) {
        L += __ffs(ne) - 1;
        break;
      }
      L += 32;
    }
    const int lit = mpos - anchor;
    if (lane == 0) seqs[nseq] = seq_pack((unsigned)lit, (unsigned)L, (unsigned)(mpos - mref));
    for (int i = lane; i < lit; i += 32) slot[nlit + i] = W.byte(anchor + i);
    nseq++;
    nlit += lit;
    p = anchor = mpos + L;
  }
  for (int i = lane; i < len - anchor; i += 32) slot[nlit + i] = W.byte(anchor + i);
  nlit += len - anchor;
  __syncwarp();

  // ---- a compressed body: literals header and literals, sequence count and
  // modes, the sequence stream; it must be smaller than the raw block ----
  const int cap = len - 1;
  ZBlock r{3u + (unsigned)len, 0, 0};
  if (nseq > 0 && nlit + 3 < cap) {
    const int k = nlit + lit_header_bytes(nlit);
    const int head = seq_header_bytes(nseq);
    const int stream = code_sequences(seqs, nseq, fse, W.c, reinterpret_cast<uint32_t*>(slot + ZBLK), lane);
    if (cap - k >= 4 && k + head + stream <= cap) {
      r = ZBlock{(unsigned)(3 + k + head + stream), 2, (unsigned)nlit};
      r.type |= (unsigned)nseq << 2;
    }
  }
  if (lane == 0) {
    blocks[b] = r;
    sizes[b] = r.size;
  }
}

// Block b into dst + off[b] (one CTA per block): its headers, then the bytes
// of its slot, or of the source for a raw or RLE block.
__global__ void __launch_bounds__(256) zstd_gather_kernel(const uint8_t* __restrict__ src, size_t n, long long nblocks,
                                                          const uint8_t* __restrict__ slots,
                                                          const ZBlock* __restrict__ blocks,
                                                          const unsigned int* __restrict__ off,
                                                          uint8_t* __restrict__ dst) {
  const long long b = blockIdx.x;
  const ZBlock B = blocks[b];
  const unsigned type = B.type & 3u;
  const int nseq = (int)(B.type >> 2);
  uint8_t* d = dst + off[b];
  const size_t s0 = (size_t)b * ZBLK;
  const unsigned len = (unsigned)((n - s0) < (size_t)ZBLK ? (n - s0) : (size_t)ZBLK);
  const int lh = type == 2 ? lit_header_bytes((int)B.nlit) : 0, sh = type == 2 ? seq_header_bytes(nseq) : 0;
  if (threadIdx.x == 0) {
    zstd::write_block_header(d, b == nblocks - 1, (int)type, type == 2 ? B.size - 3 : len);
    if (type == 2) {
      zstd::write_raw_literals_header(B.nlit, d + 3);
      uint8_t* q = d + 3 + lh + B.nlit;
      if (sh == 2) {
        q[0] = (uint8_t)nseq;
      } else {
        q[0] = (uint8_t)((nseq >> 8) + 128);
        q[1] = (uint8_t)nseq;
      }
      q[sh - 1] = 0;  // predefined modes
    }
  }
  if (type == 1) {
    if (threadIdx.x == 0) d[3] = src[s0];
    return;
  }
  if (type == 0) {
    for (unsigned i = threadIdx.x; i < len; i += blockDim.x) d[3 + i] = src[s0 + i];
    return;
  }
  const uint8_t* s = slots + (size_t)b * ZSLOT;
  uint8_t* dl = d + 3 + lh;
  for (unsigned i = threadIdx.x; i < B.nlit; i += blockDim.x) dl[i] = s[i];
  uint8_t* ds = dl + B.nlit + sh;
  const unsigned stream = B.size - (unsigned)(3 + lh + sh) - B.nlit;
  for (unsigned i = threadIdx.x; i < stream; i += blockDim.x) ds[i] = s[ZBLK + i];
}

bool g_tables_ready[64] = {};
bool g_smem_set[64] = {};

}  // namespace

size_t zstd_frame_bound(size_t n) {
  const size_t nb = n ? (n + ZBLK - 1) / ZBLK : 1;
  return zstd::kFrameHeader + n + 4 * nb;
}

size_t zstd_tmp_bytes(size_t n) {
  const size_t nb = n ? (n + ZBLK - 1) / ZBLK : 1;
  auto al = [](size_t x) { return (x + 255) / 256 * 256 + 256; };
  return al(nb * ZMAXSEQ * 8) + al(nb * ZSLOT) + al(nb * sizeof(ZBlock)) + 2 * al(4 * (nb + 1)) +
         al(scan_u32_tmp_bytes(nb));
}

int launch_zstd_frame(cpsz_b200_ctx* ctx, const uint8_t* d_in, size_t n, uint8_t* d_out, size_t out_cap,
                      size_t* out_size, void* tmp) {
  cudaStream_t st = ctx->stream;
  if (!g_tables_ready[ctx->device & 63]) {
    zstd::Tables T;
    zstd::build_tables(&T);
    // (in place before any stream's kernel reads them: the context's streams do not wait for the default one)
    CPSZ_CUDA_TRY(cudaMemcpyToSymbolAsync(c_tables, &T, sizeof(T), 0, cudaMemcpyHostToDevice, st));
    CPSZ_CUDA_TRY(cudaStreamSynchronize(st));
    g_tables_ready[ctx->device & 63] = true;
  }
  const long long nb = n ? (long long)((n + ZBLK - 1) / ZBLK) : 0;
  auto al = [](size_t x) { return (x + 255) / 256 * 256 + 256; };
  uint8_t* t = (uint8_t*)tmp;
  unsigned long long* seqs = (unsigned long long*)t;
  t += al((size_t)(nb ? nb : 1) * ZMAXSEQ * 8);
  uint8_t* slots = t;
  t += al((size_t)(nb ? nb : 1) * ZSLOT);
  ZBlock* blocks = (ZBlock*)t;
  t += al((size_t)(nb ? nb : 1) * sizeof(ZBlock));
  unsigned int* sizes = (unsigned int*)t;
  t += al(4 * (size_t)(nb + 1));
  unsigned int* off = (unsigned int*)t;
  t += al(4 * (size_t)(nb + 1));
  void* scan_tmp = t;
  uint8_t hdr[zstd::kFrameHeader + 3];
  size_t h = zstd::write_frame_header(hdr, n);
  if (nb == 0) {
    // an empty frame: one empty raw block
    zstd::write_block_header(hdr + h, true, 0, 0);
    h += 3;
    if (out_cap < h) return set_error(CPSZ_ERR_INVALID, "output capacity %zu < frame size %zu", out_cap, h);
    CPSZ_CUDA_TRY(cudaMemcpyAsync(d_out, hdr, h, cudaMemcpyHostToDevice, st));
    CPSZ_CUDA_TRY(cudaStreamSynchronize(st));
    *out_size = h;
    return CPSZ_OK;
  }
  if (n > ((size_t)1 << 32) - 4 * (size_t)nb - 64)
    return set_error(CPSZ_ERR_UNSUPPORTED, "lossless stage input of %zu bytes exceeds 4 GB", n);
  if (!g_smem_set[ctx->device & 63]) {
    CPSZ_CUDA_TRY(cudaFuncSetAttribute(zstd_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ZSMEM));
    g_smem_set[ctx->device & 63] = true;
  }
  zstd_block_kernel<<<(unsigned)((nb + ZWARPS - 1) / ZWARPS), 32 * ZWARPS, ZSMEM, st>>>(d_in, n, nb, seqs, slots,
                                                                                         blocks, sizes);
  count_launch(ctx);
  CPSZ_TRY(check_launch("zstd_block_kernel"));
  CPSZ_TRY(launch_scan_u32(ctx, sizes, off, (size_t)nb, scan_tmp));
  unsigned int total = 0;
  CPSZ_CUDA_TRY(cudaMemcpyAsync(&total, off + nb, 4, cudaMemcpyDeviceToHost, st));
  CPSZ_CUDA_TRY(cudaStreamSynchronize(st));
  const size_t fsize = h + total;
  *out_size = fsize;
  if (fsize > out_cap) return set_error(CPSZ_ERR_INVALID, "output capacity %zu < frame size %zu", out_cap, fsize);
  CPSZ_CUDA_TRY(cudaMemcpyAsync(d_out, hdr, h, cudaMemcpyHostToDevice, st));
  zstd_gather_kernel<<<(unsigned)nb, 256, 0, st>>>(d_in, n, nb, slots, blocks, off, d_out + h);
  count_launch(ctx);
  return check_launch("zstd_gather_kernel");
}

}  // namespace cpsz
