// pipeline2d.cu -- the 2D offline compressor / decompressor on one GPU.
//
// Compress (sz_compress_cp_preserve_2d_offline<float>,
// src/sz_compress_cp_preserve_2d.cpp:175-274):
//   eb2d (bounds + ids + id histogram)  ->  wave2d compress of U and V (codes)
//   -> block-order permutation + code histograms, unpredictable gather
//   -> host Huffman trees (reference tie-breaking) -> GPU bit packing
//   -> blob assembled in device memory -> one copy to the caller.
// The id tree is built on the host while the wavefront runs.
//
// Batches (compress_2d_batch) run in passes of up to 32 fields: every stage
// is issued for all fields of the pass, the wavefront is one persistent
// launch over all of them (its work queue interleaves the fields' row
// groups), and the host builds the pass's Huffman trees on all host threads.
// A single-field call is a pass of one field.
//
// Decompress (sz_decompress_cp_preserve_2d_offline<float>,
// src/sz_decompress_cp_preserve_2d.cpp:8-52): host header/tree parsing ->
// GPU Huffman decode of ids and codes -> raster permutation, unpredictable
// scatter -> wave2d decompress of U and V.
//
// Blob layout (src/sz_compress_cp_preserve_2d.cpp:258-269, src/sz_compress_3d.cpp:219-228):
//   int base(4) | double thr(2^-52) | size_t eb_size | size_t u_size | size_t v_size
//   | HUF(ids, 2048 states, 2N) | FIELD(U) | FIELD(V)
//   FIELD = int 12 | char 0 | int 32768 | meanInfo<float>{false,0} (8 B) | size_t 0
//         | size_t n_unpred | float[n_unpred] | ceil(nblocks/8) zero bytes | HUF(codes, 131072 states, N)
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <vector>

#include "host_pool.h"
#include "huffman_host.h"
#include "kernels.h"
#include "pack_group.h"
#include "tuning.h"
#include "pipeline.h"
#include "transfer.h"

namespace cpsz {

namespace {

constexpr int BS = 12;
constexpr size_t FIELD_HDR = 4 + 1 + 4 + 8 + 8 + 8;  // up to and including n_unpred
constexpr size_t BLOB_HDR = 4 + 8 + 8 + 8 + 8;
// pinned staging per field, behind the fields' id histograms (256 words each):
// the two code histograms' lists and their lengths, the unpredictable counts
constexpr size_t ID_HIST = 256 * 8;
constexpr size_t JOB_PINNED = 2 * 65536 * 8 + 64;
constexpr size_t PINNED_BASE = 4096;  // the flag word and scalars live below
// sub-batch limits: fields per pass (pinned staging) and points per pass (workspace)
constexpr int BATCH_MAX_FIELDS = 32;
constexpr size_t BATCH_MAX_POINTS = (size_t)1 << 27;
// A single field of at least this many points packs its ids on the second
// stream while the wavefront's tail runs; a smaller one (and a batch) packs
// its three streams in one launch once every tree is known: below it the
// extra copy, launches and events cost more than the packing they hide (early
// against together: 512^2 348 and 326 us, 724^2 591 and 584, 1024^2 534 and
// 545, 2048^2 942 and 970).
constexpr size_t EARLY_IDS_POINTS = (size_t)1 << 19;

// upload staging of that packing
constexpr size_t EARLY_UP = 256 * sizeof(HuffEntry) + sizeof(PackPrep) + sizeof(PackJob) + 512;

struct DevBuf {
  // arena sub-allocations of one field
  float* U;
  float* V;
  uint8_t* ids;  // 2N: U ids then V ids
  unsigned long long* hist_ids;
  uint16_t* craster[2];
  float2* pairs[2];  // per-point (value, 1/precision) pairs read by the wavefront
  uint16_t* cblocks[2];
  unsigned long long* hist_codes[2];
  unsigned long long* gbnd;
  unsigned* gdone;            // per component and row group: the wavefront is done with it; then 2 tickets, gave_up
  unsigned long long* units;  // eb2d progress word, then per-unit counters of finished vertices
  int2* uorder;               // eb2d's unit order (every band's units, band after band)
  unsigned long long* strip[2];  // strip-pass look-back words and ticket
  float* unpred[2];
  unsigned long long* enc_code[3];
  uint8_t* enc_len[3];
  unsigned long long* enc_tmp[3];
  uint32_t* bits[3];
  uint8_t* blob;
  float* logs[2];       // offline_log: log2f |U|, |V| (the unpredictable values it stores)
  uint32_t* signs[2];   // offline_log: sign maps
};

// One field of a compression pass (a pass holds one or more fields).
struct Job2D {
  const float* U_in = nullptr;
  const float* V_in = nullptr;
  int r1 = 0, r2 = 0, ngroups = 0, ncb = 0;
  size_t N = 0, nblocks = 0;
  double eb = 0;
  const double* eb_ext = nullptr;  // given per-vertex bounds (device), else derived
  bool dev_in = false;
  size_t ids_bits_cap = 0, codes_bits_cap = 0, blob_cap = 0;
  DevBuf d{};
  unsigned long long* h_hist_ids = nullptr;  // pinned, 256
  unsigned long long* h_list[2] = {nullptr, nullptr};  // pinned, 65536 each
  unsigned* h_nlist = nullptr;               // pinned, 2
  unsigned* h_nunpred = nullptr;             // pinned, 2
  HuffCodebook cb[3];
  bool tree_ok[3] = {false, false, false};
  size_t n_unpred[2] = {0, 0};
  size_t sec_bytes[3] = {0, 0, 0}, bits_bytes[3] = {0, 0, 0};
  size_t size = 0;  // blob bytes
  // device output: the blob is built in place at blob_base (blob_room bytes
  // there), the caller's buffer when it is a device buffer with room for it,
  // else the workspace blob
  unsigned char* dev_out = nullptr;
  size_t dev_cap = 0;
  uint8_t* blob_base = nullptr;
  size_t blob_room = 0;
  // host output: the blob is written straight into host memory (sections
  // copied from their device buffers), not assembled in device memory
  unsigned char* host_out = nullptr;
  size_t host_cap = 0;
  // the offline_log form: base 2, one id stream of N symbols, the two sign
  // maps (device, MSB-first bit streams) between the id section and the fields
  bool log_form = false;
  size_t n_syms(int k) const { return k || log_form ? N : 2 * N; }  // stream k: ids, codes of U / V
};

int read_flag(cpsz_b200_ctx* ctx, int* out) {
  CPSZ_CUDA_TRY(cudaMemcpyAsync(ctx->pinned, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CPSZ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  *out = *(int*)ctx->pinned;
  return CPSZ_OK;
}

// Pinned word receiving the device flag right after the wavefront of a pass
// whose wavefront ran beside the bound kernel.
int* wave_flag_snapshot(cpsz_b200_ctx* ctx) { return (int*)((char*)ctx->pinned + 2048); }
// Pinned word receiving the histogram follower's gave-up flag.
int* follow_flag_snapshot(cpsz_b200_ctx* ctx) { return (int*)((char*)ctx->pinned + 2056); }

int flag_error(int flag) {
  if (flag & FLAG_TIMEOUT) return set_error(CPSZ_ERR_TIMEOUT, "a bounded device-side wait gave up");
  if (flag & FLAG_ID_OVERFLOW)
    return set_error(CPSZ_ERR_UNSUPPORTED, "an error-bound id does not fit the 8-bit id stream (max_pwr_eb too large)");
  if (flag & (FLAG_HUFF_CORRUPT | FLAG_HUFF_RESYNC)) return set_error(CPSZ_ERR_FORMAT, "Huffman stream does not decode");
  if (flag & FLAG_RAW_RANGE) return set_error(CPSZ_ERR_FORMAT, "unpredictable-value list shorter than its codes");
  if (flag & FLAG_OUT_CAPACITY) return set_error(CPSZ_ERR_INVALID, "an output stream exceeded its buffer");
  return CPSZ_OK;
}

// While it lives, the launch wrappers (which all enqueue on ctx->stream) run
// on stream s instead of the context's main stream.
struct OnStream {
  cpsz_b200_ctx* ctx;
  cudaStream_t saved;
  OnStream(cpsz_b200_ctx* c, cudaStream_t s) : ctx(c), saved(c->stream) { c->stream = s; }
  ~OnStream() { ctx->stream = saved; }
};

int job_init(Job2D& j, const float* U, const float* V, size_t r1s, size_t r2s, double eb) {
  if (!U || !V) return set_error(CPSZ_ERR_INVALID, "null input field");
  if (r1s == 0 || r2s == 0) return set_error(CPSZ_ERR_INVALID, "empty field (%zu x %zu)", r1s, r2s);
  if (r1s > (1u << 30) || r2s > (1u << 30) || r1s * r2s > (size_t)INT32_MAX)
    return set_error(CPSZ_ERR_UNSUPPORTED, "field of %zu x %zu points exceeds 2^31 points", r1s, r2s);
  if (eb != eb) return set_error(CPSZ_ERR_INVALID, "max_pwr_eb is NaN");
  j.U_in = U;
  j.V_in = V;
  j.r1 = (int)r1s;
  j.r2 = (int)r2s;
  j.N = r1s * r2s;
  j.eb = eb;
  j.ngroups = (j.r1 + WAVE_GROUP_ROWS - 1) / WAVE_GROUP_ROWS;
  j.ncb = (j.r2 + UNIT_COLS - 1) / UNIT_COLS;
  const int nby = (j.r2 - 1) / BS + 1, nbx = (j.r1 - 1) / BS + 1;
  j.nblocks = (size_t)nbx * nby;
  j.dev_in = is_device_ptr(U) && is_device_ptr(V);
  // bit streams: Huffman averages < log2(distinct) + 1 bits per symbol
  j.ids_bits_cap = (2 * j.N * 9 + 7) / 8 + 64;
  j.codes_bits_cap = (j.N * 17 + 7) / 8 + 64;
  j.blob_cap = BLOB_HDR + 2 * FIELD_HDR + 8 * j.N + 2 * ((j.nblocks + 7) / 8) + 2 * (j.N / 8 + 1) +
               3 * (12 + 1 + 13 * 131072 + 8) +
               j.ids_bits_cap + 2 * j.codes_bits_cap + 64;
  return CPSZ_OK;
}

// Bound of a field's uploads once its trees are known: code entries and
// their tables' jobs, then the blob's small pieces (header, three trees with
// their stream sizes, field headers) and their descriptors.
size_t up_bytes_bound(const Job2D& j) {
  const size_t sym = std::min<size_t>(65536, j.N), tree = 12 + 1 + 13 * std::min<size_t>(131072, 2 * j.N + 1) + 8;
  return (256 + 2 * sym) * sizeof(HuffEntry) + BLOB_HDR + 2 * FIELD_HDR + (12 + 1 + 13 * 512 + 8) + 2 * tree +
         3 * (sizeof(PackPrep) + sizeof(PackJob)) + 24 * sizeof(CopyPiece) + 1024;
}

// Pass-wide device pieces.
struct PassBuf {
  // the setup image, one upload: thresholds, wavefront fields and items, jobs
  // of the batched kernels, eb2d's unit order
  uint8_t* image;
  size_t image_bytes;
  double* thr;
  WaveField* fields;
  WaveItem* items;
  Eb2dJob* eb;
  HistJob* hist;
  HistList* list;
  StripJob* strip;
  int2* uorder;
  // zeroed in one piece: the wavefront's queue, histograms, look-back words
  uint8_t* zero;
  size_t zero_bytes;
  int* queue;
  unsigned long long* hist_ids;
  uint8_t* gbnd;  // boundary rows, right behind (a pass over some row groups keeps part of them)
  size_t gbnd_bytes;
  uint8_t* up_ids;  // early id entries
  uint8_t* up;      // later uploads
  size_t up_bytes;
};

// The pass's workspace: with a null arena every piece is only counted (each
// padded as the arena pads it).
struct Alloc {
  cpsz_b200_ctx* ctx;  // null: count
  size_t bytes = 0;
  bool failed = false;
  void* operator()(size_t b) {
    bytes += align_up(b, 256) + 256;
    if (!ctx || failed) return nullptr;
    // a request that does not fit fails every later one too (no smaller piece
    // may land behind a failed one)
    void* p = arena_alloc(ctx, b);
    failed = !p;
    return p;
  }
};
// A run of pieces inside one allocation, 256-byte aligned each.
struct Run {
  uint8_t* base;
  size_t at = 0;
  uint8_t* take(size_t b) {
    uint8_t* p = base ? base + at : nullptr;
    at += align_up(b, 256);
    return p;
  }
};

void pass_alloc(std::vector<Job2D>& jobs, PassBuf& P, Alloc& A) {
  const size_t nj = jobs.size();
  auto image = [&](Run r) {
    P.thr = (double*)r.take(QUANT_TAB_MAX * 8);
    P.fields = (WaveField*)r.take(2 * nj * sizeof(WaveField));
    size_t groups = 0, units = 0;
    for (const Job2D& j : jobs) {
      groups += j.ngroups;
      units += (size_t)j.ngroups * j.ncb;
    }
    P.items = (WaveItem*)r.take(2 * groups * sizeof(WaveItem));
    P.eb = (Eb2dJob*)r.take(nj * sizeof(Eb2dJob));
    P.hist = (HistJob*)r.take(nj * sizeof(HistJob));
    P.list = (HistList*)r.take(2 * nj * sizeof(HistList));
    P.strip = (StripJob*)r.take(nj * sizeof(StripJob));
    P.uorder = (int2*)r.take(nj == 1 ? units * sizeof(int2) : 0);
    return r.at;
  };
  P.image_bytes = image(Run{nullptr});
  P.image = (uint8_t*)A(P.image_bytes);
  image(Run{P.image});
  auto zero = [&](Run r) {
    P.queue = (int*)r.take(256);
    P.hist_ids = (unsigned long long*)r.take(nj * ID_HIST);
    for (size_t k = 0; k < nj; k++) {
      Job2D& j = jobs[k];
      DevBuf& d = j.d;
      d.hist_ids = P.hist_ids + 256 * k;
      d.units = (unsigned long long*)r.take(((size_t)j.ngroups * j.ncb + 1) * 8);
      d.gdone = (unsigned*)r.take((2 * (size_t)j.ngroups + 4) * 4);
      for (int f = 0; f < 2; f++) {
        d.hist_codes[f] = (unsigned long long*)r.take(65536 * 8);
        d.strip[f] = (unsigned long long*)r.take(strip_scratch_bytes(j.r1, j.r2));
      }
      for (int f = 0; f < 3; f++) d.enc_tmp[f] = (unsigned long long*)r.take(huff_encode_tmp_bytes(j.n_syms(f)));
    }
    P.zero_bytes = r.at;
    P.gbnd = r.take(0);
    for (Job2D& j : jobs) j.d.gbnd = (unsigned long long*)r.take(2 * j.ngroups * wave_gbnd_pitch(j.r2) * 8);
    P.gbnd_bytes = r.at - P.zero_bytes;
    return r.at;
  };
  const size_t zb = zero(Run{nullptr});
  P.zero = (uint8_t*)A(zb);
  zero(Run{P.zero});
  P.up_bytes = 0;
  for (const Job2D& j : jobs) P.up_bytes += up_bytes_bound(j);
  P.up = (uint8_t*)A(P.up_bytes);
  P.up_ids = (uint8_t*)A(EARLY_UP);
  for (Job2D& j : jobs) {
    DevBuf& d = j.d;
    const size_t N = j.N;
    if (j.dev_in) {
      d.U = const_cast<float*>(j.U_in);
      d.V = const_cast<float*>(j.V_in);
    } else {
      d.U = (float*)A(4 * N);
      d.V = (float*)A(4 * N);
    }
    d.ids = (uint8_t*)A(2 * N);
    for (int f = 0; f < 2; f++) {
      d.craster[f] = (uint16_t*)A(2 * N);
      d.pairs[f] = (float2*)A(8 * N);
      d.cblocks[f] = (uint16_t*)A(2 * N);
      d.unpred[f] = (float*)A(4 * N);
    }
    d.uorder = P.uorder;
    for (int f = 0; f < 3; f++) {
      const size_t n = f ? 65536 : 256;
      d.enc_code[f] = (unsigned long long*)A(n * 8);
      d.enc_len[f] = (uint8_t*)A(n);
      d.bits[f] = (uint32_t*)A(f ? j.codes_bits_cap : j.ids_bits_cap);
    }
    d.blob = (uint8_t*)A(j.blob_cap);
    if (j.log_form)
      for (int f = 0; f < 2; f++) {
        d.logs[f] = (float*)A(4 * N);
        d.signs[f] = (uint32_t*)A(4 * ((N + 31) / 32));
      }
    j.blob_base = d.blob;
    j.blob_room = align_up(j.blob_cap, 256);
    if (j.dev_out && j.dev_cap >= j.blob_cap + 8) {
      j.blob_base = j.dev_out;
      j.blob_room = j.dev_cap;
    }
  }
}

// The reference's 2D blob (sz_compress_cp_preserve_2d_offline,
// src/sz_compress_cp_preserve_2d.cpp): header, the id stream's Huffman
// section, then per component its header, unpredictable floats, the all-zero
// block indicator and the code stream's Huffman section.  Every small piece is
// staged in `small`; the bit streams and unpredictable floats go to bit_dst /
// unpred_dst.
struct BlobLayout {
  // bytes [dst, dst + n) of the blob: from small[src] (ext null), from ext
  // (host memory that outlives the pass: a code tree), or zeros (zero)
  struct Piece {
    size_t dst, src, n;
    const uint8_t* ext;
    bool zero;
  };
  size_t total = 0, bit_dst[3] = {0, 0, 0}, unpred_dst[2] = {0, 0}, sign_dst = 0, sign_bytes = 0;
  std::vector<uint8_t> small;
  std::vector<Piece> pieces;
};

// offset of the id stream's bits (known once the id tree is)
size_t ids_bits_at(const Job2D& j) { return BLOB_HDR + j.cb[0].tree_bytes.size() + 8; }

int job_layout(const Job2D& j, BlobLayout& L) {
  const size_t ind_bytes = (j.nblocks + 7) / 8;
  size_t field_size[2];
  for (int f = 0; f < 2; f++) field_size[f] = FIELD_HDR + 4 * j.n_unpred[f] + ind_bytes + j.sec_bytes[1 + f];
  const size_t sign_bytes = j.log_form ? (j.N - 1) / 8 + 1 : 0;
  const size_t total = BLOB_HDR + j.sec_bytes[0] + 2 * sign_bytes + field_size[0] + field_size[1];
  L.total = total;
  L.sign_bytes = sign_bytes;
  std::vector<uint8_t>& small = L.small;
  small.reserve(BLOB_HDR + j.cb[0].tree_bytes.size() + 3 * 8 + 2 * FIELD_HDR);
  auto stage = [&](size_t dst, const void* p, size_t n) {
    L.pieces.push_back(BlobLayout::Piece{dst, small.size(), n, nullptr, false});
    small.insert(small.end(), (const uint8_t*)p, (const uint8_t*)p + n);
  };
  // the code trees and the zero indicator bytes are referenced, not copied:
  // the layout precedes the code packing, their bytes go up after it
  auto refer = [&](size_t dst, const uint8_t* p, size_t n) {
    L.pieces.push_back(BlobLayout::Piece{dst, 0, n, p, p == nullptr});
  };
  {
    uint8_t hdr[BLOB_HDR];
    const int base = j.log_form ? 2 : 4;
    const double thr = DBL_EPSILON;
    memcpy(hdr, &base, 4);
    memcpy(hdr + 4, &thr, 8);
    memcpy(hdr + 12, &j.sec_bytes[0], 8);
    memcpy(hdr + 20, &field_size[0], 8);
    memcpy(hdr + 28, &field_size[1], 8);
    stage(0, hdr, BLOB_HDR);
  }
  size_t at = BLOB_HDR;
  size_t* bit_dst = L.bit_dst;
  size_t* unpred_dst = L.unpred_dst;
  auto stage_huff = [&](int k) {
    if (k == 0) stage(at, j.cb[k].tree_bytes.data(), j.cb[k].tree_bytes.size());
    else refer(at, j.cb[k].tree_bytes.data(), j.cb[k].tree_bytes.size());
    at += j.cb[k].tree_bytes.size();
    unsigned long long nb = j.bits_bytes[k];
    stage(at, &nb, 8);
    at += 8;
    bit_dst[k] = at;
    at += j.bits_bytes[k];
  };
  stage_huff(0);
  L.sign_dst = at;  // offline_log: sign maps of U and V (copied from the device)
  at += 2 * sign_bytes;
  for (int f = 0; f < 2; f++) {
    uint8_t fh[FIELD_HDR];
    memset(fh, 0, sizeof(fh));
    const int bs = BS, radius = 32768;
    memcpy(fh, &bs, 4);
    memcpy(fh + 5, &radius, 4);
    // meanInfo<float>{false, 0}: 8 zero bytes; reg_count = 0
    unsigned long long nu = j.n_unpred[f];
    memcpy(fh + 5 + 4 + 8 + 8, &nu, 8);
    stage(at, fh, FIELD_HDR);
    at += FIELD_HDR;
    unpred_dst[f] = at;
    at += 4 * j.n_unpred[f];
    refer(at, nullptr, ind_bytes);
    at += ind_bytes;
    stage_huff(1 + f);
  }
  if (at != total) return set_error(CPSZ_ERR_INVALID, "internal: blob layout mismatch (%zu != %zu)", at, total);
  return CPSZ_OK;
}

// Upload staging that job_pieces takes for a field, its copies' table included.
size_t piece_up_bytes(const BlobLayout& L) {
  size_t b = align_up(L.small.size(), 16) + (L.pieces.size() + 5) * sizeof(CopyPiece) + 64;
  for (const BlobLayout::Piece& pc : L.pieces)
    if (pc.ext) b += align_up(pc.n, 16) + 16;
  return b;
}

// The sections of a device blob that the packers do not write, as copies for
// launch_copy_pieces: the staged small pieces (header, trees, stream sizes,
// field headers), the zero indicators, the unpredictable values, the sign maps.
int job_pieces(Job2D& j, const BlobLayout& L, UpImage& up, std::vector<CopyPiece>& out) {
  uint8_t* blob = j.blob_base;
  uint8_t *d_small, *d_ext;
  uint8_t* h = up.take(L.small.size(), &d_small);
  if (!h) return up_overrun();
  memcpy(h, L.small.data(), L.small.size());
  for (const BlobLayout::Piece& pc : L.pieces) {
    CopyPiece c{blob + pc.dst, pc.zero ? nullptr : d_small + pc.src, pc.n, 0};
    if (pc.ext) {
      if (!(h = up.take(pc.n, &d_ext))) return up_overrun();
      memcpy(h, pc.ext, pc.n);
      c.src = d_ext;
    }
    out.push_back(c);
  }
  for (int f = 0; f < 2; f++) {
    if (j.n_unpred[f])
      out.push_back(CopyPiece{blob + L.unpred_dst[f], (const uint8_t*)j.d.unpred[f], 4 * j.n_unpred[f], 0});
    if (L.sign_bytes)
      out.push_back(
          CopyPiece{blob + L.sign_dst + f * L.sign_bytes, (const uint8_t*)j.d.signs[f], L.sign_bytes, 0});
  }
  j.size = L.total;
  return CPSZ_OK;
}

// One compression pass over `jobs` (workspace reserved by the caller).
// dev_at (device memory with room for dev_room bytes, or null): the blobs are
// built there back to back if they fit.
int run_pass(cpsz_b200_ctx* ctx, std::vector<Job2D>& jobs, const StageTap* tap, uint8_t* dev_at, size_t dev_room) {
  cudaStream_t st = ctx->stream;
  const int nj = (int)jobs.size();
  // the offline_log form runs as a pass of one field
  const bool log_form = nj == 1 && jobs[0].log_form;
  const QuantTable& qt = log_form ? quant_table_2d_log() : quant_table_2d();
  LibmTables libm{};
  if (log_form) CPSZ_TRY(libm_tables_device(ctx, &libm));
  PassBuf P{};
  Alloc arena{ctx};
  pass_alloc(jobs, P, arena);
  if (arena.failed) return set_error(CPSZ_ERR_NOMEM, "workspace layout overflow");
  {
    uint8_t* base = (uint8_t*)ctx->pinned + PINNED_BASE;
    for (int k = 0; k < nj; k++) jobs[k].h_hist_ids = (unsigned long long*)(base + k * ID_HIST);
    base += nj * ID_HIST;
    for (int k = 0; k < nj; k++, base += JOB_PINNED) {
      for (int f = 0; f < 2; f++) jobs[k].h_list[f] = (unsigned long long*)base + (size_t)f * 65536;
      jobs[k].h_nlist = (unsigned*)(base + 2 * 65536 * 8);
      jobs[k].h_nunpred = jobs[k].h_nlist + 2;
    }
  }

  // Derived bounds (eb2d) signal per 128-row group, so for one field the
  // wavefront runs beside them on the high-priority stream and starts on a
  // group as soon as its pairs are written: its items (group-major over the
  // two components) come in the order eb2d finishes them.  A batch's items
  // are group-major across fields while eb2d finishes field after field, so a
  // batch (and given bounds, quant2d, which are not row-ordered) runs the
  // wavefront after the bounds with every CTA slot.
  const bool overlap =
      nj == 1 && jobs[0].eb_ext == nullptr && !log_form && tune_get(TUNE_WAVE2D_OVERLAP, jobs[0].N) != 0;
  // Host input is uploaded and bounded in bands of band_rows(j) rows (a
  // multiple of WAVE_GROUP_ROWS), band c right after its upload.
  auto band_rows = [&](const Job2D& j) -> int {
    const int K = (!j.dev_in && j.N >= ((size_t)1 << 22) && !j.eb_ext) ? tune_get(TUNE_H2D_CHUNKS, j.N) : 1;
    return (int)align_up((size_t)(j.r1 + K - 1) / K, WAVE_GROUP_ROWS);
  };

  // ---- setup: one image with the tables and every kernel's jobs, built in
  // the page-locked upload staging (no copy from it is in flight yet; the
  // pass's later uploads reuse it after this copy has run) ----
  reset_marks(ctx);
  mark(ctx, "h2d+setup");
  CPSZ_TRY(upload_reserve(ctx, P.image_bytes));
  uint8_t* const h_image = (uint8_t*)ctx->up_pinned;
  auto host = [&](auto* dev) { return reinterpret_cast<decltype(dev)>(h_image + ((uint8_t*)dev - P.image)); };
  memcpy(host(P.thr), qt.t, QUANT_TAB_MAX * 8);
  // a pass that quantizes again only some vertices starts the recursion at
  // their first row group: the groups above (and their boundary rows, which
  // the first group run reads) are the previous pass's
  const int g0 = (nj == 1 && tap && tap->recon_only && tap->requant && jobs[0].eb_ext)
                     ? std::min(std::max(tap->first_group, 0), jobs[0].ngroups)
                     : 0;
  // One large field beside its bounds: the code histograms are counted while
  // the wavefront's tail runs (hist_follow on the second stream), as its row
  // groups finish, instead of after it (below 2^22 points the histograms take
  // a few microseconds and the follower's own launch and waits cost more).
  const bool follow = overlap && nj == 1 && !tap && jobs[0].N >= ((size_t)1 << 22);
  std::vector<WaveField> hf(2 * nj);
  std::vector<int> r1v(2 * nj);
  std::vector<HistJob> hist_jobs(nj);
  std::vector<StripJob> strip_jobs(nj);
  size_t strips = 0;
  for (int k = 0; k < nj; k++) {
    Job2D& j = jobs[k];
    if (overlap) {
      // eb2d's unit order, band by band (units along diagonals of slope
      // eb2d.skew column blocks per group)
      const int R = band_rows(j), skew = tune_get(TUNE_EB2D_SKEW, j.N);
      std::vector<int2> part;
      int2* order = host(P.uorder);
      for (int r0 = 0; r0 < j.r1; r0 += R) {
        unit_order(r0 / WAVE_GROUP_ROWS, (std::min(j.r1, r0 + R) + WAVE_GROUP_ROWS - 1) / WAVE_GROUP_ROWS, j.ncb, skew,
                   part);
        order = std::copy(part.begin(), part.end(), order);
      }
    }
    StripJob& S = strip_jobs[k];
    S = StripJob{{j.d.craster[0], j.d.craster[1]},
                 {j.log_form ? j.d.logs[0] : j.d.U, j.log_form ? j.d.logs[1] : j.d.V},
                 {j.d.cblocks[0], j.d.cblocks[1]},
                 {j.d.unpred[0], j.d.unpred[1]},
                 {j.d.strip[0], j.d.strip[1]},
                 j.h_nunpred,
                 j.r1,
                 j.r2,
                 (unsigned)strips};
    strips += strip_count(j.r1, j.r2);
    hist_jobs[k] = HistJob{{j.d.craster[0], j.d.craster[1]}, {j.d.hist_codes[0], j.d.hist_codes[1]}, j.N, 0, 0};
    for (int f = 0; f < 2; f++) {
      host(P.list)[2 * k + f] = HistList{j.d.hist_codes[f], j.h_list[f], j.h_nlist + f};
      WaveField& F = hf[2 * k + f];
      F.pair = j.d.pairs[f];
      F.codes = j.d.craster[f];
      F.trace = (nj == 1 && ctx->d_wave_trace && ctx->wave_trace_len >= 2 * (size_t)j.ngroups * WAVE_WARPS * 4)
                    ? ctx->d_wave_trace + (size_t)f * j.ngroups * WAVE_WARPS * 4
                    : nullptr;
      F.out = tap ? tap->recon[f] : nullptr;
      F.gbnd = j.d.gbnd + f * j.ngroups * wave_gbnd_pitch(j.r2);
      F.pair_pitch = j.r2;
      F.code_pitch = j.r2;
      F.out_pitch = j.r2;
      F.r1 = j.r1;
      F.r2 = j.r2;
      F.unit_done = overlap ? j.d.units + 1 : nullptr;
      F.unit_ncb = j.ncb;
      F.band_wait_ns = ctx->band_wait_ns;
      F.band_extra = ctx->band_unreachable ? 1 : 0;
      F.group_done = follow ? j.d.gdone + (size_t)f * j.ngroups : nullptr;
      r1v[2 * k + f] = j.r1;
    }
  }
  if (strips > 0x7fffffffu) return set_error(CPSZ_ERR_UNSUPPORTED, "fields of %zu strips", strips);
  const unsigned hist_ctas = hist_assign_ctas(ctx->num_sms, hist_jobs.data(), nj);
  std::vector<WaveItem> items;
  build_wave_items(2 * nj, r1v.data(), items);
  if (g0 > 0) items.erase(std::remove_if(items.begin(), items.end(), [&](const WaveItem& w) { return w.group < g0; }),
                          items.end());
  const int n_items = (int)items.size();
  std::copy(hf.begin(), hf.end(), host(P.fields));
  std::copy(items.begin(), items.end(), host(P.items));
  std::copy(hist_jobs.begin(), hist_jobs.end(), host(P.hist));
  std::copy(strip_jobs.begin(), strip_jobs.end(), host(P.strip));
  // A batch of device-resident fields derives its bounds in one bound-kernel
  // launch: every field's tiles in one grid (largest field first, so the
  // small fields' tiles fill the launch's tail), each CTA finding its field in
  // a descriptor table, instead of a launch per field that leaves the SMs
  // idle while a small field's few tiles run.
  bool eb_batched = nj > 1;
  for (const Job2D& j : jobs)
    eb_batched = eb_batched && j.dev_in && !j.eb_ext && !j.log_form && j.eb >= 0 && j.eb <= 1e300;
  int eb_shape = 0, eb_tiles = 0;
  if (eb_batched) {
    size_t largest = 0;
    for (const Job2D& j : jobs) largest = std::max(largest, j.N);
    eb_shape = tune_get(TUNE_EB2D_TILE, largest);
    int tx, ty;
    eb2d_tile_shape(eb_shape, &tx, &ty);
    std::vector<int> by_size(nj);
    for (int k = 0; k < nj; k++) by_size[k] = k;
    std::stable_sort(by_size.begin(), by_size.end(), [&](int a, int b) { return jobs[a].N > jobs[b].N; });
    Eb2dJob* ebj = host(P.eb);
    for (int k : by_size) {
      const Job2D& j = jobs[k];
      Eb2dJob e;
      e.U = j.d.U;
      e.V = j.d.V;
      e.ids_u = j.d.ids;
      e.ids_v = j.d.ids + j.N;
      e.hist = j.d.hist_ids;
      e.pair_u = j.d.pairs[0];
      e.pair_v = j.d.pairs[1];
      e.max_pwr_eb = j.eb;
      e.r1 = j.r1;
      e.r2 = j.r2;
      e.tiles_x = (j.r2 + tx - 1) / tx;
      e.tile0 = eb_tiles;
      const size_t t = (size_t)e.tiles_x * ((j.r1 + ty - 1) / ty);
      if (eb_tiles + t > (size_t)INT32_MAX) {
        eb_batched = false;  // beyond one grid's tile count: a launch per field
        break;
      }
      eb_tiles += (int)t;
      *ebj++ = e;
    }
  }
  CPSZ_CUDA_TRY(cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), st));
  CPSZ_CUDA_TRY(cudaMemcpyAsync(P.image, h_image, P.image_bytes, cudaMemcpyHostToDevice, st));
  if (g0 == 0) {
    CPSZ_CUDA_TRY(cudaMemsetAsync(P.zero, 0, P.zero_bytes + P.gbnd_bytes, st));
  } else {
    const Job2D& j = jobs[0];
    CPSZ_CUDA_TRY(cudaMemsetAsync(P.zero, 0, P.zero_bytes, st));
    const size_t pitch = wave_gbnd_pitch(j.r2);
    for (int f = 0; f < 2; f++)
      CPSZ_CUDA_TRY(cudaMemsetAsync(j.d.gbnd + ((size_t)f * j.ngroups + g0) * pitch, 0,
                                    (size_t)(j.ngroups - g0) * pitch * 8, st));
  }
  double* const thr_tab = P.thr;
  int* const queue = P.queue;
  const WaveField* const d_fields = P.fields;
  const WaveItem* const d_items = P.items;
  size_t pass_points = 0;
  for (const Job2D& j : jobs) pass_points += j.N;
  // a wavefront launched beside its producer must be finished before this
  // call returns on any path (its workspace is reused by the next call)
  struct HiDrain {
    cudaStream_t s = nullptr;
    ~HiDrain() {
      if (s) cudaStreamSynchronize(s);
    }
  } hi_drain, follow_drain;
  if (overlap) {
    // The wavefront (high-priority stream, one CTA per SM) is launched before
    // its producer eb2d (stage 1), whose CTAs then fill the rest of every SM:
    // measured at 8192^2, this order takes 7.87 ms a compression against
    // 8.7-9.5 ms with eb2d enqueued first (eb2d itself runs slower behind a
    // late wavefront, which then trails it).  The order is not relied on: a
    // wavefront wait gives up once eb2d shows no progress for a while (a tool
    // that serialises kernels runs the wavefront alone first), and the pass
    // then runs its wavefront again after the bounds (see the code trees
    // below), so serialised execution costs that wait, not a failure.
    CPSZ_TRY(preload_eb2d());
    CPSZ_TRY(preload_wave2d());
    for (const Job2D& j : jobs)
      if (!j.dev_in) {  // a band and the row below it are copied at once
        const size_t band = 4 * (size_t)std::min(j.r1, band_rows(j) + 1) * j.r2;
        CPSZ_TRY(transfer_reserve(ctx, j.U_in, band));
        CPSZ_TRY(transfer_reserve(ctx, j.V_in, band));
      }
    hi_drain.s = ctx->hi;
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[3], st));
    CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->hi, ctx->ev[3], 0));
    CPSZ_TRY(launch_wave2d(ctx, false, d_fields, d_items, n_items, queue, pass_points, ctx->hi, WAVE_BESIDE));
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[4], ctx->hi));
  }

  // Stages 1-3 (bounds, wavefront, code histograms, block order) are the
  // pass's device work before the host builds the code trees.  A batch whose
  // fields are all in device memory captures them once into a CUDA graph,
  // kept on the context and replayed while the pass is the same (fields,
  // shapes, bounds, workspace, tuning table); events the host waits on are
  // recorded as external events of the graph.
  bool all_dev_in = true;
  for (const Job2D& j : jobs) all_dev_in = all_dev_in && j.dev_in;
  bool capturing = false;
  auto record = [&](cudaEvent_t e) {
    return capturing ? cudaEventRecordWithFlags(e, st, cudaEventRecordExternal) : cudaEventRecord(e, st);
  };
  auto stages_1_2 = [&]() -> int {
    // ---- stage 1: inputs and error bounds ----
    mark(ctx, "eb2d");
    // host-input uploads run on the second stream, after the pass's setup (once
    // per pass: per field it would hold each upload behind the previous field's
    // bound kernels)
    if (!all_dev_in) {
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[2], st));
      CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->ev[2], 0));
    }
    if (eb_batched)
      CPSZ_TRY(launch_eb2d_batch(ctx, P.eb, nj, eb_tiles, eb_shape, thr_tab, qt.n, qt.float_pow4));
    for (Job2D& j : jobs) {
      // beside the wavefront, eb2d runs unit by unit in the order made in the
      // setup; band_units(g0, g1) is the slice for the rows of groups [g0, g1)
      auto band_units = [&](int g0, int g1) {
        Eb2dUnits u;
        u.order = j.d.uorder + (size_t)g0 * j.ncb;
        u.n = (g1 - g0) * j.ncb;
        u.ncb = j.ncb;
        u.done = j.d.units + 1;  // [-1]: tiles finished
        return u;
      };
      if (j.log_form) {
        // offline_log: the fields whole, one id per vertex, then the logs,
        // wavefront pairs and sign maps
        if (!j.dev_in) {
          CPSZ_TRY(h2d(ctx, j.d.U, j.U_in, 4 * j.N, st));
          CPSZ_TRY(h2d(ctx, j.d.V, j.V_in, 4 * j.N, st));
        }
        CPSZ_TRY(launch_eb2d(ctx, j.d.U, j.d.V, j.r1, j.r2, j.eb, thr_tab, qt.n, j.d.ids, nullptr, j.d.hist_ids,
                             nullptr, nullptr, nullptr, 0, -1, nullptr, true));
        CPSZ_TRY(launch_log2d(ctx, j.d.U, j.d.V, j.d.ids, j.N, libm.log2f, j.d.pairs[0], j.d.pairs[1], j.d.logs[0],
                              j.d.logs[1], j.d.signs[0], j.d.signs[1]));
      } else if (j.dev_in) {
        if (j.eb_ext && nj == 1 && tap && tap->recon_only && tap->requant)
          CPSZ_TRY(launch_requant2d(ctx, j.d.U, j.d.V, j.N, j.eb_ext, thr_tab, qt.n, j.d.ids, j.d.ids + j.N,
                                    j.d.pairs[0], j.d.pairs[1], tap->requant));
        else if (j.eb_ext)
          CPSZ_TRY(launch_quant2d(ctx, j.d.U, j.d.V, j.N, j.eb_ext, thr_tab, qt.n, j.d.ids, j.d.ids + j.N,
                                  j.d.hist_ids, j.d.pairs[0], j.d.pairs[1]));
        else if (!eb_batched) {
          const Eb2dUnits u = band_units(0, j.ngroups);
          CPSZ_TRY(launch_eb2d(ctx, j.d.U, j.d.V, j.r1, j.r2, j.eb, thr_tab, qt.n, j.d.ids, j.d.ids + j.N,
                               j.d.hist_ids, j.d.pairs[0], j.d.pairs[1], nullptr, 0, -1, overlap ? &u : nullptr,
                               false, qt.float_pow4));
        }
      } else {
        // Host input: row chunks go up on the second stream and the bound kernel
        // runs band by band as soon as a band's rows and the row below it are
        // on the device, so the transfer overlaps the bound derivation.  Bands
        // start on wavefront group boundaries.  Chunk c carries its band's rows
        // and the next band's first row (which chunk c + 1 writes again, with
        // the same bytes), so band c waits for chunk c alone and only the last
        // band's bounds follow the end of the transfer.
        const int R = band_rows(j);
        const int nch = (j.r1 + R - 1) / R;
        // band c is enqueued right after chunk c's copy call (a copy from
        // pageable memory returns only once the host has staged it, so
        // enqueueing every copy first would hold the bands back until the whole
        // field was staged)
        auto band_launch = [&](int c) -> int {
          CPSZ_CUDA_TRY(cudaStreamWaitEvent(st, ctx->up_ev[c], 0));
          if (j.eb_ext)
            return launch_quant2d(ctx, j.d.U, j.d.V, j.N, j.eb_ext, thr_tab, qt.n, j.d.ids, j.d.ids + j.N,
                                  j.d.hist_ids, j.d.pairs[0], j.d.pairs[1]);
          const Eb2dUnits u = band_units(c * R / WAVE_GROUP_ROWS, (std::min(j.r1, (c + 1) * R) + WAVE_GROUP_ROWS - 1) /
                                                                     WAVE_GROUP_ROWS);
          return launch_eb2d(ctx, j.d.U, j.d.V, j.r1, j.r2, j.eb, thr_tab, qt.n, j.d.ids, j.d.ids + j.N, j.d.hist_ids,
                             j.d.pairs[0], j.d.pairs[1], nullptr, c * R, std::min(j.r1, (c + 1) * R),
                             overlap ? &u : nullptr, false, qt.float_pow4);
        };
        for (int c = 0; c < nch; c++) {
          const size_t off = (size_t)c * R * j.r2;
          const size_t cnt = (size_t)(std::min(j.r1, (c + 1) * R + 1) - c * R) * j.r2;
          CPSZ_TRY(h2d(ctx, j.d.U + off, j.U_in + off, 4 * cnt, ctx->aux));
          CPSZ_TRY(h2d(ctx, j.d.V + off, j.V_in + off, 4 * cnt, ctx->aux));
          CPSZ_CUDA_TRY(cudaEventRecord(ctx->up_ev[c], ctx->aux));
          CPSZ_TRY(band_launch(c));
        }
      }
    }
    if (!(tap && tap->recon_only))
      CPSZ_CUDA_TRY(cudaMemcpyAsync(jobs[0].h_hist_ids, P.hist_ids, nj * ID_HIST, cudaMemcpyDeviceToHost, st));
    CPSZ_CUDA_TRY(record(ctx->ev[0]));
    if (follow) {
      // the code histograms, counted on the second stream as the wavefront
      // finishes its row groups; the flag and the lists come back there
      Job2D& j = jobs[0];
      follow_drain.s = ctx->aux;
      CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->ev[0], 0));
      const uint16_t* codes[2] = {j.d.craster[0], j.d.craster[1]};
      const unsigned* gd[2] = {j.d.gdone, j.d.gdone + j.ngroups};
      unsigned long long* hc[2] = {j.d.hist_codes[0], j.d.hist_codes[1]};
      unsigned* tix = j.d.gdone + 2 * (size_t)j.ngroups;
      CPSZ_TRY(launch_hist_follow(ctx, codes, gd, j.r1, j.r2, hc, tix, (int*)(tix + 2), ctx->aux));
      CPSZ_CUDA_TRY(
          cudaMemcpyAsync(follow_flag_snapshot(ctx), tix + 2, sizeof(int), cudaMemcpyDeviceToHost, ctx->aux));
      // on the high-priority stream: its two CTAs would otherwise wait for the
      // block-order pass's tens of thousands (the host's trees start with them)
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[6], ctx->aux));
      CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->hi, ctx->ev[6], 0));
      CPSZ_TRY(launch_hist_list(ctx, P.list, 2, ctx->hi));
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[6], ctx->hi));
    }
    if (tap && tap->ids)
      CPSZ_CUDA_TRY(cudaMemcpyAsync(tap->ids, jobs[0].d.ids, 2 * jobs[0].N, cudaMemcpyDeviceToDevice, st));

    // ---- stage 2: one persistent wavefront over every field of the pass ----
    mark(ctx, "wave2d_compress");
    if (overlap) {
      // the bounds are done: the rest of each SM joins the running wavefront
      CPSZ_TRY(launch_wave2d(ctx, false, d_fields, d_items, n_items, queue, pass_points, st, WAVE_JOIN));
      CPSZ_CUDA_TRY(cudaStreamWaitEvent(st, ctx->ev[4], 0));
      // the flag as the wavefront left it, read by the host once the code
      // histograms (enqueued after it) have arrived
      CPSZ_CUDA_TRY(cudaMemcpyAsync(wave_flag_snapshot(ctx), ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, st));
      CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[1], st));
    } else {
      CPSZ_TRY(launch_wave2d(ctx, false, d_fields, d_items, n_items, queue, pass_points));
    }
    return CPSZ_OK;
  };
  auto count_codes = [&]() -> int {
    CPSZ_TRY(launch_hist_u16(ctx, hist_jobs.data(), P.hist, nj, hist_ctas));
    CPSZ_TRY(launch_hist_list(ctx, P.list, 2 * nj, st));
    CPSZ_CUDA_TRY(record(ctx->ev[6]));
    return CPSZ_OK;
  };
  bool hist_in_stage3 = !follow;
  auto stage_3 = [&]() -> int {
    mark(ctx, "blocks+hist+unpred");

    // ---- stage 3: code histograms first (the host builds the code trees from
    // them while the GPU converts to block order and gathers unpredictables);
    // a single field beside its bounds has them from the follower ----
    if (hist_in_stage3) CPSZ_TRY(count_codes());
    CPSZ_TRY(launch_strip_pass(ctx, strip_jobs.data(), P.strip, nj));
    CPSZ_CUDA_TRY(record(ctx->ev[5]));  // the unpredictable counts are on the host
    return CPSZ_OK;
  };
  const bool use_graph = nj > 1 && all_dev_in && !tap && !ctx->timing && !overlap;
  bool done = false;
  if (use_graph) {
    std::vector<uint64_t> key = {(uint64_t)nj, (uint64_t)(uintptr_t)ctx->arena.base, (uint64_t)(uintptr_t)ctx->pinned,
                                 tune_generation()};
    for (const Job2D& j : jobs) {
      uint64_t ebits;
      memcpy(&ebits, &j.eb, 8);
      key.insert(key.end(), {(uint64_t)(uintptr_t)j.U_in, (uint64_t)(uintptr_t)j.V_in, (uint64_t)j.r1,
                             (uint64_t)j.r2, ebits});
    }
    auto& cache = ctx->pass_graphs;
    auto hit = std::find_if(cache.begin(), cache.end(), [&](const cpsz_b200_ctx::PassGraph& g) { return g.key == key; });
    if (hit != cache.end()) {
      std::rotate(hit, hit + 1, cache.end());  // most recently used last
      CPSZ_CUDA_TRY(cudaGraphLaunch(cache.back().exec, st));
      count_launch(ctx, cache.back().launches);
      ctx->graph_replays++;
      done = true;
    } else {
      if (cache.size() >= cpsz_b200_ctx::kMaxPassGraphs) {
        cudaGraphExecDestroy(cache.front().exec);
        cache.erase(cache.begin());
      }
      const uint64_t launches0 = ctx->launches;
      if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        capturing = true;
        int rc = stages_1_2();
        if (rc == CPSZ_OK) rc = stage_3();
        capturing = false;
        cudaGraph_t graph = nullptr;
        const cudaError_t e = cudaStreamEndCapture(st, &graph);
        cudaGraphExec_t exec = nullptr;
        if (rc == CPSZ_OK && e == cudaSuccess && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess) {
          cache.push_back(cpsz_b200_ctx::PassGraph{key, exec, (int)(ctx->launches - launches0)});
          done = cudaGraphLaunch(exec, st) == cudaSuccess;
          ctx->graph_captures += done;
        }
        if (graph) cudaGraphDestroy(graph);
      }
      if (!done) {
        // capture unavailable or failed: the same work, launched directly
        cudaGetLastError();
        clear_error();
        ctx->launches = launches0;
      }
    }
  }
  if (!done) {
    CPSZ_TRY(stages_1_2());
    if (tap && tap->recon_only) {
      int flag = 0;
      CPSZ_TRY(read_flag(ctx, &flag));
      return flag ? flag_error(flag) : CPSZ_OK;
    }
    CPSZ_TRY(stage_3());
  }
  mark(ctx, "host_trees");
  // Host output (one field): the sections are copied from their device
  // buffers straight into the caller's memory, each right after its producer
  // when that memory is page-locked (the copies then overlap the rest), else
  // once everything is done; no blob is assembled in device memory.
  Job2D* hj = (nj == 1 && jobs[0].host_out) ? &jobs[0] : nullptr;
  const bool h_async = hj && host_kind(hj->host_out) == HOST_PINNED;
  // Page-locked output: each section's copy runs on the aux stream behind its
  // producer, so the next producer does not wait for it.  The main stream
  // joins aux before the pass ends; on an early return the guard drains aux, so
  // no copy out of the workspace outlives the call.
  struct AuxDrain {
    cudaStream_t s = nullptr;
    ~AuxDrain() {
      if (s) cudaStreamSynchronize(s);
    }
  } aux_drain;
  auto d2h_beside = [&](void* dst, const void* src, size_t n) -> int {
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[6], st));
    CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->ev[6], 0));
    aux_drain.s = ctx->aux;
    return d2h(ctx, dst, src, n, ctx->aux);
  };
  // Bit packing of stream k (0: ids, 1-2: codes of U / V).  A device blob gets
  // the bits in place, at byte `at` (the sections around it are written
  // byte by byte, and the packer ORs only zero bits into their bytes); host
  // output packs into a buffer of the stream's own that is copied out.
  auto add_stream = [&](PackGroup& G, Job2D& j, int k, size_t at) {
    uint8_t* dst = j.host_out ? (uint8_t*)j.d.bits[k] : j.blob_base + at;
    const size_t room = j.host_out ? (k ? j.codes_bits_cap : j.ids_bits_cap) : j.blob_room - at;
    G.add(j.cb[k], k ? (const void*)j.d.cblocks[k - 1] : (const void*)j.d.ids, k ? 2 : 1, k == 0, j.n_syms(k), dst,
          j.bits_bytes[k], room, j.d.enc_code[k], j.d.enc_len[k], j.d.enc_tmp[k]);
  };

  // host: the id trees (their histograms arrive with the bounds); a large
  // field's ids are packed on the aux stream as soon as the bounds are done:
  // that runs beside the wavefront's tail, which leaves most SMs idle, and the
  // main stream joins aux before the blob is finished
  const bool early_ids = nj == 1 && jobs[0].N >= EARLY_IDS_POINTS;
  auto tree_failure = [&]() {
    int fl = 0;
    CPSZ_TRY(read_flag(ctx, &fl));
    if (fl) return flag_error(fl);
    return set_error(CPSZ_ERR_UNSUPPORTED, "Huffman tree construction failed (code longer than 64 bits)");
  };
  CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[0]));
  host_parallel_for(nj, [&](int k) { jobs[k].tree_ok[0] = huff_build(jobs[k].h_hist_ids, 256, 2048, &jobs[k].cb[0]); });
  for (Job2D& j : jobs) {
    if (!j.tree_ok[0]) return tree_failure();
    j.sec_bytes[0] = huff_section_bytes(j.cb[0]);
    j.bits_bytes[0] = (j.cb[0].total_bits + 7) / 8;
    if (j.bits_bytes[0] + 8 > j.ids_bits_cap) return set_error(CPSZ_ERR_UNSUPPORTED, "Huffman stream larger than its bound");
  }
  if (early_ids) {
    Job2D& j = jobs[0];
    CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->ev[0], 0));
    aux_drain.s = ctx->aux;
    // the setup image has been copied (ev[0] follows it), so its staging is
    // free; the later uploads are staged behind these entries
    CPSZ_TRY(upload_reserve(ctx, EARLY_UP));
    UpImage up{(uint8_t*)ctx->up_pinned, P.up_ids, EARLY_UP};
    PackGroup G;
    add_stream(G, j, 0, ids_bits_at(j));
    CPSZ_TRY(G.stage(up, ctx->num_sms));
    OnStream on_aux(ctx, ctx->aux);
    CPSZ_TRY(up.send(ctx->aux));
    CPSZ_TRY(G.launch(ctx));
    if (h_async) {
      const size_t at = ids_bits_at(j);
      if (at + j.bits_bytes[0] > j.host_cap)
        return set_error(CPSZ_ERR_INVALID, "output capacity %zu too small for the blob", j.host_cap);
      CPSZ_TRY(d2h(ctx, j.host_out + at, j.d.bits[0], j.bits_bytes[0], ctx->aux));
    }
  }
  // code trees, as soon as the histograms' lists are on the host
  auto code_trees = [&]() -> int {
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[6]));
    host_parallel_for(2 * nj, [&](int q) {
      Job2D& j = jobs[q / 2];
      const int f = q % 2;
      j.tree_ok[1 + f] = huff_build_list(j.h_list[f], j.h_nlist[f], 65536, 131072, &j.cb[1 + f]);
    });
    return CPSZ_OK;
  };
  if (follow) {
    // the follower's histograms; one that gave up (its wavefront was not
    // running beside it) leaves them to be counted here
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[6]));
    if (*(volatile int*)follow_flag_snapshot(ctx)) {
      for (int f = 0; f < 2; f++) CPSZ_CUDA_TRY(cudaMemsetAsync(jobs[0].d.hist_codes[f], 0, 65536 * 8, st));
      CPSZ_TRY(count_codes());
    }
  }
  CPSZ_TRY(code_trees());
  if (overlap) {
    // The histograms are on the host, so is the flag snapshot taken before
    // them.  A wavefront wait that gave up (the bound kernel was held back
    // for seconds: a saturated or time-sliced device) left codes from
    // incomplete inputs; the bounds are complete now, so the wavefront and
    // everything after it runs again, after the bounds, and the pass goes on.
    // The id stream's packing, already enqueued, depends on the bounds only.
    CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[1]));
    const int snap = *(volatile int*)wave_flag_snapshot(ctx);
    if (snap & FLAG_TIMEOUT) {
      if (snap != FLAG_TIMEOUT) return flag_error(snap);
      CPSZ_CUDA_TRY(cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), st));
      for (WaveField& F : hf) {
        F.unit_done = nullptr;
        F.group_done = nullptr;
      }
      CPSZ_CUDA_TRY(cudaMemcpyAsync(P.fields, hf.data(), hf.size() * sizeof(WaveField), cudaMemcpyHostToDevice, st));
      for (Job2D& j : jobs) {
        CPSZ_CUDA_TRY(cudaMemsetAsync(j.d.gbnd, 0, 2 * j.ngroups * wave_gbnd_pitch(j.r2) * 8, st));
        for (int f = 0; f < 2; f++) {
          CPSZ_CUDA_TRY(cudaMemsetAsync(j.d.hist_codes[f], 0, 65536 * 8, st));
          CPSZ_CUDA_TRY(cudaMemsetAsync(j.d.strip[f], 0, strip_scratch_bytes(j.r1, j.r2), st));
        }
      }
      CPSZ_CUDA_TRY(cudaMemsetAsync(queue, 0, 64, st));
      CPSZ_TRY(launch_wave2d(ctx, false, d_fields, d_items, n_items, queue, pass_points));
      hist_in_stage3 = true;
      CPSZ_TRY(stage_3());
      CPSZ_TRY(code_trees());
      ctx->wave_reruns++;
    }
  }

  // ---- stage 4: blob layout (every section size is known once the
  // unpredictable counts are on the host) and bit packing of the codes ----
  mark(ctx, "huffman_encode");
  for (Job2D& j : jobs) {
    if (!j.tree_ok[1] || !j.tree_ok[2]) return tree_failure();
    for (int k = 1; k < 3; k++) {
      j.sec_bytes[k] = huff_section_bytes(j.cb[k]);
      j.bits_bytes[k] = (j.cb[k].total_bits + 7) / 8;
      if (j.bits_bytes[k] + 8 > j.codes_bits_cap)
        return set_error(CPSZ_ERR_UNSUPPORTED, "Huffman stream larger than its bound");
    }
  }
  CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[5]));
  std::vector<BlobLayout> lay(nj);
  size_t all_bytes = 0;
  for (int q = 0; q < nj; q++) {
    Job2D& j = jobs[q];
    j.n_unpred[0] = j.h_nunpred[0];
    j.n_unpred[1] = j.h_nunpred[1];
    CPSZ_TRY(job_layout(j, lay[q]));
    all_bytes += lay[q].total;
    if (j.host_out) {
      if (lay[q].total > j.host_cap)
        return set_error(CPSZ_ERR_INVALID, "output capacity %zu < blob size %zu", j.host_cap, lay[q].total);
    } else if (lay[q].total > j.blob_cap) {
      return set_error(CPSZ_ERR_UNSUPPORTED, "blob larger than its bound");
    }
  }
  // every size is known now: blobs with room in the caller's device memory are
  // built there (8 bytes over: the packers touch the last word of a stream)
  if (!early_ids && dev_at && all_bytes + 8 <= dev_room) {
    size_t at = 0;
    for (int q = 0; q < nj; q++) {
      jobs[q].blob_base = dev_at + at;
      jobs[q].blob_room = dev_room - at;
      at += lay[q].total;
    }
  }
  if (hj) {
    const BlobLayout& hl = lay[0];
    for (const BlobLayout::Piece& pc : hl.pieces) {
      if (pc.zero) memset(hj->host_out + pc.dst, 0, pc.n);
      else memcpy(hj->host_out + pc.dst, pc.ext ? pc.ext : hl.small.data() + pc.src, pc.n);
    }
    if (h_async)
      for (int f = 0; f < 2; f++) {
        CPSZ_TRY(d2h_beside(hj->host_out + hl.unpred_dst[f], hj->d.unpred[f], 4 * hj->n_unpred[f]));
        if (hl.sign_bytes)
          CPSZ_TRY(d2h_beside(hj->host_out + hl.sign_dst + f * hl.sign_bytes, hj->d.signs[f], hl.sign_bytes));
      }
  }
  // The streams still to be packed, in one launch; or, to page-locked host
  // output, one by one, each copied out while the next is packed.
  const int k_first = early_ids ? 1 : 0;
  std::vector<PackGroup> groups(h_async ? 3 - k_first : 1);
  for (int q = 0; q < nj; q++)
    for (int k = k_first; k < 3; k++) add_stream(groups[h_async ? k - k_first : 0], jobs[q], k, lay[q].bit_dst[k]);
  // page-locked staging of the pass's remaining uploads, behind the early id
  // entries' (whose copy may still be in flight)
  const size_t early_up = early_ids ? align_up(EARLY_UP, 256) : 0;
  size_t up_bytes = 1024;
  for (const PackGroup& G : groups) up_bytes += G.up_bytes();
  for (const BlobLayout& L : lay) up_bytes += piece_up_bytes(L);
  if (up_bytes > P.up_bytes) return set_error(CPSZ_ERR_INVALID, "internal: uploads exceed their bound");
  if (early_ids && ctx->up_cap < early_up + up_bytes) CPSZ_CUDA_TRY(cudaStreamSynchronize(ctx->aux));
  CPSZ_TRY(upload_reserve(ctx, early_up + up_bytes));
  UpImage up{(uint8_t*)ctx->up_pinned + early_up, P.up, up_bytes};
  for (PackGroup& G : groups) CPSZ_TRY(G.stage(up, ctx->num_sms));
  // the rest of a device blob (header, trees, unpredictable values, sign
  // maps): uploaded with the entries, or, for a large field, staged once the
  // packers are running
  std::vector<CopyPiece> pieces;
  uint8_t* d_pieces = nullptr;
  unsigned piece_ctas = 0;
  auto stage_pieces = [&]() -> int {
    for (int q = 0; q < nj; q++) CPSZ_TRY(job_pieces(jobs[q], lay[q], up, pieces));
    piece_ctas = assign_piece_chunks(pieces.data(), pieces.size());
    uint8_t* h = up.take(pieces.size() * sizeof(CopyPiece), &d_pieces);
    if (!h) return up_overrun();
    memcpy(h, pieces.data(), pieces.size() * sizeof(CopyPiece));
    return CPSZ_OK;
  };
  if (!hj && !early_ids) CPSZ_TRY(stage_pieces());
  CPSZ_TRY(up.send(st));
  for (size_t g = 0; g < groups.size(); g++) {
    CPSZ_TRY(groups[g].launch(ctx));
    if (h_async) {
      const int k = k_first + (int)g;
      CPSZ_TRY(d2h_beside(hj->host_out + lay[0].bit_dst[k], hj->d.bits[k], hj->bits_bytes[k]));
    }
  }
  if (aux_drain.s) {  // the aux stream's work (id packing, section copies) joins the main stream
    CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[7], ctx->aux));
    CPSZ_CUDA_TRY(cudaStreamWaitEvent(st, ctx->ev[7], 0));
  }
  // ---- stage 5: the rest of a device blob, or, for host output without
  // page-locked memory, the sections not yet copied ----
  mark(ctx, "blob_assembly");
  int assembled = CPSZ_OK;
  if (!hj) {
    if (early_ids) {
      assembled = stage_pieces();
      if (assembled == CPSZ_OK) assembled = up.send(st);
    }
    if (assembled == CPSZ_OK)
      assembled = launch_copy_pieces(ctx, (const CopyPiece*)d_pieces, (int)pieces.size(), piece_ctas);
  }
  {
    int flag = 0;
    CPSZ_TRY(read_flag(ctx, &flag));  // synchronizes the stream; a kernel's error outranks the assembly's
    if (flag) return flag_error(flag);
  }
  if (assembled != CPSZ_OK) return assembled;
  if (hj) {
    const BlobLayout& hl = lay[0];
    if (!h_async) {
      CPSZ_TRY(d2h(ctx, hj->host_out + hl.bit_dst[0], hj->d.bits[0], hj->bits_bytes[0], st));
      for (int f = 0; f < 2; f++) {
        CPSZ_TRY(d2h(ctx, hj->host_out + hl.unpred_dst[f], hj->d.unpred[f], 4 * hj->n_unpred[f], st));
        if (hl.sign_bytes)
          CPSZ_TRY(d2h(ctx, hj->host_out + hl.sign_dst + f * hl.sign_bytes, hj->d.signs[f], hl.sign_bytes, st));
      }
      for (int k = 1; k < 3; k++) CPSZ_TRY(d2h(ctx, hj->host_out + hl.bit_dst[k], hj->d.bits[k], hj->bits_bytes[k], st));
    }
    hj->size = hl.total;
  }
  mark(ctx, "end");
  if (tap) {
    Job2D& j = jobs[0];
    for (int f = 0; f < 2; f++) {
      if (tap->codes_blocks[f])
        CPSZ_CUDA_TRY(cudaMemcpyAsync(tap->codes_blocks[f], j.d.cblocks[f], 2 * j.N, cudaMemcpyDeviceToDevice, st));
      if (tap->unpred[f] && j.n_unpred[f])
        CPSZ_CUDA_TRY(
            cudaMemcpyAsync(tap->unpred[f], j.d.unpred[f], 4 * j.n_unpred[f], cudaMemcpyDeviceToDevice, st));
    }
  }
  return CPSZ_OK;
}

// Workspace and page-locked staging of a pass (its pieces are placed by run_pass).
int pass_reserve(cpsz_b200_ctx* ctx, std::vector<Job2D>& jobs) {
  PassBuf P{};
  Alloc count{nullptr};
  pass_alloc(jobs, P, count);
  CPSZ_TRY(arena_reserve(ctx, count.bytes));
  return pinned_reserve(ctx, PINNED_BASE + jobs.size() * (ID_HIST + JOB_PINNED));
}

}  // namespace

int build_wave_items(int nfields, const int* r1s, std::vector<WaveItem>& items) {
  int maxg = 0;
  for (int f = 0; f < nfields; f++) maxg = std::max(maxg, (r1s[f] + WAVE_GROUP_ROWS - 1) / WAVE_GROUP_ROWS);
  items.clear();
  for (int g = 0; g < maxg; g++)
    for (int f = 0; f < nfields; f++)
      if (g * WAVE_GROUP_ROWS < r1s[f]) items.push_back(WaveItem{f, g});
  return (int)items.size();
}

int compress_2d(cpsz_b200_ctx* ctx, const float* U_in, const float* V_in, size_t r1s, size_t r2s, double max_pwr_eb,
                Blob2D* out, const StageTap* tap, const double* eb_ext, unsigned char* host_out, size_t host_cap,
                bool log_form) {
  if (log_form && (tap || eb_ext))
    return set_error(CPSZ_ERR_INVALID, "the offline_log form takes neither stage taps nor given bounds");
  std::vector<Job2D> jobs(1);
  CPSZ_TRY(job_init(jobs[0], U_in, V_in, r1s, r2s, max_pwr_eb));
  jobs[0].log_form = log_form;
  jobs[0].eb_ext = eb_ext;
  if (host_out && host_kind(host_out) == HOST_DEVICE) {
    if (on_ctx_device(ctx, host_out)) {  // (another device's memory gets a copy)
      jobs[0].dev_out = host_out;
      jobs[0].dev_cap = host_cap;
    }
  } else {
    jobs[0].host_out = host_out;
    jobs[0].host_cap = host_cap;
  }
  CPSZ_TRY(pass_reserve(ctx, jobs));
  CPSZ_TRY(run_pass(ctx, jobs, tap, jobs[0].dev_out, jobs[0].dev_cap));
  out->d_blob = jobs[0].host_out ? nullptr : jobs[0].blob_base;
  out->size = jobs[0].size;
  out->n_unpred[0] = jobs[0].n_unpred[0];
  out->n_unpred[1] = jobs[0].n_unpred[1];
  return CPSZ_OK;
}

int compress_2d_batch(cpsz_b200_ctx* ctx, int n, const float* const* U, const float* const* V, const size_t* r1,
                      const size_t* r2, const double* ebs, unsigned char* out, size_t out_cap, size_t* offsets) {
  if (n < 0 || (n > 0 && (!U || !V || !r1 || !r2 || !ebs))) return set_error(CPSZ_ERR_INVALID, "null batch argument");
  if (!out || !offsets) return set_error(CPSZ_ERR_INVALID, "null output");
  const bool dev_out = on_ctx_device(ctx, out);
  size_t at = 0;
  int k0 = 0;
  offsets[0] = 0;
  while (k0 < n) {
    // greedy pass: up to BATCH_MAX_FIELDS fields and BATCH_MAX_POINTS points (a larger field goes alone)
    std::vector<Job2D> jobs;
    size_t pts = 0;
    int k = k0;
    while (k < n && (int)jobs.size() < BATCH_MAX_FIELDS) {
      Job2D j;
      CPSZ_TRY(job_init(j, U[k], V[k], r1[k], r2[k], ebs[k]));
      if (!jobs.empty() && pts + j.N > BATCH_MAX_POINTS) break;
      pts += j.N;
      jobs.push_back(std::move(j));
      k++;
    }
    CPSZ_TRY(pass_reserve(ctx, jobs));
    CPSZ_TRY(run_pass(ctx, jobs, nullptr, dev_out && at < out_cap ? out + at : nullptr, at < out_cap ? out_cap - at : 0));
    for (size_t q = 0; q < jobs.size(); q++) {
      const Job2D& j = jobs[q];
      if (at + j.size > out_cap)
        return set_error(CPSZ_ERR_INVALID, "output capacity %zu < %zu bytes of blobs", out_cap, at + j.size);
      if (j.blob_base != out + at) CPSZ_TRY(d2h(ctx, out + at, j.blob_base, j.size, ctx->stream));
      at += j.size;
      offsets[k0 + q + 1] = at;
    }
    // the next pass reuses the workspace
    CPSZ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    k0 = k;
  }
  return CPSZ_OK;
}

// ---- decompression ---------------------------------------------------------------

static int* again_snapshot(cpsz_b200_ctx* ctx) { return (int*)((char*)ctx->pinned + 2064); }

int probe_decode_again(cpsz_b200_ctx* ctx) {
  CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[0], ctx->stream));
  CPSZ_CUDA_TRY(cudaStreamWaitEvent(ctx->aux, ctx->ev[0], 0));
  CPSZ_CUDA_TRY(cudaMemcpyAsync(again_snapshot(ctx), ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->aux));
  CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[1], ctx->aux));
  return CPSZ_OK;
}

int seen_decode_again(cpsz_b200_ctx* ctx, bool* again) {
  CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[1]));
  *again = (*(volatile int*)again_snapshot(ctx) & FLAG_HUFF_RESYNC) != 0;
  return CPSZ_OK;
}

namespace {

struct FieldView {
  size_t n_unpred;
  size_t unpred_off;  // from blob start
  HuffDecoderHost huff;
  size_t huff_off;
};

int parse_field(const unsigned char* blob, size_t off, size_t size, size_t N, size_t nblocks, FieldView* fv) {
  if (size < FIELD_HDR) return set_error(CPSZ_ERR_FORMAT, "field blob truncated");
  const unsigned char* p = blob + off;
  int bs, radius;
  memcpy(&bs, p, 4);
  memcpy(&radius, p + 5, 4);
  unsigned char use_mean = p[9];
  unsigned long long reg_count, nu;
  memcpy(&reg_count, p + 17, 8);
  memcpy(&nu, p + 25, 8);
  if (bs != BS || radius != 32768 || use_mean != 0 || reg_count != 0)
    return set_error(CPSZ_ERR_UNSUPPORTED,
                     "field blob parameters (block %d, radius %d, mean %d, regression %llu) are not the offline "
                     "compressor's",
                     bs, radius, (int)use_mean, reg_count);
  if (nu > N || 4 * nu > size - FIELD_HDR) return set_error(CPSZ_ERR_FORMAT, "unpredictable count %llu invalid", nu);
  fv->n_unpred = nu;
  fv->unpred_off = off + FIELD_HDR;
  size_t ind = (nblocks - 1) / 8 + 1;
  size_t hoff = FIELD_HDR + 4 * nu + ind;
  if (hoff > size) return set_error(CPSZ_ERR_FORMAT, "field blob truncated before its Huffman section");
  if (!huff_parse(p + hoff, size - hoff, 65535, &fv->huff)) return CPSZ_ERR_FORMAT;
  fv->huff_off = off + hoff;
  return CPSZ_OK;
}

}  // namespace

int decompress_2d(cpsz_b200_ctx* ctx, const unsigned char* blob, size_t blob_size, size_t r1s, size_t r2s, float* U_out,
                  float* V_out, bool log_form) {
  if (!blob || !U_out || !V_out) return set_error(CPSZ_ERR_INVALID, "null pointer argument");
  if (r1s == 0 || r2s == 0) return set_error(CPSZ_ERR_INVALID, "empty field");
  if (r1s > (1u << 30) || r2s > (1u << 30) || r1s * r2s > (size_t)INT32_MAX)
    return set_error(CPSZ_ERR_UNSUPPORTED, "field of %zu x %zu points exceeds 2^31 points", r1s, r2s);
  if (blob_size < BLOB_HDR) return set_error(CPSZ_ERR_FORMAT, "blob shorter than its header");
  const int r1 = (int)r1s, r2 = (int)r2s;
  const size_t N = r1s * r2s;
  const int nby = (r2 - 1) / BS + 1, nbx = (r1 - 1) / BS + 1;
  const size_t nblocks = (size_t)nbx * nby;
  const int ngroups = (r1 + WAVE_GROUP_ROWS - 1) / WAVE_GROUP_ROWS;
  int base;
  double thr;
  unsigned long long eb_size, u_size, v_size;
  memcpy(&base, blob, 4);
  memcpy(&thr, blob + 4, 8);
  memcpy(&eb_size, blob + 12, 8);
  memcpy(&u_size, blob + 20, 8);
  memcpy(&v_size, blob + 28, 8);
  if (base != (log_form ? 2 : 4) || thr != DBL_EPSILON)
    return set_error(CPSZ_ERR_UNSUPPORTED, "blob quantizer (base %d, thr %g) is not the offline%s compressor's", base,
                     thr, log_form ? "_log" : "");
  // offline_log: the sign maps of U and V follow the id section
  const size_t sign_bytes = log_form ? (N - 1) / 8 + 1 : 0;
  const size_t avail = blob_size - BLOB_HDR;
  if (eb_size > avail || 2 * sign_bytes > avail - eb_size || u_size > avail - eb_size - 2 * sign_bytes ||
      v_size > avail - eb_size - 2 * sign_bytes - u_size)
    return set_error(CPSZ_ERR_FORMAT, "section sizes exceed the blob");
  const size_t fields_at = BLOB_HDR + eb_size + 2 * sign_bytes;
  const size_t n_ids = log_form ? N : 2 * N;
  HuffDecoderHost hid;
  if (!huff_parse(blob + BLOB_HDR, eb_size, 2047, &hid)) return CPSZ_ERR_FORMAT;
  if (hid.section_bytes > eb_size) return set_error(CPSZ_ERR_FORMAT, "id section overruns");
  if (hid.max_sym > (uint32_t)ID_MAX_2D)
    return set_error(CPSZ_ERR_UNSUPPORTED, "error-bound id %u beyond the supported range (<= %d)", hid.max_sym,
                     ID_MAX_2D);
  FieldView fv[2];
  CPSZ_TRY(parse_field(blob, fields_at, u_size, N, nblocks, &fv[0]));
  CPSZ_TRY(parse_field(blob, fields_at + u_size, v_size, N, nblocks, &fv[1]));
  LibmTables libm{};
  if (log_form) CPSZ_TRY(libm_tables_device(ctx, &libm));
  const bool dev_out = is_device_ptr(U_out) && is_device_ptr(V_out);

  // ---- workspace: what goes up (one image), what starts at zero, the rest ----
  int r1v[2] = {r1, r1};
  std::vector<WaveItem> items;
  const int n_items = build_wave_items(2, r1v, items);
  WaveField hf[2] = {};
  const HuffDecoderHost* hs[3] = {&hid, &fv[0].huff, &fv[1].huff};
  const size_t sec_at[3] = {BLOB_HDR, fv[0].huff_off, fv[1].huff_off};
  Upload up;
  const size_t up_fields = up.add(hf, sizeof(hf)), up_items = up.add(items.data(), n_items * sizeof(WaveItem));
  size_t up_tree[3], up_bits[3], up_unpred[2];
  for (int k = 0; k < 3; k++) up_tree[k] = up.add(blob + sec_at[k] + hs[k]->tree_offset, hs[k]->tree_bytes);
  const size_t up_signs = up.add(blob + BLOB_HDR + eb_size, 2 * sign_bytes);
  up_bits[0] = up.add(blob + sec_at[0] + hid.bits_offset, hid.nbytes, HUFF_DEC_PAD);
  up.cut();
  for (int f = 0; f < 2; f++) {
    up_bits[1 + f] = up.add(blob + sec_at[1 + f] + hs[1 + f]->bits_offset, hs[1 + f]->nbytes, HUFF_DEC_PAD);
    up_unpred[f] = up.add(blob + fv[f].unpred_off, 4 * fv[f].n_unpred);
    up.cut();
  }
  HuffDecJob dec[3];
  for (int k = 0; k < 3; k++) {
    dec[k].nbytes = hs[k]->nbytes;
    dec[k].node_count = hs[k]->node_count;
    dec[k].root_is_leaf = hs[k]->root_is_leaf;
    dec[k].root_sym = hs[k]->root_sym;
    dec[k].n = k ? N : n_ids;
    dec[k].out_bytes = k ? 2 : 1;
  }
  // a small blob goes up and is decoded in one piece, a large one stream by
  // stream, each decoded while the next one goes up
  const bool whole = up.bytes() <= UPLOAD_WHOLE;
  size_t dec_bytes[3];
  for (int k = 0; k < 3; k++) dec_bytes[k] = whole ? (k ? 0 : huff_decode_tmp_bytes(dec, 3)) : huff_decode_tmp_bytes(&dec[k], 1);
  const size_t strip_bytes = align_up(strip_scratch_bytes(r1, r2), 256), gbnd_bytes = 2 * ngroups * wave_gbnd_pitch(r2) * 8;
  const size_t zero_bytes = 256 + 2 * strip_bytes + gbnd_bytes;
  size_t bytes = 0;
  auto add = [&](size_t b) { bytes += align_up(b, 256) + 256; };
  add(up.bytes());
  add(zero_bytes);
  for (int f = 0; f < 2; f++) {
    if (!dev_out) add(4 * N);
    add(2 * N);  // codes in block order
    add(8 * N);  // raster pairs
  }
  add(n_ids);
  for (int k = 0; k < 3; k++) add(dec_bytes[k]);
  CPSZ_TRY(arena_reserve(ctx, bytes));
  CPSZ_TRY(pinned_reserve(ctx, 4096));
  auto A = [&](size_t b) { return (uint8_t*)arena_alloc(ctx, b); };
  cudaStream_t st = ctx->stream;
  uint8_t* d_up = A(up.bytes());
  uint8_t* d_zero = A(zero_bytes);  // the wavefront's queue, strip scratch, boundary rows
  float* dU = dev_out ? U_out : (float*)A(4 * N);
  float* dV = dev_out ? V_out : (float*)A(4 * N);
  uint8_t* ids = A(n_ids);
  uint16_t* cblocks[2];
  float2* raw[2];  // (addend, raw flag) per point; .x holds the raw value where the code is 0
  for (int f = 0; f < 2; f++) {
    cblocks[f] = (uint16_t*)A(2 * N);
    raw[f] = (float2*)A(8 * N);
  }
  void* dtmp[3];
  for (int k = 0; k < 3; k++) dtmp[k] = A(dec_bytes[k]);
  if (!dtmp[2]) return set_error(CPSZ_ERR_NOMEM, "workspace layout overflow");
  void* strip[2] = {d_zero + 256, d_zero + 256 + strip_bytes};
  unsigned long long* gbnd = (unsigned long long*)(d_zero + 256 + 2 * strip_bytes);
  for (int k = 0; k < 3; k++) {
    dec[k].bits = d_up + up_bits[k];
    dec[k].tree = d_up + up_tree[k];
    dec[k].out = k ? (void*)cblocks[k - 1] : (void*)ids;
  }
  for (int f = 0; f < 2; f++) {
    WaveField& F = hf[f];
    F.pair = raw[f];
    F.out = f ? dV : dU;
    F.gbnd = gbnd + f * ngroups * wave_gbnd_pitch(r2);
    F.pair_pitch = r2;
    F.code_pitch = r2;
    F.out_pitch = r2;
    F.r1 = r1;
    F.r2 = r2;
  }
  uint8_t* d_signs = d_up + up_signs;
  unsigned int* h_cnt = (unsigned int*)ctx->pinned + 16;

  // a copy from the caller's page-locked blob must not outlive the call
  struct Drain {
    cudaStream_t s = nullptr;
    ~Drain() {
      if (s) cudaStreamSynchronize(s);
    }
  } aux_drain, main_drain;
  main_drain.s = st;

  // A stream whose subsequences did not settle in the decoder's fixed rounds
  // (FLAG_HUFF_RESYNC) is decoded again, with rounds until they have; what is
  // queued behind the first attempt then does nothing.
  for (int attempt = 0;; attempt++) {
    const bool settle = attempt > 0;
    CPSZ_CUDA_TRY(cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), st));
    CPSZ_CUDA_TRY(cudaMemsetAsync(d_zero, 0, zero_bytes, st));
    reset_marks(ctx);
    mark(ctx, "huffman_decode");
    if (whole || settle) {
      if (!settle) CPSZ_TRY(up.send_whole(ctx, d_up, st));
      if (whole) {
        CPSZ_TRY(launch_huff_decode(ctx, dec, 3, dtmp[0], settle));
      } else {
        for (int k = 0; k < 3; k++) CPSZ_TRY(launch_huff_decode(ctx, &dec[k], 1, dtmp[k], settle));
      }
    } else {
      aux_drain.s = ctx->aux;
      for (int k = 0; k < 3; k++) {
        CPSZ_TRY(up.send_part(ctx, d_up, k, ctx->aux));
        CPSZ_CUDA_TRY(cudaEventRecord(ctx->up_ev[k], ctx->aux));
        CPSZ_CUDA_TRY(cudaStreamWaitEvent(st, ctx->up_ev[k], 0));
        CPSZ_TRY(launch_huff_decode(ctx, &dec[k], 1, dtmp[k], false));
      }
    }
    const bool probe = !settle && !dev_out;
    if (probe) {
      aux_drain.s = ctx->aux;
      CPSZ_TRY(probe_decode_again(ctx));
    }
    // ---- raster pairs, unpredictable scatter ----
    mark(ctx, "raster+scatter");
    {
      const uint16_t* cb[2] = {cblocks[0], cblocks[1]};
      // offline_log: one id stream for both components, base 2
      const uint8_t* idf[2] = {ids, log_form ? ids : ids + N};
      const float* un[2] = {(const float*)(d_up + up_unpred[0]), (const float*)(d_up + up_unpred[1])};
      const unsigned long long nun[2] = {fv[0].n_unpred, fv[1].n_unpred};
      CPSZ_TRY(launch_strip_unpass(ctx, cb, idf, un, nun, r1, r2, raw, strip, h_cnt, log_form ? 1 : 2));
    }
    // ---- wavefront ----
    mark(ctx, "wave2d_decompress");
    CPSZ_TRY(launch_wave2d(ctx, true, (const WaveField*)(d_up + up_fields), (const WaveItem*)(d_up + up_items), n_items,
                           (int*)d_zero, (size_t)r1 * r2));
    if (log_form) {
      mark(ctx, "exp2d");
      CPSZ_TRY(launch_exp2d(ctx, dU, dV, d_signs, d_signs + sign_bytes, N, libm.exp2f));
    }
    mark(ctx, "d2h");
    if (probe) {
      bool again = false;
      CPSZ_TRY(seen_decode_again(ctx, &again));
      if (again) continue;
    }
    if (!dev_out) {
      CPSZ_TRY(d2h(ctx, U_out, dU, 4 * N, st));
      CPSZ_TRY(d2h(ctx, V_out, dV, 4 * N, st));
    }
    mark(ctx, "end");
    int flag = 0;
    CPSZ_TRY(read_flag(ctx, &flag));  // synchronizes the stream
    main_drain.s = nullptr;
    if ((flag & FLAG_HUFF_RESYNC) && !settle) continue;
    if (flag) return flag_error(flag);
    break;
  }
  for (int f = 0; f < 2; f++)
    if (h_cnt[f] != fv[f].n_unpred)
      return set_error(CPSZ_ERR_FORMAT, "field %d: %u zero codes but %zu unpredictable values", f, h_cnt[f],
                       fv[f].n_unpred);
  return CPSZ_OK;
}

}  // namespace cpsz
