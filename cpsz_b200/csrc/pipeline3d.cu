// pipeline3d.cu -- the 3D offline (log) compressor / decompressor on one GPU.
//
// Compress (sz_compress_cp_preserve_3d_offline_log<float>,
// src/sz_compress_cp_preserve_3d.cpp:360-581):
//   eb3d (bounds, ids) -> log3d (log2f, signs) -> Lorenzo planes (codes)
//   -> raster compaction (codes, unpredictable triples, final ids, id
//   histogram) + code histogram -> host Huffman trees -> GPU bit packing
//   -> blob assembled in device memory.
// Decompress (sz_decompress_cp_preserve_3d_online_log<float>,
// src/sz_decompress_cp_preserve_3d.cpp:7-110): host header/tree parsing ->
// GPU Huffman decode of ids and codes -> per-point addends / raw values ->
// Lorenzo planes with exp2f and signs fused.
//
// Blob layout (src/sz_compress_cp_preserve_3d.cpp:559-578):
//   int base (2) | int radius (32768) | 3 sign bitmaps of ceil(N/8) bytes
//   | size_t n_unpred | float[n_unpred] | size_t N | HUF(ids, 512 states)
//   | size_t n_codes | HUF(codes, 131072 states)
// For a field without predictable points the code section holds a one-leaf
// tree of symbol 0 and no bits (the reference cannot encode zero symbols).
#include <cstring>
#include <vector>

#include "huffman_host.h"
#include "kernels.h"
#include "pack_group.h"
#include "transfer.h"
#include "pipeline.h"

namespace cpsz {

namespace {

int read_flag3(cpsz_b200_ctx* ctx, int* out) {
  CPSZ_CUDA_TRY(cudaMemcpyAsync(ctx->pinned, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CPSZ_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  *out = *(int*)ctx->pinned;
  return CPSZ_OK;
}

int flag_error3(int flag) {
  if (flag & FLAG_ID_OVERFLOW)
    return set_error(CPSZ_ERR_UNSUPPORTED,
                     "an error-bound id reaches the reference's unpredictable marker 24 (max_pwr_eb >= 3)");
  if (flag & FLAG_RAW_RANGE) return set_error(CPSZ_ERR_FORMAT, "code or unpredictable stream shorter than its ids");
  if (flag & (FLAG_HUFF_CORRUPT | FLAG_HUFF_RESYNC)) return set_error(CPSZ_ERR_FORMAT, "Huffman stream does not decode");
  if (flag & FLAG_OUT_CAPACITY) return set_error(CPSZ_ERR_INVALID, "an output stream exceeded its buffer");
  if (flag & FLAG_TIMEOUT) return set_error(CPSZ_ERR_TIMEOUT, "a bounded device-side wait gave up");
  return set_error(CPSZ_ERR_CUDA, "device flag %d", flag);
}

int check_dims(size_t r1, size_t r2, size_t r3) {
  if (r1 == 0 || r2 == 0 || r3 == 0) return set_error(CPSZ_ERR_INVALID, "empty field (%zu x %zu x %zu)", r1, r2, r3);
  if (r1 > (1u << 30) || r2 > (1u << 30) || r3 > (1u << 30) || r1 * r2 > (size_t)INT32_MAX ||
      r1 * r2 * r3 > ((size_t)1 << 32))
    return set_error(CPSZ_ERR_UNSUPPORTED, "field of %zu x %zu x %zu points is beyond 2^32 points", r1, r2, r3);
  return CPSZ_OK;
}

}  // namespace

int compress_3d(cpsz_b200_ctx* ctx, const float* U_in, const float* V_in, const float* W_in, size_t r1s, size_t r2s,
                size_t r3s, double max_pwr_eb, Blob3D* out, unsigned char* dev_out, size_t dev_cap) {
  if (!U_in || !V_in || !W_in) return set_error(CPSZ_ERR_INVALID, "null input field");
  CPSZ_TRY(check_dims(r1s, r2s, r3s));
  if (max_pwr_eb != max_pwr_eb) return set_error(CPSZ_ERR_INVALID, "max_pwr_eb is NaN");
  const int r1 = (int)r1s, r2 = (int)r2s, r3 = (int)r3s;
  const size_t N = r1s * r2s * r3s;
  const size_t smap = (N - 1) / 8 + 1;
  const size_t sign_words = (N + 31) / 32;
  const size_t nchunks = chunk_count(N);
  const bool dev_in = is_device_ptr(U_in) && is_device_ptr(V_in) && is_device_ptr(W_in);
  const QuantTable& qt = quant_table_3d();
  LibmTables lt;
  CPSZ_TRY(libm_tables_device(ctx, &lt));

  size_t bytes = 0;
  auto add = [&](size_t b) { bytes += align_up(b, 256) + 256; };
  if (!dev_in) add(12 * N);
  add(N);              // ids
  add(std::max(16 * N, eb3d_scratch_bytes(N)));  // pairs
  add(16 * N);         // reconstruction
  add(8 * N);          // codes per point
  add(2 * (nchunks + 1) * 4);
  add(scan_u32_tmp_bytes(nchunks));
  add(6 * N);          // compacted codes
  add(12 * N);         // unpredictable triples
  add(3 * sign_words * 4);
  add(wave3d_scratch_bytes(r1, r2));
  // zeroed in one piece: both histograms, the packers' look-back words
  const size_t tmp_ids = align_up(huff_encode_tmp_bytes(N), 256);
  const size_t zero_bytes = 256 * 8 + 65536 * 8 + tmp_ids + huff_encode_tmp_bytes(3 * N);
  add(zero_bytes);
  const size_t image_bytes = QUANT_TAB_MAX * 8 + sizeof(HistList);
  add(image_bytes);
  add(256 * 9);
  add(65536 * 9);
  const size_t syms = std::min<size_t>(65536, 3 * N + 1), tree = 12 + 13 * std::min<size_t>(131072, 2 * syms) + 8;
  const size_t up_cap = (256 + syms) * sizeof(HuffEntry) + tree + 12 + 13 * 512 + 4096;
  add(up_cap);
  const size_t ids_bits_cap = (N * 8 + 7) / 8 + 64;
  const size_t codes_bits_cap = (3 * N * 17 + 7) / 8 + 64;
  const size_t blob_cap = 8 + 3 * smap + 8 + 12 * N + 8 + 8 + 2 * (12 + 13 * 131072 + 8) + ids_bits_cap +
                          codes_bits_cap + 4096;
  add(blob_cap);
  CPSZ_TRY(arena_reserve(ctx, bytes));
  CPSZ_TRY(pinned_reserve(ctx, 65536 * 8 + 256 * 8 + 4096));
  auto A = [&](size_t b) { return arena_alloc(ctx, b); };
  cudaStream_t st = ctx->stream;
  const float *dU, *dV, *dW;
  if (dev_in) {
    dU = U_in;
    dV = V_in;
    dW = W_in;
  } else {
    float* h = (float*)A(12 * N);
    CPSZ_TRY(h2d(ctx, h, U_in, 4 * N, st));
    CPSZ_TRY(h2d(ctx, h + N, V_in, 4 * N, st));
    CPSZ_TRY(h2d(ctx, h + 2 * N, W_in, 4 * N, st));
    dU = h;
    dV = h + N;
    dW = h + 2 * N;
  }
  uint8_t* ids = (uint8_t*)A(N);
  float4* pairs = (float4*)A(std::max(16 * N, eb3d_scratch_bytes(N)));
  float4* rec = (float4*)A(16 * N);
  ushort4* codes = (ushort4*)A(8 * N);
  unsigned* chunk_cnt = (unsigned*)A((nchunks + 1) * 4);
  unsigned* chunk_off = (unsigned*)A((nchunks + 1) * 4);
  void* scan_tmp = A(scan_u32_tmp_bytes(nchunks));
  uint16_t* codes_out = (uint16_t*)A(6 * N);
  float* unpred = (float*)A(12 * N);
  uint32_t* signs = (uint32_t*)A(3 * sign_words * 4);
  void* wave_sync = A(wave3d_scratch_bytes(r1, r2));
  uint8_t* zero = (uint8_t*)A(zero_bytes);
  unsigned long long* hist_ids = (unsigned long long*)zero;
  unsigned long long* hist_codes = hist_ids + 256;
  unsigned long long* enc_tmp[2] = {hist_codes + 65536,
                                    (unsigned long long*)((uint8_t*)(hist_codes + 65536) + tmp_ids)};
  uint8_t* image = (uint8_t*)A(image_bytes);
  double* thr_tab = (double*)image;
  HistList* d_list = (HistList*)(thr_tab + QUANT_TAB_MAX);
  unsigned long long* enc_code[2] = {(unsigned long long*)A(256 * 8), (unsigned long long*)A(65536 * 8)};
  uint8_t* enc_len[2] = {(uint8_t*)A(256), (uint8_t*)A(65536)};
  uint8_t* d_up = (uint8_t*)A(up_cap);
  uint8_t* blob = (uint8_t*)A(blob_cap);
  if (!blob) return set_error(CPSZ_ERR_NOMEM, "workspace layout overflow");

  reset_marks(ctx);
  mark(ctx, "h2d+setup");
  unsigned* h_npred = (unsigned*)ctx->pinned + 4;  // the flag word lives at offset 0
  unsigned* h_nlist = h_npred + 1;
  unsigned long long* h_hist_ids = (unsigned long long*)ctx->pinned + 8;
  unsigned long long* h_list = h_hist_ids + 256;
  CPSZ_TRY(upload_reserve(ctx, image_bytes));
  memcpy(ctx->up_pinned, qt.t, QUANT_TAB_MAX * 8);
  *(HistList*)((double*)ctx->up_pinned + QUANT_TAB_MAX) = HistList{hist_codes, h_list, h_nlist};
  CPSZ_CUDA_TRY(cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), st));
  CPSZ_CUDA_TRY(cudaMemsetAsync(zero, 0, zero_bytes, st));
  CPSZ_CUDA_TRY(cudaMemcpyAsync(image, ctx->up_pinned, image_bytes, cudaMemcpyHostToDevice, st));
  mark(ctx, "eb3d");
  CPSZ_TRY(launch_eb3d(ctx, dU, dV, dW, r1, r2, r3, max_pwr_eb, thr_tab, qt.n, ids, pairs));  // (pairs: not yet written)
  mark(ctx, "log3d");
  CPSZ_TRY(launch_log3d(ctx, dU, dV, dW, ids, N, lt.log2f, pairs, signs, sign_words));
  mark(ctx, "wave3d_compress");
  CPSZ_TRY(launch_wave3d(ctx, false, pairs, rec, codes, nullptr, 0, &lt, nullptr, nullptr, nullptr, r1, r2, r3,
                          wave_sync));
  mark(ctx, "compact+hist");
  // The code histogram straight from the raster codes, so the host builds
  // the code tree while the GPU compacts: a predictable point's three codes
  // are never 0 (|q| <= 32767 around 32768), an unpredictable point's are,
  // and so is every fourth lane, so the count without symbol 0 is the
  // compacted codes' histogram.
  CPSZ_TRY(launch_hist_u16_nonzero(ctx, reinterpret_cast<const uint16_t*>(codes), 4 * N, hist_codes));
  CPSZ_TRY(launch_hist_list(ctx, d_list, 1, st));
  CPSZ_CUDA_TRY(cudaEventRecord(ctx->ev[1], st));
  CPSZ_TRY(launch_chunk_count_3d(ctx, true, codes, N, chunk_cnt));
  CPSZ_TRY(launch_scan_u32(ctx, chunk_cnt, chunk_off, nchunks, scan_tmp));
  CPSZ_TRY(launch_compact3d(ctx, codes, ids, dU, dV, dW, N, chunk_off, codes_out, unpred, hist_ids));
  CPSZ_CUDA_TRY(cudaMemcpyAsync(h_npred, chunk_off + nchunks, 4, cudaMemcpyDeviceToHost, st));
  CPSZ_CUDA_TRY(cudaMemcpyAsync(h_hist_ids, hist_ids, 256 * 8, cudaMemcpyDeviceToHost, st));
  mark(ctx, "host_trees");
  HuffCodebook cb[2];
  CPSZ_CUDA_TRY(cudaEventSynchronize(ctx->ev[1]));
  if (*h_nlist == 0) {  // no predictable point: one-leaf tree of symbol 0, no bits
    h_list[0] = 1;
    *h_nlist = 1;
  }
  if (!huff_build_list(h_list, *h_nlist, 65536, 131072, &cb[1])) return CPSZ_ERR_INVALID;
  CPSZ_CUDA_TRY(cudaStreamSynchronize(st));
  int flag = 0;
  CPSZ_TRY(read_flag3(ctx, &flag));
  if (flag) return flag_error3(flag);
  const size_t n_pred = *h_npred;
  const size_t n_codes = 3 * n_pred, n_unpred = 3 * (N - n_pred);
  if (!huff_build(h_hist_ids, 256, 512, &cb[0])) return CPSZ_ERR_INVALID;

  // ---- blob layout, then the streams packed in place (the caller's device
  // buffer if it has room: 8 bytes over, the packers touch a stream's last
  // word), the rest copied behind them ----
  mark(ctx, "huffman_encode");
  const size_t sec_bytes[2] = {huff_section_bytes(cb[0]), huff_section_bytes(cb[1])};
  const size_t bits_bytes[2] = {(cb[0].total_bits + 7) / 8, (cb[1].total_bits + 7) / 8};
  if (bits_bytes[0] + 8 > ids_bits_cap || bits_bytes[1] + 8 > codes_bits_cap)
    return set_error(CPSZ_ERR_UNSUPPORTED, "Huffman stream larger than its bound");
  const size_t total = 8 + 3 * smap + 8 + 4 * n_unpred + 8 + sec_bytes[0] + 8 + sec_bytes[1];
  if (total > blob_cap) return set_error(CPSZ_ERR_UNSUPPORTED, "blob larger than its bound");
  size_t room = blob_cap;
  if (dev_out && total + 8 <= dev_cap) {
    blob = dev_out;
    room = dev_cap;
  }
  // (the setup image has been copied: its staging is free)
  CPSZ_TRY(upload_reserve(ctx, up_cap));
  UpImage up{(uint8_t*)ctx->up_pinned, d_up, up_cap};
  std::vector<CopyPiece> pieces;
  auto stage = [&](size_t dst, const void* p, size_t n) -> int {
    uint8_t* dev;
    uint8_t* h = up.take(n, &dev);
    if (!h) return up_overrun();
    memcpy(h, p, n);
    pieces.push_back(CopyPiece{blob + dst, dev, n, 0});
    return CPSZ_OK;
  };
  size_t at = 0;
  const int hdr[2] = {2, 32768};
  CPSZ_TRY(stage(at, hdr, 8));
  at += 8;
  for (int c = 0; c < 3; c++, at += smap)
    pieces.push_back(CopyPiece{blob + at, (const uint8_t*)(signs + c * sign_words), smap, 0});
  unsigned long long v64 = n_unpred;
  CPSZ_TRY(stage(at, &v64, 8));
  at += 8;
  if (n_unpred) pieces.push_back(CopyPiece{blob + at, (const uint8_t*)unpred, 4 * n_unpred, 0});
  at += 4 * n_unpred;
  v64 = N;
  CPSZ_TRY(stage(at, &v64, 8));
  at += 8;
  PackGroup G;
  for (int k = 0; k < 2; k++) {
    if (k == 1) {
      v64 = n_codes;
      CPSZ_TRY(stage(at, &v64, 8));
      at += 8;
    }
    CPSZ_TRY(stage(at, cb[k].tree_bytes.data(), cb[k].tree_bytes.size()));
    at += cb[k].tree_bytes.size();
    unsigned long long nb = bits_bytes[k];
    CPSZ_TRY(stage(at, &nb, 8));
    at += 8;
    if (k == 0 || n_codes)
      G.add(cb[k], k ? (const void*)codes_out : (const void*)ids, k ? 2 : 1, false, k ? n_codes : N, blob + at,
            bits_bytes[k], room - at, enc_code[k], enc_len[k], enc_tmp[k]);
    at += bits_bytes[k];
  }
  if (at != total) return set_error(CPSZ_ERR_INVALID, "internal: blob layout mismatch (%zu != %zu)", at, total);
  CPSZ_TRY(G.stage(up, ctx->num_sms));
  const unsigned piece_ctas = assign_piece_chunks(pieces.data(), pieces.size());
  uint8_t* d_pieces;
  uint8_t* h_pieces = up.take(pieces.size() * sizeof(CopyPiece), &d_pieces);
  if (!h_pieces) return up_overrun();
  memcpy(h_pieces, pieces.data(), pieces.size() * sizeof(CopyPiece));
  CPSZ_TRY(up.send(st));
  CPSZ_TRY(G.launch(ctx));
  mark(ctx, "blob_assembly");
  CPSZ_TRY(launch_copy_pieces(ctx, (const CopyPiece*)d_pieces, (int)pieces.size(), piece_ctas));
  mark(ctx, "end");
  CPSZ_TRY(read_flag3(ctx, &flag));
  if (flag) return flag_error3(flag);
  out->d_blob = blob;
  out->size = total;
  out->n_unpred = n_unpred;
  out->n_codes = n_codes;
  return CPSZ_OK;
}

int decompress_3d(cpsz_b200_ctx* ctx, const unsigned char* blob, size_t blob_size, size_t r1s, size_t r2s, size_t r3s,
                  float* U_out, float* V_out, float* W_out) {
  if (!blob || !U_out || !V_out || !W_out) return set_error(CPSZ_ERR_INVALID, "null pointer argument");
  CPSZ_TRY(check_dims(r1s, r2s, r3s));
  const int r1 = (int)r1s, r2 = (int)r2s, r3 = (int)r3s;
  const size_t N = r1s * r2s * r3s;
  const size_t smap = (N - 1) / 8 + 1;
  const size_t nchunks = chunk_count(N);
  // ---- header ----
  if (blob_size < 8 + 3 * smap + 8) return set_error(CPSZ_ERR_FORMAT, "blob shorter than its header");
  int base, radius;
  memcpy(&base, blob, 4);
  memcpy(&radius, blob + 4, 4);
  if (base != 2 || radius != 32768)
    return set_error(CPSZ_ERR_UNSUPPORTED, "blob quantizer (base %d, radius %d) is not the offline compressor's", base,
                     radius);
  size_t at = 8 + 3 * smap;
  unsigned long long n_unpred, n_ids, n_codes;
  memcpy(&n_unpred, blob + at, 8);
  at += 8;
  if (n_unpred > 3 * N || (blob_size - at) / 4 < n_unpred)
    return set_error(CPSZ_ERR_FORMAT, "unpredictable count %llu invalid", n_unpred);
  const size_t unpred_at = at;
  at += 4 * n_unpred;
  if (blob_size - at < 8) return set_error(CPSZ_ERR_FORMAT, "blob truncated before the id section");
  memcpy(&n_ids, blob + at, 8);
  at += 8;
  if (n_ids != N) return set_error(CPSZ_ERR_FORMAT, "id count %llu != %zu points", n_ids, N);
  HuffDecoderHost hs[2];
  if (!huff_parse(blob + at, blob_size - at, 511, &hs[0])) return CPSZ_ERR_FORMAT;
  if (hs[0].max_sym > (uint32_t)ID_RAW_3D)
    return set_error(CPSZ_ERR_UNSUPPORTED, "error-bound id %u beyond the supported range (<= %d)", hs[0].max_sym,
                     ID_RAW_3D);
  const size_t ids_at = at;
  at += hs[0].section_bytes;
  if (blob_size - at < 8) return set_error(CPSZ_ERR_FORMAT, "blob truncated before the code section");
  memcpy(&n_codes, blob + at, 8);
  at += 8;
  if (n_codes > 3 * N) return set_error(CPSZ_ERR_FORMAT, "code count %llu invalid", n_codes);
  if (!huff_parse(blob + at, blob_size - at, 65535, &hs[1])) return CPSZ_ERR_FORMAT;
  const size_t codes_at = at;
  const bool dev_out = is_device_ptr(U_out) && is_device_ptr(V_out) && is_device_ptr(W_out);
  LibmTables lt;
  CPSZ_TRY(libm_tables_device(ctx, &lt));

  // what goes up, as one image: a small blob whole, a large one stream by
  // stream, each decoded while the next one goes up
  const size_t sec_at[2] = {ids_at, codes_at};
  Upload up;
  size_t up_tree[2], up_bits[2];
  for (int k = 0; k < 2; k++) up_tree[k] = up.add(blob + sec_at[k] + hs[k].tree_offset, hs[k].tree_bytes);
  up_bits[0] = up.add(blob + ids_at + hs[0].bits_offset, hs[0].nbytes, HUFF_DEC_PAD);
  up.cut();
  up_bits[1] = up.add(blob + codes_at + hs[1].bits_offset, hs[1].nbytes, HUFF_DEC_PAD);
  up.cut();
  const size_t up_unpred = up.add(blob + unpred_at, 4 * n_unpred), up_signs = up.add(blob + 8, 3 * smap, 16);
  up.cut();
  HuffDecJob dec[2];
  for (int k = 0; k < 2; k++) {
    dec[k].nbytes = hs[k].nbytes;
    dec[k].node_count = hs[k].node_count;
    dec[k].root_is_leaf = hs[k].root_is_leaf;
    dec[k].root_sym = hs[k].root_sym;
    dec[k].n = k ? n_codes : N;
    dec[k].out_bytes = k ? 2 : 1;
  }
  const bool whole = up.bytes() <= UPLOAD_WHOLE;
  size_t dec_bytes[2];
  for (int k = 0; k < 2; k++) dec_bytes[k] = whole ? (k ? 0 : huff_decode_tmp_bytes(dec, 2)) : huff_decode_tmp_bytes(&dec[k], 1);
  size_t bytes = 0;
  auto add = [&](size_t b) { bytes += align_up(b, 256) + 256; };
  add(up.bytes());
  if (!dev_out) add(12 * N);
  add(N);
  add(2 * n_codes + 16);
  for (int k = 0; k < 2; k++) add(dec_bytes[k]);
  add(2 * (nchunks + 1) * 4);
  add(scan_u32_tmp_bytes(nchunks));
  add(16 * N);
  add(16 * N);
  add(wave3d_scratch_bytes(r1, r2));
  CPSZ_TRY(arena_reserve(ctx, bytes));
  CPSZ_TRY(pinned_reserve(ctx, 4096));
  auto A = [&](size_t b) { return arena_alloc(ctx, b); };
  cudaStream_t st = ctx->stream;
  uint8_t* d_up = (uint8_t*)A(up.bytes());
  float* out = dev_out ? nullptr : (float*)A(12 * N);
  float* dU = dev_out ? U_out : out;
  float* dV = dev_out ? V_out : out + N;
  float* dW = dev_out ? W_out : out + 2 * N;
  const uint8_t* signs = d_up + up_signs;
  const float* unpred = (const float*)(d_up + up_unpred);
  uint8_t* ids = (uint8_t*)A(N);
  uint16_t* codes = (uint16_t*)A(2 * n_codes + 16);
  void* dtmp[2];
  for (int k = 0; k < 2; k++) dtmp[k] = A(dec_bytes[k]);
  unsigned* chunk_cnt = (unsigned*)A((nchunks + 1) * 4);
  unsigned* chunk_off = (unsigned*)A((nchunks + 1) * 4);
  void* scan_tmp = A(scan_u32_tmp_bytes(nchunks));
  float4* pairs = (float4*)A(16 * N);
  float4* rec = (float4*)A(16 * N);
  void* wave_sync = A(wave3d_scratch_bytes(r1, r2));
  if (!wave_sync) return set_error(CPSZ_ERR_NOMEM, "workspace layout overflow");
  for (int k = 0; k < 2; k++) {
    dec[k].bits = d_up + up_bits[k];
    dec[k].tree = d_up + up_tree[k];
    dec[k].out = k ? (void*)codes : (void*)ids;
  }
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
    reset_marks(ctx);
    mark(ctx, "huffman_decode");
    if (whole) {
      if (!settle) CPSZ_TRY(up.send_whole(ctx, d_up, st));
      CPSZ_TRY(launch_huff_decode(ctx, dec, 2, dtmp[0], settle));
    } else {
      for (int k = 0; k < 3; k++) {
        if (!settle) {
          aux_drain.s = ctx->aux;
          CPSZ_TRY(up.send_part(ctx, d_up, k, ctx->aux));
          CPSZ_CUDA_TRY(cudaEventRecord(ctx->up_ev[k], ctx->aux));
          CPSZ_CUDA_TRY(cudaStreamWaitEvent(st, ctx->up_ev[k], 0));
        }
        if (k < 2) CPSZ_TRY(launch_huff_decode(ctx, &dec[k], 1, dtmp[k], settle));
      }
    }
    const bool probe = !settle && !dev_out;
    if (probe) {
      aux_drain.s = ctx->aux;
      CPSZ_TRY(probe_decode_again(ctx));
    }
    mark(ctx, "prep3d");
    CPSZ_TRY(launch_chunk_count_3d(ctx, false, ids, N, chunk_cnt));
    CPSZ_TRY(launch_scan_u32(ctx, chunk_cnt, chunk_off, nchunks, scan_tmp));
    CPSZ_TRY(launch_prep3d(ctx, ids, N, chunk_off, codes, n_codes, unpred, n_unpred, pairs, &lt, dU, dV, dW));
    mark(ctx, "wave3d_decompress");
    CPSZ_TRY(launch_wave3d(ctx, true, pairs, rec, nullptr, signs, smap, &lt, dU, dV, dW, r1, r2, r3, wave_sync));
    mark(ctx, "d2h");
    if (probe) {
      bool again = false;
      CPSZ_TRY(seen_decode_again(ctx, &again));
      if (again) continue;
    }
    if (!dev_out) {
      CPSZ_TRY(d2h(ctx, U_out, dU, 4 * N, st));
      CPSZ_TRY(d2h(ctx, V_out, dV, 4 * N, st));
      CPSZ_TRY(d2h(ctx, W_out, dW, 4 * N, st));
    }
    mark(ctx, "end");
    int flag = 0;
    CPSZ_TRY(read_flag3(ctx, &flag));  // synchronizes the stream
    main_drain.s = nullptr;
    if ((flag & FLAG_HUFF_RESYNC) && !settle) continue;
    if (flag) return flag_error3(flag);
    break;
  }
  return CPSZ_OK;
}

}  // namespace cpsz
