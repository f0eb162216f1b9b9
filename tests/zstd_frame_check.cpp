// zstd_frame_check.cpp -- checks frames of the GPU lossless stage against
// cpsz_b200/csrc/zstd_format.h, byte by byte (test infrastructure, built and
// run by tests/test_gpu_lossless.py): every compressed block's literals and
// sequences are read back with a plain decoder of the predefined tables
// (RFC 8878 3.1.1.3.2 and 4.1.1), must give the block's data, and written
// again with the header's coder must give the block's bytes; headers, raw and
// RLE blocks are compared with the header's, too.
// Argument: a file of (u64 data bytes, u64 frame bytes, data, frame) records.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "zstd_format.h"

using namespace cpsz::zstd;

struct DecodeCell {
  int sym, nb, base;
};

static std::vector<DecodeCell> decode_table(const int16_t* norm, int max_sym, int log) {
  const int size = 1 << log, step = (size >> 1) + (size >> 3) + 3;
  std::vector<int> cell(size);
  int high = size - 1, pos = 0;
  for (int s = 0; s <= max_sym; s++)
    if (norm[s] == -1) cell[high--] = s;
  for (int s = 0; s <= max_sym; s++)
    for (int i = 0; i < norm[s]; i++) {
      cell[pos] = s;
      do pos = (pos + step) & (size - 1);
      while (pos > high);
    }
  std::vector<int> next(max_sym + 1);
  for (int s = 0; s <= max_sym; s++) next[s] = norm[s] == -1 ? 1 : norm[s];
  std::vector<DecodeCell> t(size);
  for (int u = 0; u < size; u++) {
    const int x = next[cell[u]]++, nb = log - highbit32((uint32_t)x);
    t[u] = DecodeCell{cell[u], nb, (x << nb) - size};
  }
  return t;
}

struct BackBits {  // the stream's bits from its end mark down
  const uint8_t* p;
  long long at;
  bool ok = true;
  BackBits(const uint8_t* s, size_t n) : p(s) {
    ok = n > 0 && s[n - 1] != 0;
    at = ok ? 8 * (long long)(n - 1) + highbit32(s[n - 1]) : 0;
  }
  uint32_t take(int nb) {
    uint32_t v = 0;
    for (int i = 0; i < nb; i++) {
      if (--at < 0) {
        ok = false;
        return 0;
      }
      v = v << 1 | ((p[at >> 3] >> (at & 7)) & 1);
    }
    return v;
  }
};

static const std::vector<DecodeCell> kLL = decode_table(kLLNorm, 35, kLLLog), kML = decode_table(kMLNorm, 52, kMLLog),
                                     kOF = decode_table(kOFNorm, 28, kOFLog);

// Checks one compressed block body; returns what is wrong, or null.
static const char* check_body(const Tables& T, const uint8_t* b, size_t n, const uint8_t* data, size_t len) {
  if (n < 2 || (b[0] & 3) != 0) return "literals are not raw";
  const int form = (b[0] >> 2) & 3;
  size_t nlit, k;
  if ((form & 1) == 0) nlit = b[0] >> 3, k = 1;
  else if (form == 1) nlit = b[0] >> 4 | (size_t)b[1] << 4, k = 2;
  else nlit = b[0] >> 4 | (size_t)b[1] << 4 | (size_t)b[2] << 12, k = 3;
  uint8_t hdr[3];
  if (write_raw_literals_header((uint32_t)nlit, hdr) != k || memcmp(hdr, b, k)) return "literals header";
  if (k + nlit + 2 > n) return "literals run past the block";
  const uint8_t* lit = b + k;
  const uint8_t* s = lit + nlit;
  const size_t sn = n - k - nlit;
  int nseq;
  size_t q;
  if (s[0] < 128) nseq = s[0], q = 1;
  else if (s[0] < 255) nseq = ((s[0] - 128) << 8) + s[1], q = 2;
  else nseq = s[1] + (s[2] << 8) + 0x7F00, q = 3;
  if (nseq == 0 || q + 1 > sn || s[q] != 0) return "sequence count or modes";
  q++;
  BackBits r(s + q, sn - q);
  uint32_t ll = r.take(kLLLog), of = r.take(kOFLog), ml = r.take(kMLLog);
  std::vector<Seq> seqs;
  std::vector<uint8_t> out;
  size_t used = 0;
  for (int i = 0; i < nseq && r.ok; i++) {
    const int oc = kOF[of].sym, mc = kML[ml].sym, lc = kLL[ll].sym;
    const uint32_t ofv = (1u << oc) + r.take(oc);
    const uint32_t mlen = ml_base(mc) + r.take(ml_bits(mc));
    const uint32_t llen = ll_base(lc) + r.take(ll_bits(lc));
    if (ofv <= 3) return "a repeat offset";
    seqs.push_back(Seq{llen, mlen, ofv - 3});
    if (used + llen > nlit) return "more literals than there are";
    out.insert(out.end(), lit + used, lit + used + llen);
    used += llen;
    if (ofv - 3 > out.size() || out.size() + mlen > len) return "a match outside the block";
    for (uint32_t j = 0; j < mlen; j++) out.push_back(out[out.size() - (ofv - 3)]);
    if (i + 1 < nseq) {
      ll = kLL[ll].base + r.take(kLL[ll].nb);
      ml = kML[ml].base + r.take(kML[ml].nb);
      of = kOF[of].base + r.take(kOF[of].nb);
    }
  }
  if (!r.ok || r.at != 0) return "bits left or missing";
  out.insert(out.end(), lit + used, lit + nlit);
  if (out.size() != len || memcmp(out.data(), data, len)) return "decoded data";
  std::vector<uint8_t> again(sn + 64);
  const size_t an = write_sequences(T, seqs.data(), nseq, again.data(), again.size());
  if (an != sn || memcmp(again.data(), s, sn)) return "sequence section";
  return nullptr;
}

int main(int argc, char** argv) {
  Tables T;
  build_tables(&T);
  FILE* f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
  if (!f) return 2;
  int kinds[3] = {0, 0, 0}, records = 0;
  uint64_t head[2];
  while (fread(head, 8, 2, f) == 2) {
    std::vector<uint8_t> d(head[0]), z(head[1]);
    if (fread(d.data(), 1, d.size(), f) != d.size() || fread(z.data(), 1, z.size(), f) != z.size()) return 2;
    uint8_t hdr[kFrameHeader];
    const size_t h = write_frame_header(hdr, d.size());
    const char* bad = z.size() < h || memcmp(hdr, z.data(), h) ? "frame header" : nullptr;
    size_t at = h, from = 0;
    bool last = false;
    while (!bad && !last) {
      if (at + 3 > z.size()) {
        bad = "frame ends early";
        break;
      }
      const uint32_t v = z[at] | z[at + 1] << 8 | z[at + 2] << 16, type = v >> 1 & 3, size = v >> 3;
      last = v & 1;
      const size_t len = std::min<size_t>(8192, d.size() - from), body = type == 1 ? 1 : size;
      if (type > 2 || at + 3 + body > z.size()) bad = "block header";
      else if (type == 0) bad = size != len || memcmp(&z[at + 3], d.data() + from, len) ? "raw block" : nullptr;
      else if (type == 1)
        bad = size != len || std::count(d.begin() + from, d.begin() + from + len, z[at + 3]) != (long)len ? "RLE block"
                                                                                                          : nullptr;
      else bad = size >= len ? "a compressed block that did not shrink" : check_body(T, &z[at + 3], size, &d[from], len);
      if (type <= 2) kinds[type]++;
      from += len;
      at += 3 + body;
      if (!bad && last != (from == d.size())) bad = "last block flag";
    }
    if (!bad && at != z.size()) bad = "bytes behind the frame";
    if (bad) {
      printf("FAIL record %d (%zu bytes) at %zu: %s\n", records, d.size(), from, bad);
      return 1;
    }
    records++;
  }
  printf("ALL OK %d frames: %d raw, %d rle, %d compressed blocks\n", records, kinds[0], kinds[1], kinds[2]);
  return 0;
}
