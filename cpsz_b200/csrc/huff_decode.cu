// huff_decode.cu -- the GPU decoder of the SZ-1.x Huffman streams
// (src/sz_huffman.cpp decode, src/sz_decompression_utils.cpp:92-108 layout).
//
// The reference's streams carry no chunk index, so decoding self-synchronises
// (after Weissenberger & Schmidt, ICPP 2018): the stream is cut into
// subsequences of DEC_S bits, one thread each.
//   table  the serialized tree, as it stands in the blob, becomes a 2^12-entry
//          table whose entry holds every whole symbol of its 12 bits that fits
//          48 bits of payload (three u16 or six u8 symbols), and for each
//          12-bit pattern that no code ends in, 2^8 entries over the next 8
//          bits (longer codes walk the tree from there bit by bit);
//   scan   a CTA stages its subsequences' bits in shared memory; every thread
//          decodes its own from the nominal start, then threads whose
//          predecessor left at another bit decode again from there, in
//          lockstep with their previous path until the two meet, round after
//          round inside the CTA.  The CTA begins DEC_PRE subsequences early,
//          so its own first start is nearly always settled, too;
//   fix    a CTA whose first start still differs from its predecessor's exit
//          repeats the rounds from that exit;
//   write  symbol counts become offsets by decoupled look-back
//          (lookback.cuh), and every thread decodes its subsequence once more
//          into 16-byte stores.  It also checks its exit against the next
//          start: a difference raises FLAG_HUFF_RESYNC, and the caller
//          decodes again with `settle`, which repeats `fix` until no start
//          moves (streams that never synchronise, as fixed-length codes whose
//          length does not divide DEC_S).
//
// Bound: the dependent chain of a look-up (shared-memory loads and shifts) and
// divergence: a warp's lanes hold different numbers of symbols.  Device time of
// a blob's streams: 8192 x 8192, eb 0.1 (402 M symbols, 86 MB) 1.43 ms, where
// one symbol per look-up, a tree walk in global memory for codes over 12 bits
// and a launch with a host wait per synchronisation round took 4.2 ms;
// 1021 x 1537, eb 0.05 0.14 ms against 1.85 (few CTAs, so the walks' latency
// was exposed: some lane of a warp met one at nearly every step); 3D 256^3,
// eb 0.05 0.90 against 2.5 ms.
// DEC_S = 512: 1024 bits leave a 1.6 M point field's streams on 20 CTAs.
#include <algorithm>

#include "kernels.h"
#include "lookback.cuh"

namespace cpsz {

namespace {

constexpr int DEC_S = 512;     // bits per subsequence
constexpr int DEC_NT = 256;    // threads per CTA
constexpr int DEC_PRE = 16;    // subsequences a scan CTA starts early
constexpr int DEC_TILE = DEC_NT - DEC_PRE;  // subsequences a scan CTA owns
constexpr int DEC_ROW = DEC_S / 32;         // words per subsequence
constexpr int DEC_WORDS = DEC_NT * DEC_ROW + 8;  // staged words (8: a code and the reader's window past the end)
constexpr int DEC_SMEM_WORDS = DEC_WORDS + DEC_WORDS / DEC_ROW + 1;
constexpr int LUT1_BITS = 12, LUT1 = 1 << LUT1_BITS;
constexpr int LUT2_BITS = 8, LUT2 = 1 << LUT2_BITS;
constexpr int MAX_CODE = 64;   // longest code; a longer walk is a corrupt tree
constexpr int DEC_MAX_JOBS = 3;
constexpr long long DEC_SPIN_LIMIT = 1ll << 22;  // look-back polls before giving up (FLAG_TIMEOUT)

// First-level entries of a 12-bit pattern, two tables:
//   write  (32 bits + 32 bits) bits 0-2 symbols in the entry, 3-6 their bits,
//          7-10 the first symbol's bits, 16-31 and the second word the payload
//   count  (16 bits) bits 0-3 all whole symbols in the pattern, 4-7 their
//          bits, 8-11 the first symbol's bits; the counting pass needs no
//          payload, so a look-up takes up to 12 symbols there
// A pattern that no code ends in: 0 symbols, bits 16-31 the pattern's
// second-level table; in the count entry COUNT_LONG | that table.
// Second-level entry: symbol << 8 | code length, or 0x80 | node << 8 (node 0: walk from the root).
constexpr uint32_t COUNT_LONG = 0x8000u;

struct DecTree {
  const uint8_t* base;  // L | R (wdt bytes each), C (4), t (1) of nc nodes; base 16-byte aligned
  int nc, wdt;
};

struct DecStream {
  const uint32_t* w;  // the stream, big-endian words
  long long nwords;   // readable words, zero behind the stream
  unsigned long long nbits;
  int nsub;
  DecTree tree;
  uint32_t* lut1;   // write entries: LUT1 words, then LUT1 payload words
  uint16_t* lutc;   // count entries
  uint32_t* lut2;
  unsigned lut2_cap;  // second-level tables of single patterns; the one behind them is for all patterns past them
  unsigned* lut2_n;
  uint8_t* rel;     // start of each subsequence, bits after its nominal start
  uint8_t* texit;   // exit of each scan tile, bits after its end
  uint16_t* cnt;    // symbols that start in each subsequence
  unsigned long long* status;  // look-back words of the write tiles
  unsigned* ticket;
  size_t n;
  void* out;
  int out_bytes;
};
struct DecStreams {
  DecStream s[DEC_MAX_JOBS];
};

__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

struct TreeNode {
  uint32_t l, r, sym;
  bool leaf;
};
// All of a node's fields at once (one memory latency per level of a walk).
__device__ __forceinline__ TreeNode tree_node(const DecTree& T, uint32_t i) {
  TreeNode n;
  const size_t nc = (size_t)T.nc;
  const uint8_t* C = T.base + 2 * (size_t)T.wdt * nc + 4 * (size_t)i;
  if (T.wdt == 1) {
    n.l = T.base[i];
    n.r = T.base[nc + i];
    n.sym = (uint32_t)C[0] | (uint32_t)C[1] << 8 | (uint32_t)C[2] << 16 | (uint32_t)C[3] << 24;
  } else if (T.wdt == 2) {
    n.l = reinterpret_cast<const uint16_t*>(T.base)[i];
    n.r = reinterpret_cast<const uint16_t*>(T.base)[nc + i];
    n.sym = *reinterpret_cast<const uint32_t*>(C);
  } else {
    n.l = reinterpret_cast<const uint32_t*>(T.base)[i];
    n.r = reinterpret_cast<const uint32_t*>(T.base)[nc + i];
    n.sym = *reinterpret_cast<const uint32_t*>(C);
  }
  n.leaf = i != 0 && T.base[(2 * (size_t)T.wdt + 4) * nc + i] != 0;  // the root of a stream with bits is an inner node
  return n;
}

// ---- table ------------------------------------------------------------------------
// Patterns per CTA: the walks are serial (a memory latency per level), so few
// patterns in many CTAs: one per warp in the second phase.
constexpr int TAB_PAT = 8;

__global__ void __launch_bounds__(256) dec_table_kernel(const __grid_constant__ DecStreams J) {
  const DecStream& S = J.s[blockIdx.y];
  if (S.nsub == 0) return;
  __shared__ uint32_t s_node[TAB_PAT], s_tab[TAB_PAT];
  __shared__ int s_n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_n = 0;
  if (blockIdx.x == 0 && S.lut2_cap < LUT1) S.lut2[(size_t)S.lut2_cap * LUT2 + threadIdx.x] = 0x80u;
  __syncthreads();
  if (threadIdx.x < TAB_PAT) {
    const uint32_t pat = blockIdx.x * TAB_PAT + lane;
    const int cap = S.out_bytes == 1 ? 6 : 3, sb = 8 * S.out_bytes;
    unsigned long long pay = 0;
    int n = 0, bits = 0, len0 = 0, nall = 0, bits_all = 0;
    const TreeNode root = tree_node(S.tree, 0);
    TreeNode nd = root;
    uint32_t node = 0;
    for (int k = 0; k < LUT1_BITS; k++) {
      node = (pat >> (LUT1_BITS - 1 - k)) & 1u ? nd.r : nd.l;
      nd = tree_node(S.tree, node);
      if (nd.leaf) {
        nall++;
        bits_all = k + 1;
        if (nall == 1) len0 = k + 1;
        if (nall <= cap) {
          pay |= (unsigned long long)nd.sym << (sb * n);
          n = nall;
          bits = k + 1;
        }
        nd = root;
      }
    }
    uint32_t hi16 = (uint32_t)(pay & 0xffffu), count = (uint32_t)(len0 << 8 | bits_all << 4 | nall);
    if (n == 0) {
      const int q = atomicAdd(&s_n, 1);
      const unsigned t = min(atomicAdd(S.lut2_n, 1u), S.lut2_cap);
      s_node[q] = node;
      s_tab[q] = t;
      hi16 = t;
      count = COUNT_LONG | t;
    }
    S.lut1[pat] = hi16 << 16 | (uint32_t)(len0 << 7 | bits << 3 | n);
    S.lut1[LUT1 + pat] = (uint32_t)(pay >> 16);
    S.lutc[pat] = (uint16_t)count;
  }
  __syncthreads();
  // lane l fills the 8 entries whose first 5 bits are l
  for (int q = warp; q < s_n; q += 8) {
    if (s_tab[q] >= S.lut2_cap) continue;
    uint32_t* tab = S.lut2 + (size_t)s_tab[q] * LUT2;
    uint32_t node[8], e[8];
    TreeNode nd[8];
    const TreeNode top = tree_node(S.tree, s_node[q]);
#pragma unroll
    for (int m = 0; m < 8; m++) {
      nd[m] = top;
      node[m] = s_node[q];
      e[m] = 0;
    }
#pragma unroll
    for (int k = 0; k < LUT2_BITS; k++) {
#pragma unroll
      for (int m = 0; m < 8; m++) {
        const uint32_t idx = (uint32_t)lane * 8 + m;
        if (e[m] == 0) {
          node[m] = (idx >> (LUT2_BITS - 1 - k)) & 1u ? nd[m].r : nd[m].l;
          nd[m] = tree_node(S.tree, node[m]);
          if (nd[m].leaf) e[m] = nd[m].sym << 8 | (uint32_t)(LUT1_BITS + k + 1);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 8; m++) tab[lane * 8 + m] = e[m] ? e[m] : 0x80u | node[m] << 8;
  }
}

// ---- bits -------------------------------------------------------------------------
// Staged word j (a subsequence's row of words is padded by one, so the lanes
// of a warp, each in its own row, meet in different banks).
struct Bits {
  const uint32_t* sm;
  __device__ __forceinline__ uint32_t word(int j) const { return sm[j + j / DEC_ROW]; }
  __device__ __forceinline__ uint32_t peek32(int pos) const {
    const int j = pos >> 5;
    return __funnelshift_l(word(j + 1), word(j), (unsigned)(pos & 31));
  }
};

// The words of subsequences g0 .. g0 + DEC_NT - 1 (g0 may be negative).
__device__ __forceinline__ void stage_bits(const DecStream& S, long long g0, uint32_t* sm) {
  const long long w0 = g0 * DEC_ROW;
#pragma unroll 4
  for (int j = threadIdx.x; j < DEC_WORDS; j += DEC_NT) {
    const long long w = w0 + j;
    sm[j + j / DEC_ROW] = (w >= 0 && w < S.nwords) ? bswap32(__ldg(S.w + w)) : 0u;
  }
}

// The rest of a code that the tables do not end: from `node`, whose code has
// LUT1_BITS + LUT2_BITS bits, or from the root (node 0: a pattern without a
// table).  Returns symbol << 8 | length, 0 beyond MAX_CODE.
__device__ __noinline__ uint32_t deep_code(DecTree T, Bits b, int pos, uint32_t node) {
  for (int l = node ? LUT1_BITS + LUT2_BITS : 0; l < MAX_CODE;) {
    const int at = pos + l;
    const uint32_t bit = (b.word(at >> 5) >> (31 - (at & 31))) & 1u;
    const TreeNode nd = tree_node(T, node);
    node = bit ? nd.r : nd.l;
    l++;
    const TreeNode c = tree_node(T, node);
    if (c.leaf) return c.sym << 8 | (uint32_t)l;
  }
  return 0;
}

// A code over 12 bits (second-level table `t`, next8 its bits after them):
// symbol << 8 | length; 0: no code.
__device__ __forceinline__ uint32_t long_code(const DecStream& S, Bits b, int pos, uint32_t t, uint32_t next8) {
  const uint32_t e = __ldg(S.lut2 + (size_t)t * LUT2 + next8);
  return e & 0x80u ? deep_code(S.tree, b, pos, e >> 8) : e;
}

// Length of the one code at `pos` (lut: count entries).
__device__ __forceinline__ int code_len(const DecStream& S, const uint16_t* lut, Bits b, int pos) {
  const uint32_t p = b.peek32(pos), m = lut[p >> (32 - LUT1_BITS)];
  if (!(m & COUNT_LONG)) return (int)(m >> 8 & 15u);
  return (int)(long_code(S, b, pos, m & (LUT1 - 1), p << LUT1_BITS >> (32 - LUT2_BITS)) & 0x7fu);
}

// Sequential reader: the next bits in a 64-bit register, more than 32 of
// them, and the word after them (loaded before it is known to be needed, so
// a refill is two selects and no branch).
struct Cursor {
  unsigned long long buf;
  uint32_t next;
  int nb, j;
  __device__ __forceinline__ void seek(const Bits& b, int pos) {
    j = pos >> 5;
    buf = ((unsigned long long)b.word(j) << 32 | b.word(j + 1)) << (pos & 31);
    nb = 64 - (pos & 31);
    j += 2;
    next = b.word(j);
  }
  __device__ __forceinline__ void skip(const Bits& b, int l) {  // l <= 32
    buf <<= l;
    nb -= l;
    const bool need = nb <= 32;
    buf |= need ? (unsigned long long)next << ((32 - nb) & 63) : 0ull;
    nb += need ? 32 : 0;
    j += need ? 1 : 0;
    next = b.word(j);
  }
  __device__ __forceinline__ int pos() const { return 32 * j - nb; }
  __device__ __forceinline__ uint32_t top12() const { return (uint32_t)(buf >> (64 - LUT1_BITS)); }
  __device__ __forceinline__ uint32_t next8() const {
    return (uint32_t)(buf >> (64 - LUT1_BITS - LUT2_BITS)) & (LUT2 - 1);
  }
};

// ---- scan -------------------------------------------------------------------------
// The path of a subsequence: its start, its exit (both in bits after the
// nominal place) and the symbols that start in it.
struct Path {
  int st, en;
  unsigned c;
};

// Decodes [pos, lim) (bits of the staged tile), whose nominal end is `end`,
// after c symbols of a path from start st.
__device__ __forceinline__ Path decode_path(const DecStream& S, const uint16_t* lut, Bits b, int st, int pos, int lim,
                                            int end, unsigned c) {
  Path p{st, 0, c};
  Cursor cur;
  cur.seek(b, pos);
  while (pos < lim) {
    const uint32_t m = lut[cur.top12()];
    const bool all = pos + LUT1_BITS <= lim;  // every symbol of the entry starts before lim
    int l = (int)(all ? m >> 4 & 15u : m >> 8 & 15u);
    unsigned n = all ? m & 15u : 1u;
    if (m & COUNT_LONG) {
      l = (int)(long_code(S, b, pos, m & (LUT1 - 1), cur.next8()) & 0x7fu);
      n = 1;
      if (l == 0) {  // no code: only on a path that did not start at one, or in a corrupt tree
        pos = lim;
        break;
      }
    }
    p.c += n;
    pos += l;
    if (l <= 32) cur.skip(b, l);
    else cur.seek(b, pos);
  }
  p.en = max(0, pos - end);
  return p;
}

// The path from start st in place of p's: the two advance in lockstep (the
// one behind first) until they meet, from where p's counts hold.  Most meet
// within a few codes; past MEET_CODES steps the new path goes on alone, an
// entry of several symbols at a time.
constexpr int MEET_CODES = 24;
__device__ __forceinline__ Path repath(const DecStream& S, const uint16_t* lut, Bits b, int row, int st, int lim,
                                       const Path& p) {
  int a = row + st, o = row + p.st;
  unsigned ca = 0, co = 0;
  for (int k = 0; k < MEET_CODES && a < lim; k++) {
    if (o == a) return Path{st, p.en, ca + p.c - co};
    const bool old = o < a;
    const int l = code_len(S, lut, b, old ? o : a);
    if (l == 0) break;
    if (old) {
      o += l;
      co++;
    } else {
      a += l;
      ca++;
    }
  }
  return decode_path(S, lut, b, st, a, lim, row + DEC_S, ca);
}

// Rounds inside a CTA until every thread starts where its predecessor left:
// thread 0 starts at st0.  At most DEC_NT rounds (round k settles thread k).
__device__ __forceinline__ Path settle(const DecStream& S, const uint16_t* lut, Bits b, int row, int lim, bool active,
                                       Path p, int st0, uint8_t* s_en) {
  s_en[threadIdx.x] = (uint8_t)p.en;
  for (;;) {
    __syncthreads();
    const int st = threadIdx.x ? s_en[threadIdx.x - 1] : st0;
    const bool move = active && st != p.st;
    if (move) p = repath(S, lut, b, row, st, lim, p);
    if (!__syncthreads_or(move)) break;
    if (move) s_en[threadIdx.x] = (uint8_t)p.en;
  }
  return p;
}

struct ScanShared {
  uint16_t lut[LUT1];
  uint32_t bits[DEC_SMEM_WORDS];
  uint8_t en[DEC_NT];
};

__device__ __forceinline__ int sub_limit(const DecStream& S, long long g, int row) {
  const long long left = (long long)S.nbits - g * DEC_S;
  return row + (int)min((long long)DEC_S, max(0ll, left));
}

__global__ void __launch_bounds__(DEC_NT) dec_scan_kernel(const __grid_constant__ DecStreams J) {
  const DecStream& S = J.s[blockIdx.y];
  if ((long long)blockIdx.x * DEC_TILE >= S.nsub) return;
  __shared__ ScanShared sh;
  const long long g0 = (long long)blockIdx.x * DEC_TILE - DEC_PRE, g = g0 + threadIdx.x;
  stage_bits(S, g0, sh.bits);
  for (int k = threadIdx.x; k < LUT1 / 2; k += DEC_NT)
    reinterpret_cast<uint32_t*>(sh.lut)[k] = __ldg(reinterpret_cast<const uint32_t*>(S.lutc) + k);
  __syncthreads();
  const Bits b{sh.bits};
  const bool active = g >= 0 && g < S.nsub;
  const int row = threadIdx.x * DEC_S, lim = sub_limit(S, g, row);
  Path p{0, 0, 0};
  if (active) p = decode_path(S, sh.lut, b, 0, row, lim, row + DEC_S, 0);
  p = settle(S, sh.lut, b, row, lim, active, p, 0, sh.en);
  if (!active || threadIdx.x < DEC_PRE) return;
  S.rel[g] = (uint8_t)p.st;
  S.cnt[g] = (uint16_t)p.c;
  if (threadIdx.x == DEC_NT - 1) S.texit[blockIdx.x] = (uint8_t)p.en;
}

__global__ void __launch_bounds__(DEC_NT) dec_fix_kernel(const __grid_constant__ DecStreams J, int* changed) {
  const DecStream& S = J.s[blockIdx.y];
  const long long g0 = (long long)blockIdx.x * DEC_TILE, g = g0 + threadIdx.x;
  if (blockIdx.x == 0 || g0 >= S.nsub) return;
  // another CTA may be moving its own exit: what is stale here shows in the next round or in the write
  const int st0 = *(volatile uint8_t*)(S.texit + blockIdx.x - 1);
  __shared__ int s_same;
  if (threadIdx.x == 0) s_same = S.rel[g0] == st0;
  __syncthreads();
  if (s_same) return;
  __shared__ ScanShared sh;
  __shared__ int s_st0;
  if (threadIdx.x == 0) s_st0 = st0;
  stage_bits(S, g0, sh.bits);
  for (int k = threadIdx.x; k < LUT1 / 2; k += DEC_NT)
    reinterpret_cast<uint32_t*>(sh.lut)[k] = __ldg(reinterpret_cast<const uint32_t*>(S.lutc) + k);
  const bool active = threadIdx.x < DEC_TILE && g < S.nsub;
  const int row = threadIdx.x * DEC_S, lim = sub_limit(S, g, row);
  Path p{0, 0, 0};
  if (active) {
    p.st = S.rel[g];
    p.c = S.cnt[g];
    p.en = threadIdx.x == DEC_TILE - 1 ? S.texit[blockIdx.x] : g + 1 < S.nsub ? S.rel[g + 1] : 0;
  }
  __syncthreads();  // every path is read before one is written
  p = settle(S, sh.lut, Bits{sh.bits}, row, lim, active, p, s_st0, sh.en);
  if (!active) return;
  S.rel[g] = (uint8_t)p.st;
  S.cnt[g] = (uint16_t)p.c;
  if (threadIdx.x == DEC_TILE - 1) S.texit[blockIdx.x] = (uint8_t)p.en;
  if (threadIdx.x == 0) *changed = 1;
}

// ---- write ------------------------------------------------------------------------
struct WriteShared {
  uint32_t lut[2 * LUT1];
  uint32_t bits[DEC_SMEM_WORDS];
  unsigned warp_sum[DEC_NT / 32];
  unsigned long long excl;
  unsigned tile;
};

// Appends symbols to memory in aligned 16-byte stores; the partial chunks at
// the two ends of the run go out in 4-byte pieces and single symbols.
template <class Out>
struct Appender {
  unsigned char* chunk;  // 16-byte aligned place of (w0, acc)
  unsigned long long w0, acc;
  int nb;     // bits of the chunk so far (with the foreign ones at its head)
  int head;   // bytes of the chunk that belong to the run before
  __device__ __forceinline__ void init(Out* p) {
    chunk = (unsigned char*)((uintptr_t)p & ~(uintptr_t)15);
    head = (int)((uintptr_t)p & 15);
    nb = 8 * head;
    w0 = acc = 0;
  }
  __device__ __forceinline__ void part(int from, int to) {  // bytes [from, to) of the chunk
    const unsigned long long lo = nb >= 64 ? w0 : acc, hi = acc;
    for (int k = from; k < to;) {
      const unsigned long long v = (k < 8 ? lo >> (8 * k) : hi >> (8 * (k - 8)));
      if ((k & 3) == 0 && k + 4 <= to) {
        *reinterpret_cast<uint32_t*>(chunk + k) = (uint32_t)v;
        k += 4;
      } else {
        *reinterpret_cast<Out*>(chunk + k) = (Out)v;
        k += (int)sizeof(Out);
      }
    }
  }
  // the low `bits` of pay (8 .. 48, whole symbols; the bits above them 0)
  __device__ __forceinline__ void add(unsigned long long pay, int bits) {
    const int s = nb & 63;
    acc |= pay << s;
    const int t = s + bits;
    if (t < 64) {
      nb += bits;
      return;
    }
    const unsigned long long rest = s ? pay >> (64 - s) : 0ull;
    if (nb < 64) {
      w0 = acc;
      nb += bits;
    } else {
      if (head) {
        part(head, 16);
        head = 0;
      } else {
        __stcs(reinterpret_cast<uint4*>(chunk), make_uint4((uint32_t)w0, (uint32_t)(w0 >> 32), (uint32_t)acc,
                                                           (uint32_t)(acc >> 32)));
      }
      chunk += 16;
      nb += bits - 128;
    }
    acc = rest;
  }
  __device__ __forceinline__ void finish() {
    if (nb >> 3 > head) part(head, nb >> 3);
  }
};

template <class Out>
__device__ __forceinline__ bool write_run(const DecStream& S, const uint32_t* lut, Bits b, int pos, size_t o,
                                          unsigned left, int* end_pos) {
  constexpr int SB = 8 * (int)sizeof(Out);
  constexpr uint32_t SMASK = sizeof(Out) == 1 ? 0xffu : 0xffffu;
  Appender<Out> ap;
  ap.init(reinterpret_cast<Out*>(S.out) + o);
  Cursor cur;
  cur.seek(b, pos);
  bool ok = true;
  while (left > 0) {
    const uint32_t i = cur.top12(), m = lut[i];
    const unsigned n = m & 7u;
    const bool all = n <= left;  // else only the entry's first symbol
    unsigned long long pay = all ? (unsigned long long)lut[LUT1 + i] << 16 | m >> 16 : m >> 16 & SMASK;
    unsigned take = all ? n : 1u;
    int l = (int)(all ? m >> 3 & 15u : m >> 7 & 15u);
    if (n == 0) {
      const int at = cur.pos();
      const uint32_t e = long_code(S, b, at, m >> 16, cur.next8());
      l = (int)(e & 0x7fu);
      if (l == 0) {
        ok = false;
        break;
      }
      pay = e >> 8 & SMASK;
      take = 1;
    }
    ap.add(pay, (int)take * SB);
    left -= take;
    if (l <= 32) cur.skip(b, l);
    else cur.seek(b, cur.pos() + l);
  }
  ap.finish();
  *end_pos = cur.pos();
  return ok;
}

__global__ void __launch_bounds__(DEC_NT) dec_write_kernel(const __grid_constant__ DecStreams J, int* flag) {
  extern __shared__ __align__(16) unsigned char dec_smem[];
  WriteShared& sh = *reinterpret_cast<WriteShared*>(dec_smem);
  const DecStream& S = J.s[blockIdx.y];
  const unsigned ntiles = (unsigned)((S.nsub + DEC_NT - 1) / DEC_NT);
  if (blockIdx.x >= ntiles) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sh.tile = atomicAdd(S.ticket, 1u);
  __syncthreads();
  const unsigned tile = sh.tile;
  const long long g0 = (long long)tile * DEC_NT, g = g0 + threadIdx.x;
  const bool active = g < S.nsub;
  const unsigned c = active ? S.cnt[g] : 0u;
  const int st = active ? S.rel[g] : 0;
  const int next = g + 1 < S.nsub ? S.rel[g + 1] : -1;
  unsigned x = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) sh.warp_sum[warp] = x;
  stage_bits(S, g0, sh.bits);
  for (int k = threadIdx.x; k < 2 * LUT1; k += DEC_NT) sh.lut[k] = __ldg(S.lut1 + k);
  __syncthreads();
  unsigned wpre = 0, agg = 0;
#pragma unroll
  for (int q = 0; q < DEC_NT / 32; q++) {
    const unsigned v = sh.warp_sum[q];
    wpre += q < warp ? v : 0u;
    agg += v;
  }
  if (warp == 0) {
    if (lane == 0) lookback_publish(S.status, tile, agg);
    const unsigned long long e = lookback_warp(S.status, tile, agg, lane, DEC_SPIN_LIMIT, flag);
    if (lane == 0) sh.excl = e;
  }
  __syncthreads();
  const unsigned long long o = sh.excl + wpre + x - c;
  if (threadIdx.x == 0 && tile == ntiles - 1 && sh.excl + agg < S.n) atomicOr(flag, FLAG_HUFF_CORRUPT);
  if (!active || o >= S.n) return;
  const unsigned take = (unsigned)min((unsigned long long)c, (unsigned long long)S.n - o);
  const int row = threadIdx.x * DEC_S;
  int end = 0;
  const bool ok = S.out_bytes == 1 ? write_run<uint8_t>(S, sh.lut, Bits{sh.bits}, row + st, o, take, &end)
                                   : write_run<uint16_t>(S, sh.lut, Bits{sh.bits}, row + st, o, take, &end);
  if (!ok) atomicOr(flag, FLAG_HUFF_CORRUPT);
  else if (take == c && next >= 0 && end - (row + DEC_S) != next) atomicOr(flag, FLAG_HUFF_RESYNC);
}

template <class Out>
__global__ void fill_kernel(Out* out, size_t n, Out v) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = v;
}

size_t sub_count(size_t nbytes) { return (8 * nbytes + DEC_S - 1) / DEC_S; }

// Workspace of a stream: what has to be zero, and the rest.
struct DecLayout {
  size_t nsub, scan_tiles, write_tiles, lut2_cap, zero, rest;
};
DecLayout dec_layout(const HuffDecJob& j) {
  DecLayout L{};
  if (j.root_is_leaf || j.n == 0) return L;
  L.nsub = sub_count(j.nbytes);
  L.scan_tiles = (L.nsub + DEC_TILE - 1) / DEC_TILE;
  L.write_tiles = (L.nsub + DEC_NT - 1) / DEC_NT;
  // Patterns that no code ends in are paths to inner nodes at depth 12: in a
  // tree fewer than half its nodes.  A node array whose nodes are shared (both
  // children one node, say: huff_parse takes any children with larger numbers)
  // can have up to 4096 of them whatever its size: those past this room share
  // one table more, whose entries have the code walked from the root.
  L.lut2_cap = std::min<size_t>(LUT1, (size_t)j.node_count / 2 + 1);
  L.zero = align_up(8 * L.write_tiles + 16, 256);
  L.rest = align_up(10 * (size_t)LUT1, 256) + align_up(4 * (L.lut2_cap + 1) * LUT2, 256) + align_up(L.nsub + 1, 256) +
           align_up(L.scan_tiles + 1, 256) + align_up(2 * (L.nsub + 1), 256);
  return L;
}

bool g_write_smem_set[64] = {};

}  // namespace

size_t huff_decode_tmp_bytes(const HuffDecJob* jobs, int nj) {
  size_t b = 256;  // the fix rounds' `changed` word
  for (int k = 0; k < nj; k++) {
    const DecLayout L = dec_layout(jobs[k]);
    b += L.zero + L.rest;
  }
  return b;
}

int launch_huff_decode(cpsz_b200_ctx* ctx, const HuffDecJob* jobs, int nj, void* tmp, bool settle) {
  if (nj < 0 || nj > DEC_MAX_JOBS) return set_error(CPSZ_ERR_INVALID, "internal: %d Huffman streams", nj);
  cudaStream_t st = ctx->stream;
  DecStreams J{};
  char* p = (char*)tmp;
  int* changed = (int*)p;
  p += 256;
  char* const zero0 = p;
  size_t zero = 0;
  unsigned scan_grid = 0, write_grid = 0;
  int nd = 0;
  DecLayout lay[DEC_MAX_JOBS];
  for (int k = 0; k < nj; k++) {
    const HuffDecJob& j = jobs[k];
    if (j.n == 0) continue;
    if (j.root_is_leaf) {
      const unsigned grid = (unsigned)std::min<size_t>((j.n + 255) / 256, (size_t)ctx->num_sms * 8);
      if (j.out_bytes == 1) fill_kernel<uint8_t><<<grid, 256, 0, st>>>((uint8_t*)j.out, j.n, (uint8_t)j.root_sym);
      else fill_kernel<uint16_t><<<grid, 256, 0, st>>>((uint16_t*)j.out, j.n, (uint16_t)j.root_sym);
      count_launch(ctx);
      CPSZ_TRY(check_launch("huffman fill"));
      continue;
    }
    const DecLayout L = dec_layout(j);
    if (L.nsub == 0) return set_error(CPSZ_ERR_FORMAT, "empty Huffman stream for %zu symbols", j.n);
    if (L.nsub > 0x7fffffffu) return set_error(CPSZ_ERR_UNSUPPORTED, "Huffman stream of %zu bytes", j.nbytes);
    DecStream& S = J.s[nd];
    S.w = (const uint32_t*)j.bits;
    S.nwords = (long long)((j.nbytes + HUFF_DEC_PAD) / 4);
    S.nbits = 8ull * j.nbytes;
    S.nsub = (int)L.nsub;
    S.tree = DecTree{j.tree, j.node_count, j.node_count <= 256 ? 1 : j.node_count <= 65536 ? 2 : 4};
    S.lut2_cap = (unsigned)L.lut2_cap;
    S.n = j.n;
    S.out = j.out;
    S.out_bytes = j.out_bytes;
    S.status = (unsigned long long*)(zero0 + zero);
    S.ticket = (unsigned*)(S.status + L.write_tiles);
    S.lut2_n = S.ticket + 1;
    zero += L.zero;
    scan_grid = std::max(scan_grid, (unsigned)L.scan_tiles);
    write_grid = std::max(write_grid, (unsigned)L.write_tiles);
    lay[nd++] = L;
  }
  if (nd == 0) return CPSZ_OK;
  p = zero0 + zero;
  for (int k = 0; k < nd; k++) {
    DecStream& S = J.s[k];
    auto take = [&](size_t b) {
      char* q = p;
      p += align_up(b, 256);
      return q;
    };
    S.lut1 = (uint32_t*)take(10 * (size_t)LUT1);
    S.lutc = (uint16_t*)(S.lut1 + 2 * LUT1);
    S.lut2 = (uint32_t*)take(4 * (lay[k].lut2_cap + 1) * LUT2);
    S.rel = (uint8_t*)take(lay[k].nsub + 1);
    S.texit = (uint8_t*)take(lay[k].scan_tiles + 1);
    S.cnt = (uint16_t*)take(2 * (lay[k].nsub + 1));
  }
  CPSZ_CUDA_TRY(cudaMemsetAsync(tmp, 0, 256 + zero, st));
  dec_table_kernel<<<dim3(LUT1 / TAB_PAT, nd), 256, 0, st>>>(J);
  dec_scan_kernel<<<dim3(scan_grid, nd), DEC_NT, 0, st>>>(J);
  dec_fix_kernel<<<dim3(scan_grid, nd), DEC_NT, 0, st>>>(J, changed);
  count_launch(ctx, 3);
  if (settle) {
    // each round settles at least one more tile
    int* h_changed = (int*)ctx->pinned;
    for (unsigned round = 0; round <= scan_grid; round++) {
      CPSZ_CUDA_TRY(cudaMemsetAsync(changed, 0, sizeof(int), st));
      dec_fix_kernel<<<dim3(scan_grid, nd), DEC_NT, 0, st>>>(J, changed);
      count_launch(ctx);
      CPSZ_CUDA_TRY(cudaMemcpyAsync(h_changed, changed, sizeof(int), cudaMemcpyDeviceToHost, st));
      CPSZ_CUDA_TRY(cudaStreamSynchronize(st));
      if (!*h_changed) break;
    }
  }
  if (!g_write_smem_set[ctx->device & 63]) {
    CPSZ_CUDA_TRY(cudaFuncSetAttribute(dec_write_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(WriteShared)));
    g_write_smem_set[ctx->device & 63] = true;
  }
  dec_write_kernel<<<dim3(write_grid, nd), DEC_NT, sizeof(WriteShared), st>>>(J, ctx->d_flag);
  count_launch(ctx);
  return check_launch("huffman decode");
}

}  // namespace cpsz
