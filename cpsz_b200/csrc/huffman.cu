// huffman.cu -- GPU side of the SZ-1.x Huffman codec used by the reference
// (src/sz_huffman.cpp): symbol histograms and the MSB-first bit packer (the
// decoder is huff_decode.cu).
//
// Encoder.  The reference's packer (encode, src/sz_huffman.cpp:217-320) emits
// the MSB-first concatenation of the codes, zero padded to a byte.  Here one
// persistent kernel reads every symbol once: a tile of 8192 consecutive
// symbols sums and scans its code lengths, packs its codes into a
// shared-memory word buffer, finds its starting bit by a decoupled look-back
// over the earlier tiles' published bit counts, and stores the buffer shifted
// onto the global 32-bit word grid with coalesced stores (atomicOr for the two
// edge words, shared with the neighbouring tiles).  Words are stored byte-swapped so
// memory holds the big-endian byte stream the reference writes.
#include <algorithm>

#include "kernels.h"
#include "lookback.cuh"

namespace cpsz {

namespace {

// ---- encoder: one pass with decoupled look-back --------------------------------------
constexpr int PK_NT = 256;                  // threads per CTA
constexpr int PK_SPT = 32;                  // symbols per thread (a contiguous run)
constexpr int PK_TILE = PK_NT * PK_SPT;     // symbols per tile
constexpr int PK_WORDS = PK_TILE;           // staged words of a tile whose codes are at most 32 bits
constexpr int PK_WIN = 1536;                // codebook entries cached in shared memory: u16 symbols
constexpr int PK_WIN_LO = 32768 - PK_WIN / 2;  // [PK_WIN_LO, PK_WIN_LO + PK_WIN) (all 256 for u8)
constexpr int PK_CTAS_PER_SM = 4;
constexpr long long PK_SPIN_LIMIT = 1ll << 22;  // look-back polls before giving up (FLAG_TIMEOUT)

__device__ __forceinline__ uint32_t bswap32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

__device__ __forceinline__ void sts_u32_if(bool p, unsigned addr, uint32_t v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u32 [%1], %2;\n\t}" ::"r"((unsigned)p),
               "r"(addr), "r"(v)
               : "memory");
}

template <class Sym>
struct PackWin {
  static constexpr int lo = sizeof(Sym) == 1 ? 0 : PK_WIN_LO;
  static constexpr int n = sizeof(Sym) == 1 ? 256 : PK_WIN;
  static constexpr int per_word = 4 / (int)sizeof(Sym);  // symbols per 32-bit register
};

// The job whose CTAs include x: the last with cta0 <= x.
template <class Job>
__device__ __forceinline__ int find_job(const Job* __restrict__ jobs, int n, unsigned x) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].cta0 <= x) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

struct PackShared {
  uint32_t words[PK_WORDS];  // the tile's packed bits from its first bit (tile-relative)
  uint32_t lcode[PK_WIN];    // codes of at most 32 bits, left-aligned (0 for longer codes)
  uint8_t len[PK_WIN];
  unsigned int warp_bits[2][PK_NT / 32];
  unsigned long long excl;
  unsigned int tile;
};

// Code length of symbol s (the cached window, else the global table).
template <class Sym>
__device__ __forceinline__ unsigned pk_len(const PackShared& sh, unsigned s, const uint8_t* __restrict__ len) {
  if (sizeof(Sym) == 1) return sh.len[s];
  const unsigned d = s - (unsigned)PackWin<Sym>::lo;
  return d < (unsigned)PackWin<Sym>::n ? sh.len[d] : __ldg(len + s);
}
// Left-aligned code of symbol s whose length l is at most 32.
template <class Sym>
__device__ __forceinline__ uint32_t pk_lcode(const PackShared& sh, unsigned s, unsigned l,
                                             const unsigned long long* __restrict__ code) {
  if (sizeof(Sym) == 1) return sh.lcode[s];
  const unsigned d = s - (unsigned)PackWin<Sym>::lo;
  if (d < (unsigned)PackWin<Sym>::n) return sh.lcode[d];
  return l ? (uint32_t)(__ldg(code + s) << (32 - l)) : 0u;
}

// Persistent packer.  Tiles of PK_TILE symbols are taken in order from a
// ticket; thread t of a tile owns its symbols t*32 .. t*32+31.
//   1. A tile is taken: its symbols are read, their code lengths (kept in
//      registers) summed and scanned in the CTA, and its bit count published
//      for the look-back (lookback.cuh).
//   2. The codes are packed tile-relative into the shared word buffer: each
//      thread appends its codes to a 32-bit register and stores every word it
//      completes (a word is completed by exactly one thread, which also zeroes
//      the bits of earlier threads in it); after a barrier each thread ORs in
//      its last, partial word.
//   3. The next tile is taken (1), and only then does warp 0 find the starting
//      bit of the one that is packed: its predecessors had that long to
//      publish, so the look-back is one round trip and waits for nobody.  A
//      ticket's count is always published without a wait on another CTA in
//      between, or the look-backs would hold one another up (a ticket taken a
//      whole tile ahead doubled the kernel's time).
//   4. The buffer goes out shifted onto the global word grid with coalesced
//      stores, the two edge words (shared with the neighbouring tiles) by
//      atomicOr.
// A tile with a code longer than 32 bits (possible only for skewed
// histograms) skips 2 and ORs its words straight into global memory.  The
// stream starts at bit `bit0` (0-31) of out[0].
//
// Bound by the latency between its barriers (a ticket, the symbols, a
// look-back, the stores) at half the chip's warps, and by issue: 45 thread
// instructions a u16 symbol, 29 an id.  Both code streams of 8192 x 8192 take
// .49 ms; .59 with the look-back directly after the packing and a 64-bit
// append under a branch.  Measured and no better: five or three CTAs an SM,
// 16 symbols a thread at 256 or 512 threads (.78-.86), codes kept beside the
// lengths (spills), a window lookup without the fallback (a sixth fewer
// instructions, the same time).
template <class Sym, bool MAP0>
__device__ __forceinline__ void pack_stream(const PackJob& J, PackShared& sh, int* __restrict__ flag) {
  const Sym* __restrict__ sym = static_cast<const Sym*>(J.sym);
  const size_t n = J.n, cap_words = J.cap_words;
  const unsigned long long* __restrict__ code = J.tab.code;
  const uint8_t* __restrict__ len = J.tab.len;
  const int nsym = J.tab.nsym, bit0 = J.bit0;
  uint32_t* __restrict__ out = J.out;
  unsigned long long* __restrict__ state = J.scratch + 1;
  unsigned int* __restrict__ ticket = reinterpret_cast<unsigned int*>(J.scratch);
  const unsigned long long ntiles = (n + PK_TILE - 1) / PK_TILE;
  unsigned long long* __restrict__ d_total = J.total_bits;
  using W = PackWin<Sym>;
  constexpr int NW = PK_SPT / W::per_word;  // registers of packed symbols
  constexpr int SB = 8 * (int)sizeof(Sym);
  constexpr unsigned SMASK = sizeof(Sym) == 1 ? 0xffu : 0xffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < W::n; i += PK_NT) {
    int v = W::lo + i;
    if (MAP0 && v == (int)ID_ZERO) v = 0;  // the stream's zero id is symbol 0
    const unsigned l = v < nsym ? len[v] : 0u;
    sh.len[i] = (uint8_t)l;
    sh.lcode[i] = (l >= 1 && l <= 32) ? (uint32_t)(code[v] << (32 - l)) : 0u;
  }
  const bool vec_ok = ((uintptr_t)sym & 15) == 0;
  const unsigned words0 = (unsigned)__cvta_generic_to_shared(&sh.words[0]);
  // A tile in flight: its symbols, their code lengths (4 to a register), the
  // thread's bits and where they start among the tile's.
  uint32_t w[NW] = {}, lw[PK_SPT / 4];
  unsigned int bits = 0, tpre = 0, agg = 0;
  bool any_long = false;
  auto sym_k = [&](int k) -> unsigned { return (w[k / W::per_word] >> (SB * (k % W::per_word))) & SMASK; };
  auto take = [&](unsigned long long tile, int par) {
    const size_t my = (size_t)tile * PK_TILE + (size_t)tid * PK_SPT;
    if (my + PK_SPT <= n && vec_ok) {
      const uint4* src = reinterpret_cast<const uint4*>(sym + my);
#pragma unroll
      for (int q = 0; q < NW / 4; q++) {
        const uint4 v = __ldcs(src + q);
        w[4 * q] = v.x;
        w[4 * q + 1] = v.y;
        w[4 * q + 2] = v.z;
        w[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < NW; q++) w[q] = 0;
#pragma unroll
      for (int k = 0; k < PK_SPT; k++)
        if (my + k < n) w[k / W::per_word] |= (uint32_t)sym[my + k] << (SB * (k % W::per_word));
    }
    unsigned int b = 0, lmax = 0;
#pragma unroll
    for (int k = 0; k < PK_SPT; k++) {
      const unsigned l = pk_len<Sym>(sh, sym_k(k), len);
      b += l;
      lmax = max(lmax, l);
      lw[k / 4] = (k % 4) ? (lw[k / 4] | (l << (8 * (k % 4)))) : l;
    }
    if (my + PK_SPT > n) {  // the stream's end: no bits past it
      b = lmax = 0;
      const int cnt = my >= n ? 0 : (int)(n - my);
#pragma unroll
      for (int k = 0; k < PK_SPT; k++) {
        if (k >= cnt) lw[k / 4] &= ~(255u << (8 * (k % 4)));
        const unsigned l = (lw[k / 4] >> (8 * (k % 4))) & 255u;
        b += l;
        lmax = max(lmax, l);
      }
    }
    unsigned int x = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh.warp_bits[par][warp] = x;
    any_long = __syncthreads_or(lmax > 32) != 0;
    unsigned int wpre = 0;
    agg = 0;
#pragma unroll
    for (int q = 0; q < PK_NT / 32; q++) {
      const unsigned int v = sh.warp_bits[par][q];
      wpre += q < warp ? v : 0u;
      agg += v;
    }
    bits = b;
    tpre = wpre + x - b;
    if (tid == 0) lookback_publish(state, tile, agg);
  };

  if (tid == 0) sh.tile = atomicAdd(ticket, 1u);
  __syncthreads();  // also: the codebook window is in place
  unsigned long long tile = sh.tile;
  if (tile >= ntiles) return;
  take(tile, 0);
  for (int par = 1;; par ^= 1) {
    unsigned int after = 0;
    if (tid == 0) after = atomicAdd(ticket, 1u);
    // 2. tile-relative packing; nobody completes the last partial word
    const bool packed = !any_long;
    const unsigned int t_agg = agg, t_pre = tpre;
    uint32_t acc = 0;  // the word at `at` so far
    unsigned nacc = tpre & 31;  // leading bits of its first word belong to earlier threads
    unsigned at = words0 + 4u * (tpre >> 5);
    if (packed) {
      if (tid == 0 && (agg & 31)) sh.words[agg >> 5] = 0;
#pragma unroll
      for (int k = 0; k < PK_SPT; k++) {
        const unsigned l = (lw[k / 4] >> (8 * (k % 4))) & 255u;
        const uint32_t c = pk_lcode<Sym>(sh, sym_k(k), l, code);
        acc |= c >> nacc;
        const uint32_t rest = __funnelshift_r(0u, c, nacc);  // the code's bits past that word
        nacc += l;
        // a completed word, as one predicated store
        const bool full = nacc >= 32;
        sts_u32_if(full, at, acc);
        acc = full ? rest : acc;
        at += full ? 4u : 0u;
        nacc &= 31;
      }
    }
    if (tid == 0) sh.tile = after;
    __syncthreads();  // every completed word is in place
    // (symbols past the stream's end have left bits below the last code's)
    if (packed && bits > 0 && nacc > 0) atomicOr(&sh.words[(at - words0) >> 2], acc & ~(0xffffffffu >> nacc));
    const unsigned long long next = sh.tile;
    if (next < ntiles) take(next, par);
    else __syncthreads();
    // 3. the starting bit, then the words onto the global grid
    if (warp == 0) {
      const unsigned long long e = lookback_warp(state, tile, t_agg, lane, PK_SPIN_LIMIT, flag);
      if (lane == 0) sh.excl = e;
    }
    __syncthreads();
    const unsigned long long excl = sh.excl;
    const unsigned long long s0 = (unsigned long long)bit0 + excl;
    const unsigned long long w_lo = s0 >> 5;
    if (packed) {
      const unsigned int shift = (unsigned int)(s0 & 31);
      const int nrel = (int)((t_agg + 31) >> 5);
      const int nout = t_agg ? (int)((shift + t_agg - 1) >> 5) + 1 : 0;
      for (int k = tid; k < nout; k += PK_NT) {
        const unsigned long long g = w_lo + (unsigned long long)k;
        if (g >= cap_words) {
          atomicOr(flag, FLAG_OUT_CAPACITY);
          break;
        }
        const uint32_t lo = k < nrel ? sh.words[k] : 0u;
        const uint32_t hi = k > 0 ? sh.words[k - 1] : 0u;
        const uint32_t v = bswap32(shift ? __funnelshift_r(lo, hi, shift) : lo);
        if (k == 0 || k == nout - 1) atomicOr(&out[g], v);  // shared with the neighbouring tiles
        else out[g] = v;
      }
    } else {
      // a code longer than 32 bits: every word ORed
      const size_t my = (size_t)tile * PK_TILE + (size_t)tid * PK_SPT;
      const unsigned int pos = (unsigned int)(s0 & 31) + t_pre;
      int wi = (int)(pos >> 5);
      int nacc = (int)(pos & 31);
      unsigned long long acc = 0;
      bool any = false;
      auto emit = [&]() {
        const unsigned long long g = w_lo + (unsigned long long)wi;
        if (g < cap_words) atomicOr(&out[g], bswap32((uint32_t)(acc >> 32)));
        else atomicOr(flag, FLAG_OUT_CAPACITY);
        wi++;
      };
      auto put = [&](uint32_t v, int l) {  // 1 <= l <= 32, v < 2^l
        acc |= (unsigned long long)v << (64 - nacc - l);
        nacc += l;
        if (nacc >= 32) {
          emit();
          acc <<= 32;
          nacc -= 32;
        }
      };
      for (int k = 0; k < PK_SPT && my + k < n; k++) {
        unsigned s = (unsigned)sym[my + k];
        if (MAP0 && s == ID_ZERO) s = 0;
        const int l = __ldg(len + s);
        const unsigned long long c = __ldg(code + s);
        any |= l > 0;
        if (l > 32) {
          put((uint32_t)(c >> 32) & (uint32_t)((1ull << (l - 32)) - 1), l - 32);
          put((uint32_t)c, 32);
        } else if (l > 0) {
          put((uint32_t)c & (uint32_t)((1ull << l) - 1), l);
        }
      }
      if (any && nacc > 0) emit();
    }
    if (tile == ntiles - 1 && tid == 0 && d_total) *d_total = excl + t_agg;
    if (next >= ntiles) break;
    tile = next;
    __syncthreads();  // the words are written again
  }
}

// The CTAs of a launch are shared out among its streams (PackJob::cta0); a CTA
// takes tiles of its own stream until they run out.  SYM: 1 u8, 2 u16, 0 both.
template <int SYM>
__global__ void __launch_bounds__(PK_NT, PK_CTAS_PER_SM)
    pack_kernel(const __grid_constant__ PackJob one, const PackJob* __restrict__ jobs, int njobs,
                int* __restrict__ flag) {
  __shared__ PackShared sh;
  __shared__ PackJob s_job;
  if (jobs) {
    if (threadIdx.x == 0) s_job = jobs[find_job(jobs, njobs, blockIdx.x)];
    __syncthreads();
  }
  const PackJob& J = jobs ? s_job : one;
  if (SYM == 2 || (SYM == 0 && J.sym_bytes == 2)) pack_stream<uint16_t, false>(J, sh, flag);
  else if (J.map_id_zero) pack_stream<uint8_t, true>(J, sh, flag);
  else pack_stream<uint8_t, false>(J, sh, flag);
}

// Before the packers: the codebook entries of a stream scattered into its
// tables, and the bytes its bits go to zeroed (the packer ORs the words two
// tiles share).  grid.y: the stream; grid.x CTAs take its entries and bytes in
// chunks of 256 and PREP_BYTES.
constexpr unsigned PREP_BYTES = 16384;
__global__ void __launch_bounds__(256) pack_prep_kernel(const PackPrep* __restrict__ jobs) {
  const PackPrep J = jobs[blockIdx.y];
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i < J.n) {
    const HuffEntry v = J.entries[i];
    J.code[v.sym] = v.code;
    J.len[v.sym] = (uint8_t)v.len;
  }
  const size_t b0 = (size_t)blockIdx.x * PREP_BYTES;
  if (b0 >= J.zero_bytes) return;
  const size_t b1 = b0 + PREP_BYTES < J.zero_bytes ? b0 + PREP_BYTES : J.zero_bytes;
  uint8_t* p = J.zero + b0;
  uint8_t* const e = J.zero + b1;
  uint8_t* const lo = (uint8_t*)(((uintptr_t)p + 15) & ~(uintptr_t)15);
  if (lo >= e) {
    for (uint8_t* q = p + threadIdx.x; q < e; q += 256) *q = 0;
    return;
  }
  uint8_t* const hi = (uint8_t*)((uintptr_t)e & ~(uintptr_t)15);
  if (p + threadIdx.x < lo) p[threadIdx.x] = 0;
  if (hi + threadIdx.x < e) hi[threadIdx.x] = 0;
  for (uint8_t* q = lo + 16 * threadIdx.x; q < hi; q += 16 * 256) *reinterpret_cast<uint4*>(q) = make_uint4(0, 0, 0, 0);
}

size_t pack_scratch_words(size_t n) { return (n + PK_TILE - 1) / PK_TILE + 1; }

// CTAs of one of `streams` streams: its share of a full device, or one per
// PK_TILES_PER_CTA tiles if that is more (a CTA loads its stream's codebook
// window once, whatever it packs).
constexpr size_t PK_TILES_PER_CTA = 4;
unsigned pack_ctas(int num_sms, size_t n, int streams) {
  const size_t ntiles = (n + PK_TILE - 1) / PK_TILE, cap = (size_t)num_sms * PK_CTAS_PER_SM;
  const size_t share = std::max((ntiles + PK_TILES_PER_CTA - 1) / PK_TILES_PER_CTA, cap / (size_t)streams);
  return (unsigned)std::min(ntiles, std::min(cap, share));
}

// ---- histogram -------------------------------------------------------------------
constexpr int HIST_NT = 512;
constexpr int HIST_LO = 32768 - 4096;  // shared window of the code histogram
constexpr int HIST_W = 8192;

// Codes concentrate on 32768 and its neighbours (prediction errors of zero and
// one quantum): those three are counted in registers and reduced once per
// warp, so the shared-memory atomics see only the spread-out remainder (no
// 32-way same-address conflicts).  Reads are 16-byte vectors where aligned.
template <bool SKIP0 = false>
__device__ __forceinline__ void hist_add(unsigned int* sh, unsigned long long* hist, unsigned v, unsigned& c_lo,
                                         unsigned& c_mid, unsigned& c_hi) {
  const unsigned d = v - 32767u;
  if (d < 3u) {
    c_lo += d == 0u;
    c_mid += d == 1u;
    c_hi += d == 2u;
  } else if (v == 0u) {
    if (!SKIP0) atomicAdd(&sh[HIST_W], 1u);
  } else if (v - (unsigned)HIST_LO < (unsigned)HIST_W) {
    atomicAdd(&sh[v - HIST_LO], 1u);
  } else {
    atomicAdd(&hist[v], 1ull);
  }
}

// Symbols t0, t0 + stride, ... of s[0, n) into the shared window / registers:
// the elements before the first 16-byte boundary, the vector body, the tail.
template <bool SKIP0 = false>
__device__ __forceinline__ void hist_span(unsigned* sh, unsigned long long* hist, const uint16_t* s, size_t n,
                                          size_t t0, size_t stride, unsigned& c_lo, unsigned& c_mid, unsigned& c_hi) {
  const size_t head = ((16 - ((uintptr_t)s & 15)) & 15) / 2;
  const size_t h = head < n ? head : n;
  if (t0 < h) hist_add<SKIP0>(sh, hist, s[t0], c_lo, c_mid, c_hi);
  const size_t nv = (n - h) / 8;
  const uint4* sv = reinterpret_cast<const uint4*>(s + h);
  for (size_t i = t0; i < nv; i += stride) {
    const uint4 w = __ldcs(sv + i);
    const unsigned ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; q++) {
      hist_add<SKIP0>(sh, hist, ws[q] & 0xffffu, c_lo, c_mid, c_hi);
      hist_add<SKIP0>(sh, hist, ws[q] >> 16, c_lo, c_mid, c_hi);
    }
  }
  for (size_t i = h + nv * 8 + t0; i < n; i += stride) hist_add<SKIP0>(sh, hist, s[i], c_lo, c_mid, c_hi);
}
// The register counts and the shared window into the global histogram.
__device__ __forceinline__ void hist_flush(unsigned* sh, unsigned long long* hist, unsigned c_lo, unsigned c_mid,
                                           unsigned c_hi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c_lo += __shfl_down_sync(0xffffffffu, c_lo, o);
    c_mid += __shfl_down_sync(0xffffffffu, c_mid, o);
    c_hi += __shfl_down_sync(0xffffffffu, c_hi, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (c_lo) atomicAdd(&sh[32767 - HIST_LO], c_lo);
    if (c_mid) atomicAdd(&sh[32768 - HIST_LO], c_mid);
    if (c_hi) atomicAdd(&sh[32769 - HIST_LO], c_hi);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < HIST_W; k += HIST_NT)
    if (sh[k]) atomicAdd(&hist[HIST_LO + k], (unsigned long long)sh[k]);
  if (threadIdx.x == 0 && sh[HIST_W]) atomicAdd(&hist[0], (unsigned long long)sh[HIST_W]);
}

// Component blockIdx.y of a field's codes into its histogram, by the field's
// share of the CTAs; SKIP0: symbol 0 is not counted.
template <bool SKIP0>
__global__ void __launch_bounds__(HIST_NT) hist_u16_kernel(const __grid_constant__ HistJob one,
                                                           const HistJob* __restrict__ jobs, int njobs) {
  __shared__ unsigned int sh[HIST_W + 1];  // window + symbol 0
  __shared__ int s_job;
  if (threadIdx.x == 0) s_job = jobs ? find_job(jobs, njobs, blockIdx.x) : 0;
  for (int k = threadIdx.x; k <= HIST_W; k += HIST_NT) sh[k] = 0;
  __syncthreads();
  const HistJob& J = jobs ? jobs[s_job] : one;
  unsigned long long* __restrict__ hist = J.hist[blockIdx.y];
  unsigned c_lo = 0, c_mid = 0, c_hi = 0;
  hist_span<SKIP0>(sh, hist, J.sym[blockIdx.y], J.n, (size_t)(blockIdx.x - J.cta0) * HIST_NT + threadIdx.x,
                   (size_t)J.ctas * HIST_NT, c_lo, c_mid, c_hi);
  hist_flush(sh, hist, c_lo, c_mid, c_hi);
}

// ---- histogram -> list ---------------------------------------------------------------
// The symbols that occur, ascending, as symbol << 40 | count, and their number,
// written straight into page-locked host memory: the host reads a few thousand
// words where it would copy and scan 65536 bins (512 KB each).
// One CTA per histogram; warp w has bins 2048 w .. 2048 w + 2047, 32 per step,
// so a step's ballot gives every lane its place.
constexpr int LIST_NT = 1024;
constexpr int LIST_STEPS = 65536 / LIST_NT;
__global__ void __launch_bounds__(LIST_NT) hist_list_kernel(const HistList* __restrict__ jobs) {
  const HistList J = jobs[blockIdx.x];
  __shared__ unsigned s_warp[LIST_NT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned bin0 = (unsigned)warp * 32 * LIST_STEPS + lane;
  unsigned n = 0;  // this lane's occurring bins
#pragma unroll 16
  for (int k = 0; k < LIST_STEPS; k++) n += J.hist[bin0 + 32 * k] != 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) n += __shfl_xor_sync(0xffffffffu, n, d);
  if (lane == 0) s_warp[warp] = n;
  __syncthreads();
  unsigned v = s_warp[lane], x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (threadIdx.x == 31) *J.count = x;
  unsigned at = __shfl_sync(0xffffffffu, x - v, warp);
#pragma unroll 16
  for (int k = 0; k < LIST_STEPS; k++) {
    const unsigned long long c = J.hist[bin0 + 32 * k];
    const unsigned m = __ballot_sync(0xffffffffu, c != 0);
    if (c) J.list[at + __popc(m & ((1u << lane) - 1u))] = (unsigned long long)(bin0 + 32 * k) << 40 | c;
    at += __popc(m);
  }
}

// ---- histogram follower ----------------------------------------------------------
// Counts a field's code histograms while its wavefront is still running:
// blockIdx.y is the component; the CTAs take slices of FOLLOW_ROWS rows in
// row order from the component's ticket, wait for the slice's row group to
// be flagged done by the wavefront (thread 0 polls with acquire loads, the
// CTA then acquires), and count the slice.  The wavefront finishes its
// groups in row order, so most of the field is counted during the
// wavefront's tail and only the last group's slices remain once it ends.
// A wait that outlasts FOLLOW_WAIT_NS (the wavefront is not running: a tool
// serialises kernels) sets *gave_up and every CTA stops; the host counts
// the histograms again.
constexpr int FOLLOW_ROWS = 8;
constexpr long long FOLLOW_WAIT_NS = 100000000ll;  // 100 ms

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ long long follow_clock_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__global__ void __launch_bounds__(HIST_NT) hist_follow_kernel(const uint16_t* __restrict__ c0,
                                                              const uint16_t* __restrict__ c1,
                                                              const unsigned* __restrict__ d0,
                                                              const unsigned* __restrict__ d1, int r1, int r2,
                                                              unsigned long long* __restrict__ h0,
                                                              unsigned long long* __restrict__ h1,
                                                              unsigned* __restrict__ tickets, int* gave_up) {
  const uint16_t* __restrict__ codes = blockIdx.y ? c1 : c0;
  const unsigned* __restrict__ done = blockIdx.y ? d1 : d0;
  unsigned long long* __restrict__ hist = blockIdx.y ? h1 : h0;
  __shared__ unsigned int sh[HIST_W + 1];
  __shared__ int s_slice;
  for (int k = threadIdx.x; k <= HIST_W; k += HIST_NT) sh[k] = 0;
  unsigned c_lo = 0, c_mid = 0, c_hi = 0;
  const int nslices = (r1 + FOLLOW_ROWS - 1) / FOLLOW_ROWS;
  for (;;) {
    if (threadIdx.x == 0) {
      int sl = (int)atomicAdd(tickets + blockIdx.y, 1u);
      if (sl < nslices) {
        const unsigned* flag = done + (sl * FOLLOW_ROWS) / WAVE_GROUP_ROWS;
        if (!ld_acquire_u32(flag)) {
          const long long t0 = follow_clock_ns();
          while (!ld_acquire_u32(flag)) {
            if (*(volatile int*)gave_up || follow_clock_ns() - t0 > FOLLOW_WAIT_NS) {
              atomicOr(gave_up, 1);
              sl = nslices;
              break;
            }
            __nanosleep(1000);
          }
        }
      }
      s_slice = sl;
    }
    __syncthreads();
    const int sl = s_slice;
    if (sl >= nslices) break;
    (void)ld_acquire_u32(done + (sl * FOLLOW_ROWS) / WAVE_GROUP_ROWS);
    const int row0 = sl * FOLLOW_ROWS, rows = min(FOLLOW_ROWS, r1 - row0);
    hist_span(sh, hist, codes + (size_t)row0 * r2, (size_t)rows * r2, threadIdx.x, HIST_NT, c_lo, c_mid, c_hi);
    __syncthreads();  // s_slice is rewritten only after every thread has read it
  }
  hist_flush(sh, hist, c_lo, c_mid, c_hi);
}

}  // namespace

size_t huff_encode_tmp_bytes(size_t n) { return align_up(pack_scratch_words(n), 32) * sizeof(unsigned long long); }

int launch_pack_prep(cpsz_b200_ctx* ctx, const PackPrep* d_jobs, int n, size_t max_entries, size_t max_zero_bytes) {
  const size_t gx = std::max((max_entries + 255) / 256, (max_zero_bytes + PREP_BYTES - 1) / PREP_BYTES);
  if (n <= 0 || gx == 0) return CPSZ_OK;
  pack_prep_kernel<<<dim3((unsigned)gx, (unsigned)n), 256, 0, ctx->stream>>>(d_jobs);
  count_launch(ctx);
  return check_launch("pack_prep_kernel");
}

unsigned pack_assign_ctas(int num_sms, PackJob* jobs, int n) {
  unsigned at = 0;
  for (int k = 0; k < n; k++) {
    jobs[k].cta0 = at;
    at += pack_ctas(num_sms, jobs[k].n, n);
  }
  return at;
}

int launch_pack(cudaStream_t st, const PackJob* jobs, const PackJob* d_jobs, int n, unsigned ctas, int* flag) {
  if (ctas == 0) return CPSZ_OK;
  bool u8 = false, u16 = false;
  for (int k = 0; k < n; k++) {
    if (jobs[k].bit0 < 0 || jobs[k].bit0 > 31)
      return set_error(CPSZ_ERR_INVALID, "internal: stream start bit %d", jobs[k].bit0);
    (jobs[k].sym_bytes == 2 ? u16 : u8) = true;
  }
  const PackJob* table = n == 1 ? nullptr : d_jobs;
  if (u8 && u16) pack_kernel<0><<<ctas, PK_NT, 0, st>>>(jobs[0], table, n, flag);
  else if (u16) pack_kernel<2><<<ctas, PK_NT, 0, st>>>(jobs[0], table, n, flag);
  else pack_kernel<1><<<ctas, PK_NT, 0, st>>>(jobs[0], table, n, flag);
  return check_launch("pack_kernel");
}

int launch_huff_encode(cpsz_b200_ctx* ctx, PackJob job) {
  if (job.n == 0) return CPSZ_OK;
  CPSZ_CUDA_TRY(cudaMemsetAsync(job.scratch, 0, pack_scratch_words(job.n) * 8, ctx->stream));
  CPSZ_TRY(launch_pack(ctx->stream, &job, nullptr, 1, pack_assign_ctas(ctx->num_sms, &job, 1), ctx->d_flag));
  count_launch(ctx);
  return CPSZ_OK;
}

// About two CTAs per SM in all, each with at least 16 symbols a thread: a CTA
// clears and flushes an 8192-bin window whatever it counts.
unsigned hist_assign_ctas(int num_sms, HistJob* jobs, int n) {
  size_t total = 0;
  for (int k = 0; k < n; k++) total += jobs[k].n;
  const size_t share = std::max<size_t>(16 * HIST_NT, (total + num_sms - 1) / num_sms);
  unsigned at = 0;
  for (int k = 0; k < n; k++) {
    jobs[k].cta0 = at;
    jobs[k].ctas = (unsigned)std::max<size_t>(1, (jobs[k].n + share - 1) / share);
    at += jobs[k].ctas;
  }
  return at;
}

int launch_hist_u16(cpsz_b200_ctx* ctx, const HistJob* jobs, const HistJob* d_jobs, int n, unsigned ctas) {
  hist_u16_kernel<false><<<dim3(ctas, 2), HIST_NT, 0, ctx->stream>>>(jobs[0], n == 1 ? nullptr : d_jobs, n);
  count_launch(ctx);
  return check_launch("hist_u16_kernel");
}

int launch_hist_u16_nonzero(cpsz_b200_ctx* ctx, const uint16_t* sym, size_t n, unsigned long long* hist) {
  if (n == 0) return CPSZ_OK;
  HistJob job{{sym, nullptr}, {hist, nullptr}, n, 0, 0};
  job.ctas = (unsigned)std::min<size_t>((size_t)ctx->num_sms * 2, (n + HIST_NT - 1) / HIST_NT);
  hist_u16_kernel<true><<<dim3(job.ctas, 1), HIST_NT, 0, ctx->stream>>>(job, nullptr, 1);
  count_launch(ctx);
  return check_launch("hist_u16_kernel");
}

int launch_hist_list(cpsz_b200_ctx* ctx, const HistList* d_jobs, int n, cudaStream_t stream) {
  if (n <= 0) return CPSZ_OK;
  hist_list_kernel<<<n, LIST_NT, 0, stream>>>(d_jobs);
  count_launch(ctx);
  return check_launch("hist_list_kernel");
}

int launch_hist_follow(cpsz_b200_ctx* ctx, const uint16_t* const codes[2], const unsigned* const group_done[2], int r1,
                       int r2, unsigned long long* const hist[2], unsigned* tickets, int* gave_up, cudaStream_t stream) {
  if (r1 <= 0 || r2 <= 0) return CPSZ_OK;
  const int nslices = (r1 + FOLLOW_ROWS - 1) / FOLLOW_ROWS;
  const int grid = std::min(nslices, ctx->num_sms);
  hist_follow_kernel<<<dim3(grid, 2), HIST_NT, 0, stream>>>(codes[0], codes[1], group_done[0], group_done[1], r1, r2,
                                                            hist[0], hist[1], tickets, gave_up);
  count_launch(ctx);
  return check_launch("hist_follow_kernel");
}

// ---- Huffman packing without any allocation ---------------------------------------------
//
// Some callers cannot allocate device memory at the point where they encode:
// an in-situ analysis hook running inside a simulation that reserved all GPU
// memory for its own pool at start-up, a plugin that is only handed
// preallocated buffers by its host framework, or a real-time loop where a
// cudaMalloc (which may synchronise the device) is not allowed.  For them
// this entry point packs a symbol stream with the same kernel as
// cpsz_b200_huffman_encode_u16 but takes its scratch -- the tile ticket and
// the per-tile look-back states -- from a fixed array in this file instead of
// a context workspace.  The array (about 64 KB) lives on every GPU that loads
// the library until the process exits, and it bounds the stream length.

constexpr size_t kNoAllocMaxSymbols = size_t(1) << 26;  // 67,108,864 symbols per call
constexpr size_t kNoAllocTiles = kNoAllocMaxSymbols / PK_TILE;
// layout: [ticket][tile states: kNoAllocTiles][flag word]
static __device__ __align__(256) unsigned long long g_noalloc_scratch[1 + kNoAllocTiles + 1];

namespace {

// The array's device address in the calling thread's current context.  It is
// looked up on every call (a lookup, no allocation): an address cached once
// per device would go stale after a device reset, or in a context the caller
// created and made current itself, and kernels given it would write to memory
// that is no longer the array.
int noalloc_scratch(unsigned long long** out) {
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess)
    return set_error(e == cudaErrorNoDevice ? CPSZ_ERR_NO_DEVICE : CPSZ_ERR_CUDA,
                     "cudaGetSymbolAddress of the no-alloc scratch: %s", cudaGetErrorString(e));
  *out = (unsigned long long*)p;
  return CPSZ_OK;
}

}  // namespace

}  // namespace cpsz

extern "C" int cpsz_b200_huffman_encode_u16_noalloc(const uint16_t* sym, size_t n, const uint64_t* code,
                                                    const uint8_t* len, unsigned char* out, size_t out_cap,
                                                    uint64_t* total_bits, void* stream) {
  using namespace cpsz;
  clear_error();
  if (!sym || !code || !len || !out || !total_bits) return set_error(CPSZ_ERR_INVALID, "null pointer argument");
  if (((uintptr_t)out & 3) != 0) return set_error(CPSZ_ERR_INVALID, "output must be 4-byte aligned");
  // the packer stores whole 32-bit words: a capacity that is not a multiple of
  // 4 would leave its last bytes unwritten without the overflow rule noticing
  if (out_cap % 4 != 0) return set_error(CPSZ_ERR_INVALID, "out_cap (%zu) must be a multiple of 4", out_cap);
  if (n > kNoAllocMaxSymbols)
    return set_error(CPSZ_ERR_INVALID, "%zu symbols exceed the no-alloc maximum of %zu symbols per call", n,
                     kNoAllocMaxSymbols);
  unsigned long long* scratch = nullptr;
  CPSZ_TRY(noalloc_scratch(&scratch));
  cudaStream_t st = (cudaStream_t)stream;
  int* flag = (int*)(scratch + 1 + kNoAllocTiles);
  // the packer ORs the edge words of every tile: the output starts at zero
  CPSZ_CUDA_TRY(cudaMemsetAsync(out, 0, out_cap, st));
  CPSZ_CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(unsigned long long), st));
  if (n == 0) {
    CPSZ_CUDA_TRY(cudaMemsetAsync(total_bits, 0, sizeof(uint64_t), st));
    return CPSZ_OK;
  }
  int dev = 0, sms = 0;
  CPSZ_CUDA_TRY(cudaGetDevice(&dev));
  CPSZ_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  PackJob job;
  job.sym = sym;
  job.n = n;
  job.sym_bytes = 2;
  job.tab = HuffEncTable{(const unsigned long long*)code, len, 65536};
  job.out = (uint32_t*)out;
  job.cap_words = out_cap / 4;
  job.scratch = scratch;
  job.total_bits = (unsigned long long*)total_bits;
  CPSZ_CUDA_TRY(cudaMemsetAsync(scratch, 0, pack_scratch_words(n) * 8, st));
  CPSZ_TRY(launch_pack(st, &job, nullptr, 1, pack_assign_ctas(sms, &job, 1), flag));
  return check_launch("huffman no-alloc encode");
}
