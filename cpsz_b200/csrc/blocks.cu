// blocks.cu -- 12x12 block-order plumbing of the 2D field blobs, and a
// generic device-wide exclusive scan.
//
// The reference emits quantization codes and unpredictable values in 12x12
// block order (blocks row-major, rows inside a block, src/sz_compress_3d.cpp:
// 126-193): element (i, j) sits at block-order position
//   bi*12*r2 + bj*12*h + li*w + lj,   h = rows of block-row bi (12, or the
//   remainder), w = columns of block bj (12, or the remainder).
#include <algorithm>

#include "kernels.h"
#include "lookback.cuh"

namespace cpsz {

namespace {

constexpr int BS = 12;
constexpr unsigned FULLM = 0xffffffffu;

// ---- generic exclusive scan (u32) ---------------------------------------------------
constexpr int SCAN_NT = 1024;
constexpr int SCAN_PER = 8;
constexpr int SCAN_CHUNK = SCAN_NT * SCAN_PER;

__device__ __forceinline__ unsigned int block_exclusive_scan(unsigned int v, unsigned int* warp_tot,
                                                             unsigned int* total) {
  unsigned int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) >= o) x += y;
  }
  if ((threadIdx.x & 31) == 31) warp_tot[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned int w = (threadIdx.x < blockDim.x / 32) ? warp_tot[threadIdx.x] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      unsigned int y = __shfl_up_sync(0xffffffffu, w, o);
      if (threadIdx.x >= o) w += y;
    }
    warp_tot[threadIdx.x] = w;
  }
  __syncthreads();
  unsigned int pre = (threadIdx.x >= 32 ? warp_tot[(threadIdx.x >> 5) - 1] : 0u) + x - v;
  if (total) *total = warp_tot[blockDim.x / 32 - 1];
  __syncthreads();
  return pre;
}

__global__ void __launch_bounds__(SCAN_NT) scan_reduce_kernel(const unsigned int* __restrict__ in, size_t n,
                                                              unsigned int* __restrict__ part) {
  __shared__ unsigned int warp_tot[32];
  size_t base = (size_t)blockIdx.x * SCAN_CHUNK;
  unsigned int s = 0;
  for (int k = 0; k < SCAN_PER; k++) {
    size_t i = base + (size_t)k * SCAN_NT + threadIdx.x;
    if (i < n) s += in[i];
  }
  unsigned int total;
  block_exclusive_scan(s, warp_tot, &total);
  if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_NT) scan_partials_kernel(unsigned int* __restrict__ part, size_t np) {
  __shared__ unsigned int warp_tot[32];
  __shared__ unsigned int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (size_t base = 0; base < np; base += SCAN_NT) {
    size_t i = base + threadIdx.x;
    unsigned int v = i < np ? part[i] : 0u;
    unsigned int total;
    unsigned int pre = block_exclusive_scan(v, warp_tot, &total);
    if (i < np) part[i] = carry + pre;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) part[np] = carry;
}

__global__ void __launch_bounds__(SCAN_NT) scan_down_kernel(const unsigned int* __restrict__ in, size_t n,
                                                            const unsigned int* __restrict__ part,
                                                            unsigned int* __restrict__ out) {
  __shared__ unsigned int warp_tot[32];
  size_t base = (size_t)blockIdx.x * SCAN_CHUNK + (size_t)threadIdx.x * SCAN_PER;
  unsigned int v[SCAN_PER];
  unsigned int s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    size_t i = base + k;
    v[k] = i < n ? in[i] : 0u;
    s += v[k];
  }
  unsigned int pre = block_exclusive_scan(s, warp_tot, nullptr) + part[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_PER; k++) {
    size_t i = base + k;
    if (i < n) out[i] = pre;
    pre += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = part[gridDim.x];
}

// ---- strips: a 12-row block row cut into runs of STRIP_BLOCKS blocks ----------------
// A strip's blocks are consecutive in block order, so its block-order image is
// one contiguous range.  A CTA holds that image in shared memory, at the
// range's own 16-byte phase, and moves it to or from global memory in 16-byte
// pieces; on the raster side it is reached four columns at a time (12 = 3 * 4,
// so four columns never leave a block's row, and their place in the image is
// 8-byte aligned).  The unpredictable values are the image's zeros in order.
//
// Bound by the latency of a strip's few dependent round trips (ticket, rows,
// look-back), hidden by other strips: small CTAs, as many as 42 registers a
// thread allow.  Both components of 8192 x 8192 take .32 ms to block order and
// .34 back (.57 and .58 with rows in shared memory, an element's place worked
// out by itself and four CTAs of 256 threads an SM; .34 and .35 with eight of
// 256, .34 and .38 with sixteen of 128).
constexpr int STRIP_BLOCKS = 32;
constexpr int STRIP_W = STRIP_BLOCKS * BS;  // 384 columns
constexpr int STRIP_NT = 128;
constexpr int STRIP_E = BS * STRIP_W;                // 4608 elements
constexpr int STRIP_IMG = STRIP_E + 16;              // shared image, with room for its phase
constexpr int STRIP_VEC = (STRIP_E / 8 + STRIP_NT - 1) / STRIP_NT;   // 16-byte vectors per thread: 5
constexpr int STRIP_GRP = (STRIP_E / 4 + STRIP_NT - 1) / STRIP_NT;   // groups of 4 columns per thread: 9
constexpr int STRIP_CTAS = 12;                       // per SM: latency is hidden by other strips
constexpr int STRIP_RUN = 36;                        // consecutive elements whose zeros a thread counts
static_assert(STRIP_NT * STRIP_RUN >= STRIP_E, "every element has its thread");

struct StripGeom {
  int bi, h, c0, W, nb, wl;
  long long out0;  // block-order position of the strip's first element
};
__device__ __forceinline__ StripGeom strip_geom(long long s, int r1, int r2, int nsc) {
  StripGeom g;
  g.bi = (int)(s / nsc);
  const int sc = (int)(s - (long long)g.bi * nsc);
  g.h = min(BS, r1 - g.bi * BS);
  g.c0 = sc * STRIP_W;
  g.W = min(STRIP_W, r2 - g.c0);
  g.nb = (g.W + BS - 1) / BS;
  g.wl = g.W - (g.nb - 1) * BS;  // width of the strip's last block (12 unless it ends the row)
  g.out0 = (long long)g.bi * BS * r2 + (long long)sc * STRIP_BLOCKS * BS * g.h;
  return g;
}

// Element e of a strip's block-order image: row and column in the strip.
// Every block but the last is 12 wide, so b = e / (12 h) clamped to the last.
__device__ __forceinline__ void strip_pos(const StripGeom& g, int e, int& li, int& col) {
  const int b = min(e / (BS * g.h), g.nb - 1);
  const int k = e - b * BS * g.h, w = b == g.nb - 1 ? g.wl : BS;
  li = k / w;
  col = b * BS + (k - li * w);
}
// The inverse: the image's element at (li, col).
__device__ __forceinline__ int strip_elem(const StripGeom& g, int li, int col) {
  const int b = col / BS, w = b == g.nb - 1 ? g.wl : BS;
  return b * BS * g.h + li * w + (col - b * BS);
}

// The strips' unpredictable counts are summed by decoupled look-back
// (lookback.cuh): a CTA takes the next strip in ticket order, so every
// earlier strip belongs to a CTA that is running or done.  One load per lane
// could not keep pace with tens of thousands of strips (windows of in-flight
// strips that had not yet published their prefix grew to hundreds), hence
// the look-back's several windows per round trip.
constexpr long long LOOKBACK_SPIN = 1ll << 24;

// Whether a zero code may be among the two halves of a word (exact when none
// is: a false alarm needs a true zero below it).
__device__ __forceinline__ unsigned zero_half(unsigned v) { return (v - 0x00010001u) & ~v & 0x80008000u; }

struct StripShared {
  __align__(16) uint16_t img[STRIP_IMG];
  unsigned int warp_z[STRIP_NT / 32];
  unsigned int idx;
  unsigned long long excl;
};

// Zeros of this thread's run of the image (the STRIP_RUN elements from
// STRIP_RUN tid on), and of all earlier threads'; total in every thread.  All
// threads call it.
__device__ __forceinline__ unsigned strip_zeros(StripShared& sh, const uint16_t* img, int E, unsigned& before,
                                                unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = (int)threadIdx.x * STRIP_RUN, n = min(STRIP_RUN, E - e0);
  unsigned z = 0;
  for (int k = 0; k < n; k++) z += img[e0 + k] == 0;
  unsigned x = z;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned y = __shfl_up_sync(FULLM, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) sh.warp_z[warp] = x;
  __syncthreads();
  before = x - z;
  total = 0;
#pragma unroll
  for (int q = 0; q < STRIP_NT / 32; q++) {
    const unsigned v = sh.warp_z[q];
    before += q < warp ? v : 0u;
    total += v;
  }
  return z;
}

// Compression, one launch for both components of every field: codes raster ->
// block order, and the unpredictable values (code 0) in block order.
__global__ void __launch_bounds__(STRIP_NT, STRIP_CTAS) strip_pass_kernel(const __grid_constant__ StripJob one,
                                                              const StripJob* __restrict__ jobs, int njobs, int* flag) {
  __shared__ StripShared sh;
  __shared__ int s_job;
  if (jobs) {
    // the last job with strip0 <= blockIdx.x: a warp counts them, its loads
    // independent of one another (a binary search's are a chain)
    if (threadIdx.x < 32) {
      int n = 0;
      for (int k = threadIdx.x; k < njobs; k += 32) n += jobs[k].strip0 <= blockIdx.x;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) n += __shfl_xor_sync(FULLM, n, d);
      if (threadIdx.x == 0) s_job = n - 1;
    }
    __syncthreads();
  }
  const StripJob& J = jobs ? jobs[s_job] : one;
  const int c = blockIdx.y, r1 = J.r1, r2 = J.r2, nsc = (r2 + STRIP_W - 1) / STRIP_W;
  const unsigned int ns = (unsigned)((r1 + BS - 1) / BS) * (unsigned)nsc;
  unsigned long long* const status = J.status[c];
  if (threadIdx.x == 0) sh.idx = atomicAdd(reinterpret_cast<unsigned int*>(status + ns), 1u);
  __syncthreads();
  const unsigned int s = sh.idx;
  const StripGeom g = strip_geom(s, r1, r2, nsc);
  const int E = g.h * g.W, phase = (int)(g.out0 & 7);
  uint16_t* const img = sh.img + phase;

  // the raster's rows into the image: four columns of full blocks at a time,
  // from the two 8-byte words that hold them (one when they are aligned)
  const uint16_t* src = J.raster[c] + (long long)g.bi * BS * r2 + g.c0;
  const int nfull = g.W / BS, ng = 3 * nfull, tot = g.h * ng;
  unsigned any = 0;
  uint2 v[STRIP_GRP];
#pragma unroll
  for (int it = 0; it < STRIP_GRP; it++) {
    const int q = threadIdx.x + it * STRIP_NT;
    if (q < tot) {
      const int li = ng == 96 ? q / 96 : q / ng, gr = q - li * ng;
      const uint16_t* p = src + (long long)li * r2 + 4 * gr;
      const unsigned a = (unsigned)((uintptr_t)p & 7);
      const uint2* w = reinterpret_cast<const uint2*>(p - a / 2);
      uint2 x = __ldg(w);
      if (a) {
        const uint2 y = __ldg(w + 1);
        const unsigned sft = 8 * (a & 3);
        const unsigned t0 = a & 4 ? x.y : x.x, t1 = a & 4 ? y.x : x.y, t2 = a & 4 ? y.y : y.x;
        x = make_uint2(__funnelshift_r(t0, t1, sft), __funnelshift_r(t1, t2, sft));
      }
      v[it] = x;
    }
  }
#pragma unroll
  for (int it = 0; it < STRIP_GRP; it++) {
    const int q = threadIdx.x + it * STRIP_NT;
    if (q < tot) {
      const int li = ng == 96 ? q / 96 : q / ng, gr = q - li * ng, b = gr / 3;
      *reinterpret_cast<uint2*>(img + (b * g.h + li) * BS + 4 * (gr - 3 * b)) = v[it];
      any |= zero_half(v[it].x) | zero_half(v[it].y);
    }
  }
  const int rem = g.W - BS * nfull;  // the field's last, narrower block
  for (int q = threadIdx.x; q < g.h * rem; q += STRIP_NT) {
    const int li = q / rem, cc = q - li * rem;
    const uint16_t x = src[(long long)li * r2 + BS * nfull + cc];
    img[nfull * BS * g.h + q] = x;
    any |= x == 0;
  }
  const bool some = __syncthreads_or(any != 0) != 0;
  unsigned before = 0, total = 0, z = 0;
  if (some) z = strip_zeros(sh, img, E, before, total);
  if (threadIdx.x == 0) lookback_publish(status, s, total);

  // the image, 16 bytes at a time between the range's ends
  uint16_t* const dst = J.blocks[c] + g.out0;
  const int head = (reinterpret_cast<uintptr_t>(J.blocks[c]) & 15) ? E : min(E, (8 - phase) & 7);
  const int nvec = (E - head) >> 3, tail0 = head + 8 * nvec;
  for (int q = threadIdx.x; q < nvec; q += STRIP_NT)
    *reinterpret_cast<uint4*>(dst + head + 8 * q) = *reinterpret_cast<const uint4*>(img + head + 8 * q);
  for (int q = threadIdx.x; q < head + (E - tail0); q += STRIP_NT) {
    const int e = q < head ? q : tail0 + (q - head);
    dst[e] = img[e];
  }

  if (threadIdx.x < 32) {
    const unsigned long long excl = lookback_warp(status, s, total, (int)threadIdx.x, LOOKBACK_SPIN, flag);
    if (threadIdx.x == 0) {
      sh.excl = excl;
      if (s == ns - 1) J.total[c] = (unsigned int)(excl + total);
    }
  }
  if (!some) return;
  __syncthreads();

  // unpredictable values, in block order
  if (z) {
    float* out = J.unpred[c] + sh.excl + before;
    const float* x = J.x[c] + (long long)g.bi * BS * r2 + g.c0;
    const int e0 = (int)threadIdx.x * STRIP_RUN, n = min(STRIP_RUN, E - e0);
    for (int k = 0; k < n; k++)
      if (img[e0 + k] == 0) {
        int li, col;
        strip_pos(g, e0 + k, li, col);
        *out++ = x[(long long)li * r2 + col];
      }
  }
}

struct StripUnpass {
  const uint16_t* blocks;      // block-order codes
  const uint8_t* ids;          // the component's error-bound ids, raster order (pitch r2)
  const float* unpred;         // unpredictable values, block order
  unsigned long long n_unpred;
  float2* pair;                // raster (pitch r2)
  unsigned long long* status;  // as in StripJob
  unsigned* total;
  int id_shift;                // p = 2^(id_shift * id) * 2^-52: 2 (offline), 1 (offline_log)
};

// Decompression side of a point: the addend 2(code - 32768) * p that the
// wavefront adds to its prediction (p = 4^id * 2^-52 for the offline blob,
// 2^id * 2^-52 for the offline_log one, 0 for id 0;
// src/sz_decompress_cp_preserve_2d.cpp:30-34 and :76-80,
// include/sz_decompression_utils.hpp:65-73), or for code 0 the raw flag with
// the raw value in .x.
__device__ __forceinline__ float2 dec_pair(unsigned int code, unsigned int id, int shift) {
  const float p = id ? __int_as_float((int)(shift * (int)id - 52 + 127) << 23) : 0.f;
  return make_float2((float)(2 * ((int)code - 32768)) * p, __int_as_float(code == 0 ? 1 : 0));
}

// Decompression, one launch for both components: block-order codes -> the
// raster pairs the wavefront reads, with the unpredictable values (block
// order) scattered into the pairs of the zero codes.  The last strip stores
// the number of zero codes, which the host checks against the stored list.
__global__ void __launch_bounds__(STRIP_NT, STRIP_CTAS) strip_unpass_kernel(StripUnpass P0, StripUnpass P1, int r1, int r2,
                                                                int nsc, unsigned int ns, int* flag) {
  __shared__ StripShared sh;
  const StripUnpass P = blockIdx.y ? P1 : P0;
  if (threadIdx.x == 0) {
    const bool again = decode_again(flag);
    const unsigned int t = atomicAdd(reinterpret_cast<unsigned int*>(P.status + ns), 1u);
    sh.idx = again ? ns : t;
  }
  __syncthreads();
  const unsigned int s = sh.idx;
  if (s >= ns) return;
  const StripGeom g = strip_geom(s, r1, r2, nsc);
  const int E = g.h * g.W, phase = (int)(g.out0 & 7);
  uint16_t* const img = sh.img + phase;

  // the block-order codes, 16 bytes at a time between the range's ends
  const uint16_t* src = P.blocks + g.out0;
  const int head = (reinterpret_cast<uintptr_t>(P.blocks) & 15) ? E : min(E, (8 - phase) & 7);
  const int nvec = (E - head) >> 3, tail0 = head + 8 * nvec;
  unsigned any = 0;
  uint4 v[STRIP_VEC];
#pragma unroll
  for (int it = 0; it < STRIP_VEC; it++) {
    const int q = threadIdx.x + it * STRIP_NT;
    if (q < nvec) v[it] = __ldg(reinterpret_cast<const uint4*>(src + head + 8 * q));
  }
#pragma unroll
  for (int it = 0; it < STRIP_VEC; it++) {
    const int q = threadIdx.x + it * STRIP_NT;
    if (q < nvec) {
      *reinterpret_cast<uint4*>(img + head + 8 * q) = v[it];
      any |= zero_half(v[it].x) | zero_half(v[it].y) | zero_half(v[it].z) | zero_half(v[it].w);
    }
  }
  for (int q = threadIdx.x; q < head + (E - tail0); q += STRIP_NT) {
    const int e = q < head ? q : tail0 + (q - head);
    const uint16_t x = src[e];
    img[e] = x;
    any |= x == 0;
  }
  const bool some = __syncthreads_or(any != 0) != 0;
  unsigned before = 0, total = 0, z = 0;
  if (some) z = strip_zeros(sh, img, E, before, total);
  if (threadIdx.x == 0) lookback_publish(P.status, s, total);

  // raster pairs
  const long long row0 = (long long)g.bi * BS;
  if ((r2 & 3) == 0 && ((reinterpret_cast<uintptr_t>(P.ids) & 3) | (reinterpret_cast<uintptr_t>(P.pair) & 15)) == 0) {
    // 4 columns per item (W is a multiple of 4 here, and so is every block's
    // width): one u32 of ids in, two 16-byte pair stores out
    const int nq = g.W >> 2, tot = g.h * nq;
    unsigned int idv[STRIP_GRP];
#pragma unroll
    for (int u = 0; u < STRIP_GRP; u++) {
      const int q = threadIdx.x + u * STRIP_NT;
      if (q < tot) {
        const int li = nq == 96 ? q / 96 : q / nq;
        idv[u] = __ldg(reinterpret_cast<const unsigned int*>(P.ids + (row0 + li) * r2 + g.c0) + (q - li * nq));
      }
    }
#pragma unroll
    for (int u = 0; u < STRIP_GRP; u++) {
      const int q = threadIdx.x + u * STRIP_NT;
      if (q < tot) {
        const int li = nq == 96 ? q / 96 : q / nq, gr = q - li * nq, b = gr / 3;
        const int w = b == g.nb - 1 ? g.wl : BS;
        const uint2 cw = *reinterpret_cast<const uint2*>(img + b * BS * g.h + li * w + 4 * (gr - 3 * b));
        const float2 a = dec_pair(cw.x & 0xffffu, idv[u] & 0xffu, P.id_shift),
                     d = dec_pair(cw.x >> 16, (idv[u] >> 8) & 0xffu, P.id_shift);
        const float2 e = dec_pair(cw.y & 0xffffu, (idv[u] >> 16) & 0xffu, P.id_shift),
                     f = dec_pair(cw.y >> 16, idv[u] >> 24, P.id_shift);
        float4* out = reinterpret_cast<float4*>(P.pair + (row0 + li) * r2 + g.c0 + 4 * gr);
        out[0] = make_float4(a.x, a.y, d.x, d.y);
        out[1] = make_float4(e.x, e.y, f.x, f.y);
      }
    }
  } else {
#pragma unroll 6
    for (int q = threadIdx.x; q < E; q += STRIP_NT) {
      const int li = g.W == STRIP_W ? q / STRIP_W : q / g.W, c = q - li * g.W;
      const long long gi = (row0 + li) * r2 + g.c0 + c;
      P.pair[gi] = dec_pair(img[strip_elem(g, li, c)], P.ids[gi], P.id_shift);
    }
  }

  if (threadIdx.x < 32) {
    const unsigned long long excl = lookback_warp(P.status, s, total, (int)threadIdx.x, LOOKBACK_SPIN, flag);
    if (threadIdx.x == 0) {
      sh.excl = excl;
      if (s == ns - 1) *P.total = (unsigned int)(excl + total);
    }
  }
  if (!some) return;
  __syncthreads();  // also: the raw values below overwrite .x of pairs stored above

  // unpredictable values, in block order
  if (z) {
    unsigned long long o = sh.excl + before;
    const int e0 = (int)threadIdx.x * STRIP_RUN, n = min(STRIP_RUN, E - e0);
    for (int k = 0; k < n; k++)
      if (img[e0 + k] == 0) {
        int li, col;
        strip_pos(g, e0 + k, li, col);
        if (o < P.n_unpred) P.pair[(row0 + li) * r2 + g.c0 + col].x = P.unpred[o];
        else atomicOr(flag, FLAG_RAW_RANGE);
        o++;
      }
  }
}

// ---- byte runs ------------------------------------------------------------------------
// Whole words of the destination from two source words each (the two sides'
// alignments differ), single bytes at a chunk's ends.
constexpr int PIECE_CHUNK = 8192;
__global__ void __launch_bounds__(256) copy_pieces_kernel(const CopyPiece* __restrict__ pieces, int n) {
  __shared__ int s_piece;
  if (threadIdx.x == 0) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (pieces[mid].chunk0 <= blockIdx.x) lo = mid;
      else hi = mid - 1;
    }
    s_piece = lo;
  }
  __syncthreads();
  const CopyPiece P = pieces[s_piece];
  const size_t c0 = (size_t)(blockIdx.x - P.chunk0) * PIECE_CHUNK;
  if (c0 >= P.n) return;
  const int len = (int)(P.n - c0 < (size_t)PIECE_CHUNK ? P.n - c0 : (size_t)PIECE_CHUNK);
  uint8_t* d = P.dst + c0;
  const uint8_t* s = P.src ? P.src + c0 : nullptr;
  const int head = min(len, (int)((4 - ((uintptr_t)d & 3)) & 3)), words = (len - head) >> 2, tail = head + 4 * words;
  if (threadIdx.x < 8) {
    const int i = threadIdx.x < 4 ? (int)threadIdx.x : tail + (int)threadIdx.x - 4;
    if (threadIdx.x < 4 ? i < head : i < len) d[i] = s ? s[i] : 0;
  }
  uint32_t* dw = reinterpret_cast<uint32_t*>(d + head);
  if (!s) {
    for (int k = threadIdx.x; k < words; k += 256) dw[k] = 0;
    return;
  }
  const uint8_t* sb = s + head;
  const unsigned sh = 8 * ((uintptr_t)sb & 3);
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(sb - ((uintptr_t)sb & 3));
  if (sh == 0) {
    for (int k = threadIdx.x; k < words; k += 256) dw[k] = sw[k];
  } else {  // sw[k + 1] holds a byte of the run, so it is readable
    for (int k = threadIdx.x; k < words; k += 256) dw[k] = __funnelshift_r(sw[k], sw[k + 1], sh);
  }
}

}  // namespace

size_t scan_u32_tmp_bytes(size_t n) { return ((n + SCAN_CHUNK - 1) / SCAN_CHUNK + 2) * sizeof(unsigned int) + 256; }

int launch_scan_u32(cpsz_b200_ctx* ctx, const unsigned int* in, unsigned int* out, size_t n, void* tmp) {
  size_t nb = (n + SCAN_CHUNK - 1) / SCAN_CHUNK;
  if (nb == 0) {
    cudaMemsetAsync(out, 0, sizeof(unsigned int), ctx->stream);
    return CPSZ_OK;
  }
  unsigned int* part = (unsigned int*)tmp;
  scan_reduce_kernel<<<(unsigned)nb, SCAN_NT, 0, ctx->stream>>>(in, n, part);
  scan_partials_kernel<<<1, SCAN_NT, 0, ctx->stream>>>(part, nb);
  scan_down_kernel<<<(unsigned)nb, SCAN_NT, 0, ctx->stream>>>(in, n, part, out);
  count_launch(ctx, 3);
  return check_launch("scan_u32");
}

unsigned assign_piece_chunks(CopyPiece* pieces, size_t n) {
  unsigned at = 0;
  for (size_t k = 0; k < n; k++) {
    pieces[k].chunk0 = at;
    at += (unsigned)std::max<size_t>(1, (pieces[k].n + PIECE_CHUNK - 1) / PIECE_CHUNK);
  }
  return at;
}

int launch_copy_pieces(cpsz_b200_ctx* ctx, const CopyPiece* d_pieces, int n, unsigned ctas) {
  if (n <= 0) return CPSZ_OK;
  copy_pieces_kernel<<<ctas, 256, 0, ctx->stream>>>(d_pieces, n);
  count_launch(ctx);
  return check_launch("copy_pieces_kernel");
}

size_t strip_count(int r1, int r2) {
  const long long nbx = (r1 + BS - 1) / BS, nsc = (r2 + STRIP_W - 1) / STRIP_W;
  return (size_t)(nbx * nsc);
}

size_t strip_scratch_bytes(int r1, int r2) { return 8 * strip_count(r1, r2) + 8; }

int launch_strip_pass(cpsz_b200_ctx* ctx, const StripJob* jobs, const StripJob* d_jobs, int n) {
  const size_t ns = jobs[n - 1].strip0 + strip_count(jobs[n - 1].r1, jobs[n - 1].r2);
  if (ns > 0x7fffffffu) return set_error(CPSZ_ERR_UNSUPPORTED, "field of %zu strips", ns);
  strip_pass_kernel<<<dim3((unsigned)ns, 2), STRIP_NT, 0, ctx->stream>>>(jobs[0], n == 1 ? nullptr : d_jobs, n,
                                                                         ctx->d_flag);
  count_launch(ctx);
  return check_launch("strip_pass_kernel");
}

int launch_strip_unpass(cpsz_b200_ctx* ctx, const uint16_t* const blocks[2], const uint8_t* const ids[2],
                        const float* const unpred[2], const unsigned long long n_unpred[2], int r1, int r2,
                        float2* const pair[2], void* const scratch[2], unsigned* total, int id_shift) {
  const size_t ns = strip_count(r1, r2);
  if (ns > 0x7fffffffu) return set_error(CPSZ_ERR_UNSUPPORTED, "field of %zu strips", ns);
  const int nsc = (r2 + STRIP_W - 1) / STRIP_W;
  StripUnpass P[2];
  for (int f = 0; f < 2; f++)
    P[f] = StripUnpass{blocks[f], ids[f], unpred[f], n_unpred[f], pair[f], (unsigned long long*)scratch[f], total + f,
                       id_shift};
  strip_unpass_kernel<<<dim3((unsigned)ns, 2), STRIP_NT, 0, ctx->stream>>>(P[0], P[1], r1, r2, nsc, (unsigned)ns,
                                                                           ctx->d_flag);
  count_launch(ctx);
  return check_launch("strip_unpass_kernel");
}

}  // namespace cpsz
