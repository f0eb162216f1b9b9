// wave3d.cu -- the 3D Lorenzo recursion of the offline (log) path on
// reconstructed log values (src/sz_compress_cp_preserve_3d.cpp:441-520,
// src/sz_decompress_cp_preserve_3d.cpp:52-104).
//
// A point's predictor reads its seven lower neighbours (i-1 / j-1 / k-1
// combinations).  One persistent kernel runs the whole recursion:
//  * a unit is W3_P planes i0 .. i0+P-1 of 32 rows j0 .. j0+31, run by one
//    CTA: compute warp p owns plane i0 + p, lane l row j0 + l, and at step t
//    the thread handles column k = t - l - p (lanes skewed by one column,
//    planes by one step), so all seven neighbours were produced at steps
//    t-1 .. t-3; one barrier of the compute warps per step;
//  * each plane keeps its last results in a ring in shared memory, two windows
//    of W3_W steps: slot t, entry l+1 = lane l's value of step t, entry 0 = row
//    j0-1 at column t+1-p (as if from a lane -1).  A point reads (i,j-1,k) from
//    its own plane's ring and (i-1,j,k), (i-1,j-1,k) from plane p-1's; the
//    other four are its own result and these three of the step before, kept
//    in registers.  Plane i0-1 is a ring loaded from the unit of the planes
//    below.  Lane 0 needs no special case;
//  * everything that touches global memory is done by W3_HELPERS warps, a
//    window of steps at a time: a row's W3_W points of a window are
//    consecutive in memory, so a warp's access covers four rows of 128 bytes
//    (a thread that fetched or stored its own point would touch 32 lines per
//    access).  During window w they store window w-1's results and codes,
//    publish the unit's progress, and load window w+1's input and boundary
//    values; the compute warps meet them at one barrier per window;
//    A compute warp reads after the step's barrier only what needs it, plane
//    p-1's value of the step before; the rest it reads ahead of it;
//  * units are dequeued in ticket order u = (i0 / P) * slabs + s from an
//    atomic counter, so a unit's producers (the planes below, the rows
//    below) hold smaller tickets, taken by CTAs that are already running:
//    every wait ends;
//  * the values of step t's slot need the unit of the planes below at
//    >= t + P + 1 steps and the unit of the rows below at >= t + 33; the
//    latter covers the unit below and behind, which that unit waited for;
//  * loads go through L2 (cp.async.cg: another SM's writes must not meet a
//    stale L1 line).
//
// What bounds it: the helpers' accesses (32 KB in, 48 KB out per window) and the
// compute warps' on one shared-memory pipe, then the step's chain and barrier.
// A unit by itself took .39 us a step, .19 with idle helpers, .14 without the
// barrier, while a 16-byte copy of four rows scattered its lines over eight
// slots (24 shared-memory wavefronts; 384^3 1.50 ms, 1.27 with a row's points
// together).  With a thread fetching its own input and storing its own result,
// eight ring reads a step and progress published behind two fences a step was
// .55-.9 us: 384^3 2.9 ms, and decoding 256^3 3.2 (most of it logarithms of
// raw points inside the recursion: prep3d takes them now), .5 here.  One, two
// or four input warps and two, four or eight storing ones are within 10 %.
// Every wait is bounded: on expiry (or once any wait has expired) the kernel
// sets FLAG_TIMEOUT and stops waiting; the host then fails the call.
//
// Step arithmetic (all float; equal to the reference's float/double mix, see
// the wavefront notes in wave2d.cu): with p = 2^(id-23) and y = |x - pred| / p
// exact, the reference's capacity test is y < 65535, the code is
// 32768 +- ((int)y + 1) >> 1 = 32768 +- floor(y/2 + 1/2), and
// (float)(pred + 2 q p) equals the float sum pred + (2q) p (no product
// overflows: logs are below 2^8).  The decoder's
// (float)(pred + 2 (code - 32768) p) is likewise pred + addend with the addend
// precomputed exactly in float; a raw point's logs are taken before the
// recursion (prep3d), exp2f and signs applied after it.
#include "kernels.h"
#include "libm_dev.cuh"

namespace cpsz {

namespace {

constexpr int W3_P = 8;         // planes per unit = compute warps per CTA
constexpr int W3_W = 8;         // steps per window
constexpr int W3_IN = 2, W3_OUT = 4;            // helper warps that load input, that store results
constexpr int W3_HELPERS = 1 + W3_IN + W3_OUT;  // and one for the boundary
constexpr int W3_COMPUTE = 32 * W3_P;
constexpr int W3_THREADS = W3_COMPUTE + 32 * W3_HELPERS;
constexpr int W3_SR = 2 * W3_W;  // slots of a computed ring, and of the input
constexpr int W3_SL = 4 * W3_W;  // slots of loaded values: the next window's arrive while the last one's are read
constexpr long long W3_WAIT_NS = 4000000000ll;

struct W3Args {
  const float4* in;  // compress: (log u, log v, log w, 1/p); decompress: addends, or a raw point's logs (w != 0)
  float4* rec;       // reconstructed log values
  ushort4* codes;    // compress: codes (0,0,0 for unpredictable points)
  int r1, r2, r3, slabs;
  int* sync;  // [0] the work queue, [1 + u] unit u's published progress
  int* flag;
};

// Rows of 33 points: a warp's 16-byte accesses to four rows of eight slots, and
// to one slot's 32 lanes, meet no bank twice.
template <bool DECOMP>
struct W3Smem {
  // Input row by row: a row's eight points of a window are 128 bytes, the point
  // of step m of row l in piece m ^ (l & 7), so that a copied line lands in one
  // place and a step's 32 lanes still read all banks.
  float4 in[W3_P][2][32][W3_W];
  float4 ring[W3_P][W3_SR][33];  // plane i0+p
  float4 below[W3_SL][33];       // plane i0-1
  float4 edge[W3_P][W3_SL];      // row j0-1 of plane i0+p: entry 0 of ring[p]'s slots to come
  ushort4 codes[DECOMP ? 1 : W3_P][W3_SR][33];
  int unit;
};

__device__ __forceinline__ long long globaltimer_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int ld_acquire_s32(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_s32(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// 16-byte cp.async through L2; zero-fills the slot when !valid (src unread)
__device__ __forceinline__ void cp16(void* smem, const void* g, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(g), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(W3_COMPUTE) : "memory"); }
__device__ __forceinline__ void store_sync() { asm volatile("bar.sync 2, %0;" ::"n"(32 * W3_OUT) : "memory"); }

__device__ __forceinline__ float comp(const float4& v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }

// A unit: its planes, rows and steps.
struct W3Unit {
  int u, s, i0, np, j0, nrows, t_end;
};

// ---- helper warps ----
// A warp covers rows l0 + 0, 4, .. 28 of slots T + m: eight accesses of four
// rows.  Where every row of a plane has its column in the field, an access is
// an address step and the access.
__device__ __forceinline__ bool w3_inner(const W3Unit& U, int r3, int T, int p) {
  return p < U.np && U.nrows == 32 && T - 31 - p >= 0 && T + W3_W - 1 - p < r3;
}

template <bool DECOMP>
__device__ __forceinline__ void w3_load_input(const W3Args& a, W3Smem<DECOMP>& M, const W3Unit& U, int T, int p0,
                                              int lane) {
  const int r3 = a.r3, l0 = lane >> 3, m = lane & 7, t = T + m;
  for (int p = p0; p < W3_P; p += W3_IN) {
    const float4* src = a.in + ((long long)(U.i0 + p) * a.r2 + U.j0 + l0) * r3 + (t - l0 - p);
    float4 (*const dst)[W3_W] = M.in[p][(T / W3_W) & 1];
    if (w3_inner(U, r3, T, p)) {
#pragma unroll
      for (int r = 0; r < 8; r++, src += 4 * (r3 - 1))
        cp16(&dst[4 * r + l0][m ^ ((4 * r + l0) & 7)], src, true);
    } else {
#pragma unroll
      for (int r = 0; r < 8; r++, src += 4 * (r3 - 1)) {
        const int l = 4 * r + l0, k = t - l - p;
        const bool act = p < U.np && l < U.nrows && k >= 0 && k < r3;
        cp16(&dst[l][m ^ (l & 7)], act ? src : a.in, act);
      }
    }
  }
}

template <bool DECOMP>
__device__ __forceinline__ void w3_load_boundary(const W3Args& a, W3Smem<DECOMP>& M, const W3Unit& U, int T,
                                                 int lane) {
  const int r3 = a.r3, l0 = lane >> 3, t = T + (lane & 7), slot = t & (W3_SL - 1);
  const long long d0 = (long long)a.r2 * r3;
  // plane i0-1: entry l+1 = row j0+l at column t-l+1, entry 0 = row j0-1 at column t+2
  const long long base = (long long)(U.i0 - 1) * d0 + (long long)U.j0 * r3;
  if (U.i0 > 0) {
    const float4* src = a.rec + base + (long long)l0 * r3 + (t - l0 + 1);
    float4* dst = &M.below[slot][l0 + 1];
    if (w3_inner(U, r3, T, -1)) {
#pragma unroll
      for (int r = 0; r < 8; r++, src += 4 * (r3 - 1)) cp16(dst + 4 * r, src, true);
    } else {
#pragma unroll
      for (int r = 0; r < 8; r++, src += 4 * (r3 - 1)) {
        const int l = 4 * r + l0, k = t - l + 1;
        const bool act = l < U.nrows && k >= 0 && k < r3;
        cp16(dst + 4 * r, act ? src : a.rec, act);
      }
    }
  } else {
    for (int r = 0; r < 8; r++) M.below[slot][4 * r + l0 + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (l0 == 0) {
    const int k = t + 2;
    const bool act = U.i0 > 0 && U.s > 0 && k >= 0 && k < r3;
    cp16(&M.below[slot][0], act ? a.rec + base - r3 + k : a.rec, act);
  }
  // row j0-1 of planes i0+p at column t+1-p
#pragma unroll
  for (int p = l0; p < W3_P; p += 4) {
    const int k = t + 1 - p;
    const bool act = U.s > 0 && p < U.np && k >= 0 && k < r3;
    cp16(&M.edge[p][slot], act ? a.rec + base + (long long)(p + 1) * d0 - r3 + k : a.rec, act);
  }
}

// Waits until the producers have reached what the loads of the window at T
// read (its last slot is t = T + W3_W - 1): lane 0 for the unit of the planes
// below, lane 1 for the unit of the rows below.  Plane i0-1's row j0+l at
// column t-l+1 is the planes-below unit's step t+P; row j0-1 of plane i0+p at
// column t+1-p is the rows-below unit's step t+32.  Targets are capped at the
// producers' step counts (the planes-below unit has P planes and these rows,
// the rows-below unit 32 rows and these planes): a step beyond them loads only
// zero fill.  `have`: the lane's last value.
__device__ __forceinline__ void w3_wait(const W3Args& a, const W3Unit& U, int T, int lane, int& have, bool& aborted) {
  const int t = T + W3_W - 1;
  const int need = lane == 0 && U.i0 > 0 ? min(t + W3_P + 1, a.r3 + U.nrows - 1 + W3_P - 1)
                   : lane == 1 && U.s > 0 ? min(t + 33, a.r3 + 31 + U.np - 1)
                                          : 0;
  const int* p = a.sync + 1 + U.u - (lane == 0 ? a.slabs : 1);
  long long t0 = 0;
  if (have < need && !aborted) {
    have = ld_acquire_s32(p);
    while (have < need) {
      const long long now = globaltimer_ns();
      if (!t0) t0 = now;
      if ((*(volatile int*)a.flag & FLAG_TIMEOUT) || now - t0 > W3_WAIT_NS) {
        atomicOr(a.flag, FLAG_TIMEOUT);
        aborted = true;
        break;
      }
      __nanosleep(20);
      have = ld_acquire_s32(p);
    }
  }
  __syncwarp();
}

template <bool DECOMP>
__device__ __forceinline__ void w3_store(const W3Args& a, const W3Smem<DECOMP>& M, const W3Unit& U, int T, int p0,
                                         int lane) {
  const int r3 = a.r3, l0 = lane >> 3, t = T + (lane & 7), slot = t & (W3_SR - 1);
  for (int p = p0; p < U.np; p += W3_OUT) {
    const long long at = ((long long)(U.i0 + p) * a.r2 + U.j0 + l0) * r3 + (t - l0 - p);
    float4* rec = a.rec + at;
    ushort4* codes = DECOMP ? nullptr : a.codes + at;
    float4 v[8];  // read before the first store: one shared-memory latency
    ushort4 c[8];
#pragma unroll
    for (int r = 0; r < 8; r++) {
      v[r] = M.ring[p][slot][4 * r + l0 + 1];
      if (!DECOMP) c[r] = M.codes[p][slot][4 * r + l0];
    }
    const bool inner = w3_inner(U, r3, T, p);
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int l = 4 * r + l0, k = t - l - p;
      if (inner || (l < U.nrows && k >= 0 && k < r3)) {
        *rec = v[r];
        if (!DECOMP) *codes = c[r];
      }
      rec += 4 * (r3 - 1);
      if (!DECOMP) codes += 4 * (r3 - 1);
    }
  }
}

template <bool DECOMP>
__device__ __forceinline__ void w3_help(const W3Args& a, W3Smem<DECOMP>& M, const W3Unit& U, int helper, int lane,
                                        bool& aborted) {
  const int nwin = (U.t_end + W3_W - 1) / W3_W;
  if (helper == 0) {  // the boundary
    int have = 0;
    w3_wait(a, U, 0, lane, have, aborted);
    w3_load_boundary(a, M, U, -W3_W, lane);
    w3_load_boundary(a, M, U, 0, lane);
    // Slot -1's entry 0 is there when the barrier opens window 0: plane p + 1
    // reads it in step 0, before the first barrier among the compute warps.
    // It is row j0-1 at column -p, which exists for p = 0 alone.
    if (lane < W3_P) {
      const bool act = U.s > 0 && lane == 0;
      cp16(&M.ring[lane][W3_SR - 1][0], act ? a.rec + ((long long)U.i0 * a.r2 + U.j0 - 1) * a.r3 : a.rec, act);
    }
    cp_wait_all();
    __syncthreads();  // window 0 starts
    for (int w = 0; w < nwin; w++) {
      if (w + 1 < nwin) {
        w3_wait(a, U, (w + 1) * W3_W, lane, have, aborted);
        w3_load_boundary(a, M, U, (w + 1) * W3_W, lane);
        cp_wait_all();
      }
      __syncthreads();  // window w is computed, window w+1 starts
    }
  } else if (helper <= W3_IN) {  // the input
    w3_load_input(a, M, U, 0, helper - 1, lane);
    cp_wait_all();
    __syncthreads();
    for (int w = 0; w < nwin; w++) {
      if (w + 1 < nwin) {
        w3_load_input(a, M, U, (w + 1) * W3_W, helper - 1, lane);
        cp_wait_all();
      }
      __syncthreads();
    }
  } else {  // the results
    auto publish = [&](int steps) {
      store_sync();  // all stores; the release makes them visible with the count
      if (helper == 1 + W3_IN && lane == 0) st_release_s32(a.sync + 1 + U.u, steps);
    };
    __syncthreads();
    for (int w = 0; w < nwin; w++) {
      if (w > 0) {
        w3_store(a, M, U, (w - 1) * W3_W, helper - 1 - W3_IN, lane);
        publish(w * W3_W);
      }
      __syncthreads();
    }
    w3_store(a, M, U, (nwin - 1) * W3_W, helper - 1 - W3_IN, lane);
    publish(U.t_end);
  }
}

// ---- compute warps ----
template <bool DECOMP>
__device__ __forceinline__ void w3_compute(const W3Args& a, W3Smem<DECOMP>& M, const W3Unit& U, int p, int lane) {
  const int r3 = a.r3;
  const float4 Z = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool mine = p < U.np && lane < U.nrows;
  // q0 = (i-1,j-1,k-1), q1 = (i-1,j-1,k), q2 = (i-1,j,k-1), q3 = (i-1,j,k),
  // q4 = (i,j-1,k-1), q5 = (i,j-1,k), q6 = (i,j,k-1)
  float4 q0 = Z, q1, q2 = Z, q4 = Z, q5, q6 = Z;
  for (int sl = W3_SR - 2; sl < W3_SR; sl++) M.ring[p][sl][lane + 1] = Z;  // steps -2 and -1
  if (lane == 0) M.ring[p][W3_SR - 2][0] = Z;  // (step -1's comes with the boundary)
  const int nwin = (U.t_end + W3_W - 1) / W3_W;
  for (int w = 0; w < nwin; w++) {
    __syncthreads();  // window w's values are loaded, window w-1 is computed
    const int cur = W3_W * (w & 1), prev = W3_W - cur;
    if (lane < W3_W) M.ring[p][cur + lane][0] = M.edge[p][(W3_W * w + lane) & (W3_SL - 1)];
    __syncwarp();
    float4 (*const R)[33] = &M.ring[p][cur];
    const float4 (*const Rp)[33] = &M.ring[p][prev];
    const float4 (*const B)[33] = p > 0 ? &M.ring[p - 1][cur] : &M.below[W3_W * (w & 3)];
    const float4 (*const Bp)[33] = p > 0 ? &M.ring[p - 1][prev] : &M.below[W3_W * ((w - 1) & 3)];
    const float4* const X = M.in[p][w & 1][lane];
    if (w == 0) {
      q1 = Bp[W3_W - 2][lane];
      q5 = Rp[W3_W - 1][lane];
    }
    float4 x = X[lane & 7];
#pragma unroll
    for (int j = 0; j < W3_W; j++) {
      if (j > 0) compute_sync();  // every plane has finished the step before
      // the one value that needs the barrier; the others were read before it
      const float4* const Bj = j > 0 ? B[j > 0 ? j - 1 : 0] : Bp[W3_W - 1];
      const float4 q3 = Bj[lane + 1];
      const int k = W3_W * w + j - lane - p;
      const bool act = mine && k >= 0 && k < r3;
      // pred = q0 + q3 + q5 + q6 - q1 - q2 - q4, left to right
      float pred[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        float v = comp(q0, c) + comp(q3, c);
        v = v + comp(q5, c);
        v = v + comp(q6, c);
        v = v - comp(q1, c);
        v = v - comp(q2, c);
        v = v - comp(q4, c);
        pred[c] = v;
      }
      float4 res;
      if (!DECOMP) {
        const float inv = x.w;  // NaN: precision 0 (unpredictable)
        const float pw = __int_as_float(0x7F000000 - __float_as_int(inv));
        bool ok = true;
        float dec[3], cf[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const float xc = comp(x, c);
          const float diff = xc - pred[c];
          const unsigned neg = __float_as_uint(diff) & 0x80000000u;
          const float h = __fmaf_rd(fabsf(diff), 0.5f * inv, 0.5f);  // y/2 + 1/2
          const float qf = __fadd_rd(h, 8388608.0f) - 8388608.0f;
          dec[c] = __fmaf_rn(qf, __uint_as_float(__float_as_uint(pw + pw) | neg), pred[c] + 0.f);
          cf[c] = __fmaf_rn(qf, __uint_as_float(0x3F800000u | neg), 8388608.0f + 32768.0f);  // code in its low 16 bits
          ok = ok & (h < 32768.0f) & (fabsf(dec[c] - xc) < pw);
        }
        res = ok ? make_float4(dec[0], dec[1], dec[2], 0.f) : make_float4(x.x, x.y, x.z, 0.f);
        M.codes[p][cur + j][lane] =
            ok ? make_ushort4((unsigned short)__float_as_uint(cf[0]), (unsigned short)__float_as_uint(cf[1]),
                              (unsigned short)__float_as_uint(cf[2]), 0)
               : make_ushort4(0, 0, 0, 0);
      } else if (__float_as_int(x.w) != 0) {
        res = make_float4(x.x, x.y, x.z, 0.f);  // raw point: its logs
      } else {
        res = make_float4(pred[0] + x.x, pred[1] + x.y, pred[2] + x.z, 0.f);
      }
      if (!act) res = Z;
      R[j][lane + 1] = res;
      q0 = q1;
      q2 = q3;
      q4 = q5;
      q6 = res;
      __syncwarp();
      q5 = R[j][lane];  // the next step's, of the row above
      q1 = Bj[lane];
      if (j + 1 < W3_W) x = X[(j + 1) ^ (lane & 7)];
    }
  }
  __syncthreads();  // the last window is computed
}

template <bool DECOMP>
__global__ void __launch_bounds__(W3_THREADS, 1) wave3d_kernel(const W3Args a) {
  extern __shared__ __align__(128) unsigned char w3_smem[];
  W3Smem<DECOMP>& M = *reinterpret_cast<W3Smem<DECOMP>*>(w3_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int units = ((a.r1 + W3_P - 1) / W3_P) * a.slabs;
  bool aborted = false;  // the boundary warp's lanes: a wait has expired; no more waiting
  for (;;) {
    __syncthreads();  // the previous unit's results are stored
    if (threadIdx.x == 0) {
      const bool again = DECOMP && decode_again(a.flag);
      const int next = atomicAdd(a.sync, 1);
      M.unit = again ? units : next;
    }
    __syncthreads();
    W3Unit U;
    U.u = M.unit;
    if (U.u >= units) break;
    const int g = U.u / a.slabs;
    U.s = U.u - g * a.slabs;
    U.i0 = g * W3_P;
    U.np = min(W3_P, a.r1 - U.i0);
    U.j0 = 32 * U.s;
    U.nrows = min(32, a.r2 - U.j0);
    U.t_end = a.r3 + U.nrows - 1 + U.np - 1;
    if (warp < W3_P) w3_compute<DECOMP>(a, M, U, warp, lane);
    else w3_help<DECOMP>(a, M, U, warp - W3_P, lane, aborted);
  }
}

// Decoded values from the reconstructed logs: 0 below log -99, else
// +-exp2f(log) (the host library's) with the stored sign.  Raw points have
// their values already (prep3d).
__global__ void __launch_bounds__(256) exp3d_kernel(const float4* __restrict__ in, const float4* __restrict__ rec,
                                                    const uint8_t* __restrict__ signs, size_t sign_bytes, LibmFn Ex,
                                                    float* __restrict__ U, float* __restrict__ V,
                                                    float* __restrict__ W, size_t n, const int* __restrict__ flag) {
  if (decode_again(flag)) return;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += stride) {
    if (__float_as_int(in[idx].w) != 0) continue;
    float out[3];
    const float4 l = rec[idx];
    const unsigned byte = (unsigned)(idx >> 3), bit = 7u - (unsigned)(idx & 7);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float lg = comp(l, c);
      const bool pos = (__ldg(signs + (size_t)c * sign_bytes + byte) >> bit) & 1u;
      if (lg < -99.f) {
        out[c] = 0.f;
      } else {
        const float e = dev::host_exp2f(lg, Ex);
        out[c] = pos ? e : -e;
      }
    }
    U[idx] = out[0];
    V[idx] = out[1];
    W[idx] = out[2];
  }
}

}  // namespace

size_t wave3d_scratch_bytes(int r1, int r2) {
  return ((size_t)((r1 + W3_P - 1) / W3_P) * ((r2 + 31) / 32) + 1) * sizeof(int);
}

int launch_wave3d(cpsz_b200_ctx* ctx, bool decompress, const float4* in, float4* rec, ushort4* codes,
                  const uint8_t* signs, size_t sign_bytes, const LibmTables* L, float* U, float* V, float* W, int r1,
                  int r2, int r3, void* scratch) {
  W3Args a{};
  a.in = in;
  a.rec = rec;
  a.codes = codes;
  a.r1 = r1;
  a.r2 = r2;
  a.r3 = r3;
  a.slabs = (r2 + 31) / 32;
  a.sync = (int*)scratch;
  a.flag = ctx->d_flag;
  CPSZ_CUDA_TRY(cudaMemsetAsync(scratch, 0, wave3d_scratch_bytes(r1, r2), ctx->stream));
  const long long units = (long long)((r1 + W3_P - 1) / W3_P) * a.slabs;
  auto kern = decompress ? wave3d_kernel<true> : wave3d_kernel<false>;
  const size_t smem = decompress ? sizeof(W3Smem<true>) : sizeof(W3Smem<false>);
  CPSZ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long ctas = units < ctx->num_sms ? units : ctx->num_sms;  // one fills an SM's shared memory
  kern<<<(int)ctas, W3_THREADS, smem, ctx->stream>>>(a);
  count_launch(ctx);
  CPSZ_TRY(check_launch("wave3d_kernel"));
  if (!decompress) return CPSZ_OK;
  const size_t n = (size_t)r1 * r2 * r3;
  const size_t blocks = (n + 255) / 256, cap = (size_t)ctx->num_sms * 8;
  exp3d_kernel<<<(int)(blocks < cap ? blocks : cap), 256, 0, ctx->stream>>>(in, rec, signs, sign_bytes, L->exp2f, U,
                                                                            V, W, n, ctx->d_flag);
  count_launch(ctx);
  return check_launch("exp3d_kernel");
}

}  // namespace cpsz
