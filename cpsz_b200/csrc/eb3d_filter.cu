// eb3d_filter.cu -- the compression path's 3D bound kernel.
//
// A vertex's bound matters only through its id, whose thresholds lie about a
// factor 2 apart (log2(1 + eb) in powers of 2), so the kernel works with an
// enclosure of every tet's bound, evaluated in single precision, and goes to
// the reference's arithmetic (dev::tet_eb) only for tets that have none and
// for vertices whose enclosure holds a threshold.
//
// The bound of a tet (src/sz_compress_cp_preserve_3d.cpp:266-358).  With the
// 24 triple products t = u_i v_j w_k, which the reference forms in float (so
// they are its values exactly), the minor M_f of face f is a signed sum of the
// face's 6 products, M the sum of the four minors, and a minor is flagged when
// M / M_f > 1.  The bound is the max over unflagged f of min(K(p_f, n_f),
// K(p'_f, n'_f)): p_f, n_f the sums of the positive and negated negative
// products of the face, p'_f, n'_f those of the other three faces, and K the
// reference's |c(p) - c(n)| / (c(p) + c(n)), c its cube root.  Write A_f =
// p_f + n_f = sum |t|, B_f the same over the other faces, O_f = M - M_f.  Then
// |p_f - n_f| = |M_f| and |p'_f - n'_f| = |O_f|, and K(p, n) grows with
// |p - n| / (p + n).  So the tet's bound is k(q), k(x) = tanh(atanh(x) / 3), of
//   q = max over unflagged f of min(|M_f| / A_f, |O_f| / B_f),
// the minimum over tets is taken on q, and k is evaluated once per vertex.
//
// Work per cube.  A face (6 products) is the minor of every tet it belongs to,
// up to sign.  The six tets of a cube stand around its diagonal c = (1,1,1),
// d = (0,0,0): tet k is (a_k, a_k+1, c, d) with a_0..a_5 the ring of the other
// six corners.  So a thread takes a cube: the six inner faces (a_k, c, d) serve
// two tets each, and the outer ones (a_k, a_k+1, c) and (a_k, a_k+1, d) are
// evaluated together, one in each word of packed f32x2 operands: 18 faces in 9
// packed evaluations, where six separate tets have 24.
//
// Errors, u = 2^-24.  A face's differences d = t - t' come with their rounding
// errors e (Knuth); M_f = ((d1 + d2) + d3) + ((e1 + e2) + e3) is within 3.1 u D_f
// of its real value, D_f = |d1| + |d2| + |d3|; O_f and M, sums of up to four of
// them, within 5.2 u D, D the sum over the tet's faces.
//  * decisions.  The reference evaluates the minors, M and the quotient in
//    double, within 2^-47 S (S = sum |t|).  With T = 8 u D + 2^-44 S, when
//    every |M_f|, |O_f| and |M| exceeds T, its M and M_f are not zero and its
//    flag f is (sign O_f == sign M_f).  Otherwise, and when all four are
//    flagged (a critical point), the tet is evaluated exactly.
//  * range.  Exact path unless every A_f >= 2^-100 and S <= 2^100 (which also
//    excludes infinities and NaN).  A tet whose products are all 0 has M = 0
//    and so the bound 0.
//  * the enclosure, for bounds up to 0.3 (max_pwr_eb <= 0.25 caps the rest; a
//    product sum that is 0 or subnormal beside one above 2^-101 gives a K of
//    the reference above 0.9, and q above 0.99).  Most bounds are small (the
//    median over a tet of a smooth noisy field is 2e-4, over the 24 tets of a
//    vertex 2e-5), so the absolute part counts.  The reference's cube root is
//    two Newton steps: c(x) = cbrt(x) (1 + e(x)) (1 + r(x)), e the steps' own
//    deviation, which between two arguments changes by at most 5e-5 |ln(x / y)|
//    + 6.3e-9, and r their float roundings, in a range of 2.5e-7; so ln(c(p) /
//    c(n)) is within 2.6e-7 + 5e-5 |ln(p / n)| of ln(p / n) / 3 = 2 atanh(k), and
//    K, whose difference is exact (Sterbenz), within 1.3e-7 + 1.5e-4 k.  The
//    float sums p, n (3.1 u relative each, all their terms positive) add 1.04 u.
//    q: 3.1 u or 5.2 u from M_f or O_f (D_f <= A_f), times dk/dq = (1 - k^2) /
//    (3 (1 - q^2)), at most 1/3 + 1.12 k up to k = 0.3; and 7 u + 9.9e-8 + u
//    relative from the sums, rcp.approx and the product, times q dk/dq <= 1.7 k.
//    k itself: one Newton step of its cubic from an approximation, 6 u relative.
//    Together 2.92e-7 + 1.6e-4 k; EB3_ABS = 3.0e-7, EB3_REL = 2e-4.
// tests/test_gpu_eb3d_filter.py recomputes this sum from the operations' maxima
// measured on the device.
//
// What stays open -- a vertex whose enclosure holds a threshold, or with a tet
// that has none -- goes to a list with the tets that can hold its minimum, and a
// second kernel evaluates those, a thread per vertex: in the marching kernel
// one open vertex would hold up its whole CTA for a thousand instructions.
//
// Bound: instruction issue.  Per tet the full evaluation (kernels3d.cu, one
// thread per tet, minors in double, exact cube roots) issues about 1025
// instructions, and each of the field's tets took it: 384^3, eb 0.05 15.5 ms. Here
// a warp issues about 1300 for a plane of its cubes (6 tets a lane) and vertices,
// 63 % of the issue slots: 4.1 ms, and 0.55 ms for the open vertices.
#include "eb_math.cuh"
#include "kernels.h"
#include "tuning.h"

namespace cpsz {

namespace {

constexpr int TK = 32, TJ = 8;                 // vertices of a CTA's column
constexpr int VK = TK + 2, VJ = TJ + 2;        // with the halo
constexpr int CK = TK + 1, CJ = TJ + 1, NCELL = CK * CJ;
constexpr int NT = 320;                        // a thread per cube (297); the first 256 take the vertices
constexpr float EB3_ABS = 3.0e-7f, EB3_REL = 2.0e-4f;  // |bound - k| <= EB3_ABS + EB3_REL k
constexpr unsigned INF_BITS = 0x7f800000u;

// A tet's entry in the table: the bits of q (ordered as unsigned integers), or
// INF_BITS (no tet), ZERO (the bound is 0) or OPEN (no enclosure); q's bits are
// above these two: q >= T / S > 2^-45.
constexpr unsigned OPEN = 0u, ZERO = 1u;

// Ring corners a_k as (dk, dj, di), and the table index (the reference's tet
// number, src/sz_compress_cp_preserve_3d.cpp:9-46) of the tet (a_k, a_k+1).
__device__ constexpr int RING[6][3] = {{0, 0, 1}, {0, 1, 1}, {0, 1, 0}, {1, 1, 0}, {1, 0, 0}, {1, 0, 1}};
__device__ constexpr int RING_TET[6] = {0, 1, 4, 5, 3, 2};
// The same tets as their first two corners in the reference's order.
__constant__ int8_t c_ab[6][2][3] = {{{0, 0, 1}, {0, 1, 1}}, {{0, 1, 0}, {0, 1, 1}}, {{0, 0, 1}, {1, 0, 1}},
                                     {{1, 0, 0}, {1, 0, 1}}, {{0, 1, 0}, {1, 1, 0}}, {{1, 0, 0}, {1, 1, 0}}};

using dev::f32x2;

struct V3 {
  float u, v, w;
};
struct V3x2 {
  f32x2 u, v, w;
};
__device__ __forceinline__ V3x2 both(const V3& a, const V3& b) {
  return V3x2{dev::pk2(a.u, b.u), dev::pk2(a.v, b.v), dev::pk2(a.w, b.w)};
}
// Per word: the face's minor det(x, y, z), sum |t| and sum |d|.
struct Face2 {
  float m[2], a[2], d[2];
};
__device__ __forceinline__ Face2 face2(const V3x2& x, const V3x2& y, const V3x2& z) {
  using namespace dev;
  const f32x2 t1 = mul2(mul2(x.u, y.v), z.w), t2 = mul2(mul2(x.u, z.v), y.w), t3 = mul2(mul2(y.u, z.v), x.w),
              t4 = mul2(mul2(y.u, x.v), z.w), t5 = mul2(mul2(z.u, x.v), y.w), t6 = mul2(mul2(z.u, y.v), x.w);
  f32x2 d1, d2, d3, e1, e2, e3;
  two_diff2(t1, t2, d1, e1);
  two_diff2(t3, t4, d2, e2);
  two_diff2(t5, t6, d3, e3);
  const f32x2 m = add2(add2(add2(d1, d2), d3), add2(add2(e1, e2), e3));
  Face2 f;
  float p[9][2];
  unpk2(m, f.m[0], f.m[1]);
  unpk2(t1, p[0][0], p[0][1]);
  unpk2(t2, p[1][0], p[1][1]);
  unpk2(t3, p[2][0], p[2][1]);
  unpk2(t4, p[3][0], p[3][1]);
  unpk2(t5, p[4][0], p[4][1]);
  unpk2(t6, p[5][0], p[5][1]);
  unpk2(d1, p[6][0], p[6][1]);
  unpk2(d2, p[7][0], p[7][1]);
  unpk2(d3, p[8][0], p[8][1]);
#pragma unroll
  for (int w = 0; w < 2; w++) {
    f.a[w] = ((fabsf(p[0][w]) + fabsf(p[1][w])) + (fabsf(p[2][w]) + fabsf(p[3][w]))) +
             (fabsf(p[4][w]) + fabsf(p[5][w]));
    f.d[w] = (fabsf(p[6][w]) + fabsf(p[7][w])) + fabsf(p[8][w]);
  }
  return f;
}

// The q of a tet from its minors, sums and difference sums; false: no
// enclosure (s: sum of all |t|).
__device__ __forceinline__ bool tet_q(const float (&M)[4], const float (&A)[4], const float (&D)[4], float& q,
                                      float& s) {
  const float m01 = M[0] + M[1], m23 = M[2] + M[3], m = m01 + m23;
  const float O[4] = {M[1] + m23, M[0] + m23, M[3] + m01, M[2] + m01};
  const float a01 = A[0] + A[1], a23 = A[2] + A[3];
  const float B[4] = {A[1] + a23, A[0] + a23, A[3] + a01, A[2] + a01};
  s = a01 + a23;
  const float T = ((D[0] + D[1]) + (D[2] + D[3])) * 4.76837158e-7f + s * 5.68434189e-14f;  // 8 u, 2^-44
  float least = fabsf(m);
  unsigned open = 0;  // sign bit: some minor is not flagged
  q = 0.f;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    least = fminf(least, fminf(fabsf(M[f]), fabsf(O[f])));
    const unsigned differ = __float_as_uint(M[f]) ^ __float_as_uint(O[f]);
    const float v = fminf(fabsf(M[f]) * dev::rcp_approx(A[f]), fabsf(O[f]) * dev::rcp_approx(B[f]));
    open |= differ;
    q = fmaxf(q, (int)differ < 0 ? v : 0.f);
  }
  const float a_min = fminf(fminf(A[0], A[1]), fminf(A[2], A[3]));
  return least > T && a_min >= 7.88860905e-31f && s <= 1.26765060e30f && (int)open < 0;
}

// k(q) = tanh(atanh(q) / 3) for q >= 0: from q = tanh 3x = (3 k + k^3) / (1 + 3 k^2),
// a Newton step on k^3 - 3 q k^2 + 3 k - q from the approximation (1 - s) / (1 + s),
// s = ((1 - q) / (1 + q))^(1/3), whose own error (2.6e-7, absolute) would widen
// the enclosure of a small k.  Near q = 1, where every k is beyond use, it only
// has to stay above 0.3 (the step's derivative 3 (1 - 2 q k + k^2) is positive
// there as for k < 1 anywhere).
__device__ __forceinline__ float k_of_q(float q) {
  const float r = fmaxf(1.f - q, 0.f) * dev::rcp_approx(1.f + q);
  const float s = dev::ex2_approx(dev::lg2_approx(r) * 0.333333343f);
  const float k = (1.f - s) * dev::rcp_approx(1.f + s);
  if (q > 0.8f) return k;
  return k - ((k * (k - 3.f * q) + 3.f) * k - q) * dev::rcp_approx(3.f * (1.f + k * (k - 2.f * q)));
}
__device__ __forceinline__ float k_low(float k) { return k - (EB3_ABS + EB3_REL * k); }
__device__ __forceinline__ float k_high(float k) { return k + (EB3_ABS + EB3_REL * k); }

// The reference's bound of tet t of the cube with corner `at`.
__device__ __noinline__ float tet_exact(const float* __restrict__ U, const float* __restrict__ V,
                                        const float* __restrict__ W, size_t at, size_t d0, size_t d1, int t) {
  size_t p[4];
#pragma unroll
  for (int x = 0; x < 2; x++) p[x] = at + c_ab[t][x][0] + c_ab[t][x][1] * d1 + c_ab[t][x][2] * d0;
  p[2] = at + 1 + d1 + d0;
  p[3] = at;
  return (float)dev::tet_eb(__ldg(U + p[0]), __ldg(U + p[1]), __ldg(U + p[2]), __ldg(U + p[3]), __ldg(V + p[0]),
                            __ldg(V + p[1]), __ldg(V + p[2]), __ldg(V + p[3]), __ldg(W + p[0]), __ldg(W + p[1]),
                            __ldg(W + p[2]), __ldg(W + p[3]));
}

__device__ __forceinline__ double min_ref(double s, double cur) { return (s < cur) ? s : cur; }

// f(e, oi, oj, ok, t) for the e-th of the 24 tets around a vertex in the
// reference's update order: tet t of the cube at the vertex minus (oi, oj, ok),
// cubes by ascending linear index, tets ascending
// (src/sz_compress_cp_preserve_3d.cpp:390-418).
template <class F>
__device__ __forceinline__ void around(const F& f) {
#pragma unroll
  for (int t = 0; t < 6; t++) f(t, 1, 1, 1, t);
  f(6, 1, 1, 0, 0);
  f(7, 1, 1, 0, 1);
  f(8, 1, 0, 1, 2);
  f(9, 1, 0, 1, 3);
  f(10, 1, 0, 0, 0);
  f(11, 1, 0, 0, 2);
  f(12, 0, 1, 1, 4);
  f(13, 0, 1, 1, 5);
  f(14, 0, 1, 0, 1);
  f(15, 0, 1, 0, 4);
  f(16, 0, 0, 1, 3);
  f(17, 0, 0, 1, 5);
#pragma unroll
  for (int t = 0; t < 6; t++) f(18 + t, 0, 0, 0, t);
}
// The same as a table: offsets packed as oi | oj << 1 | ok << 2 | t << 3.
__constant__ uint8_t c_around[24] = {7 | 0 << 3, 7 | 1 << 3, 7 | 2 << 3, 7 | 3 << 3, 7 | 4 << 3, 7 | 5 << 3,
                                     3 | 0 << 3, 3 | 1 << 3, 5 | 2 << 3, 5 | 3 << 3, 1 | 0 << 3, 1 | 2 << 3,
                                     6 | 4 << 3, 6 | 5 << 3, 2 | 1 << 3, 2 | 4 << 3, 4 | 3 << 3, 4 | 5 << 3,
                                     0 | 0 << 3, 0 | 1 << 3, 0 | 2 << 3, 0 | 3 << 3, 0 | 4 << 3, 0 | 5 << 3};

// id = (int)log2(log2(1 + s) / 2^-23), s > 0; the guess only seeds the count
__device__ __forceinline__ int id_of(const double* thr, int n, double s) {
  const float g = __log2f(__double2float_rn(s) * 1.4426950f) + 23.0f;
  return dev::count_thresholds(thr, n, s, (int)fmaxf(g, 0.f));
}

// A CTA owns a 32 (k) x 8 (j) column of vertices and marches over i, one barrier
// per plane: between two barriers it fetches vertex plane i + 2, evaluates
// cube-plane i from vertex planes i and i + 1, and finishes vertex plane i - 1
// from cube-planes i - 2 and i - 1 (three buffers of each).
// Field dimensions all >= 2, 0 <= max_pwr_eb <= 0.25.
__global__ void __launch_bounds__(NT, 2) eb3d_filter_kernel(const float* __restrict__ U, const float* __restrict__ V,
                                                            const float* __restrict__ W, int r1, int r2, int r3,
                                                            int i_chunk, double max_pwr_eb,
                                                            const double* __restrict__ thr, int thr_n,
                                                            uint8_t* __restrict__ id_q, Eb3dOpen* __restrict__ list,
                                                            unsigned* __restrict__ count, unsigned limit) {
  __shared__ float vtx[3][3][VJ][VK];
  __shared__ unsigned tets[3][6][CJ][CK];
  __shared__ double s_thr[32];
  const int k0 = blockIdx.x * TK, j0 = blockIdx.y * TJ;
  const int i_begin = blockIdx.z * i_chunk, i_end = min(r1, i_begin + i_chunk);
  const size_t d1 = (size_t)r3, d0 = (size_t)r2 * r3;
  const int kl = threadIdx.x & 31, jl = threadIdx.x >> 5;
  const int j = j0 + jl, k = k0 + kl;
  const int cj = threadIdx.x / CK, ck = threadIdx.x - cj * CK;
  const bool has_cube = threadIdx.x < NCELL;
  const bool cube_in = has_cube && j0 - 1 + cj >= 0 && j0 - 1 + cj <= r2 - 2 && k0 - 1 + ck >= 0 && k0 - 1 + ck <= r3 - 2;
  const bool vertex = jl < TJ && j < r2 && k < r3;
  for (int e = threadIdx.x; e < 32; e += NT) s_thr[e] = e < thr_n ? thr[e] : 0.0;
  const int tn = min(thr_n, 32);

  // A vertex plane goes through registers: fetched at the start of a step,
  // stored at its end.
  constexpr int PER = (VJ * VK + NT - 1) / NT;  // 2
  float pre[PER][3];
  auto fetch_plane = [&](int i) {
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int e = threadIdx.x + p * NT, jj = e / VK, kk = e - jj * VK;
      const int gj = j0 - 1 + jj, gk = k0 - 1 + kk;
      pre[p][0] = pre[p][1] = pre[p][2] = 0.f;
      if (e < VJ * VK && gj >= 0 && gj < r2 && gk >= 0 && gk < r3) {
        const size_t at = (size_t)i * d0 + (size_t)gj * d1 + gk;
        pre[p][0] = __ldg(U + at);
        pre[p][1] = __ldg(V + at);
        pre[p][2] = __ldg(W + at);
      }
    }
  };
  auto store_plane = [&](int buf) {
#pragma unroll
    for (int p = 0; p < PER; p++) {
      const int e = threadIdx.x + p * NT;
      if (e < VJ * VK) {
        (&vtx[buf][0][0][0])[e] = pre[p][0];
        (&vtx[buf][1][0][0])[e] = pre[p][1];
        (&vtx[buf][2][0][0])[e] = pre[p][2];
      }
    }
  };
  // cube-plane of the table without any tet
  auto no_cubes = [&](int buf) {
    if (has_cube)
      for (int t = 0; t < 6; t++) tets[buf][t][cj][ck] = INF_BITS;
  };

  const int i_start = max(0, i_begin - 1);  // the first cube-plane
  fetch_plane(i_start);
  store_plane(0);
  fetch_plane(i_start + 1);  // exists: i_start <= r1 - 2
  store_plane(1);
  if (i_begin == 0) no_cubes(2);  // cube-plane -1
  int va = 0;                     // buffer of planes i (vertices and cubes); i - 1 is in va - 1, i + 1 in va + 1
  for (int i = i_start; i <= i_end; i++) {
    // the step's barrier; past the limit the ids are not wanted any more
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile unsigned*)count > limit)) return;
    const int vb = va == 2 ? 0 : va + 1, vc = vb == 2 ? 0 : vb + 1;  // planes i + 1, and i + 2 or i - 1
    const bool more = i + 2 < r1 && i + 1 < i_end;
    if (more) fetch_plane(i + 2);
    if (i < i_end) {
      if (i <= r1 - 2 && cube_in) {
        auto corner = [&](int dk, int dj, int di) -> V3 {
          const int pl = di ? vb : va;
          return V3{vtx[pl][0][cj + dj][ck + dk], vtx[pl][1][cj + dj][ck + dk], vtx[pl][2][cj + dj][ck + dk]};
        };
        const V3 c = corner(1, 1, 1), d = corner(0, 0, 0);
        V3 ring[6];
#pragma unroll
        for (int r = 0; r < 6; r++) ring[r] = corner(RING[r][0], RING[r][1], RING[r][2]);
        float in_m[6], in_a[6], in_d[6];  // inner faces (a_k, c, d)
        {
          const V3x2 cc = both(c, c), dd = both(d, d);
#pragma unroll
          for (int r = 0; r < 6; r += 2) {
            const Face2 f = face2(both(ring[r], ring[r + 1]), cc, dd);
#pragma unroll
            for (int w = 0; w < 2; w++) {
              in_m[r + w] = f.m[w];
              in_a[r + w] = f.a[w];
              in_d[r + w] = f.d[w];
            }
          }
        }
        const V3x2 cd = both(c, d);
#pragma unroll
        for (int r = 0; r < 6; r++) {
          const int n = (r + 1) % 6, t = RING_TET[r];
          const Face2 o = face2(both(ring[r], ring[r]), both(ring[n], ring[n]), cd);
          // the tet's minors (a common sign aside)
          const float M[4] = {-in_m[n], in_m[r], -o.m[1], o.m[0]};
          const float A[4] = {in_a[n], in_a[r], o.a[1], o.a[0]};
          const float D[4] = {in_d[n], in_d[r], o.d[1], o.d[0]};
          float q, s;
          const bool ok = tet_q(M, A, D, q, s);
          tets[va][t][cj][ck] = ok ? __float_as_uint(q) : s == 0.f ? ZERO : OPEN;  // s 0: every product is 0
        }
      } else {
        no_cubes(va);  // beyond the field (or this thread's cube is)
      }
    }
    if (i > i_begin) {
      // vertex plane i - 1: cube-planes i - 2 (buffer vb) and i - 1 (buffer vc)
      const size_t idx = (size_t)(i - 1) * d0 + (size_t)j * d1 + k;
      auto entry = [&](int oi, int oj, int ok, int t) { return tets[oi ? vb : vc][t][jl + 1 - oj][kl + 1 - ok]; };
      bool open = false;
      float hi_k = 0.f;  // no enclosed bound above this is the least
      if (vertex) {
        unsigned least = 0xffffffffu;
        around([&](int, int oi, int oj, int ok, int t) { least = umin(least, entry(oi, oj, ok, t)); });
        int id = ID_ZERO;
        if (least > ZERO) {
          double lo = max_pwr_eb, hi = max_pwr_eb;
          if (least < INF_BITS) {
            const float kq = k_of_q(__uint_as_float(least));
            hi_k = k_high(kq);
            lo = fmin(lo, (double)k_low(kq));
            hi = fmin(hi, (double)hi_k);
          }
          if (lo > 0) {
            id = id_of(s_thr, tn, hi);
            open = id > 0 && lo < s_thr[id];
          } else {
            open = hi > 0;  // (hi is 0 if max_pwr_eb is)
          }
        } else if (least == OPEN) {
          open = true;
          unsigned rest = 0xffffffffu;
          around([&](int, int oi, int oj, int ok, int t) {
            const unsigned x = entry(oi, oj, ok, t);
            if (x != OPEN) rest = umin(rest, x);
          });
          if (rest > ZERO && rest < INF_BITS) hi_k = k_high(k_of_q(__uint_as_float(rest)));
        }
        id_q[idx] = (uint8_t)id;
      }
      const unsigned who = __ballot_sync(0xffffffffu, open);
      if (open) {
        // the enclosed tets that can hold the minimum: k_low(k(q)) <= hi_k, that
        // is q <= tanh(3 atanh(k)) where k_low(k) = hi_k (rounded up)
        const float kl_ = (hi_k + EB3_ABS) * (1.f + 1.01f * EB3_REL);
        const float ql = kl_ * (3.f + kl_ * kl_) / (1.f + 3.f * kl_ * kl_) * 1.00001f;
        const unsigned q_last = hi_k > 0.3f ? INF_BITS - 1u : __float_as_uint(ql);
        unsigned which = 0;
        around([&](int e, int oi, int oj, int ok, int t) {
          const unsigned x = entry(oi, oj, ok, t);
          if (x == OPEN || (x > ZERO && x <= q_last)) which |= 1u << e;
          if (x == ZERO) which |= 1u << 31;  // a bound of 0 among the rest
        });
        if (hi_k == 0.f) {  // no enclosed tet, or one whose bound is 0: only those without enclosure matter
          unsigned only = which & (1u << 31);
          around([&](int e, int oi, int oj, int ok, int t) {
            if (entry(oi, oj, ok, t) == OPEN) only |= 1u << e;
          });
          which = only;
        }
        const int first = __ffs(who) - 1;
        unsigned base = 0;
        if (kl == first) base = atomicAdd(count, (unsigned)__popc(who));
        base = __shfl_sync(who, base, first) + __popc(who & ((1u << kl) - 1u));
        if (base < limit) list[base] = Eb3dOpen{(unsigned)idx, (unsigned)(idx >> 32), which, 0};
      }
    }
    if (more) store_plane(vc);
    va = vb;
  }
}

// The open vertices: the reference's minimum over the listed tets (every other
// tet's bound is larger).  A warp takes 32 vertices and shares their tets out
// among its lanes.  A bound that is not a number makes the order of all 24
// matter, so that vertex runs the reference's sequence whole.
constexpr int OPEN_WARPS = 4;
__global__ void __launch_bounds__(32 * OPEN_WARPS) eb3d_open_kernel(
    const float* __restrict__ U, const float* __restrict__ V, const float* __restrict__ W, int r1, int r2, int r3,
    double max_pwr_eb, const double* __restrict__ thr, int thr_n, uint8_t* __restrict__ id_q,
    const Eb3dOpen* __restrict__ list, const unsigned* __restrict__ count, unsigned limit, int* __restrict__ flag) {
  __shared__ uint16_t s_item[OPEN_WARPS][32 * 24];  // lane | tet around it << 5
  __shared__ unsigned s_min[OPEN_WARPS][32];
  __shared__ unsigned s_nan[OPEN_WARPS];
  const unsigned n = *count;
  if (n > limit) return;
  const size_t d1 = (size_t)r3, d0 = (size_t)r2 * r3;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int my_flag = 0;
  for (unsigned q0 = (blockIdx.x * OPEN_WARPS + warp) * 32; q0 < n; q0 += gridDim.x * OPEN_WARPS * 32) {
    const Eb3dOpen o = q0 + lane < n ? list[q0 + lane] : Eb3dOpen{0, 0, 0, 0};
    const size_t idx = (size_t)o.at_hi << 32 | o.at_lo;
    const unsigned mine = o.tets & 0xffffffu;
    unsigned x = __popc(mine);
    const unsigned own = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    const unsigned total = __shfl_sync(0xffffffffu, x, 31);
    unsigned at = x - own;
    for (unsigned m = mine; m; m &= m - 1) s_item[warp][at++] = (uint16_t)(lane | (__ffs(m) - 1) << 5);
    s_min[warp][lane] = 0x7f800000u;
    if (lane == 0) s_nan[warp] = 0;
    __syncwarp();
    for (unsigned e0 = 0; e0 < total; e0 += 32) {
      const bool on = e0 + lane < total;
      const unsigned it = on ? s_item[warp][e0 + lane] : 0u;
      const int who = (int)(it & 31u);
      const size_t v_at = (size_t)__shfl_sync(0xffffffffu, o.at_hi, who) << 32 | __shfl_sync(0xffffffffu, o.at_lo, who);
      if (on) {
        const unsigned a = c_around[it >> 5];
        const float v = tet_exact(U, V, W, v_at - (a & 1) * d0 - (a >> 1 & 1) * d1 - (a >> 2 & 1), d0, d1, (int)(a >> 3));
        if (v == v) atomicMin(&s_min[warp][who], __float_as_uint(v));
        else atomicOr(&s_nan[warp], 1u << who);
      }
    }
    __syncwarp();
    if (q0 + lane < n) {
      double s = fmin(max_pwr_eb, (double)__uint_as_float(s_min[warp][lane]));
      if (o.tets >> 31) s = fmin(s, 0.0);
      if (s_nan[warp] >> lane & 1u) {
        const int i = (int)(idx / d0), j = (int)((idx - i * d0) / d1), k = (int)(idx - i * d0 - j * d1);
        s = max_pwr_eb;
        for (int e = 0; e < 24; e++) {
          const unsigned a = c_around[e];
          const int ci = i - (int)(a & 1), cj = j - (int)(a >> 1 & 1), ck = k - (int)(a >> 2 & 1);
          if (ci < 0 || ci > r1 - 2 || cj < 0 || cj > r2 - 2 || ck < 0 || ck > r3 - 2) continue;
          s = min_ref(s, (double)tet_exact(U, V, W, (size_t)ci * d0 + (size_t)cj * d1 + ck, d0, d1, (int)(a >> 3)));
        }
      }
      const int id = s > 0 ? id_of(thr, thr_n, s) : (int)ID_ZERO;
      if (id != ID_ZERO && id >= ID_RAW_3D) my_flag |= FLAG_ID_OVERFLOW;
      id_q[idx] = (uint8_t)id;
    }
    __syncwarp();
  }
  if (my_flag) atomicOr(flag, my_flag);
}

}  // namespace

bool eb3d_filter_takes(int r1, int r2, int r3, double max_pwr_eb) {
  return r1 >= 2 && r2 >= 2 && r3 >= 2 && max_pwr_eb >= 0 && max_pwr_eb <= 0.25;
}

int launch_eb3d_filter(cpsz_b200_ctx* ctx, const float* U, const float* V, const float* W, int r1, int r2, int r3,
                       double max_pwr_eb, const double* d_thr, int thr_n, uint8_t* id_q, int chunk, Eb3dOpen* list,
                       unsigned* count, unsigned limit) {
  const dim3 grid((r3 + TK - 1) / TK, (r2 + TJ - 1) / TJ, (r1 + chunk - 1) / chunk);
  eb3d_filter_kernel<<<grid, NT, 0, ctx->stream>>>(U, V, W, r1, r2, r3, chunk, max_pwr_eb, d_thr, thr_n, id_q, list,
                                                   count, limit);
  eb3d_open_kernel<<<ctx->num_sms * 8, 32 * OPEN_WARPS, 0, ctx->stream>>>(U, V, W, r1, r2, r3, max_pwr_eb, d_thr, thr_n, id_q,
                                                              list, count, limit, ctx->d_flag);
  count_launch(ctx, 2);
  return check_launch("eb3d_filter_kernel");
}

}  // namespace cpsz
