// Device helpers shared by the quartet kernels: compile-time angular-momentum
// tables, Rys roots/weights from the polynomial tables, the per-axis Rys
// vertical recurrence, and small warp utilities.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>
#include <utility>

#include "igpu_internal.hpp"

namespace igpu {

// ------------------------------------------------------------ compile time

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int tri_below(int d) { return d * (d + 1) * (d + 2) / 6; }
__host__ __device__ constexpr int n_addr(int l) { return (l + 1) * (l + 2) * (l + 3) / 6; }
// Number of Cartesian triples with degree in [lo, hi].
__host__ __device__ constexpr int nrange(int lo, int hi) { return tri_below(hi + 1) - tri_below(lo); }

// Component i (canonical order: lx descending, then ly descending) of degree l.
__host__ __device__ constexpr int comp_lx(int l, int i) {
  int lx = l, rem = i;
  while (rem >= l - lx + 1) {
    rem -= l - lx + 1;
    --lx;
  }
  return lx;
}
__host__ __device__ constexpr int comp_ly(int l, int i) {
  int lx = l, rem = i;
  while (rem >= l - lx + 1) {
    rem -= l - lx + 1;
    --lx;
  }
  return (l - lx) - rem;
}
__host__ __device__ constexpr int comp_lz(int l, int i) { return l - comp_lx(l, i) - comp_ly(l, i); }
// Degree of the k-th triple in the range starting at degree lo.
__host__ __device__ constexpr int range_deg(int lo, int k) {
  int d = lo;
  while (k >= ncart(d)) {
    k -= ncart(d);
    ++d;
  }
  return d;
}
__host__ __device__ constexpr int range_idx(int lo, int k) {
  int d = lo;
  while (k >= ncart(d)) {
    k -= ncart(d);
    ++d;
  }
  return k;
}
__host__ __device__ constexpr int range_x(int lo, int k) { return comp_lx(range_deg(lo, k), range_idx(lo, k)); }
__host__ __device__ constexpr int range_y(int lo, int k) { return comp_ly(range_deg(lo, k), range_idx(lo, k)); }
__host__ __device__ constexpr int range_z(int lo, int k) { return comp_lz(range_deg(lo, k), range_idx(lo, k)); }

// Pair class pc = l_a(l_a+1)/2 + l_b (l_a >= l_b) and back.
__host__ __device__ constexpr int pc_la(int pc) {
  int la = 0;
  while ((la + 1) * (la + 2) / 2 <= pc) ++la;
  return la;
}
__host__ __device__ constexpr int pc_lb(int pc) { return pc - pc_la(pc) * (pc_la(pc) + 1) / 2; }

// cart_index / addr (src/math/am.rs:51-55, src/engine/os_eri.rs:129-137)
__host__ __device__ inline int cart_index3(int lx, int ly, int lz) {
  int d = ly + lz;
  return d * (d + 1) / 2 + lz;
}
__host__ __device__ inline int addr3(int lx, int ly, int lz) {
  return tri_below(lx + ly + lz) + cart_index3(lx, ly, lz);
}

template <int N, typename F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
// Calls f(std::integral_constant<int, i>) for i = 0 .. N-1, fully unrolled.
template <int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl<N>(static_cast<F&&>(f), std::make_integer_sequence<int, N>{});
}

// ----------------------------------------------------------- device tables

// Each translation unit (one per bra pair class) is its own device module,
// so every module carries its own copy of these tables, filled by its
// upload_module_constants().
// Triples by global address (degree <= 20): packed lx | ly<<8 | lz<<16.
constexpr int ADDR_TAB_DEG = ADDR_TAB_DEG_HOST;
static __constant__ int c_addr_lxyz[n_addr(ADDR_TAB_DEG)];
static __constant__ double c_lag_x[MAX_ROOTS][MAX_ROOTS];
static __constant__ double c_lag_w[MAX_ROOTS][MAX_ROOTS];
static __constant__ float c_lag_xf[MAX_ROOTS][MAX_ROOTS];
static __constant__ float c_lag_wf[MAX_ROOTS][MAX_ROOTS];
static __constant__ const double* c_rys_tab;
static __constant__ const float* c_rys_tab_f;

static inline cudaError_t upload_module_constants(const ConstData& c) {
  cudaError_t e;
  if ((e = cudaMemcpyToSymbol(c_addr_lxyz, c.addr_lxyz, sizeof(int) * c.n_addr))) return e;
  if ((e = cudaMemcpyToSymbol(c_lag_x, c.lag_x, sizeof(double) * MAX_ROOTS * MAX_ROOTS))) return e;
  if ((e = cudaMemcpyToSymbol(c_lag_w, c.lag_w, sizeof(double) * MAX_ROOTS * MAX_ROOTS))) return e;
  if ((e = cudaMemcpyToSymbol(c_lag_xf, c.lag_xf, sizeof(float) * MAX_ROOTS * MAX_ROOTS))) return e;
  if ((e = cudaMemcpyToSymbol(c_lag_wf, c.lag_wf, sizeof(float) * MAX_ROOTS * MAX_ROOTS))) return e;
  if ((e = cudaMemcpyToSymbol(c_rys_tab, &c.tab, sizeof(c.tab)))) return e;
  if ((e = cudaMemcpyToSymbol(c_rys_tab_f, &c.tab_f, sizeof(c.tab_f)))) return e;
  return cudaSuccess;
}

__device__ __forceinline__ int addr_lx(int a) { return c_addr_lxyz[a] & 0xff; }
__device__ __forceinline__ int addr_ly(int a) { return (c_addr_lxyz[a] >> 8) & 0xff; }
__device__ __forceinline__ int addr_lz(int a) { return (c_addr_lxyz[a] >> 16) & 0xff; }

// ----------------------------------------------------------------- Rys

// Whether a kernel stages its N-root table in shared memory: the
// one-thread classes and the FP32 teams up to four roots (at most 46 KB per block).  FP64 teams, whose shared memory holds the
// recurrence tables of their primitive quartets, and larger N read it through
// L1 (a team evaluates one root per lane, a small part of its work).
template <int N, typename R>
__host__ __device__ constexpr bool rys_staged(int team) {
  return N <= 4 && (team == 1 || sizeof(R) == 4);
}
template <int N, typename R>
__host__ __device__ constexpr int rys_smem(int team) {
  return rys_staged<N, R>(team) ? rys_nsub<R>(N) * rys_row<R>(N) : 4;
}

template <int N, typename R>
__device__ __forceinline__ const R* rys_global() {
  if constexpr (sizeof(R) == 8)
    return c_rys_tab + rys_off<double>(N);
  else
    return c_rys_tab_f + rys_off<float>(N);
}

// Copy the N-root table into shared memory where the kernel stages it; every
// thread of the block must call it (it ends in a block barrier either way).
template <int N, typename R, int TEAM>
__device__ __forceinline__ void stage_rys_table(R* s_tab) {
  if constexpr (rys_staged<N, R>(TEAM)) {
    constexpr int PER = 16 / sizeof(R);
    const uint4* src = reinterpret_cast<const uint4*>(rys_global<N, R>());
    uint4* dst = reinterpret_cast<uint4*>(s_tab);
    for (int i = threadIdx.x; i < rys_nsub<R>(N) * rys_row<R>(N) / PER; i += blockDim.x) dst[i] = __ldg(src + i);
  }
  __syncthreads();
}

// One polynomial of NC coefficients of a table row (16-byte aligned; GLOBAL:
// read through the read-only path) by Horner's scheme.  The short intervals
// replace 17-term Chebyshev sums on intervals about six wide, and their position
// needs no rounding or division.
template <int NC, bool GLOBAL>
__device__ __forceinline__ double rys_poly(const double* c, double xi) {
  static_assert(NC % 2 == 0, "two coefficients a read");
  const double2* q = reinterpret_cast<const double2*>(c);
  auto at = [q](int k) {
    if constexpr (GLOBAL)
      return __ldg(q + k);
    else
      return q[k];
  };
  double2 t = at(NC / 2 - 1);
  double v = fma(t.y, xi, t.x);
#pragma unroll
  for (int k = NC / 2 - 2; k >= 0; --k) {
    t = at(k);
    v = fma(v, xi, t.y);
    v = fma(v, xi, t.x);
  }
  return v;
}
template <int NC, bool GLOBAL>
__device__ __forceinline__ float rys_poly(const float* c, float xi) {
  static_assert(NC % 4 == 0, "four coefficients a read");
  const float4* q = reinterpret_cast<const float4*>(c);
  auto at = [q](int k) {
    if constexpr (GLOBAL)
      return __ldg(q + k);
    else
      return q[k];
  };
  float v = 0.f;
#pragma unroll
  for (int k = NC / 4 - 1; k >= 0; --k) {
    const float4 t = at(k);
    v = k == NC / 4 - 1 ? t.w : fmaf(v, xi, t.w);
    v = fmaf(v, xi, t.z);
    v = fmaf(v, xi, t.y);
    v = fmaf(v, xi, t.x);
  }
  return v;
}

// N-point Rys quadrature at parameter T (src/math/rys.rs:174-215): the
// generalized-Laguerre(-1/2) limit above the crossover, else the tables.
// x = squared roots, w = weights.
template <int N, bool GLOBAL, typename R>
__device__ __forceinline__ void rys_roots_s(const R* tab, R T, R* x, R* w) {
  if (!rys_tabulated(N, T)) {
    const R r = rsqrt(T);
    const R inv_t = R(1) / T;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if constexpr (sizeof(R) == 8) {
        x[i] = c_lag_x[N - 1][i] * inv_t;
        w[i] = c_lag_w[N - 1][i] * (R(0.5) * r);
      } else {
        x[i] = c_lag_xf[N - 1][i] * inv_t;
        w[i] = c_lag_wf[N - 1][i] * (R(0.5) * r);
      }
    }
    return;
  }
  R xi;
  const R* row = tab + rys_interval(N, T, xi) * rys_row<R>(N);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    x[i] = rys_poly<rys_nc<R>(N), GLOBAL>(row + (2 * i) * rys_nc<R>(N), xi);
    w[i] = rys_poly<rys_nc<R>(N), GLOBAL>(row + (2 * i + 1) * rys_nc<R>(N), xi);
  }
}

// Root r of the N-point quadrature.
template <int N, bool GLOBAL, typename R>
__device__ __forceinline__ void rys_root_one(const R* tab, R T, int r, R& x, R& w) {
  if (!rys_tabulated(N, T)) {
    if constexpr (sizeof(R) == 8) {
      x = c_lag_x[N - 1][r] / T;
      w = c_lag_w[N - 1][r] * R(0.5) * rsqrt(T);
    } else {
      x = c_lag_xf[N - 1][r] / T;
      w = c_lag_wf[N - 1][r] * R(0.5) * rsqrt(T);
    }
    return;
  }
  R xi;
  const R* c = tab + rys_interval(N, T, xi) * rys_row<R>(N) + 2 * r * rys_nc<R>(N);
  x = rys_poly<rys_nc<R>(N), GLOBAL>(c, xi);
  w = rys_poly<rys_nc<R>(N), GLOBAL>(c + rys_nc<R>(N), xi);
}

// Per-axis Rys vertical recurrence g[n][m], n <= NE (bra power on A),
// m <= NF (ket power on C), seeded with g[0][0] = g00 (src/engine/rys.rs:
// 246-268; the seed scales the whole table, which folds the weight and
// prefactor into one axis).
template <int NE, int NF, typename R>
__device__ __forceinline__ void vrr_axis(R g00, R c00, R cp0, R b10, R b01, R b00,
                                         R (&g)[NE + 1][NF + 1]) {
  g[0][0] = g00;
  if constexpr (NE >= 1) g[1][0] = c00 * g00;
#pragma unroll
  for (int n = 1; n < NE; ++n) g[n + 1][0] = c00 * g[n][0] + R(n) * b10 * g[n - 1][0];
#pragma unroll
  for (int m = 0; m < NF; ++m) {
#pragma unroll
    for (int n = 0; n <= NE; ++n) {
      R t = cp0 * g[n][m];
      if (m >= 1) t += R(m) * b01 * g[n][m - 1];
      if (n >= 1) t += R(n) * b00 * g[n - 1][m];
      g[n][m + 1] = t;
    }
  }
}

// Per-primitive-quartet scalars of the Rys quadrature (src/engine/rys.rs:
// 140-166) in evaluation orientation.  For the long-range operator
// erf(omega r)/r (omega > 0, src/engine/rys.rs:163-175) the quadrature is
// taken at s*T with s = omega^2 / (rho + omega^2), every root scaled by s
// (xs) and every weight by sqrt(s) (folded into pref); omega = 0 is the
// Coulomb operator, with T and pref untouched and xs = 1.
template <typename R>
struct QuartetHdr {
  R T, pref;
  R qpq, ppq;       // q / (p + q), p / (p + q)
  R hpq;            // 1 / (2 (p + q))
  R inv2p, inv2q;   // 1 / (2 p), 1 / (2 q)
  R pqx, pqy, pqz;  // P - Q
  R pax, pay, paz;  // P - A
  R qcx, qcy, qcz;  // Q - C
  R xs;             // root scale (1 for Coulomb)
};

// r = 1 / sqrt(s) and inv = 1 / s from one rsqrt and a Newton step shared by
// both (FP32's approximate rsqrt is otherwise off by up to two units).
template <typename R>
__device__ __forceinline__ void inv_and_rsqrt(R s, R& r, R& inv) {
  const R y = rsqrt(s);
  const R e = fma(-(s * y), y, R(1));
  r = fma(R(0.5) * y, e, y);
  inv = r * r;
}

template <typename R>
__device__ __forceinline__ void erf_scale(QuartetHdr<R>& h, R rho, double omega) {
  h.xs = R(1);
  if (omega > 0.0) {
    const R w2 = R(omega) * R(omega);
    const R sc = w2 / (rho + w2);
    h.T *= sc;
    h.pref *= sqrt(sc);
    h.xs = sc;
  }
}

template <typename R>
__device__ __forceinline__ QuartetHdr<R> quartet_header(const PrimPairD& bp, const PrimPairD& kp,
                                                        double omega) {
  QuartetHdr<R> h;
  const R p = R(bp.zeta), q = R(kp.zeta);
  R r, inv;
  inv_and_rsqrt(p + q, r, inv);
  h.hpq = R(0.5) * inv;
  h.qpq = q * inv;
  h.ppq = p * inv;
  const R rho = p * h.qpq;
  // centre differences in double first: absolute coordinates would lose
  // the separation to cancellation in FP32
  h.pqx = R(bp.px - kp.px);
  h.pqy = R(bp.py - kp.py);
  h.pqz = R(bp.pz - kp.pz);
  h.T = rho * (h.pqx * h.pqx + h.pqy * h.pqy + h.pqz * h.pqz);
  h.pref = R(bp.ez) * R(kp.ez) * r;
  h.inv2p = R(bp.inv2z);
  h.inv2q = R(kp.inv2z);
  h.pax = R(bp.pax);
  h.pay = R(bp.pay);
  h.paz = R(bp.paz);
  h.qcx = R(kp.pax);
  h.qcy = R(kp.pay);
  h.qcz = R(kp.paz);
  erf_scale(h, rho, omega);
  return h;
}

// The Rys parameter T of a primitive quartet in FP64 from the double pair
// data (the same expression as quartet_header, erf scaling included).
__device__ __forceinline__ double quartet_T64(const PrimPairD& bp, const PrimPairD& kp, double omega) {
  const double p = bp.zeta, q = kp.zeta, pq = p + q;
  const double rho = p * q / pq;
  const double dx = bp.px - kp.px, dy = bp.py - kp.py, dz = bp.pz - kp.pz;
  double T = rho * (dx * dx + dy * dy + dz * dz);
  if (omega > 0.0) T *= omega * omega / (rho + omega * omega);
  return T;
}

// The FP32 launches generate roots and weights in FP64 for every quadrature
// of five or more roots (high angular momentum, l_a + l_b + l_c + l_d >= 8):
// the n where weights lose digits just below the asymptotic crossover
// (the reference's own FP64 weights lose three to four there at n = 9, 11,
// 13, src/math/rys.rs:80-89) are all among them.  Above the crossover the
// roots and weights are the closed forms c_i / T and w_i T^{-1/2}, exact to
// FP32 rounding at every n.
constexpr int ROOTS64_NR = 5;
template <int N, typename R>
__device__ __forceinline__ bool roots_in_fp64(R) {
  return sizeof(R) == 4 && N >= ROOTS64_NR;
}

// quartet_header for the FP32 launches from the FP32 pair copies; ac = the
// bra's first evaluation shell centre minus the ket's, rounded once per
// quartet.
__device__ __forceinline__ QuartetHdr<float> quartet_header_f(const PrimPairF& bp, const PrimPairF& kp, float acx,
                                                              float acy, float acz, double omega) {
  QuartetHdr<float> h;
  const float p = bp.zeta, q = kp.zeta;
  float r, inv;
  inv_and_rsqrt(p + q, r, inv);
  h.hpq = 0.5f * inv;
  h.qpq = q * inv;
  h.ppq = p * inv;
  const float rho = p * h.qpq;
  h.pqx = acx + (bp.pax - kp.pax);
  h.pqy = acy + (bp.pay - kp.pay);
  h.pqz = acz + (bp.paz - kp.paz);
  h.T = rho * (h.pqx * h.pqx + h.pqy * h.pqy + h.pqz * h.pqz);
  h.pref = bp.ez * kp.ez * r;
  h.inv2p = bp.inv2z;
  h.inv2q = kp.inv2z;
  h.pax = bp.pax;
  h.pay = bp.pay;
  h.paz = bp.paz;
  h.qcx = kp.pax;
  h.qcy = kp.pay;
  h.qcz = kp.paz;
  erf_scale(h, rho, omega);
  return h;
}

// Primitive pair q of a lane's ket: from the class's interleaved copy when
// the launch has one, else from the pair list.
__device__ __forceinline__ PrimPairD load_ket(const KernelArgs& A, int prim_off, int kpos, int q, double) {
  if (!A.kets) return A.prims[prim_off + q];
  const size_t st = A.ket_stride;
  const double* p = A.kets + (size_t)q * KET_VALS * st + kpos;
  PrimPairD k;
  k.zeta = __ldg(p);
  k.inv2z = __ldg(p + st);
  k.ez = __ldg(p + 2 * st);
  k.px = __ldg(p + 3 * st);
  k.py = __ldg(p + 4 * st);
  k.pz = __ldg(p + 5 * st);
  k.pax = __ldg(p + 6 * st);
  k.pay = __ldg(p + 7 * st);
  k.paz = __ldg(p + 8 * st);
  return k;
}
__device__ __forceinline__ PrimPairF load_ket(const KernelArgs& A, int prim_off, int kpos, int q, float) {
  if (!A.ketsf) return A.primsf[prim_off + q];
  const size_t st = A.ket_stride;
  const float* p = A.ketsf + (size_t)q * KET_VALS_F * st + kpos;
  PrimPairF k;
  k.zeta = __ldg(p);
  k.inv2z = __ldg(p + st);
  k.ez = __ldg(p + 2 * st);
  k.pax = __ldg(p + 3 * st);
  k.pay = __ldg(p + 4 * st);
  k.paz = __ldg(p + 5 * st);
  return k;
}

// ----------------------------------------------------------- misc device

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
// Identity of one screened canonical quartet with its density mask; the sum
// over the list (mod 2^64) fingerprints the list independent of order.
__device__ __forceinline__ uint64_t quartet_key(int i, int j, int k, int l, uint64_t mask) {
  uint64_t id = ((((uint64_t)i * 65536u + (uint64_t)j) * 65536u + (uint64_t)k) * 65536u) + (uint64_t)l;
  return splitmix64(id ^ splitmix64(mask + 0x5851F42D4C957F2Dull));
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace igpu
