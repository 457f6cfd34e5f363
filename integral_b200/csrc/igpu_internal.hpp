// Internal data layout shared by the host plan (plan*.cpp) and the device
// kernels (kernels.cu).  Everything here is plain data in device memory.
#pragma once
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define IGPU_HD __host__ __device__
#else
#define IGPU_HD
#endif

namespace igpu {

constexpr int MAX_L = 6;             // reference engine cap (src/engine/os.rs:34)
constexpr int MAX_GRAD_L = MAX_L - 1;
constexpr int GPU_MAX_L = 4;         // highest shell l with compiled quartet kernels
constexpr int MAX_ROOTS = 13;
constexpr int MAX_DENS = 64;
constexpr int ADDR_TAB_DEG_HOST = 20;  // degrees of the device triple table

// One shell on the device.
struct DevShell {
  double cx, cy, cz;
  int l;
  int nprim;
  int off;       // first function (AO) index
  int nfunc;     // n_cart or 2l+1
  int atom;      // index into Basis::atoms()
  int spherical;
  int prim_off;  // first primitive in the exponent/coefficient arrays
  int pad;
};

// One primitive pair of a shell pair in evaluation orientation (first shell
// A, second shell B, l_A >= l_B), surviving the 1e-32 pair screen of the
// reference (src/engine/os_eri.rs:211-244).
// The quartet kernels form every per-quartet factor from products of these
// and one rsqrt of zeta_bra + zeta_ket: no division per primitive quartet.
struct alignas(16) PrimPairD {
  double zeta;       // alpha + beta
  double inv2z;      // 1 / (2 zeta)
  double ez;         // kappa * c_A * c_B (effective coefficients) * sqrt(2 pi^{5/2}) / zeta
  double px, py, pz; // Gaussian product centre
  double pax, pay, paz;  // P - A
  double alpha;      // exponent on A (gradient raise on A)
  double beta;       // exponent on B
  double pad;
};
// sqrt(2 pi^{5/2}): the product of two pairs' ez carries the Coulomb prefactor.
constexpr double SQRT_TWO_PI_2_5 = 5.914967172795613;

// FP32 copy of one primitive pair for the FP32 launches, rounded once at
// plan creation: the FP32 header then needs no double loads or conversions.
// P - Q of a quartet is formed as (A - C) + (PA - QC), with A - C (the
// evaluation shells' centres) rounded once per quartet, so no absolute
// coordinate enters an FP32 difference.
struct alignas(16) PrimPairF {
  float zeta, inv2z, ez;
  float pax, pay, paz;
  float alpha, beta;
};

// Lane-interleaved copy of a ket class's primitive pairs for the kernels that
// run one quartet per lane: value v of primitive pair q of the ket at position
// k of the class list lies at (q * KET_VALS + v) * stride + k, so that lanes
// on consecutive kets read consecutive values.  From PrimPairD each such read
// of a warp takes one L1 wavefront per lane (96 bytes apart), which bound
// those kernels: 82-92% of the L1 rate in FP64.
constexpr int KET_VALS = 9;    // zeta, inv2z, ez, px, py, pz, pax, pay, paz
constexpr int KET_VALS_F = 6;  // zeta, inv2z, ez, pax, pay, paz

// One canonical shell pair (i >= j in the reference's sense) with its
// evaluation orientation.  An auxiliary pair of density fitting (an aux shell
// with the unit s dummy, src/df.rs:1-37) has i = the aux shell's position in
// the aux basis, j = -1 and tri = -1.
struct PairD {
  int a, b;       // evaluation orientation shells (l_a >= l_b)
  int i, j;       // canonical shells (i >= j)
  int prim_off;   // into PrimPairD array
  int nprim;      // surviving primitive pairs
  int tri;        // i*(i+1)/2 + j
  int cls;        // pair class index (l_a*(l_a+1)/2 + l_b)
  double abx, aby, abz;  // A - B
  double q;       // Schwarz bound Q[i][j]
};

// Rys tables of the n-point quadrature: below rys_t_hi(n) the roots and
// weights are polynomials on intervals of T of length 1 / rys_div(n) (a power
// of two, so that the position xi in [-1, 1] is exact in both precisions), with
// ascending coefficients.  Row s holds root 0, weight 0, root 1, ...; its stride
// is an odd multiple of 16 bytes, so that the 16-byte reads of lanes in
// different intervals start in different shared-memory banks.  Above it the
// generalised Gauss-Laguerre limit holds.
//
// A one-thread kernel spends most of its shared-memory rate on these rows (its
// lanes are in different intervals), so in FP64 n <= 2, where little else is
// done per primitive quartet, takes 8 coefficients on quarters (as far as a
// block's 48 KB allow): 1.1 to 1.2 times as fast as 12 on unit intervals in
// (20|00), (10|10), (10|00).  The others take 12, FP32 8 (4 on sixteenths gained
// nothing there), on unit intervals.
template <typename R>
IGPU_HD constexpr int rys_div(int n) {
  return sizeof(R) == 8 && n <= 2 ? 4 : 1;
}
template <typename R>
IGPU_HD constexpr int rys_nc(int n) {
  return sizeof(R) == 8 && n > 2 ? 12 : 8;
}
IGPU_HD constexpr double rys_t_hi(int n) { return 30.5 + 5.0 * n; }
template <typename R>
IGPU_HD constexpr int rys_nsub(int n) {
  return (31 + 5 * n) * rys_div<R>(n);
}
// The tables hold T < rys_t_hi(n).  A NaN compares false: the closed form, which
// takes no index, returns it.
template <typename R>
IGPU_HD constexpr bool rys_tabulated(int n, R T) {
  return T < R(rys_t_hi(n));
}
// Interval of a tabulated T and the position in it.  A negative T (a negative
// exponent gives one) extrapolates the first interval.
template <typename R>
IGPU_HD inline int rys_interval(int n, R T, R& xi) {
  const R u = T * R(rys_div<R>(n));
#ifdef __CUDA_ARCH__
  // to unsigned: this conversion saturates, so a negative u gives 0 by itself
  int s;
  if constexpr (sizeof(R) == 8)
    s = (int)__double2uint_rz(u);
  else
    s = (int)__float2uint_rz(u);
#else
  int s = (int)u;
  s = s < 0 ? 0 : s;
#endif
  xi = R(2) * (u - R(s)) - R(1);
  return s;
}
template <typename R>
IGPU_HD constexpr int rys_row(int n) {
  return 2 * n * rys_nc<R>(n) + 16 / (int)sizeof(R);
}
template <typename R>
IGPU_HD constexpr int rys_off(int n) {
  int o = 0;
  for (int k = 1; k < n; ++k) o += rys_nsub<R>(k) * rys_row<R>(k);
  return o;
}

// Task list of one class-pair launch: for each listed bra (position in the
// bra class' Q-sorted pair list) kets 0..nket-1 of the ket class' sorted
// list.  prefix[b] = sum of nket over earlier bras (64-bit).
struct TaskList {
  const int* bra_pair;          // pair index per task bra
  const int* ket_pairs;         // Q-sorted pair indices of the ket class
  const unsigned long long* prefix;  // nbra + 1 entries
  const int* ket_start;         // first ket position per bra (NULL = 0)
  int nbra;
  unsigned long long total;
};

// Constant tables every device module needs (uploaded per module).
struct ConstData {
  const int* addr_lxyz;
  int n_addr;
  const double* lag_x;   // MAX_ROOTS x MAX_ROOTS
  const double* lag_w;
  const float* lag_xf;
  const float* lag_wf;
  const double* tab;     // device Rys tables (rys_off, rys_row)
  const float* tab_f;
};

// Output modes of the quartet kernels.
enum Mode : int {
  MODE_JK = 0,
  MODE_DENSE = 1,
  MODE_SCHWARZ = 2,
  MODE_BUILDER = 3,
  MODE_GRAD = 4,
  MODE_PACKED = 5,
  MODE_DF3 = 6,  // density fitting (mu nu|P): main pair x (aux shell, unit s)
  MODE_DF2 = 7,  // density fitting (P|Q): (aux shell, unit s) x (aux shell, unit s)
  MODE_BLOCK = 8,  // one shell-quartet block in a requested shell order
};

struct JKDev {
  const double* D;       // ndens x nao x nao
  const float* Df;       // its FP32 copy, read by the FP32 launches
  const double* bounds;  // ndens x nsh x nsh  (density_shell_bounds)
  double* J;             // symmetric: one-orientation accumulators J', K'
  double* K;             //   (J = (J' + J'^T)/2 added by the finalize pass)
  int ndens;             // matrices contracted: nscreen, or 2 nscreen (symmetric parts, then antisymmetric ones)
  int nscreen;           // densities the screening sees (bounds)
  int nj;                // first matrices that have a Coulomb part
  int want_k;
  int symmetric;         // every matrix symmetric or antisymmetric (bitwise): one-orientation sums
  double threshold;
};

// Two-particle density of the gradient as product terms factor * L (x) R
// (GradDensityTerm, src/direct_grad.rs:21-25).  Per term: device pointers to
// the nao x nao matrices and to their symmetrised shell-block maxima
// (nsh x nsh, src/direct_grad.rs:292-312).  c* = Coulomb-type terms, x* =
// exchange-type terms.
struct GradDev {
  const double* const* cl;
  const double* const* cr;
  const double* const* cl_max;
  const double* const* cr_max;
  const double* cf;      // factors
  const double* const* xl;
  const double* const* xr;
  const double* const* xl_max;
  const double* const* xr_max;
  const double* xf;
  int ncoul, nexch;
  double threshold;
  double* out;           // natom x 3, dE/dR accumulated
};

struct Counters {
  unsigned long long quartets;
  unsigned long long hash;
  unsigned long long fp32_quartets;
  unsigned long long prim_quartets;
  unsigned long long skipped;
  unsigned long long pad[3];
};

// Everything a quartet kernel needs.
struct KernelArgs {
  const DevShell* shells;
  const PairD* pairs;
  const PrimPairD* prims;
  const PrimPairF* primsf;  // FP32 copy of prims (same order)
  const double* kets;       // this ket class's interleaved copies (nullptr: none)
  const float* ketsf;
  size_t ket_stride;
  const double* c2s;     // c2s matrices (ratio folded), c2s_off[l] into it
  int c2s_off[GPU_MAX_L + 3];
  int nsh;
  int nao;
  TaskList task;
  int mode;
  int fp32;              // this launch evaluates in FP32
  double* scratch;       // per-team slots for the post phase
  size_t slot_doubles;
  JKDev jk;
  GradDev grad;
  double* dense;         // nao^4 (MODE_DENSE / MODE_BUILDER); packed triangle (MODE_PACKED)
  const long long* packed_start;  // MODE_PACKED: first AO-pair index of every canonical shell pair
  double* schwarz_out;   // per pair Q (MODE_SCHWARZ)
  Counters* counters;
  int builder_swap;      // builder mode: requested bra is the evaluation ket
  const unsigned* bra_bitmap;  // optional: reference bra pairs to keep (bit per pair)
  unsigned long long* work_counter;  // next unclaimed task (dynamic chunks)
  unsigned long long chunk;          // tasks claimed per grab (per warp)
  int split;             // one-thread kernels: lanes sharing a quartet's bra primitives (power of two)
  size_t acc_offset;     // slot offset of the running bra-block J accumulators
  int kinds;             // 0 all shells Cartesian, 1 all spherical, 2 mixed
  double omega;          // 0: Coulomb 1/r; > 0: long-range erf(omega r)/r
  int naux;              // MODE_DF3 / MODE_DF2: auxiliary functions
  size_t dense_len;      // MODE_DF3 / MODE_DF2 / MODE_BLOCK: doubles in `dense`
  unsigned* store_fault; // MODE_DF3 / MODE_DF2 / MODE_BLOCK: set when an index falls outside `dense`
  int blk_shells[4];     // MODE_BLOCK: requested shells (i, j, k, l)
  int blk_dims[4];       // MODE_BLOCK: their function counts
  // FP32 launches of the mixed J/K path: a primitive quartet whose magnitude
  // bound |E_ab E_cd| 2 pi^{5/2} / (p q sqrt(p + q)) is below prim_cut is
  // skipped (0: every primitive quartet is evaluated)
  double prim_cut;
};

}  // namespace igpu
