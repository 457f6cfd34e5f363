// One-thread-per-quartet kernels of the larger Cartesian classes (symmetric
// J/K builds with many quartets).
//
// The team kernels (quartet.cuh) spread a quartet's [e0|f0] rows over lanes
// that read the 2D integrals from shared memory: (NF + 1) values per axis and
// row for NFP columns of two operations each, and a shared-memory read of a
// warp takes four times an FP64 (FP32) operation's issue.  They run at the
// shared-memory rate.  Here every lane keeps its own quartet's 2D integrals in
// registers, where their indices are compile-time constants, and the table is
// cut into row blocks instead:
//   - a group of 32 quartets (one per lane) is taken by WPG warps; each warp
//     sums its own row block(s) of all 32 tables over the primitive quartets,
//     recomputing the recurrences, while the Rys roots are shared: each warp
//     evaluates every WPG-th root and passes it on in shared memory, one
//     group barrier per primitive quartet (double buffered);
//   - the tables go to scratch, interleaved by lane (coalesced);
//   - then every warp finishes one of the block's four groups, one quartet per
//     lane: per ket component pair (c, d) the ket recurrence combines table
//     columns, the bra recurrence runs in registers, and the six image sums
//     follow while the (a, b) slice is there.
// A class uses these kernels when its launch has enough quartets to fill the
// device with groups (wide_min_tasks); smaller launches keep the teams, whose
// quartets finish sooner.
#pragma once
#include "post_thread.cuh"
#include "quartet.cuh"

namespace igpu {

template <int LA, int LB, int LC, int LD, typename R>
struct WideShape {
  using S = ClassShape<LA, LB, LC, LD>;
  // accumulators per lane: with the recurrence tables they fill the 255
  // registers of a 128-thread block at two blocks per SM
  static constexpr int BUD = sizeof(R) == 8 ? 56 : 104;
  static constexpr int RMAX = BUD / S::NFP < 1 ? 1 : BUD / S::NFP;
  static constexpr int NP = (S::NEP + RMAX - 1) / RMAX;  // row blocks
  static constexpr int WPG = NP <= 1 ? 1 : (NP <= 2 ? 2 : 4);
  static constexpr int PPW = (NP + WPG - 1) / WPG;       // row blocks per warp
  static constexpr int ROWS = (S::NEP + WPG * PPW - 1) / (WPG * PPW);
  static constexpr int NAB = ncart(LA) * ncart(LB);
  // bytes: four groups' tables
  static constexpr size_t TAB = (size_t)4 * S::NG * 32 * sizeof(R);
};
// Scratch doubles of one block: the tables of four groups, then per warp and
// lane the running bra-block J sums (bra index and ndens blocks).
template <int LA, int LB, int LC, int LD, typename R>
__host__ __device__ constexpr size_t wide_tab_doubles() {
  return (WideShape<LA, LB, LC, LD, R>::TAB + 7) / 8;
}

// Barrier of the WPG warps of group team gt: by number, since the warps reach it
// from the different row blocks that they sum (wide_rows).  Every row block, the
// empty ones too, passes the same barriers: one per primitive quartet of the
// group, skipped by all warps or none.
template <int WPG>
__device__ __forceinline__ void wide_sync(int gt) {
  if constexpr (WPG == 1)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(1 + gt), "r"(WPG * 32) : "memory");
}

// A lane whose quartet has no primitives, or none at all (!has), runs along on
// another lane's pairs (the caller's choice) with weight zero.
template <int LA, int LB, int LC, int LD, typename R, int E0>
__device__ __forceinline__ void wide_rows(const KernelArgs& A, const R* tab, R* s_roots, bool has, const PairD& pb,
                                          const PairD& pk, int kpos, int npb, int npk, int wi, int gt, int lane,
                                          R* G) {
  using S = ClassShape<LA, LB, LC, LD>;
  using W = WideShape<LA, LB, LC, LD, R>;
  constexpr int NE = S::NE, NF = S::NF, NR = S::NR, WPG = W::WPG, NFP = S::NFP;
  constexpr int NROW = E0 >= S::NEP ? 0 : (E0 + W::ROWS <= S::NEP ? W::ROWS : S::NEP - E0);
  R acc[NROW > 0 ? NROW * NFP : 1];
#pragma unroll
  for (int q = 0; q < (NROW > 0 ? NROW * NFP : 1); ++q) acc[q] = R(0);
  const float cut = (sizeof(R) == 4 && A.fp32) ? (float)A.prim_cut : 0.f;
  float acx = 0.f, acy = 0.f, acz = 0.f;
  if constexpr (sizeof(R) == 4) {
    const DevShell& sa = A.shells[pb.a];
    const DevShell& sc = A.shells[pk.a];
    acx = (float)(sa.cx - sc.cx);
    acy = (float)(sa.cy - sc.cy);
    acz = (float)(sa.cz - sc.cz);
  }
  int buf = 0;
  for (int ip = 0; ip < npb; ++ip) {
    const int bi = pb.prim_off + (ip < pb.nprim ? ip : 0);
    for (int kq = 0; kq < npk; ++kq) {
      const int kk = kq < pk.nprim ? kq : 0;
      bool live = has && ip < pb.nprim && kq < pk.nprim;
      QuartetHdr<R> h;
      if constexpr (sizeof(R) == 4) {
        const PrimPairF bp = A.primsf[bi], kp = load_ket(A, pk.prim_off, kpos, kk, 0.f);
        if (cut > 0.f) {
          live = live && prim_bound(bp, kp) >= cut;
          if (!__any_sync(0xffffffffu, live)) continue;  // the same for every warp of the group
        }
        h = quartet_header_f(bp, kp, acx, acy, acz, A.omega);
      } else {
        h = quartet_header<R>(A.prims[bi], load_ket(A, pk.prim_off, kpos, kk, 0.0), A.omega);
      }
      if (!live) h.pref = R(0);
      R* sr = s_roots + buf * (2 * NR * 32) + lane;
      for (int r = wi; r < NR; r += WPG) {
        R xr, wr;
        if constexpr (sizeof(R) == 4 && NR >= ROOTS64_NR) {
          double xd, wd;
          const double T64 = quartet_T64(A.prims[bi], load_ket(A, pk.prim_off, kpos, kk, 0.0), A.omega);
          rys_root_one<NR, true>(rys_global<NR, double>(), T64, r, xd, wd);
          xr = R(xd);
          wr = R(wd);
        } else {
          rys_root_one<NR, !rys_staged<NR, R>(1)>(tab, h.T, r, xr, wr);
        }
        sr[r * 32] = xr * h.xs;
        sr[(NR + r) * 32] = wr * h.pref;
      }
      wide_sync<WPG>(gt);
      buf ^= 1;
      if constexpr (NROW > 0) {
#pragma unroll 1
        for (int r = 0; r < NR; ++r) {
          const R xr = sr[r * 32], wr = sr[(NR + r) * 32];
          const R cq = xr * h.qpq, cp = xr * h.ppq;
          const R b00 = xr * h.hpq;
          const R b10 = (R(1) - cq) * h.inv2p;
          const R b01 = (R(1) - cp) * h.inv2q;
          R gx[NE + 1][NF + 1], gy[NE + 1][NF + 1], gz[NE + 1][NF + 1];
          vrr_axis<NE, NF, R>(R(1), h.pax - cq * h.pqx, h.qcx + cp * h.pqx, b10, b01, b00, gx);
          vrr_axis<NE, NF, R>(R(1), h.pay - cq * h.pqy, h.qcy + cp * h.pqy, b10, b01, b00, gy);
          vrr_axis<NE, NF, R>(wr, h.paz - cq * h.pqz, h.qcz + cp * h.pqz, b10, b01, b00, gz);
          static_for<NROW>([&](auto e) {
            constexpr int ei = E0 + decltype(e)::value;
            constexpr int ex = range_x(LA, ei), ey = range_y(LA, ei), ez = range_z(LA, ei);
            static_for<NFP>([&](auto f) {
              constexpr int fx = range_x(LC, decltype(f)::value), fy = range_y(LC, decltype(f)::value),
                            fz = range_z(LC, decltype(f)::value);
              acc[decltype(e)::value * NFP + decltype(f)::value] += gx[ex][fx] * gy[ey][fy] * gz[ez][fz];
            });
          });
        }
      }
    }
  }
  if constexpr (NROW > 0) {
#pragma unroll
    for (int q = 0; q < NROW * NFP; ++q) G[(size_t)(E0 * NFP + q) * 32 + lane] = acc[q];
  }
}

// The (a, b) slice of ket component pair (c, d): table columns of c and, for
// a p shell d, of c + 1_d; for a d shell the four columns of its two axes.
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void wide_slice(const R* G, int lane, int f0, int f1, int f2, int f3, R k1, R k2,
                                           const R ab[3], R (&B)[ncart(LA) * ncart(LB)]) {
  using S = ClassShape<LA, LB, LC, LD>;
  R t[S::NEP];
#pragma unroll
  for (int e = 0; e < S::NEP; ++e) {
    const R* g = G + (size_t)e * S::NFP * 32 + lane;
    R v = g[f0 * 32];
    if constexpr (LD >= 1) v = g[f1 * 32] + k1 * v;
    // d = 1_i + 1_j: (c + 1_i + 1_j) + CD_j (c + 1_i) + CD_i ((c + 1_j) + CD_j c)
    if constexpr (LD == 2) v = g[f3 * 32] + k1 * g[f2 * 32] + k2 * v;
    t[e] = v;
  }
  bra_hrr<LA, LB, 1, 1, R>(t, B, ab);  // [b][a]
}

// Index of component (degree l, index i, y + z = m) raised along axis x.
__device__ __forceinline__ int raise_index(int i, int m, int axis) { return axis == 0 ? i : i + m + axis; }

// Horizontal recurrences and the symmetric-density J/K sums of this lane's
// quartet (thread_jk's sums, the block formed slice by slice).
template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void wide_post(const KernelArgs& A, const R* G, const PairD& pb, const PairD& pk,
                                          uint64_t mask, double* acc, int lane) {
  constexpr int NA = ncart(LA), NB = ncart(LB), ND = ncart(LD), NAB = NA * NB;
  const R ab[3] = {(R)pb.abx, (R)pb.aby, (R)pb.abz};
  const R cd[3] = {(R)pk.abx, (R)pk.aby, (R)pk.abz};
  const int shl[4] = {pb.a, pb.b, pk.a, pk.b};
  const int oa = A.shells[shl[0]].off, ob = A.shells[shl[1]].off, oc = A.shells[shl[2]].off, od = A.shells[shl[3]].off;
  const unsigned w = distinct_perms(shl);
  auto Wt = [&](int p) { return (R)((w >> p) & 1u); };
  const R wab = Wt(0) + Wt(1) + Wt(2) + Wt(3), wcd = Wt(4) + Wt(5) + Wt(6) + Wt(7);
  const R wac = Wt(0) + Wt(4), wbc = Wt(1) + Wt(5), wad = Wt(2) + Wt(6), wbd = Wt(3) + Wt(7);
  const size_t nao = (size_t)A.nao, n2 = nao * nao;
  const bool want_k = A.jk.want_k != 0;
  // the (a, d) and (b, d) sums stay in registers over c where they fit, and
  // the running (a, b) sums go to their interleaved store slice by slice where
  // 36 FP64 values would spill
  constexpr bool KEEP_D = ND == 1 || (ND == 3 && (sizeof(R) == 4 || NAB <= 18));
  constexpr bool KEEP_AB = sizeof(R) == 4 || NAB <= 18;
  constexpr int NK = KEEP_D ? ND : 1;
  for (int dn = 0; dn < A.jk.ndens; ++dn) {
    if (!((mask >> dn) & 1ull)) continue;
    const R* Dm = dens_of<R>(A.jk) + dn * n2;
    double* J = A.jk.J + dn * n2;
    double* K = want_k ? A.jk.K + dn * n2 : nullptr;
    const bool want_j = dn < A.jk.nj;
    R jab[KEEP_AB ? NAB : 1], kad[NK][NA], kbd[NK][NB];
    double* const ja = acc + ((size_t)1 + (size_t)dn * NAB) * 32;
#pragma unroll
    for (int q = 0; q < (KEEP_AB ? NAB : 1); ++q) jab[q] = R(0);
#pragma unroll
    for (int d = 0; d < NK; ++d) {
#pragma unroll
      for (int a = 0; a < NA; ++a) kad[d][a] = R(0);
#pragma unroll
      for (int b = 0; b < NB; ++b) kbd[d][b] = R(0);
    }
    int c = 0;
#pragma unroll 1
    for (int m = 0; m <= LC; ++m)
#pragma unroll 1
      for (int z = 0; z <= m; ++z, ++c) {
        R kac[NA], kbc[NB], dac[NA], dbc[NB];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          kac[a] = R(0);
          dac[a] = want_k ? __ldg(Dm + (oa + a) * nao + oc + c) : R(0);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          kbc[b] = R(0);
          dbc[b] = want_k ? __ldg(Dm + (ob + b) * nao + oc + c) : R(0);
        }
        auto term = [&](int d, const R (&B)[NAB], R (&kadd)[NA], R (&kbdd)[NB]) {
          if (want_j) {
            const R dcd = __ldg(Dm + (oc + c) * nao + od + d);
            R jcd = R(0);
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                const R v = B[b * NA + a];
                if constexpr (KEEP_AB)
                  jab[a * NB + b] += v * dcd;
                else
                  ja[(a * NB + b) * 32] += (double)(wab * (v * dcd));
                jcd += v * __ldg(Dm + (oa + a) * nao + ob + b);
              }
            if (wcd != R(0)) atomicAdd(J + (oc + c) * nao + od + d, (double)(wcd * jcd));
          }
          if (want_k) {
            R dad[NA], dbd[NB];
#pragma unroll
            for (int a = 0; a < NA; ++a) dad[a] = __ldg(Dm + (oa + a) * nao + od + d);
#pragma unroll
            for (int b = 0; b < NB; ++b) dbd[b] = __ldg(Dm + (ob + b) * nao + od + d);
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                const R v = B[b * NA + a];
                kac[a] += v * dbd[b];
                kbc[b] += v * dad[a];
                kadd[a] += v * dbc[b];
                kbdd[b] += v * dac[a];
              }
          }
        };
        auto flush_d = [&](int d, R (&kadd)[NA], R (&kbdd)[NB]) {
#pragma unroll
          for (int a = 0; a < NA; ++a)
            if (wad != R(0)) atomicAdd(K + (oa + a) * nao + od + d, (double)(wad * kadd[a]));
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (wbd != R(0)) atomicAdd(K + (ob + b) * nao + od + d, (double)(wbd * kbdd[b]));
        };
        R B[NAB];
        if constexpr (LD == 0) {
          wide_slice<LA, LB, LC, LD, R>(G, lane, c, 0, 0, 0, R(0), R(0), ab, B);
          term(0, B, kad[0], kbd[0]);
        } else if constexpr (LD == 1) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            wide_slice<LA, LB, LC, LD, R>(G, lane, c, ncart(LC) + raise_index(c, m, d), 0, 0, cd[d], R(0), ab, B);
            if constexpr (KEEP_D) {
              term(d, B, kad[d], kbd[d]);
            } else {
              R kadd[NA], kbdd[NB];
#pragma unroll
              for (int a = 0; a < NA; ++a) kadd[a] = R(0);
#pragma unroll
              for (int b = 0; b < NB; ++b) kbdd[b] = R(0);
              term(d, B, kadd, kbdd);
              if (want_k) flush_d(d, kadd, kbdd);
            }
          }
        } else {
          int d = 0;
#pragma unroll 1
          for (int i = 0; i < 3; ++i)
#pragma unroll 1
            for (int j = i; j < 3; ++j, ++d) {
              // (c, 1_i + 1_j): the axis order of the components is i <= j
              const int ci = raise_index(c, m, i), cj = raise_index(c, m, j);
              const int cij = raise_index(ci, m + (i > 0), j);
              const R ki = i == 0 ? cd[0] : (i == 1 ? cd[1] : cd[2]), kj = j == 0 ? cd[0] : (j == 1 ? cd[1] : cd[2]);
              wide_slice<LA, LB, LC, LD, R>(G, lane, c, ncart(LC) + cj, ncart(LC) + ci,
                                            ncart(LC) + ncart(LC + 1) + cij, kj, ki, ab, B);
              R kadd[NA], kbdd[NB];
#pragma unroll
              for (int a = 0; a < NA; ++a) kadd[a] = R(0);
#pragma unroll
              for (int b = 0; b < NB; ++b) kbdd[b] = R(0);
              term(d, B, kadd, kbdd);
              if (want_k) flush_d(d, kadd, kbdd);
            }
        }
        if (want_k) {
#pragma unroll
          for (int a = 0; a < NA; ++a)
            if (wac != R(0)) atomicAdd(K + (oa + a) * nao + oc + c, (double)(wac * kac[a]));
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (wbc != R(0)) atomicAdd(K + (ob + b) * nao + oc + c, (double)(wbc * kbc[b]));
        }
      }
    if constexpr (KEEP_D) {
      if (want_k)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
#pragma unroll
          for (int a = 0; a < NA; ++a)
            if (wad != R(0)) atomicAdd(K + (oa + a) * nao + od + d, (double)(wad * kad[d][a]));
#pragma unroll
          for (int b = 0; b < NB; ++b)
            if (wbd != R(0)) atomicAdd(K + (ob + b) * nao + od + d, (double)(wbd * kbd[d][b]));
        }
    }
    if (KEEP_AB && want_j) {
#pragma unroll
      for (int q = 0; q < (KEEP_AB ? NAB : 1); ++q) ja[q * 32] += (double)(wab * jab[q]);
    }
  }
}

// Adds this lane's running bra-block sums to J' and clears them (acc: lane's
// first value, values 32 apart; [0] the bra pair index or -1).
template <int LA, int LB>
__device__ __forceinline__ void wide_flush(const KernelArgs& A, double* acc) {
  constexpr int NA = ncart(LA), NB = ncart(LB);
  const int bra = (int)acc[0];
  if (bra < 0) return;
  const PairD pb = A.pairs[bra];
  const size_t nao = (size_t)A.nao, n2 = nao * nao;
  const int oa = A.shells[pb.a].off, ob = A.shells[pb.b].off;
  for (int d = 0; d < A.jk.ndens; ++d) {
    double* a = acc + ((size_t)1 + (size_t)d * NA * NB) * 32;
    double* J = A.jk.J + d * n2;
    for (int q = 0; q < NA * NB; ++q) {
      const double v = a[q * 32];
      if (v != 0.0) {
        atomicAdd(J + (oa + q / NB) * nao + ob + q % NB, v);
        a[q * 32] = 0.0;
      }
    }
  }
  acc[0] = -1.0;
}

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__(128, 2) wide_kernel(KernelArgs A) {
  using S = ClassShape<LA, LB, LC, LD>;
  using W = WideShape<LA, LB, LC, LD, R>;
  constexpr int NR = S::NR, WPG = W::WPG, TEAMS = 4 / WPG;
  __shared__ __align__(16) R s_tab[rys_smem<NR, R>(1)];
  __shared__ R s_roots[TEAMS][2 * 2 * NR * 32];
  __shared__ int s_bra[128], s_ket[128];
  __shared__ uint64_t s_mask[128];
  __shared__ unsigned long long s_base;
  const R* tab = rys_staged<NR, R>(1) ? s_tab : rys_global<NR, R>();
  stage_rys_table<NR, R, 1>(s_tab);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gt = warp / WPG, wi = warp % WPG;
  double* slot = A.scratch + (size_t)blockIdx.x * A.slot_doubles;
  R* G = reinterpret_cast<R*>(slot);
  const int nacc = 1 + A.jk.ndens * W::NAB;
  double* acc = slot + A.acc_offset + (size_t)warp * 32 * nacc + lane;
  for (int q = 1; q < nacc; ++q) acc[(size_t)q * 32] = 0.0;
  acc[0] = -1.0;
  QuartetCounters cnt;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_base = atomicAdd(A.work_counter, A.chunk);
    __syncthreads();
    const unsigned long long base = s_base;
    if (base >= A.task.total) break;
    const unsigned long long end = base + A.chunk < A.task.total ? base + A.chunk : A.task.total;
    for (unsigned long long b0 = base; b0 < end; b0 += 128) {
      // phase 1: the tables of four groups of 32 quartets
      for (int g = gt; g < 4; g += TEAMS) {
        const unsigned long long t = b0 + g * 32 + lane;
        TaskCursor cur;
        int pbi, pki, kpos;
        cursor_seek(A.task, t < end ? t : b0, cur);
        cursor_decode(A.task, t < end ? t : b0, cur, pbi, pki, kpos);
        PairD pb = A.pairs[pbi];
        PairD pk = A.pairs[pki];
        const Screen sc = screen_quartet(A, pb, pk);
        const bool keep = t < end && sc.keep;
        if (wi == 0) {
          s_bra[g * 32 + lane] = keep ? pbi : -1;
          s_ket[g * 32 + lane] = pki;
          s_mask[g * 32 + lane] = sc.dens;
          if (keep) cnt.add(sc, pb, pk, A.fp32);
        }
        if (!__any_sync(0xffffffffu, keep)) continue;
        // A pair can lose every primitive to the pair screen and still be
        // listed (a threshold of zero or less keeps every bound): there is no
        // primitive 0 to run along on, in the interleaved copies or in A.prims.
        // Such lanes take the pairs of the first lane that has primitives.
        const bool has = keep && pb.nprim > 0 && pk.nprim > 0;
        const unsigned any = __ballot_sync(0xffffffffu, has);
        const int src = any ? __ffs(any) - 1 : 0;
        const int sb = __shfl_sync(0xffffffffu, pb.prim_off, src), nb = __shfl_sync(0xffffffffu, pb.nprim, src);
        const int sk = __shfl_sync(0xffffffffu, pk.prim_off, src), nk = __shfl_sync(0xffffffffu, pk.nprim, src);
        const int sp = __shfl_sync(0xffffffffu, kpos, src);
        if (!has) {
          pb.prim_off = sb;
          pb.nprim = nb;
          pk.prim_off = sk;
          pk.nprim = nk;
          kpos = sp;
        }
        // no lane with primitives: no passes, the tables are zero
        const int npb = __reduce_max_sync(0xffffffffu, has ? pb.nprim : 0);
        const int npk = __reduce_max_sync(0xffffffffu, has ? pk.nprim : 0);
        R* Gg = G + (size_t)g * S::NG * 32;
        static_for<W::PPW>([&](auto p) {
          static_for<WPG>([&](auto v) {
            constexpr int blk = decltype(p)::value * WPG + decltype(v)::value;
            if (wi == decltype(v)::value)
              wide_rows<LA, LB, LC, LD, R, blk * W::ROWS>(A, tab, s_roots[gt], has, pb, pk, kpos, npb, npk, wi, gt,
                                                          lane, Gg);
          });
          // the next row block reuses the root buffers from the start
          wide_sync<WPG>(gt);
        });
      }
      __syncthreads();
      // phase 2: warp w finishes group w
      const int pbi = s_bra[threadIdx.x];
      if (pbi >= 0) {
        const PairD pb = A.pairs[pbi];
        const PairD pk = A.pairs[s_ket[threadIdx.x]];
        if ((int)acc[0] != pbi) {
          wide_flush<LA, LB>(A, acc);
          acc[0] = (double)pbi;
        }
        wide_post<LA, LB, LC, LD, R>(A, G + (size_t)warp * S::NG * 32, pb, pk, s_mask[threadIdx.x], acc, lane);
      }
      __syncthreads();
    }
  }
  wide_flush<LA, LB>(A, acc);
  __syncwarp();
  cnt.flush(A.counters);
}

// Classes with a kernel here: Cartesian work up to d shells, from the tables
// that exceed a lane's registers to the size where the recurrences, repeated
// for every row block, cost more than the teams' shared-memory reads: (22|11)
// takes 55 ns per quartet here and 52 on a team in FP64, 12 and 24 in FP32.
template <int LA, int LB, int LC, int LD, typename R>
__host__ __device__ constexpr bool wide_class() {
  return LA <= 2 && ClassShape<LA, LB, LC, LD>::NG > 81 &&
         ClassShape<LA, LB, LC, LD>::NG <= (sizeof(R) == 8 ? 256 : 300);
}

}  // namespace igpu
