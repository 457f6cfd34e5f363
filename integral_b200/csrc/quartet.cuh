// Shell-quartet kernels of the two-electron path.
//
// One launch handles one angular class (la,lb|lc,ld) in evaluation
// orientation (la >= lb, lc >= ld, bra class >= ket class) over a task list
// of (bra pair, ket pair) quartets that survived the Schwarz product screen.
//
// Phase 1 builds the contracted table G[e][f] = sum over primitive quartets
// and Rys roots of Ix[ex][fx] Iy[ey][fy] Iz[ez][fz] (the [e0|f0] integrals,
// e of degree la..la+lb on A, f of degree lc..lc+ld on C) by Rys quadrature
// with the vertical recurrence of src/engine/rys.rs:234-268.  Doing the
// horizontal recurrence once per shell quartet on the contracted table is the
// early-contraction scheme of the reference's OS/HGP engine
// (src/engine/os_eri.rs:1-12) applied to Rys 2D integrals.
//   TEAM == 1 : one thread per quartet, everything in registers.
//   TEAM >= 2 : a team of TEAM lanes per quartet; roots and the 3*nroots
//               per-axis tables are built cooperatively in shared memory and
//               every lane accumulates its own rows of G, of the bra or the
//               ket side (register tiles walked in passes, TeamSweep).
// The class's Rys table is staged in shared memory where rys_staged says so.
// Phase 2 (post.cuh) runs the horizontal recurrences, the Cartesian ->
// spherical transform and the mode-specific consumer on the team.
#pragma once
#include "device_common.cuh"
#include "post.cuh"
#include "post_thread.cuh"

namespace igpu {

template <int LA, int LB, int LC, int LD>
struct ClassShape {
  static constexpr int NE = LA + LB;
  static constexpr int NF = LC + LD;
  static constexpr int LT = NE + NF;
  static constexpr int NR = LT / 2 + 1;
  static constexpr int NEP = nrange(LA, NE);
  static constexpr int NFP = nrange(LC, NF);
  static constexpr int NG = NEP * NFP;
};

// Lanes per quartet: one thread while the whole G table fits in registers,
// otherwise the smallest team of 8, 16 or 32 lanes covering the rows (teams
// of 2 or 4 lanes measured slower: the per-primitive root and recurrence
// work is then spread over too few lanes).
__host__ __device__ constexpr int team_for(int nep, int nfp) {
  if (nep * nfp <= 81) return 1;
  if (nep <= 8) return 8;
  if (nep <= 16) return 16;
  return 32;
}
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr int team_size() {
  return team_for(nrange(LA, LA + LB), nrange(LC, LC + LD));
}

// Accumulators per lane and pass.
template <typename R>
__host__ __device__ constexpr int max_acc() { return sizeof(R) == 8 ? 64 : 96; }

// How a team sums its table.  Rows of one side (e of the bra, or f of the ket
// when `ket`) go one to a lane over groups of `gp` lanes, the other side's
// components are the columns; the team's T / gp groups take different primitive
// quartets of a round.  A pass holds rp row slots and fch columns per lane and
// recomputes the 2D tables.
struct TeamSweep {
  bool ket;
  int gp, rl, nchunk, fch, rp, npass;
  long cost;
};
// The cheapest of the lane-rows, by a count of SM cycles per root (times 32):
// a row slot loads 3 (N + 1) axis values, N the columns' side, once per column
// chunk, and spends two operations per column; a warp's FP64 shared load takes
// four times its multiply-add (likewise in FP32).  Rows on the bra side alone
// cost (33|21) 2.7 times as much: 74 rows of 21 loads for 16 columns against 16
// rows of 21 for 74.
__host__ __device__ constexpr TeamSweep team_sweep(int la, int lb, int lc, int ld, int T, int bp, int max_acc) {
  const int ne = la + lb, nf = lc + ld;
  const int nep = nrange(la, ne), nfp = nrange(lc, nf);
  TeamSweep best{};
  best.cost = 1L << 60;
  for (int side = 0; side < 2; ++side)
    for (int gp = T; gp >= 4; gp /= 2) {
      TeamSweep w{};
      w.ket = side == 1;
      const int rows = w.ket ? nfp : nep, cols = w.ket ? nep : nfp;
      const int loads = 3 * ((w.ket ? ne : nf) + 1);
      w.gp = gp;
      w.rl = (rows + gp - 1) / gp;
      w.nchunk = (cols + max_acc - 1) / max_acc;
      w.fch = (cols + w.nchunk - 1) / w.nchunk;
      int rp = w.nchunk > 1 ? 1 : max_acc / cols;
      rp = rp < w.rl ? rp : w.rl;
      rp = rp < 6 ? rp : 6;  // three offsets a row slot
      const int rpass = (w.rl + rp - 1) / rp;
      w.rp = (w.rl + rpass - 1) / rpass;
      w.npass = ((w.rl + w.rp - 1) / w.rp) * w.nchunk;
      const int groups = T / gp < bp ? T / gp : bp;
      w.cost = (long)w.npass * 10 * (ne + 1) * (nf + 1) + (long)(T / groups) * w.rl * (2 * w.nchunk * loads + cols);
      if (w.cost < best.cost) best = w;
    }
  return best;
}

template <int LA, int LB, int LC, int LD, typename R>
struct TeamShape {
  using S = ClassShape<LA, LB, LC, LD>;
  static constexpr int T = team_size<LA, LB, LC, LD>();
  // Primitive quartets set up per round: as many as fit a shared-memory
  // budget of 56 KB (FP32: 48) per 128-thread block (power of two, at most T).
  static constexpr int GTAB = (S::NE + 1) * (S::NF + 1);
  // x, w, g[3][NR][GTAB] of one primitive quartet, an odd number of values:
  // the lanes that build different quartets' tables store at this stride, and
  // an even one shares few banks (it was 96 for (22|10): every lane of a store
  // in one bank)
  static constexpr int PRIM_TAB = (2 * S::NR + 3 * S::NR * GTAB) | 1;
  static constexpr int BUDGET = ((sizeof(R) == 8 ? 56 : 48) * 1024 / 128) * (T == 1 ? 1 : T) / (int)sizeof(R);
  static constexpr int BP0 = BUDGET / PRIM_TAB;
  static constexpr int BP = BP0 >= T ? T : (BP0 >= 16 ? 16 : (BP0 >= 8 ? 8 : (BP0 >= 4 ? 4 : (BP0 >= 2 ? 2 : 1))));
  static constexpr int SUB = T / BP;  // lanes sharing one primitive quartet in a round
  static constexpr int SMEM_PER_TEAM = T == 1 ? 0 : BP * PRIM_TAB;  // in R units
  static constexpr TeamSweep SW = team_sweep(LA, LB, LC, LD, T < 4 ? 4 : T, BP, max_acc<R>());
  // Per-team shared memory: the primitive tables of phase 1, reused by the
  // post phase for the team's copy of the Cartesian block (16-byte multiple).
  // Classes whose copies would need more than 96 KB per 128-thread block
  // (f shells) read the block from the scratch slot instead.
  static constexpr int STAGE_BYTES0 = T == 1 ? 0 : jk_stage_doubles(LA, LB, LC, LD) * 8;
  static constexpr bool STAGE = T > 1 && (128 / T) * STAGE_BYTES0 <= 96 * 1024;
  static constexpr int STAGE_BYTES = STAGE ? STAGE_BYTES0 : 0;
  static constexpr int TAB_BYTES = SMEM_PER_TEAM * (int)sizeof(R);
  static constexpr int TEAM_BYTES = ((TAB_BYTES > STAGE_BYTES ? TAB_BYTES : STAGE_BYTES) + 15) / 16 * 16;
};

// Magnitude bound of one primitive quartet's contribution, |E_ab E_cd| times
// the Coulomb prefactor 2 pi^{5/2} / (p q sqrt(p + q)) (every Rys weight sum
// and Boys value is <= 1); evaluated in FP32 for the primitive screen of the
// FP32 launches.
__device__ __forceinline__ float prim_bound(const PrimPairF& b, const PrimPairF& k) {
  return fabsf(b.ez * k.ez) * rsqrtf(b.zeta + k.zeta);
}

// Largest primitive-quartet count the team screen compacts (16 x 16 primitive
// pairs); quartets with more run every primitive quartet.
constexpr int MAX_SURV = 256;

// ------------------------------------------------------------- TEAM == 1

template <int LA, int LB, int LC, int LD, typename R>
__device__ __forceinline__ void accumulate_thread(const KernelArgs& A, const R* tab, const PairD& pb,
                                                  const PairD& pk, int kpos, int sub, int split, R (&G)[ClassShape<LA, LB, LC, LD>::NG]) {
  using S = ClassShape<LA, LB, LC, LD>;
  constexpr int NE = S::NE, NF = S::NF, NR = S::NR;
#pragma unroll
  for (int q = 0; q < S::NG; ++q) G[q] = R(0);
  const float cut = (sizeof(R) == 4 && A.fp32) ? (float)A.prim_cut : 0.f;
  float acx = 0.f, acy = 0.f, acz = 0.f;
  if constexpr (sizeof(R) == 4) {
    const DevShell& sa = A.shells[pb.a];
    const DevShell& sc = A.shells[pk.a];
    acx = (float)(sa.cx - sc.cx);
    acy = (float)(sa.cy - sc.cy);
    acz = (float)(sa.cz - sc.cz);
  }
  for (int ip = sub; ip < pb.nprim; ip += split) {
    for (int kq = 0; kq < pk.nprim; ++kq) {
      QuartetHdr<R> h;
      if constexpr (sizeof(R) == 4) {
        const PrimPairF bp = A.primsf[pb.prim_off + ip];
        const PrimPairF kp = load_ket(A, pk.prim_off, kpos, kq, 0.f);
        if (cut > 0.f && prim_bound(bp, kp) < cut) continue;
        h = quartet_header_f(bp, kp, acx, acy, acz, A.omega);
      } else {
        h = quartet_header<R>(A.prims[pb.prim_off + ip], load_ket(A, pk.prim_off, kpos, kq, 0.0), A.omega);
      }
      R x[NR], w[NR];
      if constexpr (sizeof(R) == 4) {
        // FP32 launch: quadratures of five or more roots (high l) take
        // FP64 roots and weights
        if (roots_in_fp64<NR, R>(h.T)) {
          const double T64 = quartet_T64(A.prims[pb.prim_off + ip], A.prims[pk.prim_off + kq], A.omega);
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            double xd, wd;
            rys_root_one<NR, true>(rys_global<NR, double>(), T64, r, xd, wd);
            x[r] = R(xd);
            w[r] = R(wd);
          }
        } else {
          rys_roots_s<NR, !rys_staged<NR, R>(1)>(tab, h.T, x, w);
        }
      } else {
        rys_roots_s<NR, !rys_staged<NR, R>(1)>(tab, h.T, x, w);
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const R xr = x[r] * h.xs;
        const R cq = xr * h.qpq, cp = xr * h.ppq;
        const R b00 = xr * h.hpq;
        const R b10 = (R(1) - cq) * h.inv2p;
        const R b01 = (R(1) - cp) * h.inv2q;
        R gx[NE + 1][NF + 1], gy[NE + 1][NF + 1], gz[NE + 1][NF + 1];
        vrr_axis<NE, NF, R>(R(1), h.pax - cq * h.pqx, h.qcx + cp * h.pqx, b10, b01, b00, gx);
        vrr_axis<NE, NF, R>(R(1), h.pay - cq * h.pqy, h.qcy + cp * h.pqy, b10, b01, b00, gy);
        vrr_axis<NE, NF, R>(w[r] * h.pref, h.paz - cq * h.pqz, h.qcz + cp * h.pqz, b10, b01, b00, gz);
        static_for<S::NEP>([&](auto e) {
          constexpr int ex = range_x(LA, decltype(e)::value);
          constexpr int ey = range_y(LA, decltype(e)::value);
          constexpr int ez = range_z(LA, decltype(e)::value);
          static_for<S::NFP>([&](auto f) {
            constexpr int fx = range_x(LC, decltype(f)::value);
            constexpr int fy = range_y(LC, decltype(f)::value);
            constexpr int fz = range_z(LC, decltype(f)::value);
            G[decltype(e)::value * S::NFP + decltype(f)::value] += gx[ex][fx] * gy[ey][fy] * gz[ez][fz];
          });
        });
      }
    }
  }
}

// --------------------------------------------------------------- TEAM > 1

// One pass over all primitive quartets accumulating the columns
// [C0, C0 + fch) of this lane's rows in row slots [K0, K0 + rp).
template <int LA, int LB, int LC, int LD, typename R, int K0, int C0>
__device__ __forceinline__ void team_pass(const KernelArgs& A, const R* tab, const PairD& pb, const PairD& pk,
                                          R* sm, int lane, unsigned tmask, double* G, const unsigned short* surv,
                                          int npr, bool g32) {
  using S = ClassShape<LA, LB, LC, LD>;
  using TS = TeamShape<LA, LB, LC, LD, R>;
  constexpr TeamSweep SW = TS::SW;
  constexpr int NE = S::NE, NF = S::NF, NR = S::NR, T = TS::T;
  constexpr bool KET = SW.ket;
  constexpr int GP = SW.gp, GROUPS = T / GP;
  constexpr int NROW = KET ? S::NFP : S::NEP, NCOL = KET ? S::NEP : S::NFP;
  constexpr int RLO = KET ? LC : LA, CLO = KET ? LA : LC;  // lowest degrees
  constexpr int NL = KET ? NE : NF;                        // axis power of the columns' side
  constexpr int RST = KET ? 1 : NF + 1, CST = KET ? NF + 1 : 1;
  constexpr int CW = C0 + SW.fch <= NCOL ? SW.fch : NCOL - C0;
  constexpr int GT = TS::GTAB;
  constexpr int ROWS = SW.rl - K0 < SW.rp ? SW.rl - K0 : SW.rp;
  // unrolled, the loads of later roots are hoisted into registers that large
  // tiles do not leave
  constexpr int ROOTS_UNROLL = ROWS * CW * (int)sizeof(R) / 4 <= 40 ? NR : 1;
  const int gl = lane % GP, grp = lane / GP;
  R acc[ROWS][CW];
#pragma unroll
  for (int k = 0; k < ROWS; ++k)
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[k][c] = R(0);
  int rx0[ROWS], ry0[ROWS], rz0[ROWS];
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    const int row = gl + GP * (K0 + k);
    const int a = tri_below(RLO) + (row < NROW ? row : 0);
    rx0[k] = addr_lx(a) * RST;
    ry0[k] = addr_ly(a) * RST;
    rz0[k] = addr_lz(a) * RST;
  }
  // Rounds of BP primitive quartets: SUB lanes set up each one (roots, then
  // the 3*NR per-axis tables) into its shared-memory slot, then every lane
  // accumulates its rows over the whole round.
  constexpr int BP = TS::BP, SUB = TS::SUB, PT = TS::PRIM_TAB;
  const int npk = pk.nprim;
  const int myp = lane % BP;
  const int sub = lane / BP;
  float acx = 0.f, acy = 0.f, acz = 0.f;
  if constexpr (sizeof(R) == 4) {
    const DevShell& sa = A.shells[pb.a];
    const DevShell& sc = A.shells[pk.a];
    acx = (float)(sa.cx - sc.cx);
    acy = (float)(sa.cy - sc.cy);
    acz = (float)(sa.cz - sc.cz);
  }
  for (int base = 0; base < npr; base += BP) {
    const int nb = npr - base < BP ? npr - base : BP;
    const bool active = myp < nb;
    R* mys = sm + myp * PT;
    QuartetHdr<R> h;
    if (active) {
      const int pidx = surv ? (int)surv[base + myp] : base + myp;
      const int ip = pidx / npk, kq = pidx - ip * npk;
      if constexpr (sizeof(R) == 4)
        h = quartet_header_f(A.primsf[pb.prim_off + ip], A.primsf[pk.prim_off + kq], acx, acy, acz, A.omega);
      else
        h = quartet_header<R>(A.prims[pb.prim_off + ip], A.prims[pk.prim_off + kq], A.omega);
      // FP32 launch: quadratures of five or more roots (high l) take
      // FP64 roots and weights
      const bool r64 = roots_in_fp64<NR, R>(h.T);
      const double T64 = r64 ? quartet_T64(A.prims[pb.prim_off + ip], A.prims[pk.prim_off + kq], A.omega) : 0.0;
      for (int r = sub; r < NR; r += SUB) {
        R xr, wr;
        if (r64) {
          double xd, wd;
          rys_root_one<NR, true>(rys_global<NR, double>(), T64, r, xd, wd);
          xr = R(xd);
          wr = R(wd);
        } else {
          rys_root_one<NR, !rys_staged<NR, R>(T)>(tab, h.T, r, xr, wr);
        }
        mys[r] = xr * h.xs;
        mys[NR + r] = wr * h.pref;
      }
    }
    __syncwarp(tmask);
    if (active) {
      for (int t = sub; t < 3 * NR; t += SUB) {
        const int axis = t / NR, r = t - axis * NR;
        const R xr = mys[r];
        const R cq = xr * h.qpq, cp = xr * h.ppq;
        const R b00 = xr * h.hpq;
        const R b10 = (R(1) - cq) * h.inv2p;
        const R b01 = (R(1) - cp) * h.inv2q;
        const R pqa = axis == 0 ? h.pqx : (axis == 1 ? h.pqy : h.pqz);
        const R paa = axis == 0 ? h.pax : (axis == 1 ? h.pay : h.paz);
        const R qca = axis == 0 ? h.qcx : (axis == 1 ? h.qcy : h.qcz);
        R g[NE + 1][NF + 1];
        vrr_axis<NE, NF, R>(axis == 2 ? mys[NR + r] : R(1), paa - cq * pqa, qca + cp * pqa, b10, b01, b00, g);
        R* dst = mys + 2 * NR + (axis * NR + r) * GT;
#pragma unroll
        for (int n = 0; n <= NE; ++n)
#pragma unroll
          for (int m = 0; m <= NF; ++m) dst[n * (NF + 1) + m] = g[n][m];
      }
    }
    __syncwarp(tmask);
    for (int p = grp; p < nb; p += GROUPS) {
      const R* gt = sm + p * PT + 2 * NR;
#pragma unroll ROOTS_UNROLL
      for (int r = 0; r < NR; ++r) {
        const R* tx = gt + (0 * NR + r) * GT;
        const R* ty = gt + (1 * NR + r) * GT;
        const R* tz = gt + (2 * NR + r) * GT;
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
          if (SW.rl * GP > NROW && gl + GP * (K0 + k) >= NROW) continue;
          R rx[NL + 1], ry[NL + 1], rz[NL + 1];
#pragma unroll
          for (int m = 0; m <= NL; ++m) {
            rx[m] = tx[rx0[k] + m * CST];
            ry[m] = ty[ry0[k] + m * CST];
            rz[m] = tz[rz0[k] + m * CST];
          }
          static_for<CW>([&](auto c) {
            constexpr int ci = C0 + decltype(c)::value;
            constexpr int cx = range_x(CLO, ci), cy = range_y(CLO, ci), cz = range_z(CLO, ci);
            acc[k][decltype(c)::value] += rx[cx] * ry[cy] * rz[cz];
          });
        }
      }
    }
    __syncwarp(tmask);
  }
#pragma unroll
  for (int k = 0; k < ROWS; ++k) {
    // the groups' sums over their primitive quartets
#pragma unroll
    for (int o = GP; o < T; o *= 2)
#pragma unroll
      for (int c = 0; c < CW; ++c) acc[k][c] += __shfl_xor_sync(tmask, acc[k][c], o);
    const int row = gl + GP * (K0 + k);
    if (grp == 0 && row < NROW) {
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        const size_t at = KET ? (size_t)(C0 + c) * S::NFP + row : (size_t)row * S::NFP + C0 + c;
        if (sizeof(R) == 4 && g32)
          reinterpret_cast<float*>(G)[at] = (float)acc[k][c];  // FP32 post phase: the table stays in FP32
        else
          G[at] = (double)acc[k][c];
      }
    }
  }
}

template <int LA, int LB, int LC, int LD, typename R, int P>
__device__ __forceinline__ void team_passes(const KernelArgs& A, const R* tab, const PairD& pb, const PairD& pk,
                                            R* sm, int lane, unsigned tmask, double* G, const unsigned short* surv,
                                            int npr, bool g32) {
  using TS = TeamShape<LA, LB, LC, LD, R>;
  if constexpr (P < TS::SW.npass) {
    team_pass<LA, LB, LC, LD, R, P / TS::SW.nchunk * TS::SW.rp, P % TS::SW.nchunk * TS::SW.fch>(
        A, tab, pb, pk, sm, lane, tmask, G, surv, npr, g32);
    __syncwarp(tmask);
    team_passes<LA, LB, LC, LD, R, P + 1>(A, tab, pb, pk, sm, lane, tmask, G, surv, npr, g32);
  }
}

// Primitive screen of one quartet on a team of T lanes: the indices
// ip * nprim_ket + kq of the primitive quartets whose bound reaches `cut`,
// in order, into `list`; returns their count.
template <int T>
__device__ __forceinline__ int screen_prims(const KernelArgs& A, const PairD& pb, const PairD& pk, float cut,
                                            unsigned short* list, int lane, unsigned tmask) {
  const int npk = pk.nprim, npr = pb.nprim * npk;
  const int shift = ((threadIdx.x & 31) / T) * T;  // the team's first lane in the warp
  int n = 0;
  for (int b0 = 0; b0 < npr; b0 += T) {
    const int pidx = b0 + lane;
    bool keep = false;
    if (pidx < npr) {
      const int ip = pidx / npk, kq = pidx - ip * npk;
      keep = prim_bound(A.primsf[pb.prim_off + ip], A.primsf[pk.prim_off + kq]) >= cut;
    }
    const unsigned bal = (__ballot_sync(tmask, keep) & tmask) >> shift;
    if (keep) list[n + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)pidx;
    n += __popc(bal);
  }
  __syncwarp(tmask);
  return n;
}

// ------------------------------------------------------------------ kernel

// Minimum resident 128-thread blocks per SM (register budget): team
// classes 3 (168 registers; measured faster than the unconstrained
// allocation, whose unrolled J/K sums take up to 255), FP64 teams with an f or
// g bra 2 (their row tiles spill at 168: mixed J/K of 8 atoms with spherical f
// shells 198 against 181 ms), thread-per-quartet
// classes by the size of their register-resident G table (spilling large
// tables costs more than the occupancy gains).
#ifndef IGPU_FP32_TEAM_MINB
#define IGPU_FP32_TEAM_MINB 3
#endif
template <int LA, int LB, int LC, int LD, typename R>
__host__ __device__ constexpr int quartet_min_blocks() {
  return team_size<LA, LB, LC, LD>() > 1
             ? (sizeof(R) == 4 ? IGPU_FP32_TEAM_MINB : (LA >= 3 ? 2 : 3))
             : (ClassShape<LA, LB, LC, LD>::NG <= 9 ? 5 : (ClassShape<LA, LB, LC, LD>::NG <= 27 ? 3 : 1));
}

template <int LA, int LB, int LC, int LD, typename R>
__global__ void __launch_bounds__(128, quartet_min_blocks<LA, LB, LC, LD, R>()) quartet_kernel(KernelArgs A) {
  using S = ClassShape<LA, LB, LC, LD>;
  using TS = TeamShape<LA, LB, LC, LD, R>;
  constexpr int T = TS::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) R s_tab[rys_smem<S::NR, R>(T)];
  constexpr bool SCREEN = sizeof(R) == 4 && T > 1;
  __shared__ unsigned short s_surv[SCREEN ? (128 / T) * MAX_SURV : 1];
  // compile-time shaped J/K sums: every spherical class, Cartesian blocks up
  // to (ff|ff); the larger ones (Cartesian g shells) take the runtime sums
  constexpr bool CT_CART = ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD) <= 10000;
  __shared__ int s_hrr[T > 1 ? HrrTab<LA, LB, LC, LD>::TOTAL : 1];
  // the spherical post phase runs in the launch's arithmetic up to f shells,
  // in FP64 beyond
  using PX = std::conditional_t<CT_CART, R, double>;
  __shared__ PX s_c2s[T > 1 ? 4 * C2S_TILE : 1];
  if constexpr (T > 1) {
    build_hrr_tab<LA, LB, LC, LD>(s_hrr);
    stage_c2s<LA, LB, LC, LD, PX>(A, s_c2s);
  }
  const R* tab = rys_staged<S::NR, R>(T) ? s_tab : rys_global<S::NR, R>();
  stage_rys_table<S::NR, R, T>(s_tab);  // its __syncthreads also publishes s_hrr, s_c2s
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int team = tid / T;
  const int lane = threadIdx.x % T;
  const int nteams = (gridDim.x * blockDim.x) / T;
  const unsigned tmask = T == 32 ? 0xffffffffu : (((1u << T) - 1u) << ((threadIdx.x % 32) / T * T));
  unsigned char* team_smem = smem_raw + (size_t)(threadIdx.x / T) * TS::TEAM_BYTES;
  R* sm = reinterpret_cast<R*>(team_smem);
  double* stage = TS::STAGE ? reinterpret_cast<double*>(team_smem) : nullptr;
  R* stage_r = TS::STAGE ? reinterpret_cast<R*>(team_smem) : nullptr;
  // a team's slot, then its running bra-block accumulators; one-thread teams
  // keep a warp's accumulators together, interleaved by lane
  constexpr int AS = T == 1 ? 32 : 1;
  double* slot = A.scratch + (size_t)team * A.slot_doubles;
  double* acc = slot + A.acc_offset;
  if constexpr (T == 1) {
    double* warp = A.scratch + (size_t)(team & ~31) * A.slot_doubles;
    slot = warp + (size_t)(team & 31) * A.acc_offset;
    acc = warp + 32 * A.acc_offset + (team & 31);
  }
  QuartetCounters cnt;
  (void)nteams;
  const bool use_acc = A.mode == MODE_JK && A.jk.symmetric;
  if (use_acc) {
    // the scratch slot is shared with earlier launches: clear the running
    // bra-block accumulators before first use
    const int nacc = A.jk.ndens * ncart(LA) * ncart(LB);
    for (int q = lane; q < nacc; q += T) acc[(1 + q) * AS] = 0.0;
    if (lane == 0) acc[0] = -1.0;
  }
  __syncwarp(tmask);

  // Warps claim contiguous chunks of the task list; the teams of a warp
  // interleave inside a chunk, so consecutive quartets (same bra pair, same
  // primitive-pair count) stay on the same lanes.
  // In a one-thread launch of few quartets, `split` lanes share one: each sums
  // every split-th bra primitive, and the first finishes the quartet.
  const int split = T == 1 && A.split > 1 ? A.split : 1;
  const int TPW = 32 / (T * split);
  const int tw = (threadIdx.x & 31) / (T * split);
  const int sub = T == 1 ? (threadIdx.x & 31) % split : 0;
  for (;;) {
    unsigned long long base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(A.work_counter, A.chunk);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= A.task.total) break;
    const unsigned long long end = base + A.chunk < A.task.total ? base + A.chunk : A.task.total;
    TaskCursor cur;
    if (base + tw < end) cursor_seek(A.task, base + tw, cur);
    for (unsigned long long g = base + tw; g < end; g += TPW) {
      int pbi, pki, kpos;
      cursor_decode(A.task, g, cur, pbi, pki, kpos);
      const PairD pb = A.pairs[pbi];
      const PairD pk = A.pairs[pki];
      Screen sc = screen_quartet(A, pb, pk);
      if (!sc.keep) continue;
      if (lane == 0 && sub == 0) cnt.add(sc, pb, pk, A.fp32);
      if constexpr (T == 1) {
        R G[S::NG];
        accumulate_thread<LA, LB, LC, LD, R>(A, tab, pb, pk, kpos, sub, split, G);
        if (split > 1) {
          const unsigned group = ((1u << split) - 1u) << ((threadIdx.x & 31) - sub);  // split <= 16
#pragma unroll
          for (int q = 0; q < S::NG; ++q)
            for (int o = 1; o < split; o *= 2) G[q] += __shfl_xor_sync(group, G[q], o);
          if (sub) continue;
        }
        if (use_acc && A.kinds != 2) {
          // the post phase runs in the launch's arithmetic (FP32 launches
          // read the FP32 densities); J/K accumulate in FP64
          if (A.kinds == 0)
            thread_post_jk<LA, LB, LC, LD, false, R>(A, G, pb, pk, sc, acc, pbi);
          else
            thread_post_jk<LA, LB, LC, LD, true, R>(A, G, pb, pk, sc, acc, pbi);
          continue;
        }
#pragma unroll
        for (int q = 0; q < S::NG; ++q) slot[q] = (double)G[q];
      } else {
        const unsigned short* surv = nullptr;
        int npr = pb.nprim * pk.nprim;
        if constexpr (SCREEN) {
          if (A.fp32 && A.prim_cut > 0.0 && npr <= MAX_SURV) {
            unsigned short* list = s_surv + (threadIdx.x / T) * MAX_SURV;
            npr = screen_prims<T>(A, pb, pk, (float)A.prim_cut, list, lane, tmask);
            surv = list;
            if (npr == 0) continue;  // the whole quartet is below the screen
          }
        }
        team_passes<LA, LB, LC, LD, R, 0>(A, tab, pb, pk, sm, lane, tmask, slot, surv, npr,
                                          CT_CART && use_acc && A.kinds != 2);
      }
      __syncwarp(tmask);
      // in the launch's arithmetic; everything else, and the runtime sums, in
      // FP64
      if constexpr (T > 1 && CT_CART) {
        if (use_acc && A.kinds == 0) {
          post_quartet_jk_cart<LA, LB, LC, LD, T, R>(A, pb, pk, sc, slot, lane, tmask, pbi, stage_r, s_hrr);
          continue;
        }
      }
      if constexpr (T > 1) {
        if (use_acc && A.kinds == 1) {
          post_quartet_jk_sph<LA, LB, LC, LD, T, PX>(A, pb, pk, sc, slot, lane, tmask, pbi,
                                                     reinterpret_cast<PX*>(stage), s_hrr, s_c2s);
          continue;
        }
      }
      post_quartet<LA, LB, LC, LD, T>(A, s_hrr, pb, pk, sc, slot, lane, T, tmask, pbi, stage, acc, AS);
      __syncwarp(tmask);
    }
  }
  if (use_acc) flush_bra_acc(A, acc, AS, lane, T, tmask);
  cnt.flush(A.counters);
}

}  // namespace igpu
