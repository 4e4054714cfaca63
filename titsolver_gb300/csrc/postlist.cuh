// postlist.cuh - the post-integration stage (post.cuh) on the neighbour lists
// of the step (pairlist.cuh): the lists hold every pair within the support
// radius at the end of the step's stages as well (the last stage checks the
// displacement bound like the others and leaves the home state alone), so
// the stage needs no sort, no gather and no cell walk of its own, and small
// runs take several lanes per particle.
//
// Same sums and decisions as post.cuh, in FP64 in both forms.  GB300's FP64
// pipe bounds k_lpost_sums, so a pair costs about a third of the FP64
// operations of a direct transcription: the kernel gradient from the seeds
// of pairlist.cuh, the tank's constants and 1 / gamma applied once per
// particle, the symmetric L summed as such, and no quotients.
#pragma once

#include "pairlist.cuh"
#include "post.cuh"

namespace tg {

template<int D, int F>
struct ListPostArgs {
  ListArgs<D, F> L;   // pin, pos_in, dat_in: the state after the last stage
  PostArgs<D, F> P;   // the post-integration buffers and constants
};

// Target of a lane: slot i, lane tl of its team; false for walls' slots and
// past the end (uniform over a team).
template<int D, int F, int Team>
__device__ __forceinline__ bool list_target(const ListArgs<D, F>& A, int64_t& i, int& tl,
                                            uint32_t& id) {
  i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / Team;
  tl = Team == 1 ? 0 : static_cast<int>(threadIdx.x % Team);
  if (i >= A.S.n || *A.stop != 0u) return false;
  id = A.S.Y.id[i];
  return true;
}

// FP64 position of slot j.
template<int D, int F>
__device__ __forceinline__ void list_pos(const ListArgs<D, F>& A, uint32_t j, double* y) {
  if constexpr (F == TG_FP64) {
    load_pos(A.pos_in, j, y);
  } else {
#pragma unroll
    for (int k = 0; k < D; ++k) y[k] = __ldg(A.pin[k] + j);
  }
}

// The reference's predicate |x - y|^2 <= R^2: by the high words of a fused
// sum where they differ by more than one, else on the reference's rounding.
template<int D>
__device__ __forceinline__ bool list_near(const double* x, const double* y, double R2, double* d,
                                          double& s2) {
  s2 = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    d[k] = x[k] - y[k];
    s2 = k == 0 ? d[0] * d[0] : fma(d[k], d[k], s2);
  }
  const int hi = __double2hiint(s2), r2hi = __double2hiint(R2);
  if (hi < r2hi - 1) return true;
  if (hi > r2hi + 1) return false;
  double t[3];
  return dist2_exact<D>(x, y, t) <= R2;
}

// Calls fn(j) for the entries of slot i that lane tl takes.
template<int D, int F, int Team, class Fn>
__device__ __forceinline__ void list_entries(const ListArgs<D, F>& A, int64_t i, int tl, Fn&& fn) {
  const uint32_t m = A.cnt[i];
  const uint4* groups = reinterpret_cast<const uint4*>(A.list) + (list_at(i, 0, A.cap) >> 2);
  for (uint32_t p = 4 * tl; p < m; p += 4 * Team) {
    const uint4 g = groups[(p >> 2) * 32];
    const uint32_t js[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (uint32_t q = 0; q < 4u; ++q) {
      if (p + q < m) fn(js[q]);
    }
  }
}

template<int Team>
__device__ __forceinline__ double team_sum(double v) {
#pragma unroll
  for (int o = Team / 2; o > 0; o >>= 1) {
    v += __shfl_xor_sync(team_mask<Team>(), v, o, Team);
  }
  return v;
}

template<int D, int F, int K, int Team>
__global__ void __launch_bounds__(128) k_lpost_sums(ListPostArgs<D, F> Q) {
  const ListArgs<D, F>& A = Q.L;
  const PostArgs<D, F>& P = Q.P;
  int64_t i;
  int tl;
  uint32_t id;
  if (!list_target<D, F, Team>(A, i, tl, id)) return;
  const TankDev& T = A.S.tanks[tank_of_key(A.S.skey[i], A.S.tank_off, A.S.ntanks)];
  double rho_a, va[3];
  post_neighbour<D>(A.dat_in, static_cast<uint32_t>(i), T, rho_a, va);
  if (id & kWallBit) {
    if (tl == 0) {
      P.rho_raw[i] = rho_a;
      P.phi[i] = kPhiMax;
    }
    return;
  }
  double pa[3];
  list_pos(A, static_cast<uint32_t>(i), pa);
  constexpr int kSym = D * (D + 1) / 2;
  double N[D] = {}, Ls[kSym] = {}, gv[D * D] = {}, gr[D] = {};
  int32_t count = 0;
  const double tiny2 = 6.0554544523933395e-06 * 6.0554544523933395e-06;
  const double mhinv2 = -0.5 * T.hinv, R2 = T.radius2;
  list_entries<D, F, Team>(A, i, tl, [&](uint32_t j) {
    double y[3], d[3], s2;
    list_pos(A, j, y);
    if (!list_near<D>(pa, y, R2, d, s2)) return;
    ++count;
    if (s2 < tiny2) return;  // normalize(r_ab) is zero
    const auto b = load_dat(A.dat_in, j);
    double rho_b, ib;
    if constexpr (F == TG_FP64) {
      rho_b = b.rho;
      ib = b.invrho;
    } else {
      rho_b = T.rho0 + static_cast<double>(b.drho);
      ib = rcp_f64(rho_b);
    }
    const double y0 = rsqrt_seed(s2);
    const double r0 = s2 * y0;
    const double e = fma(-r0, y0, 1.0);
    const double ep = e * fma(e, 0.375, 0.5);
    const double r = fma(r0, ep, r0);
    double t = fma(r, mhinv2, 1.0);
    if (static_cast<unsigned>(__double2hiint(t)) > 0x3ff00000u) t = 0.0;
    double rinv = 0.0;
    if constexpr (!KernelPoly<K>::deriv_over_q) rinv = fma(y0, ep, y0);
    const double c = ib * list_g<K>(t, KernelPoly<K>::deriv_over_q ? 0.0 : r * T.hinv, rinv);
    const double vb[3] = {b.vx, b.vy, b.vz};
    const double drb = rho_b - rho_a;
    double w[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      w[k] = c * d[k];
      N[k] += w[k];
      gr[k] = fma(drb, w[k], gr[k]);
    }
    int q = 0;
#pragma unroll
    for (int a2 = 0; a2 < D; ++a2) {
      const double dva = vb[a2] - va[a2];
#pragma unroll
      for (int b2 = 0; b2 < D; ++b2) gv[a2 * D + b2] = fma(dva, w[b2], gv[a2 * D + b2]);
#pragma unroll
      for (int b2 = a2; b2 < D; ++b2, ++q) Ls[q] = fma(d[a2], w[b2], Ls[q]);
    }
  });
  if constexpr (Team > 1) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      N[k] = team_sum<Team>(N[k]);
      gr[k] = team_sum<Team>(gr[k]);
    }
#pragma unroll
    for (int k = 0; k < kSym; ++k) Ls[k] = team_sum<Team>(Ls[k]);
#pragma unroll
    for (int k = 0; k < D * D; ++k) gv[k] = team_sum<Team>(gv[k]);
#pragma unroll
    for (int o = Team / 2; o > 0; o >>= 1) {
      count += __shfl_xor_sync(team_mask<Team>(), count, o, Team);
    }
    if (tl != 0) return;
  }
  // The constants of m / rho_b grad W, and 1 / gamma; face boundaries
  // (fluid_equations.hpp:335-349) add their terms, already divided by it.
  const FaceArgs& fc = A.S.fc;
  const double s = fc.on ? T.list_s / fc.gamma[i] : T.list_s;
  double L[D * D];
  int q = 0;
#pragma unroll
  for (int a2 = 0; a2 < D; ++a2) {
    N[a2] *= s;
    gr[a2] *= s;
#pragma unroll
    for (int b2 = 0; b2 < D; ++b2) gv[a2 * D + b2] *= s;
#pragma unroll
    for (int b2 = a2; b2 < D; ++b2, ++q) L[a2 * D + b2] = L[b2 * D + a2] = -s * Ls[q];
  }
  if (fc.on) {
    int c[3] = {0, 0, 0};
    cell_from_key<D>(T, A.curkey[i], c);
    const uint32_t gcell = global_cell<D>(T, c);
    if (fc.cell_start[gcell + 1] > fc.cell_start[gcell]) {
      const double* f0 = fc.post_face + kPostFaceSums<D> * static_cast<size_t>(i);
#pragma unroll
      for (int k = 0; k < D; ++k) {
        N[k] += f0[k];
        gr[k] += f0[D + 2 * D * D + k];
      }
#pragma unroll
      for (int k = 0; k < D * D; ++k) {
        L[k] += f0[D + k];
        gv[k] += f0[D + D * D + k];
      }
    }
  }
  // The entries do not hold the particle itself, which the reference counts.
  post_store_sums<D, F>(P, i, N, L, gv, gr, count + 1);
}

template<int D, int F, int Team>
__global__ void __launch_bounds__(128) k_lpost_phi(ListPostArgs<D, F> Q) {
  const ListArgs<D, F>& A = Q.L;
  const PostArgs<D, F>& P = Q.P;
  int64_t i;
  int tl;
  uint32_t id;
  if (!list_target<D, F, Team>(A, i, tl, id) || (id & kWallBit)) return;
  const TankDev& T = A.S.tanks[tank_of_key(A.S.skey[i], A.S.tank_off, A.S.ntanks)];
  double pa[3], Na[3];
  list_pos(A, static_cast<uint32_t>(i), pa);
#pragma unroll
  for (int k = 0; k < D; ++k) Na[k] = P.N[i * D + k];
  const uint32_t m = A.cnt[i];
  const uint4* groups = reinterpret_cast<const uint4*>(A.list) + (list_at(i, 0, A.cap) >> 2);
  bool visible = false;
  // Team-uniform trips: any lane's hit ends the search.
  for (uint32_t p0 = 0; p0 < m; p0 += 4 * Team) {
    const uint32_t p = p0 + 4u * tl;
    if (p < m) {
      const uint4 g = groups[(p >> 2) * 32];
      const uint32_t js[4] = {g.x, g.y, g.z, g.w};
      for (uint32_t q = 0; q < 4u && p + q < m && !visible; ++q) {
        double y[3], d[3];
        list_pos(A, js[q], y);
        const double s2 = dist2_exact<D>(pa, y, d);
        if (s2 > T.radius2) continue;
        const double na = dot_rn(Na, d, D);
        visible = na > 0.0 && __dmul_rn(na, na) >= __dmul_rn(P.cos2_fov, s2);
      }
    }
    if constexpr (Team > 1) {
      visible = __any_sync(team_mask<Team>(), visible);
    }
    if (visible) break;
  }
  if (tl != 0) return;
  const int cutoff = D == 2 ? 8 : 26;
  P.phi[i] = visible && P.count[i] > cutoff ? kPhiMax : kPhiMin;
}

template<int D, int F, int K, int Team>
__global__ void __launch_bounds__(128) k_lpost_near(ListPostArgs<D, F> Q) {
  const ListArgs<D, F>& A = Q.L;
  const PostArgs<D, F>& P = Q.P;
  int64_t i;
  int tl;
  uint32_t id;
  if (!list_target<D, F, Team>(A, i, tl, id)) return;
  const double phi = P.phi[i];
  if ((id & kWallBit) || !bits_eq(phi, kPhiMax)) {
    if (tl == 0) P.phi2[i] = phi;
    return;
  }
  const TankDev& T = A.S.tanks[tank_of_key(A.S.skey[i], A.S.tank_off, A.S.ntanks)];
  double pa[3];
  list_pos(A, static_cast<uint32_t>(i), pa);
  // The closest surface neighbour, the lowest upload index on ties (the
  // reference takes the first minimum in index order); none: id ~0.
  uint32_t best = 0, best_id = 0xffffffffu;
  double best_d2 = __longlong_as_double(0x7ff0000000000000ll);
  list_entries<D, F, Team>(A, i, tl, [&](uint32_t j) {
    if (!bits_eq(P.phi[j], kPhiMin)) return;
    double y[3], d[3];
    list_pos(A, j, y);
    const double s2 = dist2_exact<D>(pa, y, d);
    if (s2 > T.radius2) return;
    const uint32_t jid = A.S.Y.id[j] & kIdMask;
    if (s2 < best_d2 || (s2 == best_d2 && jid < best_id)) {
      best = j;
      best_id = jid;
      best_d2 = s2;
    }
  });
#pragma unroll
  for (int o = Team / 2; o > 0; o >>= 1) {
    const unsigned mask = team_mask<Team>();
    const double d2 = __shfl_xor_sync(mask, best_d2, o, Team);
    const uint32_t j = __shfl_xor_sync(mask, best, o, Team);
    const uint32_t jid = __shfl_xor_sync(mask, best_id, o, Team);
    if (d2 < best_d2 || (d2 == best_d2 && jid < best_id)) {
      best = j;
      best_id = jid;
      best_d2 = d2;
    }
  }
  if (tl != 0) return;
  double out = phi;
  if (best_id != 0xffffffffu) {
    double y[3], d[3], Nb[3];
    list_pos(A, best, y);
#pragma unroll
    for (int k = 0; k < D; ++k) {
      d[k] = __dsub_rn(pa[k], y[k]);
      Nb[k] = P.N[static_cast<size_t>(best) * D + k];
    }
    out = phi * (fabs(dot_rn(Nb, d, D)) / (KernelPoly<K>::unit_radius * T.h));
  }
  P.phi2[i] = out;
}

// The home state: far particles shifted, with the keys of their positions.
template<int D, int F>
__global__ void __launch_bounds__(128) k_lpost_shift(ListPostArgs<D, F> Q) {
  using R = typename StageArgs<D, F>::R;
  const ListArgs<D, F>& A = Q.L;
  const StageArgs<D, F>& S = A.S;
  int64_t i;
  int tl;
  uint32_t id;
  if (!list_target<D, F, 1>(A, i, tl, id)) return;
  if (id & kWallBit) {
    list_commit_wall(A, i, id);
    return;
  }
  const uint32_t key = S.skey[i];
  const TankDev& T = S.tanks[tank_of_key(key, S.tank_off, S.ntanks)];
  double p[3] = {0.0, 0.0, 0.0}, v[3], rho;
  list_pos(A, static_cast<uint32_t>(i), p);
  post_neighbour<D>(A.dat_in, static_cast<uint32_t>(i), T, rho, v);
  post_apply_shift<D, F>(Q.P, i, T, p, v, rho);
  Q.P.rho_raw[i] = rho;
  R dv[3] = {R(0), R(0), R(0)};
#pragma unroll
  for (int k = 0; k < D; ++k) dv[k] = S.Y.dv[k][i];
  post_commit<D, F>(S, i, id, key, T, p, v, rho, dv, S.Y.drho[i]);
}

template<int D, int F, int K, int Team>
__global__ void __launch_bounds__(128) k_lpost_fs(ListPostArgs<D, F> Q) {
  const ListArgs<D, F>& A = Q.L;
  const PostArgs<D, F>& P = Q.P;
  const StageArgs<D, F>& S = A.S;
  int64_t i;
  int tl;
  uint32_t id;
  if (!list_target<D, F, Team>(A, i, tl, id)) return;
  if ((id & kWallBit) || bits_eq(P.phi2[i], kPhiMax)) return;
  const TankDev& T = S.tanks[tank_of_key(S.X.pkey[i], S.tank_off, S.ntanks)];
  double pa[3], xa[3];
  list_pos(A, static_cast<uint32_t>(i), pa);  // prepare positions: the neighbour set
#pragma unroll
  for (int k = 0; k < D; ++k) xa[k] = S.X.pos[k][i];  // shifted: the kernel values
  double alpha = 0.0, rho_t = 0.0;
  const auto pair = [&](uint32_t j) {
    double y[3], d[3], s2;
    list_pos(A, j, y);
    if (!list_near<D>(pa, y, T.radius2, d, s2)) return;
    double x2 = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const double x = xa[k] - S.X.pos[k][j];
      x2 = fma(x, x, x2);
    }
    const double W = KernelPoly<K>::value(T.hinv * sqrt_f64(x2));
    alpha = fma(rcp_f64(P.rho_raw[j]), W, alpha);
    rho_t += W;
  };
  if (tl == 0) pair(static_cast<uint32_t>(i));  // the list leaves out the particle itself
  list_entries<D, F, Team>(A, i, tl, pair);
  if constexpr (Team > 1) {
    alpha = team_sum<Team>(alpha);
    rho_t = team_sum<Team>(rho_t);
    if (tl != 0) return;
  }
  const double mw = T.m * T.w;
  post_commit_density<D, F>(P, S, i, T, alpha * mw, rho_t * mw);
}

}  // namespace tg
