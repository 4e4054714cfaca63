// density.cuh - summation density over a point cloud
// (fluid_equations.hpp:498-502 form, self included): rho_a = sum_b m W_ab,
// with neighbour counts and order-independent hashes of the neighbour sets.
//   FP64 positions: FP64 predicate and sum.
//   FP32 positions: the positions are rounded to float once; predicate and
//   kernel in FP32, compensated sum.
#pragma once

#include "pairlist.cuh"

namespace tg {

template<int D>
struct CloudArgs {
  const void* pos;  // Pos64_* or Pos32_* absolute positions, cell order
  // One array per axis: FP64 form tank-local FP32 coordinates, FP32 form the
  // offsets from the cell corner.
  const float* local[3];
  const uint64_t* hash;  // FP32 form: hash of every point's id, cell order
  const uint32_t* id;
  const uint32_t* skey;  // sorted keys
  const uint32_t* cell_start;
  const TankDev* tanks;
  const uint32_t* tank_off;
  int ntanks;
  int64_t n;
  int k;             // cells per radius; 0: the tank's own (TankDev::pad)
  double* rho;       // by upload id
  int32_t* counts;   // by upload id
  uint64_t* hashes;  // by upload id
  const uint32_t* id_base;
};

// Records of the cloud in cell order: positions, ids, and what the form's
// pass reads beside them (local coordinates, or hashes).
template<int D, bool F32>
__global__ void __launch_bounds__(256)
    k_cloud_records(const double* __restrict__ px, const double* __restrict__ py,
                    const double* __restrict__ pz, const uint32_t* __restrict__ id_in,
                    const uint32_t* __restrict__ perm, CloudArgs<D> A, void* rec,
                    uint32_t* __restrict__ id_out, float* lx, float* ly, float* lz,
                    uint64_t* __restrict__ hash) {
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= A.n) return;
  const uint32_t s = perm[j];
  const double x = px[s], y = py[s], z = D == 3 ? pz[s] : 0.0;
  const uint32_t id = id_in[s];
  id_out[j] = id;
  const uint32_t tk = tank_of_key(A.skey[j], A.tank_off, A.ntanks);
  if constexpr (F32) {
    if constexpr (D == 2) {
      static_cast<Pos32_2*>(rec)[j] = Pos32_2{float(x), float(y)};
    } else {
      static_cast<Pos32_3*>(rec)[j] = Pos32_3{float(x), float(y), float(z), 0.f};
    }
    const TankDev& T = A.tanks[tk];
    const double p[3] = {float(x), float(y), float(z)};
    int c[3] = {0, 0, 0};
    float o[3] = {0.f, 0.f, 0.f};
    cell_from_key<D>(T, A.skey[j], c);
    cell_offset<D>(T, c, p, o);
    lx[j] = o[0];
    ly[j] = o[1];
    if constexpr (D == 3) lz[j] = o[2];
    hash[j] = splitmix64(static_cast<uint64_t>((id & kIdMask) - A.id_base[tk]) + 1u);
  } else {
    const TankDev& T = A.tanks[tk];
    lx[j] = __double2float_rn(x - T.lo[0]);
    ly[j] = __double2float_rn(y - T.lo[1]);
    if constexpr (D == 2) {
      static_cast<Pos64_2*>(rec)[j] = Pos64_2{x, y};
    } else {
      static_cast<Pos64_3*>(rec)[j] = Pos64_3{x, y, z, 0.0};
      lz[j] = __double2float_rn(z - T.lo[2]);
    }
  }
}

// f(q) at s2 = |r_ab|^2 in FP64.  The Wendland polynomials take q = 2 - 2 t
// with t = 1 - q/2 cut to [0, 1], which is 0 also for a NaN.
template<int K>
__device__ __forceinline__ double density_value(double s2, double hinv) {
  const double r = sqrt_f64(s2);
  if constexpr (KernelPoly<K>::deriv_over_q) {
    double t = fma(r, -0.5 * hinv, 1.0);
    if (static_cast<unsigned>(__double2hiint(t)) > 0x3ff00000u) t = 0.0;
    const double q = fma(-2.0, t, 2.0);
    const double t2 = t * t;
    if constexpr (K == TG_KERNEL_WENDLAND_C2) {
      return fma(2.0, q, 1.0) * (t2 * t2);
    } else if constexpr (K == TG_KERNEL_WENDLAND_C4) {
      return fma(fma(35.0 / 12.0, q, 3.0), q, 1.0) * (t2 * t2 * t2);
    } else {
      const double t4 = t2 * t2;
      return fma(fma(fma(4.0, q, 6.25), q, 4.0), q, 1.0) * (t4 * t4);
    }
  } else {
    return KernelPoly<K>::value(r * hinv);
  }
}

constexpr int kDensityBlock = 128;

// FP64 form, one warp per point.  GB300's FP64 pipe takes 16 cycles for an
// instruction of a warp, however few of its lanes need it, so the candidates
// are culled on FP32 coordinates first (list_slack_f covers their rounding)
// and those left gather in a queue of the warp, which is emptied 32 at a
// time: the FP64 work runs on full warps.  Near the grid's border, where
// clamped points may be anywhere, nothing is culled.  (60,001 points, 3D:
// one thread per point 4.69 ms, with queues per thread 3.59 ms, where FP64
// instructions ran with 10 of 32 lanes active.)
template<int D, int K>
__global__ void __launch_bounds__(kDensityBlock) k_density64(CloudArgs<D> A) {
  __shared__ uint32_t s_queue[kDensityBlock / 32][64];
  uint32_t* queue = s_queue[threadIdx.x >> 5];
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (i >= A.n) return;  // whole warps
  const uint32_t key = A.skey[i];
  const uint32_t tk = tank_of_key(key, A.tank_off, A.ntanks);
  const TankDev& T = A.tanks[tk];
  const int k = A.k > 0 ? A.k : static_cast<int>(T.pad);
  const uint32_t base = A.id_base[tk];
  int c[3] = {0, 0, 0};
  cell_from_key<D>(T, key, c);
  using P = std::conditional_t<D == 2, Pos64_2, Pos64_3>;
  const P* pr = static_cast<const P*>(A.pos);
  double pa[3] = {0.0, 0.0, 0.0};
  load_pos(pr, static_cast<uint32_t>(i), pa);
  // FP32 geometry only where its squares are ordinary numbers, and row clips
  // only where the offsets from the cell corner are small.
  float xl[3] = {0.f, 0.f, 0.f}, oc[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int a = 0; a < D; ++a) {
    xl[a] = A.local[a][i];
    oc[a] = xl[a] - static_cast<float>(c[a]) * T.cs_f;
  }
  const bool cull = T.cull_r2_f >= 1e-30f && T.cull_r2_f <= 1e30f &&
                    T.list_slack_f <= T.R_f && target_band<D>(T, c, k).lo > 0.f;
  const float RL = T.R_f + T.list_slack_f;
  const float RL2 = cull ? RL * RL : __int_as_float(0x7f800000);
  const double R2 = T.radius2, hinv = T.hinv;
  const int r2hi = __double2hiint(R2);
  int32_t cnt = 0;
  uint64_t hs = 0;
  double acc = 0.0;
  int nq = 0;
  const auto entry = [&](uint32_t j) {
    double pb[3], d[3];
    load_pos(pr, j, pb);
    double s2 = 0.0;
#pragma unroll
    for (int a = 0; a < D; ++a) {
      d[a] = pa[a] - pb[a];
      s2 = a == 0 ? d[0] * d[0] : fma(d[a], d[a], s2);
    }
    // The reference's predicate, not |r_ab|^2 > R^2 (so a NaN stays in): by
    // the high words, on its own rounding where those are within one.
    const int hi = __double2hiint(s2);
    if (hi > r2hi + 1 && hi <= 0x7ff00000) return;
    if (hi >= r2hi - 1 && hi <= r2hi + 1 && dist2_exact<D>(pa, pb, d) > R2) return;
    acc += density_value<K>(s2, hinv);
    ++cnt;
    hs += splitmix64(static_cast<uint64_t>((A.id[j] & kIdMask) - base) + 1u);
  };
  for_shared_rows<D, 32>(T, c, k, A.cell_start, lane, 0xffffffffu, cull ? oc : nullptr, RL2,
                         [&](uint32_t s, uint32_t e) {
    for (uint32_t j0 = s; j0 < e; j0 += 32) {
      const uint32_t j = j0 + lane;
      bool in = j < e;
      if (in) {
        const float dx = xl[0] - __ldg(A.local[0] + j);
        const float dy = xl[1] - __ldg(A.local[1] + j);
        float s2 = dx * dx + dy * dy;
        if constexpr (D == 3) {
          const float dz = xl[2] - __ldg(A.local[2] + j);
          s2 = fmaf(dz, dz, s2);
        }
        in = !(s2 > RL2);
      }
      const unsigned hit = __ballot_sync(0xffffffffu, in);
      if (in) queue[nq + __popc(hit & ((1u << lane) - 1u))] = j;
      nq += __popc(hit);
      __syncwarp();
      if (nq >= 32) {
        nq -= 32;
        const uint32_t q = queue[nq + lane];
        __syncwarp();
        entry(q);
      }
    }
  });
  if (lane < nq) entry(queue[lane]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    hs += __shfl_xor_sync(0xffffffffu, hs, o);
  }
  if (lane != 0) return;
  const uint32_t id = A.id[i] & kIdMask;
  if (A.rho != nullptr) A.rho[id] = T.w * T.m * acc;
  if (A.counts != nullptr) A.counts[id] = cnt;
  if (A.hashes != nullptr) A.hashes[id] = hs;
}

// FP32 form, one thread per point: the walk over the candidates bounds it
// (about a thousand per point in the clusters, 75% of the issue slots).  The
// predicate is the reference's on the rounded positions, uncontracted; the
// hashes and the offsets from the cell corner are made once per point with
// the records.  Measured on 4M points (3D, 70% lattice, 30% in clusters), us
// per call: 9587 with the hash made per pair, IEEE square roots and FP64
// offsets per thread; this form 6474; 8 lanes per point sharing the rows
// 11992; every candidate's value without a branch 9533; warps that lie in one
// cell walking together with a queue per lane 12408.  Relative L2 error
// against 64 bits at 4M, 125,236 and 13,838 points: 2.7e-8, 2.7e-8, 2.8e-8
// (the rounding of the results to FP32) against 4.8e-8, 6.3e-8, 8.6e-8 with
// 1/h in one word, the weight in FP32 and IEEE square roots.
template<int D, int K>
__global__ void __launch_bounds__(kDensityBlock) k_density32(CloudArgs<D> A) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  const uint32_t key = A.skey[i];
  const TankDev& T = A.tanks[tank_of_key(key, A.tank_off, A.ntanks)];
  int c[3] = {0, 0, 0};
  cell_from_key<D>(T, key, c);
  using P = std::conditional_t<D == 2, Pos32_2, Pos32_3>;
  const P* pr = static_cast<const P*>(A.pos);
  float pa[3] = {0.f, 0.f, 0.f}, oc[3] = {0.f, 0.f, 0.f};
  load_pos(pr, static_cast<uint32_t>(i), pa);
#pragma unroll
  for (int a = 0; a < D; ++a) oc[a] = A.local[a][i];
  // 1/h in two words: its rounding would move every q the same way, and the
  // sum keeps that.
  const float R2 = T.radius2_f, hinv = T.hinv_f;
  const float hinv_lo = static_cast<float>(T.hinv - static_cast<double>(hinv));
  int32_t cnt = 0;
  uint64_t hs = 0;
  Kahan acc;
  for_cells<D, false>(T, c, A.k, A.cell_start, [&](uint32_t s, uint32_t e, int, int, int) {
    for (uint32_t j = s; j < e; ++j) {
      float pb[3], d[3];
      load_pos(pr, j, pb);
      const float s2 = dist2_exact<D>(pa, pb, d);
      if (s2 > R2) continue;
      const float r = sqrt_newton(s2);
      acc.add(KernelPoly<K>::value(fmaf(r, hinv, r * hinv_lo)));
      ++cnt;
      hs += __ldg(A.hash + j);
    }
  }, oc);
  const uint32_t id = A.id[i] & kIdMask;
  if (A.rho != nullptr) {
    A.rho[id] = T.w * T.m * (static_cast<double>(acc.s) - static_cast<double>(acc.c));
  }
  if (A.counts != nullptr) A.counts[id] = cnt;
  if (A.hashes != nullptr) A.hashes[id] = hs;
}

}  // namespace tg
