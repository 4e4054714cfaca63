// pairlist.cuh - one time step on neighbour lists.
//
// The SSPRK stages of a step move a particle by a few percent of the support
// radius R at most, so one neighbour list per particle, built at the step's
// start from a single sort and taken a little wider than R, holds every
// neighbour of all the stages.  A step then runs as
//   sort + cell table (sort.cu, sort_near.cu)
//   k_list_gather   state into cell order, records, dt and |v| reductions
//   k_list_build    lists of the fluid particles and of the walls near fluid
//   per stage: k_list_walls (wall extrapolation), k_list_forces (pair sums,
//   update, and the records of the next stage)
// in place of a sort, a reorder and a cell walk per stage.
//
// Validity.  A list of radius R + 2 delta holds every pair that comes within
// R while no particle is more than delta from where the step began.  delta
// is dt max|v| of the tank (the first stage moves by exactly dt v) plus a
// margin for the accelerations, and every stage checks it: a particle beyond
// delta, or a list past its capacity, raises *stop.  The last stage and all
// later kernels then leave the home state as the step found it, and the host
// repeats the step, or its chain, with a sort per stage and goes on with lists
// (tg_step, listpolicy.cuh).  Nothing is approximated:
// every entry's |r_ab| is taken anew in every stage, and an entry beyond R
// adds nothing: by the predicate |r_ab| <= R, or, in the compensated form
// with a Wendland kernel, by the kernel itself, whose clamped factor
// max(1 - |r_ab| / R, 0) makes each of its terms an exact zero there.
//
// Chains.  The steps within one tg_step call share the lists (kListChain at
// a time; in the plain form only those of small runs, whose sorts and builds
// are chains of short launches): the lists are as much wider, and the first
// step's last stage hands its state on in the records.  The home state
// is written by the chain's last step, so a stop repeats the whole chain.
//
// Positions of the compensated form are 32-bit fixed point, in units of
// 2^-28 cells modulo 2^32: a difference is exact while it is below 8 cells,
// whatever the cells of the two particles are, so no cell offsets enter the
// pair loop and r_ab keeps the relative precision of FP32.  (A listed pair is
// within R + 2 delta when the lists are built and each of the two then moves
// delta <= R / 4 at most: R + 4 delta <= 2 R <= 6 cells at 3 cells per radius.)  The unit stays in the pair
// loop; the constants absorb it.
#pragma once

#include "engine.cuh"
#include "fluid.cuh"

namespace tg {

// Fixed point of a coordinate: 2^52 + 2^51 puts the integer part of
// (p - lo) * inv_unit into the low mantissa bits.
__device__ __forceinline__ int fixed_coord(double p, double lo, double inv_unit) {
  return __double2loint(fma(p - lo, inv_unit, 6755399441055744.0));
}

template<int D, int F>
struct ListArgs {
  StageArgs<D, F> S;      // X home state, Y.pos / Y.id the step start in cell
                          // order, Udst the start's velocity and density
  using R = typename StageArgs<D, F>::R;
  using DatRec = typename Layout<D, F>::DatRec;
  // FP64 positions; the compensated form's sit in its data records.
  using PosRec = std::conditional_t<F == TG_FP64, typename Layout<D, F>::PosRec, int4>;
  const PosRec* pos_in;
  PosRec* pos_out;
  DatRec* dat_in;         // the wall pass writes the walls' entries
  DatRec* dat_out;
  double* pin[3];         // FP64 positions of this stage
  double* pout[3];
  float4* lrec;           // tank-local FP32 positions (w: sign = wall)
  uint32_t* list;         // tiles of 32 slots: 4-entry groups, group-major
  uint32_t* cnt;          // entries of each slot
  uint32_t* curkey;       // current cell keys (face walls), or null
  unsigned* vmax;         // per tank: max |v| as float bits
  uint32_t* stop;
  int64_t n_walls;
  int cap;                // entries per slot, a multiple of 4
  float margin;           // acceleration share of delta, in R
  int first, last;
  // Chains: steps that share the lists.  dt_build: the first step's dt (S.dt:
  // the present step's).  carry: the last stage of a step that another one
  // follows, which leaves its state as that step's start (positions in pout,
  // velocity and density in next) and folds its time step into dt_next.
  int chain, carry;
  const double* dt_build;
  double* dt_next;
  StartBuf<R> next;
  float* travel;          // path since the build up to the present step's
                          // start, or null in the first step
  float* travel_out;
  int post;               // the last stage of a step with post-integration:
                          // keeps the rates in Y and leaves X to that
  double w0;              // 1 - S.w_new, and both in the form's type
  R w0r, wr;
};

// Entry p of slot s.
__device__ __forceinline__ size_t list_at(int64_t s, uint32_t p, int cap) {
  return static_cast<size_t>(s >> 5) * (static_cast<size_t>(cap) << 5) +
         (static_cast<size_t>(p >> 2) << 7) + ((s & 31) << 2) + (p & 3u);
}

// The displacement bound of a tank's particles in this step.
template<int D, int F>
__device__ __forceinline__ float list_delta(const ListArgs<D, F>& A, const TankDev& T,
                                            uint32_t tk) {
  const float d = static_cast<float>(A.chain) *
                  (static_cast<float>(A.dt_build[tk]) * __uint_as_float(A.vmax[tk]) * 1.0001f +
                   A.margin * T.R_f);
  return fminf(d, 0.25f * T.R_f);  // also for a tank without fluid (dt = inf)
}

// The compensated form's record is one 32-byte Dat32 per particle, read by
// one load: in 2D the fixed-point coordinates take the words vz and pad, in
// 3D those of c, 1/rho and pad, which the pair loop recomputes from rho - rho0
// (5 instructions against a second 16-byte gather: the pass is bound by the
// L1 wavefronts of its gathers).
template<int D>
__device__ __forceinline__ void set_coords(Dat32& r, const int* q) {
  if constexpr (D == 2) {
    r.vz = __int_as_float(q[0]);
    r.pad = __int_as_float(q[1]);
  } else {
    r.c = __int_as_float(q[0]);
    r.invrho = __int_as_float(q[1]);
    r.pad = __int_as_float(q[2]);
  }
}
template<int D>
__device__ __forceinline__ void get_coords(const Dat32& r, int* q) {
  if constexpr (D == 2) {
    q[0] = __float_as_int(r.vz);
    q[1] = __float_as_int(r.pad);
  } else {
    q[0] = __float_as_int(r.c);
    q[1] = __float_as_int(r.invrho);
    q[2] = __float_as_int(r.pad);
  }
}

// Records: tank constants of a fluid particle (common to the gather and the
// stages), and their stores.
// The plain form's pad word holds the potential H(rho) of a tank with walls,
// once per particle instead of once per wall and neighbour.
template<int D>
__device__ __forceinline__ Dat64 fluid_record(const PhysDev& P, const TankDev& T, const double* v,
                                              double rho, bool walls) {
  double pr, c;
  tait_f64(P, T, rho, pr, c);
  const double inv = 1.0 / rho;
  return Dat64{v[0], v[1], D == 3 ? v[2] : 0.0, rho, pr * inv * inv, c, inv,
               walls ? potential_f64(P, T, rho) : 0.0};
}
template<int D>
__device__ __forceinline__ Dat32 fluid_record(const PhysDev& P, const TankDev& T, const float* v,
                                              float rho, bool) {
  float pr, c;
  tait_f32(P, T, rho, pr, c);
  const float inv = __frcp_rn(T.rho0_f + rho);
  return Dat32{v[0], v[1], D == 3 ? v[2] : 0.f, rho, pr * inv * inv, c, inv, 0.f};
}
template<int D>
__device__ __forceinline__ void store_list_record(const typename Layout<D, TG_FP64>::PosRec* pos,
                                                  Dat64* dat, int64_t j, const TankDev&,
                                                  const double* p, const Dat64& rec) {
  auto* out = const_cast<typename Layout<D, TG_FP64>::PosRec*>(pos);
  if constexpr (D == 2) {
    out[j] = Pos64_2{p[0], p[1]};
  } else {
    out[j] = Pos64_3{p[0], p[1], p[2], 0.0};
  }
  dat[j] = rec;
}
template<int D>
__device__ __forceinline__ void store_list_record(const int4*, Dat32* dat, int64_t j,
                                                  const TankDev& T, const double* p, Dat32 rec) {
  int q[3] = {0, 0, 0};
#pragma unroll
  for (int k = 0; k < D; ++k) q[k] = fixed_coord(p[k], T.lo[k], T.list_inv_unit);
  set_coords<D>(rec, q);
  dat[j] = rec;
}

// FluidEquations::compute_time_step (fluid_equations.hpp:205-230) of one
// particle, in either form (rho: the density, or its deviation).
__device__ __forceinline__ float time_step(const PhysDev& P, const TankDev& T, float speed,
                                           float accel, float drho, float c) {
  const float h = T.h_f;
  const float dt_ac = P.cfl_f * h / (c + speed);
  const float dt_vi = P.c_visc_f * h * h * (T.rho0_f + drho) / P.mu_f;
  const float dt_fo = P.c_force_f * sqrtf(h / fmaxf(accel, P.g_f));
  return fminf(dt_ac, fminf(dt_vi, dt_fo));
}

__device__ __forceinline__ double time_step(const PhysDev& P, const TankDev& T, double speed,
                                            double accel, double rho, double c) {
  const double h = T.h;
  const double dt_ac = P.cfl * h / (c + speed);
  const double dt_vi = P.c_visc * h * h * rho / P.mu;
  const double dt_fo = P.c_force * sqrt(h / fmax(accel, P.g));
  return fmin(dt_ac, fmin(dt_vi, dt_fo));
}

// Minimum over a tank, from the lanes that are here: one atomic for those of
// one tank, and only where it would lower the result.
__device__ __forceinline__ void fold_time_step(double* dt, uint32_t tk, float mine) {
  const unsigned here = __activemask();
  int same = 0;
  __match_all_sync(here, tk, &same);
  unsigned bits = __float_as_uint(mine);  // positive floats order like their bits
  if (same) bits = __reduce_min_sync(here, bits);
  if (same && static_cast<int>(threadIdx.x & 31u) != __ffs(here) - 1) return;
  const double d = static_cast<double>(__uint_as_float(bits));
  if (d < *static_cast<volatile double*>(dt + tk)) atomic_min_pos(dt + tk, d);
}

__device__ __forceinline__ void fold_time_step(double* dt, uint32_t tk, double mine) {
  if (mine < *static_cast<volatile double*>(dt + tk)) atomic_min_pos(dt + tk, mine);
}

// ---------------------------------------------------------------------------
// Gather into cell order.
template<int D, int F>
__global__ void __launch_bounds__(256) k_list_gather(ListArgs<D, F> A) {
  if (*A.stop != 0u) return;
  using R = typename StageArgs<D, F>::R;
  const StageArgs<D, F>& S = A.S;
  const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool valid = j < S.n;
  double dt_a = __longlong_as_double(0x7ff0000000000000ll);
  float v_a = 0.f;
  uint32_t tk = 0xffffffffu;
  float xl[3] = {0.f, 0.f, 0.f};
  bool fluid = false, wall = false;
  if (valid) {
    const uint32_t src = S.perm[j];
    const uint32_t id = S.X.id[src];
    tk = tank_of_key(S.skey[j], S.tank_off, S.ntanks);
    const TankDev& T = S.tanks[tk];
    wall = (id & kWallBit) != 0;
    fluid = !wall;
    double p[3] = {0.0, 0.0, 0.0};
    R v[3] = {R(0), R(0), R(0)};
#pragma unroll
    for (int k = 0; k < D; ++k) {
      p[k] = S.X.pos[k][src];
      S.Y.pos[k][j] = p[k];
    }
    local_coords<D>(T, p, xl);
    S.Y.id[j] = id;
    A.lrec[j] = make_float4(xl[0], xl[1], xl[2], wall ? -1.f : 1.f);
    typename ListArgs<D, F>::DatRec rec;
    if (wall) {
      // rho(0): the wall pass overwrites the walls near fluid.
      rec = wall_record<D>(S.phys, T, R(0), false);
    } else {
#pragma unroll
      for (int k = 0; k < D; ++k) {
        v[k] = S.X.vel[k][src];
        S.Udst.vel[k][j] = v[k];
      }
      const R rho = S.X.rho[src];
      S.Udst.rho[j] = rho;
      rec = fluid_record<D>(S.phys, T, v, rho, A.n_walls > 0);
      R a2 = R(0), v2 = R(0);
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const R a = S.X.dv[k][src];
        a2 += a * a;
        v2 += v[k] * v[k];
      }
      const R speed = sqrt(v2);
      dt_a = static_cast<double>(time_step(S.phys, T, speed, sqrt(a2), rho, rec.c));
      if constexpr (F == TG_FP64) v_a = __double2float_ru(speed);
      else v_a = speed;
    }
    store_list_record<D>(A.pos_in, A.dat_in, j, T, p, rec);
  }
  // The walls' slots, one atomic per warp.
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const unsigned wm = __ballot_sync(0xffffffffu, wall);
  if (wm != 0u) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(S.wall_count, static_cast<uint32_t>(__popc(wm)));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (wall) S.wall_list[base + __popc(wm & ((1u << lane) - 1u))] = static_cast<uint32_t>(j);
  }
  if (S.fbox != nullptr) fold_fluid_box<D>(S.fbox, S.ntanks, tk, fluid, xl);
  // Per-tank reductions: the warp's extremes when it lies in one tank, and
  // an atomic only where it would move the result (one address per tank).
  const uint32_t t0 = __reduce_min_sync(0xffffffffu, fluid ? tk : 0xffffffffu);
  const bool one = __all_sync(0xffffffffu, !fluid || tk == t0);
  if (one && t0 != 0xffffffffu) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dt_a = fmin(dt_a, __shfl_xor_sync(0xffffffffu, dt_a, o));
      v_a = fmaxf(v_a, __shfl_xor_sync(0xffffffffu, v_a, o));
    }
  }
  if ((one && lane == 0 && t0 != 0xffffffffu) || (!one && fluid)) {
    const uint32_t t = one ? t0 : tk;
    if (dt_a < *static_cast<volatile double*>(S.dt + t)) atomic_min_pos(S.dt + t, dt_a);
    if (__float_as_uint(v_a) > *static_cast<volatile unsigned*>(A.vmax + t)) {
      atomicMax(A.vmax + t, __float_as_uint(v_a));
    }
  }
}

// ---------------------------------------------------------------------------
// The walls that fluid can reach during the step: those within the list
// radius of their tank's fluid bounding box.
template<int D, int F>
__global__ void __launch_bounds__(256) k_list_select(ListArgs<D, F> A) {
  if (*A.stop != 0u) return;
  const StageArgs<D, F>& S = A.S;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  bool act = false;
  uint32_t e = 0;
  if (t < A.n_walls) {
    e = S.wall_list[t];
    const uint32_t tk = tank_of_key(S.skey[e], S.tank_off, S.ntanks);
    const TankDev& T = S.tanks[tk];
    const float4 x = A.lrec[e];
    const float xl[3] = {x.x, x.y, x.z};
    const float reach = sqrtf(T.wall_skip_r2_f) +
                        2.f * list_delta(A, T, tk);
    act = !beyond_fluid<D>(S.fbox, S.ntanks, tk, reach * reach, xl);
  }
  const unsigned mask = __ballot_sync(0xffffffffu, act);
  const int lane = static_cast<int>(threadIdx.x & 31u);
  uint32_t base = 0;
  if (lane == 0 && mask != 0u) {
    base = atomicAdd(S.wall_count + 1, static_cast<uint32_t>(__popc(mask)));
  }
  base = __shfl_sync(0xffffffffu, base, 0);
  if (act) S.wall_active[base + __popc(mask & ((1u << lane) - 1u))] = e;
}

// ---------------------------------------------------------------------------
// Lists.  A target's candidates are the rows of cells that its list radius
// RL reaches, each clipped to RL along x; they are tested on tank-local FP32
// coordinates (list_slack_f covers their rounding).  A target whose block
// of cells reaches a border cell of the grid, where clamped particles lie
// outside their cell's box, takes whole rows and tests FP64 positions.
// Accepted entries leave in groups of four (16-byte stores).

struct ListRows {
  int y0, y1, z0, z1, x0, x1;  // the block of cells
  int x, yb, zb, span;         // its centre, unclipped corner and width
  float RL, RL2;
  bool border;
};

template<int D>
__device__ __forceinline__ ListRows list_rows(const TankDev& T, const int* c, const float* xl,
                                              float RL) {
  ListRows W;
  W.RL = RL;
  W.RL2 = RL * RL;
  const float inv = T.inv_cs_f;
  const int kk = static_cast<int>(ceilf(RL * inv));
  W.border = c[0] - kk <= 0 || c[0] + kk >= T.nc[0] - 1 || c[1] - kk <= 0 ||
             c[1] + kk >= T.nc[1] - 1;
  if constexpr (D == 3) W.border = W.border || c[2] - kk <= 0 || c[2] + kk >= T.nc[2] - 1;
  W.x = c[0];
  W.yb = c[1] - kk;
  W.zb = D == 3 ? c[2] - kk : 0;
  W.span = 2 * kk + 1;
  W.x0 = max(c[0] - kk, 0);
  W.x1 = min(c[0] + kk, T.nc[0] - 1);
  W.y0 = max(c[1] - kk, 0);
  W.y1 = min(c[1] + kk, T.nc[1] - 1);
  W.z0 = D == 3 ? max(c[2] - kk, 0) : 0;
  W.z1 = D == 3 ? min(c[2] + kk, T.nc[2] - 1) : 0;
  if (!W.border) {
    // The rows whose box comes within RL (floor of finite values).
    W.y0 = max(W.y0, static_cast<int>(floorf((xl[1] - RL) * inv)));
    W.y1 = min(W.y1, static_cast<int>(floorf((xl[1] + RL) * inv)));
    if constexpr (D == 3) {
      W.z0 = max(W.z0, static_cast<int>(floorf((xl[2] - RL) * inv)));
      W.z1 = min(W.z1, static_cast<int>(floorf((xl[2] + RL) * inv)));
    }
  }
  return W;
}

// Record range of row (y, z); empty when the row is out of reach.
template<int D>
__device__ __forceinline__ void list_row(const TankDev& T, const ListRows& W, const float* xl,
                                         const uint32_t* __restrict__ cstart, int y, int z,
                                         uint32_t& s, uint32_t& e) {
  int x0 = W.x0, x1 = W.x1;
  if (!W.border) {
    const float cs = T.cs_f;
    const float ylo = static_cast<float>(y) * cs;
    const float gy = fmaxf(fmaxf(ylo - xl[1], xl[1] - (ylo + cs)), 0.f);
    float rem = W.RL2 - gy * gy;
    if constexpr (D == 3) {
      const float zlo = static_cast<float>(z) * cs;
      const float gz = fmaxf(fmaxf(zlo - xl[2], xl[2] - (zlo + cs)), 0.f);
      rem -= gz * gz;
    }
    if (rem < 0.f) {
      s = e = 0u;
      return;
    }
    const float w = sqrtf(rem);
    x0 = max(x0, static_cast<int>(floorf((xl[0] - w) * T.inv_cs_f)));
    x1 = min(x1, static_cast<int>(floorf((xl[0] + w) * T.inv_cs_f)));
    if (x1 < x0) {
      s = e = 0u;
      return;
    }
  }
  uint32_t row = T.cell_off + static_cast<uint32_t>(y) * T.nc[0];
  if constexpr (D == 3) row += static_cast<uint32_t>(z) * T.nc[1] * T.nc[0];
  s = __ldg(cstart + 2 * (row + x0));
  e = __ldg(cstart + 2 * (row + x1 + 1));
}

// |r_a - r_b|^2 <= RL^2 on the FP64 step-start positions.
template<int D>
__device__ __forceinline__ bool list_near_fp64(double* const* pos, int64_t a, uint32_t b,
                                               double RL) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const double d = pos[k][a] - pos[k][b];
    s = fma(d, d, s);
  }
  return s <= RL * RL;
}

// Candidates loaded together, and 128-thread blocks per SM: the build waits
// for its loads, so warps count most.  Measured sort + build per step, 3D 2M
// / 2D 1.28M fluid particles, in ms (candidates x blocks): 2 x 12 1.03 / .338
// (2 x 8 1.15 / .358, 2 x 10 1.07 / .341, 2 x 16 1.08 / .358, 1 x 16 1.07 /
// .363, 4 x 8 1.10 / .347, 4 x 12 1.25 / .343); loading one record ahead of
// the test instead 1.23 / .385.
constexpr uint32_t kListScan = 2;
constexpr int kListBuildBlocks = 12;

// Appends accepted entries to a list in groups of four.
struct ListWriter {
  uint4* out;
  uint32_t cap, cnt = 0, e0 = 0, e1 = 0, e2 = 0;
  __device__ __forceinline__ void add(uint32_t j) {
    if ((cnt & 3u) == 3u && cnt < cap) out[(cnt >> 2) * 32] = make_uint4(e2, e1, e0, j);
    e2 = e1;
    e1 = e0;
    e0 = j;
    ++cnt;
  }
  // The last group: its entries were shifted in, the newest in e0.
  __device__ __forceinline__ void finish() {
    const uint32_t tail = cnt & 3u;
    if (tail == 0u || cnt >= cap) return;
    out[(cnt >> 2) * 32] = tail == 1u   ? make_uint4(e0, 0u, 0u, 0u)
                           : tail == 2u ? make_uint4(e1, e0, 0u, 0u)
                                        : make_uint4(e2, e1, e0, 0u);
  }
};

// The list of slot i, by Team lanes (lane tl of the team).  Wall targets list fluid entries only.  A warp with a border target
// takes the FP64 test for all its targets: kept apart, so that the common
// loop holds no FP64 instruction (selected per candidate, they issued for
// every candidate and the build of 2M particles took 9.2 ms).
template<int D, int F, int Team, bool Wall, bool Border>
__device__ __forceinline__ void build_list(const ListArgs<D, F>& A, const TankDev& T,
                                           const ListRows& W, const float* xl, int64_t i,
                                           bool target, int tl, unsigned tmask) {
  const StageArgs<D, F>& S = A.S;
  const uint32_t ia = static_cast<uint32_t>(i);
  const auto accept = [&](const float4& b, uint32_t j) {
    bool near;
    if constexpr (!Border) {
      const float dx = xl[0] - b.x, dy = xl[1] - b.y;
      float s2 = dx * dx + dy * dy;
      if constexpr (D == 3) {
        const float dz = xl[2] - b.z;
        s2 = fmaf(dz, dz, s2);
      }
      near = s2 <= W.RL2;
    } else {
      near = list_near_fp64<D>(S.Y.pos, i, j, static_cast<double>(W.RL));
    }
    return near && j != ia && !(Wall && b.w < 0.f);
  };
  const uint32_t cap = static_cast<uint32_t>(A.cap);
  uint32_t cnt = 0;
  if constexpr (Team == 1) {
    ListWriter w;
    w.out = reinterpret_cast<uint4*>(A.list) + (list_at(i, 0, A.cap) >> 2);
    w.cap = cap;
    // Every lane takes its rows by their offset from its own cell's row (out
    // of reach or not), so that the lanes of a row of cells, most of a warp,
    // walk the same rows together.
    for (int z = W.zb; z < W.zb + (D == 3 ? W.span : 1); ++z) {
      for (int y = W.yb; y < W.yb + W.span; ++y) {
        uint32_t s = 0, e = 0;
        if (y >= W.y0 && y <= W.y1 && z >= W.z0 && z <= W.z1) {
          list_row<D>(T, W, xl, S.cell_start, y, z, s, e);
        }
        // Batches of candidates in flight; lrec is readable kListScan - 1
        // records past the last.
        for (uint32_t j = s; j < e; j += kListScan) {
          float4 b[kListScan];
#pragma unroll
          for (uint32_t q = 0; q < kListScan; ++q) b[q] = A.lrec[j + q];
#pragma unroll
          for (uint32_t q = 0; q < kListScan; ++q) {
            if (j + q < e && accept(b[q], j + q)) w.add(j + q);
          }
        }
      }
    }
    w.finish();
    cnt = w.cnt;
  } else {
    // The team's lanes share every row; lanes without a target sit out.
    if (target) {
      const int c[3] = {W.x, W.yb + (W.span >> 1), D == 3 ? W.zb + (W.span >> 1) : 0};
      const float o[3] = {xl[0] - static_cast<float>(c[0]) * T.cs_f,
                          xl[1] - static_cast<float>(c[1]) * T.cs_f,
                          D == 3 ? xl[2] - static_cast<float>(c[2]) * T.cs_f : 0.f};
      const unsigned below = tmask & ((1u << (threadIdx.x & 31u)) - 1u);
      for_shared_rows<D, Team>(T, c, W.span >> 1, S.cell_start, tl, tmask, Border ? nullptr : o,
                               W.RL2, [&](uint32_t s, uint32_t e) {
        for (uint32_t j0 = s; j0 < e; j0 += Team) {
          const uint32_t j = j0 + tl;
          const bool acc = j < e && accept(A.lrec[j < e ? j : s], j);
          const unsigned hit = __ballot_sync(tmask, acc) & tmask;
          const uint32_t p = cnt + __popc(hit & below);
          if (acc && p < cap) A.list[list_at(i, p, A.cap)] = j;
          cnt += __popc(hit);
        }
      });
    }
  }
  if (target && tl == 0) {
    A.cnt[i] = min(cnt, cap);
    if (cnt > cap) atomicOr(A.stop, kStopCapacity);
  }
}

// Called by whole warps; lanes without a target take part in the votes.
template<int D, int F, int Team, bool Wall>
__device__ __forceinline__ void build_lists(const ListArgs<D, F>& A, int64_t i, bool target,
                                            int tl, unsigned tmask) {
  const StageArgs<D, F>& S = A.S;
  const TankDev* T = S.tanks;
  ListRows W{0, -1, 0, -1, 0, 0, 0, 0, 0, 0, 0.f, 0.f, false};
  float xl[3] = {0.f, 0.f, 0.f};
  if (target) {
    const uint32_t key = S.skey[i];
    const uint32_t tk = tank_of_key(key, S.tank_off, S.ntanks);
    T = S.tanks + tk;
    int c[3] = {0, 0, 0};
    cell_from_key<D>(*T, key, c);
    const float4 x = A.lrec[i];
    xl[0] = x.x;
    xl[1] = x.y;
    xl[2] = x.z;
    W = list_rows<D>(*T, c, xl, T->R_f + T->list_slack_f + 2.f * list_delta(A, *T, tk));
  }
  if (__any_sync(0xffffffffu, W.border)) {
    build_list<D, F, Team, Wall, true>(A, *T, W, xl, i, target, tl, tmask);
  } else {
    build_list<D, F, Team, Wall, false>(A, *T, W, xl, i, target, tl, tmask);
  }
}

// Blocks below fluid_blocks take the slots in order (walls excepted), the
// others the listed walls in turn.
template<int D, int F, int Team>
__global__ void __launch_bounds__(128, kListBuildBlocks) k_list_build(ListArgs<D, F> A, unsigned fluid_blocks) {
  if (*A.stop != 0u) return;
  const StageArgs<D, F>& S = A.S;
  const int tl = Team == 1 ? 0 : static_cast<int>(threadIdx.x % Team);
  const unsigned tmask = team_mask<Team>();
  if (blockIdx.x < fluid_blocks) {
    const int64_t i =
        (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / Team;
    const bool target = i < S.n && !(S.Y.id[i] & kWallBit);
    build_lists<D, F, Team, false>(A, target ? i : 0, target, tl, tmask);
    return;
  }
  const bool all = S.fbox == nullptr;
  const uint32_t* walls = all ? S.wall_list : S.wall_active;
  const int64_t count = all ? S.wall_count[0] : S.wall_count[1];
  const int64_t step = static_cast<int64_t>(gridDim.x - fluid_blocks) * blockDim.x / Team;
  // Warp-uniform trips: the team form votes across the warp.
  const int64_t w0 = (static_cast<int64_t>(blockIdx.x - fluid_blocks) * blockDim.x +
                      (threadIdx.x & ~31u)) / Team;
  const int in_warp = static_cast<int>((threadIdx.x & 31u) / Team);
  for (int64_t w = w0; w < count; w += step) {
    const bool target = w + in_warp < count;
    const int64_t i = target ? walls[w + in_warp] : 0;
    build_lists<D, F, Team, true>(A, i, target, tl, tmask);
  }
}

// ---------------------------------------------------------------------------
// Pair arithmetic.

// g(q) with grad W = S g r_ab (r_ab in the pair loop's unit, S the tank's
// list_s*): Wendland kernels f'(q)/q without its constant, as a polynomial
// in t = 1 - q/2 >= 0; B-splines f'(q) / |r_ab|.
template<int K, class T>
__device__ __forceinline__ T list_g(T t, T q, T rinv) {
  if constexpr (K == TG_KERNEL_WENDLAND_C2) {
    return t * t * t;
  } else if constexpr (K == TG_KERNEL_WENDLAND_C4) {
    const T t2 = t * t;  // (1 + 5/2 q) = 6 - 5 t
    return (T(6) - T(5) * t) * (t2 * t2 * t);
  } else if constexpr (K == TG_KERNEL_WENDLAND_C6) {
    const T t2 = t * t;  // 2 + 7 q + 8 q^2 = 48 - 78 t + 32 t^2
    const T t4 = t2 * t2;
    return (T(48) + t * (T(32) * t - T(78))) * (t4 * t2 * t);
  } else {
    return KernelPoly<K>::deriv(q) * rinv;
  }
}

__device__ __forceinline__ Dat32 load_dat_wide(const Dat32* p, uint32_t j) {
  Dat32 r;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(r.vx), "=f"(r.vy), "=f"(r.vz), "=f"(r.drho), "=f"(r.P), "=f"(r.c), "=f"(r.invrho),
        "=f"(r.pad)
      : "l"(p + j));
  return r;
}

// Compensated form, one target.
template<int D, int F, int K, int Phys>
struct ListPairF32 {
  Dat32 a;
  int x[3];
  float hq, ah, ca_ah, eps2, dk, mu2, rho_a2, rho0, inv_rho0, cs0;
  int visc, diff;
  bool kahan;
  Kahan drho, dv[3];
  float pd, pv[3];

  __device__ __forceinline__ void init(const ListArgs<D, F>& A, const TankDev& T, int64_t i) {
    a = A.dat_in[i];
    get_coords<D>(a, x);
    if constexpr (D == 3) {
      float pr;
      tait_f32(A.S.phys, T, a.drho, pr, a.c);
      a.invrho = __frcp_rn(T.rho0_f + a.drho);
    }
    hq = T.list_hq_f;
    ah = T.list_ah_f;
    ca_ah = a.c * ah;
    eps2 = T.list_eps2_f;
    dk = T.list_dk_f;
    mu2 = T.list_mu2_f * a.invrho;
    rho0 = T.rho0_f;
    rho_a2 = 2.f * T.rho0_f + a.drho;
    inv_rho0 = T.inv_rho0_f;
    cs0 = T.cs0_f;
    visc = A.S.phys.viscosity;
    diff = A.S.phys.diffusion;
    kahan = A.S.kahan != 0;
  }
  // r_ab in fixed-point units, and its square.
  __device__ __forceinline__ float rab(const Dat32& b, float* d) const {
    int y[3];
    get_coords<D>(b, y);
    float s2 = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      d[k] = __int2float_rn(static_cast<int>(static_cast<unsigned>(x[k]) -
                                             static_cast<unsigned>(y[k])));
      s2 = fmaf(d[k], d[k], s2);
    }
    return s2;
  }
  __device__ __forceinline__ void open() {
    pd = 0.f;
    pv[0] = pv[1] = pv[2] = 0.f;
  }
  __device__ __forceinline__ void close() {
    if (Phys != kPhysGeneric || kahan) {
      drho.add(pd);
#pragma unroll
      for (int k = 0; k < D; ++k) dv[k].add(pv[k]);
    } else {
      drho.s += pd;
#pragma unroll
      for (int k = 0; k < D; ++k) dv[k].s += pv[k];
    }
  }
  // PairF32::add in the unit of r_ab, without the tank's factor list_s_f.
  __device__ __forceinline__ void add(const ListArgs<D, F>& A, const TankDev& T, const float* d,
                                      float s2, const Dat32& b) {
    const int df = Phys == kPhysTextbook    ? TG_DIFF_MOLTENI
                   : Phys == kPhysReference ? TG_DIFF_FERRARI
                                            : diff;
    const int vs = Phys == kPhysTextbook    ? TG_VISC_MONAGHAN
                   : Phys == kPhysReference ? TG_VISC_MORRIS
                                            : visc;
    float cb, ib;
    if constexpr (D == 2) {
      cb = b.c;
      ib = b.invrho;
    } else {
      if constexpr (Phys == kPhysGeneric) {
        float pr;
        tait_f32(A.S.phys, T, b.drho, pr, cb);
      } else {  // the presets' Tait law, xi = 7
        const float xr = fmaf(b.drho, inv_rho0, 1.f);
        cb = cs0 * (xr * xr * xr);
      }
      ib = rcp_newton(rho0 + b.drho);
    }
    const float rinv = rsqrt_seed(s2);
    const float r = s2 * rinv;
    // t = max(1 - q/2, 0): 0 also for the NaN of a coincident particle.
    const float t = fmaxf(fmaf(r, -0.5f * hq, 1.f), 0.f);
    const float g = list_g<K>(t, r * hq, rinv);
    const float vb[3] = {b.vx, b.vy, b.vz};
    const float va[3] = {a.vx, a.vy, a.vz};
    float vd = 0.f;
#pragma unroll
    for (int k = 0; k < D; ++k) vd = fmaf(va[k] - vb[k], d[k], vd);
    const float drab = a.drho - b.drho;
    float cont = vd;
    if (df == TG_DIFF_FERRARI) {
      cont += fmaxf(a.c, cb) * drab * r * ib;
    } else if (df == TG_DIFF_MOLTENI) {
      cont += dk * drab * ib;
    }
    pd = fmaf(g, cont, pd);
    float Pi;
    if (vs == TG_VISC_MORRIS) {
      Pi = mu2 * vd * ib * (rinv * rinv);
    } else {
      Pi = __fdividef(fminf(vd, 0.f) * fmaf(cb, ah, ca_ah), (s2 + eps2) * (rho_a2 + b.drho));
    }
    const float coef = (Pi - (a.P + b.P)) * g;
#pragma unroll
    for (int k = 0; k < D; ++k) pv[k] = fmaf(coef, d[k], pv[k]);
  }
};

// FP64 form, one target.  GB300's FP64 pipe bounds this form, so the pair
// costs as few FP64 operations as the sums allow: one reciprocal square root
// and one quotient, each from the hardware seed (relative error below 2^-19)
// by the third-order iteration of rcp_f64 and sqrt_f64 in the residual e
// (truncation 5 e^3 / 16 < 2^-55 and e^3 < 2^-57), and comparisons on the high
// words.
template<int D, int F, int K>
struct ListPairF64 {
  Dat64 a;
  double x[3];
  double mhinv2, hinv, ah, eps2, dk, mu2;
  double R2;
  int visc, diff, r2hi;
  unsigned within;  // high words of normal numbers clearly below R^2
  double drho, dv[3];

  __device__ __forceinline__ void init(const ListArgs<D, F>& A, const TankDev& T, int64_t i) {
    a = A.dat_in[i];
    load_pos(A.pos_in, static_cast<uint32_t>(i), x);
    hinv = T.hinv;
    mhinv2 = -0.5 * T.hinv;
    ah = A.S.phys.alpha * T.h;
    eps2 = T.visc_eps2;
    dk = T.diff_k;
    mu2 = 2.0 * A.S.phys.mu * a.invrho;
    R2 = T.radius2;
    r2hi = __double2hiint(R2);
    within = static_cast<unsigned>(max(r2hi - 1 - 0x00100000, 0));
    visc = A.S.phys.viscosity;
    diff = A.S.phys.diffusion;
    drho = dv[0] = dv[1] = dv[2] = 0.0;
  }
  // r_ab, |r_ab|^2 and the reference's predicate: decided by the high words
  // except where they are within one of R^2's, there on the reference's own
  // rounding (dist2_exact).  Particles whose squared distance is a subnormal
  // number, which the seed would flush, add nothing: the reference's unit
  // vector is 0 there.
  __device__ __forceinline__ bool near(const double* y, double* d, double& s2) const {
    s2 = 0.0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      d[k] = x[k] - y[k];
      s2 = k == 0 ? d[0] * d[0] : fma(d[k], d[k], s2);
    }
    const int hi = __double2hiint(s2);
    if (static_cast<unsigned>(hi - 0x00100000) < within) return true;
    if (hi < 0x00100000) return s2 == 0.0;
    if (hi > r2hi + 1) return false;
    double t[3];
    return dist2_exact<D>(x, y, t) <= R2;
  }
  __device__ __forceinline__ void add(const double* d, double s2, const Dat64& b) {
    // r = s2 / sqrt(s2).
    const double y0 = rsqrt_seed(s2);
    const double r0 = s2 * y0;
    const double e = fma(-r0, y0, 1.0);
    const double ep = e * fma(e, 0.375, 0.5);
    const double r = fma(r0, ep, r0);
    double t = fma(r, mhinv2, 1.0);
    // 0 for t < 0 and for the NaN of a coincident particle: t <= 1, so its
    // high word lies in [0, 0x3ff00000].
    if (static_cast<unsigned>(__double2hiint(t)) > 0x3ff00000u) t = 0.0;
    double rinv = 0.0;
    if (!KernelPoly<K>::deriv_over_q || visc == TG_VISC_MORRIS) rinv = fma(y0, ep, y0);
    const double g = list_g<K>(t, KernelPoly<K>::deriv_over_q ? 0.0 : r * hinv, rinv);
    const double vb[3] = {b.vx, b.vy, b.vz};
    const double va[3] = {a.vx, a.vy, a.vz};
    double vd = (va[0] - vb[0]) * d[0];
#pragma unroll
    for (int k = 1; k < D; ++k) vd = fma(va[k] - vb[k], d[k], vd);
    const double drab = a.rho - b.rho;
    double cont = vd;
    if (diff == TG_DIFF_FERRARI) {
      cont = fma(fmax(a.c, b.c) * drab * r, b.invrho, cont);
    } else if (diff == TG_DIFF_MOLTENI) {
      cont = fma(dk * drab, b.invrho, cont);
    }
    drho = fma(g, cont, drho);
    const double Pab = a.P + b.P;
    double coef;
    if (visc == TG_VISC_MORRIS) {
      coef = fma(mu2 * vd * b.invrho, rinv * rinv, -Pab);
    } else {
      coef = -Pab;
      if (__double2hiint(vd) < 0) {  // approaching
        const double den = (s2 + eps2) * (a.rho + b.rho);
        const double z0 = rcp_seed(den);
        const double f = fma(-den, z0, 1.0);
        const double q0 = (ah * vd * (a.c + b.c)) * z0;
        coef += fma(q0, fma(f, f, f), q0);
      }
    }
    coef *= g;
#pragma unroll
    for (int k = 0; k < D; ++k) dv[k] = fma(coef, d[k], dv[k]);
  }
};

// ---------------------------------------------------------------------------
// Wall extrapolation (k_walls) over the walls' lists: teams of lanes take the
// listed walls in turn, the lanes the list's groups of four entries.  Four
// lanes, eight for the small runs whose passes are chains of latencies
// (measured in ms per step for 8 / 4 / 2 lanes: 24 3D tanks .163 / .129 /
// .131, 3D 2M .121 / .101 / .097, plain 3D 250k .366 / .297 / .297, 2D 1.28M
// .037 / .039 / .050; 800 particles with shifting 297 / 310 us per step).
template<int D, int F, int K, int Team>
__global__ void __launch_bounds__(128) k_list_walls(ListArgs<D, F> A) {
  if (*A.stop != 0u) return;
  const StageArgs<D, F>& S = A.S;
  const bool all = S.fbox == nullptr;
  const uint32_t* list = all ? S.wall_list : S.wall_active;
  const int64_t count = all ? S.wall_count[0] : S.wall_count[1];
  const int tl = static_cast<int>(threadIdx.x % Team);
  const unsigned tmask = team_mask<Team>();
  const int64_t teams = static_cast<int64_t>(gridDim.x) * blockDim.x / Team;
  for (int64_t w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / Team;
       w < count; w += teams) {
    const uint32_t ew = list[w];
    const TankDev& T = S.tanks[tank_of_key(S.skey[ew], S.tank_off, S.ntanks)];
    const uint32_t m = A.cnt[ew];
    const uint4* groups = reinterpret_cast<const uint4*>(A.list) + (list_at(ew, 0, A.cap) >> 2);
    double ne[3] = {0.0, 0.0, 0.0};
    if (S.fc.on) normalize_d<D>(S.fc.ggam + D * static_cast<size_t>(ew), ne);
    if constexpr (F == TG_FP64) {
      double pe[3] = {0.0, 0.0, 0.0};
      load_pos(A.pos_in, ew, pe);
      double Ss = 0.0, H = 0.0;
      for (uint32_t p = 4 * tl; p < m; p += 4 * Team) {
        const uint4 g = groups[(p >> 2) * 32];
        const uint32_t js[4] = {g.x, g.y, g.z, g.w};
        for (uint32_t q = 0; q < 4u && p + q < m; ++q) {
          double pb[3], d[3];
          load_pos(A.pos_in, js[q], pb);
          const double s2 = dist2_exact<D>(pb, pe, d);
          if (s2 > T.radius2) continue;
          const Dat64 b = load_dat(A.dat_in, js[q]);
          const double VW = b.invrho * KernelPoly<K>::value(sqrt_f64(s2) * T.hinv);
          double Hb = b.pad;
          if (S.fc.on) Hb += S.phys.g * dot_d<D>(d, ne) * ne[1];
          Ss += VW;
          H = fma(VW, Hb, H);
        }
      }
#pragma unroll
      for (int o = Team / 2; o > 0; o >>= 1) {
        Ss += __shfl_xor_sync(tmask, Ss, o, Team);
        H += __shfl_xor_sync(tmask, H, o, Team);
      }
      if (tl == 0) {
        const double Hs = fabs(Ss * (T.m * T.w)) <= 6.0554544523933395e-06 ? 0.0 : H / Ss;
        A.dat_in[ew] = wall_record<D>(S.phys, T, wall_density_f64(S.phys, T, Hs), true);
      }
    } else {
      const float hq = T.list_hq_f;
      ListPairF32<D, F, K, kPhysGeneric> own;  // coordinates only
      const Dat32 e = A.dat_in[ew];
      get_coords<D>(e, own.x);
      Kahan Ss, H;
      for (uint32_t p = 4 * tl; p < m; p += 4 * Team) {
        const uint4 g = groups[(p >> 2) * 32];
        const uint32_t js[4] = {g.x, g.y, g.z, g.w};
        for (uint32_t q = 0; q < 4u && p + q < m; ++q) {
          const Dat32 b = load_dat(A.dat_in, js[q]);
          float d[3];
          const float s2 = own.rab(b, d);
          if (s2 > T.list_hi_f) continue;
          if (s2 >= T.list_lo_f && !within_fp64<D>(A.pin, ew, js[q], T.radius2)) continue;
          const float W = T.w_f * KernelPoly<K>::value(sqrt_newton(s2) * hq);
          const float ib = D == 2 ? b.invrho : rcp_newton(T.rho0_f + b.drho);
          const float Vb = T.m_f * ib;
          float Hb = potential_f32(S.phys, T, b.drho);
          if (S.fc.on) {
            float dn = 0.f;  // r_be = -d
#pragma unroll
            for (int k = 0; k < D; ++k) dn += d[k] * static_cast<float>(ne[k]);
            Hb -= S.phys.g_f * (dn * T.list_unit_f) * static_cast<float>(ne[1]);
          }
          Ss.add(Vb * W);
          H.add(Vb * Hb * W);
        }
      }
      float Sv = Ss.value(), Hv = H.value();
#pragma unroll
      for (int o = Team / 2; o > 0; o >>= 1) {
        Sv += __shfl_xor_sync(tmask, Sv, o, Team);
        Hv += __shfl_xor_sync(tmask, Hv, o, Team);
      }
      if (tl == 0) {
        const float Hs = fabsf(Sv) <= 6.0554544523933395e-06f ? 0.f : Hv / Sv;
        Dat32 rec = wall_record<D>(S.phys, T, deviation_from_potential_f32(S.phys, T, Hs), true);
        set_coords<D>(rec, own.x);
        A.dat_in[ew] = rec;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Pair sums over the lists, then the update: Euler step, SSPRK combination,
// and the next stage's records (or, in the last stage, the home state with
// the keys of the new positions).

template<int D, int F>
__device__ __forceinline__ void list_commit_wall(const ListArgs<D, F>& A, int64_t e, uint32_t id) {
  using R = typename StageArgs<D, F>::R;
  const StageArgs<D, F>& S = A.S;
  if (!A.last) {
    if (A.first) {  // the other record buffer gets the wall's fixed part
      A.dat_out[e] = A.dat_in[e];
      if constexpr (F == TG_FP64) A.pos_out[e] = A.pos_in[e];
#pragma unroll
      for (int k = 0; k < D; ++k) A.pout[k][e] = S.Y.pos[k][e];
      if (A.curkey != nullptr) A.curkey[e] = S.skey[e];
    } else {
#pragma unroll
      for (int k = 0; k < D; ++k) A.pout[k][e] = S.Y.pos[k][e];
    }
    return;
  }
  const uint32_t key = S.skey[e];
  double p[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < D; ++k) {
    p[k] = S.Y.pos[k][e];
    S.X.pos[k][e] = p[k];
    S.X.vel[k][e] = R(0);
    S.X.dv[k][e] = R(0);
  }
  if constexpr (F == TG_FP64) {
    S.X.rho[e] = A.dat_in[e].rho;
  } else {
    S.X.rho[e] = A.dat_in[e].drho;
    const TankDev& T = S.tanks[tank_of_key(key, S.tank_off, S.ntanks)];
    int c[3] = {0, 0, 0};
    float o[3] = {0.f, 0.f, 0.f};
    cell_from_key<D>(T, key, c);
    cell_offset<D>(T, c, p, o);
#pragma unroll
    for (int k = 0; k < D; ++k) S.X.off[k][e] = o[k];
  }
  S.X.drho[e] = R(0);
  S.X.id[e] = id;
  S.X.pkey[e] = key;  // read before the key write: the buffers may alias
  S.X.key[e] = key;
}

template<int D, int F>
__device__ __forceinline__ void list_epilogue(const ListArgs<D, F>& A, int64_t i, uint32_t id,
                                              uint32_t key, uint32_t tk, const TankDev& T,
                                              const typename StageArgs<D, F>::R* va,
                                              typename StageArgs<D, F>::R rho_self,
                                              const typename StageArgs<D, F>::R* dv,
                                              typename StageArgs<D, F>::R drho) {
  using R = typename StageArgs<D, F>::R;
  const StageArgs<D, F>& S = A.S;
  const double dt = S.dt[tk];
  const R dtr = static_cast<R>(dt);
  const float dtf = static_cast<float>(dtr);
  double pn[3] = {0.0, 0.0, 0.0};
  R vn[3] = {R(0), R(0), R(0)};
#pragma unroll
  for (int k = 0; k < D; ++k) {
    pn[k] = fma(dt, static_cast<double>(va[k]), A.pin[k][i]);
    vn[k] = va[k] + dtr * dv[k];
  }
  R rn = rho_self + dtr * drho;
  // The displacement since the step's start, for the bound: dt v in the
  // first stage, so that the second starts from u_n + dt v_n and ends at
  // w dt (v_n + v) from u_n (few FP64 operations: their pipe is what the
  // compensated form's update is bound by); the third's only where
  // post-integration follows, from the positions.
  float dis[3] = {0.f, 0.f, 0.f};
  if (S.lincomb) {
    const R wr = A.wr, w0r = A.w0r;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const R v0 = S.Udst.vel[k][i];
      dis[k] = static_cast<float>(wr) * dtf * (static_cast<float>(v0) + static_cast<float>(va[k]));
      pn[k] = fma(A.w0, S.Y.pos[k][i], S.w_new * pn[k]);
      vn[k] = w0r * v0 + wr * vn[k];
    }
    rn = w0r * S.Udst.rho[i] + wr * rn;
  } else {
#pragma unroll
    for (int k = 0; k < D; ++k) dis[k] = dtf * static_cast<float>(va[k]);
  }
  if (!A.last) {
    float d2 = 0.f;
    if (A.post || A.carry) {
#pragma unroll
      for (int k = 0; k < D; ++k) dis[k] = __double2float_rn(pn[k] - S.Y.pos[k][i]);
    }
    if (A.post) {
#pragma unroll
      for (int k = 0; k < D; ++k) S.Y.dv[k][i] = dv[k];
      S.Y.drho[i] = drho;
    }
#pragma unroll
    for (int k = 0; k < D; ++k) {
      d2 = fmaf(dis[k], dis[k], d2);
      A.pout[k][i] = pn[k];
    }
    float far = sqrtf(d2);
    if (A.travel != nullptr) far += A.travel[i];
    if (!(far <= list_delta(A, T, tk))) atomicOr(A.stop, kStopMoved);
    if (A.curkey != nullptr) {
      int cn[3] = {0, 0, 0};
      bool outside = false;
      cell_of<D>(T, pn, cn, outside);
      A.curkey[i] = key_of(flat_cell<D>(T, cn), false);
    }
    const auto rec = fluid_record<D>(S.phys, T, vn, rn, A.n_walls > 0);
    if (A.carry) {
      A.travel_out[i] = far * 1.00001f;
      R v2 = R(0), a2 = R(0);
#pragma unroll
      for (int k = 0; k < D; ++k) {
        A.next.vel[k][i] = vn[k];
        v2 += vn[k] * vn[k];
        a2 += dv[k] * dv[k];
      }
      A.next.rho[i] = rn;
      fold_time_step(A.dt_next, tk, time_step(S.phys, T, sqrt(v2), sqrt(a2), rn, rec.c));
    }
    store_list_record<D>(A.pos_out, A.dat_out, i, T, pn, rec);
    return;
  }
  int c[3] = {0, 0, 0};
  cell_from_key<D>(T, key, c);
  commit_fluid<D, F>(S, i, id, T, c, pn, vn, rn, dv, drho);
}

// Launch bounds (128-thread blocks per SM) and records in flight per lane of
// the pair loop.  FP64: its pipe is the limit (87% busy).  Compensated: the
// gathers take 80% of the L1's throughput and the pairs 56% of the issue slots
// at the same time (3D 2M fluid: 0.470 ms per launch, 1.448 for the walk over
// cells).  Measured for the three passes of a step (in a chain of
// two) at 2M (3D) / 1.28M (2D) fluid particles in ms, blocks x records: 3D
// 7 x 2 1.59, 6 x 4 1.585, 8 x 2 1.62, 6 x 2 1.62, 9 x 2 1.75, 5 x 4 1.69,
// 8 x 1 1.68; 2D 9 x 2 .631, 8 x 2 .642, 10 x 2 .665, 7 x 2 .656, 8 x 4 .638,
// 10 x 1 .636.  With a predicate per entry and a check of the list's end: 3D
// 1.69, 2D .631.
template<int D, int F>
constexpr int list_min_blocks() {
  return F == TG_FP64 ? 4 : D == 3 ? 7 : 9;
}
constexpr uint32_t kListBatch = 2;

// Team lanes per target take the list's groups of four entries in turn.
// The compensated sums take one add per two groups.
template<int D, int F, int K, int Phys, int Team>
__global__ void __launch_bounds__(128, list_min_blocks<D, F>()) k_list_forces(ListArgs<D, F> A) {
  using R = typename StageArgs<D, F>::R;
  if (*A.stop != 0u) return;
  const StageArgs<D, F>& S = A.S;
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / Team;
  const int tl = Team == 1 ? 0 : static_cast<int>(threadIdx.x % Team);
  if (i >= S.n) return;  // uniform over a team, as are the exits below
  const uint32_t id = S.Y.id[i];
  if (id & kWallBit) {
    if (tl == 0) list_commit_wall(A, i, id);
    return;
  }
  const uint32_t key = S.skey[i];
  const uint32_t tk = tank_of_key(key, S.tank_off, S.ntanks);
  const TankDev& T = S.tanks[tk];
  const uint32_t m = A.cnt[i];
  const uint4* groups = reinterpret_cast<const uint4*>(A.list) + (list_at(i, 0, A.cap) >> 2);
  const bool faces = S.fc.on;
  R va[3], dv[3] = {R(0), R(0), R(0)}, drho, rho_self;
  if constexpr (F == TG_FP64) {
    ListPairF64<D, F, K> acc;
    acc.init(A, T, i);
    for (uint32_t p = 4 * tl; p < m; p += 4 * Team) {
      const uint4 g = groups[(p >> 2) * 32];
      const uint32_t js[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (uint32_t q = 0; q < 4u; ++q) {
        if (p + q >= m) break;
        double y[3], d[3], s2;
        load_pos(A.pos_in, js[q], y);
        const Dat64 b = load_dat(A.dat_in, js[q]);
        if (acc.near(y, d, s2)) acc.add(d, s2, b);
      }
    }
    if constexpr (Team > 1) {
      const unsigned mask = team_mask<Team>();
#pragma unroll
      for (int o = Team / 2; o > 0; o >>= 1) {
        acc.drho += __shfl_xor_sync(mask, acc.drho, o, Team);
#pragma unroll
        for (int k = 0; k < D; ++k) acc.dv[k] += __shfl_xor_sync(mask, acc.dv[k], o, Team);
      }
      if (tl != 0) return;
    }
    drho = acc.drho * T.list_s;
#pragma unroll
    for (int k = 0; k < D; ++k) dv[k] = acc.dv[k] * T.list_s;
    va[0] = acc.a.vx;
    va[1] = acc.a.vy;
    va[2] = acc.a.vz;
    rho_self = acc.a.rho;
  } else {
    ListPairF32<D, F, K, Phys> acc;
    acc.init(A, T, i);
    // B-splines: entries in the band around R^2 wait for the FP64 predicate
    // until the list is done (kBandCap of them; more take a second pass).
    // Wendland kernels need no predicate: beyond R their t is cut to 0, and
    // in the band t <= 2^-15 makes g at most t^3 = 2^-45 of its peak, below
    // the rounding of every sum it could enter.
    constexpr bool kBand = !KernelPoly<K>::deriv_over_q;
    const float lo = T.list_lo_f, hi = T.list_hi_f;
    extern __shared__ uint32_t s_band[];
    uint32_t* slots = s_band + threadIdx.x;
    uint32_t nb = 0;
    const auto pair = [&](const Dat32& b, uint32_t j) {
      float d[3];
      float s2 = acc.rab(b, d);
      if constexpr (kBand) {
        if (s2 >= lo && s2 <= hi) {
          if (nb < static_cast<uint32_t>(kBandCap)) slots[nb * blockDim.x] = j;
          ++nb;
        }
        // Entries beyond the radius add zero (the kernel vanishes at twice
        // the radius): no branch between the pairs.
        if (!(s2 < lo)) s2 = 4.f * hi;
      }
      acc.add(A, T, d, s2, b);
    };
    acc.open();
    uint32_t p = 4 * tl, done = 0;
    uint4 g = p < m ? groups[tl * 32] : make_uint4(0u, 0u, 0u, 0u);
    for (; p + 4u <= m; p += 4 * Team) {
      const uint32_t js[4] = {g.x, g.y, g.z, g.w};
      if (p + 4u * Team < m) g = groups[((p >> 2) + Team) * 32];  // the next entries
#pragma unroll
      for (uint32_t q0 = 0; q0 < 4u; q0 += kListBatch) {
        Dat32 b[kListBatch];
#pragma unroll
        for (uint32_t q = 0; q < kListBatch; ++q) b[q] = load_dat_wide(A.dat_in, js[q0 + q]);
#pragma unroll
        for (uint32_t q = 0; q < kListBatch; ++q) pair(b[q], js[q0 + q]);
      }
      if ((++done & 1u) == 0u) {
        acc.close();
        acc.open();
      }
    }
    if (p < m) {  // the last group, up to three entries
      pair(load_dat_wide(A.dat_in, g.x), g.x);
      if (p + 1u < m) pair(load_dat_wide(A.dat_in, g.y), g.y);
      if (p + 2u < m) pair(load_dat_wide(A.dat_in, g.z), g.z);
    }
    acc.close();
    if (kBand && nb != 0u) {
      const auto decide = [&](uint32_t j) {
        const Dat32 b = load_dat_wide(A.dat_in, j);
        float d[3];
        const float s2 = acc.rab(b, d);
        if (s2 < lo || s2 > hi) return;
        if (within_fp64<D>(A.pin, static_cast<uint32_t>(i), j, T.radius2)) {
          acc.add(A, T, d, s2, b);
        }
      };
      acc.open();
      if (nb <= static_cast<uint32_t>(kBandCap)) {
        for (uint32_t e = 0; e < nb; ++e) decide(slots[e * blockDim.x]);
      } else {
        for (uint32_t p = 4 * tl; p < m; p += 4 * Team) {
          const uint4 g = groups[(p >> 2) * 32];
          const uint32_t js[4] = {g.x, g.y, g.z, g.w};
          for (uint32_t q = 0; q < 4u && p + q < m; ++q) decide(js[q]);
        }
      }
      acc.close();
    }
    if constexpr (Team > 1) {
      const unsigned mask = team_mask<Team>();
#pragma unroll
      for (int o = Team / 2; o > 0; o >>= 1) {
        acc.drho.merge(__shfl_xor_sync(mask, acc.drho.s, o, Team),
                       __shfl_xor_sync(mask, acc.drho.c, o, Team));
#pragma unroll
        for (int k = 0; k < D; ++k) {
          acc.dv[k].merge(__shfl_xor_sync(mask, acc.dv[k].s, o, Team),
                          __shfl_xor_sync(mask, acc.dv[k].c, o, Team));
        }
      }
      if (tl != 0) return;
    }
    drho = acc.drho.value() * T.list_s_f;
#pragma unroll
    for (int k = 0; k < D; ++k) dv[k] = acc.dv[k].value() * T.list_s_f;
    va[0] = acc.a.vx;
    va[1] = acc.a.vy;
    va[2] = acc.a.vz;
    rho_self = acc.a.drho;
  }
  // Face boundaries divide by gamma and add the face terms before gravity.
  if (faces) {
    double drho_f = drho;
    double dv_f[3] = {static_cast<double>(dv[0]), static_cast<double>(dv[1]),
                      static_cast<double>(dv[2])};
    apply_face_terms(S, i, drho_f, dv_f);
    drho = static_cast<R>(drho_f);
#pragma unroll
    for (int k = 0; k < D; ++k) dv[k] = static_cast<R>(dv_f[k]);
  } else {
    dv[1] -= static_cast<R>(S.phys.g);
  }
  list_epilogue<D, F>(A, i, id, key, tk, T, va, rho_self, dv, drho);
}

}  // namespace tg
