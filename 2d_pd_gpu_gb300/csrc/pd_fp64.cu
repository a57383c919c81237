// FP64 explicit NOSB step (the plain form).  Compiled with --fmad=false: the
// only fused multiply-adds are the explicit fma() calls, written in the same
// places as the oracle's restatement, so results are bit-identical to it.
//
// Two threads per particle, one per component, bonds walked in family order
// through the SELL-32 layout (a warp's load of a slot is half a coalesced line).
// Per-particle sums are sequential in family order, with no atomics, so results
// are deterministic and independent of the launch shape.
//
// Reference correspondence (src/main_seq.cpp):
//   k_drift / pass B tail : applyVelocityBC :28-36, updatePositions :386-393,
//                           applyFixedBC :38-46
//   k_pass_a              : computeShapeTensors :71-156 (n1=n2=0: one K per
//                           particle), computeStressTensor :204-268,
//                           S = sigma K^-1 of computeForceDensityStates :355
//   k_pass_b              : computeVelocity :396-470 in gather form
//                           f_i = sum_j V_j (S_i + S_j) xi_ij (= T_ij - T_ji)
// FP64 operations per bond: pass A 11 (d 2, stretch test 5, D 4) + 2 with the
// zero-energy-mode penalty (sum V_j d), pass B 4.  The stretch test runs in
// FP64 only where stretch_fp32 cannot prove its outcome: about as near to the
// limit s2 |xi|^2 as the larger of 1e-6 s2 |xi|^2 and 2.4e-7 (|u_i| + |u_j|) |xi|
// (on a plate that has moved by 30 |xi|, at s_c = 5e-4: 1.4 % of the limit).  For
// nearly every bond pass A costs 8 FP64 operations.
#include "pd_internal.h"
#include "pd_walk.cuh"

namespace pd {

namespace {

__device__ __forceinline__ int64_t slot0(const Fp64Args& a, int64_t i, int* w) {
  const int64_t c = i >> 5;
  *w = a.chunk_w[c];
  return a.chunk_base[c] + (i & 31);
}

// Threads per block of the passes (32 particles): small blocks spread a small
// plate over the chip (200 x 200, per step: 43 us against 47 with 128 threads
// and 72 with 256) and end a large one evenly.
constexpr int kPairBlock = 64;
// Bonds per group of the passes' walks, two groups in flight (step with bonds
// breaking, us, pass A 1, 2, 3 bonds: 100 x 100 particles 16.8, 16.3, 16.2, 1M 686,
// 685, 711; pass B 2, 4: 1M 685, 710).  With bond breaking each thread of a pair
// runs the FP32 stretch test of one of a group's two bonds.
constexpr int kWalkA = 2, kWalkB = 2;
// Up to this many particles a pass lets the next one launch at its blocks' exit
// only: launched while some SMs still hold blocks of this pass, the next one's
// blocks crowd onto the others, and all of them fit at once, so nothing evens that
// out (step, us: 150 x 150 particles 23.6 -> 20.0, 170 x 170 31.4 -> 22.9, with bonds
// breaking 34 -> 23.6; 220 x 220 41.4 -> 37.0; 1M 686.4 against 687.3).
constexpr int64_t kExitTrigger = 60000;

// The passes run two threads per particle: thread h = 0 sums the x components
// (d11, d12, the penalty's x; f.x), h = 1 the y components.  Every sum keeps
// its operations and its order, none is computed twice, and each thread's
// serial chain of FP64 operations is half as long: an FP64 instruction keeps
// its SM quarter busy for 64 cycles, and that chain is what a plate too small
// to fill the chip waits for.
__device__ __forceinline__ double comp(const double2* p, int64_t i, int h) {
  return reinterpret_cast<const double*>(p)[2 * i + h];
}
__device__ __forceinline__ void set_comp(double2* p, int64_t i, int h, double v) {
  reinterpret_cast<double*>(p)[2 * i + h] = v;
}

// K^-1 and m/V of particle i over its intact bonds (oracle: kinv_of); true: singular
// (the caller counts it).
__device__ bool kinv_update(const Fp64Args& a, int64_t i) {
  int w;
  const int64_t s0 = slot0(a, i, &w);
  double k11 = 0.0, k12 = 0.0, k22 = 0.0, mx = 0.0, my = 0.0;
  int nal = 0;
  for (int k = 0; k < w; ++k) {
    const int64_t s = s0 + (int64_t)k * kChunk;
    if (a.nbr[s] < 0) continue;
    const double2 e = a.bxi[s];
    const double2 t = a.bgeo[s];
    k11 = fma(t.x, e.x, k11);
    k12 = fma(t.x, e.y, k12);
    k22 = fma(t.y, e.y, k22);
    mx = mx + t.x;
    my = my + t.y;
    ++nal;
  }
  const double det = fma(k11, k22, -(k12 * k12));
  const int32_t fam = a.fam[i];
  const bool failed = fam > 0 && (double)a.broken[i] / (double)fam > a.damage_fail;
  if (nal == 0 || failed || !(det > a.det_guard * (k11 * k22))) {
    a.kinv01[i] = make_double2(0.0, 0.0);
    a.kinv22[i] = 0.0;
    a.mt[i] = make_double2(0.0, 0.0);
    a.singular[i] = 1;
    return true;
  }
  const double r = 1.0 / det;
  a.kinv01[i] = make_double2(k22 * r, -k12 * r);
  a.kinv22[i] = k11 * r;
  const double rv = 1.0 / a.vol[i];
  a.mt[i] = make_double2(mx * rv, my * rv);
  a.singular[i] = 0;
  return false;
}

// From more than this many of a warp's particles on, each updates itself: the warp
// form takes ~19 FP64 instructions of the pipe per particle, one lane each ~180 in all
// (a step in which all of 1M particles lose bonds 1902 -> 1127 us, of which the counters'
// one addition per warp instead of per particle is most).
constexpr int kManyLost = 8;

// Pass A's update of the particles that lost bonds (newly > 0 in their lane):
// broken count, damage, K^-1 and m/V, by the whole warp.  Eight lanes take a
// particle, four particles at a time: lanes 0 .. 4 each sum one of k11, k12,
// k22, mx, my in family order, lanes 0 .. 2 share one division (1 / det,
// 1 / V, damage) and lanes 0 .. 4 one product; kinv_update's operations
// (x + t is fma(t, 1, x)).  One thread alone has a chain of ~240 dependent FP64
// operations here instead of ~45, each of which waits for its turn on the pipe,
// and its pass waits for it (300 x 300 plate with bonds breaking, pass A:
// 87 us against 72).
__device__ __noinline__ void kinv_update_warp(const Fp64Args& a, int64_t i, int64_t s0, int w, int newly) {
  const int lane = threadIdx.x & 31, c = lane & 7, g0 = lane & 24;
  unsigned todo = __ballot_sync(0xffffffffu, newly > 0);
  if (__popc(todo) > kManyLost) {
    bool bad = false;
    if (newly > 0) {
      const int32_t broken = a.broken[i] + newly;
      a.broken[i] = broken;
      a.damage[i] = (double)broken / (double)a.fam[i];
      bad = kinv_update(a, i);
    }
    const int all = __reduce_add_sync(0xffffffffu, newly), nbad = __popc(__ballot_sync(0xffffffffu, bad));
    if (lane == 0) {
      atomicAdd(a.counters + CNT_BROKEN, (unsigned long long)all);
      if (nbad) atomicAdd(a.counters + CNT_SINGULAR, (unsigned long long)nbad);
    }
    return;
  }
  while (todo) {
    unsigned rest = todo;  // this lane's particle: that of the (lane / 8)-th lane left to do
    for (int q = lane >> 3; q > 0; --q) rest &= rest - 1;
    const bool have = rest != 0;
    const int src = have ? __ffs((int)rest) - 1 : 0;
    const int64_t gi = __shfl_sync(0xffffffffu, i, src), gs = __shfl_sync(0xffffffffu, s0, src);
    const int gw = __shfl_sync(0xffffffffu, w, src), gn = __shfl_sync(0xffffffffu, newly, src);
    double sum = 0.0, num = 1.0, den = 1.0;
    int nal = 0, broken = 0, fam = 1;
    if (have) {
      broken = a.broken[gi] + gn;
      fam = a.fam[gi];
      if (c == 1) den = a.vol[gi];
      if (c == 2) {
        num = (double)broken;
        den = (double)fam;
      }
      const double* P = reinterpret_cast<const double*>(a.bgeo) + (c == 2 || c == 4 ? 1 : 0);  // V_j xi
      const double* Q = reinterpret_cast<const double*>(a.bxi) + (c == 0 ? 0 : 1);             // xi
      if (c < 5) {
#pragma unroll 4
        for (int k = 0; k < gw; ++k) {
          const int64_t s = gs + (int64_t)k * kChunk;
          const bool live = a.nbr[s] >= 0;
          const double p = P[2 * s], q = c < 3 ? Q[2 * s] : 1.0;
          if (live) {
            sum = fma(p, q, sum);
            ++nal;
          }
        }
      }
    }
    const double k11 = __shfl_sync(0xffffffffu, sum, g0), k12 = __shfl_sync(0xffffffffu, sum, g0 + 1),
                 k22 = __shfl_sync(0xffffffffu, sum, g0 + 2);
    nal = __shfl_sync(0xffffffffu, nal, g0);
    const double det = fma(k11, k22, -(k12 * k12));
    if (c == 0) den = det;
    const double quo = num / den;
    const double r = __shfl_sync(0xffffffffu, quo, g0), rv = __shfl_sync(0xffffffffu, quo, g0 + 1),
                 damage = __shfl_sync(0xffffffffu, quo, g0 + 2);
    const bool bad = nal == 0 || damage > a.damage_fail || !(det > a.det_guard * (k11 * k22));
    if (have) {
      const double x = c == 0 ? k22 : c == 1 ? -k12 : c == 2 ? k11 : sum;
      const double out = bad ? 0.0 : x * (c < 3 ? r : rv);
      if (c < 2)
        set_comp(a.kinv01, gi, c, out);
      else if (c == 2)
        a.kinv22[gi] = out;
      else if (c < 5)
        set_comp(a.mt, gi, c - 3, out);
      else if (c == 5)
        a.singular[gi] = bad ? 1 : 0;
      else if (c == 6) {
        a.broken[gi] = broken;
        a.damage[gi] = damage;
      } else {
        atomicAdd(a.counters + CNT_BROKEN, (unsigned long long)gn);
        if (bad) atomicAdd(a.counters + CNT_SINGULAR, 1ull);
      }
    }
    for (int q = 0; q < 4 && todo; ++q) todo &= todo - 1;
  }
}

__global__ void __launch_bounds__(kBlock) k_init_geometry(Fp64Args a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n && kinv_update(a, i)) atomicAdd(a.counters + CNT_SINGULAR, 1ull);
}

// Velocity BC, drift, fixed BC of particle i; an = f_i / rho.
__device__ __forceinline__ void drift_one(const Fp64Args& a, int64_t i, double2& v, double2& u, double anx,
                                          double any) {
  const int g = a.bc[i];
  const int kind = g ? a.gkind[g - 1] : PD_BC_NONE;
  if (kind == PD_BC_VELOCITY) v = a.gval[g - 1];
  u.x = u.x + (v.x * a.dt + (0.5 * anx) * a.dt2);
  u.y = u.y + (v.y * a.dt + (0.5 * any) * a.dt2);
  if (kind == PD_BC_FIXED) u = make_double2(0.0, 0.0);
}

__device__ __forceinline__ void drift_particle(const Fp64Args& a, int64_t i) {
  double2 v = a.in_v ? a.in_v[i] : a.v[i], u = a.in_u ? a.in_u[i] : a.u[i];
  const double2 f = a.in_f ? a.in_f[i] : a.f[i];
  if (a.in_f) a.f[i] = f;
  drift_one(a, i, v, u, f.x * a.inv_rho, f.y * a.inv_rho);
  a.v[i] = v;
  a.u[i] = u;
  a.u32[i] = make_float2((float)u.x, (float)u.y);
}

__global__ void __launch_bounds__(kBlock) k_drift(Fp64Args a) {
  const int64_t i = a.i0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n) drift_particle(a, i);
}

// The FP32 shadow of u for particles i0 <= i < n; with in_u / in_v / in_a
// set (pd_compute_velocity on page-locked buffers), u, velocity and acce are
// first read from host memory into the device state.
__global__ void __launch_bounds__(kBlock) k_shadow(Fp64Args a) {
  const int64_t i = a.i0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double2 u = a.in_u ? a.in_u[i] : a.u[i];
  if (a.in_u) a.u[i] = u;
  if (a.in_v) a.v[i] = a.in_v[i];
  if (a.in_a) a.acc[i] = a.in_a[i];
  a.u32[i] = make_float2((float)u.x, (float)u.y);
}

// The stretch test in FP32 from the shadows of u and xi: 1 the FP64 test would
// say intact, -1 it would say broken, 0 too close to call (the FP64 test runs).
// With f = fl32(u32_j - u32_i), S_c = 2|xi_c| + |f_c| and delta_c a bound on
// |f_c - d_c| (the shadows' and the difference's rounding, <= 2^-24 each of
// |u_j|, |u_i| and |f|), the FP64 test's q = d.(2 xi + d) differs from
// f.(2 xi + f) by at most sum delta_c (2 S_c + delta_c), and xi's and the
// evaluation's rounding add at most 4 * 2^-24 sum |f_c| S_c; the limit's own
// relative error is below 6 * 2^-24.  The margins taken (6.0e-8, 3e-7 and 1e-6)
// are above these and the FP64 evaluation's ~1e-15.  These are relative errors, which
// hold while nothing that counts is below FP32's normal range (s2 itself, |xi|^2, the
// limit): limits outside 1e-30 .. 1e30 leave it to FP64, so do infinities and NaN, and
// outside 1e-30 <= s2 <= 1e6 the host passes s2 = 0, a limit of 0.  Inside, |xi|^2 >=
// 1e-36, and what underflows elsewhere is below 1e-36 of a limit's 1e-30.
// A test that bounds |d| alone leaves every rotating or compressed bond to FP64
// too, which in the few warps of a fracture zone is what the whole pass waits
// for (300 x 300 plate with bonds breaking: see k_pass_a).
__device__ __forceinline__ int stretch_fp32(float2 ui, float2 uj, float2 e, float s2) {
  const float fx = uj.x - ui.x, fy = uj.y - ui.y;
  const float dx = 6.0e-8f * (fabsf(uj.x) + fabsf(ui.x) + fabsf(fx));
  const float dy = 6.0e-8f * (fabsf(uj.y) + fabsf(ui.y) + fabsf(fy));
  const float sx = fmaf(2.0f, fabsf(e.x), fabsf(fx)), sy = fmaf(2.0f, fabsf(e.y), fabsf(fy));
  const float q = fmaf(fx, fmaf(2.0f, e.x, fx), fy * fmaf(2.0f, e.y, fy));
  const float err = fmaf(3.0e-7f, fmaf(fabsf(fx), sx, fabsf(fy) * sy),
                         fmaf(dx, fmaf(2.0f, sx, dx), dy * fmaf(2.0f, sy, dy)));
  const float lim = s2 * fmaf(e.x, e.x, e.y * e.y);
  if (!(lim > 1.0e-30f && lim < 1.0e30f)) return 0;
  if (q + err < 0.999999f * lim) return 1;
  return q - err > 1.000001f * lim ? -1 : 0;
}

// The same in FP64 (the oracle's operations).
__device__ __noinline__ bool stretch_fp64(const Fp64Args& a, int64_t i, int64_t j, int64_t s) {
  const double2 e = a.bxi[s], ui = a.u[i], uj = a.u[j];
  const double dx = uj.x - ui.x, dy = uj.y - ui.y;
  return fma(dx, fma(2.0, e.x, dx), dy * fma(2.0, e.y, dy)) > a.s2 * fma(e.x, e.x, e.y * e.y);
}

// Additions and products as fma, with the constant in a register: on this GPU a
// DFMA of three registers leaves the FP64 pipe in 16 cycles per warp and SM; a
// DADD, a DMUL, or a DFMA with an operand from the arguments or an immediate,
// in 19 (measured, 4 to 16 warps).  x + y = fma(x, 1, y) and x y = fma(x, y, -0)
// round the same exact value once and keep the sign of a zero.
struct FpConst {
  double one, neg_one, neg_zero;
};
// A value the compiler cannot place in a uniform register or fold (all lanes call it).
__device__ __forceinline__ double in_register(double x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ FpConst fp_const(const Fp64Args& a) {
  return FpConst{in_register(a.one), in_register(a.neg_one), in_register(a.neg_zero)};
}
__device__ __forceinline__ double add1(const FpConst& a, double x, double y) { return fma(x, a.one, y); }
__device__ __forceinline__ double sub1(const FpConst& a, double x, double y) { return fma(y, a.neg_one, x); }
__device__ __forceinline__ double mul1(const FpConst& a, double x, double y) { return fma(x, y, a.neg_zero); }

// Pass A's stretch tests of particle i ahead of its sums, its bonds dealt to the two threads of
// the pair in turn; broken ones are marked.  Returns the number this thread broke, and the number it left intact.
constexpr int kTests = 7;  // in flight (1M particles: 2, 4, 7, 14: 712, 696, 684, 682 us per step at 10 blocks per SM)
__device__ __forceinline__ int test_bonds(const Fp64Args& a, int64_t i, int h, int64_t s0, int w, float2 ui32,
                                          int* intact) {
  int newly = 0, live = 0, jn[kTests];
  auto indices = [&](int k) {
#pragma unroll
    for (int q = 0; q < kTests; ++q) jn[q] = k + 2 * q < w ? a.nbr[s0 + (int64_t)(k + 2 * q) * kChunk] : -1;
  };
  indices(h);
  for (int k = h; k < w; k += 2 * kTests) {
    int j[kTests], least = 1;
    float2 u[kTests], e[kTests];
#pragma unroll
    for (int q = 0; q < kTests; ++q) {
      j[q] = jn[q];
      u[q] = a.u32[j[q] < 0 ? i : (int64_t)j[q]];
      e[q] = __ldcs(&a.bxi32[j[q] < 0 ? s0 : s0 + (int64_t)(k + 2 * q) * kChunk]);
    }
    indices(k + 2 * kTests);
    int v[kTests];
#pragma unroll
    for (int q = 0; q < kTests; ++q) {
      v[q] = j[q] >= 0 ? stretch_fp32(ui32, u[q], e[q], a.s2f) : 1;
      least = min(least, v[q]);
      live += j[q] >= 0 ? 1 : 0;
    }
    if (least <= 0) {
#pragma unroll
      for (int q = 0; q < kTests; ++q) {
        const int64_t s = s0 + (int64_t)(k + 2 * q) * kChunk;
        if (v[q] <= 0 && (v[q] < 0 || stretch_fp64(a, i, j[q], s))) {
          a.nbr[s] = -2 - j[q];
          ++newly;
        }
      }
    }
  }
  *intact = live - newly;
  return newly;
}

// From this many particles (of the plate) on, pass A tests a particle's bonds before it sums them:
// the sums then need 80 registers instead of 96 and no branch, and other warps' sums keep the FP64
// pipe busy under the tests (step with bonds breaking, us, 500 x 500 particles 176.7 -> 175.9,
// 800 x 800 441 -> 435, 1M 683.5 -> 672, 2M 1356 -> 1329).  A smaller plate waits for the tests
// (400 x 400 117.5 -> 118.1, 100 x 100 15.3 -> 15.9).  Where fewer than 3/4 of a warp's slots hold
// intact bonds it takes them one by one and leaves out those that no lane has a bond in (1M particles,
// all but 10 M of 28 M bonds broken: 697 -> 518 us).
constexpr int64_t kTestsFirst = 250000;

// Pass A of component h of particle i (stretch tests, D, penalty sum, stress,
// W).  All 32 lanes of the warp call it, lanes 2k and 2k + 1 with the same
// particle; ok = false: the lane has none.
// Bonds are taken kWalkA at a time: while one group's terms are summed the next
// one's bond data and neighbours' state are on their way, and the indices of the
// one after it.  Without bond breaking a group has no branch (an empty slot's terms
// are -0, which changes no sum).  In a plate too small to fill the chip a warp has
// its SM quarter to itself and waits for each of these in turn (step, us, against
// one group at a time: 30 x 31 particles 17.4 -> 13.5, with bonds breaking 16.5 ->
// 13.7; 100 x 100 17.7 -> 14.5, 17.4 -> 15.5; 401 x 399 120.4 -> 113.9, 120.9 ->
// 117.5; 1M 683 -> 664, 688 -> 683; 250 x 250 52.2 -> 49.8, but 51.7 -> 52.6).
template <bool BREAK, bool HG, bool TESTS_FIRST>
__device__ __forceinline__ void pass_a_particle(const Fp64Args& a, int64_t i, int h, bool ok) {
  int w = 0;
  int64_t s0 = 0;
  double ui = 0.0;
  float2 ui32 = make_float2(0.f, 0.f);
  if (ok) {
    s0 = slot0(a, i, &w);
    ui = comp(a.u, i, h);
    if (BREAK) ui32 = a.u32[i];
  }
  const FpConst K = fp_const(a);
  double d1 = 0.0, d2 = 0.0, ah = 0.0;  // row h of D, component h of the penalty sum
  int newly = 0;
  bool few = false;                             // (the warp's) fewer than 3/4 of the slots hold intact bonds
  constexpr bool TEST = BREAK && !TESTS_FIRST;  // among the sums
  if (BREAK && TESTS_FIRST) {
    int intact;
    newly = test_bonds(a, i, h, s0, w, ui32, &intact);
    newly += __shfl_xor_sync(0xffffffffu, newly, 1);
    __syncwarp();  // (the marks are read by both threads)
    few = 4 * (int)__reduce_add_sync(0xffffffffu, intact) < 3 * (int)__reduce_add_sync(0xffffffffu, w) / 2;
  }
  const float s2 = TEST ? a.s2f : 0.f;
  struct Group {
    int j[kWalkA];
    double uj[kWalkA], vj[kWalkA];
    double2 t[kWalkA];
    float2 uj32, e32;  // of the bond this thread tests
  };
  static_assert(!TEST || kWalkA == 2, "one bond of a group for each thread of the pair to test");
  const int most = TEST ? __reduce_max_sync(0xffffffffu, w) : w;  // (the pair exchanges run in every lane)
  const int64_t self = TEST && !ok ? a.n - 1 : i;                 // what an empty slot reads
  int jn[kWalkA];
  auto indices = [&](int k) {
#pragma unroll
    for (int q = 0; q < kWalkA; ++q) jn[q] = k + q < w ? a.nbr[s0 + (int64_t)(k + q) * kChunk] : -1;
  };
  auto request = [&](Group& g, int k) {
    const int64_t s = s0 + (int64_t)k * kChunk;
#pragma unroll
    for (int q = 0; q < kWalkA; ++q) {
      g.j[q] = jn[q];
      const int64_t jj = g.j[q] < 0 ? self : (int64_t)g.j[q];
      const int64_t sq = g.j[q] < 0 ? s0 : s + (int64_t)q * kChunk;
      g.uj[q] = comp(a.u, jj, h);
      g.t[q] = __ldcs(&a.bgeo[sq]);
      if (HG) g.vj[q] = a.vol[jj];
    }
    if (TEST) {
      const int jo = h ? g.j[1] : g.j[0];
      g.uj32 = a.u32[jo < 0 ? self : (int64_t)jo];
      g.e32 = __ldcs(&a.bxi32[jo < 0 ? s0 : s + (int64_t)h * kChunk]);
    }
  };
  auto sums = [&](const Group& g, int k) {
    int v[2] = {1, 1};
    if (TEST) {  // (both bonds tested by both threads: 100 x 100 particles 16.0 against 15.5 us per step)
      const int mine = stretch_fp32(ui32, g.uj32, g.e32, s2), other = __shfl_xor_sync(0xffffffffu, mine, 1);
      v[0] = h ? other : mine;
      v[1] = h ? mine : other;
    }
#pragma unroll
    for (int q = 0; q < kWalkA; ++q) {
      const bool on = g.j[q] >= 0;
      if (TEST) {
        if (!on) continue;
        const int64_t s = s0 + (int64_t)(k + q) * kChunk;
        if (v[q] <= 0 && (v[q] < 0 || stretch_fp64(a, i, g.j[q], s))) {
          // both threads of the pair find the same; the second one does not store, and if it
          // reads the slot after the first one's store it skips the bond there
          if (h == 0) a.nbr[s] = -2 - g.j[q];
          ++newly;
          continue;
        }
      }
      const double dh = TEST || on ? sub1(K, g.uj[q], ui) : -0.0;
      d1 = fma(dh, TEST || on ? g.t[q].x : 1.0, d1);
      d2 = fma(dh, TEST || on ? g.t[q].y : 1.0, d2);
      if (HG) ah = fma(TEST || on ? g.vj[q] : 1.0, dh, ah);
    }
  };
  if (BREAK && TESTS_FIRST && few) {  // slots that no lane has a bond in cost nothing here
    const int widest = __reduce_max_sync(0xffffffffu, w);  // (every lane votes)
    const int64_t mine = ok ? i : a.n - 1;
#pragma unroll 1
    for (int k = 0; k < widest; ++k) {
      const int64_t s = k < w ? s0 + (int64_t)k * kChunk : s0;
      const int j = k < w ? a.nbr[s] : -1;
      if (!__any_sync(0xffffffffu, j >= 0)) continue;  // (a vote: predicated off, the sums would keep the pipe busy)
      const bool on = j >= 0;
      const int64_t jj = on ? (int64_t)j : mine;
      const double dh = on ? sub1(K, comp(a.u, jj, h), ui) : -0.0;
      const double2 t = a.bgeo[s];
      d1 = fma(dh, on ? t.x : 1.0, d1);
      d2 = fma(dh, on ? t.y : 1.0, d2);
      if (HG) ah = fma(on ? a.vol[jj] : 1.0, dh, ah);
    }
  } else if (most > 0) {
    Group g0, g1;
    indices(0);
    request(g0, 0);
    indices(kWalkA);
    for (int k = 0; k < most; k += 2 * kWalkA) {
      request(g1, k + kWalkA);
      indices(k + 2 * kWalkA);
      sums(g0, k);
      request(g0, k + 2 * kWalkA);
      indices(k + 3 * kWalkA);
      if (k + kWalkA < most) sums(g1, k + kWalkA);
    }
  }
  // late, so that the next pass's blocks do not take the places of this pass's waiting ones
  if (!a.exit_trigger) grid_dep_launch();
  if (HG && ok) set_comp(a.hg, i, h, mul1(K, a.k_hg2, ah));
  if (BREAK) {
    if (TEST) newly = __shfl_sync(0xffffffffu, newly, threadIdx.x & 30);  // the first thread's count
    if (__any_sync(0xffffffffu, newly != 0)) {
      __syncwarp();  // (other lanes read the marks)
      kinv_update_warp(a, i, s0, w, h == 0 ? newly : 0);
      __syncwarp();  // (its stores, by either form, are read below by both threads of a pair)
    }
  }
  double2 k01 = make_double2(0.0, 0.0);
  double k22 = 0.0, vi = 0.0;
  bool singular = true;
  if (ok) {
    singular = a.singular[i];
    k01 = a.kinv01[i];
    k22 = a.kinv22[i];
    vi = a.vol[i];
  }
  const double k11 = k01.x, k12 = k01.y;
  // row h of G = D K^-1 = F - I, and of the symmetric stress: thread 0 has
  // (s11, s12), thread 1 (s12, s22)
  const double g1 = fma(d1, k11, mul1(K, d2, k12)), g2 = fma(d1, k12, mul1(K, d2, k22));
  const double diag = h ? g2 : g1, other = __shfl_xor_sync(0xffffffffu, diag, 1);
  const double off = h ? g1 : g2, cross = __shfl_xor_sync(0xffffffffu, off, 1);
  const double e11 = h ? other : diag, e22 = h ? diag : other, e12 = mul1(K, 0.5, add1(K, off, cross));
  const double sd = fma(h ? a.c12 : a.c11, e11, mul1(K, h ? a.c11 : a.c12, e22));
  const double s12 = mul1(K, a.c33, e12);
  const double sa = h ? s12 : sd, sb = h ? sd : s12;
  if (!ok) return;
  double w1 = fma(sa, k11, mul1(K, sb, k12)), w2 = fma(sa, k12, mul1(K, sb, k22));
  if (HG) {  // W = V (sigma K^-1 - k G)
    const double kh = -a.k_hg;
    w1 = fma(kh, g1, w1);
    w2 = fma(kh, g2, w2);
  }
  double2 W = make_double2(mul1(K, vi, w1), mul1(K, vi, w2));
  if (singular) W = make_double2(0.0, 0.0);
  (h ? a.w23 : a.w01)[i] = W;
}

// (10 blocks per SM, pass B 12: with registers to spare the compiler keeps the walk's
// loads where they stand; left to itself it saves registers and moves them to their uses)
template <bool BREAK, bool HG, bool TESTS_FIRST = false>
__global__ void __launch_bounds__(kPairBlock, TESTS_FIRST ? 12 : 10) k_pass_a(Fp64Args a) {
  const int64_t i = a.i0 + (int64_t)blockIdx.x * (kPairBlock / 2) + (threadIdx.x >> 1);
  grid_dep_wait();  // nothing is read before the previous pass has completed
  pass_a_particle<BREAK, HG, TESTS_FIRST>(a, i, threadIdx.x & 1, i < a.n);
}

// Pass B of component h of particle i (force gather, kick; MODE 1 adds the
// next drift, MODE 2 is the drop-in kick with acce in/out).
template <int MODE, bool HG>
__device__ __forceinline__ void pass_b_particle(const Fp64Args& a, const FpConst& K, int64_t i, int h) {
  int w;
  const int64_t s0 = slot0(a, i, &w);
  const double2* W = h ? a.w23 : a.w01;
  const double2 wi = W[i], m = a.mt[i];
  double f = fma(wi.x, m.x, HG ? fma(wi.y, m.y, comp(a.hg, i, h)) : mul1(K, wi.y, m.y));
  // requested before the walk (1M-particle plate: 252 -> 243 us)
  double v = comp(a.v, i, h), ao = comp(MODE == 2 ? a.acc : a.f, i, h), u = MODE == 1 ? comp(a.u, i, h) : 0.0;
  struct Group {
    int j[kWalkB];
    double2 nb[kWalkB], e[kWalkB];
  };
  int jn[kWalkB];
  auto indices = [&](int k) {
#pragma unroll
    for (int q = 0; q < kWalkB; ++q) jn[q] = k + q < w ? __ldcs(&a.nbr[s0 + (int64_t)(k + q) * kChunk]) : -1;
  };
  auto request = [&](Group& g, int k) {
    const int64_t s = s0 + (int64_t)k * kChunk;
#pragma unroll
    for (int q = 0; q < kWalkB; ++q) {
      g.j[q] = jn[q];
      g.nb[q] = W[g.j[q] < 0 ? i : (int64_t)g.j[q]];
      g.e[q] = __ldcs(&a.bxi[g.j[q] < 0 ? s0 : s + (int64_t)q * kChunk]);
    }
  };
  auto sums = [&](const Group& g) {
#pragma unroll
    for (int q = 0; q < kWalkB; ++q) {
      if (g.j[q] < 0) continue;
      f = fma(g.nb[q].x, g.e[q].x, f);
      f = fma(g.nb[q].y, g.e[q].y, f);
    }
  };
  if (w > 0) {
    Group g0, g1;
    indices(0);
    request(g0, 0);
    indices(kWalkB);
    for (int k = 0; k < w; k += 2 * kWalkB) {
      request(g1, k + kWalkB);
      indices(k + 2 * kWalkB);
      sums(g0);
      request(g0, k + 2 * kWalkB);
      indices(k + 3 * kWalkB);
      sums(g1);
    }
  }
  if (!a.exit_trigger) grid_dep_launch();
  if (MODE != 2) ao = mul1(K, ao, a.inv_rho);
  const double an = mul1(K, f, a.inv_rho);
  v = add1(K, v, mul1(K, mul1(K, 0.5, add1(K, ao, an)), a.dt));
  set_comp(a.f, i, h, f);
  if (MODE == 2) set_comp(a.acc, i, h, an);
  if (MODE == 1) {  // drift_one of the component
    const int g = a.bc[i];
    const int kind = g ? a.gkind[g - 1] : PD_BC_NONE;
    if (kind == PD_BC_VELOCITY) v = comp(a.gval, g - 1, h);
    u = add1(K, u, add1(K, mul1(K, v, a.dt), mul1(K, mul1(K, 0.5, an), a.dt2)));
    if (kind == PD_BC_FIXED) u = 0.0;
    set_comp(a.u, i, h, u);
    reinterpret_cast<float*>(a.u32)[2 * i + h] = (float)u;
  }
  set_comp(a.v, i, h, v);
  if (a.out_v) {  // pd_step_host's last pass, or the drop-in call: the results straight to host memory
    if (MODE == 2)
      set_comp(a.out_a, i, h, an);
    else
      set_comp(a.out_u, i, h, MODE == 1 ? u : comp(a.u, i, h));
    set_comp(a.out_v, i, h, v);
    set_comp(a.out_f, i, h, f);
  }
}

template <int MODE, bool HG>
__global__ void __launch_bounds__(kPairBlock, 12) k_pass_b(Fp64Args a) {
  const int64_t i = a.i0 + (int64_t)blockIdx.x * (kPairBlock / 2) + (threadIdx.x >> 1);
  grid_dep_wait();
  const FpConst K = fp_const(a);
  if (i < a.n) pass_b_particle<MODE, HG>(a, K, i, threadIdx.x & 1);
}

// ---- batched plates: phase 0 drift, 1 pass A, 2 pass B + next drift, 3 pass B
// (ok = false: a lane past the tile's end, which only the warp-wide parts call for)
__device__ __forceinline__ void batch_particle(const Fp64Args& p, int64_t i, int h, bool ok, int phase) {
  const bool hg = p.k_hg != 0.0;
  if (phase == 0) {
    if (ok && h == 0) drift_particle(p, i);
  } else if (phase == 1) {
    if (p.brk)
      hg ? pass_a_particle<true, true, false>(p, i, h, ok) : pass_a_particle<true, false, false>(p, i, h, ok);
    else
      hg ? pass_a_particle<false, true, false>(p, i, h, ok) : pass_a_particle<false, false, false>(p, i, h, ok);
  } else {
    const FpConst K = fp_const(p);
    if (!ok) return;
    if (phase == 2)
      hg ? pass_b_particle<1, true>(p, K, i, h) : pass_b_particle<1, false>(p, K, i, h);
    else
      hg ? pass_b_particle<0, true>(p, K, i, h) : pass_b_particle<0, false>(p, K, i, h);
  }
}

__device__ __forceinline__ void batch_phase(const Fp64Args* __restrict__ plates, const BatchTile* __restrict__ tiles,
                                            int ntiles, int phase) {
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchTile T = tiles[t];
    const Fp64Args& p = plates[T.plate];
    for (int k0 = 0; k0 < 2 * T.count; k0 += blockDim.x) {  // whole warps in every round
      const int k = k0 + threadIdx.x;
      batch_particle(p, T.first + (k >> 1), k & 1, k < 2 * T.count, phase);
    }
  }
}

__global__ void __launch_bounds__(256) k_batch_persistent(const Fp64Args* __restrict__ plates,
                                                          const BatchTile* __restrict__ tiles, int ntiles, int nsteps,
                                                          GridBarrier* bar, const BarrierLimits lim) {
  const unsigned nb = gridDim.x;
  batch_phase(plates, tiles, ntiles, 0);
  for (int s = 0; s < nsteps; ++s) {
    if (!grid_sync(bar, nb, lim)) return;
    batch_phase(plates, tiles, ntiles, 1);
    if (!grid_sync(bar, nb, lim)) return;
    batch_phase(plates, tiles, ntiles, s + 1 < nsteps ? 2 : 3);
  }
}

__global__ void __launch_bounds__(256) k_batch_phase(const Fp64Args* __restrict__ plates,
                                                     const BatchTile* __restrict__ tiles, int ntiles, int phase) {
  batch_phase(plates, tiles, ntiles, phase);
}

}  // namespace

int batch_occupancy_fp64(const BatchLaunch& cfg) {
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_batch_persistent, cfg.block, 0) != cudaSuccess) return 0;
  return nb;
}

cudaError_t launch_batch_fp64(const Fp64Args* d_plates, const BatchTile* d_tiles, int ntiles, int nsteps,
                              const BatchLaunch& cfg, GridBarrier* d_bar, int nsm, cudaStream_t s) {
  if (ntiles <= 0 || nsteps <= 0) return cudaSuccess;
  if (!cfg.persistent) {
    const unsigned g = (unsigned)ntiles;
    k_batch_phase<<<g, cfg.block, 0, s>>>(d_plates, d_tiles, ntiles, 0);
    for (int k = 0; k < nsteps; ++k) {
      k_batch_phase<<<g, cfg.block, 0, s>>>(d_plates, d_tiles, ntiles, 1);
      k_batch_phase<<<g, cfg.block, 0, s>>>(d_plates, d_tiles, ntiles, k + 1 < nsteps ? 2 : 3);
    }
    return cudaGetLastError();
  }
  int occ = batch_occupancy_fp64(cfg);
  int bps = cfg.blocks_per_sm < occ ? cfg.blocks_per_sm : occ;
  if (bps < 1) return cudaErrorInvalidConfiguration;
  int grid = nsm * bps;
  if (grid > ntiles) grid = ntiles;
  cudaError_t e = cudaMemsetAsync(d_bar, 0, sizeof(GridBarrier), s);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)grid);
  lc.blockDim = dim3((unsigned)cfg.block);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, k_batch_persistent, d_plates, d_tiles, ntiles, nsteps, d_bar, cfg.limits);
}

namespace {
// reach[k] / low[k] = the largest / smallest id among slab k's particles
// (k*slab .. k*slab + slab - 1) and their neighbours
__global__ void k_slab_reach(int64_t n, const int64_t* __restrict__ row_ptr, const int32_t* __restrict__ col,
                             int64_t slab, int32_t* reach, int32_t* low) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t m = (int32_t)i, l = (int32_t)i;
  for (int64_t k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
    m = col[k] > m ? col[k] : m;
    l = col[k] < l ? col[k] : l;
  }
  atomicMax(&reach[i / slab], m);
  atomicMin(&low[i / slab], l);
}
}  // namespace

void launch_slab_reach(int64_t n, const int64_t* row_ptr, const int32_t* col, int64_t slab, int32_t* reach,
                       int32_t* low, cudaStream_t s) {
  if (n > 0) k_slab_reach<<<(unsigned)blocks_for(n), kBlock, 0, s>>>(n, row_ptr, col, slab, reach, low);
}

void launch_init_geometry_fp64(const Fp64Args& a, cudaStream_t s) {
  if (a.n > 0) k_init_geometry<<<(unsigned)blocks_for(a.n), kBlock, 0, s>>>(a);
}

void launch_drift_fp64(const Fp64Args& a, cudaStream_t s) {
  if (a.n > a.i0) k_drift<<<(unsigned)blocks_for(a.n - a.i0), kBlock, 0, s>>>(a);
}

void launch_shadow_fp64(const Fp64Args& a, cudaStream_t s) {
  if (a.n > a.i0) k_shadow<<<(unsigned)blocks_for(a.n - a.i0), kBlock, 0, s>>>(a);
}

// pdl: launched with programmatic stream serialization (the blocks start
// while the previous kernel on the stream drains, and wait for it first).
static void launch_pass(void (*kernel)(Fp64Args), const Fp64Args& a, bool pdl, cudaStream_t s) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3((unsigned)blocks_for(2 * (a.n - a.i0), kPairBlock));
  lc.blockDim = dim3(kPairBlock);
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = pdl ? 1 : 0;
  Fp64Args b = a;
  b.exit_trigger = a.exit_trigger && a.n - a.i0 <= kExitTrigger;
  cudaLaunchKernelEx(&lc, kernel, b);
}

void launch_pass_a_fp64(const Fp64Args& a, bool breaking, cudaStream_t s, bool pdl) {
  if (a.n <= a.i0) return;
  const bool hg = a.k_hg != 0.0;
  if (breaking && a.plate >= kTestsFirst)
    launch_pass(hg ? k_pass_a<true, true, true> : k_pass_a<true, false, true>, a, pdl, s);
  else if (breaking)
    launch_pass(hg ? k_pass_a<true, true> : k_pass_a<true, false>, a, pdl, s);
  else
    launch_pass(hg ? k_pass_a<false, true> : k_pass_a<false, false>, a, pdl, s);
}

void launch_pass_b_fp64(const Fp64Args& a, int mode, cudaStream_t s, bool pdl) {
  if (a.n <= a.i0) return;
  const bool hg = a.k_hg != 0.0;
  if (mode == 0)
    launch_pass(hg ? k_pass_b<0, true> : k_pass_b<0, false>, a, pdl, s);
  else if (mode == 1)
    launch_pass(hg ? k_pass_b<1, true> : k_pass_b<1, false>, a, pdl, s);
  else
    launch_pass(hg ? k_pass_b<2, true> : k_pass_b<2, false>, a, pdl, s);
}

}  // namespace pd
