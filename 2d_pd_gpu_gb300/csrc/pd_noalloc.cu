// pd_compute_velocity_noalloc: one FP64 force + kick on caller-owned device
// buffers, for callers that must not allocate device memory.
//
// Who needs it: a host application that owns every device allocation through
// its own pool (and forbids other allocators in its address space), and code
// on a latency-critical path, where cudaMalloc/cudaFree would synchronise
// the device.  Such a caller hands in its own buffers for inputs and
// outputs; the only memory beyond them is the per-particle scratch between
// the two kernels (W, m / V and the zero-energy-mode penalty term, 8 doubles
// per particle), and that lives in the file-scope array below, sized for
// PD_NOALLOC_MAX_PARTICLES particles (8 * 8 * 65536 B = 4 MiB, held by every
// device that loads the library until the process exits).
//
// The arithmetic is the FP64 form's, operation for operation (this file is
// compiled with --fmad=false, like pd_fp64.cu), walking the caller's CSR
// families directly; with the same inputs and no broken bonds its results
// equal pd_compute_velocity's bit for bit.
//
// The caller's CSR is checked on the device as it is walked: a particle whose
// row is not a range inside [row_ptr[0] = 0, row_ptr[n]], or whose family
// names an index outside [0, n), reads nothing out of range and gets NaN in
// its velocity, acce and netF (so do the particles whose families reach it),
// which the caller sees in its own outputs without a synchronisation.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "pd_internal.h"

namespace {

constexpr int kNoallocBlock = 64;  // 32 particles: small blocks spread a small call over the chip

constexpr int kScratchPerParticle = 8;  // W (4) + m / V (2) + penalty term (2)

// The scratch.  Every call shares it and it keeps the previous call's
// contents; each call writes every entry it later reads, so nothing needs
// clearing.  Two calls whose kernels overlap on the GPU (different streams,
// or different host threads) race on it.
static __device__ __align__(256) double g_noalloc_scratch[(size_t)PD_NOALLOC_MAX_PARTICLES * kScratchPerParticle];

struct NoallocArgs {
  int64_t n;
  const double2* x;
  const double* vol;
  const int64_t* row_ptr;
  const int32_t* col;
  const double2* u;
  double2* v;
  double2* acc;
  double2* f;
  double2* w01;  // scratch
  double2* w23;  // scratch
  double2* mt;   // scratch
  double2* hg;   // scratch
  double c11, c12, c33, dt, inv_rho, det_guard, k_hg;
  double one, neg_one, neg_zero;  // 1, -1, -0
};

// A particle's row [r0, r1) is walkable when it lies inside [0, row_ptr[n]]
// (the caller's col holds row_ptr[n] entries) and row_ptr[0] is 0.
__device__ __forceinline__ bool row_ok(const NoallocArgs& a, int64_t i, int64_t* r0, int64_t* r1) {
  *r0 = a.row_ptr[i];
  *r1 = a.row_ptr[i + 1];
  return a.row_ptr[0] == 0 && 0 <= *r0 && *r0 <= *r1 && *r1 <= a.row_ptr[a.n];
}

// A value in a register: a DFMA of three registers takes 16 cycles of the FP64
// pipe per warp and SM, a DADD, DMUL or DFMA with a constant operand 19, so the
// bond loops write x - y = fma(y, -1, x), x + y = fma(x, 1, y), x y = fma(x, y, -0)
// (one rounding of the same value each): a call on 256 x 255 particles 104 -> 91 us.
__device__ __forceinline__ double in_register(double x) { return __shfl_sync(0xffffffffu, x, 0); }

// The warp's longest row (the pair exchanges of a walk run in every lane).
__device__ __forceinline__ int64_t longest(int64_t len) {
  for (int o = 16; o; o >>= 1) {
    const int64_t t = __shfl_xor_sync(0xffffffffu, len, o);
    len = t > len ? t : len;
  }
  return len;
}

// Stress and W of particle i from its sums: row h of D (d1, d2), K^-1; the
// lanes of a particle's pair exchange what the symmetric stress needs.  All
// lanes of the warp call it.
__device__ __forceinline__ double2 w_row(const NoallocArgs& a, int h, double d1, double d2, double q11, double q12,
                                         double q22, double vi) {
  const double g1 = fma(d1, q11, d2 * q12), g2 = fma(d1, q12, d2 * q22);
  const double diag = h ? g2 : g1, other = __shfl_xor_sync(0xffffffffu, diag, 1);
  const double off = h ? g1 : g2, cross = __shfl_xor_sync(0xffffffffu, off, 1);
  const double e11 = h ? other : diag, e22 = h ? diag : other, e12 = 0.5 * (off + cross);
  const double sd = fma(h ? a.c12 : a.c11, e11, (h ? a.c11 : a.c12) * e22);
  const double s12 = a.c33 * e12;
  const double sa = h ? s12 : sd, sb = h ? sd : s12, kh = -a.k_hg;
  return make_double2(vi * fma(kh, g1, fma(sa, q11, sb * q12)), vi * fma(kh, g2, fma(sa, q12, sb * q22)));
}

// What pass A leaves of component h of particle i.  singular: no stress.
__device__ __forceinline__ void store_a(const NoallocArgs& a, int64_t i, int h, bool ok, bool singular, double hg,
                                        double mt, double2 W) {
  const double q = nan("");
  if (!ok) hg = mt = W.x = W.y = q;
  else if (singular) mt = W.x = W.y = 0.0;
  reinterpret_cast<double*>(a.hg)[2 * i + h] = hg;
  reinterpret_cast<double*>(a.mt)[2 * i + h] = mt;
  (h ? a.w23 : a.w01)[i] = W;
}

// Pass A: K^-1 and m/V over the given family, D, stress, W (no bond breaking).
// Two threads per particle, thread h summing component h (k11, k12 or k22; m_h,
// row h of D, the penalty's h): 9 of the 17 FP64 operations of a bond each, the
// sums in family order as ever.  An FP64 instruction keeps its SM quarter busy
// for 64 cycles, so a thread's chain is what a call waits for.
constexpr int kNoallocWalk = 4;  // bonds in flight per thread (2: 24.0 us against 21.6 per 30 x 31 call)

// A warp's rows, up to `most` bonds: whole groups of bonds(k, their indices, the
// group's size, what to request next), whose terms need no branch (a call on 256 x 255
// particles 91.5 -> 90.2 us), then the rest one by one.
template <typename Index, typename Bonds>
__device__ __forceinline__ void walk_row(int64_t most, Index index, Bonds bonds) {
  int jn[kNoallocWalk];
  auto ask = [&](int64_t k) {
#pragma unroll
    for (int q = 0; q < kNoallocWalk; ++q) jn[q] = index(k + q);
  };
  int64_t k = 0;
  ask(0);
  for (; k + kNoallocWalk <= most; k += kNoallocWalk) {
    int j[kNoallocWalk];
#pragma unroll
    for (int q = 0; q < kNoallocWalk; ++q) j[q] = jn[q];
    bonds(k, j, std::integral_constant<int, kNoallocWalk>{}, [&] { ask(k + kNoallocWalk); });
  }
  for (; k < most; ++k) {
    int j = index(k);
    bonds(k, &j, std::integral_constant<int, 1>{}, [] {});
  }
}

__global__ void __launch_bounds__(kNoallocBlock) k_noalloc_pass_a(NoallocArgs a) {
  const int64_t p = (int64_t)blockIdx.x * (kNoallocBlock / 2) + (threadIdx.x >> 1);
  const int h = threadIdx.x & 1;
  const bool have = p < a.n;
  const int64_t i = have ? p : a.n - 1;  // (a lane past the end repeats the last particle and stores nothing)
  const double xi = reinterpret_cast<const double*>(a.x)[2 * i + h], ui = reinterpret_cast<const double*>(a.u)[2 * i + h];
  int64_t r0, r1;
  bool ok = row_ok(a, i, &r0, &r1);
  double ka = 0.0, kb = 0.0, m = 0.0;     // h = 0: k11, k12; h = 1: k22 (in kb)
  double d1 = 0.0, d2 = 0.0, ah = 0.0;
  const int64_t len = ok ? r1 - r0 : 0;
  const double one = in_register(a.one), neg1 = in_register(a.neg_one), neg0 = in_register(a.neg_zero);
  const int64_t most = longest(len);
  // the neighbour of bond k (past the row: the particle itself)
  auto index = [&](int64_t k) { return k < len ? a.col[r0 + k] : (int)i; };
  // U bonds j[0 .. U) from bond k on, without a branch each; next(): after their requests
  auto bonds = [&](int64_t k, int* j, auto u, auto next) {
    constexpr int U = decltype(u)::value;
    double xj[U], uj[U], vj[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (j[q] < 0 || j[q] >= a.n) {  // a bad index: read nothing of it, poison this particle
        ok = false;
        j[q] = (int)i;
      }
      xj[q] = reinterpret_cast<const double*>(a.x)[2 * (int64_t)j[q] + h];
      uj[q] = reinterpret_cast<const double*>(a.u)[2 * (int64_t)j[q] + h];
      vj[q] = a.vol[j[q]];
    }
    next();
#pragma unroll
    for (int q = 0; q < U; ++q) {
      double e = fma(xi, neg1, xj[q]), t = fma(vj[q], e, neg0), d = fma(ui, neg1, uj[q]);
      if (k + q >= len) {  // zeros, which change no sum
        e = t = 0.0;
        d = -0.0;
        vj[q] = 1.0;
      }
      const double e2 = __shfl_xor_sync(0xffffffffu, e, 1), t2 = __shfl_xor_sync(0xffffffffu, t, 1);
      const double tx = h ? t2 : t, ty = h ? t : t2;
      ka = fma(t, e, ka);   // k11 | k22
      kb = fma(t, e2, kb);  // k12 (h = 0)
      m = fma(t, one, m);
      d1 = fma(d, tx, d1);
      d2 = fma(d, ty, d2);
      ah = fma(vj[q], d, ah);
    }
  };
  walk_row(most, index, bonds);
  // (pass B is let go at the blocks' exit: launched while some SMs still hold blocks of this
  // pass, its blocks crowd onto the others: calls on 120 x 120, 170 x 170 and 190 x 190 particles
  // 29.8, 51.7 and 58.8 us against 24.6, 40.7 and 52.8)
  const double k11 = __shfl_sync(0xffffffffu, ka, threadIdx.x & 30), k12 = __shfl_sync(0xffffffffu, kb, threadIdx.x & 30),
               k22 = __shfl_sync(0xffffffffu, ka, (threadIdx.x & 30) + 1);
  const double det = fma(k11, k22, -(k12 * k12));
  const bool singular = r1 == r0 || !(det > a.det_guard * (k11 * k22));
  const double vi = a.vol[i], quo = 1.0 / (h ? vi : det);
  const double r = __shfl_sync(0xffffffffu, quo, threadIdx.x & 30), rv = __shfl_sync(0xffffffffu, quo, (threadIdx.x & 30) + 1);
  const double2 W = w_row(a, h, d1, d2, k22 * r, -k12 * r, k11 * r, vi);
  if (have) store_a(a, i, h, ok, singular, (2.0 * a.k_hg) * ah, m * rv, W);
}

// Pass A of a small call: 16 lanes per particle.  The lanes take 16 bonds at a
// time, form each bond's xi, V xi, d (6 operations, one bond per lane) into
// shared memory, and then 11 of them run one of the 11 sums each over these
// bonds, in family order: a chain of ~40 FP64 operations per particle instead
// of ~290.  It costs twice the two-thread form's FP64 issue per particle, so it
// serves the calls that leave most of the chip idle.
constexpr int kNoallocSmallBlock = 64;
constexpr int kNoallocSmall = 4096;

__global__ void __launch_bounds__(kNoallocSmallBlock) k_noalloc_pass_a_small(NoallocArgs a) {
  enum { EX, EY, T0, T1, DX, DY, V, NV };
  __shared__ double val[kNoallocSmallBlock / 16][NV][16];
  const int64_t p = (int64_t)blockIdx.x * (kNoallocSmallBlock / 16) + (threadIdx.x >> 4);
  const int c = threadIdx.x & 15;
  const bool have = p < a.n;
  const int64_t i = have ? p : a.n - 1;
  double(*S)[16] = val[threadIdx.x >> 4];
  // sum c adds S[pc] * S[qc] (sums 3 and 4, of m: S[pc] * 1, which is S[pc])
  const int pc = c < 2 ? T0 : c == 2 ? T1 : c == 3 ? T0 : c == 4 ? T1 : c < 7 ? DX : c < 9 ? DY : V;
  const int qc = c == 0 ? EX : c < 3 ? EY : c == 5 || c == 7 ? T0 : c < 9 ? T1 : c == 9 ? DX : DY;
  const bool sums_m = c == 3 || c == 4;
  const double2 xi = a.x[i], ui = a.u[i];
  int64_t r0, r1;
  bool ok = row_ok(a, i, &r0, &r1);
  const int64_t len = ok ? r1 - r0 : 0;
  int64_t most = len;  // of the warp's two particles
  const int64_t t = __shfl_xor_sync(0xffffffffu, most, 16);
  most = t > most ? t : most;
  double sum = 0.0;
  for (int64_t k0 = 0; k0 < most; k0 += 16) {
    if (k0 + c < len) {
      int j = a.col[r0 + k0 + c];
      if (j < 0 || j >= a.n) {
        ok = false;
        j = (int)i;
      }
      const double2 xj = a.x[j], uj = a.u[j];
      const double vj = a.vol[j], ex = xj.x - xi.x, ey = xj.y - xi.y;
      S[EX][c] = ex;
      S[EY][c] = ey;
      S[T0][c] = vj * ex;
      S[T1][c] = vj * ey;
      S[DX][c] = uj.x - ui.x;
      S[DY][c] = uj.y - ui.y;
      S[V][c] = vj;
    }
    __syncwarp();
    const int m = (int)(len - k0 < 16 ? len - k0 : 16);
    for (int k = 0; k < m; ++k) sum = fma(S[pc][k], sums_m ? 1.0 : S[qc][k], sum);
    __syncwarp();
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int g0 = threadIdx.x & 16, h = c & 1;
  ok = ((__ballot_sync(0xffffffffu, ok) >> g0) & 0xffffu) == 0xffffu;
  auto get = [&](int q) { return __shfl_sync(0xffffffffu, sum, g0 + q); };
  const double k11 = get(0), k12 = get(1), k22 = get(2), m = get(3 + h), d1 = get(5 + 2 * h), d2 = get(6 + 2 * h),
               ah = get(9 + h);
  const double det = fma(k11, k22, -(k12 * k12));
  const bool singular = r1 == r0 || !(det > a.det_guard * (k11 * k22));
  const double vi = a.vol[i], quo = 1.0 / (h ? vi : det);
  const double r = __shfl_sync(0xffffffffu, quo, g0), rv = __shfl_sync(0xffffffffu, quo, g0 + 1);
  const double2 W = w_row(a, h, d1, d2, k22 * r, -k12 * r, k11 * r, vi);
  if (have && c < 2) store_a(a, i, h, ok, singular, (2.0 * a.k_hg) * ah, m * rv, W);
}

// Pass B: gather force, velocity-Verlet kick, acce := f / rho; component h of
// a particle per thread, as pass A.
__global__ void __launch_bounds__(kNoallocBlock) k_noalloc_pass_b(NoallocArgs a) {
  const int64_t p = (int64_t)blockIdx.x * (kNoallocBlock / 2) + (threadIdx.x >> 1);
  const int h = threadIdx.x & 1;
  const bool have = p < a.n;
  const int64_t i = have ? p : a.n - 1;
  asm volatile("griddepcontrol.wait;" ::: "memory");  // pass A's scratch
  const double2* Wr = h ? a.w23 : a.w01;
  const double2 wi = Wr[i], m = a.mt[i];
  const double xi = reinterpret_cast<const double*>(a.x)[2 * i + h];
  const double hg = reinterpret_cast<const double*>(a.hg)[2 * i + h];
  const double ao = reinterpret_cast<const double*>(a.acc)[2 * i + h];
  double v = reinterpret_cast<const double*>(a.v)[2 * i + h];
  double f = fma(wi.x, m.x, fma(wi.y, m.y, hg));
  int64_t r0, r1;
  bool ok = row_ok(a, i, &r0, &r1);
  const int64_t len = ok ? r1 - r0 : 0, most = longest(len);
  const double neg1 = in_register(a.neg_one);
  auto index = [&](int64_t k) { return k < len ? a.col[r0 + k] : (int)i; };
  auto bonds = [&](int64_t k, int* j, auto u, auto next) {
    constexpr int U = decltype(u)::value;
    double xj[U];
    double2 wj[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (j[q] < 0 || j[q] >= a.n) {
        ok = false;
        j[q] = (int)i;
      }
      xj[q] = reinterpret_cast<const double*>(a.x)[2 * (int64_t)j[q] + h];
      wj[q] = Wr[j[q]];
    }
    next();
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const double e = fma(xi, neg1, xj[q]), e2 = __shfl_xor_sync(0xffffffffu, e, 1);
      const bool on = k + q < len;  // past the row: -0, which changes no sum
      f = fma(on ? wj[q].x : 1.0, on ? (h ? e2 : e) : -0.0, f);
      f = fma(on ? wj[q].y : 1.0, on ? (h ? e : e2) : -0.0, f);
    }
  };
  walk_row(most, index, bonds);
  if (!ok) f = nan("");
  const double an = f * a.inv_rho;
  v = v + (0.5 * (ao + an)) * a.dt;
  if (!have) return;
  reinterpret_cast<double*>(a.v)[2 * i + h] = v;
  reinterpret_cast<double*>(a.f)[2 * i + h] = f;
  reinterpret_cast<double*>(a.acc)[2 * i + h] = an;
}

// Device address of the scratch.  In host code the array's name is only a
// host-side stand-in, so the address is looked up with cudaGetSymbolAddress
// in the CUDA context that is current at the call, once per context, and
// cached under that context's unique id (cuCtxGetId: never reused in a
// process, so a context destroyed by cudaDeviceReset cannot leave a stale
// address behind; its replacement is looked up afresh).  The driver entry
// points come through the runtime, so the library does not link libcuda.
std::mutex g_scratch_mu;
struct ScratchEntry {
  unsigned long long ctx_id;
  double* ptr;
};
constexpr int kScratchCache = 64;
ScratchEntry g_scratch_cache[kScratchCache] = {};
int g_scratch_next = 0;
PFN_cuCtxGetCurrent_v4000 g_ctx_get_current = nullptr;
PFN_cuCtxGetId_v12000 g_ctx_get_id = nullptr;

// The current context's id; 0 with *err set when it cannot be had.
unsigned long long current_context_id(cudaError_t* err) {
  *err = cudaSuccess;
  if (!g_ctx_get_current || !g_ctx_get_id) {
    cudaDriverEntryPointQueryResult q1, q2;
    void* f1 = nullptr;
    void* f2 = nullptr;
    cudaError_t e1 = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1);
    cudaError_t e2 = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2);
    if (e1 != cudaSuccess || e2 != cudaSuccess || q1 != cudaDriverEntryPointSuccess ||
        q2 != cudaDriverEntryPointSuccess || !f1 || !f2) {
      *err = e1 != cudaSuccess ? e1 : (e2 != cudaSuccess ? e2 : cudaErrorSymbolNotFound);
      return 0;
    }
    g_ctx_get_current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(f1);
    g_ctx_get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(f2);
  }
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (g_ctx_get_current(&c) == CUDA_SUCCESS && !c) {
    // No context bound to this thread yet: bind the current device's primary
    // context, as any runtime call would (a context the caller made current
    // itself is left as it is).
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
    g_ctx_get_current(&c);
  }
  if (!c || g_ctx_get_id(c, &id) != CUDA_SUCCESS) {
    *err = cudaErrorDeviceUninitialized;
    return 0;
  }
  return id;
}

void set_err(char* errbuf, int errlen, const char* msg) {
  if (errbuf && errlen > 0) {
    std::strncpy(errbuf, msg, (size_t)errlen - 1);
    errbuf[errlen - 1] = '\0';
  }
}

}  // namespace

extern "C" int pd_compute_velocity_noalloc(int64_t n, const double* x, const double* vol, const int64_t* row_ptr,
                                           const int32_t* col, const double* u, double* velocity, double* acce,
                                           double* netF, const pd_params* p, void* stream, char* errbuf,
                                           int errlen) {
  if (n < 0 || n > PD_NOALLOC_MAX_PARTICLES) {
    char m[160];
    std::snprintf(m, sizeof(m), "pd_compute_velocity_noalloc: n = %lld is outside [0, %d] (PD_NOALLOC_MAX_PARTICLES)",
                  (long long)n, PD_NOALLOC_MAX_PARTICLES);
    set_err(errbuf, errlen, m);
    return PD_ERR_CAPACITY;
  }
  if (!p) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: NULL params");
    return PD_ERR_ARG;
  }
  if (!(p->rho > 0.0) || !(p->dt > 0.0)) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: rho and dt must be positive");
    return PD_ERR_ARG;
  }
  // What this path does not implement is refused, not ignored.
  if (p->precision != PD_FP64) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: FP64 only (precision must be PD_FP64)");
    return PD_ERR_ARG;
  }
  if (p->n1 != 0.0 || p->n2 != 0.0) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: classic weights only (n1 = n2 = 0)");
    return PD_ERR_ARG;
  }
  if (p->s_c > 0.0) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: no bond breaking here (s_c must be 0)");
    return PD_ERR_ARG;
  }
  if (!x || !vol || !row_ptr || (!col && n > 0) || !u || !velocity || !acce || !netF) {
    set_err(errbuf, errlen, "pd_compute_velocity_noalloc: NULL argument");
    return PD_ERR_ARG;
  }
  if (n == 0) return PD_OK;
  cudaError_t e = cudaSuccess;
  double* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    const unsigned long long id = current_context_id(&e);
    if (id == 0) {
      char m[200];
      std::snprintf(m, sizeof(m), "pd_compute_velocity_noalloc: no current CUDA context: %s", cudaGetErrorString(e));
      set_err(errbuf, errlen, m);
      return PD_ERR_CUDA;
    }
    for (int k = 0; k < kScratchCache; ++k)
      if (g_scratch_cache[k].ctx_id == id) scratch = g_scratch_cache[k].ptr;
    if (!scratch) {  // first call in this context: set-up
      void* q = nullptr;
      e = cudaGetSymbolAddress(&q, g_noalloc_scratch);
      if (e != cudaSuccess || !q) {
        char m[200];
        std::snprintf(m, sizeof(m), "pd_compute_velocity_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        set_err(errbuf, errlen, m);
        return PD_ERR_CUDA;
      }
      scratch = static_cast<double*>(q);
      g_scratch_cache[g_scratch_next] = {id, scratch};
      g_scratch_next = (g_scratch_next + 1) % kScratchCache;
    }
  }
  NoallocArgs a;
  a.n = n;
  a.x = reinterpret_cast<const double2*>(x);
  a.vol = vol;
  a.row_ptr = row_ptr;
  a.col = col;
  a.u = reinterpret_cast<const double2*>(u);
  a.v = reinterpret_cast<double2*>(velocity);
  a.acc = reinterpret_cast<double2*>(acce);
  a.f = reinterpret_cast<double2*>(netF);
  a.w01 = reinterpret_cast<double2*>(scratch);
  a.w23 = reinterpret_cast<double2*>(scratch + 2 * (size_t)PD_NOALLOC_MAX_PARTICLES);
  a.mt = reinterpret_cast<double2*>(scratch + 4 * (size_t)PD_NOALLOC_MAX_PARTICLES);
  a.hg = reinterpret_cast<double2*>(scratch + 6 * (size_t)PD_NOALLOC_MAX_PARTICLES);
  const double pre = p->E / (1.0 - p->nu * p->nu);  // plane stress, as pd_create's contexts
  a.c11 = pre;
  a.c12 = p->nu * pre;
  a.c33 = (1.0 - p->nu) * pre;
  a.dt = p->dt;
  a.inv_rho = 1.0 / p->rho;
  a.det_guard = p->det_guard;
  a.k_hg = p->k_hg;
  a.one = 1.0;
  a.neg_one = -1.0;
  a.neg_zero = -0.0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n <= kNoallocSmall) {
    constexpr int per = kNoallocSmallBlock / 16;
    k_noalloc_pass_a_small<<<(unsigned)((n + per - 1) / per), kNoallocSmallBlock, 0, s>>>(a);
  } else {
    k_noalloc_pass_a<<<(unsigned)((2 * n + kNoallocBlock - 1) / kNoallocBlock), kNoallocBlock, 0, s>>>(a);
  }
  e = cudaGetLastError();
  if (e == cudaSuccess) {  // pass B's blocks start while pass A drains, and wait for it
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)((2 * n + kNoallocBlock - 1) / kNoallocBlock));
    lc.blockDim = dim3(kNoallocBlock);
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    e = cudaLaunchKernelEx(&lc, k_noalloc_pass_b, a);
  }
  if (e != cudaSuccess) {
    char m[200];
    std::snprintf(m, sizeof(m), "pd_compute_velocity_noalloc: launch: %s", cudaGetErrorString(e));
    set_err(errbuf, errlen, m);
    return PD_ERR_CUDA;
  }
  return PD_OK;
}
