// common.cuh -- shared definitions for the GB300 likelihood kernels (sm_103a).
//
// Covariance functions of libKriging src/lib/Covariance.cpp (the same functions, in product form):
//   gauss      Cov :24-36   DlnCovDtheta :38-50
//   exp        Cov :65-75   DlnCovDtheta :77-88
//   matern3_2  Cov :104-116 DlnCovDtheta :118-130
//   matern5_2  Cov :149-161 DlnCovDtheta :163-179
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace lkg {

enum Kernel : int { KGAUSS = 0, KEXP = 1, KMATERN32 = 2, KMATERN52 = 3 };

constexpr int MAX_D = 32;  // largest input dimension the fused kernels accept

struct CudaError : std::runtime_error {
  explicit CudaError(const std::string& s) : std::runtime_error(s) {}
};

inline void check_cuda(cudaError_t e, const char* what, const char* file, int line) {
  if (e != cudaSuccess)
    throw CudaError(std::string("CUDA error in ") + what + " (" + file + ":" + std::to_string(line) +
                    "): " + cudaGetErrorString(e));
}
#define LKG_CUDA(x) ::lkg::check_cuda((x), #x, __FILE__, __LINE__)
#define LKG_LAUNCH(what) ::lkg::check_cuda(cudaGetLastError(), what, __FILE__, __LINE__)

// Chains of short dependent kernels: a kernel launched with chained = true may start while the one before it in its stream
// still runs.  It does there what needs none of that one's results (barriers, tensor memory, tables, operands that the whole
// chain only reads) and then waits in chain_wait() for its end and its writes.  Every CTA of such a kernel calls
// chain_wait() before it returns, reads what the chain writes, or writes anything: a kernel of the chain then ends
// after all those before it.  chain_next() lets the next one start; it costs nothing where that one is not chained.  The
// gap between two kernels of a graph, with the prologue, is what this saves.  Only single matrices are chained: the
// launches of a batch fill the chip, and kernels that wait cost it more than the gaps (64 matrices of 2048 rows: 74.1 ms
// unchained, 76.1 chained).  One matrix: n = 1003 LL + gradient 2.23 -> 2.10 ms, predict of 1000 points at n = 200 293 -> 268
// us, of 5003 at n = 4001 7.80 -> 7.43 ms.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// No chains in launches of this thread while one lives: for batched evaluations that run beside others, whose SMs waiting
// kernels would hold.  (Predictions of submodels beside one another keep theirs: 200 points on 24 submodels of 150 to 2500
// rows take 3.5 ms chained, 4.0 unchained, 5000 points 22.0 and 22.2.)
inline thread_local int t_unchained = 0;
struct Unchained {
  explicit Unchained(bool on) : on_(on) { t_unchained += on_; }
  ~Unchained() { t_unchained -= on_; }
  Unchained(const Unchained&) = delete;
  Unchained& operator=(const Unchained&) = delete;

 private:
  int on_;
};

// wall clock of the device in nanoseconds, for waits that give up
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t));
  return t;
}

template <class... KA, class... A>
void launch_chained(bool chained, void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = chained && !t_unchained ? 1 : 0;
  LKG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<KA>(args)...));
}

// x 2^k for a normal x and result: an integer operation (an FP64 product takes an issue slot of the scarce pipe)
__device__ __forceinline__ double times_pow2(double x, int k) {
  return __hiloint2double(__double2hiint(x) + k * 0x00100000, __double2loint(x));
}

// 1 / sqrt(x) as FP32 gives it, for 2^-99 <= x < 2^99 (rsqrt_seed_range, read off the bits): the conversions, to nearest
// even, are integer operations
__device__ __forceinline__ bool rsqrt_seed_range(double x) {
  const int hi = __double2hiint(x);
  return hi >= 0x39C00000 && hi < 0x46200000;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  constexpr unsigned long long kBias = 896ull << 52;  // FP64 exponent bias minus FP32's
  unsigned long long xb = (unsigned long long)__double_as_longlong(x) - kBias;
  xb += 0x0FFFFFFFull + ((xb >> 29) & 1ull);
  const float seed = rsqrtf(__int_as_float((int)(xb >> 29)));
  return __longlong_as_double((long long)(((unsigned long long)(unsigned)__float_as_int(seed) << 29) + kBias));
}

// ---------------------------------------------------------------------------------------------------------------
// device covariance functions.  dx is X_j - X_i (sign irrelevant for Cov and DlnCovDtheta)
// ---------------------------------------------------------------------------------------------------------------
// Product forms (no per-dimension division or log1p): with c_k = s / |theta_k| (s = 1, sqrt(3), sqrt(5)) and
// t_k = c_k |dx_k|,
//   gauss     exp(-0.5 sum (dx_k / theta_k)^2)
//   exp       exp(-sum t_k)
//   matern3_2 prod (1 + t_k) exp(-sum t_k)              = exp(-sum (t_k - log1p t_k))
//   matern5_2 prod (1 + t_k + t_k^2 / 3) exp(-sum t_k)  = exp(-sum (t_k - log1p(t_k + t_k^2 / 3)))
// They take an eighth of the FP64 instructions of the log1p form, and these bound the covariance kernels (GB300 issues one
// FP64 warp instruction per 19 clocks and SM).
//
// In plain FP64 (cov_fast_*: gradient sums, Vecchia blocks, pairs of submodels) the value carries the rounding of sum t_k,
// which is several times the exponent that it nearly cancels with the product, and one rounding per factor: 2.5 units of
// 2^-53 (rms) at d = 8 and theta of three times the distances, where the log1p form has 0.6.  The matrices and
// cross-covariances that go into factors and solves take CovValue: from d = 5 on (the kernels' template for eight and more
// dimensions) CovSum, whose values are as accurate as the log1p form's.
template <int K>
__device__ __forceinline__ double cov_scale() {
  if constexpr (K == KMATERN32) return sqrt(3.0);
  else if constexpr (K == KMATERN52) return sqrt(5.0);
  else return 1.0;
}

// accumulate one dimension: sum_state (the exponent argument) and prod_state (the polynomial product)
template <int K>
__device__ __forceinline__ void cov_fast_term(double dx, double ck, double& sum_state, double& prod_state) {
  if constexpr (K == KGAUSS) {
    const double v = dx * ck;
    sum_state = fma(v, v, sum_state);
  } else {
    const double t = fabs(dx) * ck;
    sum_state += t;
    if constexpr (K == KMATERN32) prod_state *= (1.0 + t);
    if constexpr (K == KMATERN52) prod_state *= fma(t, t * (1.0 / 3.0), 1.0 + t);
  }
}

// prod_state exp(-sum_state), also where the exponential alone leaves the FP64 range: past 700 it is taken in two
// halves, and past 1500 the value is below the smallest double for any d <= 32 (prod <= (1 + 1500 / 32 + (1500 /
// 32)^2 / 3)^32 < e^214).  An infinite or NaN sum falls through to inf * 0 = NaN, as in the log1p form.  The range test
// reads the high word: a compare of doubles would take an FP64 issue slot of every pair.
template <int K>
__device__ __forceinline__ double cov_fast_finish(double sum_state, double prod_state) {
  if constexpr (K == KGAUSS) return exp(-0.5 * sum_state);
  else if constexpr (K == KEXP) return exp(-sum_state);
  else {
    const int hi = __double2hiint(sum_state);
    if (hi >= 0x4085E000 && hi < 0x7FF00000) {  // 700 <= sum < infinity
      if (sum_state > 1500.0) return 0.0;
      const double h = exp(-0.5 * sum_state);
      return prod_state * h * h;
    }
    return prod_state * exp(-sum_state);
  }
}

// The scale of one dimension for CovSum: c = cov_scale / |theta| in FP64 and what c lacks of it, relative to c, with the
// rounding of the square root: true scale = c (1 + rest)
struct CovScale {
  double c;
  float rest;
};
template <int K>
__device__ __forceinline__ CovScale cov_scale_of(double theta) {
  constexpr double kRoot = K == KMATERN32 ? 5.7937e-17 : K == KMATERN52 ? -4.8586e-17 : 0.0;  // of sqrt(3), sqrt(5) in FP64
  const double s = cov_scale<K>(), th = fabs(theta), c = s / th;
  const double rest = fma(-c, th, s) / s + kRoot;
  return {c, fabs(rest) < 1.0 ? (float)rest : 0.0f};
}

// The same value with sum t_k (sum t_k^2) in fixed point (64 fraction bits, by integer operations, exact but for 2^-64 a term: integer
// instructions are cheap beside an FP64 one) and, for the Materns, the rounding errors of the product, which fma gives
// exactly, summed in FP32 relative to it, with the effect of the scale's rounding; all go into the value at the end.  As many
// FP64 operations per dimension as the plain form: the fused update p + p a replaces 1 + a and the product, and pays for
// the error; four more per pair.  Measured, n = 4096, d = 8, matern5_2: the build of R 1.27 ms, 1.29 in the plain form, 9.81
// with the division and log1p per dimension; R_on of 5003 points against 4001, d = 6: 2.67 ms, 2.52, 17.7.
template <int K>
struct CovSum {
  static constexpr unsigned kHuge = 2048u, kInf = 1u << 20, kNan = 1u << 26;  // of 32 terms at most: no overflow
  double p = 1.0;                  // Materns: the product
  unsigned long long frac = 0ull;  // sum t, gauss: sum t^2: ip + frac 2^-64
  unsigned ip = 0u;
  float r = 0.0f;  // relative correction of the value

  __device__ __forceinline__ void add(double dx, const CovScale& k) {
    const double t = fabs(dx) * k.c;
    const float tf = fminf(narrowed(t), 2048.0f);  // the value is zero beyond
    if constexpr (K == KGAUSS) {
      add_fixed(t * t);
      r = fmaf(-k.rest * tf, tf, r);
    } else {
      add_fixed(t);
      if constexpr (K == KEXP) r = fmaf(-k.rest, tf, r);
      // - t dlnC/dt = t^2 / (1 + t), t^2 (1 + t) / (3 + 3 t + t^2)
      if constexpr (K == KMATERN32) r = fmaf(-k.rest, __fdividef(tf * tf, 1.0f + tf), r);
      if constexpr (K == KMATERN52) r = fmaf(-k.rest, __fdividef(tf * tf * (1.0f + tf), fmaf(tf, tf + 3.0f, 3.0f)), r);
      if constexpr (K != KEXP) {
        double a = t;  // the factor minus one
        if constexpr (K == KMATERN52) a = fma(t, t * (1.0 / 3.0), t);
        const double pn = fma(p, a, p);
        const double e = fma(p, a, p - pn);
        // e / pn in FP32: e with pn's exponent taken off, over pn's significand
        const int he = __double2hiint(e), hp = __double2hiint(pn), fe = ((he >> 20) & 0x7FF) - (hp >> 20) + 127;
        const int eb = (he & 0x80000000) | (fe << 23) | ((he & 0xFFFFF) << 3) | (int)((unsigned)__double2loint(e) >> 29);
        r += __fdividef(fe > 0 ? __int_as_float(eb) : 0.0f, __int_as_float(0x3F800000 | ((hp & 0xFFFFF) << 3)));
        p = pn;
      }
    }
  }

  __device__ __forceinline__ double value() const {
    if (ip >= kNan) return __longlong_as_double(0x7FF8000000000000ll);
    const double hi = __longlong_as_double((long long)(0x40B0000000000000ull | ((unsigned long long)(ip & 4095u) << 40) |
                                                       (frac >> 24))) -
                      4096.0;  // ip and the 40 leading fraction bits: exact
    const float lo = (float)(unsigned)(frac & 0xFFFFFFull) * 0x1p-64f;
    if constexpr (K == KGAUSS || K == KEXP) {
      constexpr float h = K == KGAUSS ? 0.5f : 1.0f;
      if (ip >= kHuge) return 0.0;
      const double e = exp(-(double)h * hi);
      return fma(widened(r - h * lo), e, e);
    } else {
      if (ip >= 700u) {  // the exponential alone leaves the FP64 range
        if (ip >= kInf) return __longlong_as_double(0x7FF8000000000000ll);  // infinity times 0, as in the log1p form
        // past 1500 the value is below the smallest double for any d <= 32 (p <= (1 + 1500 / 32 + (1500 / 32)^2 / 3)^32 <
        // e^214)
        if (ip >= 1500u) return 0.0;
        const double h = exp(-0.5 * hi);
        return fma(p * h, widened(r - lo), p * h) * h;
      }
      const double e = exp(-hi), y = p * e;
      return y + fma(y, widened(r - lo), fma(p, e, -y));
    }
  }

 private:
  __device__ __forceinline__ void add_fixed(double t) {
    const int hi = __double2hiint(t), e = hi >> 20, q = e - 1022;  // t = m 2^(q - 64) with m's leading bit 63
    const unsigned long long m = ((unsigned long long)__double_as_longlong(t) << 11) | 0x8000000000000000ull;
    unsigned long long f, up, i;  // the shifts give zero past 63
    asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(m), "r"(-q));
    asm("shl.b64 %0, %1, %2;" : "=l"(up) : "l"(m), "r"(q));
    asm("shr.u64 %0, %1, %2;" : "=l"(i) : "l"(m), "r"(64 - q));
    if (q > 0) f = up;
    unsigned w = (unsigned)i;
    if (q > 11) w = e < 2047 ? kHuge : (hi & 0xFFFFF) | __double2loint(t) ? kNan : kInf;
    frac += f;
    ip += w + (frac < f ? 1u : 0u);
  }
  // t >= 0 cut to FP32 by integer operations
  static __device__ __forceinline__ float narrowed(double t) {
    const int hi = __double2hiint(t), e = hi >> 20;
    if (e <= 896) return 0.0f;
    if (e >= 1151) return 2048.0f;
    return __int_as_float(((e - 896) << 23) | ((hi & 0xFFFFF) << 3) | (int)((unsigned)__double2loint(t) >> 29));
  }
  // an FP32 number below 1 as FP64 by integer operations (zero becomes 2^-127)
  static __device__ __forceinline__ double widened(float x) {
    const unsigned b = __float_as_uint(x);
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7FFFFFFFu) >> 3) + (896u << 20))), (int)(b << 29));
  }
};

template <int K>
struct CovPlain {
  double s = 0.0, p = 1.0;
  __device__ __forceinline__ void add(double dx, const CovScale& k) { cov_fast_term<K>(dx, k.c, s, p); }
  __device__ __forceinline__ double value() const { return cov_fast_finish<K>(s, p); }
};

// The line lies where the plain form's error shows: with it, and the digit products, results are 0.4 (d = 2) to 0.9 (d = 4)
// times as far from 80-bit arithmetic as with DFMA products on log1p-form matrices, and 1.1 to 1.9 times from d = 6 on; CovSum
// brings those to 0.3 .. 0.7 (geometric means of LL, gradient, leave-one-out and predictions, 382 outputs of Matern designs).
// Below it smooth designs without noise are so ill-conditioned that results show every rounding of R (gradients in two
// dimensions move by 2e-9), so they keep theirs.
template <int K, int DM>
using CovValue = std::conditional_t<(DM <= 4), CovPlain<K>, CovSum<K>>;

// dlnC/dtheta_k with inv = 1 / theta_k and ck = s / theta_k
template <int K>
__device__ __forceinline__ double dlncov_fast(double dx, double inv, double ck) {
  if constexpr (K == KGAUSS) {
    const double v = dx * inv;
    return v * v * inv;
  } else if constexpr (K == KEXP) {
    return fabs(dx) * inv * inv;
  } else if constexpr (K == KMATERN32) {
    const double t = fabs(dx) * ck;
    return (t * t) / (1.0 + t) * inv;
  } else {
    const double t = fabs(dx) * ck;
    const double a = 1.0 + t, b = t * t * (1.0 / 3.0);
    return (a * b) / (a + b) * inv;
  }
}

// dispatch a runtime kernel id to a template functor call
template <typename F>
inline void dispatch_kernel(int k, F&& f) {
  switch (k) {
    case KGAUSS: f.template operator()<KGAUSS>(); break;
    case KEXP: f.template operator()<KEXP>(); break;
    case KMATERN32: f.template operator()<KMATERN32>(); break;
    case KMATERN52: f.template operator()<KMATERN52>(); break;
    default: throw std::invalid_argument("Unsupported covariance kernel id " + std::to_string(k));
  }
}

inline int kernel_from_name(const std::string& s) {
  if (s == "gauss") return KGAUSS;
  if (s == "exp") return KEXP;
  if (s == "matern3_2") return KMATERN32;
  if (s == "matern5_2") return KMATERN52;
  throw std::invalid_argument("Unsupported covariance kernel: " + s);
}

inline const char* kernel_name(int k) {
  switch (k) {
    case KGAUSS: return "gauss";
    case KEXP: return "exp";
    case KMATERN32: return "matern3_2";
    case KMATERN52: return "matern5_2";
  }
  return "?";
}

inline int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Launch<kernel, DM>::run(args...) for the runtime kernel id and the smallest DM in {4, 8, 16, 32} holding d
template <template <int, int> class Launch, typename... Args>
void dispatch_kd(int kernel, int d, Args&&... args) {
  auto go = [&](auto kc) {
    constexpr int KK = decltype(kc)::value;
    if (d <= 4) Launch<KK, 4>::run(args...);
    else if (d <= 8) Launch<KK, 8>::run(args...);
    else if (d <= 16) Launch<KK, 16>::run(args...);
    else if (d <= 32) Launch<KK, 32>::run(args...);
    else throw std::invalid_argument("input dimension d > 32 is not supported by the GPU kernels");
  };
  switch (kernel) {
    case KGAUSS: go(std::integral_constant<int, KGAUSS>{}); break;
    case KEXP: go(std::integral_constant<int, KEXP>{}); break;
    case KMATERN32: go(std::integral_constant<int, KMATERN32>{}); break;
    case KMATERN52: go(std::integral_constant<int, KMATERN52>{}); break;
    default: throw std::invalid_argument("Unsupported covariance kernel id");
  }
}

}  // namespace lkg
