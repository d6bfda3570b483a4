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

// No chains in launches of this thread while one lives: for evaluations that run beside others, whose SMs waiting kernels
// would hold.
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
// Every covariance build uses them: within a few ulps of the true value, as the log1p form is (whose exponent carries
// one rounding of each t_k), and an eighth of its FP64 instructions, which bound these kernels (GB300 issues one
// FP64 warp instruction per 19 clocks and SM).  Measured, n = 4096, d = 8, matern5_2: the build of R takes 1.29 ms
// against 9.81 ms with the division and log1p per dimension; R_on of 5003 points against 4001, d = 6: 2.52 against
// 17.7 ms.
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
