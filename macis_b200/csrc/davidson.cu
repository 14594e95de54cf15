// Single-vector Davidson on the GPU, replacing macis::davidson
// (include/macis/solvers/davidson.hpp:129-225) and diagonal_guess (:62-68).
//
// Basis V and A*V live in HBM (N x (max_m+1) FP64 each). Per iteration:
//   AV_i = H V_i                                  (spmv.cu)
//   row i of the Rayleigh matrix V^T AV           (multi-dot, FP64)
//   k x k symmetric eigenproblem on the host      (cyclic Jacobi, FP64)
//   X = V c, R = AV c - lambda X, |R|, W = -R/(D - lambda)   (one fused pass)
//   CGS2 of W against V, normalise                (davidson.hpp:111-126)
// The reference recomputes the full k x k product with gemm every
// iteration; only its lower triangle enters syev (rayleigh_ritz.hpp:73-75),
// and the entries of earlier rows do not change, so only the new row is
// formed. Reductions are two-stage with a fixed order (deterministic).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <vector>

#include "internal.hpp"
#include "primitives.cuh"

namespace mb {

constexpr int DV_THREADS = 512;
constexpr int DV_WARPS = DV_THREADS / 32;
constexpr int DV_CHUNK = 8;  // columns held by one multi-dot block

// The vector kernels of one iteration form a chain of short launches (for a
// basis that L2 holds, each runs 2-4 us, about a launch latency), so they
// are launched with programmatic serialization: the launch work of a kernel
// overlaps its predecessor and dav_wait holds its first access back until
// the predecessor has completed and its writes are visible.
__device__ __forceinline__ void dav_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Sum of acc[c] over the warp for 8 values at once: each step halves the
// values a lane holds, 9 shuffles instead of 40. Lane l ends with the sum of
// value ((l >> 4) & 1) * 4 + ((l >> 3) & 1) * 2 + ((l >> 2) & 1).
__device__ __forceinline__ double warp_sum8(double (&acc)[DV_CHUNK]) {
  const int lane = threadIdx.x & 31;
  double b[4], c[2];
  {
    const bool hi = lane & 16;
#pragma unroll
    for(int j = 0; j < 4; ++j) {
      const double send = hi ? acc[j] : acc[j + 4];
      b[j] = (hi ? acc[j + 4] : acc[j]) + __shfl_xor_sync(0xffffffffu, send, 16);
    }
  }
  {
    const bool hi = lane & 8;
#pragma unroll
    for(int j = 0; j < 2; ++j) {
      const double send = hi ? b[j] : b[j + 2];
      c[j] = (hi ? b[j + 2] : b[j]) + __shfl_xor_sync(0xffffffffu, send, 8);
    }
  }
  const bool hi = lane & 4;
  const double send = hi ? c[0] : c[1];
  double d = (hi ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, send, 4);
  d += __shfl_xor_sync(0xffffffffu, d, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  return d;
}

// True in the last of `n` blocks to arrive at *done (which it resets); the
// partial sums the other blocks wrote before arriving are then visible.
__device__ __forceinline__ bool last_block(unsigned* done, unsigned n) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if(threadIdx.x == 0) {
    last = atomicAdd(done, 1u) == n - 1;
    if(last) *done = 0;
  }
  __syncthreads();
  if(last) __threadfence();
  return last;
}

// Sum of p[0], p[stride], ... (nb terms) by one warp, in a fixed order.
__device__ __forceinline__ double warp_sum_partials(const double* p, int nb,
                                                    int stride) {
  const int lane = threadIdx.x & 31;
  double a = 0;
  for(int b = lane; b < nb; b += 32) a += __ldcg(p + size_t(b) * stride);
#pragma unroll
  for(int o = 16; o; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// out[c] = A[:, c] . v for c < ncol: block (x, y) sums rows x, x + gridDim.x,
// ... (in units of DV_THREADS) of the DV_CHUNK columns from DV_CHUNK y, and
// the last block of a chunk adds the chunk's partial sums in a fixed order
// (one launch instead of two per 8 columns). HBM-bound for long vectors.
__global__ void __launch_bounds__(DV_THREADS)
    multidot_k(const double* __restrict__ A, int64_t lda, int ncol,
               const double* __restrict__ v, int64_t n, double* partial,
               unsigned* done, double* out) {
  __shared__ double sh[DV_WARPS][DV_CHUNK];
  dav_wait();
  const int c0 = int(blockIdx.y) * DV_CHUNK;
  const int nc = ncol - c0 < DV_CHUNK ? ncol - c0 : DV_CHUNK;
  const double* Ac = A + c0 * lda;
  double acc[DV_CHUNK];
#pragma unroll
  for(int c = 0; c < DV_CHUNK; ++c) acc[c] = 0;
  for(int64_t i = int64_t(blockIdx.x) * DV_THREADS + threadIdx.x; i < n;
      i += int64_t(gridDim.x) * DV_THREADS) {
    const double x = v[i];
#pragma unroll
    for(int c = 0; c < DV_CHUNK; ++c)
      if(c < nc) acc[c] += Ac[i + c * lda] * x;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double a = warp_sum8(acc);
  if((lane & 3) == 0) sh[wid][(lane >> 4) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = a;
  __syncthreads();
  double* pc = partial + size_t(blockIdx.y) * gridDim.x * DV_CHUNK;
  if(threadIdx.x < DV_CHUNK) {
    double t = 0;
#pragma unroll
    for(int w = 0; w < DV_WARPS; ++w) t += sh[w][threadIdx.x];
    pc[blockIdx.x * DV_CHUNK + threadIdx.x] = t;
  }
  if(last_block(done + blockIdx.y, gridDim.x) && wid < nc) {
    const double t = warp_sum_partials(pc + wid, int(gridDim.x), DV_CHUNK);
    if(lane == 0) out[c0 + wid] = t;
  }
}

// Block sum of acc into partial[blockIdx.x]; the last block writes the total.
__device__ __forceinline__ void grid_sum(double acc, double* partial,
                                         unsigned* done, double* out) {
  __shared__ double sh[DV_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for(int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if(lane == 0) sh[wid] = acc;
  __syncthreads();
  if(threadIdx.x == 0) {
    double t = 0;
    for(int w = 0; w < DV_WARPS; ++w) t += sh[w];
    partial[blockIdx.x] = t;
  }
  if(last_block(done, gridDim.x) && wid == 0) {
    const double t = warp_sum_partials(partial, int(gridDim.x), 1);
    if(lane == 0) *out = t;
  }
}

// v -= A[:, 0:k] coef; with norm2 != nullptr also *norm2 = v . v after it.
__global__ void __launch_bounds__(DV_THREADS)
    cgs_update_k(const double* __restrict__ A, int64_t lda, int k,
                 const double* __restrict__ coef, double* v, int64_t n,
                 double* partial, unsigned* done, double* norm2) {
  __shared__ double cf[1024];
  dav_wait();
  for(int c = threadIdx.x; c < k; c += blockDim.x) cf[c] = coef[c];
  __syncthreads();
  double acc = 0;
  for(int64_t i = int64_t(blockIdx.x) * DV_THREADS + threadIdx.x; i < n;
      i += int64_t(gridDim.x) * DV_THREADS) {
    double s = 0;
#pragma unroll 8
    for(int c = 0; c < k; ++c) s += A[i + c * lda] * cf[c];
    const double x = v[i] - s;
    v[i] = x;
    acc += x * x;
  }
  if(norm2) grid_sum(acc, partial, done, norm2);
}

__global__ void scale_k(double* v, int64_t n, const double* nrm2) {
  dav_wait();
  const double inv = 1. / sqrt(*nrm2);
  for(int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += int64_t(gridDim.x) * blockDim.x)
    v[i] *= inv;
}

// Ritz coefficients passed with the launch (no copy to the device) up to
// this many; longer vectors come from device memory.
constexpr int DV_PARAM_COEF = 128;
struct RitzCoef {
  double c[DV_PARAM_COEF];
  const double* dev;  // used when not null
};

// X = V c; R = AV c - lam X; *rn2 = |R|^2; W = -R / (D - lam) into W.
__global__ void __launch_bounds__(DV_THREADS)
    ritz_residual_k(const double* __restrict__ V, const double* __restrict__ AV,
                    int64_t n, int k, const __grid_constant__ RitzCoef rc,
                    double lam, const double* __restrict__ D,
                    double* __restrict__ X, double* __restrict__ W,
                    double* partial, unsigned* done, double* rn2) {
  __shared__ double cf[1024];
  dav_wait();
  for(int j = threadIdx.x; j < k; j += blockDim.x)
    cf[j] = rc.dev ? rc.dev[j] : rc.c[j];
  __syncthreads();
  double acc = 0;
  for(int64_t i = int64_t(blockIdx.x) * DV_THREADS + threadIdx.x; i < n;
      i += int64_t(gridDim.x) * DV_THREADS) {
    double x = 0, av = 0;
#pragma unroll 8
    for(int j = 0; j < k; ++j) {
      x += V[i + j * n] * cf[j];
      av += AV[i + j * n] * cf[j];
    }
    const double r = av - lam * x;
    X[i] = x;
    W[i] = -r / (D[i] - lam);
    acc += r * r;
  }
  grid_sum(acc, partial, done, rn2);
}

// X = unit vector at the first minimum of D (diagonal_guess,
// davidson.hpp:62-68), one block.
__global__ void __launch_bounds__(1024)
    unit_guess_k(const double* D, int64_t n, double* X) {
  __shared__ double sv[32];
  __shared__ int64_t si[32];
  // every thread starts from entry 0, so a NaN there stays the choice and
  // one elsewhere is never chosen, as in a sequential scan
  double v = D[0];
  int64_t at = 0;
  auto take = [&](double w, int64_t j) {
    if(w < v || (w == v && j < at)) {
      v = w;
      at = j;
    }
  };
  for(int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    take(D[i], i);
    X[i] = 0.0;
  }
  for(int o = 16; o; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    const int64_t j = __shfl_xor_sync(0xffffffffu, at, o);
    take(w, j);
  }
  if((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = v;
    si[threadIdx.x >> 5] = at;
  }
  __syncthreads();
  if(threadIdx.x == 0) {
    for(int w = 1; w < int(blockDim.x >> 5); ++w) take(sv[w], si[w]);
    X[at] = 1.0;
  }
}

// Lowest `nwant` eigenpairs of the k x k Rayleigh matrix, given by its lower
// triangle (column-major, ld k) as dsyev with Uplo::Lower reads it
// (lobpcgxx/rayleigh_ritz.hpp:75). Householder reduction to tridiagonal
// form, Sturm-sequence bisection for each wanted eigenvalue, inverse
// iteration on the tridiagonal matrix, back-transformation and modified
// Gram-Schmidt among the returned vectors. W ascending; Vec columns.
void small_syev_lowest(int k, const double* lower, int nwant, double* W,
                       double* Vec) {
  std::vector<double> a(size_t(k) * k);
  for(int j = 0; j < k; ++j)
    for(int i = j; i < k; ++i) a[i + size_t(j) * k] = a[j + size_t(i) * k] = lower[i + size_t(j) * k];
  std::vector<double> d(k), e(k, 0.0);
  std::vector<std::vector<double>> refl;  // Householder vectors (length k)
  // tridiagonalise: A <- H A H with H = I - 2 v v^T acting on rows/cols j+1..
  for(int j = 0; j + 2 < k; ++j) {
    double nrm = 0;
    for(int i = j + 1; i < k; ++i) nrm += a[i + size_t(j) * k] * a[i + size_t(j) * k];
    nrm = std::sqrt(nrm);
    std::vector<double> v(k, 0.0);
    const double x0 = a[j + 1 + size_t(j) * k];
    if(nrm == 0) {
      refl.push_back(v);
      continue;
    }
    const double alpha = x0 > 0 ? -nrm : nrm;
    v[j + 1] = x0 - alpha;
    for(int i = j + 2; i < k; ++i) v[i] = a[i + size_t(j) * k];
    double vn = 0;
    for(int i = j + 1; i < k; ++i) vn += v[i] * v[i];
    vn = std::sqrt(vn);
    if(vn == 0) {
      refl.push_back(std::vector<double>(k, 0.0));
      continue;
    }
    for(int i = j + 1; i < k; ++i) v[i] /= vn;
    // p = A v ; K = v.p ; q = p - K v ; A <- A - 2 v q^T - 2 q v^T
    std::vector<double> p(k, 0.0);
    for(int c = j; c < k; ++c) {  // column c (= row c: a is symmetric)
      const double* ac = a.data() + size_t(c) * k;
      double s4[4] = {0, 0, 0, 0};  // four chains: the sum is latency-bound
      int r = j + 1;
      for(; r + 3 < k; r += 4)
        for(int q = 0; q < 4; ++q) s4[q] += ac[r + q] * v[r + q];
      for(; r < k; ++r) s4[0] += ac[r] * v[r];
      p[c] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    }
    double K = 0;
    for(int r = j + 1; r < k; ++r) K += v[r] * p[r];
    for(int r = j; r < k; ++r) p[r] -= K * v[r];
    for(int c = j; c < k; ++c)
      for(int r = j; r < k; ++r)
        a[r + size_t(c) * k] -= 2 * (v[r] * p[c] + p[r] * v[c]);
    refl.push_back(v);
  }
  for(int i = 0; i < k; ++i) d[i] = a[i + size_t(i) * k];
  for(int i = 0; i + 1 < k; ++i) e[i] = a[i + 1 + size_t(i) * k];
  // Gershgorin bounds
  double lo = d[0], hi = d[0];
  for(int i = 0; i < k; ++i) {
    const double r = (i ? std::fabs(e[i - 1]) : 0) + (i + 1 < k ? std::fabs(e[i]) : 0);
    lo = std::min(lo, d[i] - r);
    hi = std::max(hi, d[i] + r);
  }
  const double span = std::max({hi - lo, std::fabs(lo), std::fabs(hi), 1e-30});
  lo -= 1e-12 * span;
  hi += 1e-12 * span;
  const double tiny = 1e-15 * span;  // pivot floor of the shifted solves
  auto count_below = [&](double x) {  // Sturm count of eigenvalues < x
    int c = 0;
    double q = d[0] - x;
    if(q < 0) ++c;
    for(int i = 1; i < k; ++i) {
      if(q == 0) q = 1e-300;
      q = d[i] - x - e[i - 1] * e[i - 1] / q;
      if(q < 0) ++c;
    }
    return c;
  };
  nwant = std::min(nwant, k);
  std::vector<std::vector<double>> ztri;  // eigenvectors of the tridiagonal
  for(int m = 0; m < nwant; ++m) {
    double l = lo, h = hi;  // the m-th eigenvalue has count_below(x) > m
    for(int it = 0; it < 200 && h - l > 4e-16 * std::max(std::fabs(l), std::fabs(h)) + 1e-300; ++it) {
      const double mid = 0.5 * (l + h);
      if(count_below(mid) > m)
        h = mid;
      else
        l = mid;
    }
    W[m] = 0.5 * (l + h);
    // inverse iteration on T - lambda I (tridiagonal LU with pivoting-free
    // elimination, shifted slightly to stay regular)
    const double lam = W[m] + 1e-14 * span;
    auto floor_piv = [&](double x) {
      return std::fabs(x) < tiny ? (x < 0 ? -tiny : tiny) : x;
    };
    // start vector: deterministic, different per wanted pair
    std::vector<double> z(k), w2(k);
    for(int i = 0; i < k; ++i)
      z[i] = 1.0 + 0.5 * std::sin(0.7 * (i + 1) * (m + 1) + 0.3 * m);
    for(int it = 0; it < 5; ++it) {
      std::vector<double> dd(k), rhs = z;
      dd[0] = floor_piv(d[0] - lam);
      for(int i = 1; i < k; ++i) {
        const double f = e[i - 1] / dd[i - 1];
        dd[i] = floor_piv(d[i] - lam - f * e[i - 1]);
        rhs[i] -= f * rhs[i - 1];
      }
      w2[k - 1] = rhs[k - 1] / dd[k - 1];
      for(int i = k - 2; i >= 0; --i) w2[i] = (rhs[i] - e[i] * w2[i + 1]) / dd[i];
      // keep it orthogonal to the vectors of (nearly) equal eigenvalues
      for(int p = 0; p < m; ++p) {
        if(std::fabs(W[p] - W[m]) > 1e-7 * span) continue;
        double s2 = 0;
        for(int i = 0; i < k; ++i) s2 += ztri[p][i] * w2[i];
        for(int i = 0; i < k; ++i) w2[i] -= s2 * ztri[p][i];
      }
      double nn = 0;
      for(double x : w2) nn += x * x;
      nn = std::sqrt(nn);
      if(!(nn > 0) || !std::isfinite(nn)) break;
      for(int i = 0; i < k; ++i) z[i] = w2[i] / nn;
    }
    ztri.push_back(z);
    // back-transform: y = H_0 H_1 ... H_{k-3} z
    for(int r = int(refl.size()) - 1; r >= 0; --r) {
      const auto& v = refl[r];
      double s2 = 0;
      for(int i = 0; i < k; ++i) s2 += v[i] * z[i];
      for(int i = 0; i < k; ++i) z[i] -= 2 * s2 * v[i];
    }
    double nn = 0;
    for(double x : z) nn += x * x;
    nn = std::sqrt(nn);
    for(int i = 0; i < k; ++i) Vec[i + size_t(m) * k] = z[i] / nn;
  }
}

// out[:, j] = A[:, 0:k] Q[:, j] for j < keep (Q column-major, ld k): a thread
// keeps 8 output columns of its row in registers while it reads the row once.
// out may be A when keep <= 8 (a row is read whole before it is written).
__global__ void basis_rotate_k(const double* A, int64_t n, int k,
                               const double* __restrict__ Q, int keep,
                               double* out) {
  dav_wait();
  for(int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += int64_t(gridDim.x) * blockDim.x) {
    for(int j0 = 0; j0 < keep; j0 += DV_CHUNK) {
      double s[DV_CHUNK];
#pragma unroll
      for(int j = 0; j < DV_CHUNK; ++j) s[j] = 0;
#pragma unroll 4
      for(int c = 0; c < k; ++c) {
        const double a = A[i + c * n];
#pragma unroll
        for(int j = 0; j < DV_CHUNK; ++j)
          if(j0 + j < keep) s[j] += a * __ldg(Q + c + (j0 + j) * k);
      }
#pragma unroll
      for(int j = 0; j < DV_CHUNK; ++j)
        if(j0 + j < keep) out[i + (j0 + j) * n] = s[j];
    }
  }
}

// Phase timings of the last solve on this host thread
// (macis_b200_davidson_last_stats).
static thread_local macis_b200_davidson_stats g_dav_stats{};
const macis_b200_davidson_stats& davidson_last_stats() { return g_dav_stats; }

namespace {
// Device time per phase, summed over the solve: marks recorded on the solver
// stream at the phase boundaries of an iteration, read at the next
// synchronisation behind them.
struct PhaseMarks {
  static constexpr int N = 6;
  struct Set {  // the marks of one iteration
    cudaEvent_t e[N];
    double* acc[N] = {};  // where the time from mark i to mark i + 1 goes
  } set[2];
  int cur = 0;
  cudaStream_t s;
  explicit PhaseMarks(cudaStream_t st) : s(st) {
    for(auto& x : set)
      for(auto& y : x.e) cudaEventCreate(&y);
  }
  PhaseMarks(const PhaseMarks&) = delete;
  ~PhaseMarks() {
    for(auto& x : set)
      for(auto& y : x.e) cudaEventDestroy(y);
  }
  void mark(int i, double* into) {
    cudaEventRecord(set[cur].e[i], s);
    set[cur].acc[i] = into;
  }
  void wait(int i) const { MB_CUDA(cudaEventSynchronize(set[cur].e[i])); }
  // adds the phases of a set; its marks must have completed
  void collect(int which) {
    Set& x = set[which];
    for(int i = 0; i + 1 < N; ++i) {
      float ms = 0.f;
      if(x.acc[i] && cudaEventElapsedTime(&ms, x.e[i], x.e[i + 1]) == cudaSuccess)
        *x.acc[i] += ms;
      x.acc[i] = nullptr;
    }
  }
};

// Page-locked host memory the kernels write the few numbers into that the
// host needs each iteration.
struct HostResults {
  double* p = nullptr;
  cudaStream_t s;
  HostResults(size_t n, cudaStream_t st) : s(st) {
    MB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&p), n * 8, cudaHostAllocMapped));
  }
  HostResults(const HostResults&) = delete;
  ~HostResults() {
    cudaStreamSynchronize(s);  // kernels in flight may still write here
    cudaFreeHost(p);
  }
};

struct DavCtx {
  cudaStream_t s;
  int64_t n;
  unsigned nb;      // row blocks of the vector kernels
  double* partial;
  unsigned* done;   // arrival counters: one per column chunk, and one more
  double* dots;     // up to 1024 coefficients, then a norm
  DavCtx(cudaStream_t st, int64_t nn, int ncol, Arena& A) : s(st), n(nn) {
    nb = grid_for(size_t(nn), DV_THREADS, size_t(num_sms()) * 4);
    const size_t chunks = size_t(ncol + DV_CHUNK - 1) / DV_CHUNK;
    partial = A.get<double>(size_t(nb) * DV_CHUNK * (chunks + 1));
    done = A.get<unsigned>(chunks + 1);
    MB_CUDA(cudaMemsetAsync(done, 0, (chunks + 1) * sizeof(unsigned), st));
    dots = A.get<double>(1026);
  }
  template <class... P, class... Q>
  void launch(void (*kern)(P...), dim3 g, int threads, Q&&... args) const {
    cudaLaunchConfig_t c{};
    c.gridDim = g;
    c.blockDim = dim3(unsigned(threads));
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    MB_CUDA(cudaLaunchKernelEx(&c, kern, P(args)...));
    note_launch();
  }
  // out[0:ncol) = A^T v (columns of length n, leading dimension lda). Row
  // blocks: all of the vector's for short vectors, about 4 blocks an SM over
  // all chunks for long ones.
  void multidot(const double* A, int64_t lda, int ncol, const double* v,
                double* out) const {
    const unsigned ch = unsigned(ncol + DV_CHUNK - 1) / DV_CHUNK;
    const unsigned want = std::max(1u, unsigned(num_sms()) * 4 / ch);
    launch(multidot_k, dim3(std::min(nb, want), ch), DV_THREADS, A, lda, ncol,
           v, n, partial, done, out);
  }
  unsigned rows_grid() const {
    return std::min(nb, unsigned(num_sms()) * 4);
  }
  // gram_schmidt (davidson.hpp:111-126): CGS2 against K columns, normalise
  void cgs2(const double* Vb, int K, double* w) const {
    for(int pass = 0; pass < 2; ++pass) {
      multidot(Vb, n, K, w, dots);
      launch(cgs_update_k, dim3(rows_grid()), DV_THREADS, Vb, n, K, dots, w, n,
             partial, done, pass ? dots + 1024 : nullptr);
    }
    launch(scale_k, dim3(grid_for(size_t(n), 256, size_t(num_sms()) * 8)), 256,
           w, n, dots + 1024);
  }
};
}  // namespace

int davidson_device(const macis_b200_csr* A, int64_t max_m, double tol,
                    bool use_guess, double* X, double* E, int64_t* niter,
                    int restart_keep, int64_t max_iter) {
  MB_REQUIRE(A->m == A->n, MACIS_B200_EINVAL, "Davidson needs a square matrix");
  DavOperator op;
  op.n = A->m;
  op.diag = A->diag;
  op.s = A->stream;
  op.apply = [A](const double* x, double* y) {
    spmv_device_x64(A, 1.0, x, 0.0, y, A->stream);
  };
  return davidson_op(op, max_m, tol, use_guess, X, E, niter, restart_keep,
                     max_iter);
}

int davidson_op(const DavOperator& op, int64_t max_m, double tol,
                bool use_guess, double* X, double* E, int64_t* niter,
                int restart_keep, int64_t max_iter) {
  const int64_t N = op.n;
  MB_REQUIRE(N > 0, MACIS_B200_EINVAL, "Davidson: empty matrix");
  MB_REQUIRE(max_m >= 1 && max_m <= 1000, MACIS_B200_EINVAL,
             "Davidson: max_m must be in [1, 1000]");
  MB_REQUIRE(restart_keep >= 0 && restart_keep < max_m, MACIS_B200_EINVAL,
             "Davidson: restart_keep must be in [0, max_m)");
  NvtxRange nv("macis_b200: Davidson");
  cudaStream_t s = op.s;
  Arena Ar(s);
  const auto t_wall = std::chrono::steady_clock::now();
  macis_b200_davidson_stats st{};
  PhaseMarks marks(s);
  max_m = std::min<int64_t>(max_m, N);
  if(restart_keep >= max_m) restart_keep = int(max_m) - 1;
  const double* D = op.diag;
  if(!use_guess) unit_guess_k<<<1, 1024, 0, s>>>(D, N, X), note_launch();
  double* V = Ar.get<double>(size_t(N) * (max_m + 1));
  double* AV = Ar.get<double>(size_t(N) * (max_m + 1));
  double* tmp = restart_keep > DV_CHUNK
                    ? Ar.get<double>(size_t(N) * restart_keep)
                    : nullptr;
  const int ld = int(max_m + 1);
  DavCtx ctx(s, N, ld, Ar);
  // host-visible results: the Rayleigh row (ld), then |R|^2
  HostResults res(size_t(ld) + 1, s);
  MB_CUDA(cudaMemcpyAsync(V, X, N * 8, cudaMemcpyDeviceToDevice, s));
  op.apply(V, AV);
  MB_CUDA(cudaMemcpyAsync(V + N, AV, N * 8, cudaMemcpyDeviceToDevice, s));
  ctx.cgs2(V, 1, V + N);

  std::vector<double> Cl(size_t(ld) * ld, 0.0), lower, W(ld), Vec;
  // first entry of the Rayleigh matrix, V_0 . AV_0
  ctx.multidot(AV, N, 1, V, res.p);
  MB_CUDA(cudaStreamSynchronize(s));
  Cl[0] = res.p[0];
  double* d_c = Ar.get<double>(size_t(ld) * ld + 2);
  bool converged = false;
  int64_t iter = 1;
  double lam0 = 0;
  int64_t i = 1;  // index of the newest basis vector (AV_i not yet formed)
  for(;; ++iter) {
    const int k = int(i + 1);
    marks.cur = int(iter & 1);
    marks.mark(0, &st.apply_ms);
    op.apply(V + i * N, AV + i * N);
    // new row of V^T AV: V_i . AV_c for c <= i (lower triangle)
    marks.mark(1, &st.rayleigh_ms);
    ctx.multidot(AV, N, k, V + i * N, res.p);
    marks.mark(2, nullptr);
    st.vector_bytes += double(N) * (k + 1) * 8;
    MB_CUDA(cudaStreamSynchronize(s));
    marks.collect(marks.cur ^ 1);
    for(int c = 0; c < k; ++c) Cl[i + size_t(c) * ld] = res.p[c];
    lower.assign(size_t(k) * k, 0.0);
    for(int c = 0; c < k; ++c)
      for(int r = c; r < k; ++r) lower[r + size_t(c) * k] = Cl[r + size_t(c) * ld];
    // the lowest pair; a restart of a full basis takes restart_keep of them
    const int nwant = k >= max_m ? std::max(1, std::min(restart_keep, k)) : 1;
    Vec.assign(size_t(k) * nwant, 0.0);
    small_syev_lowest(k, lower.data(), nwant, W.data(), Vec.data());
    lam0 = W[0];
    RitzCoef rc;
    rc.dev = nullptr;
    if(k <= DV_PARAM_COEF) {
      std::copy(Vec.begin(), Vec.begin() + k, rc.c);
    } else {
      rc.dev = d_c;
    }
    if(rc.dev || nwant > 1)
      MB_CUDA(cudaMemcpyAsync(d_c, Vec.data(), size_t(k) * nwant * 8,
                              cudaMemcpyHostToDevice, s));
    double* R = V + size_t(k) * N;
    marks.mark(3, &st.residual_ms);
    ctx.launch(ritz_residual_k, dim3(ctx.rows_grid()), DV_THREADS, V, AV, N, k,
               rc, lam0, D, X, R, ctx.partial, ctx.done, res.p + ld);
    marks.mark(4, &st.ortho_ms);
    st.vector_bytes += double(N) * (2.0 * k + 3) * 8;
    // the next direction is orthonormalised behind the residual while the
    // host waits for its norm (not used when that has converged)
    const bool full = k >= max_m;
    if(!full && !(max_iter > 0 && iter >= max_iter)) {
      ctx.cgs2(V, k, R);
      st.vector_bytes += double(N) * (4.0 * k + 9) * 8;
    }
    marks.mark(5, nullptr);
    marks.wait(4);
    if(std::sqrt(res.p[ld]) < tol) {
      converged = true;
      break;
    }
    if(full) {
      // the reference stops here (davidson.hpp:161, 221)
      if(!restart_keep || (max_iter > 0 && iter >= max_iter)) break;
      // thick restart: keep the lowest restart_keep Ritz vectors
      const int keep = restart_keep;
      const dim3 g(grid_for(size_t(N), 256, size_t(num_sms()) * 8));
      // two rotations (read k columns, write keep), the copy of R, then CGS2
      // over keep columns
      st.vector_bytes += double(N) * (2.0 * k + 2.0 * keep + 2) * 8 +
                         double(N) * (4.0 * keep + 9) * 8;
      for(double* B : {V, AV}) {
        ctx.launch(basis_rotate_k, g, 256, B, N, k, d_c, keep, tmp ? tmp : B);
        if(tmp)
          MB_CUDA(cudaMemcpyAsync(B, tmp, size_t(N) * keep * 8,
                                  cudaMemcpyDeviceToDevice, s));
      }
      MB_CUDA(cudaMemcpyAsync(V + size_t(keep) * N, R, N * 8,
                              cudaMemcpyDeviceToDevice, s));
      std::fill(Cl.begin(), Cl.end(), 0.0);
      for(int c = 0; c < keep; ++c) Cl[c + size_t(c) * ld] = W[c];
      ctx.cgs2(V, keep, V + size_t(keep) * N);
      marks.mark(5, nullptr);
      i = keep;
    } else {
      if(max_iter > 0 && iter >= max_iter) break;
      i = k;
    }
  }
  MB_CUDA(cudaGetLastError());
  MB_CUDA(cudaStreamSynchronize(s));
  marks.collect(0);
  marks.collect(1);
  st.iterations = iter;
  st.wall_ms = std::chrono::duration<double, std::milli>(
                   std::chrono::steady_clock::now() - t_wall)
                   .count();
  g_dav_stats = st;
  *E = lam0;
  *niter = iter;
  return converged ? 0 : MACIS_B200_ENOCONV;
}

}  // namespace mb
