// Single-vector Davidson on the GPU, replacing macis::davidson
// (include/macis/solvers/davidson.hpp:129-225) and diagonal_guess (:62-68).
//
// Basis V and A*V live in HBM (N x (max(max_m, 2) + 1) FP64 each). Per iteration:
//   AV_i = H V_i                                  (spmv.cu)
//   row i of the Rayleigh matrix V^T AV           (multidot_k, FP64)
//   k x k symmetric eigenproblem on the host      (eig.cpp, lowest pair)
//   X = V c, R = AV c - lambda X, |R|, W = -R/(D - lambda), then CGS2 of W
//   against V and its norm (davidson.hpp:111-126) (dav_step_k, one launch)
// The reference recomputes the full k x k product with gemm every
// iteration; only its lower triangle enters syev (rayleigh_ritz.hpp:73-75),
// and the entries of earlier rows do not change, so only the new row is
// formed. Reductions are two-stage with a fixed order (deterministic).
//
// For a basis that L2 holds, an iteration is bound by launches and by the
// two round trips to the host, so it is three launches (product, Rayleigh
// row, step), the kernels write what the host needs (the row, |R|^2, phase
// times) to page-locked memory with a sequence number that the host polls,
// and the host decides on convergence while the step still orthonormalises.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.hpp"
#include "primitives.cuh"

namespace mb {

constexpr int DV_THREADS = 512;
constexpr int DV_WARPS = DV_THREADS / 32;
constexpr int DV_CHUNK = 8;  // columns held by one multi-dot block

// Waits for the preceding kernel of the stream: these kernels are launched
// with programmatic serialization, so that their launch work overlaps it.
__device__ __forceinline__ void dav_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// What the kernels report to the host, in page-locked host memory.
struct DavReport {
  volatile unsigned row_seq;   // the Rayleigh row of this number is there
  volatile unsigned res_seq;   // |R|^2 of this number is there
  volatile unsigned err;       // a grid barrier gave up
  volatile double rn2;
  // phase boundaries, ns: the product's start, the row's kernel, the step's
  // residual, its end
  volatile unsigned long long t_app0, t_row0, t_row1, t_res0, t_res1, t_end;
  volatile double row[1];      // an entry per basis column
};

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

// rep->row[c] = A[:, c] . v for c < ncol: block (x, y) sums rows x, x +
// gridDim.x, ... (in units of DV_THREADS) of the DV_CHUNK columns from
// DV_CHUNK y, the last block of a chunk adds the chunk's partial sums in a
// fixed order, and the last chunk reports. HBM-bound for long vectors.
// done: one counter per chunk, one for the chunks; t0: scratch, and the start
// of the product before it, which is reported with the row (a product that
// wrote it to host memory itself ended about 2 us later).
__global__ void __launch_bounds__(DV_THREADS)
    multidot_k(const double* __restrict__ A, int64_t lda, int ncol,
               const double* __restrict__ v, int64_t n, double* partial,
               unsigned* done, unsigned long long* t0, DavReport* rep,
               unsigned seq) {
  __shared__ double sh[DV_WARPS][DV_CHUNK];
  dav_wait();
  if(blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *t0 = gpu_time_ns();
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
  if(!last_block(done + blockIdx.y, gridDim.x)) return;
  if(wid < nc) {
    const double t = warp_sum_partials(pc + wid, int(gridDim.x), DV_CHUNK);
    if(lane == 0) rep->row[c0 + wid] = t;
  }
  __threadfence_system();  // before the report of the last chunk
  if(last_block(done + gridDim.y, gridDim.y) && threadIdx.x == 0) {
    const ulonglong2 t = __ldcg(reinterpret_cast<const ulonglong2*>(t0));
    rep->t_row0 = t.x;
    rep->t_app0 = t.y;
    rep->t_row1 = gpu_time_ns();
    __threadfence_system();
    rep->row_seq = seq;
  }
}

// Ritz coefficients passed with the launch (no copy to the device) up to
// this many; longer vectors come from device memory.
constexpr int DV_PARAM_COEF = 128;
struct RitzCoef {
  double c[DV_PARAM_COEF];
  const double* dev;  // used when not null
};

struct StepArgs {
  const double* V;
  const double* AV;
  int64_t n;
  int k;             // basis vectors
  int ritz;          // form X and the correction W (else W is given)
  int ortho;         // CGS2 and normalise W
  double lam;
  const double* D;
  double* X;
  double* W;
  double* partial;   // 2 x k x blocks, then 2 x blocks
  unsigned* done;    // arrival counter
  unsigned* bar;     // barrier counter, grows by `blocks` per barrier
  unsigned bar0;     // its value before this launch
  DavReport* rep;
  unsigned seq;
};

// Barrier over the blocks of a cooperative launch (they are all resident).
// The wait is bounded: a block that gives up reports it and the kernel ends.
constexpr int DV_SPIN_LIMIT = 1 << 24;  // polls of about 0.5 us
__device__ __forceinline__ bool grid_barrier(const StepArgs& a,
                                             unsigned& target) {
  __shared__ bool ok;
  target += gridDim.x;
  __syncthreads();
  if(gridDim.x == 1) return true;
  if(threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.bar, 1u);
    ok = false;
    for(int t = 0; t < DV_SPIN_LIMIT; ++t) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
      if(int(v - target) >= 0) {
        ok = true;
        break;
      }
    }
    if(!ok) a.rep->err = 1;
  }
  __syncthreads();
  return ok;
}

__device__ __forceinline__ double block_sum(double acc, double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for(int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __syncthreads();
  if(lane == 0) sh[wid] = acc;
  __syncthreads();
  double t = 0;
  for(int w = 0; w < DV_WARPS; ++w) t += sh[w];
  return t;
}

// One step behind the Rayleigh row: Ritz vector, residual and correction,
//   X = V c; R = AV c - lam X; |R|^2; W = -R / (D - lam),
// then gram_schmidt (davidson.hpp:111-126), W -= V (V^T W) twice and W /= |W|.
// A thread keeps its rows through all phases; the column sums meet at three
// grid barriers (their partial sums added by every block in the same order).
// One cooperative launch: as five launches the same work took 2 to 4 us each
// on a basis of 63,504 x 40, about a launch latency, whatever its size.
// For long vectors it streams V three times and AV once from HBM.
__global__ void __launch_bounds__(DV_THREADS, 2)
    dav_step_k(StepArgs a, const __grid_constant__ RitzCoef rc) {
  __shared__ double cf[1024];
  __shared__ double shc[2][DV_WARPS][DV_CHUNK];
  __shared__ double shb[DV_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n = a.n;
  const int k = a.k, nb = int(gridDim.x);
  const int64_t i0 = int64_t(blockIdx.x) * DV_THREADS + threadIdx.x;
  const int64_t di = int64_t(nb) * DV_THREADS;
  const double* __restrict__ V = a.V;
  double* W = a.W;
  double* pn = a.partial + size_t(2) * k * nb;  // |R|^2, then |W|^2
  unsigned target = a.bar0;
  if(blockIdx.x == 0 && threadIdx.x == 0 && a.ritz) a.rep->t_res0 = gpu_time_ns();
  if(a.ritz) {
    for(int j = threadIdx.x; j < k; j += DV_THREADS)
      cf[j] = rc.dev ? rc.dev[j] : rc.c[j];
    __syncthreads();
    const double* __restrict__ AV = a.AV;
    double acc = 0;
    for(int64_t i = i0; i < n; i += di) {
      double x = 0, av = 0;
#pragma unroll 8
      for(int j = 0; j < k; ++j) {
        x += V[i + j * n] * cf[j];
        av += AV[i + j * n] * cf[j];
      }
      const double r = av - a.lam * x;
      a.X[i] = x;
      W[i] = -r / (a.D[i] - a.lam);
      acc += r * r;
    }
    const double t = block_sum(acc, shb);
    if(threadIdx.x == 0) pn[blockIdx.x] = t;
    if(last_block(a.done, unsigned(nb)) && wid == 0) {
      const double s = warp_sum_partials(pn, nb, 1);
      if(lane == 0) {
        a.rep->rn2 = s;
        a.rep->t_res1 = gpu_time_ns();
        __threadfence_system();
        a.rep->res_seq = a.seq;
      }
    }
  }
  if(a.ortho) {
    for(int pass = 0; pass < 2; ++pass) {
      // column sums of V^T W over this block's rows
      double* pc = a.partial + size_t(pass) * k * nb;
      for(int c0 = 0; c0 < k; c0 += DV_CHUNK) {
        double acc[DV_CHUNK];
#pragma unroll
        for(int c = 0; c < DV_CHUNK; ++c) acc[c] = 0;
        for(int64_t i = i0; i < n; i += di) {
          const double x = W[i];
#pragma unroll
          for(int c = 0; c < DV_CHUNK; ++c)
            if(c0 + c < k) acc[c] += V[i + (c0 + c) * n] * x;
        }
        double (*sh)[DV_CHUNK] = shc[(c0 / DV_CHUNK) & 1];
        const double t = warp_sum8(acc);
        if((lane & 3) == 0)
          sh[wid][(lane >> 4) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)] = t;
        __syncthreads();
        if(threadIdx.x < DV_CHUNK && c0 + int(threadIdx.x) < k) {
          double u = 0;
#pragma unroll
          for(int w = 0; w < DV_WARPS; ++w) u += sh[w][threadIdx.x];
          pc[size_t(c0 + threadIdx.x) * nb + blockIdx.x] = u;
        }
      }
      if(!grid_barrier(a, target)) return;
      for(int c = wid; c < k; c += DV_WARPS) {
        const double u = warp_sum_partials(pc + size_t(c) * nb, nb, 1);
        if(lane == 0) cf[c] = u;
      }
      __syncthreads();
      double acc = 0;
      for(int64_t i = i0; i < n; i += di) {
        double s = 0;
#pragma unroll 8
        for(int c = 0; c < k; ++c) s += V[i + c * n] * cf[c];
        const double x = W[i] - s;
        W[i] = x;
        acc += x * x;
      }
      if(pass) {
        const double t = block_sum(acc, shb);
        if(threadIdx.x == 0) pn[nb + blockIdx.x] = t;
      } else {
        __syncthreads();  // cf is rewritten behind the next barrier
      }
    }
    if(!grid_barrier(a, target)) return;
    if(wid == 0) {
      const double s = warp_sum_partials(pn + nb, nb, 1);
      if(lane == 0) shb[0] = 1. / sqrt(s);
    }
    __syncthreads();
    const double inv = shb[0];
    for(int64_t i = i0; i < n; i += di) W[i] *= inv;
  }
  if(blockIdx.x == 0 && threadIdx.x == 0) a.rep->t_end = gpu_time_ns();
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
struct DavCtx {
  cudaStream_t s;
  int64_t n;
  unsigned nb;            // row blocks
  unsigned step_blocks;   // blocks of a step (all resident)
  double* partial;
  unsigned* done;         // arrival counters: per column chunk, of the chunks
  unsigned* bar;
  unsigned long long* t0;  // starts of the row's kernel and of the product
  unsigned nbar = 0;      // barrier arrivals so far
  unsigned seq = 0;
  DavReport* rep = nullptr;
  std::shared_ptr<PinnedPool> pool;
  DavCtx(cudaStream_t st, int64_t nn, int ncol, Arena& A,
         const std::shared_ptr<PinnedPool>& pin)
      : s(st), n(nn), pool(pin ? pin : std::make_shared<PinnedPool>()) {
    nb = grid_for(size_t(nn), DV_THREADS, size_t(num_sms()) * 4);
    int per_sm = 0;
    MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dav_step_k,
                                                          DV_THREADS, 0));
    step_blocks = std::min(nb, unsigned(num_sms() * std::min(2, std::max(1, per_sm))));
    const size_t chunks = size_t(ncol + DV_CHUNK - 1) / DV_CHUNK;
    partial = A.get<double>(std::max(size_t(nb) * DV_CHUNK * chunks,
                                     (size_t(2) * ncol + 2) * step_blocks));
    done = A.get<unsigned>(chunks + 3);
    bar = done + chunks + 2;
    MB_CUDA(cudaMemsetAsync(done, 0, (chunks + 3) * sizeof(unsigned), st));
    t0 = A.get<unsigned long long>(2);
    const size_t bytes = sizeof(DavReport) + size_t(ncol) * 8;
    MB_REQUIRE(bytes <= PinnedPool::BYTES, MACIS_B200_EINVAL,
               "Davidson: subspace too large");
    rep = static_cast<DavReport*>(pool->take());
    memset(static_cast<void*>(rep), 0, bytes);
  }
  DavCtx(const DavCtx&) = delete;
  ~DavCtx() {
    cudaStreamSynchronize(s);  // kernels in flight may still report
    if(rep) pool->give(rep);
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
  // rep->row[0:ncol) = A^T v (columns of length n). Row blocks: all of the
  // vector's for short vectors, about 4 blocks an SM over all chunks for long
  // ones.
  void multidot(const double* A, int ncol, const double* v) {
    const unsigned ch = unsigned(ncol + DV_CHUNK - 1) / DV_CHUNK;
    const unsigned want = std::max(1u, unsigned(num_sms()) * 4 / ch);
    launch(multidot_k, dim3(std::min(nb, want), ch), DV_THREADS, A, n, ncol, v,
           n, partial, done, t0, rep, ++seq);
  }
  void step(StepArgs a, const RitzCoef& rc) {
    a.n = n;
    a.partial = partial;
    a.done = done;
    a.bar = bar;
    a.bar0 = nbar;
    a.rep = rep;
    a.seq = a.ritz ? ++seq : seq;
    if(a.ortho && step_blocks > 1) nbar += 3 * step_blocks;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(step_blocks);
    c.blockDim = dim3(DV_THREADS);
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    MB_CUDA(cudaLaunchKernelEx(&c, dav_step_k, a, rc));
    note_launch();
  }
  // Waits for the report numbered seq: polls for about the time that the
  // vector work of a short iteration takes, then leaves the waiting to the
  // runtime (long products).
  void wait(const volatile unsigned& flag) const {
    const auto t = std::chrono::steady_clock::now();
    while(flag != seq) {
      if(std::chrono::steady_clock::now() - t > std::chrono::microseconds(300)) {
        MB_CUDA(cudaStreamSynchronize(s));
        MB_REQUIRE(flag == seq, MACIS_B200_ETIMEOUT,
                   "Davidson: a grid barrier timed out");
      }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    MB_REQUIRE(!rep->err, MACIS_B200_ETIMEOUT,
               "Davidson: a grid barrier timed out");
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
  op.pinned = A->pinned;
  op.apply = [A](const double* x, double* y, unsigned long long* t0) {
    spmv_device_x64(A, 1.0, x, 0.0, y, A->stream, t0);
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
  max_m = std::min<int64_t>(max_m, N);
  if(restart_keep >= max_m) restart_keep = int(max_m) - 1;
  const double* D = op.diag;
  if(!use_guess || N == 1) unit_guess_k<<<1, 1024, 0, s>>>(D, N, X), note_launch();
  auto wall_ms = [&] {
    return std::chrono::duration<double, std::milli>(
               std::chrono::steady_clock::now() - t_wall)
        .count();
  };
  if(N == 1) {  // no second basis vector: the product of the unit vector
    double* y = Ar.get<double>(1);
    op.apply(X, y, nullptr);
    *E = to_host(y, s);
    *niter = st.iterations = 1;
    st.wall_ms = wall_ms();
    g_dav_stats = st;
    return std::isfinite(*E) ? 0 : MACIS_B200_ENOCONV;
  }
  // the first step has two basis vectors, whatever max_m, and writes a third
  const int64_t cols = std::max<int64_t>(max_m, 2) + 1;
  double* V = Ar.get<double>(size_t(N) * cols);
  double* AV = Ar.get<double>(size_t(N) * cols);
  double* tmp = restart_keep > DV_CHUNK
                    ? Ar.get<double>(size_t(N) * restart_keep)
                    : nullptr;
  const int ld = int(cols);
  DavCtx ctx(s, N, ld, Ar, op.pinned);
  RitzCoef rc;
  rc.dev = nullptr;
  StepArgs sa{};
  sa.V = V;
  sa.AV = AV;
  sa.D = D;
  sa.X = X;
  auto orthonormalise = [&](int k, double* w) {
    StepArgs o = sa;
    o.k = k;
    o.ortho = 1;
    o.W = w;
    ctx.step(o, rc);
  };
  MB_CUDA(cudaMemcpyAsync(V, X, N * 8, cudaMemcpyDeviceToDevice, s));
  op.apply(V, AV, nullptr);
  MB_CUDA(cudaMemcpyAsync(V + N, AV, N * 8, cudaMemcpyDeviceToDevice, s));
  orthonormalise(1, V + N);

  std::vector<double> Cl(size_t(ld) * ld, 0.0), lower, W(ld), Vec;
  // first entry of the Rayleigh matrix, V_0 . AV_0
  ctx.multidot(AV, 1, V);
  ctx.wait(ctx.rep->row_seq);
  Cl[0] = ctx.rep->row[0];
  double* d_c = Ar.get<double>(size_t(ld) * ld + 2);
  auto ms = [](unsigned long long a, unsigned long long b) {
    return b > a ? double(b - a) * 1e-6 : 0.0;
  };
  bool converged = false;
  int64_t iter = 1;
  double lam0 = 0;
  int64_t i = 1;  // index of the newest basis vector (AV_i not yet formed)
  for(;; ++iter) {
    const int k = int(i + 1);
    op.apply(V + i * N, AV + i * N, ctx.t0 + 1);
    // new row of V^T AV: V_i . AV_c for c <= i (lower triangle)
    ctx.multidot(AV, k, V + i * N);
    st.vector_bytes += double(N) * (k + 1) * 8;
    ctx.wait(ctx.rep->row_seq);
    // the step before has ended too: its last phase; then the product, timed
    // from its own start (the GPU may have waited for the host before it), and
    // the row
    if(iter > 1) st.ortho_ms += ms(ctx.rep->t_res1, ctx.rep->t_end);
    st.apply_ms += ms(ctx.rep->t_app0, ctx.rep->t_row0);
    st.rayleigh_ms += ms(ctx.rep->t_row0, ctx.rep->t_row1);
    for(int c = 0; c < k; ++c) Cl[i + size_t(c) * ld] = ctx.rep->row[c];
    lower.assign(size_t(k) * k, 0.0);
    for(int c = 0; c < k; ++c)
      for(int r = c; r < k; ++r) lower[r + size_t(c) * k] = Cl[r + size_t(c) * ld];
    // the lowest pair; a restart of a full basis takes restart_keep of them
    const bool full = k >= max_m;
    const int nwant = full ? std::max(1, std::min(restart_keep, k)) : 1;
    Vec.assign(size_t(k) * nwant, 0.0);
    small_syev_lowest(k, lower.data(), nwant, W.data(), Vec.data());
    lam0 = W[0];
    if(k <= DV_PARAM_COEF)
      std::copy(Vec.begin(), Vec.begin() + k, rc.c);
    else
      rc.dev = d_c;
    if(rc.dev || nwant > 1)
      MB_CUDA(cudaMemcpyAsync(d_c, Vec.data(), size_t(k) * nwant * 8,
                              cudaMemcpyHostToDevice, s));
    double* R = V + size_t(k) * N;
    const bool last = max_iter > 0 && iter >= max_iter;
    StepArgs a = sa;
    a.k = k;
    a.ritz = 1;
    // the next direction is orthonormalised while the host looks at |R|^2
    // (for nothing when that has converged)
    a.ortho = !full && !last;
    a.lam = lam0;
    a.W = R;
    ctx.step(a, rc);
    st.vector_bytes += double(N) * (2.0 * k + 3) * 8;
    if(a.ortho) st.vector_bytes += double(N) * (4.0 * k + 9) * 8;
    ctx.wait(ctx.rep->res_seq);
    st.residual_ms += ms(ctx.rep->t_res0, ctx.rep->t_res1);
    if(std::sqrt(ctx.rep->rn2) < tol) {
      converged = true;
      break;
    }
    if(full) {
      // the reference stops here (davidson.hpp:161, 221)
      if(!restart_keep || last) break;
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
      orthonormalise(keep, V + size_t(keep) * N);
      i = keep;
    } else {
      if(last) break;
      i = k;
    }
  }
  MB_CUDA(cudaGetLastError());
  MB_CUDA(cudaStreamSynchronize(s));
  st.iterations = iter;
  st.wall_ms = wall_ms();
  g_dav_stats = st;
  *E = lam0;
  *niter = iter;
  return converged ? 0 : MACIS_B200_ENOCONV;
}

}  // namespace mb
