// CSR Hamiltonian build on the GPU -- the B200 replacement of
// DoubleLoopHamiltonianGenerator::make_csr_hamiltonian_block_
// (include/macis/hamiltonian_generator/double_loop.hpp:31-98).
//
// The reference tests every (bra, ket) pair. Here the ket determinants are
// grouped by alpha string and only alpha strings within two excitations of
// the bra alpha are visited ("sorted double loop over unique alpha strings
// and their beta partners"):
//
//  * Direct-product path (CAS / full-CI spaces, the order of
//    generate_hilbert_space, sd_operations.hpp:461-476): det i = (A, B) with
//    A = i / UB, B = i % UB. Per alpha string A the list of A' within two
//    excitations and per beta string B the lists of B' within one and two
//    excitations are precomputed with their packed (hole, particle, sign)
//    data, so a row is emitted as the concatenation over ascending A' of the
//    ascending B' lists: columns come out sorted with no search and no sort,
//    and every entry costs one list read and one integral gather.
//  * General path (selected spaces): kets sorted by (alpha, beta); per row
//    the connected alpha groups are scanned with popcount tests (exact-beta
//    binary search for alpha doubles); candidates are sorted by column in
//    shared memory (rows above 1024 candidates go through the radix sort).
//
// Both paths count candidates first (|h| > thresh applied in the fill), so
// rows are written once at their final position unless some element falls
// below the threshold, in which case a compaction pass closes the gaps.
// Matrix elements follow the reference summation order exactly
// (common.cuh), so values are bit-identical to the reference.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "internal.hpp"
#include "primitives.cuh"

namespace mb {

constexpr int HB_WARPS = 4;
constexpr int HB_THREADS = 32 * HB_WARPS;
constexpr int GEN_CAP = 1024;  // candidates sorted in shared memory per warp
// bytes of candidate lists up to which the free memory is not asked for
constexpr uint64_t GEN_LIST_ASK = uint64_t(256) << 20;

template <int NSW>
__device__ __forceinline__ int sp_cmp(const Spin<NSW>& a, const Spin<NSW>& b) {
#pragma unroll
  for(int j = NSW - 1; j >= 0; --j) {
    if(a.w[j] < b.w[j]) return -1;
    if(a.w[j] > b.w[j]) return 1;
  }
  return 0;
}

template <int NSW>
__device__ __forceinline__ Spin<NSW> ld_spin(const uint64_t* p, size_t i) {
  Spin<NSW> s;
#pragma unroll
  for(int j = 0; j < NSW; ++j) s.w[j] = p[i * NSW + j];
  return s;
}
template <int NSW>
__device__ __forceinline__ void st_spin(uint64_t* p, size_t i, Spin<NSW> s) {
#pragma unroll
  for(int j = 0; j < NSW; ++j) p[i * NSW + j] = s.w[j];
}

__device__ __forceinline__ int warp_incl_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for(int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, v, o);
    if(lane >= o) v += y;
  }
  return v;
}

// ----------------------------------------------------- spin extraction
template <int NBITS>
__global__ void split_spins_k(const uint64_t* dets, size_t n, uint64_t* a,
                              uint64_t* b) {
  using D = DetTraits<NBITS>;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    const uint64_t* d = dets + i * D::NW;
    if(a) st_spin<D::NSW>(a, i, D::alpha(d));
    if(b) st_spin<D::NSW>(b, i, D::beta(d));
  }
}

// ------------------------------------------------ direct-product detection
template <int NBITS>
__global__ void first_alpha_change_k(const uint64_t* dets, size_t n,
                                     unsigned long long* first) {
  // block-wide minimum first, one atomic per block
  using D = DetTraits<NBITS>;
  __shared__ unsigned long long wmin[32];
  const auto a0 = D::alpha(dets);
  unsigned long long best = ~0ull;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x)
    if(!(D::alpha(dets + i * D::NW) == a0)) {
      best = i;
      break;  // later i of this thread are larger
    }
  for(int o = 16; o; o >>= 1) {
    const unsigned long long y = __shfl_xor_sync(0xffffffffu, best, o);
    best = y < best ? y : best;
  }
  if((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = best;
  __syncthreads();
  if(threadIdx.x == 0) {
    for(int w = 1; w < int(blockDim.x >> 5); ++w) best = wmin[w] < best ? wmin[w] : best;
    if(best != ~0ull) atomicMin(first, best);
  }
}

// Flags any determinant that breaks the (A = i/UB, B = i%UB) product layout,
// is zero, or changes the electron count of a spin.
template <int NBITS>
__global__ void dp_check_k(const uint64_t* dets, size_t n, size_t ub,
                           int* bad) {
  using D = DetTraits<NBITS>;
  const auto a0 = D::alpha(dets), b0 = D::beta(dets);
  const int pa = sp_popc(a0), pb = sp_popc(b0);
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    const uint64_t* d = dets + i * D::NW;
    const auto a = D::alpha(d), b = D::beta(d);
    const size_t A = i / ub, B = i % ub;
    bool ok = a == D::alpha(dets + A * ub * D::NW) &&
              b == D::beta(dets + B * D::NW) && sp_popc(a) == pa &&
              sp_popc(b) == pb && (pa + pb) > 0;
    if(!ok) atomicOr(bad, 1);
  }
}

template <int NBITS>
__global__ void gather_block_spins_k(const uint64_t* dets, size_t ua,
                                     size_t ub, uint64_t* alphas,
                                     uint64_t* betas) {
  using D = DetTraits<NBITS>;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
      i < (ua > ub ? ua : ub); i += size_t(gridDim.x) * blockDim.x) {
    if(i < ua) st_spin<D::NSW>(alphas, i, D::alpha(dets + i * ub * D::NW));
    if(i < ub) st_spin<D::NSW>(betas, i, D::beta(dets + i * D::NW));
  }
}

// ----------------------------------------------------- spin connectivity
// What the direct-product plan needs to know before it can allocate.
struct DPTotals {
  int64_t na, n2, n4, nnz;      // entries of the lists, of the matrix
  int dup;                      // some string occurs twice
  int l2max, l4max;             // longest beta lists
  unsigned long long dropped;   // elements below the threshold (fill)
};

// Per string l the connected strings of the same list: at popcount 0, 2 and
// 4 (cls[3 l ..]), within 2 (cnt2) and within 4 (cnt4). Warp per string.
// Strings that occur twice and the longest lists are noted on the way, which
// a sort of the strings and a copy of all list offsets were needed for.
template <int NSW>
__global__ void dp_conn_count_k(const uint64_t* strs, size_t ns, int32_t* cls,
                                int64_t* cnt2, int64_t* cnt4, int beta,
                                DPTotals* tot) {
  const int lane = threadIdx.x & 31;
  const size_t nwarp = size_t(gridDim.x) * (blockDim.x >> 5);
  for(size_t l = size_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      l < ns; l += nwarp) {
    const Spin<NSW> L = ld_spin<NSW>(strs, l);
    int c0 = 0, c2 = 0, c4 = 0;
    for(size_t r = lane; r < ns; r += 32) {
      const int p = sp_popc(L ^ ld_spin<NSW>(strs, r));
      c0 += p == 0;
      c2 += p == 2;
      c4 += p == 4;
    }
#pragma unroll
    for(int o = 16; o; o >>= 1) {
      c0 += __shfl_xor_sync(0xffffffffu, c0, o);
      c2 += __shfl_xor_sync(0xffffffffu, c2, o);
      c4 += __shfl_xor_sync(0xffffffffu, c4, o);
    }
    if(lane == 0) {
      cls[3 * l] = c0;
      cls[3 * l + 1] = c2;
      cls[3 * l + 2] = c4;
      cnt2[l] = c0 + c2;
      cnt4[l] = c0 + c2 + c4;
      if(c0 > 1) atomicOr(&tot->dup, 1);
      if(beta) {
        atomicMax(&tot->l2max, c0 + c2);
        atomicMax(&tot->l4max, c0 + c2 + c4);
      }
    }
  }
}

struct DPData {
  int64_t UA, UB;
  const uint64_t* ua;      // UA spins
  const uint64_t* ub;      // UB spins
  const int64_t* aoff;     // UA+1
  const int32_t* acol;     // A'
  const uint32_t* ainfo;   // packed, pa in bits 29..31
  const int64_t* l2off;    // UB+1
  const int32_t* l2col;
  const uint32_t* l2info;
  const int64_t* l4off;    // UB+1
  const int32_t* l4col;
  const uint32_t* l4info;
  // same-spin parts of the single-excitation elements (dp_pg_k)
  // at string x no nv (the electron counts of a product space are fixed)
  const double* pga;
  const double* pgb;
  // signed G value of every double of the alpha and beta L4 lists (0 for
  // the other entries): the fill reads it with the list entry instead of
  // gathering G
  const double* aval;
  const double* l4val;
};

// Occupied and empty orbitals of a spin string, in ascending order, into
// occ[0..no) and vir[0..n-no) (one orbital per lane).
template <int NSW>
__device__ __forceinline__ void spin_lists(const Spin<NSW>& s, int n, int lane,
                                           uint8_t* occ, uint8_t* vir) {
  for(int i = lane; i < n; i += 32) {
    int below = 0;  // occupied orbitals below i
#pragma unroll
    for(int w = 0; w < NSW; ++w) {
      const int lo = 64 * w;
      if(i > lo)
        below += __popcll(s.w[w] &
                          (i - lo >= 64 ? ~0ull : ((1ull << (i - lo)) - 1)));
    }
    if(sp_test(s, i))
      occ[below] = uint8_t(i);
    else
      vir[i - below] = uint8_t(i);
  }
}

// Same-spin part of every single excitation of every spin string s:
//   pg[s no nv + i nv + j] = T(v,o) + sum_{p in occ(s)} G_red(p,v,o)
// with v the i-th occupied and o the j-th empty orbital of s, summed in the
// order of matrix_element_2 (matrix_elements.hpp:86-104: T, then the
// same-spin G_red terms by ascending p). The element of a determinant adds
// the other-spin V_red terms to this partial sum in the same order, so the
// split is bit-exact. One warp per string.
template <int NSW>
__global__ void dp_pg_k(Ints I, const uint64_t* strings, int64_t ns,
                        double* pg) {
  __shared__ uint8_t lists[8][256];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = I.n, n2 = n * n;
  uint8_t* occ = lists[wid];
  uint8_t* vir = occ + 128;
  for(int64_t st = int64_t(blockIdx.x) * 8 + wid; st < ns;
      st += int64_t(gridDim.x) * 8) {
    const Spin<NSW> sp = ld_spin<NSW>(strings, st);
    const int no = sp_popc(sp), nv = n - no;
    __syncwarp();
    spin_lists<NSW>(sp, n, lane, occ, vir);
    __syncwarp();
    double* out = pg + st * no * nv;
    for(int u = lane; u < no * nv; u += 32) {
      const int v = occ[u / nv], o = vir[u % nv];
      double h = __ldg(I.T + v + o * n);
      const double* Gov = I.G_red + v * n + o * n2;
      for(int k = 0; k < no; ++k) h += __ldg(Gov + occ[k]);
      out[u] = h;
    }
  }
}

__global__ void dp_rowcount_k(const int32_t* na, const int64_t* l2cnt,
                              const int64_t* l4cnt, int64_t r0, int64_t nrows,
                              int64_t UB, int64_t* cnt) {
  for(int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nrows;
      i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t A = (r0 + i) / UB, B = (r0 + i) % UB;
    cnt[i] = int64_t(na[3 * A]) * l4cnt[B] + int64_t(na[3 * A + 1]) * l2cnt[B] +
             int64_t(na[3 * A + 2]);
  }
}

// Diagonal matrix elements of a determinant list (matrix_element_diag).
template <int NBITS>
__global__ void hdiag_k(Ints I, const uint64_t* dets, size_t n, double* out) {
  using D = DetTraits<NBITS>;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    const uint64_t* d = dets + i * D::NW;
    out[i] = me_diag(I, D::alpha(d), D::beta(d));
  }
}

template <typename VT>
__device__ __forceinline__ VT store_val(double h, bool is_diag);
template <>
__device__ __forceinline__ double store_val<double>(double h, bool) {
  return h;
}
template <>
__device__ __forceinline__ float store_val<float>(double h, bool is_diag) {
  return is_diag ? 0.0f : float(h);
}

// Direct-product fill. A CTA of DP_WARPS warps takes DP_WARPS rows that
// share one beta string B (rows (A..A+DP_WARPS-1, B)); the beta lists L2(B), L4(B)
// and the signed values of L4's beta doubles are staged once in shared
// memory.
// Each warp first evaluates all Slater-Condon singles of its bra into a
// shared table F[spin][v*n + o] (per-string partial sums plus the other-spin
// terms, reference summation order), then emits the row: entries are produced in ascending column order
// as the concatenation over connected alpha strings A' of the beta lists,
// two 32-entry rounds in flight, threshold compaction by ballot and
// streaming stores (the output must not evict the integrals from L2).
constexpr int DP_WARPS = 12;
// resident CTAs per SM: 24 warps of 80 registers (measured on the
// CAS(12e,12o) fill: 24 warps at 80 registers beat 32 at 64 by 7 %; of the
// 24-warp shapes 12 x 2 is ~1.5 % ahead of 8 x 3 and 6 x 4, since 12 rows
// share each staged beta list)
constexpr int DP_CTAS = 2;
constexpr int DP_THREADS = 32 * DP_WARPS;

struct DPShared {
  int n;
  int64_t l2max, l4max;
  size_t f_off, l2_off, l4_off, l4v_off, occ_off, bytes;
};

__host__ __device__ inline DPShared dp_shared_layout(int n, int64_t l2max,
                                                     int64_t l4max) {
  DPShared L;
  L.n = n;
  L.l2max = l2max;
  L.l4max = l4max;
  size_t o = 0;
  L.f_off = o;
  o += size_t(DP_WARPS) * 2 * n * n * 8;
  L.l2_off = o;
  o += size_t(l2max) * 8;
  L.l4_off = o;
  o += size_t(l4max) * 8;
  L.l4v_off = o;
  o += size_t(l4max) * 8;
  L.occ_off = o;
  o += size_t(DP_WARPS) * 4 * 128;  // occ/vir lists, both spins
  L.bytes = (o + 15) & ~size_t(15);
  return L;
}

// Packed list words of the fill (y of a uint2 whose x is the partner
// string index): bits 0..27 an integral offset, bits 29..30 the excitation
// class (0 none, 1 single, 2 double), bit 31 the fermionic sign.
//   alpha list:  single -> pair index a = v1 + o1 n (row a of VT) in bits
//                0..13, singles-table index v1 n + o1 in bits 14..27
//                double -> G offset of (v1,o1,v2,o2)
//   beta L2:     single -> pair index b = v1 + o1 n (column b of VT)
//   beta L4:     single -> singles-table index n^2 + v1 n + o1
//                double -> G offset
__device__ __forceinline__ uint32_t dp_encode(uint32_t e, int p, int n,
                                              int which) {
  const uint32_t n2 = uint32_t(n) * n;
  const uint32_t sg = (e >> 28) & 1u;
  uint32_t off = 0, cls = 0;
  const uint32_t o1 = ex_o1(e), v1 = ex_v1(e), o2 = ex_o2(e), v2 = ex_v2(e);
  if(p == 2) {
    cls = 1;
    if(which == 0)  // pair index (row of VT) | singles-table index << 14
      off = (v1 + o1 * n) | ((v1 * n + o1) << 14);
    else if(which == 1)
      off = v1 + o1 * n;  // pair index: column of VT
    else
      off = n2 + v1 * n + o1;
  } else if(p == 4) {
    cls = 2;
    off = v1 + n * (o1 + n * (v2 + n * o2));
  }
  return off | (cls << 29) | (sg << 31);
}

// The lists of dp_conn_count_k, encoded: for every string the strings within
// 4 (ascending; encoding `which`, and the signed G value of the doubles, 0
// for the others) and, when col2 is given, those within 2 (encoding 1). The
// excitation is seen from bra = the string. Warp per string.
template <int NSW>
__global__ void dp_conn_fill_k(const uint64_t* strs, size_t ns, int n,
                               int which, const double* G, const int64_t* off4,
                               int32_t* col4, uint32_t* info4, double* val4,
                               const int64_t* off2, int32_t* col2,
                               uint32_t* info2) {
  const int lane = threadIdx.x & 31;
  const size_t nwarp = size_t(gridDim.x) * (blockDim.x >> 5);
  for(size_t l = size_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      l < ns; l += nwarp) {
    const Spin<NSW> L = ld_spin<NSW>(strs, l);
    int64_t p4 = off4[l], p2 = col2 ? off2[l] : 0;
    for(size_t r0 = 0; r0 < ns; r0 += 32) {
      const size_t r = r0 + lane;
      Spin<NSW> R = sp_zero<NSW>();
      int p = 99;
      if(r < ns) {
        R = ld_spin<NSW>(strs, r);
        p = sp_popc(L ^ R);
      }
      const unsigned m4 = __ballot_sync(0xffffffffu, p <= 4);
      if(!m4) continue;
      const unsigned m2 = __ballot_sync(0xffffffffu, p <= 2);
      if(p <= 4) {
        uint32_t e = 0;
        if(p == 2)
          e = single_ex(L, R);
        else if(p == 4)
          e = double_ex(L, R);
        const int64_t x = p4 + __popc(m4 & lanemask_lt());
        const uint32_t w = dp_encode(e, p, n, which);
        double v = 0.0;
        if(p == 4) {
          v = __ldg(G + (w & 0x0FFFFFFFu));
          if(w >> 31) v = -v;
        }
        col4[x] = int32_t(r);
        info4[x] = w;
        val4[x] = v;
        if(col2 && p <= 2) {
          const int64_t y = p2 + __popc(m2 & lanemask_lt());
          col2[y] = int32_t(r);
          info2[y] = dp_encode(e, p, n, 1);
        }
      }
      p4 += __popc(m4);
      p2 += __popc(m2);
    }
  }
}

// VT[a n^2 + b] = V[a + b n^2] for pair indices a, b < n^2
__global__ void v_pair_transpose_k(const double* V, double* VT, int n) {
  const size_t n2 = size_t(n) * n, n4 = n2 * n2;
  for(size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < n4;
      x += size_t(gridDim.x) * blockDim.x)
    VT[(x % n2) * n2 + x / n2] = V[x];
}

const double* ham_vt(macis_b200_ham* h) {
  if(!h->VT) {
    const int n = h->norb;
    const size_t n4 = size_t(n) * n * n * n;
    MB_CUDA(dev_malloc(&h->VT, n4 * 8));
    v_pair_transpose_k<<<grid_for(n4, 256, 8 * num_sms()), 256, 0, h->stream>>>(
        h->V, h->VT, n), note_launch();
    MB_CUDA(cudaGetLastError());
  }
  return h->VT;
}

__device__ __forceinline__ double sgnd(uint32_t w, double v) {
  return (w >> 31) ? -v : v;  // == sign * v for sign in {+1, -1}
}

template <int NBITS, typename CI, typename VT>
__global__ void __launch_bounds__(DP_THREADS, DP_CTAS)
    dp_fill_k(Ints I, const double* __restrict__ Vt, DPData d, DPShared L,
              const double* __restrict__ hdiag,
              const int64_t* __restrict__ rowptr, CI* __restrict__ colind,
              VT* __restrict__ nzval, double* __restrict__ diag,
              int64_t* __restrict__ rowcnt, double thresh, int64_t r0,
              int64_t nrows, unsigned long long* __restrict__ ndropped) {
  constexpr int NSW = DetTraits<NBITS>::NSW;
  extern __shared__ __align__(16) unsigned char dsm[];
  // alpha-single segments of the current chunk: (row position, column
  // base, VT row offset, sign bit) and the alpha-single value
  __shared__ int4 seg_d[DP_WARPS][32];
  __shared__ double seg_single[DP_WARPS][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n = L.n;
  const int n2 = n * n;
  double* F = reinterpret_cast<double*>(dsm + L.f_off) + size_t(wid) * 2 * n2;
  const uint2* sl2 = reinterpret_cast<const uint2*>(dsm + L.l2_off);
  const uint2* sl4 = reinterpret_cast<const uint2*>(dsm + L.l4_off);
  const double* sl4v = reinterpret_cast<const double*>(dsm + L.l4v_off);
  uint8_t* occl = dsm + L.occ_off + size_t(wid) * 512;  // occ[2][128]
  uint8_t* virl = occl + 256;                           // vir[2][128]
  const double* __restrict__ gVT = Vt;
  const int32_t UB = int32_t(d.UB);
  const int64_t A_lo = r0 / d.UB, A_hi = (r0 + nrows - 1) / d.UB;
  const int64_t nachunk = (A_hi - A_lo + DP_WARPS) / DP_WARPS;
  const int64_t nitems = nachunk * d.UB;
  for(int64_t item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int32_t B = int32_t(item % d.UB);
    const int64_t ac = item / d.UB;
    const int64_t l2b = d.l2off[B], l4b = d.l4off[B];
    const int32_t n2l = int32_t(d.l2off[B + 1] - l2b);
    const int32_t n4l = int32_t(d.l4off[B + 1] - l4b);
    __syncthreads();  // previous item's lists are no longer read
    uint2* wl2 = reinterpret_cast<uint2*>(dsm + L.l2_off);
    uint2* wl4 = reinterpret_cast<uint2*>(dsm + L.l4_off);
    const bool s2 = n2l <= L.l2max, s4 = n4l <= L.l4max;
    if(s2)
      for(int x = threadIdx.x; x < n2l; x += DP_THREADS)
        wl2[x] = make_uint2(uint32_t(d.l2col[l2b + x]), d.l2info[l2b + x]);
    if(s4)
      for(int x = threadIdx.x; x < n4l; x += DP_THREADS) {
        wl4[x] = make_uint2(uint32_t(d.l4col[l4b + x]), d.l4info[l4b + x]);
        reinterpret_cast<double*>(dsm + L.l4v_off)[x] = d.l4val[l4b + x];
      }
    __syncthreads();
    const int64_t A = A_lo + ac * DP_WARPS + wid;
    const int64_t grow = A * d.UB + B;
    if(A > A_hi || grow < r0 || grow >= r0 + nrows) continue;
    const int32_t row = int32_t(grow - r0);
    const Spin<NSW> sp[2] = {ld_spin<NSW>(d.ua, A), ld_spin<NSW>(d.ub, B)};
    // occupied / virtual lists, one orbital per lane
    int no[2], nv[2];
#pragma unroll
    for(int S = 0; S < 2; ++S) {
      no[S] = sp_popc(sp[S]);
      nv[S] = n - no[S];
      spin_lists<NSW>(sp[S], n, lane, occl + S * 128, virl + S * 128);
    }
    __syncwarp();
    // singles table: F[spin][v*n + o] = (T(v,o) + sum_{p in occ_same}
    // G_red(p,v,o)) + sum_{p in occ_other} V_red(p,v,o)
    // (matrix_elements.hpp:86-104 without the sign), v occupied and o empty
    // in the bra. The bracket is the per-string partial sum of dp_pg_k.
    {
      const int nsa = no[0] * nv[0], nsb = no[1] * nv[1];
      const double* __restrict__ pga = d.pga + A * nsa;
      const double* __restrict__ pgb = d.pgb + int64_t(B) * nsb;
      // i = u / nv by a float product: (u + 0.5) / nv stays >= 0.5 / nv
      // away from an integer, far above the rounding error for u < 2^14
      const float rva = 1.0f / float(nv[0] > 0 ? nv[0] : 1);
      const float rvb = 1.0f / float(nv[1] > 0 ? nv[1] : 1);
      for(int t = lane; t < nsa + nsb; t += 32) {
        // selects instead of no[S] / nv[S]: a dynamic index would put the
        // arrays in local memory
        const int S = t < nsa ? 0 : 1;
        const int u = S ? t - nsa : t;
        const int nvS = S ? nv[1] : nv[0];
        const int noO = S ? no[0] : no[1];
        const int i = int((float(u) + 0.5f) * (S ? rvb : rva));
        const int v = occl[S * 128 + i], o = virl[S * 128 + (u - i * nvS)];
        double h = __ldg((S ? pgb : pga) + u);
        const double* Vov = I.V_red + v * n + o * n2;
        const uint8_t* po = occl + (1 - S) * 128;
#pragma unroll 4
        for(int k = 0; k < noO; ++k) h += __ldg(Vov + po[k]);
        F[S * n2 + v * n + o] = h;
      }
    }
    __syncwarp();
    const double hd = hdiag[row];
    const int64_t out0 = rowptr[row];
    CI* __restrict__ rc = colind + out0;
    VT* __restrict__ rv = nzval + out0;
    int32_t pos = 0, dropped = 0;  // dropped: this lane's count
    uint2 el = make_uint2(0u, 0u);  // this lane's entry of the beta L2 list
    if(lane < n2l)
      el = s2 ? sl2[lane]
              : make_uint2(uint32_t(__ldg(d.l2col + l2b + lane)),
                           __ldg(d.l2info + l2b + lane));
    // beta L2 entries 32..63 (n2l <= 64): each lane also holds entry lane + 32
    // and emits it in the same segment iteration as entry lane
    const bool fold = n2l > 32 && n2l <= 64;
    uint2 el2 = make_uint2(0u, 0u);
    const bool has2 = fold && lane + 32 < n2l;
    if(has2)
      el2 = s2 ? sl2[lane + 32]
               : make_uint2(uint32_t(__ldg(d.l2col + l2b + lane + 32)),
                            __ldg(d.l2info + l2b + lane + 32));
    using CS = typename std::conditional<sizeof(CI) == 4, int, long long>::type;
    CS* __restrict__ rcs = reinterpret_cast<CS*>(rc);
    // entries whose column differs from the row (every phase but the
    // same-alpha segment): no diagonal test
    auto put = [&](bool act, int32_t p, int32_t col, double h) {
      if(act) {
        const bool keep = fabs(h) > thresh;
        dropped += !keep;
        __stcs(rcs + p, CS(keep ? col : -1));
        __stcs(rv + p, store_val<VT>(h, false));
      }
    };
    auto put_d = [&](bool act, int32_t p, int32_t col, double h) {
      if(act) {
        const bool keep = fabs(h) > thresh;
        dropped += !keep;
        const bool isd = keep && col == row;
        __stcs(rcs + p, CS(keep ? col : -1));
        __stcs(rv + p, store_val<VT>(h, isd));
        if(isd) diag[row] = h;
      }
    };
    const int64_t c1 = d.aoff[A + 1];
    // the next chunk of the alpha list is loaded while this one is emitted
    int32_t nx_col = 0;
    uint32_t nx_ai = 0;
    double nx_val = 0.0;
    {
      const int64_t j = d.aoff[A] + lane;
      if(j < c1) {
        nx_col = __ldg(d.acol + j);
        nx_ai = __ldg(d.ainfo + j);
        nx_val = __ldg(d.aval + j);
      }
    }
    for(int64_t c = d.aoff[A]; c < c1; c += 32) {
      const int64_t j = c + lane;
      int32_t colA = 0;
      uint32_t ai = 0;
      double aval = 0.0;
      int cls = 3, cnt = 0;
      if(j < c1) {
        colA = nx_col * UB;
        ai = nx_ai;
        aval = nx_val;
        cls = int((ai >> 29) & 3u);
        cnt = cls == 0 ? n4l : cls == 1 ? n2l : 1;
      }
      if(j + 32 < c1) {
        nx_col = __ldg(d.acol + j + 32);
        nx_ai = __ldg(d.ainfo + j + 32);
        nx_val = __ldg(d.aval + j + 32);
      }
      const int incl = warp_incl_scan(cnt);
      const int32_t spos = pos + incl - cnt;
      pos += __shfl_sync(0xffffffffu, incl, 31);
      // (1) alpha doubles: beta unchanged, one entry each
      {
        put(cls == 2, spos, colA + B, aval);
      }
      // (2) the same-alpha segment: every beta string within two excitations
      unsigned m0 = __ballot_sync(0xffffffffu, cls == 0);
      while(m0) {
        const int L0 = __ffs(m0) - 1;
        m0 &= m0 - 1;
        const int32_t sp0 = __shfl_sync(0xffffffffu, spos, L0);
        const int32_t cA = __shfl_sync(0xffffffffu, colA, L0);
        for(int32_t t = lane; t - lane < n4l; t += 32) {
          const bool act = t < n4l;
          double h = 0;
          int32_t col = 0;
          if(act) {
            const uint2 ent = s4 ? sl4[t]
                                 : make_uint2(uint32_t(__ldg(d.l4col + l4b + t)),
                                              __ldg(d.l4info + l4b + t));
            const uint32_t cb = (ent.y >> 29) & 3u, off = ent.y & 0x0FFFFFFFu;
            // singles from this row's table (shared; offsets < 2 n^2),
            // doubles already signed
            const double vf = F[off < uint32_t(2 * n2) ? off : 0u];
            const double vd = s4 ? sl4v[t] : __ldg(d.l4val + l4b + t);
            col = cA + int32_t(ent.x);
            h = cb == 0 ? hd : cb == 1 ? sgnd(ent.y, vf) : vd;
          }
          put_d(act, sp0 + t, col, h);
        }
      }
      // (3) alpha singles: one segment of n2l entries (beta within one
      // excitation) per connected alpha string. Each lane keeps its beta
      // list entry for the row; the warp sweeps the segments.
      const unsigned m2 = __ballot_sync(0xffffffffu, cls == 1);
      if(cls == 1) {
        const int rk = __popc(m2 & lanemask_lt());
        const uint32_t pa_ = ai & 0x3FFFu;  // v1 + o1 n
        seg_d[wid][rk] = make_int4(spos, colA, int(pa_ * uint32_t(n2)),
                                   int(ai & 0x80000000u));
        seg_single[wid][rk] = sgnd(ai, F[(ai >> 14) & 0x3FFFu]);
      }
      __syncwarp();
      const int k2 = __popc(m2);
      if(fold) {
        const bool bsame = ((el.y >> 29) & 3u) == 0;
        const uint32_t boff = el.y & 0x0FFFFFFFu, bsg = el.y & 0x80000000u;
        const bool bsame2 = ((el2.y >> 29) & 3u) == 0;
        const uint32_t boff2 = el2.y & 0x0FFFFFFFu, bsg2 = el2.y & 0x80000000u;
        CS* __restrict__ rcl = rcs + lane;
        VT* __restrict__ rvl = rv + lane;
        for(int q = 0; q < k2; ++q) {
          const int4 sd = seg_d[wid][q];
          const double sgl = seg_single[wid][q];
          const double v = __ldg(gVT + uint32_t(sd.z + int(boff)));
          const double v2 = has2 ? __ldg(gVT + uint32_t(sd.z + int(boff2))) : 0.0;
          const double hv = __hiloint2double(
              __double2hiint(v) ^ (sd.w ^ int(bsg)), __double2loint(v));
          const double h = bsame ? sgl : hv;
          const bool keep = fabs(h) > thresh;
          dropped += keep ? 0 : 1;
          const uint32_t p = uint32_t(sd.x);
          __stcs(rcl + p, CS(keep ? sd.y + int32_t(el.x) : -1));
          __stcs(rvl + p, store_val<VT>(h, false));
          if(has2) {
            const double hv2 = __hiloint2double(
                __double2hiint(v2) ^ (sd.w ^ int(bsg2)), __double2loint(v2));
            const double h2 = bsame2 ? sgl : hv2;
            const bool keep2 = fabs(h2) > thresh;
            dropped += keep2 ? 0 : 1;
            __stcs(rcl + p + 32, CS(keep2 ? sd.y + int32_t(el2.x) : -1));
            __stcs(rvl + p + 32, store_val<VT>(h2, false));
          }
        }
      } else if(lane < n2l) {
        // branch-free body: the same-beta entry (offset 0) also loads from
        // its VT row and then selects the alpha-single value
        const bool bsame = ((el.y >> 29) & 3u) == 0;
        const uint32_t boff = el.y & 0x0FFFFFFFu, bsg = el.y & 0x80000000u;
        const int32_t elx = int32_t(el.x);
        CS* __restrict__ rcl = rcs + lane;
        VT* __restrict__ rvl = rv + lane;
#pragma unroll 2
        for(int q = 0; q < k2; ++q) {
          const int4 sd = seg_d[wid][q];
          const double sgl = seg_single[wid][q];
          const double v = __ldg(gVT + uint32_t(sd.z + int(boff)));
          // sign of the element: one XOR on the high word
          const double hv = __hiloint2double(
              __double2hiint(v) ^ (sd.w ^ int(bsg)), __double2loint(v));
          const double h = bsame ? sgl : hv;
          const bool keep = fabs(h) > thresh;
          dropped += keep ? 0 : 1;
          const uint32_t p = uint32_t(sd.x);
          __stcs(rcl + p, CS(keep ? sd.y + elx : -1));
          __stcs(rvl + p, store_val<VT>(h, false));
        }
      }
      if(n2l > 64) {  // list entries 32.. of every segment, flattened
        const int32_t w2 = n2l - 32;
        const int32_t tot2 = k2 * w2;
        const float invw = 1.0f / float(w2);
        for(int32_t e = lane; e < tot2; e += 32) {
          int sg = int(float(e) * invw);
          if(sg * w2 > e) --sg;
          if((sg + 1) * w2 <= e) ++sg;
          const int32_t t = 32 + e - sg * w2;
          const uint2 ent = s2 ? sl2[t]
                               : make_uint2(uint32_t(__ldg(d.l2col + l2b + t)),
                                            __ldg(d.l2info + l2b + t));
          const int4 sd = seg_d[wid][sg];
          const double sgl = seg_single[wid][sg];
          const double v = __ldg(gVT + uint32_t(sd.z + int(ent.y & 0x0FFFFFFFu)));
          const double hv = __hiloint2double(
              __double2hiint(v) ^ (sd.w ^ int(ent.y & 0x80000000u)),
              __double2loint(v));
          const double h = ((ent.y >> 29) & 3u) == 0 ? sgl : hv;
          const bool keep = fabs(h) > thresh;
          dropped += keep ? 0 : 1;
          const uint32_t p = uint32_t(sd.x + t);
          __stcs(rcs + p, CS(keep ? sd.y + int32_t(ent.x) : -1));
          __stcs(rv + p, store_val<VT>(h, false));
        }
      }
      __syncwarp();
    }
#pragma unroll
    for(int o = 16; o > 0; o >>= 1)
      dropped += __shfl_xor_sync(0xffffffffu, dropped, o);
    if(lane == 0) {
      rowcnt[row] = int64_t(pos) - dropped;
      if(dropped) atomicAdd(ndropped, (unsigned long long)dropped);
    }
  }
}

__global__ void dp_totals_k(const int64_t* aoff, size_t ua, const int64_t* l2off,
                            const int64_t* l4off, size_t ub,
                            const int64_t* rowptr, size_t nbra, DPTotals* t) {
  t->na = aoff[ua];
  t->n2 = l2off[ub];
  t->n4 = l4off[ub];
  t->nnz = rowptr[nbra];
}

// Removes the entries marked with column -1 while packing rows to their
// final offsets (builds with dropped elements).
template <typename CI, typename VT>
__global__ void compact_marked_k(const int64_t* oldptr, const int64_t* newptr,
                                 size_t m, const CI* ci, const VT* nz, CI* ci2,
                                 VT* nz2) {
  const int lane = threadIdx.x & 31;
  const size_t nwarp = size_t(gridDim.x) * (blockDim.x >> 5);
  for(size_t r = size_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      r < m; r += nwarp) {
    const int64_t s = oldptr[r], e = oldptr[r + 1];
    int64_t o = newptr[r];
    for(int64_t b = s; b < e; b += 32) {
      const int64_t i = b + lane;
      CI c = 0;
      VT v = 0;
      bool keep = false;
      if(i < e) {
        c = ci[i];
        v = nz[i];
        keep = c >= 0;
      }
      const unsigned msk = __ballot_sync(0xffffffffu, keep);
      if(keep) {
        const int64_t p = o + __popc(msk & lanemask_lt());
        ci2[p] = c;
        nz2[p] = v;
      }
      o += __popc(msk);
    }
  }
}

// -------------------------------------------------------- general path
template <int NBITS>
struct GenKey {
  // sort key with the alpha string most significant
  static constexpr int KW = NBITS == 64 ? 1 : (NBITS == 128 ? 2 : 4);
};

template <int NBITS>
__global__ void gen_keys_k(const uint64_t* dets, size_t n, uint64_t* keys,
                           uint32_t* idx) {
  using D = DetTraits<NBITS>;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    const uint64_t* d = dets + i * D::NW;
    const auto a = D::alpha(d), b = D::beta(d);
    if constexpr(NBITS == 64) {
      keys[i] = (a.w[0] << 32) | b.w[0];
    } else if constexpr(NBITS == 128) {
      keys[2 * i] = b.w[0];
      keys[2 * i + 1] = a.w[0];
    } else {
      keys[4 * i] = b.w[0];
      keys[4 * i + 1] = b.w[1];
      keys[4 * i + 2] = a.w[0];
      keys[4 * i + 3] = a.w[1];
    }
    idx[i] = uint32_t(i);
  }
}

template <int NBITS>
__device__ __forceinline__ void key_spins(const uint64_t* keys, size_t i,
                                          Spin<DetTraits<NBITS>::NSW>& a,
                                          Spin<DetTraits<NBITS>::NSW>& b) {
  if constexpr(NBITS == 64) {
    a.w[0] = keys[i] >> 32;
    b.w[0] = keys[i] & 0xffffffffull;
  } else if constexpr(NBITS == 128) {
    b.w[0] = keys[2 * i];
    a.w[0] = keys[2 * i + 1];
  } else {
    b.w[0] = keys[4 * i];
    b.w[1] = keys[4 * i + 1];
    a.w[0] = keys[4 * i + 2];
    a.w[1] = keys[4 * i + 3];
  }
}

// What the host reads back of a sorted list.
struct GenInfo {
  uint32_t groups;  // alpha groups
  uint32_t mixed;   // the nonzero determinants' electron counts differ
  uint32_t counts;  // of the last determinant: alpha + 256 beta
};

// flags[i] = 1 at the first nonzero key of each alpha group; zero keys
// (zero determinants, which the reference skips, first in the order) get 0.
// Electron counts are compared with the last key's.
template <int NBITS>
__global__ void gen_group_flags_k(const uint64_t* keys, size_t n,
                                  uint32_t* flags, GenInfo* info) {
  constexpr int NSW = DetTraits<NBITS>::NSW;
  Spin<NSW> la, lb;
  key_spins<NBITS>(keys, n - 1, la, lb);
  const int na = sp_popc(la), nb = sp_popc(lb);
  if(blockIdx.x == 0 && threadIdx.x == 0) info->counts = uint32_t(na + 256 * nb);
  bool mixed = false;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    Spin<NSW> a, b;
    key_spins<NBITS>(keys, i, a, b);
    const int ca = sp_popc(a), cb = sp_popc(b);
    uint32_t f = 0;
    if(ca + cb != 0) {
      mixed |= ca != na || cb != nb;
      f = 1;
      if(i > 0) {
        Spin<NSW> pa, pb;
        key_spins<NBITS>(keys, i - 1, pa, pb);
        const bool pzero = sp_popc(pa) + sp_popc(pb) == 0;
        f = (pzero || !(pa == a)) ? 1 : 0;
      }
    }
    flags[i] = f;
  }
  if(mixed) info->mixed = 1;
}

// Group tables: goff[g] (first sorted position), galpha[g]; sorted strings;
// per original index its group (or -1 for zero determinants).
template <int NBITS>
__global__ void gen_groups_k(const uint64_t* keys, const uint32_t* idx,
                             const uint32_t* flags, const uint32_t* gid_excl,
                             size_t n, int64_t* goff, uint64_t* galpha,
                             uint64_t* salpha, uint64_t* sbeta,
                             int32_t* rowgroup) {
  constexpr int NSW = DetTraits<NBITS>::NSW;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    Spin<NSW> a, b;
    key_spins<NBITS>(keys, i, a, b);
    st_spin<NSW>(salpha, i, a);
    st_spin<NSW>(sbeta, i, b);
    const bool zero = sp_popc(a) + sp_popc(b) == 0;
    const uint32_t g = gid_excl[i] + flags[i] - 1;
    if(flags[i]) {
      goff[g] = int64_t(i);
      st_spin<NSW>(galpha, g, a);
    }
    if(rowgroup) rowgroup[idx[i]] = zero ? -1 : int32_t(g);
  }
}

__global__ void gen_group_end_k(int64_t* goff, uint32_t ng, int64_t end) {
  goff[ng] = end;
}

// ---- beta-major view of the kets: a row's alpha-double connections are the
// kets with its own beta whose alpha is 4 bits away, found by walking the
// kets of that beta when there are fewer of them than alpha-double groups.

// Sort keys with the beta string most significant.
template <int NBITS>
__global__ void gen_bkeys_k(const uint64_t* dets, size_t n, uint64_t* keys,
                            uint32_t* idx) {
  using D = DetTraits<NBITS>;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    const uint64_t* d = dets + i * D::NW;
    const auto a = D::alpha(d), b = D::beta(d);
    if constexpr(NBITS == 64) {
      keys[i] = (b.w[0] << 32) | a.w[0];
    } else if constexpr(NBITS == 128) {
      keys[2 * i] = a.w[0];
      keys[2 * i + 1] = b.w[0];
    } else {
      keys[4 * i] = a.w[0];
      keys[4 * i + 1] = a.w[1];
      keys[4 * i + 2] = b.w[0];
      keys[4 * i + 3] = b.w[1];
    }
    idx[i] = uint32_t(i);
  }
}

template <int NBITS>
__device__ __forceinline__ void bkey_spins(const uint64_t* keys, size_t i,
                                           Spin<DetTraits<NBITS>::NSW>& a,
                                           Spin<DetTraits<NBITS>::NSW>& b) {
  if constexpr(NBITS == 64) {
    b.w[0] = keys[i] >> 32;
    a.w[0] = keys[i] & 0xffffffffull;
  } else if constexpr(NBITS == 128) {
    a.w[0] = keys[2 * i];
    b.w[0] = keys[2 * i + 1];
  } else {
    a.w[0] = keys[4 * i];
    a.w[1] = keys[4 * i + 1];
    b.w[0] = keys[4 * i + 2];
    b.w[1] = keys[4 * i + 3];
  }
}

// amaj[idx[m]] = m: original ket index -> alpha-major sorted position.
__global__ void gen_invert_k(const uint32_t* idx, size_t n, uint32_t* amaj) {
  for(size_t m = size_t(blockIdx.x) * blockDim.x + threadIdx.x; m < n;
      m += size_t(gridDim.x) * blockDim.x)
    amaj[idx[m]] = uint32_t(m);
}

// mgroup[m] = alpha group of sorted position m (-1 stays for zero dets).
__global__ void gen_mgroup_k(const int64_t* goff, uint32_t ng,
                             int32_t* mgroup) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = int64_t(gridDim.x) * (blockDim.x >> 5);
  for(int64_t gi = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      gi < int64_t(ng); gi += nw)
    for(int64_t m = goff[gi] + lane; m < goff[gi + 1]; m += 32)
      mgroup[m] = int32_t(gi);
}

// Per beta-major position: its alpha string and alpha-major position; flags
// at the first position of every distinct beta.
template <int NBITS>
__global__ void gen_bmajor_k(const uint64_t* bkeys, const uint32_t* bidx,
                             size_t n, const uint32_t* amaj, uint64_t* bm_alpha,
                             uint32_t* bm_m, uint32_t* bflags) {
  constexpr int NSW = DetTraits<NBITS>::NSW;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    Spin<NSW> a, b;
    bkey_spins<NBITS>(bkeys, i, a, b);
    st_spin<NSW>(bm_alpha, i, a);
    bm_m[i] = amaj[bidx[i]];
    uint32_t f = 1;
    if(i > 0) {
      Spin<NSW> pa, pb;
      bkey_spins<NBITS>(bkeys, i - 1, pa, pb);
      f = (pb == b) ? 0u : 1u;
    }
    bflags[i] = f;
  }
}

// Distinct betas (sorted) and the start of each in beta-major order.
template <int NBITS>
__global__ void gen_bgroups_k(const uint64_t* bkeys, const uint32_t* bflags,
                              const uint32_t* bgx, size_t n, int64_t* bgoff,
                              uint64_t* bgbeta) {
  constexpr int NSW = DetTraits<NBITS>::NSW;
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x) {
    if(!bflags[i]) continue;
    Spin<NSW> a, b;
    bkey_spins<NBITS>(bkeys, i, a, b);
    bgoff[bgx[i]] = int64_t(i);
    st_spin<NSW>(bgbeta, bgx[i], b);
  }
}

// Alpha connectivity between bra groups and ket groups: (ket group, pa).
// Count pass (col == nullptr): cnt[l] = all connected groups, cnt4[l] =
// those at pa == 4. Fill pass: the pa <= 3 entries of bra group l first, in
// ket-group order, then its pa == 4 entries from off[l] + cnt[l] - cnt4[l].
template <int NSW>
__global__ void gen_aconn_k(const uint64_t* balpha, size_t nb,
                            const uint64_t* kalpha, size_t nk,
                            const int64_t* off, int64_t* cnt, int64_t* cnt4,
                            int32_t* col, uint8_t* pa_out) {
  const int lane = threadIdx.x & 31;
  const size_t nwarp = size_t(gridDim.x) * (blockDim.x >> 5);
  for(size_t l = size_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      l < nb; l += nwarp) {
    const Spin<NSW> L = ld_spin<NSW>(balpha, l);
    int64_t c = 0, c4 = 0;
    const int64_t base = off ? off[l] : 0;
    const int64_t base4 = col ? base + cnt[l] - cnt4[l] : 0;
    for(size_t r0 = 0; r0 < nk; r0 += 32) {
      const size_t r = r0 + lane;
      int p = 99;
      if(r < nk) p = sp_popc(L ^ ld_spin<NSW>(kalpha, r));
      const bool hit = p <= 3, hit4 = p == 4;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      const unsigned m4 = __ballot_sync(0xffffffffu, hit4);
      if(col && (hit || hit4)) {
        const int64_t pos = hit ? base + c + __popc(m & lanemask_lt())
                                : base4 + c4 + __popc(m4 & lanemask_lt());
        col[pos] = int32_t(r);
        pa_out[pos] = uint8_t(p);
      }
      c += __popc(m);
      c4 += __popc(m4);
    }
    if(!col && lane == 0) {
      cnt[l] = c + c4;
      cnt4[l] = c4;
    }
  }
}

struct GenData {
  const int32_t* rowgroup;  // bra row -> bra group (-1: zero det)
  const int64_t* aoff;      // bra group -> aconn range
  const int32_t* acol;      // ket group
  const uint8_t* apa;
  const int64_t* goff;      // ket group -> sorted range
  const uint64_t* salpha;   // sorted ket alphas
  const uint64_t* sbeta;    // sorted ket betas
  const uint32_t* sidx;     // sorted ket -> original index
  // beta hash tables of the large ket groups (gen_hsize_k / gen_hinsert_k)
  const int64_t* hoff;      // ket group -> table range (empty: no table)
  const int32_t* htab;      // sorted position - group start, -1 empty
  const int32_t* gbpop;     // ket group -> common beta popcount (-1: none)
  int n;                    // orbitals
  const int64_t* a4cnt;     // bra group -> its pa == 4 entries (at the end)
  // beta-major view of the kets (gen_bmajor_k / gen_bgroups_k)
  const uint64_t* bgbeta;   // distinct ket betas, sorted
  const int64_t* bgoff;     // their ranges in beta-major order
  int64_t nbgb;             // number of distinct ket betas
  const uint64_t* bm_alpha; // per beta-major position: alpha string
  const uint32_t* bm_m;     // per beta-major position: alpha-major position
  const int32_t* mgroup;    // alpha-major position -> ket group (-1: none)
  bool mixed;               // electron counts differ in the lists
};

// Ket groups of at least GEN_HASH_MIN members get a hash table of their
// betas so that a bra row connected to them by an alpha single excitation
// can look up its own beta single excitations instead of testing every
// member (a few hundred lookups against up to ~1e5 member tests for the
// large groups of ASCI spaces).
constexpr int64_t GEN_HASH_MIN = 256;

template <int NSW>
__device__ __forceinline__ uint64_t spin_hash(const Spin<NSW>& a) {
  uint64_t x = 0;
#pragma unroll
  for(int w = 0; w < NSW; ++w) x = (x ^ a.w[w]) * 0x9E3779B97F4A7C15ull;
  x ^= x >> 29;
  x *= 0xBF58476D1CE4E5B9ull;
  return x ^ (x >> 32);
}

// Per ket group (one warp each): the table size (a power of two >= 2 G for
// groups of G >= GEN_HASH_MIN members whose betas share one popcount, else
// 0) and that popcount (-1 when the group has no table).
template <int NSW>
__global__ void gen_hsize_k(const int64_t* goff, uint32_t ng,
                            const uint64_t* sbeta, int64_t* hsz,
                            int32_t* gbpop) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = int64_t(gridDim.x) * (blockDim.x >> 5);
  for(int64_t gi = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      gi < int64_t(ng); gi += nw) {
    const int64_t m0 = goff[gi], m1 = goff[gi + 1];
    int64_t sz = 0;
    int pc = -1;
    if(m1 - m0 >= GEN_HASH_MIN) {
      pc = sp_popc(ld_spin<NSW>(sbeta, m0));
      bool same = true;
      for(int64_t m = m0 + lane; m < m1; m += 32)
        same = same && sp_popc(ld_spin<NSW>(sbeta, m)) == pc;
      same = __all_sync(0xffffffffu, same);
      if(same) {
        sz = 1;
        while(sz < 2 * (m1 - m0)) sz <<= 1;
      } else {
        pc = -1;
      }
    }
    if(lane == 0) {
      hsz[gi] = sz;
      gbpop[gi] = pc;
    }
  }
}

// Inserts the first sorted position of every distinct beta of a ket group
// into its table (linear probing; the table has at least twice as many
// slots as entries, so every insertion finds a free slot). One thread per
// member: a warp per group left the largest groups (1e4 members) to one warp.
template <int NSW>
__global__ void gen_hinsert_k(const int64_t* goff, const int32_t* mgroup,
                              size_t n, const uint64_t* sbeta,
                              const int64_t* hoff, int32_t* htab) {
  for(size_t m = size_t(blockIdx.x) * blockDim.x + threadIdx.x; m < n;
      m += size_t(gridDim.x) * blockDim.x) {
    const int32_t gi = mgroup[m];
    if(gi < 0) continue;
    const int64_t h0 = hoff[gi], hs = hoff[gi + 1] - h0;
    if(hs == 0) continue;
    const uint64_t mask = uint64_t(hs) - 1;
    const int64_t m0 = goff[gi];
    const Spin<NSW> b = ld_spin<NSW>(sbeta, m);
    if(int64_t(m) > m0 && ld_spin<NSW>(sbeta, m - 1) == b) continue;  // duplicate
    uint64_t slot = spin_hash<NSW>(b) & mask;
    for(int64_t t = 0; t < hs; ++t) {
      if(atomicCAS(htab + h0 + slot, -1, int32_t(int64_t(m) - m0)) == -1) break;
      slot = (slot + 1) & mask;
    }
  }
}

// Next row of a kernel whose warps take rows from a counter: rows differ by
// orders of magnitude in work (the members of the largest alpha groups test
// 1e4 kets more than others), so a fixed assignment leaves a long tail.
__device__ __forceinline__ int64_t next_row(unsigned* ctr) {
  unsigned r = 0;
  if((threadIdx.x & 31) == 0) r = atomicAdd(ctr, 1u);
  return int64_t(__shfl_sync(0xffffffffu, r, 0));
}

// Enumerates the candidate kets of one bra row warp-synchronously; calls
// emit(active, sorted_pos, pa, pb) for chunks of <= 32.
template <int NSW, class F>
__device__ __forceinline__ void gen_enumerate(const GenData& g, int32_t rg,
                                              Spin<NSW> ba, Spin<NSW> bb,
                                              uint8_t* ov, F&& emit) {
  const int lane = threadIdx.x & 31;
  // occupied / empty orbitals of the bra beta (ov[0..128), ov[128..256)),
  // for the hash lookups of its single excitations
  const int nob = sp_popc(bb), nvb = g.n - nob;
  const int nenum = 1 + nob * nvb;  // the beta itself and its singles
  const float rnv = 1.0f / float(nvb > 0 ? nvb : 1);
  __syncwarp();
  spin_lists<NSW>(bb, g.n, lane, ov, ov + 128);
  __syncwarp();
  // the kets with beta bb (beta-major range [b0, b1))
  int b0 = 0, b1 = 0;
  {
    int lo = 0, hi = int(g.nbgb);
    while(lo < hi) {
      const int mid = (lo + hi) >> 1;
      if(sp_cmp(ld_spin<NSW>(g.bgbeta, mid), bb) < 0)
        lo = mid + 1;
      else
        hi = mid;
    }
    if(lo < int(g.nbgb) && ld_spin<NSW>(g.bgbeta, lo) == bb) {
      b0 = int(g.bgoff[lo]);
      b1 = int(g.bgoff[lo + 1]);
    }
  }
  const int64_t c1 = g.aoff[rg + 1];
  const int64_t c4 = c1 - g.a4cnt[rg];  // the pa == 4 entries start here
  // alpha doubles through the kets of beta bb when they are fewer than the
  // alpha-double groups (each of which would take a binary search)
  const bool by_beta = b1 - b0 < c1 - c4;
  const int64_t cend = by_beta ? c4 : c1;
  if(by_beta) {
    for(int p0 = b0; p0 < b1; p0 += 32) {
      const int p = p0 + lane;
      const bool act = p < b1 && sp_popc(ld_spin<NSW>(g.bm_alpha, p) ^ ba) == 4;
      int64_t m = 0;
      if(act) m = g.bm_m[p];
      emit(act && g.mgroup[m] >= 0, m, 4, 0);
    }
  }
  for(int64_t c = g.aoff[rg]; c < cend; c += 32) {
    const int64_t j = c + lane;
    const bool valid = j < cend;
    int pa = 99;
    int m0 = 0, m1 = 0;  // this lane's group
    int64_t h0 = 0, hs = 0;
    bool probe = false;
    if(valid) {
      const int32_t kg = g.acol[j];
      pa = g.apa[j];
      m0 = int(g.goff[kg]);
      m1 = int(g.goff[kg + 1]);
      if(pa == 2) {
        h0 = g.hoff[kg];
        hs = g.hoff[kg + 1] - h0;
        probe = hs > 0 && g.gbpop[kg] == nob && m1 - m0 > 8 * nenum;
      }
    }
    // alpha doubles (pa == 4): only the identical beta can connect
    int lo = 0, hi = 0;
    if(valid && pa == 4) {
      int a = m0, b = m1;
      while(a < b) {  // lower bound
        const int mid = (a + b) >> 1;
        if(sp_cmp(ld_spin<NSW>(g.sbeta, mid), bb) < 0)
          a = mid + 1;
        else
          b = mid;
      }
      lo = a;
      b = m1;
      while(a < b) {  // upper bound
        const int mid = (a + b) >> 1;
        if(sp_cmp(ld_spin<NSW>(g.sbeta, mid), bb) <= 0)
          a = mid + 1;
        else
          b = mid;
      }
      hi = a;
    }
    const int rem = hi - lo;
    const int maxrem = __reduce_max_sync(0xffffffffu, rem);
    for(int r = 0; r < maxrem; ++r) emit(r < rem, lo + r, 4, 0);
    // pa <= 3: the members of small groups, taken together
    const bool scan = valid && pa <= 3;
    const int small = scan && m1 - m0 <= 32 ? m1 - m0 : 0;
    int incl = warp_incl_scan(small);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int mbase = m0 - (incl - small);  // member e of the run is mbase + e
    for(int e0 = 0; e0 < total; e0 += 32) {
      const int e = e0 + lane;
      int L = 0;  // lanes whose members end at or before e
#pragma unroll
      for(int st = 16; st; st >>= 1)
        if(__shfl_sync(0xffffffffu, incl, L + st - 1) <= e) L += st;
      const int src = L < 32 ? L : 31;
      const int64_t m = __shfl_sync(0xffffffffu, mbase, src) + e;
      const int ppa = __shfl_sync(0xffffffffu, pa, src);
      int pb = 99;
      if(e < total) pb = sp_popc(ld_spin<NSW>(g.sbeta, m) ^ bb);
      emit(pb <= 4 - ppa, m, ppa, pb);
    }
    // the larger groups, one at a time
    unsigned big = __ballot_sync(0xffffffffu, scan && m1 - m0 > 32);
    while(big) {
      const int L = __ffs(big) - 1;
      big &= big - 1;
      const int ppa = __shfl_sync(0xffffffffu, pa, L);
      const int limit = 4 - ppa;
      const int gm0 = __shfl_sync(0xffffffffu, m0, L);
      const int gm1 = __shfl_sync(0xffffffffu, m1, L);
      if(__shfl_sync(0xffffffffu, int(probe), L)) {
        // alpha single into a large group: only betas within one
        // excitation of bb connect, and all of them have bb's popcount
        const int64_t gh0 = __shfl_sync(0xffffffffu, h0, L);
        const int64_t ghs = __shfl_sync(0xffffffffu, hs, L);
        const uint64_t mask = uint64_t(ghs) - 1;
        for(int u0 = 0; u0 < nenum; u0 += 32) {
          const int u = u0 + lane;
          int plo = 0, phi = 0;
          int pbv = 0;
          if(u < nenum) {
            Spin<NSW> q = bb;
            if(u > 0) {
              const int i = int((float(u - 1) + 0.5f) * rnv);
              const int jv = (u - 1) - i * nvb;
              q = sp_flip(sp_flip(q, ov[i]), ov[128 + jv]);
              pbv = 2;
            }
            uint64_t slot = spin_hash<NSW>(q) & mask;
            for(int64_t t = 0; t < ghs; ++t) {
              const int32_t r = g.htab[gh0 + slot];
              if(r < 0) break;
              if(ld_spin<NSW>(g.sbeta, gm0 + r) == q) {
                plo = gm0 + r;
                phi = plo + 1;
                while(phi < gm1 && ld_spin<NSW>(g.sbeta, phi) == q) ++phi;
                break;
              }
              slot = (slot + 1) & mask;
            }
          }
          const int prem = phi - plo;
          const int mr = __reduce_max_sync(0xffffffffu, prem);
          for(int r = 0; r < mr; ++r) emit(r < prem, plo + r, 2, pbv);
        }
        continue;
      }
      // four loads in flight: groups are a few hundred members, and the loop
      // waits for each load (one copy of emit, see gen_pairs)
      for(int mb = gm0; mb < gm1; mb += 128) {
        uint32_t pbs = 0;  // their four distances, a byte each
#pragma unroll
        for(int u = 0; u < 4; ++u) {
          const int m = mb + 32 * u + lane;
          const int pb = m < gm1 ? sp_popc(ld_spin<NSW>(g.sbeta, m) ^ bb) : 255;
          pbs |= uint32_t(pb) << (8 * u);
        }
#pragma unroll 1
        for(int m = mb; m < gm1 && m < mb + 128; m += 32, pbs >>= 8) {
          const int pb = int(pbs & 255u);
          emit(pb <= limit, m + lane, ppa, pb);
        }
      }
    }
  }
}

// The connected kets of a row are a few of the members that gen_enumerate
// tests (1.5 % on an n = 48 list of 1.5e5 determinants), so its chunks of 32
// hold one or two each. gen_pairs queues them and calls eval(on, m,
// is_double) with 32 at a time, doubles and the rest (singles, the diagonal,
// lists of mixed electron counts) apart: an element then costs a lane's share
// of the warp's instructions and not all of them. eval is expanded once in the
// queueing, which stands at five places of the enumeration, and once at the
// end: with a copy per kind of pair and unrolled chunk (18 in all) a warp
// waited half of its time for instructions, and the matrix-free product on an
// n = 64 list took 3.93 and not 2.46 ms (2.97 with eval as a call), form_rdms on
// CAS(9,9) 0.94 and not 0.89. q: 128 entries of shared memory per warp.
template <bool MIXED, int NSW, class F>
__device__ __forceinline__ void gen_pairs(const GenData& g, int32_t rg,
                                          Spin<NSW> ba, Spin<NSW> bb,
                                          uint8_t* ov, uint32_t* q, F&& eval) {
  const int lane = threadIdx.x & 31;
  int n0 = 0, n1 = 0;  // queued: others, doubles
  gen_enumerate<NSW>(g, rg, ba, bb, ov,
                     [&](bool act, int64_t m, int pa, int pb) {
    const unsigned any = __ballot_sync(0xffffffffu, act);
    if(!any) return;
    const bool dbl = !MIXED && pa + pb == 4 && !(pa & 1);
    const unsigned md = __ballot_sync(0xffffffffu, act && dbl), mo = any & ~md;
    if(act) {
      const int at = dbl ? 64 + n1 + __popc(md & lanemask_lt())
                         : n0 + __popc(mo & lanemask_lt());
      q[at] = uint32_t(m);
    }
    n0 += __popc(mo);
    n1 += __popc(md);
#pragma unroll 1
    while(n0 >= 32 || n1 >= 32) {
      const bool d = n0 < 32;
      uint32_t* qc = d ? q + 64 : q;
      __syncwarp();
      eval(true, int64_t(qc[lane]), d);
      const int left = (d ? n1 : n0) - 32;
      const uint32_t t = lane < left ? qc[32 + lane] : 0;
      __syncwarp();
      if(lane < left) qc[lane] = t;
      if(d)
        n1 = left;
      else
        n0 = left;
    }
  });
  __syncwarp();
#pragma unroll 1
  for(int c = 0; c < 2; ++c) {
    const int nc = c ? n1 : n0;
    if(nc) eval(lane < nc, int64_t(lane < nc ? q[64 * c + lane] : 0), c == 1);
  }
  __syncwarp();
}
constexpr int GEN_SCRATCH = 256 + 128 * 4;  // bytes per warp: ov, q

// H(bra, ket) of a connected pair, evaluated by class. MIXED: the lists hold
// several electron counts, and every pair takes the general element; in
// instantiations of their own, for the test of each pair made the matrix-free
// product of the usual lists 3 % slower.
template <bool MIXED, int NSW>
__device__ __forceinline__ double gen_element(const Ints& I, bool dbl,
                                              Spin<NSW> ba, Spin<NSW> bb,
                                              Spin<NSW> ka, Spin<NSW> kb,
                                              double hd) {
  if(!MIXED && dbl) return me_double(I, ba, bb, ka, kb);
  if(ka == ba && kb == bb) return hd;
  return me_generic<MIXED>(I, ba, bb, ka, kb);
}

// Candidates per row, and the rows' candidates themselves (sorted positions)
// as far as `list` holds them: a row of at most GEN_CAP takes its run of the
// list when it is done (list_off: its start, -1 when it found no room or is
// longer), so the fill need not enumerate again.
template <int NBITS>
__global__ void __launch_bounds__(HB_THREADS)
    gen_list_k(GenData g, const uint64_t* bra, int64_t nbra, int64_t* cnt,
               uint32_t* list, unsigned long long cap,
               unsigned long long* used, int64_t* list_off, unsigned* ctr) {
  using D = DetTraits<NBITS>;
  __shared__ uint8_t s_ov[HB_WARPS][256];
  __shared__ uint32_t s_m[HB_WARPS][GEN_CAP];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t* sm = s_m[wid];
  for(int64_t row; (row = next_row(ctr)) < nbra;) {
    const int32_t rg = g.rowgroup[row];
    int c = 0;
    if(rg >= 0) {
      const auto ba = D::alpha(bra + row * D::NW);
      const auto bb = D::beta(bra + row * D::NW);
      gen_enumerate<D::NSW>(g, rg, ba, bb, s_ov[wid],
                            [&](bool act, int64_t m, int, int) {
        const unsigned msk = __ballot_sync(0xffffffffu, act);
        if(act) {
          const int pos = c + __popc(msk & lanemask_lt());
          if(pos < GEN_CAP) sm[pos] = uint32_t(m);
        }
        c += __popc(msk);
      });
    }
    __syncwarp();
    unsigned long long off = 0;
    if(lane == 0) {
      cnt[row] = c;
      off = c && c <= GEN_CAP ? atomicAdd(used, (unsigned long long)c) : cap;
      list_off[row] = off + c <= cap ? int64_t(off) : -1;
    }
    off = __shfl_sync(0xffffffffu, off, 0);
    if(off + c <= cap)
      for(int i = lane; i < c; i += 32) list[off + i] = sm[i];
    __syncwarp();
  }
}

// Fill: a row's candidates go to a per-warp shared buffer as (column, sorted
// position), are sorted by column with a bitonic network, evaluated in that
// order with every lane busy and written in place; singles (sums over the
// occupied orbitals) are put off and evaluated together. Elements at or below
// the threshold are marked with column -1. Rows with more than GEN_CAP
// candidates are written unsorted to the long-row scratch (lkey/lval at
// loff[row]) and finished by the radix sort.
template <int NBITS, bool MIXED, typename CI, typename VT>
__global__ void __launch_bounds__(HB_THREADS)
    gen_fill_k(Ints I, GenData g, const uint64_t* bra, int64_t row_a,
               int64_t row_b, const double* __restrict__ hdiag,
               const int64_t* __restrict__ rowptr,
               const uint32_t* __restrict__ list,
               const int64_t* __restrict__ list_off,
               const int64_t* __restrict__ loff, int64_t lbase0,
               const uint32_t* __restrict__ lidx, uint64_t* lkey,
               double* lval, CI* __restrict__ colind, VT* __restrict__ nzval,
               double* __restrict__ diag, int64_t* __restrict__ rowcnt,
               double thresh, unsigned* ctr, unsigned long long* ndropped) {
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  __shared__ uint64_t s_key[HB_WARPS][GEN_CAP];
  __shared__ __align__(16) uint8_t s_scr[HB_WARPS][GEN_SCRATCH];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t* bk = s_key[wid];
  uint8_t* ov = s_scr[wid];
  uint32_t* q = reinterpret_cast<uint32_t*>(ov + 256);
  for(int64_t row; (row = row_a + next_row(ctr)) < row_b;) {
    const int32_t rg = g.rowgroup[row];
    const int64_t ncand = rowptr[row + 1] - rowptr[row];
    if(rg < 0 || ncand == 0) {
      if(lane == 0) rowcnt[row] = 0;
      continue;
    }
    const uint64_t* bd = bra + row * D::NW;
    const Spin<NSW> ba = D::alpha(bd), bb = D::beta(bd);
    const double hd = hdiag[row];
    if(ncand > GEN_CAP) {
      // long rows: (long-row index, column) sort keys and values into this
      // chunk's scratch; rowcnt comes from the long-row pass
      const int64_t lbase = loff[row] - lbase0;
      const uint64_t lhi = uint64_t(lidx[row]) << 32;
      int64_t c = 0;
      gen_pairs<MIXED>(g, rg, ba, bb, ov, q, [&](bool act, int64_t m, bool dbl) {
        const unsigned msk = __ballot_sync(0xffffffffu, act);
        if(act) {
          const int64_t pos = lbase + c + __popc(msk & lanemask_lt());
          lkey[pos] = lhi | g.sidx[m];
          lval[pos] = gen_element<MIXED>(I, dbl, ba, bb, ld_spin<NSW>(g.salpha, m),
                                       ld_spin<NSW>(g.sbeta, m), hd);
        }
        c += __popc(msk);
      });
      continue;
    }
    const int c = int(ncand);
    const int64_t lo = list_off[row];
    if(lo >= 0) {
      for(int i = lane; i < c; i += 32) {
        const uint32_t m = list[lo + i];
        bk[i] = (uint64_t(g.sidx[m]) << 32) | m;
      }
    } else {
      int n = 0;
      gen_enumerate<NSW>(g, rg, ba, bb, ov, [&](bool act, int64_t m, int, int) {
        const unsigned msk = __ballot_sync(0xffffffffu, act);
        if(act)
          bk[n + __popc(msk & lanemask_lt())] =
              (uint64_t(g.sidx[m]) << 32) | uint32_t(m);
        n += __popc(msk);
      });
    }
    int P = 1;
    while(P < c) P <<= 1;
    for(int i = c + lane; i < P; i += 32) bk[i] = ~0ull;
    __syncwarp();
    for(int k = 2; k <= P; k <<= 1)
      for(int jj = k >> 1; jj > 0; jj >>= 1) {
        for(int t = lane; t < (P >> 1); t += 32) {
          const int i = 2 * t - (t & (jj - 1));  // the pair (i, i + jj)
          const uint64_t x = bk[i], y = bk[i + jj];
          if((x > y) == ((i & k) == 0)) {
            bk[i] = y;
            bk[i + jj] = x;
          }
        }
        __syncwarp();
      }
    const int64_t out0 = rowptr[row];
    CI* __restrict__ rc = colind + out0;
    VT* __restrict__ rv = nzval + out0;
    int dropped = 0, nq = 0;
    auto put = [&](int i, uint32_t col, double h) {
      const bool keep = fabs(h) > thresh;
      const bool isd = keep && int64_t(col) == row;
      dropped += !keep;
      rc[i] = keep ? CI(col) : CI(-1);
      rv[i] = store_val<VT>(h, isd);
      if(isd) diag[row] = h;
    };
    auto others = [&](int cnt) {  // queued positions of singles / diagonal
      if(lane < cnt) {
        const int i = int(q[lane]);
        const uint64_t key = bk[i];
        const uint32_t m = uint32_t(key);
        put(i, uint32_t(key >> 32),
            gen_element<MIXED>(I, false, ba, bb, ld_spin<NSW>(g.salpha, m),
                             ld_spin<NSW>(g.sbeta, m), hd));
      }
    };
    for(int i0 = 0; i0 < c; i0 += 32) {
      const int i = i0 + lane;
      bool put_off = false;
      if(i < c) {
        const uint64_t key = bk[i];
        const uint32_t m = uint32_t(key);
        const Spin<NSW> ka = ld_spin<NSW>(g.salpha, m);
        const Spin<NSW> kb = ld_spin<NSW>(g.sbeta, m);
        const int ca = sp_popc(ba ^ ka), cb = sp_popc(bb ^ kb);
        if(!MIXED && ca + cb == 4 && !(ca & 1))
          put(i, uint32_t(key >> 32), me_double(I, ba, bb, ka, kb));
        else
          put_off = true;
      }
      const unsigned msk = __ballot_sync(0xffffffffu, put_off);
      if(put_off) q[nq + __popc(msk & lanemask_lt())] = uint32_t(i);
      nq += __popc(msk);
      if(nq >= 32) {
        __syncwarp();
        others(32);
        nq -= 32;
        const uint32_t t = lane < nq ? q[32 + lane] : 0;
        __syncwarp();
        if(lane < nq) q[lane] = t;
      }
    }
    __syncwarp();
    others(nq);
    dropped = __reduce_add_sync(0xffffffffu, dropped);
    if(lane == 0) {
      rowcnt[row] = ncand - dropped;
      if(dropped) atomicAdd(ndropped, (unsigned long long)dropped);
    }
    __syncwarp();
  }
}

// Long rows: the keys (row_rank << 32 | col) were radix-sorted with their
// FP64 values; write them back, marking what the threshold drops.
template <typename CI, typename VT>
__global__ void long_rows_write_k(const int64_t* lrows, int64_t nl,
                                  const int64_t* loff_sorted, int64_t base0,
                                  const uint64_t* keys, const double* vals,
                                  const int64_t* rowptr, CI* colind,
                                  VT* nzval, double* diag, int64_t* rowcnt,
                                  double thresh, unsigned long long* ndropped) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarp = int64_t(gridDim.x) * (blockDim.x >> 5);
  for(int64_t r = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      r < nl; r += nwarp) {
    const int64_t row = lrows[r];
    const int64_t b = loff_sorted[r] - base0, e = loff_sorted[r + 1] - base0;
    const int64_t out0 = rowptr[row];
    int dropped = 0;
    for(int64_t i = b + lane; i < e; i += 32) {
      const uint32_t col = uint32_t(keys[i] & 0xffffffffull);
      const double h = vals[i];
      const bool keep = fabs(h) > thresh;
      const bool isd = keep && int64_t(col) == row;
      dropped += !keep;
      colind[out0 + i - b] = keep ? CI(col) : CI(-1);
      nzval[out0 + i - b] = store_val<VT>(h, isd);
      if(isd) diag[row] = h;
    }
    dropped = __reduce_add_sync(0xffffffffu, dropped);
    if(lane == 0) {
      rowcnt[row] = e - b - dropped;
      if(dropped) atomicAdd(ndropped, (unsigned long long)dropped);
    }
  }
}

__global__ void long_flags_k(const int64_t* rowptr, size_t n, uint32_t* f) {
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x)
    f[i] = (rowptr[i + 1] - rowptr[i]) > GEN_CAP ? 1u : 0u;
}

__global__ void long_list_k(const int64_t* rowptr, size_t n,
                            const uint32_t* f, const uint32_t* fpos,
                            int64_t* lrows, int64_t* lcnt, int64_t* loff_row) {
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x)
    if(f[i]) {
      lrows[fpos[i]] = int64_t(i);
      lcnt[fpos[i]] = rowptr[i + 1] - rowptr[i];
    }
}

__global__ void long_rowoff_k(const int64_t* lrows, const int64_t* loff,
                              int64_t nl, int64_t* loff_row) {
  for(int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < nl;
      r += int64_t(gridDim.x) * blockDim.x)
    loff_row[lrows[r]] = loff[r];
}

template <typename CI>
__global__ void rowptr_cast_k(const int64_t* in, size_t n, CI* out) {
  for(size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
      i += size_t(gridDim.x) * blockDim.x)
    out[i] = CI(in[i]);
}

// ----------------------------------------------------------- driver
// General-path tables of a (bra, ket) pair: kets sorted by (alpha, beta)
// with their alpha groups, the bra rows' groups, the alpha connectivity of
// bra groups to ket groups (pa <= 3 first, pa == 4 last), beta hash tables
// of the large ket groups and the beta-major view of the kets. Everything
// lives in A; `sub` says that bra is the contiguous block of ket starting
// at row r0.
template <int NBITS>
static GenData gen_plan(macis_b200_ham* h, const uint64_t* bra, size_t nbra,
                        const uint64_t* ket, size_t nket, bool sub, int64_t r0,
                        Arena& A) {
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  cudaStream_t s = A.s;
  const int sms = num_sms();
  constexpr int KW = GenKey<NBITS>::KW;
  auto sort_side = [&](const uint64_t* dets, size_t n, uint64_t*& keys,
                       uint32_t*& idx, int64_t*& goff, uint64_t*& galpha,
                       uint64_t*& salpha, uint64_t*& sbeta, int32_t* rowgroup) {
    keys = A.get<uint64_t>(n * KW);
    idx = A.get<uint32_t>(n);
    uint64_t* k2 = A.get<uint64_t>(n * KW);
    uint32_t* i2 = A.get<uint32_t>(n);
    gen_keys_k<NBITS><<<grid_for(n, 256, 8 * sms), 256, 0, s>>>(dets, n,
                                                               keys, idx), note_launch();
    radix_sort<KW, uint32_t>(keys, idx, k2, i2, n, A);
    A.release(k2);
    A.release(i2);
    uint32_t* flags = A.get<uint32_t>(n);
    uint32_t* gx = A.get<uint32_t>(n);
    auto* d_info = A.get<GenInfo>(1);
    MB_CUDA(cudaMemsetAsync(d_info, 0, sizeof(GenInfo), s));
    gen_group_flags_k<NBITS><<<grid_for(n, 256, 8 * sms), 256, 0, s>>>(
        keys, n, flags, d_info), note_launch();
    exclusive_scan<uint32_t, uint32_t>(flags, gx, n, &d_info->groups, A);
    const GenInfo info = to_host(d_info, s);
    const uint32_t ng = info.groups;
    goff = A.get<int64_t>(ng + 1);
    galpha = A.get<uint64_t>((ng + 1) * NSW);
    salpha = A.get<uint64_t>(n * NSW);
    sbeta = A.get<uint64_t>(n * NSW);
    gen_groups_k<NBITS><<<grid_for(n, 256, 8 * sms), 256, 0, s>>>(
        keys, idx, flags, gx, n, goff, galpha, salpha, sbeta, rowgroup),
        note_launch();
    A.release(keys);
    A.release(flags);
    A.release(gx);
    gen_group_end_k<<<1, 1, 0, s>>>(goff, ng, int64_t(n)), note_launch();
    return info;
  };
  uint64_t *kkeys, *kalpha, *ksalpha, *ksbeta;
  uint32_t* kidx;
  int64_t* kgoff;
  int32_t* rowgroup = A.get<int32_t>(sub ? nket : nbra);
  const GenInfo ki = sort_side(ket, nket, kkeys, kidx, kgoff, kalpha, ksalpha,
                               ksbeta, sub ? rowgroup : nullptr);
  const uint32_t nkg = ki.groups;
  bool mixed = ki.mixed;
  if(sub) rowgroup += r0;
  const uint64_t* balpha = kalpha;
  uint32_t nbg = nkg;
  if(!sub) {
    uint64_t *bkeys, *bsalpha, *bsbeta, *bal;
    uint32_t* bidx;
    int64_t* bgoff;
    const GenInfo bi = sort_side(bra, nbra, bkeys, bidx, bgoff, bal, bsalpha,
                                 bsbeta, rowgroup);
    nbg = bi.groups;
    mixed = mixed || bi.mixed || bi.counts != ki.counts;
    A.release(bsalpha);
    A.release(bsbeta);
    balpha = bal;
  }
  // alpha connectivity bra groups -> ket groups
  int64_t* acnt = A.get<int64_t>(nbg + 1);
  int64_t* acnt4 = A.get<int64_t>(nbg + 1);
  int64_t* aoff = A.get<int64_t>(nbg + 1);
  const unsigned ga = grid_for(size_t(nbg) * 32, 256, 16 * sms);
  gen_aconn_k<NSW><<<ga, 256, 0, s>>>(balpha, nbg, kalpha, nkg, nullptr,
                                      acnt, acnt4, nullptr, nullptr), note_launch();
  exclusive_scan<int64_t, int64_t>(acnt, aoff, nbg, aoff + nbg, A);
  const int64_t natot = to_host(aoff + nbg, s);
  int32_t* acol = A.get<int32_t>(natot + 1);
  uint8_t* apa = A.get<uint8_t>(natot + 1);
  gen_aconn_k<NSW><<<ga, 256, 0, s>>>(balpha, nbg, kalpha, nkg, aoff, acnt,
                                      acnt4, acol, apa), note_launch();
  int32_t* mgroup = A.get<int32_t>(nket);
  MB_CUDA(cudaMemsetAsync(mgroup, 0xFF, nket * 4, s));
  gen_mgroup_k<<<grid_for(size_t(nkg) * 32, 256, 16 * sms), 256, 0, s>>>(
      kgoff, nkg, mgroup), note_launch();
  // beta hash tables of the large ket groups
  int64_t* hoff = A.get<int64_t>(nkg + 1);
  int32_t* gbpop = A.get<int32_t>(nkg + 1);
  int32_t* htab;
  {
    int64_t* hsz = A.get<int64_t>(nkg + 1);
    const unsigned gh = grid_for(size_t(nkg) * 32, 256, 16 * sms);
    gen_hsize_k<NSW><<<gh, 256, 0, s>>>(kgoff, nkg, ksbeta, hsz, gbpop), note_launch();
    exclusive_scan<int64_t, int64_t>(hsz, hoff, nkg, hoff + nkg, A);
    A.release(hsz);
    const int64_t htot = to_host(hoff + nkg, s);
    htab = A.get<int32_t>(size_t(std::max<int64_t>(htot, 1)));
    MB_CUDA(cudaMemsetAsync(htab, 0xFF, size_t(std::max<int64_t>(htot, 1)) * 4, s));
    if(htot > 0)
      gen_hinsert_k<NSW><<<grid_for(nket, 256, 16 * sms), 256, 0, s>>>(
          kgoff, mgroup, nket, ksbeta, hoff, htab), note_launch();
  }
  // beta-major view of the kets
  uint64_t *bm_alpha, *bgbeta;
  uint32_t* bm_m;
  int64_t* bgoff;
  int64_t nbgb = 0;
  {
    uint64_t* bkeys = A.get<uint64_t>(nket * KW);
    uint32_t* bidx = A.get<uint32_t>(nket);
    uint64_t* k2 = A.get<uint64_t>(nket * KW);
    uint32_t* i2 = A.get<uint32_t>(nket);
    gen_bkeys_k<NBITS><<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(
        ket, nket, bkeys, bidx), note_launch();
    radix_sort<KW, uint32_t>(bkeys, bidx, k2, i2, nket, A);
    A.release(k2);
    A.release(i2);
    uint32_t* amaj = A.get<uint32_t>(nket);
    gen_invert_k<<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(kidx, nket,
                                                             amaj), note_launch();
    bm_alpha = A.get<uint64_t>(nket * NSW);
    bm_m = A.get<uint32_t>(nket);
    uint32_t* bfl = A.get<uint32_t>(nket);
    uint32_t* bgx = A.get<uint32_t>(nket + 1);
    gen_bmajor_k<NBITS><<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(
        bkeys, bidx, nket, amaj, bm_alpha, bm_m, bfl), note_launch();
    exclusive_scan<uint32_t, uint32_t>(bfl, bgx, nket, bgx + nket, A);
    nbgb = int64_t(to_host(bgx + nket, s));
    bgoff = A.get<int64_t>(size_t(nbgb) + 1);
    bgbeta = A.get<uint64_t>((size_t(nbgb) + 1) * NSW);
    gen_bgroups_k<NBITS><<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(
        bkeys, bfl, bgx, nket, bgoff, bgbeta), note_launch();
    gen_group_end_k<<<1, 1, 0, s>>>(bgoff, uint32_t(nbgb), int64_t(nket)), note_launch();
    A.release(bkeys);
    A.release(bidx);
    A.release(amaj);
    A.release(bfl);
    A.release(bgx);
  }
  GenData gd{rowgroup, aoff, acol, apa, kgoff, ksalpha, ksbeta, kidx,
             hoff, htab, gbpop, h->norb, acnt4,
             bgbeta, bgoff, nbgb, bm_alpha, bm_m, mgroup, mixed};
  return gd;
}

template <int NBITS, typename CI, typename VT>
static void build_impl(macis_b200_ham* h, const uint64_t* bra, size_t nbra,
                       const uint64_t* ket, size_t nket, double thresh,
                       macis_b200_csr* out) {
  bool general_fill_timed = false;  // the chunked general fill sums its own time
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  cudaStream_t s = h->stream;
  Arena A(s);
  const Ints I = h->ints();
  const int sms = num_sms();
  // bra may be a contiguous row block of the ket list (the row partition of
  // make_dist_csr_hamiltonian, csr_hamiltonian.hpp:49-82)
  const bool sub = bra >= ket && bra + nbra * D::NW <= ket + nket * D::NW &&
                   (bra - ket) % D::NW == 0;
  const int64_t r0 = sub ? int64_t((bra - ket) / D::NW) : 0;

  out->m = int64_t(nbra);
  out->n = int64_t(nket);
  MB_CUDA(dev_malloc_async(&out->diag, std::max<size_t>(nbra, 1) * 8, s));
  MB_CUDA(cudaMemsetAsync(out->diag, 0, std::max<size_t>(nbra, 1) * 8, s));
  int64_t* rowptr64 = A.get<int64_t>(nbra + 1);
  int64_t* rowcnt = A.get<int64_t>(nbra + 1);
  int64_t* nnz_d = A.get<int64_t>(1);
  double* hdiag = A.get<double>(nbra + 1);

  struct Ev {
    cudaEvent_t e[2];
    Ev() { cudaEventCreate(&e[0]); cudaEventCreate(&e[1]); }
    ~Ev() { cudaEventDestroy(e[0]); cudaEventDestroy(e[1]); }
    cudaEvent_t& operator[](int i) { return e[i]; }
  } ev;
  if(nbra == 0 || nket == 0) {
    out->nnz = 0;
    MB_CUDA(dev_malloc_async(&out->rowptr, (nbra + 1) * sizeof(CI), s));
    MB_CUDA(cudaMemsetAsync(out->rowptr, 0, (nbra + 1) * sizeof(CI), s));
    MB_CUDA(dev_malloc_async(&out->colind, 256, s));
    MB_CUDA(dev_malloc_async(&out->nzval, 256, s));
    MB_CUDA(cudaStreamSynchronize(s));
    return;
  }
  MB_REQUIRE(nket < (size_t(1) << 31), MACIS_B200_ECAPACITY,
             "ket list longer than 2^31 determinants");

  hdiag_k<NBITS><<<grid_for(nbra, 256, 8 * sms), 256, 0, s>>>(I, bra, nbra,
                                                              hdiag), note_launch();

  // ---------------------------------------------- direct-product check
  bool direct = false;
  size_t UA = 0, UB = 0;
  uint64_t *ua = nullptr, *ub = nullptr;
  if(sub) {
    auto* first = A.get<unsigned long long>(1);
    const unsigned long long big = ~0ull;
    MB_CUDA(cudaMemcpyAsync(first, &big, 8, cudaMemcpyHostToDevice, s));
    first_alpha_change_k<NBITS><<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(
        ket, nket, first), note_launch();
    unsigned long long f = to_host(first, s);
    UB = f == big ? nket : size_t(f);
    if(UB > 0 && nket % UB == 0) {
      UA = nket / UB;
      int* bad = A.get<int>(1);
      MB_CUDA(cudaMemsetAsync(bad, 0, 4, s));
      dp_check_k<NBITS><<<grid_for(nket, 256, 8 * sms), 256, 0, s>>>(
          ket, nket, UB, bad), note_launch();
      ua = A.get<uint64_t>(UA * NSW);
      ub = A.get<uint64_t>(UB * NSW);
      gather_block_spins_k<NBITS><<<grid_for(std::max(UA, UB), 256, 8 * sms),
                                    256, 0, s>>>(ket, UA, UB, ua, ub), note_launch();
      const int hb = to_host(bad, s);
      // the fill keeps a singles table of 2 norb^2 doubles per warp in
      // shared memory: spaces whose orbitals make it too large (norb above
      // ~33) take the general path even when they have the product layout
      direct = hb == 0 && UA < (size_t(1) << 31) &&
               UB < (size_t(1) << 31) && h->norb <= 127 &&
               dp_shared_layout(int(h->norb), 512, 1024).bytes <= 220 * 1024;
    }
  }

  int64_t nnz_ub = 0;
  // the matrix is the arena's until the build has succeeded
  CI* colind = nullptr;
  VT* nzval = nullptr;
  // direct product: connectivity counts and row sizes, read back together
  DPTotals tot{};
  DPTotals* d_tot = A.get<DPTotals>(1);
  MB_CUDA(cudaMemsetAsync(d_tot, 0, sizeof(DPTotals), s));
  int64_t *aoff = nullptr, *l2off = nullptr, *l4off = nullptr;
  if(direct) {
    int32_t* cls_a = A.get<int32_t>(3 * UA);
    int32_t* cls_b = A.get<int32_t>(3 * UB);
    int64_t* cnt = A.get<int64_t>(2 * (UA + UB));
    int64_t *ca2 = cnt, *ca4 = ca2 + UA, *cb2 = ca4 + UA, *cb4 = cb2 + UB;
    dp_conn_count_k<NSW><<<grid_for(UA * 32, 256, 16 * sms), 256, 0, s>>>(
        ua, UA, cls_a, ca2, ca4, 0, d_tot), note_launch();
    dp_conn_count_k<NSW><<<grid_for(UB * 32, 256, 16 * sms), 256, 0, s>>>(
        ub, UB, cls_b, cb2, cb4, 1, d_tot), note_launch();
    aoff = A.get<int64_t>(UA + 1);
    l2off = A.get<int64_t>(UB + 1);
    l4off = A.get<int64_t>(UB + 1);
    exclusive_scan<int64_t, int64_t>(ca4, aoff, UA, aoff + UA, A);
    exclusive_scan<int64_t, int64_t>(cb2, l2off, UB, l2off + UB, A);
    exclusive_scan<int64_t, int64_t>(cb4, l4off, UB, l4off + UB, A);
    dp_rowcount_k<<<grid_for(nbra, 256, 8 * sms), 256, 0, s>>>(
        cls_a, cb2, cb4, r0, int64_t(nbra), int64_t(UB), rowcnt), note_launch();
    exclusive_scan<int64_t, int64_t>(rowcnt, rowptr64, nbra, rowptr64 + nbra, A);
    dp_totals_k<<<1, 1, 0, s>>>(aoff, UA, l2off, l4off, UB, rowptr64, nbra,
                                d_tot), note_launch();
    tot = to_host(d_tot, s);
    direct = !tot.dup;  // a string twice: not a product space after all
  }
  if(direct) {
    out->direct_product = true;
    nnz_ub = tot.nnz;
    out->nnz_candidates = nnz_ub;
    colind = A.get<CI>(size_t(nnz_ub));
    nzval = A.get<VT>(size_t(nnz_ub));
    // orbital lists of the kernels below hold 128 entries per spin
    MB_REQUIRE(nket < (size_t(1) << 31) && h->norb <= 127,
               MACIS_B200_ECAPACITY,
               "direct-product fill needs < 2^31 determinants, norb < 128");
    int32_t* acol = A.get<int32_t>(tot.na + 1);
    uint32_t* ainfo = A.get<uint32_t>(tot.na + 1);
    double* aval = A.get<double>(tot.na + 1);
    int32_t* l2col = A.get<int32_t>(tot.n2 + 1);
    uint32_t* l2info = A.get<uint32_t>(tot.n2 + 1);
    int32_t* l4col = A.get<int32_t>(tot.n4 + 1);
    uint32_t* l4info = A.get<uint32_t>(tot.n4 + 1);
    double* l4val = A.get<double>(tot.n4 + 1);
    dp_conn_fill_k<NSW><<<grid_for(UA * 32, 256, 16 * sms), 256, 0, s>>>(
        ua, UA, h->norb, 0, I.G, aoff, acol, ainfo, aval, nullptr, nullptr,
        nullptr), note_launch();
    dp_conn_fill_k<NSW><<<grid_for(UB * 32, 256, 16 * sms), 256, 0, s>>>(
        ub, UB, h->norb, 2, I.G, l4off, l4col, l4info, l4val, l2off, l2col,
        l2info), note_launch();
    // same-spin partial sums of the singles, per alpha and per beta string:
    // at most norb^2 / 4 singles per string
    const size_t nsing = size_t(h->norb) * h->norb / 4 + 1;
    double* pga = A.get<double>(UA * nsing);
    double* pgb = A.get<double>(UB * nsing);
    dp_pg_k<NSW><<<grid_for(UA * 32, 256, 8 * sms), 256, 0, s>>>(
        I, ua, int64_t(UA), pga), note_launch();
    dp_pg_k<NSW><<<grid_for(UB * 32, 256, 8 * sms), 256, 0, s>>>(
        I, ub, int64_t(UB), pgb), note_launch();
    DPData d{int64_t(UA), int64_t(UB), ua, ub, aoff, acol, ainfo,
             l2off, l2col, l2info, l4off, l4col, l4info,
             pga, pgb, aval, l4val};
    // shared-memory plan: the longest beta lists, per-warp singles tables
    int64_t l2max = tot.l2max, l4max = tot.l4max;
    const int nn = h->norb;
    // The integrals of the singles are read through L1 rather than staged in
    // shared memory: per-CTA copies would take the L1 capacity that the
    // G / V gathers need (measured: staging made the C2 fill 10% slower).
    l2max = std::min<int64_t>(l2max, 2048);
    l4max = std::min<int64_t>(l4max, 4096);
    DPShared Ls = dp_shared_layout(nn, l2max, l4max);
    if(Ls.bytes > 200 * 1024) {
      Ls = dp_shared_layout(nn, std::min<int64_t>(l2max, 512),
                            std::min<int64_t>(l4max, 1024));
    }
    MB_REQUIRE(Ls.bytes <= 220 * 1024, MACIS_B200_EINVAL,
               "norb too large for the direct-product fill");
    MB_CUDA(cudaFuncSetAttribute(dp_fill_k<NBITS, CI, VT>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(Ls.bytes)));
    // shared-memory carveout: the smallest that keeps DP_CTAS CTAs resident
    // (dynamic + static shared memory + the 1 KB the SM reserves per CTA),
    // the rest is L1. The carveout is a preference that the driver maps to
    // one of a few sizes, so it is raised until the occupancy query agrees.
    int per_sm = 0;
    {
      cudaFuncAttributes fa;
      MB_CUDA(cudaFuncGetAttributes(&fa, dp_fill_k<NBITS, CI, VT>));
      const size_t per_cta = Ls.bytes + fa.sharedSizeBytes + 1024;
      int pct = int(std::min<size_t>(
          100, (DP_CTAS * per_cta * 100 + 228 * 1024 - 1) / (228 * 1024)));
      for(;;) {
        MB_CUDA(cudaFuncSetAttribute(
            dp_fill_k<NBITS, CI, VT>,
            cudaFuncAttributePreferredSharedMemoryCarveout, pct));
        MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, dp_fill_k<NBITS, CI, VT>, DP_THREADS, Ls.bytes));
        if(per_sm >= DP_CTAS || pct >= 100) break;
        pct = std::min(100, pct + 5);
      }
    }
    const unsigned g = unsigned(std::max(1, per_sm) * sms);
    ham_vt(h);
    NvtxRange nv_fill("macis_b200: direct-product fill");
    cudaEventRecord(ev[0], s);
    dp_fill_k<NBITS, CI, VT><<<g, DP_THREADS, Ls.bytes, s>>>(
        I, h->VT, d, Ls, hdiag, rowptr64, colind, nzval, out->diag, rowcnt, thresh,
        r0, int64_t(nbra), &d_tot->dropped), note_launch();
    cudaEventRecord(ev[1], s);
    MB_CUDA(cudaGetLastError());
  } else {
    // ------------------------------------------------ general path
    GenData gd = gen_plan<NBITS>(h, bra, nbra, ket, nket, sub, r0, A);
    const unsigned gr = grid_for(nbra, HB_WARPS, size_t(sms) * 16);
    // candidate lists of the rows, as far as a tenth of the memory holds
    // them (4 B per candidate, at most GEN_CAP per row). What is free is asked
    // for long lists alone: the query takes 60 us and, on a shared host, up to
    // milliseconds, as much as the build of a few hundred determinants.
    unsigned* ctr = A.get<unsigned>(1);
    auto* used = A.get<unsigned long long>(1);
    int64_t* list_off = A.get<int64_t>(nbra);
    uint64_t cap = std::min<uint64_t>(uint64_t(nbra) * GEN_CAP,
                                      candidate_list_limit());
    size_t avail = 0;
    if(4 * cap > GEN_LIST_ASK) {
      avail = device_bytes_available();
      cap = std::min<uint64_t>(cap, avail / 40);
    }
    auto have = [](auto&& get) {  // memory that may be missing
      try {
        get();
      } catch(const Error& e) {
        if(e.code != MACIS_B200_ENOMEM) throw;
        cudaGetLastError();  // the allocation's
        return false;
      }
      return true;
    };
    uint32_t* list = nullptr;
    if(!have([&] { list = A.get<uint32_t>(cap); })) cap = 0;
    MB_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned), s));
    MB_CUDA(cudaMemsetAsync(used, 0, 8, s));
    gen_list_k<NBITS><<<gr, HB_THREADS, 0, s>>>(
        gd, bra, int64_t(nbra), rowcnt, list, cap, used, list_off, ctr),
        note_launch();
    exclusive_scan<int64_t, int64_t>(rowcnt, rowptr64, nbra, rowptr64 + nbra, A);
    nnz_ub = to_host(rowptr64 + nbra, s);
    // a matrix that needs their memory goes without the lists
    auto drop_list = [&] {
      A.release(list);
      list = nullptr;
      MB_CUDA(cudaMemsetAsync(list_off, 0xFF, nbra * 8, s));
    };
    if(list && avail &&
       1.05 * double(nnz_ub) * (sizeof(CI) + sizeof(VT)) + 1073741824.0 +
               4.0 * double(cap) > double(avail))
      drop_list();
    out->nnz_candidates = nnz_ub;
    auto get_matrix = [&] {
      colind = A.get<CI>(size_t(nnz_ub));
      nzval = A.get<VT>(size_t(nnz_ub));
    };
    if(!list) {
      get_matrix();
    } else if(!have(get_matrix)) {
      if(colind) A.release(colind);
      drop_list();
      get_matrix();
    }
    // long rows
    uint32_t* lf = A.get<uint32_t>(nbra + 1);
    uint32_t* lpos = A.get<uint32_t>(nbra + 1);
    long_flags_k<<<grid_for(nbra, 256, 8 * sms), 256, 0, s>>>(rowptr64, nbra, lf), note_launch();
    exclusive_scan<uint32_t, uint32_t>(lf, lpos, nbra, lpos + nbra, A);
    const uint32_t nl = to_host(lpos + nbra, s);
    out->long_rows = nl;
    int64_t *lrows = nullptr, *lcnt = nullptr, *loff = nullptr,
            *loff_row = nullptr;
    int64_t ltot = 0;
    std::vector<int64_t> h_lrows, h_loff;
    if(nl) {
      lrows = A.get<int64_t>(nl + 1);
      lcnt = A.get<int64_t>(nl + 1);
      loff = A.get<int64_t>(nl + 1);
      loff_row = A.get<int64_t>(nbra);
      long_list_k<<<grid_for(nbra, 256, 8 * sms), 256, 0, s>>>(
          rowptr64, nbra, lf, lpos, lrows, lcnt, loff_row), note_launch();
      exclusive_scan<int64_t, int64_t>(lcnt, loff, nl, loff + nl, A);
      ltot = to_host(loff + nl, s);
      long_rowoff_k<<<grid_for(nl, 256, 4 * sms), 256, 0, s>>>(lrows, loff, nl,
                                                              loff_row), note_launch();
      h_lrows.resize(nl);
      h_loff.resize(nl + 1);
      MB_CUDA(cudaMemcpyAsync(h_lrows.data(), lrows, nl * 8,
                              cudaMemcpyDeviceToHost, s));
      MB_CUDA(cudaMemcpyAsync(h_loff.data(), loff, (nl + 1) * 8,
                              cudaMemcpyDeviceToHost, s));
      MB_CUDA(cudaStreamSynchronize(s));
    }
    // Long rows are finished in chunks of consecutive rows whose scratch
    // (key + value, and the sort's second copy: 32 B per entry) fits in
    // what is free; short rows of the chunk are written by the same launch.
    int64_t lchunk = int64_t(0.7 * double(device_bytes_available()) / 32.0);
    lchunk = std::min<int64_t>(std::max<int64_t>(lchunk, int64_t(1) << 20),
                               int64_t(RS_MAX_RECORDS));
    float fill_ms_tot = 0.f;
    int64_t la = 0;  // next long row (list index)
    int64_t row_a = 0;
    do {
      int64_t lb = la;  // long rows [la, lb) in this chunk
      while(lb < int64_t(nl) && (lb == la || h_loff[lb + 1] - h_loff[la] <= lchunk))
        ++lb;
      const int64_t row_b = lb < int64_t(nl) ? h_lrows[lb] : int64_t(nbra);
      const int64_t cbase = nl ? h_loff[la] : 0;
      const int64_t centries = nl ? h_loff[lb] - cbase : 0;
      Arena C(s);
      uint64_t* lkey = C.get<uint64_t>(centries + 1);
      double* lval = C.get<double>(centries + 1);
      cudaEventRecord(ev[0], s);
      MB_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned), s));
      auto fill = gd.mixed ? gen_fill_k<NBITS, true, CI, VT>
                           : gen_fill_k<NBITS, false, CI, VT>;
      fill<<<gr, HB_THREADS, 0, s>>>(
          I, gd, bra, row_a, row_b, hdiag, rowptr64, list, list_off, loff_row,
          cbase, lpos, lkey, lval, colind, nzval, out->diag, rowcnt, thresh,
          ctr, &d_tot->dropped), note_launch();
      cudaEventRecord(ev[1], s);
      MB_CUDA(cudaGetLastError());
      MB_CUDA(cudaEventSynchronize(ev[1]));
      float ms = 0.f;
      MB_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      fill_ms_tot += ms;
      if(lb > la) {
        uint64_t* lk2 = C.get<uint64_t>(centries + 1);
        double* lv2 = C.get<double>(centries + 1);
        radix_sort<1, double>(lkey, lval, lk2, lv2, size_t(centries), C);
        long_rows_write_k<CI, VT><<<grid_for(size_t(lb - la) * 32, 256, 8 * sms),
                                    256, 0, s>>>(
            lrows + la, lb - la, loff + la, cbase, lkey, lval, rowptr64,
            colind, nzval, out->diag, rowcnt, thresh, &d_tot->dropped),
            note_launch();
        MB_CUDA(cudaGetLastError());
      }
      la = lb;
      row_a = row_b;
    } while(row_a < int64_t(nbra));
    out->fill_ms = fill_ms_tot;
    general_fill_timed = true;
    // the compaction below takes a second copy of the matrix: nothing of the
    // candidates is held beside it
    if(list) A.release(list);
  }

  // ------------------------------------------- exact row pointer + compaction
  int64_t* newptr = rowptr64;
  int64_t nnz = nnz_ub;
  // (when nothing was dropped the candidate row pointer stands)
  if(to_host(&d_tot->dropped, s) != 0) {
    newptr = A.get<int64_t>(nbra + 1);
    exclusive_scan<int64_t, int64_t>(rowcnt, newptr, nbra, newptr + nbra, A);
    nnz = to_host(newptr + nbra, s);
  }
  out->nnz = nnz;
  if(sizeof(CI) == 4)
    MB_REQUIRE(nnz <= int32_index_limit(), MACIS_B200_ECAPACITY,
               "nnz exceeds the int32 index range; use 64-bit indices");
  if(nnz != nnz_ub) {
    CI* ci2 = A.get<CI>(size_t(nnz));
    VT* nz2 = A.get<VT>(size_t(nnz));
    compact_marked_k<CI, VT><<<grid_for(nbra * 32, 256, 16 * sms), 256, 0, s>>>(
        rowptr64, newptr, nbra, colind, nzval, ci2, nz2), note_launch();
    A.release(colind);
    A.release(nzval);
    colind = ci2;
    nzval = nz2;
  }
  MB_CUDA(dev_malloc_async(&out->rowptr, (nbra + 1) * sizeof(CI), s));
  rowptr_cast_k<CI><<<grid_for(nbra + 1, 256, 8 * sms), 256, 0, s>>>(
      newptr, nbra + 1, static_cast<CI*>(out->rowptr)), note_launch();
  A.keep(colind);
  A.keep(nzval);
  out->colind = colind;
  out->nzval = nzval;
  MB_CUDA(cudaGetLastError());
  MB_CUDA(cudaStreamSynchronize(s));
  if(!general_fill_timed) cudaEventElapsedTime(&out->fill_ms, ev[0], ev[1]);
}

macis_b200_csr* build_csr_device(macis_b200_ham* h, const uint64_t* bra,
                                 size_t nbra, const uint64_t* ket, size_t nket,
                                 double thresh, int idx_bytes, int val_bytes) {
  NvtxRange nv("macis_b200: CSR build");
  MB_REQUIRE(idx_bytes == 4 || idx_bytes == 8, MACIS_B200_EINVAL,
             "Unsupported index_t");
  MB_REQUIRE(val_bytes == 4 || val_bytes == 8, MACIS_B200_EINVAL,
             "val_bytes must be 4 or 8");
  auto* out = new macis_b200_csr;
  out->idx_bytes = idx_bytes;
  out->val_bytes = val_bytes;
  out->device = h->device;
  out->pinned = h->pinned;
  MB_CUDA(cudaStreamCreateWithFlags(&out->stream, cudaStreamNonBlocking));
  out->own_stream = true;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, h->stream);
  try {
#define MB_BUILD(NB)                                                          \
  if(idx_bytes == 4 && val_bytes == 8)                                        \
    build_impl<NB, int32_t, double>(h, bra, nbra, ket, nket, thresh, out);    \
  else if(idx_bytes == 4)                                                     \
    build_impl<NB, int32_t, float>(h, bra, nbra, ket, nket, thresh, out);     \
  else if(val_bytes == 8)                                                     \
    build_impl<NB, int64_t, double>(h, bra, nbra, ket, nket, thresh, out);    \
  else                                                                        \
    build_impl<NB, int64_t, float>(h, bra, nbra, ket, nket, thresh, out);
    if(h->nbits == 64) {
      MB_BUILD(64)
    } else if(h->nbits == 128) {
      MB_BUILD(128)
    } else {
      MB_BUILD(256)
    }
#undef MB_BUILD
  } catch(...) {
    cudaStreamSynchronize(h->stream);
    if(out->rowptr) cudaFreeAsync(out->rowptr, h->stream);
    if(out->colind) cudaFreeAsync(out->colind, h->stream);
    if(out->nzval) cudaFreeAsync(out->nzval, h->stream);
    if(out->diag) cudaFreeAsync(out->diag, h->stream);
    cudaStreamSynchronize(h->stream);
    cudaStreamDestroy(out->stream);
    delete out;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    throw;
  }
  cudaEventRecord(e1, h->stream);
  cudaEventSynchronize(e1);
  cudaEventElapsedTime(&out->build_ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return out;
}

}  // namespace mb

// ------------------------------------------------ matrix-free H x
// The operator keeps its own stream and a copy of the generator's integral
// pointers: the generator must outlive every product, but destroying the
// operator never touches it.
struct macis_b200_hop {
  std::shared_ptr<mb::PinnedPool> pinned;
  mb::Ints I{};
  int nbits = 64;
  cudaStream_t stream = nullptr;
  int64_t n = 0;
  double thresh = 0.0;
  bool mixed = false;
  uint64_t* dets = nullptr;  // device copy of the determinant list
  double* diag = nullptr;    // H_ii
  mb::Arena* A = nullptr;    // owns dets, diag and the enumeration tables
  unsigned* ctr = nullptr;   // next row and finished blocks of a product
  mb::GenData g{};
};

namespace mb {

// y = alpha H x + beta y, one warp per row: the candidates of the general
// build's enumeration (gen_enumerate), each element evaluated, thresholded
// as in the build and accumulated into the row sum (no storage). mixed:
// off-diagonal elements rounded to FP32 first, as in an FP32-valued CSR.
// ctr: {next row, finished blocks}, both 0 before and after: the last block
// clears them, so that a product is one stream operation and two that are
// enqueued at once by several host threads follow one another.
template <int NBITS, bool MIXED>
__global__ void __launch_bounds__(HB_THREADS)
    gen_apply_k(Ints I, GenData g, const uint64_t* dets, int64_t n,
                const double* __restrict__ hdiag, double thresh, int mixed,
                double alpha, const double* __restrict__ x, double beta,
                double* __restrict__ y, unsigned* ctr,
                unsigned long long* t0) {
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  __shared__ __align__(16) uint8_t s_scr[HB_WARPS][GEN_SCRATCH];
  note_start(t0);
  const int lane = threadIdx.x & 31;
  uint8_t* ov = s_scr[threadIdx.x >> 5];
  for(int64_t row; (row = next_row(ctr)) < n;) {
    const int32_t rg = g.rowgroup[row];
    double acc = 0.0;
    if(rg >= 0) {
      const uint64_t* bd = dets + row * D::NW;
      const Spin<NSW> ba = D::alpha(bd), bb = D::beta(bd);
      const double hd = hdiag[row];
      gen_pairs<MIXED>(g, rg, ba, bb, ov, reinterpret_cast<uint32_t*>(ov + 256),
                     [&](bool act, int64_t m, bool dbl) {
        if(act) {
          const uint32_t col = g.sidx[m];
          double h = gen_element<MIXED>(I, dbl, ba, bb, ld_spin<NSW>(g.salpha, m),
                                      ld_spin<NSW>(g.sbeta, m), hd);
          if(fabs(h) > thresh) {
            if(mixed && int64_t(col) != row) h = double(float(h));
            acc += h * x[col];
          }
        }
      });
#pragma unroll
      for(int o = 16; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if(lane == 0) y[row] = alpha * acc + (beta != 0.0 ? beta * y[row] : 0.0);
  }
  __syncthreads();  // this block takes no more rows
  if(threadIdx.x == 0 && atomicAdd(ctr + 1, 1u) == gridDim.x - 1) {
    ctr[0] = 0;
    ctr[1] = 0;
  }
}

macis_b200_hop* hop_create(macis_b200_ham* h, const uint64_t* dets, size_t n,
                           double thresh, bool mixed, bool device_ptrs) {
  MB_REQUIRE(n > 0, MACIS_B200_EINVAL, "empty determinant list");
  MB_REQUIRE(n < (size_t(1) << 31), MACIS_B200_ECAPACITY,
             "matrix-free H needs < 2^31 determinants");
  const size_t nw = size_t(h->nbits / 64);
  const int sms = num_sms();
  const Ints I = h->ints();
  auto* op = new macis_b200_hop;
  op->pinned = h->pinned;
  op->I = I;
  op->nbits = h->nbits;
  op->n = int64_t(n);
  op->thresh = thresh;
  op->mixed = mixed;
  if(cudaStreamCreateWithFlags(&op->stream, cudaStreamNonBlocking) !=
     cudaSuccess) {
    delete op;
    MB_REQUIRE(false, MACIS_B200_ECUDA, "stream creation failed");
  }
  cudaStream_t s = op->stream;
  try {
    op->A = new Arena(s);
    op->dets = op->A->get<uint64_t>(n * nw);
    MB_CUDA(cudaMemcpyAsync(op->dets, dets, n * nw * 8,
                            device_ptrs ? cudaMemcpyDeviceToDevice
                                        : cudaMemcpyHostToDevice, s));
    op->diag = op->A->get<double>(n);
    op->ctr = op->A->get<unsigned>(2);
    MB_CUDA(cudaMemsetAsync(op->ctr, 0, 2 * sizeof(unsigned), s));
#define MB_HOP_PLAN(NB)                                                     \
  hdiag_k<NB><<<grid_for(n, 256, 8 * sms), 256, 0, s>>>(I, op->dets, n,     \
                                                        op->diag),          \
      note_launch();                                                        \
  op->g = gen_plan<NB>(h, op->dets, n, op->dets, n, true, 0, *op->A);
    if(h->nbits == 64) {
      MB_HOP_PLAN(64)
    } else if(h->nbits == 128) {
      MB_HOP_PLAN(128)
    } else {
      MB_HOP_PLAN(256)
    }
#undef MB_HOP_PLAN
    MB_CUDA(cudaStreamSynchronize(s));
  } catch(...) {
    cudaStreamSynchronize(s);
    delete op->A;
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    delete op;
    throw;
  }
  return op;
}

void hop_apply(const macis_b200_hop* op, double alpha, const double* x,
               double beta, double* y, unsigned long long* t0) {
  cudaStream_t s = op->stream;
  const unsigned gr = grid_for(size_t(op->n), HB_WARPS, size_t(num_sms()) * 16);
  const Ints I = op->I;
#define MB_HOP_APPLY(NB)                                                     \
  (op->g.mixed ? gen_apply_k<NB, true> : gen_apply_k<NB, false>)             \
      <<<gr, HB_THREADS, 0, s>>>(I, op->g, op->dets, op->n, op->diag,        \
                                 op->thresh, op->mixed ? 1 : 0, alpha, x,    \
                                 beta, y, op->ctr, t0),                      \
      note_launch();
  if(op->nbits == 64) {
    MB_HOP_APPLY(64)
  } else if(op->nbits == 128) {
    MB_HOP_APPLY(128)
  } else {
    MB_HOP_APPLY(256)
  }
#undef MB_HOP_APPLY
  MB_CUDA(cudaGetLastError());
}

void hop_destroy(macis_b200_hop* op) {
  if(!op) return;
  cudaStreamSynchronize(op->stream);
  delete op->A;
  cudaStreamSynchronize(op->stream);
  cudaStreamDestroy(op->stream);
  delete op;
}

int64_t hop_size(const macis_b200_hop* op) { return op->n; }
const double* hop_diag(const macis_b200_hop* op) { return op->diag; }
cudaStream_t hop_stream(const macis_b200_hop* op) { return op->stream; }
const std::shared_ptr<PinnedPool>& hop_pinned(const macis_b200_hop* op) {
  return op->pinned;
}

}  // namespace mb

// ------------------------------------------------ 1- and 2-RDMs
namespace mb {

__device__ __forceinline__ void rdm_add(double* a, size_t i, double v) {
  atomicAdd(a + i, v);
}

// Sums of rdm_contributions (include/macis/util/rdms.hpp:15-131) over all
// (bra, ket) pairs, one entry for what the reference adds to several: a pair
// costs 1 atomic instead of 2 (opposite-spin doubles), 1 instead of 4 (same
// spin), and a single 1 per occupied orbital instead of 4 or 2; rdm_expand_k
// then forms every element of the 2-RDM from the entries that reach it.
// Indices as the 2-RDM's, (p,q,r,s) at p + n (q + n (r + n s)). The sums take
// twice the 2-RDM's memory and two passes over it; DIRECT kernels add every
// pair to the 2-RDM itself and need neither (form_rdms_device chooses).
struct RdmSums {
  double* trdm;   // the 2-RDM (DIRECT)
  double* os;     // n^4: (v1, o1, v2, o2), alpha and beta excitation
  double* ss;     // n^4: (v1, o1, v2, o2) of double_ex, both spins
  double* ss1;    // n^3: (v1, o1, p), p occupied in the excited spin
  double* os1;    // n^3: (v1, o1, p), p occupied in the other spin
  double* diag;   // per row: the sum over its pairs with itself
  double* dss;    // n^2: (p, q) both occupied in one spin, over both spins
  double* dos;    // n^2: p occupied in alpha, q in beta
};

// One pair in the reference's dispatch (:15-66); pairs of the diagonal branch
// return true. MIXED: the list holds several electron counts; pairs that
// differ by 2 or 4 electrons of a spin contribute nothing.
template <bool DIRECT, bool MIXED, int NSW>
__device__ __forceinline__ bool rdm_pair(Spin<NSW> ba, Spin<NSW> bb,
                                         Spin<NSW> ka, Spin<NSW> kb,
                                         double val, int n, double* ordm,
                                         bool two, const RdmSums& S) {
  const int ca = sp_popc(ba ^ ka), cb = sp_popc(bb ^ kb);
  if(ca + cb > 4) return false;
  if(MIXED && (unbalanced(ba, ka) || unbalanced(bb, kb))) return false;
  auto at = [n](int p, int q, int r) { return size_t(p) + size_t(n) * (q + size_t(n) * r); };
  auto t4 = [&](int p, int q, int r, int s, double v) {
    rdm_add(S.trdm, idx4(p, q, r, s, n), v);
  };
  if((ca == 4 || cb == 4) && two) {  // rdm_contributions_4, :15-25
    const uint32_t e = ca == 4 ? double_ex(ba, ka) : double_ex(bb, kb);
    const int o1 = ex_o1(e), v1 = ex_v1(e), o2 = ex_o2(e), v2 = ex_v2(e);
    if constexpr(DIRECT) {
      const double v = val * (ex_sgn(e) * 0.5);
      t4(v1, o1, v2, o2, v);
      t4(v2, o1, v1, o2, -v);
      t4(v1, o2, v2, o1, -v);
      t4(v2, o2, v1, o1, v);
    } else {
      rdm_add(S.ss, idx4(v1, o1, v2, o2, n), val * ex_sgn(e));
    }
  } else if(ca == 2 && cb == 2 && two) {  // rdm_contributions_22, :27-41
    const uint32_t ea = single_ex(ba, ka), eb = single_ex(bb, kb);
    const int o1 = ex_o1(ea), v1 = ex_v1(ea), o2 = ex_o1(eb), v2 = ex_v1(eb);
    const double sg = ex_sgn(ea) * ex_sgn(eb);
    if constexpr(DIRECT) {
      t4(v1, o1, v2, o2, val * (sg * 0.5));
      t4(v2, o2, v1, o1, val * (sg * 0.5));
    } else {
      rdm_add(S.os, idx4(v1, o1, v2, o2, n), val * sg);
    }
  } else if(ca == 2 || cb == 2) {  // rdm_contributions_2, :43-66
    const bool a = ca == 2;
    const uint32_t e = a ? single_ex(ba, ka) : single_ex(bb, kb);
    const int o1 = ex_o1(e), v1 = ex_v1(e);
    const double v = ex_sgn(e) * val;
    rdm_add(ordm, size_t(v1) + size_t(n) * o1, v);
    if(two) {
      for(Spin<NSW> s = a ? ba : bb; sp_popc(s);) {
        const int p = sp_lowest(s);
        s = sp_flip(s, p);
        if constexpr(DIRECT) {
          t4(v1, o1, p, p, 0.5 * v);
          t4(p, p, v1, o1, 0.5 * v);
          t4(v1, p, p, o1, -0.5 * v);
          t4(p, o1, v1, p, -0.5 * v);
        } else {
          rdm_add(S.ss1, at(v1, o1, p), v);
        }
      }
      for(Spin<NSW> s = a ? bb : ba; sp_popc(s);) {
        const int p = sp_lowest(s);
        s = sp_flip(s, p);
        if constexpr(DIRECT) {
          t4(v1, o1, p, p, 0.5 * v);
          t4(p, p, v1, o1, 0.5 * v);
        } else {
          rdm_add(S.os1, at(v1, o1, p), v);
        }
      }
    }
  } else {
    return true;  // rdm_contributions_diag, :68-99
  }
  return false;
}

// form_rdms (double_loop.hpp:117-165) over one determinant list: every
// (bra, ket) pair within four spin-orbital differences with |C_i C_j| >
// 1e-16 adds its contributions. One warp per bra row; the pairs come from
// the general build's enumeration; sums are atomic (order not fixed). The
// contributions of the diagonal branch depend on the bra alone: their sum
// per row goes to S.diag.
template <int NBITS, bool DIRECT, bool MIXED>
__global__ void __launch_bounds__(HB_THREADS)
    rdm_k(GenData g, const uint64_t* dets, int64_t n, const double* C,
          int norb, double* ordm, int two, RdmSums S, unsigned* ctr) {
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  __shared__ __align__(16) uint8_t s_scr[HB_WARPS][GEN_SCRATCH];
  uint8_t* ov = s_scr[threadIdx.x >> 5];
  for(int64_t row; (row = next_row(ctr)) < n;) {
    const int32_t rg = g.rowgroup[row];
    double dsum = 0.0;
    if(rg >= 0) {
      const uint64_t* bd = dets + row * D::NW;
      const Spin<NSW> ba = D::alpha(bd), bb = D::beta(bd);
      const double ci = C[row];
      gen_pairs<MIXED>(g, rg, ba, bb, ov, reinterpret_cast<uint32_t*>(ov + 256),
                     [&](bool act, int64_t m, bool) {
        if(!act) return;
        const double val = ci * C[g.sidx[m]];
        if(!(fabs(val) > 1e-16)) return;
        if(rdm_pair<DIRECT, MIXED>(ba, bb, ld_spin<NSW>(g.salpha, m),
                                   ld_spin<NSW>(g.sbeta, m), val, norb, ordm,
                                   two != 0, S))
          dsum += val;
      });
#pragma unroll
      for(int o = 16; o > 0; o >>= 1)
        dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
    }
    if((threadIdx.x & 31) == 0) S.diag[row] = dsum;
  }
}

// Diagonal branch: the rows' sums over the pairs of orbitals occupied in
// them. A block takes DG_ROWS rows and a pair of orbitals a thread, and adds
// one partial sum per pair: atomics per orbital pair and block, not per row
// (every row adds to the pairs of the deepest orbitals). With all pairs in one
// block, 300 determinants of 100 orbitals had 3 blocks for 10,000 pairs.
constexpr int DG_ROWS = 128;
constexpr int DG_THREADS = 256;
template <int NBITS, bool DIRECT>
__global__ void rdm_diag_k(const uint64_t* dets, int64_t n, const double* w,
                           int norb, double* ordm, int two, RdmSums S) {
  using D = DetTraits<NBITS>;
  constexpr int NSW = D::NSW;
  __shared__ uint64_t sd[DG_ROWS * D::NW];
  __shared__ double sw[DG_ROWS];
  const int64_t r0 = int64_t(blockIdx.x) * DG_ROWS;
  const int nr = int(n - r0 < DG_ROWS ? n - r0 : DG_ROWS);
  for(int i = threadIdx.x; i < nr * D::NW; i += blockDim.x)
    sd[i] = dets[r0 * D::NW + i];
  for(int i = threadIdx.x; i < nr; i += blockDim.x) sw[i] = w[r0 + i];
  __syncthreads();
  const int npair = two ? norb * norb : norb;
  const int x = blockIdx.y * blockDim.x + threadIdx.x;
  if(x < npair) {
    const int p = two ? x % norb : x, q = two ? x / norb : x;
    double one = 0.0, ss = 0.0, os = 0.0;
    for(int r = 0; r < nr; ++r) {
      const double v = sw[r];
      const Spin<NSW> a = D::alpha(sd + r * D::NW), b = D::beta(sd + r * D::NW);
      const int ap = sp_test(a, p), bp = sp_test(b, p);
      const int aq = sp_test(a, q), bq = sp_test(b, q);
      if(p == q) one += double(ap + bp) * v;
      ss += double((ap & aq) + (bp & bq)) * v;
      if(ap & bq) os += v;
    }
    if(p == q && one != 0.0) rdm_add(ordm, size_t(p) * (norb + 1), one);
    if(DIRECT && two) {
      const double same = 0.5 * ss, opp = 0.5 * os;
      if(ss != 0.0) rdm_add(S.trdm, idx4(p, q, p, q, norb), -same);
      if(ss != 0.0 || os != 0.0)
        rdm_add(S.trdm, idx4(p, p, q, q, norb), same + opp);
      if(os != 0.0) rdm_add(S.trdm, idx4(q, q, p, p, norb), opp);
    } else if(two) {
      if(ss != 0.0) rdm_add(S.dss, size_t(x), ss);
      if(os != 0.0) rdm_add(S.dos, size_t(x), os);
    }
  }
}

// trdm += the elements formed from the sums (rdms.hpp:15-99 gathered by
// target element instead of scattered by pair).
__global__ void rdm_expand_k(RdmSums S, int n, double* trdm) {
  const size_t n2 = size_t(n) * n, n4 = n2 * n2;
  for(size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < n4;
      x += size_t(gridDim.x) * blockDim.x) {
    const int p = int(x % n), q = int(x / n % n), r = int(x / n2 % n),
              s = int(x / n2 / n);
    auto a4 = [n](int i, int j, int k, int l) { return idx4(i, j, k, l, n); };
    auto a3 = [n](int i, int j, int k) { return size_t(i) + size_t(n) * (j + size_t(n) * k); };
    double v = S.os[x] + S.os[a4(r, s, p, q)];
    v += S.ss[x] + S.ss[a4(r, s, p, q)] - S.ss[a4(r, q, p, s)] - S.ss[a4(p, s, r, q)];
    if(r == s) v += S.ss1[a3(p, q, r)] + S.os1[a3(p, q, r)];
    if(p == q) v += S.ss1[a3(r, s, p)] + S.os1[a3(r, s, p)];
    if(q == r) v -= S.ss1[a3(p, s, q)];
    if(p == s) v -= S.ss1[a3(r, q, p)];
    if(p == q && r == s)
      v += S.dss[p + n * r] + S.dos[p + n * r] + S.dos[r + n * p];
    if(p == r && q == s) v -= S.dss[p + n * q];
    trdm[x] += 0.5 * v;
  }
}

// ordm (n^2) and trdm (n^4, may be null) are device arrays the results are
// added to; dets and C device arrays of length n.
void form_rdms_device(macis_b200_ham* h, const uint64_t* dets, size_t n,
                      const double* C, double* ordm, double* trdm) {
  if(n == 0) return;
  MB_REQUIRE(n < (size_t(1) << 31), MACIS_B200_ECAPACITY,
             "RDMs need < 2^31 determinants");
  cudaStream_t s = h->stream;
  Arena A(s);
  const unsigned gr = grid_for(n, HB_WARPS, size_t(num_sms()) * 16);
  unsigned* ctr = A.get<unsigned>(1);
  MB_CUDA(cudaMemsetAsync(ctr, 0, sizeof(unsigned), s));
  const size_t n1 = size_t(h->norb), n3 = n1 * n1 * n1, n4 = n3 * n1;
  RdmSums S{};
  S.trdm = trdm;
  S.diag = A.get<double>(n);
  const int two = trdm ? 1 : 0;
  const dim3 gd(grid_for(n, DG_ROWS),
                grid_for(two ? n1 * n1 : n1, DG_THREADS));
  // Without the memory for the sums, or for the plan beside them, the pairs go
  // straight to the 2-RDM; so do those of short lists, where the passes over
  // the sums cost more than the additions that they save. Selected lists of
  // norb^2 / 20, 4 norb^2 and 16 norb^2 determinants, sums / straight: n = 24
  // 0.36 / 0.32, 0.40 / 0.39, 0.53 / 0.55 ms; n = 48 0.44 / 0.33, 0.73 / 0.65,
  // 1.47 / 1.72; n = 100 2.58 / 0.41, 6.5 / 4.6, 22.9 / 22.7. CAS spaces (more
  // pairs a determinant) lie above the line: CAS(9,8) 0.81 / 1.32 ms.
  auto sums = [&] {
    const size_t tot = 2 * n4 + 2 * n3 + 2 * n1 * n1;
    if(!trdm || n <= 4 * n1 * n1) return false;
    try {
      S.os = A.get<double>(tot);
    } catch(const Error& e) {
      if(e.code != MACIS_B200_ENOMEM) throw;
      cudaGetLastError();  // the allocation's
      return false;
    }
    MB_CUDA(cudaMemsetAsync(S.os, 0, tot * 8, s));
    S.ss = S.os + n4;
    S.ss1 = S.ss + n4;
    S.os1 = S.ss1 + n3;
    S.dss = S.os1 + n3;
    S.dos = S.dss + n1 * n1;
    return true;
  };
#define MB_RDM_RUN(NB, DIRECT)                                               \
  (g.mixed ? rdm_k<NB, DIRECT, true> : rdm_k<NB, DIRECT, false>)             \
      <<<gr, HB_THREADS, 0, s>>>(g, dets, int64_t(n), C, h->norb, ordm, two, \
                                 S, ctr),                                    \
      note_launch();                                                         \
  rdm_diag_k<NB, DIRECT><<<gd, DG_THREADS, 0, s>>>(                          \
      dets, int64_t(n), S.diag, h->norb, ordm, two, S),                      \
      note_launch();
#define MB_RDM(NB)                                                           \
  {                                                                          \
    const GenData g = gen_plan<NB>(h, dets, n, dets, n, true, 0, P);         \
    if(S.os || !trdm) {                                                      \
      MB_RDM_RUN(NB, false)                                                  \
    } else {                                                                 \
      MB_RDM_RUN(NB, true)                                                   \
    }                                                                        \
  }
  auto run = [&] {
    Arena P(s);
    if(h->nbits == 64) {
      MB_RDM(64)
    } else if(h->nbits == 128) {
      MB_RDM(128)
    } else {
      MB_RDM(256)
    }
  };
  if(!sums()) {
    run();
  } else {
    try {
      run();
    } catch(const Error& e) {  // the plan: nothing is added yet
      if(e.code != MACIS_B200_ENOMEM) throw;
      cudaGetLastError();
      A.release(S.os);
      S.os = nullptr;
      run();
    }
  }
  if(S.os)
    rdm_expand_k<<<grid_for(n4, 256, 16 * num_sms()), 256, 0, s>>>(
        S, h->norb, trdm), note_launch();
#undef MB_RDM_RUN
#undef MB_RDM
  MB_CUDA(cudaGetLastError());
  MB_CUDA(cudaStreamSynchronize(s));
}

}  // namespace mb
