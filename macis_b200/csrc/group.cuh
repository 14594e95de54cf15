// Grouping of the ASCI search's raw contributions by determinant, without
// sorting them: a search only needs the contributions to one determinant next
// to each other, in generation order (so that they are summed as the
// reference sums them), not the determinants in order.
//
// The records are partitioned by up to four stable 8-bit digit passes over a
// 32-bit hash of the key, enough digits that a bucket of equal hash holds a
// few distinct keys, and one pass over the partitioned records finds for each
// record whether an earlier one of its bucket has its key, and sums the
// others' scores. A full sort of the keys needs a pass for every byte in which
// they vary: 6 to 7 for ranked keys, 12 to 26 for determinants.
#pragma once
#include "primitives.cuh"

namespace mb {

template <int NW>
__device__ __forceinline__ uint32_t key_hash(const Key<NW>& k) {
  uint64_t h = 0;
#pragma unroll
  for(int j = 0; j < NW; ++j) {
    h = (h ^ k.w[j]) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 32;
  }
  return uint32_t((h * 0xD6E8FEB86659FD93ull) >> 32);
}

template <int NW>
struct HashDigit {  // the byte of the key's hash at bit `shift`
  int shift;
  __device__ __forceinline__ unsigned operator()(const Key<NW>& k) const {
    return (key_hash<NW>(k) >> shift) & 255u;
  }
};

// Hash digits for n records: buckets of at most about 8 distinct keys. Each
// digit pass moves every record once; a bucket of m keys costs each record m
// / 2 comparisons with records that are in L1.
inline int group_digits(size_t n) {
  int np = 1;
  while(np < 4 && (n >> (8 * np)) > 8) ++np;
  return np;
}

constexpr int GS_THREADS = 256;
constexpr int GS_IPT = 8;
constexpr int GS_TILE = GS_THREADS * GS_IPT;

// Counters of a grouping pass.
struct GroupCounts {
  unsigned long long out;      // candidates written
  unsigned long long unique;   // distinct keys
  unsigned long long scored;   // of these with a nonzero |sum| >= tcut
  unsigned long long pruned;   // of those with |sum| > ptol
};

// For records [i0, i1) of the partitioned (keys, rv, n): the first record of
// each key sums the key's scores in order. Sums that are nonzero and whose
// |sum| bits are at least max(tcut, tout) are appended to (okeys, osum), in
// no fixed order. sh: shift of the bucket hash. One read of the records and,
// with a threshold, next to no writes: on the n = 48 search of 2.7e9
// contributions the flag, scan, start and sum passes over a full sort, and
// the core filter, compaction and selection over the 1.6e9 sums they left,
// took the sort and merge phases from 228 + 1 to 311 + 90 ms.
template <int NW>
__global__ void __launch_bounds__(GS_THREADS)
    group_sum_k(const uint64_t* __restrict__ keys,
                const double* __restrict__ rv, size_t n, size_t i0, size_t i1,
                int sh, uint64_t tcut, uint64_t tout, double ptol,
                uint64_t* __restrict__ okeys, double* __restrict__ osum,
                GroupCounts* cnt) {
  __shared__ uint32_t scan_sh[GS_THREADS / 32 + 1];
  __shared__ unsigned long long base_sh;
  __shared__ uint32_t tot_sh[3];
  if(threadIdx.x < 3) tot_sh[threadIdx.x] = 0;
  const uint64_t tmin = tcut > tout ? tcut : tout;
  uint32_t nuniq = 0, nscored = 0, npruned = 0;
  for(size_t t0 = i0 + size_t(blockIdx.x) * GS_TILE; t0 < i1;
      t0 += size_t(gridDim.x) * GS_TILE) {
    double sum[GS_IPT];
    unsigned take = 0;
#pragma unroll
    for(int r = 0; r < GS_IPT; ++r) {
      const size_t i = t0 + size_t(r) * GS_THREADS + threadIdx.x;
      sum[r] = 0.0;
      if(i >= i1) continue;
      const Key<NW> k = load_key<NW>(keys, i);
      const uint32_t h = key_hash<NW>(k) >> sh;
      bool head = true;
      for(size_t j = i; j > 0;) {
        const Key<NW> q = load_key<NW>(keys, --j);
        if(key_eq<NW>(q, k)) {
          head = false;
          break;
        }
        if((key_hash<NW>(q) >> sh) != h) break;
      }
      if(!head) continue;
      double a = rv[i];
      for(size_t j = i + 1; j < n; ++j) {
        const Key<NW> q = load_key<NW>(keys, j);
        if(key_eq<NW>(q, k))
          a += rv[j];
        else if((key_hash<NW>(q) >> sh) != h)
          break;
      }
      ++nuniq;
      const double m = fabs(a);
      const uint64_t bits = uint64_t(__double_as_longlong(m));
      if(!(-m < 0.0) || bits < tcut) continue;  // zero or NaN, or too small
      ++nscored;
      npruned += m > ptol;
      if(bits >= tmin) {
        take |= 1u << r;
        sum[r] = a;
      }
    }
    uint32_t total;
    const uint32_t pre =
        block_excl_scan<uint32_t>(uint32_t(__popc(take)), scan_sh, &total);
    if(total) {  // uniform: the block's total
      if(threadIdx.x == 0) base_sh = atomicAdd(&cnt->out, (unsigned long long)total);
      __syncthreads();
      size_t o = size_t(base_sh) + pre;
#pragma unroll
      for(int r = 0; r < GS_IPT; ++r)
        if(take >> r & 1) {
          const size_t i = t0 + size_t(r) * GS_THREADS + threadIdx.x;
          store_key<NW>(okeys, o, load_key<NW>(keys, i));
          osum[o++] = sum[r];
        }
      __syncthreads();  // base_sh is rewritten by the next tile
    }
  }
  __syncthreads();
  atomicAdd(&tot_sh[0], nuniq);
  atomicAdd(&tot_sh[1], nscored);
  atomicAdd(&tot_sh[2], npruned);
  __syncthreads();
  if(threadIdx.x == 0) {
    atomicAdd(&cnt->unique, (unsigned long long)tot_sh[0]);
    atomicAdd(&cnt->scored, (unsigned long long)tot_sh[1]);
    atomicAdd(&cnt->pruned, (unsigned long long)tot_sh[2]);
  }
}

// How many distinct keys of the sorted list core (nc entries) are among the
// scored / pruned keys of the partitioned records (subtracted from the
// counts of group_sum_k: core determinants are no candidates).
template <int NW>
__global__ void group_core_k(const uint64_t* keys, const double* rv, size_t n,
                             int sh, uint64_t tcut, double ptol,
                             const uint64_t* core, size_t nc,
                             GroupCounts* cnt) {
  for(size_t c = size_t(blockIdx.x) * blockDim.x + threadIdx.x; c < nc;
      c += size_t(gridDim.x) * blockDim.x) {
    const Key<NW> k = load_key<NW>(core, c);
    if(c > 0 && key_eq<NW>(load_key<NW>(core, c - 1), k)) continue;
    const uint32_t h = key_hash<NW>(k) >> sh;
    size_t lo = 0, hi = n;  // first record of the bucket
    while(lo < hi) {
      const size_t mid = (lo + hi) >> 1;
      if((key_hash<NW>(load_key<NW>(keys, mid)) >> sh) < h)
        lo = mid + 1;
      else
        hi = mid;
    }
    double a = 0.0;
    bool found = false;
    for(; lo < n; ++lo) {
      const Key<NW> q = load_key<NW>(keys, lo);
      if(key_eq<NW>(q, k)) {
        a = found ? a + rv[lo] : rv[lo];
        found = true;
      } else if((key_hash<NW>(q) >> sh) != h) {
        break;
      }
    }
    const double m = fabs(a);
    if(!found || !(-m < 0.0) || uint64_t(__double_as_longlong(m)) < tcut)
      continue;
    atomicAdd(&cnt->scored, 1ull);
    if(m > ptol) atomicAdd(&cnt->pruned, 1ull);
  }
}

}  // namespace mb
