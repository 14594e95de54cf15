// Grouping of the ASCI search's raw contributions by determinant, without
// sorting them: a search only needs the contributions to one determinant next
// to each other, in generation order (so that they are summed as the
// reference sums them), not the determinants in order.
//
// The records are partitioned by up to four stable 8-bit digit passes over a
// 32-bit hash of the key, enough digits that a bucket of equal hash holds about
// 20 records at most, and one pass over the partitioned records finds the
// records of each key in their bucket and sums their scores. A full sort of
// the keys needs a pass for every byte in which they vary: 6 to 7 for number
// keys, 12 to 26 for determinants.
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

// One-word keys are stored mixed by a bijection, so that their hash is their
// upper half and a digit pass forms no hash.
__host__ __device__ __forceinline__ uint64_t mix_key(uint64_t k) {
  k *= 0x9E3779B97F4A7C15ull;
  k ^= k >> 32;
  return k * 0xD6E8FEB86659FD93ull;
}
constexpr uint64_t odd_inverse(uint64_t a) {  // Newton: 5 bits, doubled 4 times
  uint64_t x = (3 * a) ^ 2;
  for(int i = 0; i < 4; ++i) x *= 2 - a * x;
  return x;
}
__host__ __device__ __forceinline__ uint64_t unmix_key(uint64_t k) {
  constexpr uint64_t i1 = odd_inverse(0x9E3779B97F4A7C15ull),
                     i2 = odd_inverse(0xD6E8FEB86659FD93ull);
  k *= i2;
  k ^= k >> 32;
  return k * i1;
}

// The hash of a record's key; MIXED: the key is a mixed word.
template <int NW, bool MIXED>
__device__ __forceinline__ uint32_t rec_hash(const Key<NW>& k) {
  if constexpr(MIXED)
    return uint32_t(k.w[0] >> 32);
  else
    return key_hash<NW>(k);
}

template <int NW, bool MIXED>
struct HashDigit {  // the byte of the key's hash at bit `shift`
  int shift;
  __device__ __forceinline__ unsigned operator()(const Key<NW>& k) const {
    return (rec_hash<NW, MIXED>(k) >> shift) & 255u;
  }
};

// Hash digits for n records: 20 per bucket at most, of which a window of 32
// still ends a whole bucket. A digit pass moves every record once (9.3 ms of
// 1e9 16-byte records, 10.6 when the line was drawn: for 2.9e8 records a
// fourth pass then took 3.1 ms and their sums 4.0 in place of 6.5 ms); fuller
// buckets are read one key after another.
inline int group_digits(size_t n) {
  int np = 1;
  while(np < 4 && (n >> (8 * np)) > 20) ++np;
  return np;
}

constexpr int GS_THREADS = 128;
constexpr int GS_WARPS = GS_THREADS / 32;
template <int NW>
struct GroupTile {  // 18 to 20 KB of keys and scores for the four warps
  static constexpr int IPT = NW == 1 ? 8 : NW == 2 ? 5 : 3;
  static constexpr int N = 32 * IPT;   // records per warp
  static constexpr int SPAN = N + 32;  // with those a last bucket may go on in
};

// Counters of a grouping pass.
struct GroupCounts {
  unsigned long long out;      // candidates written
  unsigned long long unique;   // distinct keys
  unsigned long long scored;   // of these with a nonzero |sum| >= tcut
  unsigned long long pruned;   // of those with |sum| > ptol
};

// For the buckets of the partitioned (keys, rv, n) that begin in [0, n1): the
// scores of each distinct key are summed in order. Sums that are nonzero and
// whose |sum| bits are at least max(tcut, tout) are appended to (okeys, osum),
// in no fixed order. sh: shift of the bucket hash. One read of the records
// and, with a threshold, next to no writes: with a full sort, the flag, scan,
// start and sum passes over it, and the core filter, compaction and selection
// over the 1.6e9 sums they left, the sort and merge phases of the n = 48 search
// of 2.7e9 contributions took 311 + 90 ms; with this 163 + 1 ms.
//
// A warp stages a tile and goes through it 32 records at a time, each time
// from the start of a bucket to the end of the last whole one in the window:
// the records of a key are then lanes that match, and their sum is a shuffle
// per record. 2.7e9 records with 1.6e9 keys: 33.4 ms, 1.1e9 with 1.05e9: 9.2.
// A thread per record, comparing with its neighbours until its bucket ends,
// took 57.8 and 11.8 ms, for a warp waits for the lane with the longest bucket;
// matching the buckets of one record too, 38.7 and 18.3. What bounds it is the
// latency of match and shuffles; more resident blocks (10 or 12 for 7) made it
// 10 to 25 % slower. Buckets longer than a window are read from memory by the
// whole warp, one distinct key after another.
template <int NW, bool MIXED>
__global__ void __launch_bounds__(GS_THREADS)
    group_sum_k(const uint64_t* __restrict__ keys,
                const double* __restrict__ rv, size_t n, size_t n1, int sh,
                uint64_t tcut, uint64_t tout, double ptol,
                uint64_t* __restrict__ okeys, double* __restrict__ osum,
                GroupCounts* cnt) {
  constexpr unsigned ALL = 0xffffffffu;
  constexpr int TILE = GroupTile<NW>::N, SPAN = GroupTile<NW>::SPAN;
  __shared__ uint64_t s_key[GS_WARPS][NW][SPAN];
  __shared__ double s_rv[GS_WARPS][SPAN];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t (*sk)[SPAN] = s_key[wid];
  double* sv = s_rv[wid];
  const uint64_t tmin = tcut > tout ? tcut : tout;
  uint32_t nuniq = 0, nscored = 0, npruned = 0;
  auto bucket = [&](const Key<NW>& k) { return rec_hash<NW, MIXED>(k) >> sh; };
  auto accept = [&](double a) {  // a finished sum: is it to be written?
    ++nuniq;
    const double m = fabs(a);
    const uint64_t bits = uint64_t(__double_as_longlong(m));
    if(!(-m < 0.0) || bits < tcut) return false;  // zero or NaN, or too small
    ++nscored;
    npruned += m > ptol;
    return bits >= tmin;
  };
  // the lanes of a window that hold the lane's key
  auto match = [&](const Key<NW>& k) {
    unsigned p = ALL;
#pragma unroll
    for(int w = 0; w < NW; ++w)
      p &= __match_any_sync(ALL, (unsigned long long)k.w[w]);
    return p;
  };
  for(size_t t0 = (size_t(blockIdx.x) * GS_WARPS + wid) * TILE; t0 < n1;
      t0 += size_t(gridDim.x) * GS_WARPS * TILE) {
    const int ny = int(n - t0 < size_t(SPAN) ? n - t0 : size_t(SPAN));
    const int nt = int(n1 - t0 < size_t(TILE) ? n1 - t0 : size_t(TILE));
    uint32_t b0 = 0;  // the bucket before the tile
    if(t0 > 0) b0 = bucket(load_key<NW>(keys, t0 - 1));
    {
      Key<NW> k[SPAN / 32];
      double v[SPAN / 32];
#pragma unroll
      for(int u = 0; u < SPAN / 32; ++u) {
        const int y = 32 * u + lane;
        if(y < ny) {
          k[u] = load_key<NW>(keys, t0 + y);
          v[u] = rv[t0 + y];
        }
      }
#pragma unroll
      for(int u = 0; u < SPAN / 32; ++u) {
        const int y = 32 * u + lane;
        if(y < ny) {
#pragma unroll
          for(int w = 0; w < NW; ++w) sk[w][y] = k[u].w[w];
          sv[y] = v[u];
        }
      }
    }
    __syncwarp();
    auto staged = [&](int y) {
      Key<NW> k;
#pragma unroll
      for(int w = 0; w < NW; ++w) k.w[w] = sk[w][y];
      return k;
    };
    int x = 0;  // records done
    while(t0 > 0 && x < nt) {  // those of a bucket of an earlier tile
      const int y = x + lane;
      const unsigned other =
          __ballot_sync(ALL, y >= ny || bucket(staged(y)) != b0);
      if(other) {
        x += __ffs(other) - 1;
        break;
      }
      x += 32;
    }
    int kept = 0;  // sums to be written, in place of records that are done
    while(x < nt) {
      const int y = x + lane;
      const bool in = y < ny;
      Key<NW> k{};
      double v = 0.0;
      if(in) {
        k = staged(y);
        v = sv[y];
      }
      const uint32_t b = bucket(k);
      const uint32_t bp = __shfl_up_sync(ALL, b, 1);
      // lanes at which a bucket begins (lane 0 does; the end of the records
      // counts too), and the end of the whole buckets that begin in the tile
      const unsigned starts =
          __ballot_sync(ALL, in ? lane == 0 || b != bp : t0 + y >= n);
      const unsigned beyond = nt - x < 32 ? starts >> (nt - x) << (nt - x) : 0u;
      const int e = beyond ? __ffs(beyond) - 1 : 31 - __clz(starts);
      if(e == 0) {
        const size_t g0 = t0 + x;
        const uint32_t bg = __shfl_sync(ALL, b, 0);
        Key<NW> kg;  // the bucket's first key
#pragma unroll
        for(int w = 0; w < NW; ++w)
          kg.w[w] = __shfl_sync(ALL, (unsigned long long)k.w[w], 0);
        // lane's record from position p on: is it in the bucket?
        auto fetch = [&](size_t p, Key<NW>& q, double& s) {
          q = Key<NW>{};
          s = 0.0;
          if(p + lane >= n) return false;
          q = load_key<NW>(keys, p + lane);
          s = rv[p + lane];
          return bucket(q) == bg;
        };
        size_t end = 0;  // of the bucket
        for(size_t c = g0; !end; c += 32) {
          Key<NW> q;
          double s;
          const unsigned mi = __ballot_sync(ALL, fetch(c, q, s));
          if(mi != ALL) end = c + __popc(mi);
          const unsigned pq = match(q) & mi;
          const bool lead = (mi >> lane & 1) && !(pq & lanemask_lt()) &&
                            !(c > g0 && key_eq<NW>(q, kg));
          for(unsigned m = __ballot_sync(ALL, lead); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            Key<NW> kk;
#pragma unroll
            for(int w = 0; w < NW; ++w)
              kk.w[w] = __shfl_sync(ALL, (unsigned long long)q.w[w], src);
            bool seen = false;  // in an earlier window of the bucket
            for(size_t p = c; p > g0 && !seen; p -= 32)
              seen = __any_sync(
                  ALL, key_eq<NW>(load_key<NW>(keys, p - 32 + lane), kk));
            if(seen) continue;
            double a = __shfl_sync(ALL, s, src);
            unsigned me = __shfl_sync(ALL, pq, src);
            for(me &= me - 1; me; me &= me - 1)
              a += __shfl_sync(ALL, s, __ffs(me) - 1);
            for(size_t p = c + 32; !end || p < end; p += 32) {
              Key<NW> qn;
              double sn;
              const bool inb = fetch(p, qn, sn);
              const unsigned mb = __ballot_sync(ALL, inb);
              me = __ballot_sync(ALL, inb && key_eq<NW>(qn, kk));
              if(me == ALL) {
#pragma unroll
                for(int l = 0; l < 32; ++l) a += __shfl_sync(ALL, sn, l);
              } else {
                for(; me; me &= me - 1)
                  a += __shfl_sync(ALL, sn, __ffs(me) - 1);
              }
              if(mb != ALL) break;
            }
            if(lane == src && accept(a)) {
              const size_t o = size_t(atomicAdd(&cnt->out, 1ull));
              store_key<NW>(okeys, o, q);
              osum[o] = a;
            }
          }
        }
        x = end - t0 < size_t(nt) ? int(end - t0) : nt;
        continue;
      }
      // buckets of one record are left out of the match: its time grows with
      // the number of different values
      const bool alone = (starts >> lane & 1) && (starts >> lane >> 1 & 1);
      const unsigned some = __ballot_sync(ALL, lane < e && !alone);
      unsigned peers = 1u << lane;
      if(some) {
        Key<NW> q{};
        if(some >> lane & 1) q = k;
        const unsigned p = match(q);
        if(some >> lane & 1) peers = p & some;
      }
      const bool first = lane < e && !(peers & lanemask_lt());
      unsigned rest = first ? peers & (peers - 1) : 0u;
      double a = v;
      while(__any_sync(ALL, rest)) {
#pragma unroll
        for(int u = 0; u < 2; ++u) {
          const double t = __shfl_sync(ALL, v, rest ? __ffs(rest) - 1 : lane);
          if(rest) a += t;
          rest &= rest - 1;
        }
      }
      const bool take = first && accept(a);
      const unsigned tm = __ballot_sync(ALL, take);
      if(tm) {
        __syncwarp();  // the window has been read
        if(take) {
          const int o = kept + __popc(tm & lanemask_lt());
#pragma unroll
          for(int w = 0; w < NW; ++w) sk[w][o] = k.w[w];
          sv[o] = a;
        }
        kept += __popc(tm);
      }
      x += e;
    }
    if(kept) {
      __syncwarp();
      unsigned long long o0 = 0;
      if(lane == 0) o0 = atomicAdd(&cnt->out, (unsigned long long)kept);
      o0 = __shfl_sync(ALL, o0, 0);
      for(int j = lane; j < kept; j += 32) {
        store_key<NW>(okeys, size_t(o0) + j, staged(j));
        osum[size_t(o0) + j] = sv[j];
      }
    }
    __syncwarp();  // the staged records are rewritten
  }
  nuniq = __reduce_add_sync(ALL, nuniq);
  nscored = __reduce_add_sync(ALL, nscored);
  npruned = __reduce_add_sync(ALL, npruned);
  if(lane == 0) {
    atomicAdd(&cnt->unique, (unsigned long long)nuniq);
    atomicAdd(&cnt->scored, (unsigned long long)nscored);
    atomicAdd(&cnt->pruned, (unsigned long long)npruned);
  }
}

// How many distinct keys of the sorted list core (nc entries) are among the
// scored / pruned keys of the partitioned records (subtracted from the
// counts of group_sum_k: core determinants are no candidates).
template <int NW, bool MIXED>
__global__ void group_core_k(const uint64_t* keys, const double* rv, size_t n,
                             int sh, uint64_t tcut, double ptol,
                             const uint64_t* core, size_t nc,
                             GroupCounts* cnt) {
  for(size_t c = size_t(blockIdx.x) * blockDim.x + threadIdx.x; c < nc;
      c += size_t(gridDim.x) * blockDim.x) {
    Key<NW> k = load_key<NW>(core, c);
    if(c > 0 && key_eq<NW>(load_key<NW>(core, c - 1), k)) continue;
    if constexpr(MIXED) k.w[0] = mix_key(k.w[0]);
    const uint32_t h = rec_hash<NW, MIXED>(k) >> sh;
    size_t lo = 0, hi = n;  // first record of the bucket
    while(lo < hi) {
      const size_t mid = (lo + hi) >> 1;
      if((rec_hash<NW, MIXED>(load_key<NW>(keys, mid)) >> sh) < h)
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
      } else if((rec_hash<NW, MIXED>(q) >> sh) != h) {
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
