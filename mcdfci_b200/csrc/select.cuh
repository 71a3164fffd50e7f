// Radix selection of the m largest 64-bit keys held by one CTA, shared by the
// column kernel (a column's candidates) and the leader (the picks).
#pragma once

#include "device_common.cuh"

namespace mcd {

struct SelectScratch {
  alignas(16) unsigned hist[2][256];
  unsigned cnt[32], max[32];
  unsigned bin, in_bin, need;
  unsigned long long few[32], edge;  // the keys of a bin with at most 32
  unsigned n_few, tied;
};

// What to keep of the CTA's keys: all with key >= edge, but of those equal to
// edge only `need` when tied.  total: the keys there are (0 is no key).
struct SelectEdge {
  unsigned long long edge;
  unsigned need, total;
  bool tied;
};

// The key of a score: scores are +0 or positive, so their bit patterns order
// like their values; 0 is left for "none".
__device__ __forceinline__ unsigned long long score_key(double score) {
  return static_cast<unsigned long long>(__double_as_longlong(score)) + 1ull;
}

// `each(f)` calls f(key) for every key of the calling thread.  A pass counts
// the keys by their distance below `ref` in units of 2^lo: first the top 15
// bits (the exponent and three mantissa bits) down from the largest key, with
// all keys 255 or more steps below it in the last bin, then eight bits at a
// time within the bin that holds the want-th largest, until the keys at and
// above a bin are exactly `want`.  One warp scans the histogram: with every
// warp scanning it for itself a pass has one barrier less, but the callers
// are bound by instruction issue (up to eight warps per scheduler).  Called by the whole CTA (at least
// 256 threads), with a barrier since the scratch was last used.
template <class Each>
__device__ __forceinline__ SelectEdge select_edge(SelectScratch& S, unsigned want, Each each) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  unsigned cnt = 0, mx = 0;
  each([&](unsigned long long key) {
    cnt += key != 0ull ? 1u : 0u;
    mx = max(mx, static_cast<unsigned>(key >> 49));
  });
  cnt = __reduce_add_sync(~0u, cnt);
  mx = __reduce_max_sync(~0u, mx);
  if (lane == 0) {
    S.cnt[warp] = cnt;
    S.max[warp] = mx;
  }
  if (tid < 256) S.hist[0][tid] = 0u;
  if (tid == 0) S.n_few = 0u;
  __syncthreads();
  SelectEdge r;
  r.total = __reduce_add_sync(~0u, lane < nw ? S.cnt[lane] : 0u);
  r.edge = 1ull;
  r.need = want;
  r.tied = false;
  if (r.total <= want) return r;
  unsigned long long ref = __reduce_max_sync(~0u, lane < nw ? S.max[lane] : 0u);
  unsigned long long limit = ~0ull;  // distances counted (the first passes: all)
  int lo = 49, buf = 0;
#pragma unroll 1
  while (true) {
    each([&](unsigned long long key) {
      const unsigned long long y = key >> lo, d = ref - y;
      if (key != 0ull && y <= ref && d < limit) atomicAdd(&S.hist[buf][d < 255ull ? static_cast<unsigned>(d) : 255u], 1u);
    });
    if (tid < 256) S.hist[buf ^ 1][tid] = 0u;
    __syncthreads();
    if (warp == 0) {
      // The bin of the need-th largest: lane l holds bins 8l .. 8l+7.
      const uint4 u0 = *reinterpret_cast<const uint4*>(&S.hist[buf][8 * lane]);
      const uint4 u1 = *reinterpret_cast<const uint4*>(&S.hist[buf][8 * lane + 4]);
      const unsigned c[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
      const unsigned t = ((c[0] + c[1]) + (c[2] + c[3])) + ((c[4] + c[5]) + (c[6] + c[7]));
      unsigned run = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(~0u, run, o);
        if (lane >= o) run += v;
      }
      const int src = __ffs(__ballot_sync(~0u, run >= r.need)) - 1;
      if (lane == src) {
        run -= t;
        unsigned bin = 8u * lane, in_bin = c[0];
#pragma unroll
        for (int j = 0; j < 7; ++j) {
          if (run + in_bin < r.need) {
            run += in_bin;
            in_bin = c[j + 1];
            ++bin;
          }
        }
        S.bin = bin;
        S.in_bin = in_bin;
        S.need = r.need - run;
      }
    }
    __syncthreads();
    buf ^= 1;
    const unsigned bin = S.bin, in_bin = S.in_bin;
    r.need = S.need;
    const bool rest = limit == ~0ull && bin == 255u;  // the bin of everything further down
    if (!rest) r.edge = (ref - bin) << lo;
    if (in_bin == r.need) break;
    if (rest) {
      ref -= 255ull;
      continue;
    }
    if (in_bin <= 32u) {
      // Few keys are left to choose from (often an equal pair, which digits
      // would separate last or never): rank them by counting.
      const unsigned long long bin_key = ref - bin;
      each([&](unsigned long long key) {
        if (key != 0ull && (key >> lo) == bin_key) S.few[atomicAdd(&S.n_few, 1u)] = key;
      });
      __syncthreads();
      if (warp == 0) {
        const unsigned long long mine = static_cast<unsigned>(lane) < in_bin ? S.few[lane] : 0ull;
        unsigned above = 0, equal = 0, rank = 0;
#pragma unroll 4
        for (unsigned j = 0; j < in_bin; ++j) {
          const unsigned long long o = S.few[j];
          above += o > mine ? 1u : 0u;
          equal += o == mine ? 1u : 0u;
          rank += o > mine || (o == mine && j < static_cast<unsigned>(lane)) ? 1u : 0u;
        }
        if (static_cast<unsigned>(lane) < in_bin && rank == r.need - 1u) {
          S.edge = mine;
          S.need = r.need - above;
          S.tied = equal > r.need - above ? 1u : 0u;
        }
      }
      __syncthreads();
      r.edge = S.edge;
      r.need = S.need;
      r.tied = S.tied != 0u;
      break;
    }
    if (lo == 0) {
      r.tied = true;
      break;
    }
    const int w = lo < 8 ? lo : 8;
    lo -= w;
    limit = 1ull << w;
    ref = ((ref - bin) << w) | (limit - 1ull);
  }
  if (r.edge == 0ull) r.edge = 1ull;
  return r;
}

}  // namespace mcd
