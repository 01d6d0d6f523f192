// small_kernels.cuh -- a whole solve of at most kSmallMaxN people in one
// launch of one CTA.
//
// Such a solve is all latency: five launches, two resets, nine event records
// and two copies around about 20 us of work.  Here everything is in shared
// memory: her rank of him takes a byte, and so does a woman, so a man's list is
// n 2-byte words (woman << 8 | her rank of him), and a chain's step is a
// handful of shared reads.  The outcome goes straight into the caller's match
// and the host's (pinned) control block.
//   It decides what the precheck and the modes of the larger solves decide --
// distinct first choices, the mode that would have served, whether the men
// share one list -- and refuses what they refuse: women's rows that are no
// permutations, entries of the men's lists out of range, a man rejected by
// every woman; where all first choices are distinct only those are read.
//
// n = 97 uniform, from call to return: 136 -> 61 us.
//   Men who share one list would make all n (n + 1) / 2 proposals, and where the
// women share one too, all of them displace someone.  One warp takes the women
// in the list's order instead: each has the best man whom no woman before her
// has (the only stable matching there is).
#pragma once

#include "common.cuh"
#include "solve_kernels.cuh"

namespace smpb200 {

constexpr int kSmallMaxN = 256;

// Shared memory: list words and ranks (n n each), one seen-bit per pair, the
// women's words and the men's positions.
__host__ __device__ constexpr size_t small_smem(int n) {
  const size_t n2 = static_cast<size_t>(n) * n;
  return ((n2 * 2 + 15) & ~static_cast<size_t>(15)) + ((n2 + 15) & ~static_cast<size_t>(15)) +
         static_cast<size_t>(n) * (4 * 8 + 4 + 2) + 16;
}

__global__ void __launch_bounds__(1024, 1) k_small(const int32_t *__restrict__ pref_m,
                                                   const int32_t *__restrict__ pref_w, int n, int K,
                                                   int allow_perfect, int32_t *match, int32_t *also, Control *out,
                                                   int first_man) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const size_t n2 = static_cast<size_t>(n) * n;
  uint16_t *list = reinterpret_cast<uint16_t *>(smem_raw);
  unsigned char *rank = smem_raw + ((n2 * 2 + 15) & ~static_cast<size_t>(15));
  uint32_t *seen = reinterpret_cast<uint32_t *>(rank + ((n2 + 15) & ~static_cast<size_t>(15)));  // [n][8]
  uint32_t *word = seen + 8 * n;  // rank << 16 | man, all ones = free
  uint16_t *spos = reinterpret_cast<uint16_t *>(word + n);
  __shared__ int s_distinct, s_differ, s_status, s_bad, s_next, s_deep, s_late;
  __shared__ unsigned int s_hops;
  __shared__ uint32_t s_row0[kSmallMaxN / 32];  // women the first man's list has named
  __shared__ unsigned long long s_props;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const auto refuse = [&](int v) {
    if (atomicCAS(&s_status, 0, kStatusInvalidInput) == 0) s_bad = v;
  };
  if (tid == 0) {
    s_distinct = s_differ = s_status = s_bad = s_next = s_deep = s_late = 0;
    s_hops = 0;
    s_props = 0;
  }
  if (tid < kSmallMaxN / 32) s_row0[tid] = 0;
  for (int i = tid; i < 8 * n; i += 1024) seen[i] = 0;
  for (int i = tid; i < n; i += 1024) {
    word[i] = 0xFFFFFFFFu;
    spos[i] = 0;
  }
  __syncthreads();
  int first = -1;
  if (tid < n) {
    first = __ldg(pref_m + static_cast<size_t>(tid) * n);
    if (static_cast<unsigned>(first) >= static_cast<unsigned>(n))
      refuse(first);
    else if (atomicExch(word + first, 0u) == 0xFFFFFFFFu)
      atomicAdd(&s_distinct, 1);
  }
  __syncthreads();
  const int distinct = s_distinct;
  const bool perfect = allow_perfect && distinct == n && s_status == 0;
  const int mode = 4 * distinct >= n ? kModeQuery : kModeRank;
  if (perfect) {
    if (tid < n) {
      match[tid] = first;
      if (also) also[tid] = first;
    }
  } else {
    const int total = static_cast<int>(n2);
    for (int i = tid; i < n; i += 1024) word[i] = 0xFFFFFFFFu;
    for (int t = tid; t < total; t += 1024) {
      const int w = t / n, r = t - w * n;
      const int m = __ldg(pref_w + t);
      if (static_cast<unsigned>(m) >= static_cast<unsigned>(n)) {
        refuse(m);
      } else {
        const uint32_t bit = 1u << (m & 31);
        if (atomicOr(seen + 8 * w + (m >> 5), bit) & bit) refuse(m);  // named twice
        rank[w * n + m] = static_cast<unsigned char>(r);
      }
    }
    __syncthreads();
    bool differ = false;
    for (int t = tid; t < total; t += 1024) {
      const int m = t / n, r = t - m * n;
      const int w = __ldg(pref_m + t);
      differ |= distinct == 1 && w != __ldg(pref_m + r);
      if (static_cast<unsigned>(w) >= static_cast<unsigned>(n)) {
        // beyond the prefix of a query-mode solve it counts only if a man's
        // proposals go there (the rank mode that starts over refuses it)
        if (mode == kModeQuery && r >= K)
          s_late = 1;
        else
          refuse(w);
        list[t] = 0;
      } else {
        const uint32_t bit = 1u << (w & 31);
        if (m == 0 && distinct == 1 && mode == kModeRank && (atomicOr(s_row0 + (w >> 5), bit) & bit)) {
          if (first_man) refuse(w);
          differ = true;  // no list to share
        }
        list[t] = static_cast<uint16_t>((w << 8) | rank[w * n + m]);
      }
    }
    if (differ) s_differ = 1;
    // (all warps or none: one that refuses a man in the chains must not keep lanes
    // of a later one out)
    const bool refused = __syncthreads_or(s_status != 0);
    const bool shared = mode == kModeRank && distinct == 1 && n >= 2 && !s_differ;
    if (!refused && shared) {
      if (tid < 32) {
        // a lane keeps men lane, 32 + lane, ...; the next woman's ranks of them are
        // loaded while this one's best is found
        constexpr int kMen = kSmallMaxN / 32;
        uint32_t gone[kMen], r[kMen], next[kMen];  // gone: all ones once taken
        const auto load = [&](int w, uint32_t (&to)[kMen]) {
#pragma unroll
          for (int j = 0; j < kMen; ++j)
            to[j] = lane + 32 * j < n ? (static_cast<uint32_t>(rank[w * n + lane + 32 * j]) << 16) | (lane + 32 * j) : 0u;
        };
#pragma unroll
        for (int j = 0; j < kMen; ++j) gone[j] = lane + 32 * j < n ? 0u : 0xFFFFFFFFu;
        int w = list[0] >> 8, after = list[min(1, n - 1)] >> 8;
        load(w, r);
        for (int k = 0; k < n; ++k) {
          load(after, next);
          const int w2 = after;
          after = list[min(k + 2, n - 1)] >> 8;
          uint32_t best = 0xFFFFFFFFu;
#pragma unroll
          for (int j = 0; j < kMen; ++j) best = min(best, r[j] | gone[j]);
          best = __reduce_min_sync(kFullMask, best);
          const int m = static_cast<int>(best & 0xFFFFu);
#pragma unroll
          for (int j = 0; j < kMen; ++j) gone[j] |= m == lane + 32 * j ? 0xFFFFFFFFu : 0u;
          if (lane == 0) {
            word[w] = best;  // (a woman the list names twice leaves another free: refused below)
            spos[m] = static_cast<uint16_t>(k);
          }
          w = w2;
#pragma unroll
          for (int j = 0; j < kMen; ++j) r[j] = next[j];
        }
      }
    } else if (!refused) {  // the chains: a warp each, 32 choices at a time
      unsigned int hops = 0;
      int m = -1, pos = 0;
      for (;;) {
        if (m < 0) {
          int i = 0;
          if (lane == 0) i = atomicAdd(&s_next, 1);
          m = __shfl_sync(kFullMask, i, 0);
          if (m >= n) break;
          pos = 0;
        }
        if (pos >= n) {  // rejected by every woman: his list is no permutation
          if (lane == 0) refuse(m);
          break;
        }
        const int r = pos + lane;
        const uint32_t e = r < n ? list[m * n + r] : 0u;
        const uint32_t cur = r < n ? lds_relaxed_u32(word + (e >> 8)) : 0u;
        const unsigned hit = __ballot_sync(kFullMask, (e & 0xFFu) < (cur >> 16));
        if (!hit) {
          pos += 32;
          continue;
        }
        const int j = __ffs(hit) - 1;
        uint32_t old = 0;
        if (lane == j) {
          spos[m] = static_cast<uint16_t>(r);
          old = atom_min_relaxed_shared(word + (e >> 8), ((e & 0xFFu) << 16) | static_cast<uint32_t>(m));
          if ((old >> 16) <= (e & 0xFFu)) old = 0;  // someone better got there first
        }
        old = __shfl_sync(kFullMask, old, j);
        if (old == 0) {
          // (an accepted proposal displaces a rank above his, or nobody)
          pos += j;
          continue;
        }
        hops++;
        m = old == 0xFFFFFFFFu ? -1 : static_cast<int>(old & 0xFFFFu);
        if (m >= 0) pos = spos[m] + 1;
      }
      if (lane == 0 && hops) atomicAdd(&s_hops, hops);
    }
    __syncthreads();
    if (!s_status && tid < n) {
      const uint32_t v = word[tid];
      if (v == 0xFFFFFFFFu) {
        refuse(tid);
      } else {
        match[v & 0xFFFFu] = tid;
        if (also) also[v & 0xFFFFu] = tid;
      }
      atomicAdd(&s_props, spos[tid] + 1ull);
      if (spos[tid] >= K) s_deep = 1;
    }
    __syncthreads();
  }
  if (tid == 0) {
    if (s_late && s_deep) refuse(-1);
    const bool shared = !perfect && mode == kModeRank && distinct == 1 && n >= 2 && !s_differ;
    out->status = s_status;
    out->bad_value = s_bad;
    out->perfect = perfect;
    out->mode = mode;
    out->distinct = distinct;
    out->retry = !perfect && mode == kModeQuery && s_deep;  // the query mode would have started over
    out->swap_out = shared && !s_status;
    out->proposals = perfect ? static_cast<unsigned long long>(n) : s_props;
    out->bulk_proposals = out->proposals;
    out->tail_proposals = 0;
    out->bulk_hops = s_hops;
    out->tail_hops = 0;
    out->tail_men = 0;
    out->tail_done = 0;
    out->round_done = 0;
    out->blocking = 0;
    out->check_proposals = 0;
    __threadfence_system();
  }
}

}  // namespace smpb200
