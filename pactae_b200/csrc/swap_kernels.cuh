// Single solves whose men all share one list: the women propose.
//
// When every man ranks the women in the same order L, the stable matching is
// unique (each woman, taken in L's order, gets her best man not taken by a
// woman before her), so the women-proposing run returns the matching the
// men-proposing Gale-Shapley of the reference returns
// (src/smp/smp_engine_gs_1.cu:47-98).  The men's run would make n(n+1)/2
// proposals -- the man who ends with L[k] proposed to L[0..k] -- and needs the
// full rank matrix; the women's run makes about n ln n proposals and ranks
// every proposer by one inverted row, pos[w] = position of w in L.
//
//   k_swap_pos     pos = inverse of pref_m row 0; row 0 must be a permutation
//   k_swap_screen  every pref_m row equals row 0 (else swap_fail), and every
//                  pref_w row is a permutation (else the invalid-input status)
//   k_swap_gs      the women's proposals, one warp per chain
//   k_swap_rows_check, k_swap_mark_full
//                  host-input solves: the parts of pref_w sent, checked, and
//                  which rows are whole
//   k_swap_match   match[m] from the men's final bids; the men's proposal count
//   k_swap_direct  women who share one list M as well: match[M[k]] = L[k]
//                  (the k-th man of the women's list with the k-th woman of
//                  the men's), no proposals
#pragma once

#include "common.cuh"
#include "solve_kernels.cuh"

namespace smpb200 {

// pos[L[r]] = r, with pos preset to -1; an entry out of range or seen twice
// makes row 0 no permutation: invalid input (refuse), or no list to share.
__global__ void k_swap_pos(const int32_t *__restrict__ pref_m, int32_t *__restrict__ pos, int n, Control *ctrl,
                           int refuse) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    const int w = __ldg(pref_m + r);
    if (static_cast<unsigned>(w) >= static_cast<unsigned>(n) || atomicCAS(pos + w, -1, r) != -1) {
      if (refuse)
        report(ctrl, kStatusInvalidInput, w);
      else
        ctrl->swap_fail = 1;
    }
  }
}

// Rows t = 1 .. n-1 compare pref_m row t with row 0; rows t = n .. 2n-1
// check that pref_w row t-n is a permutation with a shared bitmap.  A solve
// whose men's rows were compared on the host (host-input solves) starts at
// t0 = n: only row 0 of pref_m is then on the device.  Row
// bodies move in 16-byte loads (row_span: rows start off 16-byte boundaries
// when n is not a multiple of 4).  Once a pref_m row differs, the solve
// takes the men's rank-mode pass, which checks pref_w itself: the CTAs stop.
// (One colour byte per man with plain stores and a check pass, instead of the
// bitmap's shared atomics, took 1.85 ms against 1.47 ms at n = 30000.  Where the
// women share one list too, comparing with row 0 instead of marking: 1.96 -> 1.30.)
__host__ __device__ constexpr size_t swap_screen_smem(int n) { return ((static_cast<size_t>(n) + 31) / 32) * 4; }

// Fewer than n / 4 distinct first choices (count_alike).
__device__ __forceinline__ bool women_alike(const Control *ctrl, int n) {
  return 4ll * ld_volatile_s32(&ctrl->distinct_w) < n;
}

// Does this thread's share of row t differ from row 0?  Chunk by chunk where
// both rows start at the same 16-byte offset (all rows when n is a multiple of
// 4), else each chunk against four entries of row 0.
__device__ __forceinline__ bool row_differs(const int32_t *__restrict__ pref, int t, int n) {
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const RowSpan s = row_span(pref, t, n);
  bool differs = false;
  const auto other = [](int4 v, int4 u) { return v.x != u.x || v.y != u.y || v.z != u.z || v.w != u.w; };
  int i = tid;
  if (s.head == row_span(pref, 0, n).head) {
    const int4 *q0 = reinterpret_cast<const int4 *>(pref + s.head);
    for (; i + nthr < s.nq; i += 2 * nthr) {
      const int4 v = __ldcs(s.rq + i);
      const int4 v2 = __ldcs(s.rq + i + nthr);
      differs |= other(v, __ldg(q0 + i)) || other(v2, __ldg(q0 + i + nthr));
    }
    if (i < s.nq) differs |= other(__ldcs(s.rq + i), __ldg(q0 + i));
  } else {
    for (; i < s.nq; i += nthr) {
      const int c = s.head + 4 * i;
      differs |= other(__ldcs(s.rq + i),
                       make_int4(__ldg(pref + c), __ldg(pref + c + 1), __ldg(pref + c + 2), __ldg(pref + c + 3)));
    }
  }
  if (tid < s.head) differs |= __ldcs(s.row + tid) != __ldg(pref + tid);
  const int c0 = s.head + 4 * s.nq;
  if (tid < s.tail) differs |= __ldcs(s.row + c0 + tid) != __ldg(pref + c0 + tid);
  return differs;
}

__global__ void __launch_bounds__(256) k_swap_screen(const int32_t *__restrict__ pref_m,
                                                     const int32_t *__restrict__ pref_w, int n, Control *ctrl,
                                                     int t0, int alike_cta, int only_try = 0) {
  if (only_try && !__syncthreads_or(threadIdx.x == 0 && ld_volatile_s32(&ctrl->swap_try))) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *seen = reinterpret_cast<uint32_t *>(smem_raw);
  __shared__ int s_stop;
  __shared__ int s_row;
  __shared__ int s_wsame;  // no pref_w row has differed from row 0 yet
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const int words = (n + 31) >> 5;
  bool bad = false;
  int bad_value = 0;
  // Rows are taken in turn, each CTA's next one while it works on the last: a
  // CTA that waits for the proposals' CTA to leave its SM then takes fewer.
  // Those from alike_cta on leave after their first where the women's lists are
  // alike (and not all the same, as it seems): a second CTA of the proposals gets
  // their place.
  int next = t0 + static_cast<int>(blockIdx.x);
  const bool leaves = tid == 0 && static_cast<int>(blockIdx.x) >= alike_cta && women_alike(ctrl, n) &&
                      ld_volatile_s32(&ctrl->distinct_w) > 1;
  for (;;) {
    if (tid == 0) {
      s_row = next;
      s_stop = next >= 2 * n || ld_volatile_s32(&ctrl->swap_fail) || ld_volatile_s32(&ctrl->status);
      s_wsame = !ld_volatile_s32(&ctrl->w_differ);
      next = leaves ? 2 * n : t0 + static_cast<int>(gridDim.x) + atomicAdd(&ctrl->screen_next, 1);
    }
    __syncthreads();
    if (s_stop) break;
    const int t = s_row;
    if (t < n) {
      // pref_m row t against row 0
      if (__syncthreads_or(row_differs(pref_m, t, n)) && tid == 0) atomicExch(&ctrl->swap_fail, 1);
    } else {
      // pref_w row t - n: every value in range and seen once.  While no row
      // has differed it is compared with row 0 first (the women may share one
      // list as well): a row equal to row 0 needs no check of its own.
      if (s_wsame && t > n) {
        if (!__syncthreads_or(row_differs(pref_w, t - n, n))) continue;
        if (tid == 0) atomicExch(&ctrl->w_differ, 1);  // one flag per CTA and row
      }
      for (int i = tid; i < words; i += nthr) seen[i] = 0u;
      __syncthreads();
      const RowSpan s = row_span(pref_w, t - n, n);
      // n entries in range that set n bits are a permutation: no atomic's
      // result is waited for, the bits are counted at the end
      const auto mark = [&](int v) {
        if (static_cast<unsigned>(v) < static_cast<unsigned>(n)) {
          atomicOr(seen + (v >> 5), 1u << (v & 31));
        } else {
          bad = true;
          bad_value = v;
        }
      };
      const auto mark4 = [&](int4 v) {
        mark(v.x);
        mark(v.y);
        mark(v.z);
        mark(v.w);
      };
      int i = tid;
      for (; i + nthr < s.nq; i += 2 * nthr) {
        const int4 v = __ldcs(s.rq + i);
        const int4 u = __ldcs(s.rq + i + nthr);
        mark4(v);
        mark4(u);
      }
      if (i < s.nq) mark4(__ldcs(s.rq + i));
      if (tid < s.head) mark(__ldcs(s.row + tid));
      if (tid < s.tail) mark(__ldcs(s.row + s.head + 4 * s.nq + tid));
      __syncthreads();
      for (int k = tid; k < words; k += nthr) {
        const uint32_t full = k < n / 32 ? 0xFFFFFFFFu : (1u << (n & 31)) - 1u;
        if (seen[k] != full) {  // someone is named twice, and this man not at all
          bad = true;
          bad_value = 32 * k + __ffs(~seen[k]) - 1;
        }
      }
      __syncthreads();  // the bitmap is cleared for the next row only after this one
    }
  }
  if (bad) report(ctrl, kStatusInvalidInput, bad_value);
  // the last CTA tells the proposals running beside the screen that it is over
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&ctrl->screen_ctas, 1) == static_cast<int>(gridDim.x) - 1) atomicExch(&ctrl->screen_done, 1);
  }
}

// near[w][r] = woman w's r-th choice for r < kSwapNear, in 16 bits (0xFFFF where
// it is out of range).  A displaced woman's next choices are then in a table of
// 128 bytes per woman that stays in L2; her row is a DRAM access, which takes
// several microseconds while the screen streams both lists.
constexpr int kSwapNear = 64;
__global__ void __launch_bounds__(256) k_swap_near(const int32_t *__restrict__ pref_w, uint16_t *__restrict__ near, int n) {
  const size_t total = static_cast<size_t>(n) * kSwapNear;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int w = static_cast<int>(t / kSwapNear);
    const int r = static_cast<int>(t % kSwapNear);
    if (r < n) near[t] = static_cast<uint16_t>(min(static_cast<uint32_t>(__ldg(pref_w + static_cast<size_t>(w) * n + r)), 0xFFFFu));
  }
}

// The women's proposals.  A man's bid word is pos[w] << 32 | r for the woman
// w he holds and her position r in her list (~0 while he is free), so
// atomicMin keeps the woman the men prefer and hands back the one it
// displaced together with where she resumes.  Each warp carries one woman:
// her next 32 men are read at once, the first man whose current word is
// worse than hers takes her proposal, and a displaced woman continues in the
// same warp.
//   Rows on the device: with full == nullptr every woman's whole row; else
// woman w's whole row where full[w] is set and her first `depth` entries
// otherwise (host-input solves send only those).  A woman who reaches the
// end of what the device holds of her row stops and is appended to `over`
// as (w, position), to resume once her row has been sent (start/start_count
// then list the women this launch resumes, instead of women 0..n-1 from
// position 0).  Gale-Shapley's result does not depend on that order.  An
// entry out of range is reported; a woman who runs out of her whole row
// (input that is not a permutation) too.
//   beside = 1: the screen runs at the same time.  The proposals are a chain of L2
// round trips that leaves the memory idle, the screen a stream that leaves
// the SMs idle: n = 30000 congested took 1.31 ms and then 0.82 ms.  An entry
// that is not a permutation's is the screen's to report here; the proposals
// give up when it has found that the men's lists differ, that the input is
// invalid, or that the women share one list too (they would make n (n + 1) / 2
// contended proposals) -- at once if even their first choices are all alike.
// Two CTAs per SM where the women's lists are alike (women_alike: the proposals
// contend, and there are many times more of them), one where they are not and
// the screen sets the time: it leaves them that much room.
//   beside = 2: after the screen, what is left of the proposals, with four CTAs
// per SM.  (n = 30000, women correlated with sigma 0.2 / 0.01 / 0.0003: 3.4, 5.2
// and 17.9 ms all after the screen; 3.7, 13.0 and 49 with one CTA per SM beside it
// and to the end; 2.8, 4.5 and 14.8 so.)
__global__ void __launch_bounds__(256) k_swap_gs(const int32_t *__restrict__ pref_m,
                                                 const int32_t *__restrict__ pref_w,
                                                 const int32_t *__restrict__ pos,
                                                 unsigned long long *__restrict__ bid, int n, Control *ctrl,
                                                 const uint8_t *__restrict__ full, int depth,
                                                 int2 *__restrict__ over, const int2 *__restrict__ start,
                                                 int start_count, int beside, const uint16_t *__restrict__ near,
                                                 int alike_cta = 0) {
  const int lane = threadIdx.x & 31;
  const int total = start ? start_count : n;
  int w = -1, r0 = 0;
  uint32_t key = 0;
  unsigned steps = 0;
  if (beside) {  // (one look for the CTA, as with the gates)
    int closed = 0;
    if (threadIdx.x == 0 && beside == 1)
      closed = ld_volatile_s32(&ctrl->distinct_w) <= 1 || ld_volatile_s32(&ctrl->swap_fail) ||
               ld_volatile_s32(&ctrl->status) ||
               (static_cast<int>(blockIdx.x) >= alike_cta && !women_alike(ctrl, n));
    if (threadIdx.x == 0 && beside == 2)
      closed = ld_volatile_s32(&ctrl->swap_fail) || ld_volatile_s32(&ctrl->status) || !ld_volatile_s32(&ctrl->w_differ);
    if (__syncthreads_or(closed)) return;
  }
  for (;;) {
    // Now and then only: thousands of warps reading these flags at every step
    // would queue at one L2 slice.
    if (beside && (++steps & 31) == 0) {
      int stop = 0;
      if (lane == 0)
        stop = ld_volatile_s32(&ctrl->swap_fail) || ld_volatile_s32(&ctrl->status) ||
               (ld_volatile_s32(&ctrl->screen_done) && !ld_volatile_s32(&ctrl->w_differ));
      if (__shfl_sync(kFullMask, stop, 0)) return;
    }
    if (w < 0) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&ctrl->swap_next, 1);
      i = __shfl_sync(kFullMask, i, 0);
      if (i >= total) break;
      if (start) {
        const int2 e = start[i];
        w = e.x;
        r0 = e.y;
      } else {
        w = i;
        r0 = 0;
      }
      key = static_cast<uint32_t>(__ldg(pos + w));
    }
    const int lim = (full == nullptr || full[w]) ? n : depth;  // entries of her row on the device
    if (r0 >= lim) {
      if (lane == 0) {
        if (lim >= n) {
          report(ctrl, kStatusInvalidInput, w);
        } else {
          // at most n: a woman who stops holds no man, so nothing sends her
          // back into this launch
          const int k = atomicAdd(&ctrl->swap_over, 1);
          if (k < n)
            over[k] = make_int2(w, r0);
          else
            report(ctrl, kStatusInvalidInput, w);
        }
      }
      w = -1;
      continue;
    }
    const int r = r0 + lane;
    const bool in_row = r < lim;
    const int m = !in_row                ? 0
                  : near && r < kSwapNear ? static_cast<int>(__ldg(near + w * kSwapNear + r))
                                          : __ldg(pref_w + static_cast<size_t>(w) * n + r);
    const bool valid = static_cast<unsigned>(m) < static_cast<unsigned>(n);
    const bool open = in_row && valid && static_cast<uint32_t>(ld_relaxed_u64(bid + m) >> 32) > key;
    const unsigned hit = __ballot_sync(kFullMask, open);
    const unsigned bad = __ballot_sync(kFullMask, in_row && !valid);
    if (bad) {  // an entry out of range
      if (lane == __ffs(bad) - 1) report(ctrl, kStatusInvalidInput, m);
      w = -1;
      continue;
    }
    if (!hit) {
      r0 = min(r0 + 32, lim);
      continue;
    }
    const int f = __ffs(hit) - 1;
    unsigned long long old = 0;
    if (lane == f)
      old = atomicMin(bid + m, (static_cast<unsigned long long>(key) << 32) | static_cast<uint32_t>(r));
    old = __shfl_sync(kFullMask, old, f);
    if (static_cast<uint32_t>(old >> 32) < key) {  // a woman the men prefer got there first
      r0 += f + 1;
      continue;
    }
    if (old == ~0ull) {  // he was free: the chain ends
      w = -1;
      continue;
    }
    key = static_cast<uint32_t>(old >> 32);
    w = __ldg(pref_m + key);
    r0 = static_cast<int>(old & 0xFFFFFFFFull) + 1;
  }
}

// Host-input shared-list solves: checks the entries of pref_w the device
// holds -- the first `cols` of every row (rows == nullptr: rows 0..count-1)
// or of the listed rows -- are in range and name no man twice.  One row per
// CTA at a time, n bits of shared memory.
__global__ void __launch_bounds__(256) k_swap_rows_check(const int32_t *__restrict__ pref_w, int n,
                                                         const int32_t *__restrict__ rows, int count, int cols,
                                                         Control *ctrl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *seen = reinterpret_cast<uint32_t *>(smem_raw);
  const int words = (n + 31) >> 5;
  bool bad = false;
  int bad_value = 0;
  for (int i = blockIdx.x; i < count; i += gridDim.x) {
    const int w = rows ? __ldg(rows + i) : i;
    for (int k = threadIdx.x; k < words; k += blockDim.x) seen[k] = 0u;
    __syncthreads();
    if (static_cast<unsigned>(w) < static_cast<unsigned>(n)) {
      const int32_t *row = pref_w + static_cast<size_t>(w) * n;
      for (int r = threadIdx.x; r < cols; r += blockDim.x) {
        const int v = __ldg(row + r);
        if (static_cast<unsigned>(v) >= static_cast<unsigned>(n)) {
          bad = true;
          bad_value = v;
          continue;
        }
        const uint32_t bit = 1u << (v & 31);
        if (atomicOr(seen + (v >> 5), bit) & bit) {
          bad = true;
          bad_value = v;
        }
      }
    } else if (threadIdx.x == 0) {
      bad = true;
      bad_value = w;
    }
    __syncthreads();  // the bitmap is cleared for the next row only after this one
  }
  if (bad) report(ctrl, kStatusInvalidInput, bad_value);
}

// full[rows[i]] = 1 for the rows now whole on the device.
__global__ void k_swap_mark_full(uint8_t *__restrict__ full, const int32_t *__restrict__ rows, int count, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const int w = __ldg(rows + i);
    if (static_cast<unsigned>(w) < static_cast<unsigned>(n)) full[w] = 1;
  }
}

// The outcome of the screen and the proposals beside it: nothing where the
// men's lists differ or the input is invalid; the pairing rank for rank where
// the women share one list too; else match[m] = the woman m holds.  swap_out
// says that match[] is complete.
__global__ void k_swap_outcome(const int32_t *__restrict__ pref_m, const int32_t *__restrict__ pref_w,
                               const unsigned long long *__restrict__ bid, int32_t *__restrict__ match, int n,
                               Control *ctrl, int only_try = 0) {
  if (only_try && !ld_volatile_s32(&ctrl->swap_try)) return;
  if (ld_volatile_s32(&ctrl->swap_fail) || ld_volatile_s32(&ctrl->status)) return;
  const bool alike = !ld_volatile_s32(&ctrl->w_differ);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    if (alike) {
      match[__ldg(pref_w + k)] = __ldg(pref_m + k);
    } else {
      const unsigned long long b = bid[k];
      // (a man left without a woman: reported by the proposals)
      match[k] = b == ~0ull ? -1 : __ldg(pref_m + static_cast<uint32_t>(b >> 32));
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl->swap_out = 1;
    ctrl->proposals = static_cast<unsigned long long>(n) * (static_cast<unsigned long long>(n) + 1) / 2;
    ctrl->bulk_proposals = ctrl->proposals;
    ctrl->tail_proposals = 0;
  }
}

// match[m] = the woman m holds; the men's proposal count of the same
// matching is n(n+1)/2 (final positions 0 .. n-1 in the shared list).
__global__ void k_swap_match(const int32_t *__restrict__ pref_m, const unsigned long long *__restrict__ bid,
                             int32_t *__restrict__ match, int n, Control *ctrl) {
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
    const unsigned long long b = bid[m];
    if (b == ~0ull) {
      report(ctrl, kStatusInvalidInput, m);
      match[m] = -1;
    } else {
      match[m] = __ldg(pref_m + static_cast<uint32_t>(b >> 32));
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl->proposals = static_cast<unsigned long long>(n) * (static_cast<unsigned long long>(n) + 1) / 2;
    ctrl->bulk_proposals = ctrl->proposals;
    ctrl->tail_proposals = 0;
  }
}

// Both sides share one list each (L for the men, M for the women): the k-th
// man of M and the k-th woman of L pair up.  The men's proposal count is
// again n(n+1)/2.
__global__ void k_swap_direct(const int32_t *__restrict__ pref_m, const int32_t *__restrict__ pref_w,
                              int32_t *__restrict__ match, int n, Control *ctrl) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
    match[__ldg(pref_w + k)] = __ldg(pref_m + k);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctrl->proposals = static_cast<unsigned long long>(n) * (static_cast<unsigned long long>(n) + 1) / 2;
    ctrl->bulk_proposals = ctrl->proposals;
    ctrl->tail_proposals = 0;
  }
}

}  // namespace smpb200
