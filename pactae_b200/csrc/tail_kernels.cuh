// tail_kernels.cuh -- the end of a query-mode solve: the last free men's
// displacement chains, in one CTA.
//
// The last chain is the critical path of a uniform solve: thousands of
// displacements, one after the other.  A man displaced here goes to the first
// woman after his position who would take him, and about nine in ten would
// not.  k_tail_lists finds them on all SMs when the bulk hands over: a man's
// first kTailCand women, after his position, who prefer him to their partner
// at that moment.  Women only improve, so nobody else can take him until that
// list is used up.
//   One thread follows a chain (a warp each, its other lanes idle): a step is
// a handful of dependent shared reads, and every shuffle, ballot or branch on
// it costs as much as one of them.
//   Where shared memory holds at least four entries of every list (kExact), a
// step reads those and the four women's words, and proposes to the first who
// still takes him.  Entries that have rejected a man reject him again, so a
// list is read from its start and keeps no state.
//   Else the lists are in L2, 350 cycles away, and shared memory holds only the
// woman each begins with.  While she has not changed partners since the lists
// were made she takes him, whatever the ranks: one bit of her word says so,
// and a step is two shared reads and a compare-and-swap.  Her new rank is not
// read but left for whoever needs it ("lazy": it stands in the list of the man
// she holds).  Where she has changed the list is read.  Lists age as women
// change, so a thread that has read enough of them ends the segment: all
// chains are parked and the lists made anew (one more pair of launches).
//   The last few chains are followed by one thread, one after the other: with
// nobody else writing, a proposal is a plain store, and steps go four to a
// branch, each predicated on the one before.
//   k_tail_out writes the matching and finds the positions.
//
// Measured (uniform, mean of eight seeds; before: one kernel, a warp-wide
// look at the next 32 choices per step, 630 cycles of which an L2 round trip
// is 350): tail at n = 30000 1.92 -> 1.16 ms, n = 16411 1.28 -> 0.83, n = 8000
// 0.38 -> 0.30, n = 2000 0.19 -> 0.15.  The last chain's step takes 160 cycles
// with lists in L2 (850 where the list is read: one in sixteen before a segment
// ends), 215 with exact lists.  A four-entry list read from L2 at every step,
// without the first-woman test, took 545.
#pragma once

#include "common.cuh"
#include "solve_kernels.cuh"

namespace smpb200 {

constexpr int kTailCand = 16;  // candidates per man: four 16-byte groups
constexpr uint32_t kTailNone = 0xFFFFFFFFu;
constexpr int kTailMaxN = 32767;  // men in 15 bits, ranks below 0x7FFF

// Words: all ones = free, else rank << 16 | man.  Where the lists are in L2 a
// woman who has changed since they were made has kTailChanged set in the
// man's half; lazy words are kTailLazy | kTailChanged | man.
constexpr uint32_t kTailLazy = 0x80000000u;
constexpr uint32_t kTailChanged = 0x8000u;

struct TailBufs {
  uint32_t *list;   // [n][kTailCand]: woman << 16 | her rank of him; kTailNone past the end
  uint32_t *word;   // [n]: the women's words at the end of a segment (never lazy or changed)
  int32_t *park[2]; // [n]: men without a woman, segment k's in park[k & 1]
  uint16_t *first;  // [n]: the first list entry's woman, tail_people(n) if none
  uint16_t *from;   // [n]: the prefix entry a man's search starts at
  uint16_t *end;    // [n]: the prefix entry of his last list entry, if the list is full
};
__host__ __device__ constexpr size_t tail_people(int n) { return (static_cast<size_t>(n) + 7) & ~static_cast<size_t>(7); }
__host__ __device__ constexpr size_t tail_bytes(int n) { return tail_people(n) * (4 * kTailCand + 4 + 4 + 4 + 2 + 2 + 2); }

// The query-mode tail runs (the other kernels of the mode test the same).
__device__ __forceinline__ bool tail_open(const Control *ctrl) {
  return ld_volatile_s32(&ctrl->mode) == kModeQuery && gate_open(kGateMain, ctrl) && !ld_volatile_s32(&ctrl->retry) &&
         !ld_volatile_s32(&ctrl->tail_done);
}

// One man's list: entries of his prefix from `start` whose women rank him
// below cut[w], the rank of their partner (0xFFFF: free).
__device__ __forceinline__ void tail_list(const uint32_t *__restrict__ row, int Kn, int start, int m,
                                          const uint16_t *cut, const TailBufs &b, int none, int lane) {
  uint32_t *list = b.list + static_cast<size_t>(m) * kTailCand;
  int count = 0;
  for (int base = start; base < Kn && count < kTailCand; base += 96) {
    uint32_t raw[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int r = base + 32 * u + lane;
      raw[u] = r < Kn ? __ldg(row + r) : kTailNone;
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const bool takes = raw[u] != kTailNone && (raw[u] & 0xFFFFu) < cut[raw[u] >> 16];
      const unsigned hit = __ballot_sync(kFullMask, takes);
      const int at = count + __popc(hit & ((1u << lane) - 1u));
      if (takes && at < kTailCand) {
        list[at] = raw[u];
        if (at == 0) b.first[m] = static_cast<uint16_t>(raw[u] >> 16);
        if (at == kTailCand - 1) b.end[m] = static_cast<uint16_t>(base + 32 * u + lane);
      }
      count += __popc(hit);
    }
  }
  if (count + lane < kTailCand) list[count + lane] = kTailNone;
  if (count == 0 && lane == 0) b.first[m] = static_cast<uint16_t>(none);
}

// Lists of every man.  In segment 0 a man is found through the woman he holds
// (the bulk's words), in the queue the bulk left, or among those who never
// proposed, and his position is kept; later ones start from it again, since
// every woman in between rejects him still.
constexpr int kTailListBlock = 512;

template <bool kFirst>
__global__ void __launch_bounds__(kTailListBlock) k_tail_lists(const uint32_t *__restrict__ prefix, int K,
                                                               const unsigned long long *__restrict__ bid,
                                                               const int2 *__restrict__ tail_queue, TailBufs b, int n,
                                                               Control *ctrl) {
  if (!tail_open(ctrl)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t *cut = reinterpret_cast<uint16_t *>(smem_raw);
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int Kn = min(K, n);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int warp = (blockIdx.x * blockDim.x + tid) >> 5;
#pragma unroll 8
  for (int w = tid; w < n; w += kTailListBlock)
    cut[w] = kFirst ? static_cast<uint16_t>(min(bid_rank(__ldg(bid + w)), 0xFFFFu))
                    : static_cast<uint16_t>(__ldg(b.word + w) >> 16);
  __syncthreads();
  if (kFirst) {
    const int queued = ctrl->tail_count;
    const int first_unstarted = min(ctrl->next_man, n);
    const int total = queued + (n - first_unstarted);
    if (warp == 0 && lane == 0) ctrl->tail_left = total;
    for (int i = warp; i < n + total; i += warps) {
      int m, start;
      if (i < n) {
        const unsigned long long w = __ldg(bid + i);
        if (w == kFree) continue;
        m = static_cast<int>(bid_man(w));
        start = static_cast<int>(bid_pos(w)) + 1;
      } else if (i < n + queued) {
        const int2 e = tail_queue[i - n];
        m = e.x;
        start = e.y;
      } else {
        m = first_unstarted + (i - n - queued);
        start = 0;
      }
      if (lane == 0) {
        b.from[m] = static_cast<uint16_t>(start);
        if (i >= n) b.park[0][i - n] = m;
      }
      tail_list(prefix + static_cast<size_t>(m) * K, Kn, start, m, cut, b, static_cast<int>(tail_people(n)), lane);
    }
  } else {
    for (int m = warp; m < n; m += warps)
      tail_list(prefix + static_cast<size_t>(m) * K, Kn, b.from[m], m, cut, b, static_cast<int>(tail_people(n)),
                lane);
  }
}

// Why the chains stop: few are left (one thread goes on with them), the lists
// are too old (the segment ends), the solve cannot go on here.
constexpr int kTailFew = 1, kTailOld = 2, kTailOver = 3;
// Chains that one thread follows one after the other.  With the lists in L2 a
// step costs it about 0.4 of what it costs threads that must propose
// atomically; with exact lists the two differ little, and only the last one
// gains.
constexpr int tail_alone(bool exact) { return exact ? 1 : 3; }

// Shared memory: words (4 bytes) per person, then E list entries per man, or,
// with E = 0, first women (2 bytes) and one word that is never free to take.
__host__ __device__ constexpr size_t tail_q_smem(int n, int E) {
  return E > 0 ? tail_people(n) * (4 + 4 * static_cast<size_t>(E)) : tail_people(n) * 6 + 16;
}

// One segment.  E: list entries of each man held in shared memory (0, 4, 8
// or 16); slow_limit (E = 0): lists a thread reads from L2 before it ends the
// segment (0: never).
template <int E>
__global__ void __launch_bounds__(1024, 1) k_tail_q(const int32_t *__restrict__ pref_m,
                                                    const uint32_t *__restrict__ prefix, int K,
                                                    const unsigned long long *__restrict__ bid, Control *ctrl,
                                                    TailBufs b, int32_t *match, int32_t *also, int n, int segment,
                                                    int slow_limit) {
  constexpr bool kExact = E > 0;
  constexpr int kAlone = tail_alone(kExact);
  if (segment == 0 && ld_volatile_s32(&ctrl->mode) == kModeQuery && ld_volatile_s32(&ctrl->perfect)) {
    write_perfect(pref_m, match, n, ctrl, also);
    return;
  }
  if (!tail_open(ctrl)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int np = static_cast<int>(tail_people(n));
  uint32_t *sbid = reinterpret_cast<uint32_t *>(smem_raw);
  uint4 *slist = reinterpret_cast<uint4 *>(smem_raw + static_cast<size_t>(np) * 4);       // kExact
  uint16_t *sfirst = reinterpret_cast<uint16_t *>(smem_raw + static_cast<size_t>(np) * 4 + 16);  // else, after sbid[np]
  __shared__ int s_next;
  __shared__ int s_left;    // chains that have not ended
  __shared__ int s_parked;
  __shared__ int s_stop;    // kTailFew, kTailOld or kTailOver (below)
  __shared__ unsigned int s_hops;
  const int tid = threadIdx.x;
  const int Kn = min(K, n);
  const uint4 *glist = reinterpret_cast<const uint4 *>(b.list);
  const int total = ctrl->tail_left;
  const int32_t *waiting = b.park[segment & 1];
  int32_t *parked = b.park[(segment & 1) ^ 1];
  if (segment == 0) {
#pragma unroll 8
    for (int i = tid; i < n; i += 1024) {
      const unsigned long long w = __ldg(bid + i);
      sbid[i] = w == kFree ? 0xFFFFFFFFu : (bid_rank(w) << 16) | bid_man(w);
    }
  } else {
#pragma unroll 4
    for (int i = tid; i < np / 4; i += 1024)
      reinterpret_cast<uint4 *>(sbid)[i] = __ldcg(reinterpret_cast<const uint4 *>(b.word) + i);  // (written below)
  }
  if (kExact) {
    constexpr int kGroups = kExact ? E / 4 : 1;
#pragma unroll 4
    for (int i = tid; i < n * kGroups; i += 1024)
      slist[i] = __ldg(glist + static_cast<size_t>(i / kGroups) * (kTailCand / 4) + i % kGroups);
  } else {
#pragma unroll 4
    for (int i = tid; i < np / 8; i += 1024)
      reinterpret_cast<uint4 *>(sfirst)[i] = __ldg(reinterpret_cast<const uint4 *>(b.first) + i);
    if (tid == 0) sbid[np] = kTailChanged;  // the word of a man with an empty list
  }
  if (tid == 0) {
    s_next = 0;
    s_left = total;
    s_parked = 0;
    s_stop = total <= kAlone ? kTailFew : 0;
    s_hops = 0;
    if (segment == 0) ctrl->tail_men = total;
  }
  __syncthreads();

  // the q-th four entries of man m's list
  const auto group = [&](int m, int q) {
    if (kExact && 4 * q < E) return slist[m * (E / 4) + q];
    return __ldg(glist + m * (kTailCand / 4) + q);
  };
  // a word's rank, read where it stands if it is lazy
  const auto rank_of = [&](uint32_t w) -> uint32_t {
    if (!kExact && w != 0xFFFFFFFFu && (w & kTailLazy))
      return __ldg(b.list + static_cast<size_t>(w & 0x7FFFu) * kTailCand) & 0xFFFFu;
    return w >> 16;
  };
  const auto word_of = [&](uint32_t e) { return e != kTailNone ? lds_relaxed_u32(sbid + (e >> 16)) : 0u; };

  // Whoever takes man m first in his list from its q-th group on, or in the
  // prefix after it: her entry and her word.  kTailNone if nobody does.
  int slow = 0;  // lists read from L2, or, kExact, used up altogether
  const auto search = [&](int m, int q, uint32_t &word) -> uint32_t {
    for (; q < kTailCand / 4; ++q) {
      const uint4 g = group(m, q);
      const uint32_t e[4] = {g.x, g.y, g.z, g.w};
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = word_of(e[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if ((e[k] & 0xFFFFu) < rank_of(w[k])) {
          word = w[k];
          return e[k];
        }
      if (g.w == kTailNone) return kTailNone;  // the list held every woman of his prefix who might
    }
    if (kExact) slow++;
    for (int r = b.end[m] + 1; r < Kn; r += 8) {
      uint32_t e[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = r + k < Kn ? __ldg(prefix + static_cast<size_t>(m) * K + r + k) : kTailNone;
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        const uint32_t w = word_of(e[k]);
        if ((e[k] & 0xFFFFu) < rank_of(w)) {
          word = w;
          return e[k];
        }
      }
    }
    return kTailNone;
  };
  // beyond the prefix (the rank-mode round starts over), or, where the
  // prefix is the whole list, rejected by every woman
  const auto nobody = [&](int m) {
    s_stop = kTailOver;
    if (Kn < n)
      atomicExch(&ctrl->retry, 1);
    else
      report(ctrl, kStatusInvalidInput, m);
  };
  const auto stopped = [&]() { return *reinterpret_cast<volatile int *>(&s_stop); };
  unsigned int hops = 0;
  if ((tid & 31) == 0) {
    int m = -1;
    const auto next_man = [&]() {
      const int i = stopped() ? total : atomicAdd(&s_next, 1);
      if (i >= total) return false;
      m = waiting[i];
      return true;
    };
    const auto ended = [&]() {  // at a free woman
      if (atomicSub(&s_left, 1) == kAlone + 1) atomicMax(&s_stop, kTailFew);
      return !next_man();
    };
    if (next_man()) {
      for (;;) {
        if (stopped()) {
          parked[atomicAdd(&s_parked, 1)] = m;
          break;
        }
        if constexpr (kExact) {
          const uint4 g = slist[m * (E / 4)];
          const uint32_t w0 = word_of(g.x), w1 = word_of(g.y), w2 = word_of(g.z), w3 = word_of(g.w);
          // (kTailNone's rank, 0xFFFF, is below no word's)
          const bool t0 = (g.x & 0xFFFFu) < (w0 >> 16), t1 = (g.y & 0xFFFFu) < (w1 >> 16),
                     t2 = (g.z & 0xFFFFu) < (w2 >> 16), t3 = (g.w & 0xFFFFu) < (w3 >> 16);
          uint32_t e = t0 ? g.x : t1 ? g.y : t2 ? g.z : g.w;
          if (!(t0 || t1 || t2 || t3)) {
            uint32_t word = 0;
            e = g.w == kTailNone ? kTailNone : search(m, 1, word);
            if (e == kTailNone) {
              nobody(m);
              break;
            }
            if (slow_limit > 0 && slow >= slow_limit) atomicMax(&s_stop, kTailOld);
          }
          const uint32_t old = atom_min_relaxed_shared(sbid + (e >> 16), (e << 16) | static_cast<uint32_t>(m));
          if ((old >> 16) <= (e & 0xFFFFu)) continue;  // someone better got there first
          hops++;
          if (old != 0xFFFFFFFFu)
            m = static_cast<int>(old & 0xFFFFu);
          else if (ended())
            break;
        } else {
          const uint32_t w = sfirst[m];
          const uint32_t word = lds_relaxed_u32(sbid + w);
          if (!(word & (kTailLazy | kTailChanged))) {  // (a free woman's word has both)
            if (atomicCAS(sbid + w, word, kTailLazy | kTailChanged | static_cast<uint32_t>(m)) == word) {
              hops++;
              m = static_cast<int>(word & 0x7FFFu);
            }
            continue;
          }
          // she has changed, or is free, or there is none
          slow++;
          uint32_t seen = 0;
          const uint32_t e = w < static_cast<uint32_t>(np) ? search(m, 0, seen) : kTailNone;
          if (e == kTailNone) {
            nobody(m);
            break;
          }
          if (atomicCAS(sbid + (e >> 16), seen, (e << 16) | kTailChanged | static_cast<uint32_t>(m)) != seen) continue;
          hops++;
          if (seen != 0xFFFFFFFFu)
            m = static_cast<int>(seen & 0x7FFFu);
          else if (ended())
            break;
          if (slow_limit > 0 && slow >= slow_limit) atomicMax(&s_stop, kTailOld);
        }
      }
    }
  }
  __syncthreads();
  const int why = s_stop;
  __syncthreads();
  if (why == kTailOver) return;
  if (why == kTailFew && tid == 0) {
    // the parked men and those nobody took up, one after the other
    const int few = s_parked;
    const int taken = min(s_next, total);
    const int count = few + (total - taken);
    int over = 0, kept = 0;
    slow = 0;
    for (int i = 0; i < count; ++i) {
      int m = i < few ? parked[i] : waiting[taken + i - few];
      for (bool on = !over; on;) {
        uint32_t e, seen = 0;
        if constexpr (kExact) {
          const uint4 g = slist[m * (E / 4)];
          const uint32_t w0 = word_of(g.x), w1 = word_of(g.y), w2 = word_of(g.z), w3 = word_of(g.w);
          const bool t0 = (g.x & 0xFFFFu) < (w0 >> 16), t1 = (g.y & 0xFFFFu) < (w1 >> 16),
                     t2 = (g.z & 0xFFFFu) < (w2 >> 16), t3 = (g.w & 0xFFFFu) < (w3 >> 16);
          e = t0 ? g.x : t1 ? g.y : t2 ? g.z : g.w;
          seen = t0 ? w0 : t1 ? w1 : t2 ? w2 : w3;
          if (!(t0 || t1 || t2 || t3)) e = g.w == kTailNone ? kTailNone : search(m, 1, seen);
        } else {
          for (;;) {
            bool ok = true;
            uint32_t w = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              w = sfirst[m];
              const uint32_t word = lds_relaxed_u32(sbid + w);
              ok = ok && !(word & (kTailLazy | kTailChanged));
              if (ok) {
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(smem_addr(sbid + w)),
                             "r"(kTailLazy | kTailChanged | static_cast<uint32_t>(m)) : "memory");
                m = static_cast<int>(word & 0x7FFFu);
                hops++;
              }
            }
            if (!ok) break;
          }
          slow++;
          const uint32_t w = sfirst[m];
          e = w < static_cast<uint32_t>(np) ? search(m, 0, seen) : kTailNone;
        }
        if (e == kTailNone) {
          nobody(m);
          over = 1;
          break;
        }
        sbid[e >> 16] = (e << 16) | (kExact ? 0u : kTailChanged) | static_cast<uint32_t>(m);
        hops++;
        on = seen != 0xFFFFFFFFu;
        m = static_cast<int>(seen & (kExact ? 0xFFFFu : 0x7FFFu));
        if (on && slow_limit > 0 && slow >= slow_limit) {
          // the lists are too old; the men left go to the front of the next
          // segment's list
          on = false;
          parked[kept++] = m;  // (entry i or before: read already)
          for (int j = i + 1; j < count; ++j) parked[kept++] = j < few ? parked[j] : waiting[taken + j - few];
          i = count;
        }
      }
    }
    s_parked = kept;
    s_next = total;
    if (over) s_stop = kTailOver;
  }
  if ((tid & 31) == 0 && hops) atomicAdd(&s_hops, hops);
  __syncthreads();
  if (s_stop == kTailOver) return;
  // men whom nobody took up wait for the next segment, too
  for (int i = min(s_next, total) + tid; i < total; i += 1024) parked[atomicAdd(&s_parked, 1)] = waiting[i];
  // the words without their marks
#pragma unroll 8
  for (int w = tid; w < n; w += 1024) {
    const uint32_t v = sbid[w];
    if constexpr (kExact) {
      b.word[w] = v;
    } else {
      const bool lazy = v != 0xFFFFFFFFu && (v & kTailLazy);
      const uint32_t rank = lazy ? __ldg(b.list + static_cast<size_t>(v & 0x7FFFu) * kTailCand) : v >> 16;
      b.word[w] = v == 0xFFFFFFFFu ? v : (rank << 16) | (v & 0x7FFFu);
    }
  }
  __syncthreads();
  if (tid == 0) {
    ctrl->tail_left = s_parked;
    ctrl->tail_hops += s_hops;
    ctrl->tail_done = s_parked == 0;
  }
}

// match[] (and also[], see write_perfect) and the proposal count: a man's position is where the woman he
// ended with stands in his prefix, at or after the entry before `from`.
__global__ void __launch_bounds__(256) k_tail_out(const uint32_t *__restrict__ prefix, int K, TailBufs b,
                                                  int32_t *match, int32_t *also, int n, Control *ctrl) {
  if (ld_volatile_s32(&ctrl->mode) != kModeQuery || !gate_open(kGateMain, ctrl) || !ld_volatile_s32(&ctrl->tail_done)) return;
  const int lane = threadIdx.x & 31;
  const int Kn = min(K, n);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long props = 0;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += warps) {
    const uint32_t word = __ldg(b.word + w);
    if (word == 0xFFFFFFFFu) {
      if (lane == 0) report(ctrl, kStatusInvalidInput, w);
      continue;
    }
    const int m = static_cast<int>(word & 0xFFFFu);
    int found = -1;
    for (int base = max(static_cast<int>(b.from[m]) - 1, 0); base < Kn && found < 0; base += 32) {
      const int r = base + lane;
      const uint32_t raw = r < Kn ? __ldg(prefix + static_cast<size_t>(m) * K + r) : kTailNone;
      const unsigned hit = __ballot_sync(kFullMask, raw != kTailNone && static_cast<int>(raw >> 16) == w);
      if (hit) found = base + __ffs(hit) - 1;
    }
    if (lane == 0) {
      if (found < 0) report(ctrl, kStatusInvalidInput, w);
      match[m] = w;
      if (also) also[m] = w;
      props += static_cast<unsigned long long>(found + 1);
    }
  }
  if (lane == 0 && props) atomicAdd(&ctrl->proposals, props);
}

}  // namespace smpb200
