// round_kernels.cuh -- the rank-mode proposals of one solve (uint16 ranks, bids
// that fit one SM's shared memory): a sequence of identical launches, each of
// which scans a batch of men on every SM and resolves it on one.
//
// In lists that resemble one another (common scores, common groups, one
// shared list with a twist) a man is rejected by hundreds or thousands of
// women before one takes him.  The rejections are cheap to find out in bulk;
// the acceptances are serial chains.  So a step
//   scans    the next men on all SMs, each against the women's partners as
//            the step before left them: his first kCand women who would take
//            him, with her rank of him and her position in his list.  Women
//            only improve, so a woman left out would reject him at any later
//            time: this list replaces his preference row;
//   resolves them on the CTA that finishes scanning last: a warp per
//            displacement chain, or eight lanes, bids and positions in shared memory, every
//            choice read from the candidate lists.  A man whose list is used
//            up is parked and scanned again, from where he stopped, in the
//            next step.
// Steps follow one another on the stream: the launch boundary is the only
// barrier between them and no CTA ever waits for another.  The men start in
// the order the women like them (k_order_*): a man then meets women who hold
// the men that will keep them, instead of taking free ones he loses again.
// When all men have started and some are parked, every man is scanned again
// (refresh): without it a chain through men whose lists are old would cost a
// step per displacement.
//
// Gale-Shapley's result and proposal count do not depend on the order in
// which men propose, and the proposal count is taken from the final
// positions, so none of this shows in the outputs.
//
// Measured on one B200 against k_bulk, k_tail and k_tail_coop over ranks by
// position, which still serve int32 ranks, lists whose bids no SM holds, and men
// who are alike among women who are not (bulk_rank_pays in smp_b200.cu):
// RANDOM(5) n = 15013 18.7 -> 4.0 ms (18.7 M displacements -> 98 thousand),
// n = 30000 58.8 -> 9.6; SOLO n = 10007 43.6 -> 3.0; correlated n = 30000
// 10.8 -> 7.9, n = 2000 0.57 -> 0.53, n = 97 0.25 -> 0.22.  A step of the
// n = 30000 correlated solve takes about 36 us to scan (592 rows of two
// lists: 100 MB, half the copy rate), 2 us to load the state, 64 us to
// resolve and 10 us between launches.  The resolver is bound by the latency
// of a displacement (0.46 us by warp, an L2 read of the next window on it; 0.5
// to 0.74 by eight lanes, where four chains wait for one another) and, at 32
// warps with a chain each, by the SM's issue slots (0.58 us): 24 or 16 warps
// take 7.4 and 8.6 ms for RANDOM(5)'s proposals where 32 take 6.9.  Batches of
// 296 and 1184 men were slower than 592 (9.4 and 6.3 against 6.8 ms
// correlated, 10.6 and 13.3 against 8.5 ms RANDOM(5), n = 30000): a man skips
// those of his own batch one by one, and a step costs what it costs.  Scanning
// a batch ahead while the last one is resolved does not pay for the same
// reason: the men then skip two batches.
#pragma once

#include "common.cuh"
#include "solve_kernels.cuh"

namespace smpb200 {

// ---------------------------------------------------------------------------
// The men by popularity (alone, with k_bulk: RANDOM(5) n = 30000 58.8 -> 23.2
// ms, correlated 453 -> 149 thousand displacements).  score[m] = mean rank of m over up to 64 women
// spread over the rank matrix, in kOrderBuckets steps; k_order_sort counts
// the buckets and lays the men out bucket by bucket.  The order within a
// bucket is arbitrary: any order gives the same matching.
// (Men liked in one order by the women numbered i n / 64 and in the reverse by all
// others, n = 4000: 78 ms with those sampled, 3.2 as it is.)
// ---------------------------------------------------------------------------
constexpr uint32_t kOrderBuckets = 8192;
constexpr int kOrderSamples = 64;

template <typename RankT>
__global__ void __launch_bounds__(256) k_order_score(const RankT *__restrict__ rank, size_t ld,
                                                     uint32_t *__restrict__ score, int n, Control *ctrl, int gate) {
  if (!cta_gate_open(gate, ctrl)) return;
  const int samples = min(n, kOrderSamples);
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
    unsigned long long sum = 0;
#pragma unroll 16
    for (int i = 0; i < samples; ++i) {
      const size_t w = static_cast<size_t>(order_sample(i, samples, n));
      sum += static_cast<uint32_t>(__ldg(rank + w * ld + m));
    }
    const unsigned long long b = sum * kOrderBuckets / (static_cast<unsigned long long>(n) * samples);
    score[m] = b < kOrderBuckets ? static_cast<uint32_t>(b) : kOrderBuckets - 1;
  }
}

// One CTA.
__global__ void __launch_bounds__(1024) k_order_sort(const uint32_t *__restrict__ score, int32_t *__restrict__ order,
                                                     int n, Control *ctrl, int gate) {
  if (!cta_gate_open(gate, ctrl)) return;
  __shared__ uint32_t hist[kOrderBuckets];
  __shared__ uint32_t warp_sum[32];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  constexpr int kPer = kOrderBuckets / 1024;
  for (int i = tid; i < static_cast<int>(kOrderBuckets); i += 1024) hist[i] = 0;
  __syncthreads();
  for (int m = tid; m < n; m += 1024) atomicAdd(&hist[score[m]], 1u);
  __syncthreads();
  uint32_t before[kPer], sum = 0;  // exclusive sums of this thread's buckets
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    before[k] = sum;
    sum += hist[tid * kPer + k];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t v = __shfl_up_sync(kFullMask, incl, off);
    if (lane >= off) incl += v;
  }
  if (lane == 31) warp_sum[tid >> 5] = incl;
  __syncthreads();
  if (tid < 32) {
    uint32_t v = warp_sum[tid];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t u = __shfl_up_sync(kFullMask, v, off);
      if (tid >= off) v += u;
    }
    warp_sum[tid] = v;
  }
  __syncthreads();
  const uint32_t base = incl - sum + (tid >= 32 ? warp_sum[(tid >> 5) - 1] : 0u);
#pragma unroll
  for (int k = 0; k < kPer; ++k) hist[tid * kPer + k] = base + before[k];
  __syncthreads();
  for (int m = tid; m < n; m += 1024) order[atomicAdd(&hist[score[m]], 1u)] = m;
}

// ---------------------------------------------------------------------------
// State of the rounds between launches.
// ---------------------------------------------------------------------------
// Entries per candidate list (n if fewer).  Where the lists are alike a batch
// takes about as many women as it has men, so a list must reach past that: with
// 32 entries RANDOM(5) n = 2000 took 63 ms.
constexpr int kCand = 1024;
constexpr int kRoundBlock = 1024;
constexpr int kTeam = 256;       // threads that scan one man
constexpr int kTeams = kRoundBlock / kTeam;
constexpr int kScanUnroll = 8;   // entries per thread and scan step
constexpr int kWide = 8;         // windows of 32 a chain looks ahead at first
constexpr uint32_t kNoCand = 0xFFFFFFFFu;

struct RoundSlot {
  int32_t parked;      // men in the step's parked list
  int32_t new0, new1;  // then the men order[new0 .. new1)
  int32_t refresh;     // every man is scanned
};
struct RoundCtl {
  RoundSlot slot[2];   // step t works on slot t & 1 and fills the other
  int32_t arrived[2];  // CTAs of step t that have scanned their men
  int32_t checked[2];  // rows of step t's new men taken for their range check
  int32_t done;        // the matching is complete and written
  int32_t calm;        // 1: few proposals of the step before came too late; -1: many did at four times the chains
};

struct RoundBufs {
  RoundCtl *ctl;
  uint32_t *cand;     // [n][cap]: woman << 16 | her rank of him; kNoCand past the end
  uint16_t *cpos;     // [n][cap]: her position in his list
  uint32_t *word;     // [n]: rank << 16 | man, all ones = free
  uint16_t *cut;      // [n]: word >> 16, what the scans compare with
  uint16_t *at;       // [n]: the entry of his list a man has reached (his wife, or his last rejection)
  int32_t *parkq[2];  // [n]
  int cap;
};

__host__ __device__ constexpr size_t round_words(int n) { return (static_cast<size_t>(n) + 7) & ~static_cast<size_t>(7); }
__host__ __device__ constexpr int round_cap(int n) {
  return n < kCand ? static_cast<int>(round_words(n)) : kCand;
}
__host__ __device__ constexpr size_t round_bitmap_bytes(int n) {
  return (round_words(n) / 8 + 15) & ~static_cast<size_t>(15);
}
constexpr int kBallots = kScanUnroll * (kTeam / 32);             // of one team and scan step
constexpr size_t kBallotBytes = 2 * kBallots * sizeof(uint32_t);  // of two scan steps
// Shared memory: the resolver's words and list entries; a scanner's cut-offs
// and, per team, a bitmap and its ballots.
__host__ __device__ constexpr size_t round_smem_bytes(int n) {
  const size_t resolve = round_words(n) * 6;
  const size_t scan = round_words(n) * 2 + kTeams * (round_bitmap_bytes(n) + kBallotBytes);
  return resolve > scan ? resolve : scan;
}

// With the resolver's table of the list entry after each man's position.
__host__ __device__ constexpr size_t round_table_bytes(int n) {
  const size_t resolve = round_words(n) * 10;
  return resolve > round_smem_bytes(n) ? resolve : round_smem_bytes(n);
}

// Every woman free, no man started, the first men in step 0's slot.  A
// rank-mode solve whose first choices are all distinct is finished here.
__global__ void __launch_bounds__(1024) k_round_reset(const int32_t *__restrict__ pref_m, RoundBufs b,
                                                      int32_t *__restrict__ match, int n, int batch, Control *ctrl,
                                                      int gate) {
  if (gate == kGateModeRank && ld_volatile_s32(&ctrl->perfect) && ld_volatile_s32(&ctrl->mode) == kModeRank) {
    write_perfect(pref_m, match, n, ctrl);
    return;
  }
  if (!gate_open(gate, ctrl)) return;
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < static_cast<int>(round_words(n)); i += stride) {
    b.word[i] = 0xFFFFFFFFu;
    b.cut[i] = 0xFFFFu;
    b.at[i] = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    RoundCtl c = {};
    c.slot[0].new1 = min(n, batch);
    *b.ctl = c;
  }
}

__device__ __forceinline__ void team_sync(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeam) : "memory");
}

// The i-th man of a step's scan.
__device__ __forceinline__ int round_item(const RoundSlot &slot, const int32_t *__restrict__ parkq,
                                          const int32_t *__restrict__ order, int i, bool &started) {
  started = true;
  if (slot.refresh) return i;
  if (i < slot.parked) return parkq[i];
  started = false;
  return __ldg(order + slot.new0 + (i - slot.parked));
}

// Scans a step's men, one per team of kTeam threads at a time.  The man's
// row of rankT is compared with the women's cut-offs (both in index order:
// 16-byte loads) into a bitmap of the women who would take him; his
// preference row then streams past it, and the women whose bit is set are
// kept in order, up to cap, with their ranks.  A man who holds a woman keeps
// her as entry 0.
__device__ __forceinline__ void round_scan(const int32_t *__restrict__ pref_m, const uint16_t *__restrict__ rankT,
                                           size_t ld, const int32_t *__restrict__ order, const RoundBufs &b,
                                           const RoundSlot &slot, const int32_t *__restrict__ parkq, int items, int n,
                                           unsigned char *smem, Control *ctrl) {
  static_assert(kBallots == 64, "two ballots per lane");
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int team = tid / kTeam;
  const int tt = tid % kTeam;
  const int tw = tt >> 5;
  const int nw = static_cast<int>(round_words(n));
  const int cap = b.cap;
  uint16_t *cut = reinterpret_cast<uint16_t *>(smem);
  unsigned char *bits =
      smem + static_cast<size_t>(nw) * 2 + static_cast<size_t>(team) * (round_bitmap_bytes(n) + kBallotBytes);
  const uint32_t *bitw = reinterpret_cast<const uint32_t *>(bits);
  uint32_t *ballots = reinterpret_cast<uint32_t *>(bits + round_bitmap_bytes(n));
  // (the resolver writes word[], cut[] and at[] later in this launch: no ld.nc)
  uint4 *cut4 = reinterpret_cast<uint4 *>(cut);
  const int chunks = nw / 8;
#pragma unroll 4
  for (int i = tid; i < chunks; i += kRoundBlock) cut4[i] = __ldcg(reinterpret_cast<const uint4 *>(b.cut) + i);
  __syncthreads();
  for (int i = static_cast<int>(blockIdx.x) * kTeams + team; i < items; i += static_cast<int>(gridDim.x) * kTeams) {
    bool started;
    const int m = round_item(slot, parkq, order, i, started);
    uint32_t *out = b.cand + static_cast<size_t>(m) * cap;
    uint16_t *outp = b.cpos + static_cast<size_t>(m) * cap;
    int start = 0, count = 0;
    if (started) {
      const int k = __ldcg(b.at + m);
      const uint32_t e = out[k];
      const int p = outp[k];
      team_sync(team);  // read before the list is written over
      start = p + 1;
      if ((__ldcg(b.word + (e >> 16)) & 0xFFFFu) == static_cast<uint32_t>(m)) {  // she holds him
        if (tt == 0) {
          out[0] = e;
          outp[0] = static_cast<uint16_t>(p);
        }
        count = 1;
      }
    }
    const uint4 *rr = reinterpret_cast<const uint4 *>(rankT + static_cast<size_t>(m) * ld);
    for (int c0 = tt; c0 < chunks; c0 += 4 * kTeam) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + k * kTeam;
        v[k] = c < chunks ? __ldcs(rr + c) : make_uint4(~0u, ~0u, ~0u, ~0u);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + k * kTeam;
        if (c < chunks) {
          const uint4 q = cut4[c];
          const uint32_t rv[4] = {v[k].x, v[k].y, v[k].z, v[k].w}, qv[4] = {q.x, q.y, q.z, q.w};
          uint32_t byte = 0;
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            byte |= ((rv[h] & 0xFFFFu) < (qv[h] & 0xFFFFu) ? 1u : 0u) << (2 * h);
            byte |= ((rv[h] >> 16) < (qv[h] >> 16) ? 1u : 0u) << (2 * h + 1);
          }
          bits[c] = static_cast<unsigned char>(byte);
        }
      }
    }
    const int32_t *row = pref_m + static_cast<size_t>(m) * n;
    const uint16_t *rrow = rankT + static_cast<size_t>(m) * ld;
    int wv[kScanUnroll];
#pragma unroll
    for (int u = 0; u < kScanUnroll; ++u) {
      const int r = start + u * kTeam + tt;
      wv[u] = r < n ? __ldcs(row + r) : 0;
    }
    team_sync(team);  // the bitmap is complete
    int buf = 0;
    bool bad = false;
    int bad_value = 0;
    for (int base = start; base < n && count < cap; base += kScanUnroll * kTeam) {
      uint32_t mine[kScanUnroll];
      int cur[kScanUnroll];
#pragma unroll
      for (int u = 0; u < kScanUnroll; ++u) {
        const int r = base + u * kTeam + tt;
        const int w = wv[u];
        bool hit = false;
        if (r < n) {
          if (static_cast<unsigned>(w) < static_cast<unsigned>(n)) {
            hit = (bitw[w >> 5] >> (w & 31)) & 1u;
          } else {
            bad = true;
            bad_value = w;
          }
        }
        cur[u] = w;
        mine[u] = __ballot_sync(kFullMask, hit);
      }
#pragma unroll
      for (int u = 0; u < kScanUnroll; ++u) {  // the next step's entries
        const int r = base + (kScanUnroll + u) * kTeam + tt;
        wv[u] = r < n ? __ldcs(row + r) : 0;
      }
      if (lane == 0) {
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) ballots[kBallots * buf + u * (kTeam / 32) + tw] = mine[u];
      }
      team_sync(team);
      // candidates before each ballot, in list order
      const int low = __popc(ballots[kBallots * buf + lane]);  // ballots lane and 32 + lane
      const int high = __popc(ballots[kBallots * buf + 32 + lane]);
      int incl = low | (high << 16);  // both halves in one scan: at most 1024 each
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(kFullMask, incl, off);
        if (lane >= off) incl += v;
      }
      const int sums = __shfl_sync(kFullMask, incl, 31);
      const int total = (sums & 0xFFFF) + (sums >> 16);
      if (total) {
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
          const int idx = u * (kTeam / 32) + tw;
          const int both = __shfl_sync(kFullMask, incl, idx & 31);
          const int through = idx < 32 ? both & 0xFFFF : (sums & 0xFFFF) + (both >> 16);
          const int at = count + through - __popc(mine[u]) + __popc(mine[u] & ((1u << lane) - 1u));
          if (((mine[u] >> lane) & 1u) && at < cap) {
            out[at] = (static_cast<uint32_t>(cur[u]) << 16) | __ldg(rrow + cur[u]);
            outp[at] = static_cast<uint16_t>(base + u * kTeam + tt);
          }
        }
      }
      count += total;
      buf ^= 1;
    }
    // the end of a list that has room left: one window, all any chain reads past it
    if (tt < 32 && count + tt < cap) out[count + tt] = kNoCand;
    // entry 0 is his wife, or none before it has been tried: also what a
    // resolver that reads at[m] too early may see
    if (tt == 0) b.at[m] = 0;
    if (bad) report(ctrl, kStatusInvalidInput, bad_value);
    team_sync(team);  // before the next man's bitmap
  }
}

// Every entry of pref_m is range-checked once, whatever the solve needs of
// it: the whole rows of the men a step starts.  The CTAs that do not resolve
// take them in turn after they have handed their lists over.
__device__ __forceinline__ void round_check(const int32_t *__restrict__ pref_m, const int32_t *__restrict__ order,
                                            int begin, int end, int32_t *taken, int n, Control *ctrl) {
  __shared__ int s_row;
  const int tid = threadIdx.x;
  bool bad = false;
  int bad_value = 0;
  const auto look = [&](int v) {
    if (static_cast<unsigned>(v) >= static_cast<unsigned>(n)) {
      bad = true;
      bad_value = v;
    }
  };
  for (;;) {
    if (tid == 0) s_row = begin + atomicAdd(taken, 1);
    __syncthreads();
    const int i = s_row;
    __syncthreads();
    if (i >= end) break;
    const RowSpan s = row_span(pref_m, __ldg(order + i), n);
    if (tid < s.head) look(__ldcs(s.row + tid));
    for (int k = tid; k < s.nq; k += kRoundBlock) {
      const int4 q = __ldcs(s.rq + k);
      look(q.x);
      look(q.y);
      look(q.z);
      look(q.w);
    }
    if (tid < s.tail) look(__ldcs(s.row + s.head + 4 * s.nq + tid));
  }
  if (bad) report(ctrl, kStatusInvalidInput, bad_value);
}

// The words and list entries between global and shared memory.
__device__ __forceinline__ void round_state_in(const RoundBufs &b, uint32_t *sbid, uint16_t *spos, int nw) {
#pragma unroll 4
  for (int i = threadIdx.x; i < nw / 4; i += kRoundBlock)
    reinterpret_cast<uint4 *>(sbid)[i] = __ldcg(reinterpret_cast<const uint4 *>(b.word) + i);
#pragma unroll 4
  for (int i = threadIdx.x; i < nw / 8; i += kRoundBlock)
    reinterpret_cast<uint4 *>(spos)[i] = __ldcg(reinterpret_cast<const uint4 *>(b.at) + i);
}

// match[] and the proposal count, after every chain has ended.
__device__ __forceinline__ void round_finish(const RoundBufs &b, const uint32_t *sbid, const uint16_t *spos,
                                             int32_t *__restrict__ match, int n, Control *ctrl,
                                             unsigned long long *s_props) {
  unsigned long long props = 0;
  for (int w = threadIdx.x; w < n; w += kRoundBlock) {
    const uint32_t word = sbid[w];
    if (word == 0xFFFFFFFFu) {
      report(ctrl, kStatusInvalidInput, w);
      continue;
    }
    match[word & 0xFFFFu] = w;
  }
  for (int m = threadIdx.x; m < n; m += kRoundBlock)
    props += __ldcg(b.cpos + static_cast<size_t>(m) * b.cap + spos[m]) + 1ull;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) props += __shfl_down_sync(kFullMask, props, off);
  if ((threadIdx.x & 31) == 0) atomicAdd(s_props, props);
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->proposals = *s_props;
    ctrl->bulk_proposals = *s_props;
  }
}

// What the chains of a step work on.
struct RoundChains {
  const int32_t *order;
  const int32_t *parkq;
  RoundBufs b;
  RoundSlot slot;
  uint32_t *sbid;   // shared: the women's words
  uint16_t *spos;   // shared: the entries the men have reached
  uint32_t *snext;  // shared, chains_by_warp: the entries after those
  int32_t *park;    // the men parked for the next step
  int *s_next, *s_parked, *s_stop;
  int ready, n;
  Control *ctrl;
};

// Displacements, and proposals that met someone better who had just got there.
struct RoundCount {
  unsigned int hops, lost;
};

// A chain per warp.  kTable: with a table of the list entry after each man's
// position; a man dropped tries it without a look at his list, 0.1 us on a
// displacement instead of 0.5.  That pays in a refresh step, where every list
// is new, his wife its first entry, and the one after it most often takes him.
// (With the table in every step, RANDOM(5) n = 15013 took 6.4 ms for 4.0 and
// correlated n = 30000 10.6 for 8.6: filling it reads a line per man, it takes
// L1 from the scans, and two entries in five had been overtaken.)  Counts in
// lane 0.
template <bool kTable>
__device__ __forceinline__ RoundCount chains_by_warp(const RoundChains &q) {
  const int n = q.n;
  const int cap = q.b.cap;
  const int lane = threadIdx.x & 31;
  uint32_t *sbid = q.sbid;
  uint16_t *spos = q.spos;
  uint32_t *snext = q.snext;
  if (kTable) {
    if (q.slot.refresh) {
#pragma unroll 8
      for (int i = threadIdx.x; i < n; i += kRoundBlock) {
        const int r = spos[i] + 1;
        snext[i] = r < cap ? q.b.cand[static_cast<uint32_t>(i * cap + r)] : kNoCand;
      }
    } else {
      for (int i = threadIdx.x; i < n; i += kRoundBlock) snext[i] = kNoCand;
    }
    __syncthreads();
  }
  unsigned int hops = 0, lost = 0;
  int m = -1, pos = 0;    // the man and the list entry to try next
  uint32_t raw = 0;       // this lane's entry pos + lane of his list
  uint32_t one = kNoCand;  // kTable: entry pos, where the table has it (raw is not read then)
  const auto entry = [&](int man, int r) { return r < cap ? q.b.cand[static_cast<uint32_t>(man * cap + r)] : kNoCand; };
  // Moves on to the first window at or after pos that holds a candidate or
  // the end of the list, looking at kWide windows per round trip.
  const auto skip = [&]() {
    for (;;) {
      uint32_t rv[kWide];
#pragma unroll
      for (int u = 0; u < kWide; ++u) rv[u] = entry(m, pos + 32 * u + lane);
      int hit = -1;
#pragma unroll
      for (int u = 0; u < kWide; ++u) {
        // entries past a list's end window are leftovers: any index below n will do
        const uint32_t w = min(rv[u] >> 16, static_cast<uint32_t>(n - 1));
        const uint32_t word = lds_relaxed_u32(sbid + w);
        if (__any_sync(kFullMask, rv[u] == kNoCand || (rv[u] & 0xFFFFu) < (word >> 16)) && hit < 0) {
          hit = u;
          raw = rv[u];
        }
      }
      if (hit >= 0) {
        pos += 32 * hit;
        return;
      }
      pos += 32 * kWide;
    }
  };
  const auto next_man = [&]() {
    int i = 0;
    if (lane == 0) i = *reinterpret_cast<volatile int *>(q.s_stop) ? q.ready : atomicAdd(q.s_next, 1);
    i = __shfl_sync(kFullMask, i, 0);
    if (i >= q.ready) return false;
    m = i < q.slot.parked ? q.parkq[i] : __ldg(q.order + q.slot.new0 + (i - q.slot.parked));
    pos = 0;
    one = kNoCand;
    skip();
    return true;
  };
  for (bool more = next_man(); more;) {
    if (kTable && one != kNoCand) {
      const uint32_t rk = one & 0xFFFFu;
      uint32_t old = 0;
      if (lane == 0) {
        spos[m] = static_cast<uint16_t>(pos);
        snext[m] = kNoCand;
        old = atom_min_relaxed_shared(sbid + (one >> 16), (rk << 16) | static_cast<uint32_t>(m));
      }
      old = __shfl_sync(kFullMask, old, 0);
      if ((old >> 16) > rk) {
        hops++;
        if (old == 0xFFFFFFFFu) {
          more = next_man();
          continue;
        }
        m = static_cast<int>(old & 0xFFFFu);
        pos = spos[m] + 1;
        one = snext[m];
        if (one != kNoCand) continue;
      } else {
        one = kNoCand;
        pos++;
      }
      raw = entry(m, pos + lane);
    }
    const bool ok = raw != kNoCand;  // a window past a list's end holds nothing else
    const int w = ok ? static_cast<int>(raw >> 16) : 0;
    const uint32_t rk = raw & 0xFFFFu;
    const uint32_t cur = ok ? lds_relaxed_u32(sbid + w) : 0u;
    const uint32_t hp = (ok && cur != 0xFFFFFFFFu) ? spos[cur & 0xFFFFu] : 0u;
    const unsigned cm = __ballot_sync(kFullMask, ok && rk < (cur >> 16));
    if (cm == 0) {
      const unsigned end = __ballot_sync(kFullMask, !ok);
      if (end) {
        if (pos + __ffs(end) - 1 < cap) {  // the list held every woman left: rejected by all of them
          if (lane == 0) {
            report(q.ctrl, kStatusInvalidInput, m);
            *q.s_stop = 1;
          }
          break;
        }
        if (lane == 0) {
          spos[m] = static_cast<uint16_t>(cap - 1);
          q.park[atomicAdd(q.s_parked, 1)] = m;
        }
        more = next_man();
      } else {
        pos += 32;
        skip();
      }
      continue;
    }
    const int j = __ffs(cm) - 1;
    const unsigned long long info =
        __shfl_sync(kFullMask, (static_cast<unsigned long long>(hp | (rk << 16)) << 32) | cur, j);
    const uint32_t hw = static_cast<uint32_t>(info);
    const int hm = static_cast<int>(hw & 0xFFFFu);
    const int hpos = static_cast<int>((info >> 32) & 0xFFFFu) + 1;
    const uint32_t rkj = static_cast<uint32_t>(info >> 48);
    // the window of the man she would drop, while the proposal is under way
    uint32_t next_raw = 0;
    if (hw != 0xFFFFFFFFu) next_raw = entry(hm, hpos + lane);
    uint32_t old = 0;
    const uint32_t after = kTable ? __shfl_down_sync(kFullMask, raw, 1) : kNoCand;
    if (lane == j) {
      spos[m] = static_cast<uint16_t>(pos + j);
      if (kTable) snext[m] = j < 31 ? after : kNoCand;
      old = atom_min_relaxed_shared(sbid + w, (rk << 16) | static_cast<uint32_t>(m));
    }
    old = __shfl_sync(kFullMask, old, j);
    if (old == hw && (old >> 16) > rkj && hw != 0xFFFFFFFFu) {
      hops++;
      m = hm;
      pos = hpos;
      raw = next_raw;
      if (kTable) one = snext[m];
      continue;
    }
    if ((old >> 16) <= rkj) {  // someone better got there first: read the bids again
      lost++;
      continue;
    }
    hops++;
    if (old == 0xFFFFFFFFu) {
      more = next_man();  // the chain ended at a free woman
      continue;
    }
    m = static_cast<int>(old & 0xFFFFu);
    pos = spos[m] + 1;
    raw = entry(m, pos + lane);
    if (kTable) one = snext[m];
  }
  return lane == 0 ? RoundCount{hops, lost} : RoundCount{0, 0};
}

// A chain per eight lanes, four in a warp: a window of a list is 16 bytes per
// lane.  At 32 chains the SM's issue slots were the bound (0.58 us on a
// displacement), here a step's longest chain is (70 windows of 0.74 us where
// the mean is 30 of 1.1): correlated n = 30000 8.6 -> 7.9 ms, n = 8000 1.54 ->
// 1.37, SOLO n = 10007 3.3 -> 3.0.  Counts in the first lane of each eight.
//   Where lists are old a window rejects him whole, and eight lanes take as long
// for it as a warp for eight.  A group that has passed more than kDeepWindows
// windows and kDeepPerHop a displacement parks its man at the next one: he is
// scanned again, and where all men have started so is everyone.  (Where n is not
// above kCand no list runs out, so nothing else would park him: SOLO n = 600,
// one chain that passes nine windows a displacement, took 5.9 ms for 1.1.)
constexpr unsigned int kDeepWindows = 32;
constexpr unsigned int kDeepPerHop = 4;
__device__ __forceinline__ RoundCount chains_by_group(const RoundChains &q) {
  const int n = q.n;
  const int cap = q.b.cap;
  const int lane = threadIdx.x & 31;
  const int gl = lane & 7;
  const int g0 = lane & 24;
  uint32_t *sbid = q.sbid;
  uint16_t *spos = q.spos;
  const auto window = [&](int man, int pos) {  // from the 16-byte boundary at or before pos
    const int r = (pos & ~3) + 4 * gl;
    return r < cap ? *reinterpret_cast<const uint4 *>(q.b.cand + static_cast<uint32_t>(man * cap + r))
                   : make_uint4(kNoCand, kNoCand, kNoCand, kNoCand);
  };
  unsigned int hops = 0, lost = 0, passed = 0;
  bool has = false, out = false;  // a man; no more of them
  bool fresh = false;             // his window is still to be loaded
  int m = 0, pos = 0;             // the man and the list entry to try next
  uint4 v = make_uint4(kNoCand, kNoCand, kNoCand, kNoCand);
  for (;;) {
    const bool ask = !has && !out;
    if (__any_sync(kFullMask, ask)) {
      int i = 0;
      if (ask && gl == 0) i = *reinterpret_cast<volatile int *>(q.s_stop) ? q.ready : atomicAdd(q.s_next, 1);
      i = __shfl_sync(kFullMask, i, g0);
      if (ask) {
        has = i < q.ready;
        out = !has;
        fresh = has;
        if (has) m = i < q.slot.parked ? q.parkq[i] : __ldg(q.order + q.slot.new0 + (i - q.slot.parked));
        pos = 0;
      }
    }
    if (!__any_sync(kFullMask, has)) break;
    if (fresh) v = window(m, pos);
    fresh = false;
    const int at = (pos & ~3) + 4 * gl;
    const uint32_t e[4] = {v.x, v.y, v.z, v.w};
    int f = -1;              // this lane's first entry that takes him, and her word
    uint32_t fe = 0, fw = 0;
    bool end = false;
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      // (a window past a list's end holds nothing else; leftovers are not reached)
      const uint32_t word = lds_relaxed_u32(sbid + min(e[k] >> 16, static_cast<uint32_t>(n - 1)));
      end |= e[k] == kNoCand;
      if (at + k >= pos && e[k] != kNoCand && (e[k] & 0xFFFFu) < (word >> 16)) {
        f = k;
        fe = e[k];
        fw = word;
      }
    }
    const unsigned hits = (__ballot_sync(kFullMask, has && f >= 0) >> g0) & 0xFFu;
    const unsigned ends = (__ballot_sync(kFullMask, has && end) >> g0) & 0xFFu;
    const unsigned short_end = (__ballot_sync(kFullMask, has && end && at < cap) >> g0) & 0xFFu;
    const bool found = hits != 0;
    const int src = found ? g0 + __ffs(hits) - 1 : lane;
    const uint32_t rk = __shfl_sync(kFullMask, fe, src) & 0xFFFFu;
    const uint32_t hw = __shfl_sync(kFullMask, fw, src);
    if (has && !found) {
      pos = (pos & ~3) + 32;  // every entry before it has rejected him
      if (!ends && ++passed <= kDeepWindows + kDeepPerHop * hops) {
        fresh = true;
      } else {
        if (gl == 0) {
          if (short_end) {  // the list held every woman left: rejected by all of them
            report(q.ctrl, kStatusInvalidInput, m);
            *q.s_stop = 1;
          } else {
            spos[m] = static_cast<uint16_t>(min(pos, cap) - 1);
            q.park[atomicAdd(q.s_parked, 1)] = m;
          }
        }
        has = false;
      }
    }
    // the window of the man she would drop, while the proposal is under way
    int hpos = 0;
    uint4 hv = v;
    if (found && hw != 0xFFFFFFFFu) {
      hpos = spos[hw & 0xFFFFu] + 1;
      hv = window(static_cast<int>(hw & 0xFFFFu), hpos);
    }
    uint32_t old = 0;
    if (found && lane == src) {
      spos[m] = static_cast<uint16_t>(at + f);
      old = atom_min_relaxed_shared(sbid + (fe >> 16), (fe << 16) | static_cast<uint32_t>(m));
    }
    old = __shfl_sync(kFullMask, old, src);
    if (found && (old >> 16) <= rk) lost++;  // someone better got there first: read the bids again
    if (found && (old >> 16) > rk) {
      hops++;
      has = old != 0xFFFFFFFFu;  // else the chain ended at a free woman
      m = static_cast<int>(old & 0xFFFFu);
      if (old == hw) {
        pos = hpos;
        v = hv;
      } else if (has) {
        pos = spos[m] + 1;
        fresh = true;
      }
    }
  }
  return gl == 0 ? RoundCount{hops, lost} : RoundCount{0, 0};
}

// One step.  kTable: the steps past the first ceil(n / batch), by which all men
// may have started, if the table fits.  The others work their chains by warp
// or by eight lanes, as the step before found the men calm or crowded.  Where
// many make for the same women, four times the chains at a time triple the
// displacements (RANDOM(5) n = 15013: 101 to 308 thousand, 4.0 to 6.4 ms) and
// a quarter of the proposals come too late; in correlated lists one in 200
// does by warp and one in 50 by eight lanes.
constexpr unsigned int kCalmWarp = 64;   // fewer than one in so many late
constexpr unsigned int kCalmGroup = 16;
template <bool kTable>
__global__ void __launch_bounds__(kRoundBlock, 1)
    k_round(const int32_t *__restrict__ pref_m, const uint16_t *__restrict__ rankT, size_t ld,
            const int32_t *__restrict__ order, RoundBufs b, int32_t *__restrict__ match, int n, int batch, int t,
            Control *ctrl, int gate) {
  __shared__ int s_go;
  __shared__ int s_next, s_parked, s_stop;
  __shared__ unsigned long long s_props;
  __shared__ unsigned int s_hops, s_lost;
  const int tid = threadIdx.x;
  if (tid == 0) s_go = gate_open(gate, ctrl) && !ld_volatile_s32(&b.ctl->done);
  __syncthreads();  // read once: another CTA may report an error meanwhile
  if (!s_go) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const RoundSlot slot = b.ctl->slot[t & 1];
  const int32_t *parkq = b.parkq[t & 1];
  const int ready = slot.parked + (slot.new1 - slot.new0);
  const int items = slot.refresh ? n : ready;
  if (static_cast<int>(blockIdx.x) * kTeams < items)
    round_scan(pref_m, rankT, ld, order, b, slot, parkq, items, n, smem_raw, ctrl);
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    s_go = atomicAdd(&b.ctl->arrived[t & 1], 1) == static_cast<int>(gridDim.x) - 1;
    s_next = 0;
    s_parked = 0;
    s_stop = 0;
    s_props = 0;
    s_hops = 0;
    s_lost = 0;
  }
  __syncthreads();
  if (!s_go) {
    round_check(pref_m, order, slot.new0, slot.new1, &b.ctl->checked[t & 1], n, ctrl);
    return;
  }
  __threadfence();  // the other CTAs' lists
  // ---- the last CTA resolves ----
  const int nw = static_cast<int>(round_words(n));
  uint32_t *sbid = reinterpret_cast<uint32_t *>(smem_raw);
  uint16_t *spos = reinterpret_cast<uint16_t *>(smem_raw + static_cast<size_t>(nw) * 4);
  uint32_t *snext = reinterpret_cast<uint32_t *>(smem_raw + static_cast<size_t>(nw) * 6);  // kTable
  int32_t *park = b.parkq[(t & 1) ^ 1];
  round_state_in(b, sbid, spos, nw);
  __syncthreads();
  const RoundChains q = {order,   parkq,     b,       slot,  sbid, spos,
                         snext,   park,      &s_next, &s_parked, &s_stop, ready, n, ctrl};
  const bool calm = !kTable && b.ctl->calm > 0;
  const RoundCount count = kTable ? chains_by_warp<true>(q) : calm ? chains_by_group(q) : chains_by_warp<false>(q);
  if (count.hops) atomicAdd(&s_hops, count.hops);
  if (count.lost) atomicAdd(&s_lost, count.lost);
  __syncthreads();
  if (tid == 0 && ld_volatile_s32(&ctrl->status)) s_stop = 1;  // read once
  __syncthreads();
  if (s_stop) return;
  const int parked = s_parked;
  const bool done = parked == 0 && slot.new1 >= n;
  if (tid == 0) {
    RoundSlot nx;
    nx.parked = parked;
    nx.new0 = slot.new1;
    nx.new1 = min(n, slot.new1 + max(batch - parked, batch / 4));
    nx.refresh = parked > 0 && slot.new1 >= n;
    b.ctl->slot[(t & 1) ^ 1] = nx;
    b.ctl->arrived[(t & 1) ^ 1] = 0;
    b.ctl->checked[(t & 1) ^ 1] = 0;
    const bool few = s_lost * (calm ? kCalmGroup : kCalmWarp) < s_hops;
    if (few && b.ctl->calm == 0)
      b.ctl->calm = 1;
    else if (!few && calm)
      b.ctl->calm = -1;  // for good
    b.ctl->done = done;
    ctrl->round_done = done;
    ctrl->bulk_hops += s_hops;
  }
  if (done) {
    round_finish(b, sbid, spos, match, n, ctrl, &s_props);
  } else {
    for (int i = tid; i < nw / 4; i += kRoundBlock) {
      const uint4 v = reinterpret_cast<const uint4 *>(sbid)[i];
      reinterpret_cast<uint4 *>(b.word)[i] = v;
      reinterpret_cast<uint2 *>(b.cut)[i] = make_uint2(__byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x7632));
    }
    for (int i = tid; i < nw / 8; i += kRoundBlock)
      reinterpret_cast<uint4 *>(b.at)[i] = reinterpret_cast<const uint4 *>(spos)[i];
  }
}

// ---------------------------------------------------------------------------
// The last launch of the sequence, one CTA: if the steps did not finish the
// solve, every man still parked or not started is followed straight through
// the preference lists, so the sequence ends whatever the input.  A man's
// position is kept as entry 0 of his list from here on.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kRoundBlock, 1)
    k_round_last(const int32_t *__restrict__ pref_m, const uint16_t *__restrict__ rankT, size_t ld,
                 const int32_t *__restrict__ order, RoundBufs b, int32_t *__restrict__ match, int n, int t,
                 Control *ctrl, int gate) {
  if (!gate_open(gate, ctrl) || ld_volatile_s32(&b.ctl->done)) return;
  __shared__ int s_next, s_stop;
  __shared__ unsigned long long s_props;
  __shared__ unsigned int s_hops;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int nw = static_cast<int>(round_words(n));
  uint32_t *sbid = reinterpret_cast<uint32_t *>(smem_raw);
  uint16_t *spos = reinterpret_cast<uint16_t *>(smem_raw + static_cast<size_t>(nw) * 4);
  const RoundSlot slot = b.ctl->slot[t & 1];
  const int32_t *parkq = b.parkq[t & 1];
  const int total = slot.parked + (n - slot.new0);
  round_state_in(b, sbid, spos, nw);
  if (tid == 0) {
    s_next = 0;
    s_stop = 0;
    s_props = 0;
    s_hops = 0;
  }
  __syncthreads();
  unsigned int hops = 0;
  int m = -1, from = 0;
  const auto next_man = [&]() {
    int i = 0;
    if (lane == 0) i = atomicAdd(&s_next, 1);
    i = __shfl_sync(kFullMask, i, 0);
    if (i >= total) return false;
    if (i < slot.parked) {
      m = parkq[i];
      from = __ldcg(b.cpos + static_cast<size_t>(m) * b.cap + spos[m]) + 1;
    } else {
      m = __ldg(order + slot.new0 + (i - slot.parked));
      from = 0;
    }
    return true;
  };
  for (bool more = next_man(); more;) {
    if (warp_flag(&s_stop)) break;
    const int32_t *row = pref_m + static_cast<size_t>(m) * n;
    const uint16_t *rrow = rankT + static_cast<size_t>(m) * ld;
    bool taken = false;
    for (; from < n && !taken; from += 32) {
      const int r = from + lane;
      const int w = r < n ? __ldg(row + r) : 0;
      const bool valid = static_cast<unsigned>(w) < static_cast<unsigned>(n);
      if (__any_sync(kFullMask, !valid)) break;
      const uint32_t rk = __ldg(rrow + w);
      unsigned cm = __ballot_sync(kFullMask, r < n && rk < (lds_relaxed_u32(sbid + w) >> 16));
      while (cm) {
        const int j = __ffs(cm) - 1;
        uint32_t old = 0;
        if (lane == j) {
          b.cpos[static_cast<size_t>(m) * b.cap] = static_cast<uint16_t>(r);
          spos[m] = 0;
          __threadfence_block();
          old = atom_min_relaxed_shared(sbid + w, (rk << 16) | static_cast<uint32_t>(m));
          __threadfence_block();
        }
        old = __shfl_sync(kFullMask, old, j);
        const uint32_t rkj = __shfl_sync(kFullMask, rk, j);
        __syncwarp();  // the displaced man's position, as lane j would see it
        if ((old >> 16) > rkj) {
          hops++;
          taken = true;
          if (old == 0xFFFFFFFFu) {
            more = next_man();
          } else {
            m = static_cast<int>(old & 0xFFFFu);
            from = __ldcg(b.cpos + static_cast<size_t>(m) * b.cap + spos[m]) + 1;
          }
          from -= 32;  // the loop's step
          break;
        }
        cm &= cm - 1;  // someone better got there first
      }
    }
    if (!taken) {  // an entry out of range, or rejected by every woman
      if (lane == 0) {
        report(ctrl, kStatusInvalidInput, m);
        s_stop = 1;
      }
      break;
    }
  }
  if (lane == 0 && hops) atomicAdd(&s_hops, hops);
  __syncthreads();
  if (s_stop) return;
  if (tid == 0) {
    b.ctl->done = 1;
    ctrl->round_done = 1;
    ctrl->bulk_hops += s_hops;
  }
  round_finish(b, sbid, spos, match, n, ctrl, &s_props);
  // the rows of the men who never started a step
  round_check(pref_m, order, slot.new0, n, &b.ctl->checked[t & 1], n, ctrl);
}

}  // namespace smpb200
