// batch_kernels.cuh -- many independent instances in one persistent launch.
//
// The reference solves one instance per engine object
// (benchmark/smp_engine_exec.h:6-32); a batch here is a device table of
// instances that CTAs pull from a queue, largest first.  One CTA solves one
// instance at a time, start to finish:
//   1. inversion: the women's rows become a uint16 rank matrix -- in shared
//      memory when it fits the CTA's rank region (small instances), else in
//      the CTA's own slab in global memory -- and are checked to be
//      permutations;
//   2. proposals: the bid words (rank << 16 | man) and each man's position
//      live in shared memory, and warps follow displacement chains exactly as
//      the single-instance tail kernel does, looking ahead up to kMaxSub
//      windows of 32 choices per step;
//   3. match[m] = w, the proposal count and a status go back to the table.
// The same kernel launched with one instance per launch is the plain
// per-instance baseline the batched launch is measured against.
#pragma once

#include "common.cuh"
#include "smp_b200.h"
#include "step.cuh"

namespace smpb200 {

// Device-side row of the instance table (the host mirrors smp_instance).
struct BatchInstance {
  const int32_t *pref_m;
  const int32_t *pref_w;
  int32_t *match;
  int32_t n;
  int32_t status;
  unsigned long long proposals;
};

// Shared memory for one instance of size n: bids and positions, padded to
// 16 bytes; the rank region for small instances follows.
__host__ __device__ constexpr size_t batch_smem_bytes(int max_n) {
  return (static_cast<size_t>(max_n) * 4 + static_cast<size_t>(max_n) * 2 + 15) & ~static_cast<size_t>(15);
}

// Rank rows are padded to a multiple of 8 entries (16 bytes).
__host__ __device__ __forceinline__ int batch_ld(int n) { return (n + 7) & ~7; }

// Entries of one CTA's slab: the padded rank matrix of the largest instance,
// then what a hard instance keeps per man (batch_hard): its candidate list and
// the starting order, both ways round.
constexpr int kHardCand = 64;
__host__ __device__ __forceinline__ size_t batch_slab_elems(int max_n) {
  const size_t ld = static_cast<size_t>(batch_ld(max_n));
  return ld * max_n + ld * kHardCand * (sizeof(uint2) / sizeof(uint16_t)) + 2 * ld;
}

// Inversion of pref_w through a shared buffer of `elems` slots, in groups of
// as many rows as fit it.  The buffer is the image of the group's rank rows:
// the CTA streams the group's entries, one contiguous span of pref_w, with
// 16-byte loads, scatters each rank to its slot, and copies the image to the
// slab 16 bytes at a time (kStore), checking that every slot was written.
// The k-th group writes rank | (k & 1) << 15, so a slot it missed keeps the
// other colour and the image needs no clearing (n <= 16384 here).  The next
// group's first loads are under way while the image is copied out.  A matrix
// that fits the buffer whole is left in it (one group, colour 0).
//   What bounds it is the latency of one CTA's loads and the random 2-byte
// shared stores.  Groups of at most one row per warp, cleared before and with
// no loads ahead, took 7.0 ms for n = 4096 (67 MB) on one 512-thread CTA; this
// takes 3.5 with 4 loads ahead and 3.2 with 8 (2.9 with 1024 threads).
constexpr int kBatchAhead = 8;  // 16-byte loads per thread under way between groups

// kNum: man m's rank goes to column num[m] (shared memory) instead of m.
template <bool kStore, bool kNum = false>
__device__ __forceinline__ void batch_invert(const int32_t *__restrict__ pref_w, uint16_t *slab, int n, uint16_t *buf,
                                             int elems, bool &bad, const uint16_t *num = nullptr) {
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  const int ld = batch_ld(n);
  const int G = min(elems / ld, n);
  const uint32_t by_n = 0xFFFFFFFFu / static_cast<uint32_t>(n) + 1;  // e / n = umulhi(e, by_n) for e < 2^17 (n > 1)
  const int row_chunks = ld / 8;
  uint4 *b4 = reinterpret_cast<uint4 *>(buf);
  const auto put = [&](int e, int v, uint32_t cbit) {  // entry e of the group
    const int g = n > 1 ? static_cast<int>(__umulhi(static_cast<uint32_t>(e), by_n)) : e;
    if (static_cast<unsigned>(v) < static_cast<unsigned>(n))
      buf[g * ld + (kNum ? num[v] : v)] = static_cast<uint16_t>(static_cast<uint32_t>(e - g * n) | cbit);
    else
      bad = true;
  };
  const auto put4 = [&](int e, int4 q, uint32_t cbit) {
    int g = n > 1 ? static_cast<int>(__umulhi(static_cast<uint32_t>(e), by_n)) : e;
    int r = e - g * n;
    const uint32_t v[4] = {static_cast<uint32_t>(q.x), static_cast<uint32_t>(q.y), static_cast<uint32_t>(q.z),
                           static_cast<uint32_t>(q.w)};
    if (r + 4 <= n && max(max(v[0], v[1]), max(v[2], v[3])) < static_cast<uint32_t>(n)) {
      uint16_t *row = buf + g * ld;
      const uint32_t first = static_cast<uint32_t>(r) | cbit;
#pragma unroll
      for (int k = 0; k < 4; ++k) row[kNum ? num[v[k]] : v[k]] = static_cast<uint16_t>(first + k);
      return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (v[k] < static_cast<uint32_t>(n))
        buf[g * ld + (kNum ? num[v[k]] : v[k])] = static_cast<uint16_t>(static_cast<uint32_t>(r) | cbit);
      else
        bad = true;
      if (++r == n) {
        r = 0;
        ++g;
      }
    }
  };
  struct Span {
    const int32_t *p;
    const int4 *q;
    int head, nq, count;
  };
  const auto span_of = [&](int w0) {
    Span s;
    s.p = pref_w + static_cast<size_t>(w0) * n;
    s.count = min(G, n - w0) * n;
    s.head = min(s.count, static_cast<int>(((16u - (reinterpret_cast<uintptr_t>(s.p) & 15u)) & 15u) >> 2));
    s.q = reinterpret_cast<const int4 *>(s.p + s.head);
    s.nq = (s.count - s.head) >> 2;
    return s;
  };
  int4 a[kBatchAhead];
  int edge = 0;  // one of the at most 6 entries outside the 16-byte chunks
  const auto ahead = [&](const Span &s) {
#pragma unroll
    for (int j = 0; j < kBatchAhead; ++j) {
      const int i = tid + j * nthr;
      a[j] = i < s.nq ? __ldcs(s.q + i) : make_int4(0, 0, 0, 0);
    }
    const int rest = s.count - 4 * s.nq;
    if (tid < rest) edge = __ldcs(s.p + (tid < s.head ? tid : 4 * s.nq + tid));
  };
  Span s = span_of(0);
  ahead(s);
  for (int c = tid; c < G * row_chunks; c += nthr) b4[c] = make_uint4(~0u, ~0u, ~0u, ~0u);
  __syncthreads();
  uint32_t cbit = 0;
  for (int w0 = 0; w0 < n; w0 += G, cbit ^= 0x8000u) {
#pragma unroll
    for (int j = 0; j < kBatchAhead; ++j) {
      const int i = tid + j * nthr;
      if (i < s.nq) put4(s.head + 4 * i, a[j], cbit);
    }
    if (tid < s.count - 4 * s.nq) put(tid < s.head ? tid : 4 * s.nq + tid, edge, cbit);
    int i = tid + kBatchAhead * nthr;
    for (; i + 3 * nthr < s.nq; i += 4 * nthr) {
      int4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = __ldcs(s.q + i + j * nthr);
#pragma unroll
      for (int j = 0; j < 4; ++j) put4(s.head + 4 * (i + j * nthr), v[j], cbit);
    }
    for (; i < s.nq; i += nthr) put4(s.head + 4 * i, __ldcs(s.q + i), cbit);
    __syncthreads();
    const int rows = min(G, n - w0);
    if (w0 + G < n) {
      s = span_of(w0 + G);
      ahead(s);
    }
    const uint32_t want = cbit | (cbit << 16);
    uint4 *out = reinterpret_cast<uint4 *>(slab + static_cast<size_t>(w0) * ld);
    for (int c = tid; c < rows * row_chunks; c += nthr) {
      uint4 v = b4[c];
      const int left = n - 8 * (c % row_chunks);
      uint32_t m[4] = {0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u};
      if (left < 8) {  // slots past n hold anything
#pragma unroll
        for (int h = 0; h < 4; ++h) m[h] = (2 * h < left ? 0x8000u : 0u) | (2 * h + 1 < left ? 0x80000000u : 0u);
      }
      bad |= (((v.x ^ want) & m[0]) | ((v.y ^ want) & m[1]) | ((v.z ^ want) & m[2]) | ((v.w ^ want) & m[3])) != 0u;
      if (kStore) {
        v.x &= 0x7FFF7FFFu;
        v.y &= 0x7FFF7FFFu;
        v.z &= 0x7FFF7FFFu;
        v.w &= 0x7FFF7FFFu;
        out[c] = v;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Hard instances: fewer than n / 4 distinct first choices, too large for the
// shared rank region.  Their men reject hundreds of women per acceptance, and
// reading her 2-byte rank of him from her row costs a 32-byte sector per
// rejection: n = 4096, sigma = 0.05 took 11.9 ms on one 512-thread CTA, 8.5
// this way (6.4 with 1024 threads), n = 1024 1.01 and 0.68 ms.  One CTA does
// here what the rounds of a single solve do on all SMs (round_kernels.cuh):
//   - the men are numbered in the order the women like them (the sum of their
//     ranks with 32 women), and the inversion writes column num[m];
//   - 64 men at a time, in that order: their columns, contiguous in every row
//     of the slab, are compared with the women's cut-offs and turned over by
//     ballots into one row of bits per man in shared memory;
//   - a warp per man streams his list past his bits and keeps the first
//     kHardCand women who would take him, with rank and position;
//   - warps follow the displacement chains through these lists.  Every entry
//     of a list that has rejected him once rejects him again, so a displaced
//     man's list is simply tried from its start; a man whose list is used up
//     goes on in his preference row.
// The lists also stop at an entry out of range, which counts only if a chain
// reaches it.
// ---------------------------------------------------------------------------
constexpr int kHardMen = 64;       // men per round at most
constexpr int kHardSamples = 32;
constexpr int kHardBuckets = 1024;
constexpr int kHardMinRegion = 16384;  // shared rank entries it needs (32 KB)
constexpr uint32_t kHardNone = 0xFFFFFFFFu;
constexpr uint32_t kHardBad = 0xFFFFFFFEu;

// Orders the men: num (shared) and the same in global memory with its inverse.
__device__ __forceinline__ void hard_order(const int32_t *__restrict__ pref_w, uint32_t *score, uint16_t *num,
                                           uint32_t *hist, uint16_t *ord_g, uint16_t *num_g, int n) {
  const int tid = threadIdx.x;
  const int nthr = blockDim.x;
  for (int m = tid; m < n; m += nthr) score[m] = 0;
  for (int i = tid; i < kHardBuckets; i += nthr) hist[i] = 0;
  __syncthreads();
  for (int i = 0; i < kHardSamples; ++i) {
    const int32_t *row = pref_w + static_cast<size_t>(order_sample(i, kHardSamples, n)) * n;
    for (int r = tid; r < n; r += nthr) {
      const int m = __ldg(row + r);
      if (static_cast<unsigned>(m) < static_cast<unsigned>(n)) atomicAdd(score + m, static_cast<uint32_t>(r));
    }
  }
  __syncthreads();
  const auto bucket = [&](int m) {  // score < 32 n <= 2^19
    return min(static_cast<uint32_t>(kHardBuckets - 1), score[m] * (kHardBuckets / kHardSamples) / static_cast<uint32_t>(n));
  };
  for (int m = tid; m < n; m += nthr) atomicAdd(hist + bucket(m), 1u);
  __syncthreads();
  if (tid < 32) {
    uint32_t sum = 0;
    for (int k = 0; k < kHardBuckets / 32; ++k) sum += hist[tid * (kHardBuckets / 32) + k];
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(kFullMask, incl, off);
      if (tid >= off) incl += v;
    }
    uint32_t at = incl - sum;
    for (int k = 0; k < kHardBuckets / 32; ++k) {
      const uint32_t c = hist[tid * (kHardBuckets / 32) + k];
      hist[tid * (kHardBuckets / 32) + k] = at;
      at += c;
    }
  }
  __syncthreads();
  for (int m = tid; m < n; m += nthr) {
    const uint32_t at = atomicAdd(hist + bucket(m), 1u);
    num[m] = static_cast<uint16_t>(at);
    num_g[m] = static_cast<uint16_t>(at);
    ord_g[at] = static_cast<uint16_t>(m);
  }
  __syncthreads();
}

// The proposals, after the inversion and with every woman free.  status is
// set where an invalid entry is reached.
__device__ __forceinline__ void batch_hard(const int32_t *__restrict__ pref_m, const uint16_t *slab, uint2 *list,
                                           const uint16_t *ord_g, const uint16_t *num_g, uint32_t *sbid,
                                           uint16_t *spos, uint32_t *bits, int bit_words, int n, int *next,
                                           volatile int *status) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  const int ld = batch_ld(n);
  const int stride = ((n + 31) / 32) | 1;  // words per man's bits: odd, so 32 men's words fall in 32 banks
  const int men = min(kHardMen, bit_words / stride) & ~7;
  for (int i0 = 0; i0 < n; i0 += men) {
    const int nb = min(men, n - i0);
    if (tid == 0) *next = 0;
    // bits of 32 women x 32 men at a time: a lane holds her ranks of them
    for (int blk = warp; blk * 32 < n; blk += nwarps) {
      const int w = blk * 32 + lane;
      const uint32_t cut = w < n ? sbid[w] >> 16 : 0u;
      const uint16_t *ranks = slab + static_cast<size_t>(w < n ? w : 0) * ld + i0;
      for (int h = 0; h < nb; h += 32) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          v[q] = h + 8 * q < nb ? *reinterpret_cast<const uint4 *>(ranks + h + 8 * q) : make_uint4(~0u, ~0u, ~0u, ~0u);
        uint32_t mine = 0;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
          const uint4 &q = v[k >> 3];
          const uint32_t word = (k >> 1 & 3) == 0 ? q.x : (k >> 1 & 3) == 1 ? q.y : (k >> 1 & 3) == 2 ? q.z : q.w;
          const unsigned b = __ballot_sync(kFullMask, (k & 1 ? word >> 16 : word & 0xFFFFu) < cut);
          if (lane == k) mine = b;
        }
        if (h + lane < men) bits[(h + lane) * stride + blk] = mine;
      }
    }
    __syncthreads();
    for (int j = warp; j < nb; j += nwarps) {
      const int m = ord_g[i0 + j];
      const int32_t *row = pref_m + static_cast<size_t>(m) * n;
      const uint32_t *mb = bits + j * stride;
      uint2 *out = list + static_cast<size_t>(m) * kHardCand;
      int found = 0;
      for (int base = 0; base < n && found < kHardCand; base += 512) {
        int w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int r = base + 32 * u + lane;
          w[u] = r < n ? __ldg(row + r) : 0;
        }
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int r = base + 32 * u + lane;
          const bool off = static_cast<unsigned>(w[u]) >= static_cast<unsigned>(n);
          const bool hit = r < n && (off || ((mb[w[u] >> 5] >> (w[u] & 31)) & 1u));
          const unsigned mask = __ballot_sync(kFullMask, hit);
          const int at = found + __popc(mask & ((1u << lane) - 1u));
          if (hit && at < kHardCand)
            out[at] = make_uint2(off ? kHardBad
                                     : (static_cast<uint32_t>(w[u]) << 16) | slab[static_cast<size_t>(w[u]) * ld + i0 + j],
                                 static_cast<uint32_t>(r));
          found += __popc(mask);
        }
      }
      for (int k = found + lane; k < kHardCand; k += 32) out[k] = make_uint2(kHardNone, kHardNone);
    }
    __syncthreads();
    int m = -1;
    uint2 e0 = make_uint2(kHardNone, kHardNone), e1 = e0;
    const auto load = [&](int man, uint2 &a, uint2 &b) {
      a = list[static_cast<size_t>(man) * kHardCand + lane];
      b = list[static_cast<size_t>(man) * kHardCand + 32 + lane];
    };
    const auto next_man = [&]() {
      int i = 0;
      if (lane == 0) i = *status ? nb : atomicAdd(next, 1);
      i = __shfl_sync(kFullMask, i, 0);
      if (i >= nb) return false;
      m = ord_g[i0 + i];
      load(m, e0, e1);
      return true;
    };
    for (bool more = next_man(); more;) {
      const bool in0 = e0.x < kHardBad, in1 = e1.x < kHardBad;
      const uint32_t w0 = in0 ? lds_relaxed_u32(sbid + (e0.x >> 16)) : 0u;
      const uint32_t w1 = in1 ? lds_relaxed_u32(sbid + (e1.x >> 16)) : 0u;
      const unsigned c0 = __ballot_sync(kFullMask, e0.x == kHardBad || (e0.x & 0xFFFFu) < (w0 >> 16));
      const unsigned c1 = __ballot_sync(kFullMask, e1.x == kHardBad || (e1.x & 0xFFFFu) < (w1 >> 16));
      uint32_t word, pick = 0, r = 0;
      uint2 n0 = e0, n1 = e1;
      if (c0 | c1) {
        const int src = __ffs(c0 ? c0 : c1) - 1;
        pick = __shfl_sync(kFullMask, c0 ? e0.x : e1.x, src);
        r = __shfl_sync(kFullMask, c0 ? e0.y : e1.y, src);
        word = __shfl_sync(kFullMask, c0 ? w0 : w1, src);
        if (pick == kHardBad) {
          if (lane == 0) *status = SMP_ERR_INVALID_INPUT;
          break;
        }
        // the list of the man she would drop, while the proposal is under way
        if (word != 0xFFFFFFFFu) load(static_cast<int>(word & 0xFFFFu), n0, n1);
      } else {
        // used up: on in his preference row
        word = 0xFFFFFFFFu;
        const uint32_t end = __shfl_sync(kFullMask, e1.y, 31);
        bool stop = end == kHardNone;  // the list held every woman left
        const int32_t *row = pref_m + static_cast<size_t>(m) * n;
        const uint16_t *col = slab + num_g[m];
        int base = stop ? n : max(static_cast<int>(end), static_cast<int>(spos[m])) + 1;
        bool got = false;
        for (; base < n && !got && !stop; base += 128) {
          int w[4];
          uint32_t rk[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int at = base + 32 * u + lane;
            w[u] = at < n ? __ldg(row + at) : -1;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            rk[u] = static_cast<unsigned>(w[u]) < static_cast<unsigned>(n) ? col[static_cast<size_t>(w[u]) * ld] : 0xFFFFu;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int at = base + 32 * u + lane;
            const bool off = at < n && rk[u] == 0xFFFFu;
            const bool takes = rk[u] != 0xFFFFu && rk[u] < (lds_relaxed_u32(sbid + w[u]) >> 16);
            const unsigned hit = __ballot_sync(kFullMask, off || takes);
            if (hit && !got && !stop) {
              const int src = __ffs(hit) - 1;
              stop = __shfl_sync(kFullMask, off, src);
              got = !stop;
              pick = __shfl_sync(kFullMask, (static_cast<uint32_t>(w[u]) << 16) | rk[u], src);
              r = static_cast<uint32_t>(base + 32 * u + src);
            }
          }
        }
        if (!got) {  // an entry out of range, or rejected by every woman
          if (lane == 0) *status = SMP_ERR_INVALID_INPUT;
          break;
        }
      }
      const uint32_t rk = pick & 0xFFFFu;
      uint32_t old = 0;
      if (lane == 0) {
        spos[m] = static_cast<uint16_t>(r);
        old = atom_min_relaxed_shared(sbid + (pick >> 16), (rk << 16) | static_cast<uint32_t>(m));
      }
      old = __shfl_sync(kFullMask, old, 0);
      if ((old >> 16) <= rk) continue;  // someone better got there first
      if (old == 0xFFFFFFFFu) {
        more = next_man();
        continue;
      }
      m = static_cast<int>(old & 0xFFFFu);
      if (old == word) {
        e0 = n0;
        e1 = n1;
      } else {
        load(m, e0, e1);
      }
    }
    __syncthreads();
    if (*status) return;
  }
}

// rank_smem_elems: uint16 slots of shared memory after the bids; an instance
// whose n*n rank matrix fits there keeps it on chip (small instances), the
// others use the CTA's slab in global memory.
template <int kMaxSub>
__global__ void __launch_bounds__(1024, 1) k_batch(BatchInstance *__restrict__ table, const int32_t *__restrict__ order,
                                               int count, int *queue, uint16_t *__restrict__ slabs,
                                               size_t slab_elems, int max_n, int dynamic, int rank_smem_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint32_t *sbid = reinterpret_cast<uint32_t *>(smem_raw);
  uint16_t *spos = reinterpret_cast<uint16_t *>(smem_raw + static_cast<size_t>(max_n) * 4);
  uint16_t *srank = reinterpret_cast<uint16_t *>(smem_raw + batch_smem_bytes(max_n));
  __shared__ int s_idx;
  __shared__ int s_next_man;
  __shared__ int s_status;
  __shared__ int s_bad;
  __shared__ unsigned long long s_props;
  __shared__ int s_swap;
  __shared__ int s_distinct;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nwarps = blockDim.x >> 5;
  uint16_t *const slab = slabs + static_cast<size_t>(blockIdx.x) * slab_elems;

  for (int round = 0;; ++round) {
    if (tid == 0) s_idx = dynamic ? atomicAdd(queue, 1) : (round == 0 ? static_cast<int>(blockIdx.x) : count);
    __syncthreads();
    const int k = s_idx;
    if (k >= count) return;
    BatchInstance *inst = table + order[k];
    const int n = inst->n;
    const int32_t *pref_m = inst->pref_m;
    const int32_t *pref_w = inst->pref_w;
    if (n <= 0 || n > max_n || n > 65535) {
      if (tid == 0) {
        inst->status = SMP_ERR_UNSUPPORTED;
        inst->proposals = 0;
      }
      __syncthreads();
      continue;
    }
    uint16_t *const rank =
        static_cast<long long>(n) * batch_ld(n) <= static_cast<long long>(rank_smem_elems) ? srank : slab;
    if (tid == 0) {
      s_next_man = 0;
      s_status = 0;
      s_bad = 0;
      s_props = 0;
      s_distinct = 0;
      s_swap = 2 * n <= rank_smem_elems && n >= 16;  // n >= 16: a row fits the bid words' memory
    }
    __syncthreads();

    // 0. Do all men share one list?  Then the stable matching is unique --
    // woman pi_1 gets her favourite man, pi_2 her favourite of the rest, ...
    // -- so the women-proposing run finds the same matching, with about
    // n ln n proposals instead of the men's n (n + 1) / 2; and the men's
    // proposal count is n (n + 1) / 2, each woman's place in the shared list
    // counted once.  The first choices are screened first; the full
    // comparison reads pref_m once.
    volatile int *swap_flag = &s_swap;
    if (*swap_flag) {
      const int first = __ldg(pref_m);
      for (int m = tid; m < n; m += blockDim.x)
        if (__ldg(pref_m + static_cast<size_t>(m) * n) != first) *swap_flag = 0;
    }
    __syncthreads();
    uint16_t *const inv = srank;      // inv[w] = her place in the shared list
    uint16_t *const row0 = srank + n;  // the shared list
    if (s_swap) {
      for (int w = tid; w < n; w += blockDim.x) inv[w] = 0xFFFFu;
      __syncthreads();
      for (int r = tid; r < n; r += blockDim.x) {
        const int w = __ldg(pref_m + r);
        if (static_cast<unsigned>(w) < static_cast<unsigned>(n)) {
          row0[r] = static_cast<uint16_t>(w);
          inv[w] = static_cast<uint16_t>(r);
        } else {
          *swap_flag = 0;  // the ordinary path reports it
        }
      }
      __syncthreads();
      for (int w = tid; w < n; w += blockDim.x)
        if (inv[w] == 0xFFFFu) *swap_flag = 0;  // not a permutation: the ordinary path reports it
      for (int m = 1 + warp; m < n; m += nwarps) {
        int go = 0;
        if (lane == 0) go = *swap_flag;
        if (!__shfl_sync(kFullMask, go, 0)) break;  // the whole warp leaves together
        const int32_t *row = pref_m + static_cast<size_t>(m) * n;
        bool same = true;
        for (int r = lane; r < n; r += 32) same &= __ldg(row + r) == static_cast<int>(row0[r]);
        if (!__all_sync(kFullMask, same) && lane == 0) *swap_flag = 0;
      }
      __syncthreads();
    }
    if (s_swap) {
      // the women's lists must be permutations too: checked in groups of
      // rows through the bid words' shared memory, which is free until now
      bool bad = false;
      batch_invert<false>(pref_w, slab, n, reinterpret_cast<uint16_t *>(smem_raw),
                          static_cast<int>(batch_smem_bytes(max_n) / 2), bad);
      if (bad) s_status = SMP_ERR_INVALID_INPUT;
      __syncthreads();
      for (int m = tid; m < n; m += blockDim.x) {
        sbid[m] = 0xFFFFFFFFu;  // the men, holding no woman
        spos[m] = 0;            // the women's positions (a racing relaxed read sees 0, never leftovers)
      }
      __syncthreads();
      {
        // women propose down their lists; every man ranks a woman by her
        // place in the shared list
        const SharedBids bids{sbid, spos};
        const auto keep_going = [&]() { return !warp_flag(&s_status); };
        int m = -1, pos = 0, S = 1, bad_value = 0;
        Ahead ahead;
        unsigned long long settled = 0;
        unsigned int hops = 0;
        while (keep_going()) {
          if (m < 0) {
            int i = 0;
            if (lane == 0) i = atomicAdd(&s_next_man, 1);
            i = __shfl_sync(kFullMask, i, 0);
            if (i >= n) break;
            m = i;
            pos = 0;
            S = 1;
          }
          const int rc = man_step<kMaxSub, true, false, 1, 3>(bids, keep_going, pref_w,
                                                               static_cast<const uint16_t *>(inv),
                                                               static_cast<const uint32_t *>(nullptr), 0, n, false,
                                                               lane, m, pos, S, ahead, settled, hops, bad_value);
          if (rc == kStepMoved || rc == kStepMatchedFree) continue;
          if (rc == kStepBad && lane == 0) s_status = SMP_ERR_INVALID_INPUT;
          break;
        }
      }
      __syncthreads();
      if (!s_status)
        for (int m = tid; m < n; m += blockDim.x) {
          const uint32_t b = sbid[m];
          if (b == 0xFFFFFFFFu) {
            s_bad = 1;
            continue;
          }
          inst->match[m] = static_cast<int32_t>(b & 0xFFFFu);
        }
      __syncthreads();
      if (tid == 0) {
        inst->status = s_status ? s_status : (s_bad ? SMP_ERR_INVALID_INPUT : SMP_OK);
        inst->proposals = s_status || s_bad ? 0ull : static_cast<unsigned long long>(n) * (n + 1) / 2;
      }
      __syncthreads();
      continue;
    }
    // Hard: few distinct first choices, counted in a bitmap.
    bool hard = rank == slab && rank_smem_elems >= kHardMinRegion;
    if (hard) {
      uint32_t *seen = reinterpret_cast<uint32_t *>(srank);
      const int words = (n + 31) / 32;
      for (int i = tid; i < words; i += blockDim.x) seen[i] = 0;
      __syncthreads();
      for (int m = tid; m < n; m += blockDim.x) {
        const int w = __ldg(pref_m + static_cast<size_t>(m) * n);
        if (static_cast<unsigned>(w) < static_cast<unsigned>(n)) atomicOr(seen + (w >> 5), 1u << (w & 31));
      }
      __syncthreads();
      int some = 0;
      for (int i = tid; i < words; i += blockDim.x) some += __popc(seen[i]);
      if (some) atomicAdd(&s_distinct, some);
      __syncthreads();
      hard = 4 * s_distinct < n;
    }
    const size_t top = static_cast<size_t>(batch_ld(max_n));
    uint2 *const list = reinterpret_cast<uint2 *>(slab + top * max_n);
    uint16_t *const ord_g = slab + top * max_n + top * kHardCand * (sizeof(uint2) / sizeof(uint16_t));
    uint16_t *const num_g = ord_g + top;
    if (hard) {
      bool bad = false;
      hard_order(pref_w, sbid, spos, reinterpret_cast<uint32_t *>(srank), ord_g, num_g, n);
      batch_invert<true, true>(pref_w, slab, n, srank, rank_smem_elems, bad, spos);
      if (bad) s_status = SMP_ERR_INVALID_INPUT;
    }
    // Positions start at 0, so a relaxed read of a displaced man's position
    // that races with his own store returns an earlier position (resuming
    // there only repeats rejected proposals), never leftover shared memory.
    for (int w = tid; w < n; w += blockDim.x) {
      sbid[w] = 0xFFFFFFFFu;
      spos[w] = 0;
    }
    __syncthreads();

    // 1. inversion, through the shared region where it holds a row
    bool bad = false;
    const int ld = batch_ld(n);
    if (hard) {
      // done
    } else if (rank == srank) {
      batch_invert<false>(pref_w, slab, n, srank, rank_smem_elems, bad);
    } else if (rank_smem_elems >= ld) {
      batch_invert<true>(pref_w, slab, n, srank, rank_smem_elems, bad);
    } else {  // one row per warp, checked by reading it back
      for (int w = warp; w < n; w += nwarps) {
        const int32_t *row = pref_w + static_cast<size_t>(w) * n;
        uint16_t *out = rank + static_cast<size_t>(w) * ld;
        for (int r = lane; r < n; r += 32) {
          const int m = __ldg(row + r);
          if (static_cast<unsigned>(m) < static_cast<unsigned>(n)) {
            out[m] = static_cast<uint16_t>(r);
          } else {
            bad = true;
          }
        }
        __syncwarp();
        for (int r = lane; r < n; r += 32) {
          const int m = __ldg(row + r);
          if (static_cast<unsigned>(m) < static_cast<unsigned>(n) && out[m] != r) bad = true;
        }
      }
    }
    if (bad) s_status = SMP_ERR_INVALID_INPUT;
    __syncthreads();

    // 2. proposal chains, warp per free man (the step the tail kernel uses)
    if (hard) {
      if (!s_status)
        batch_hard(pref_m, slab, list, ord_g, num_g, sbid, spos, reinterpret_cast<uint32_t *>(srank),
                   rank_smem_elems / 2, n, &s_next_man, &s_status);
    } else {
      const SharedBids bids{sbid, spos};
      const auto keep_going = [&]() { return !warp_flag(&s_status); };
      int m = -1, pos = 0, S = 1, bad_value = 0;
      Ahead ahead;
      unsigned long long settled = 0;
      unsigned int hops = 0;
      while (keep_going()) {
        if (m < 0) {
          int i = 0;
          if (lane == 0) i = atomicAdd(&s_next_man, 1);
          i = __shfl_sync(kFullMask, i, 0);
          if (i >= n) break;
          m = i;
          pos = 0;
          S = 1;
        }
        const int rc = man_step<kMaxSub, true, false, 1, 4>(bids, keep_going, pref_m, static_cast<const uint16_t *>(rank),
                                                      static_cast<const uint32_t *>(nullptr),
                                         0, n, false, lane, m, pos, S, ahead, settled, hops, bad_value);
        if (rc == kStepMoved || rc == kStepMatchedFree) continue;
        if (rc == kStepBad && lane == 0) s_status = SMP_ERR_INVALID_INPUT;
        break;
      }
    }
    __syncthreads();

    // 3. outputs
    if (!s_status) {
      unsigned long long props = 0;
      for (int w = tid; w < n; w += blockDim.x) {
        const uint32_t b = sbid[w];
        if (b == 0xFFFFFFFFu) {
          s_bad = 1;
          continue;
        }
        inst->match[b & 0xFFFFu] = w;
      }
      for (int mm = tid; mm < n; mm += blockDim.x) props += spos[mm] + 1ull;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) props += __shfl_down_sync(kFullMask, props, off);
      if (lane == 0) atomicAdd(&s_props, props);
    }
    __syncthreads();
    if (tid == 0) {
      inst->status = s_status ? s_status : (s_bad ? SMP_ERR_INVALID_INPUT : SMP_OK);
      inst->proposals = s_status || s_bad ? 0ull : s_props;
    }
    __syncthreads();
  }
}

}  // namespace smpb200
