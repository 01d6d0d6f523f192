// check_kernels.cuh -- the stability checker (no counterpart in the reference):
// counts the blocking pairs of a matching, and its proposals (the sum over
// men of the wife's position + 1).
//
// A pair (m, w) blocks if w comes before m's wife in his list and m before
// w's husband in hers.  Whether she would take him is one bit:
//   k_check_husband   husband[w] = m for match[m] = w (husband preset to -1);
//                     a woman matched twice or an out-of-range wife is reported
//   k_check_bits      bits[w][m] = woman w ranks m above her husband: her row is
//                     inverted in shared memory, as in the rank inversion, and
//                     compared with her husband's rank on its way out; a row
//                     that is not a permutation is reported
//   k_check_near      a warp per man walks the start of his list
//   k_check_transpose bitsT[m][w], so that a longer walk reads one row of bits
//   k_check_scan      and goes on with those who have not met their wife yet
// pref_w is read once, n^2 / 8 bytes of bits are written, transposed and read.
// With the rank matrix in the bits' place the scan read her 2-byte rank of him
// from her row, a 32-byte sector for every entry: n = 12007 correlated took
// 1.24 ms; with bits 0.37, and with two ranks compared per subtraction 0.33.
// Uniform n = 8464, where near choices are all there are: 0.175 ms with the
// transpose, 0.144 without (rank matrix: 0.15).
//   Above n = 65535 a row does not fit shared memory: k_check_prank and
// k_check_scan_rank read the int32 rank matrix.
#pragma once

#include "common.cuh"
#include "solve_kernels.cuh"

namespace smpb200 {

__global__ void k_check_husband(const int32_t *__restrict__ match, int32_t *husband, int n, Control *ctrl) {
  const int stride = gridDim.x * blockDim.x;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += stride) {
    const int w = match[m];
    if (static_cast<unsigned>(w) >= static_cast<unsigned>(n) || atomicExch(husband + w, m) != -1)
      report(ctrl, kStatusInvalidInput, w);
  }
}

// Bytes per row of bits: whole 32-byte sectors.
__host__ __device__ constexpr size_t check_row_bytes(int n) {
  return ((static_cast<size_t>(n) + 255) / 256) * 32;
}

__global__ void __launch_bounds__(512) k_check_bits(const int32_t *__restrict__ pref_w,
                                                    const int32_t *__restrict__ husband,
                                                    unsigned char *__restrict__ bits, int n, Control *ctrl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint16_t *srow = reinterpret_cast<uint16_t *>(smem_raw);
  const uint4 *s4 = reinterpret_cast<const uint4 *>(smem_raw);
  const int chunks = (n + 7) / 8;
  const int row_bytes = static_cast<int>(check_row_bytes(n));
  bool bad = false;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    load_row(pref_w + static_cast<size_t>(w) * n, srow, srow, chunks, n, bad);
    const int h = __ldg(husband + w);
    const uint32_t limit = static_cast<unsigned>(h) < static_cast<unsigned>(n) ? srow[h] : 0u;
    bad |= static_cast<unsigned>(h) >= static_cast<unsigned>(n);
    unsigned char *out = bits + static_cast<size_t>(w) * row_bytes;
    if (n <= kColorMaxN) {
      // ranks take 15 bits: bit 15 says that a slot is unset, and, set before
      // the subtraction, which of two ranks is below the limit
      const uint32_t lim2 = limit | (limit << 16);
      for (int c = threadIdx.x; c < row_bytes; c += blockDim.x) {
        uint32_t byte = 0;
        if (c < chunks) {
          const uint4 v = s4[c];
          uint32_t unset = (v.x | v.y | v.z | v.w) & 0x80008000u;
          const uint32_t x = (~((v.x | 0x80008000u) - lim2) & 0x80008000u) >> 15 |
                             (~((v.y | 0x80008000u) - lim2) & 0x80008000u) >> 13 |
                             (~((v.z | 0x80008000u) - lim2) & 0x80008000u) >> 11 |
                             (~((v.w | 0x80008000u) - lim2) & 0x80008000u) >> 9;
          byte = (x & 0x55u) | ((x >> 15) & 0xAAu);
          const int left = n - 8 * c;
          if (left < 8) {  // slots past n keep the fill
            byte &= (1u << left) - 1u;
            const uint32_t q[4] = {v.x, v.y, v.z, v.w};
            unset = 0;
            for (int k = 0; k < left; ++k) unset |= (k & 1 ? q[k >> 1] >> 16 : q[k >> 1]) & 0x8000u;
          }
          bad |= unset != 0;
        }
        out[c] = static_cast<unsigned char>(byte);
      }
    } else {
      for (int c = threadIdx.x; c < row_bytes; c += blockDim.x) {
        uint32_t byte = 0;
        if (c < chunks) {
          const uint4 v = s4[c];
          const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t r = k & 1 ? q[k >> 1] >> 16 : q[k >> 1] & 0xFFFFu;
            if (c * 8 + k < n) bad |= r == 0xFFFFu;  // a slot no entry named
            byte |= (r < limit ? 1u : 0u) << k;      // slots past n keep the fill, 0xFFFF
          }
        }
        out[c] = static_cast<unsigned char>(byte);
      }
    }
    __syncthreads();
  }
  if (bad) report(ctrl, kStatusInvalidInput, -1);
}

// 256 x 256 bits per CTA: a 32-byte sector per row in and out.  A warp turns
// 32 x 32 bits over in five exchange steps.
__global__ void __launch_bounds__(256) k_check_transpose(const unsigned char *__restrict__ bits,
                                                         unsigned char *__restrict__ bits_t, int n,
                                                         const Control *ctrl) {
  if (!ld_volatile_s32(&ctrl->check_deep)) return;
  __shared__ uint32_t tile[8][256];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int v = tid >> 5;
  const size_t row_bytes = check_row_bytes(n);
  const int r0 = blockIdx.y * 256;  // rows read, columns written
  const int c0 = blockIdx.x * 256;
  uint4 a = make_uint4(0, 0, 0, 0), b = a;
  if (r0 + tid < n) {
    const uint4 *src = reinterpret_cast<const uint4 *>(bits + static_cast<size_t>(r0 + tid) * row_bytes + c0 / 8);
    a = src[0];
    b = src[1];
  }
  const uint32_t in[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int k = 0; k < 8; ++k) tile[k][tid] = in[k];
  __syncthreads();
  uint32_t out[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    uint32_t x = tile[v][32 * k + lane];
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int j = 16; j; j >>= 1) {
      const uint32_t y = __shfl_xor_sync(kFullMask, x, j);
      x = (lane & j) ? (((y >> j) & mask) | (x & ~mask)) : (((y << j) & ~mask) | (x & mask));
      mask ^= mask << (j >> 1);
    }
    out[k] = x;
  }
  const int row = c0 + 32 * v + lane;
  if (row < n) {
    uint4 *dst = reinterpret_cast<uint4 *>(bits_t + static_cast<size_t>(row) * row_bytes + r0 / 8);
    dst[0] = make_uint4(out[0], out[1], out[2], out[3]);
    dst[1] = make_uint4(out[4], out[5], out[6], out[7]);
  }
}

// A warp per man, in two kernels.  k_check_near walks his first kCheckNear
// choices with the bits as they are, 32 bytes of L2 each: uniform lists end
// there, and where all do the transpose is not made.  k_check_scan goes on with
// the others (deep[m] set), the man's row of bits in shared memory and 256
// choices in flight.  A first choice out of range is reported; entries after
// the wife count for nothing.
constexpr int kCheckWarps = 8;
constexpr int kCheckNear = 128;

__device__ __forceinline__ void check_sums(unsigned long long blocking, unsigned long long props, Control *ctrl) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    blocking += __shfl_down_sync(kFullMask, blocking, off);
    props += __shfl_down_sync(kFullMask, props, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (blocking) atomicAdd(&ctrl->blocking, blocking);
    if (props) atomicAdd(&ctrl->check_proposals, props);
  }
}

__global__ void __launch_bounds__(32 * kCheckWarps) k_check_near(const int32_t *__restrict__ pref_m,
                                                                 const unsigned char *__restrict__ bits,
                                                                 const int32_t *__restrict__ match,
                                                                 unsigned char *__restrict__ deep, int n,
                                                                 Control *ctrl) {
  const int lane = threadIdx.x & 31;
  const size_t row_bytes = check_row_bytes(n);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long blocking = 0, props = 0;
  for (int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < n; m += warps) {
    const int wife = __ldg(match + m);
    const int32_t *row = pref_m + static_cast<size_t>(m) * n;
    int found = -1;  // the wife's position
    for (int base = 0; base < min(n, kCheckNear) && found < 0; base += 32) {
      const int r = base + lane;
      const int w = r < n ? __ldg(row + r) : -1;
      const unsigned hit = __ballot_sync(kFullMask, r < n && w == wife);
      if (hit) found = base + __ffs(hit) - 1;
      if (r < n && (found < 0 || r < found)) {
        if (static_cast<unsigned>(w) < static_cast<unsigned>(n))
          blocking += (__ldg(bits + static_cast<size_t>(w) * row_bytes + (m >> 3)) >> (m & 7)) & 1u;
        else if (r == 0)
          report(ctrl, kStatusInvalidInput, w);
      }
    }
    if (lane == 0) {
      deep[m] = found < 0 && n > kCheckNear;
      if (found >= 0)
        props += static_cast<unsigned long long>(found + 1);
      else if (n > kCheckNear)
        ctrl->check_deep = 1;
      else
        report(ctrl, kStatusInvalidInput, m);
    }
  }
  check_sums(blocking, props, ctrl);
}

__global__ void __launch_bounds__(32 * kCheckWarps) k_check_scan(const int32_t *__restrict__ pref_m,
                                                                 const unsigned char *__restrict__ bits_t,
                                                                 const int32_t *__restrict__ match,
                                                                 const unsigned char *__restrict__ deep, int n,
                                                                 Control *ctrl) {
  if (!ld_volatile_s32(&ctrl->check_deep)) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int row_bytes = static_cast<int>(check_row_bytes(n));
  uint4 *srow = reinterpret_cast<uint4 *>(smem_raw + static_cast<size_t>(threadIdx.x >> 5) * row_bytes);
  const uint32_t *sbits = reinterpret_cast<const uint32_t *>(srow);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long blocking = 0, props = 0;
  for (int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < n; m += warps) {
    if (!deep[m]) continue;
    const int wife = __ldg(match + m);
    const int32_t *row = pref_m + static_cast<size_t>(m) * n;
    const uint4 *brow = reinterpret_cast<const uint4 *>(bits_t + static_cast<size_t>(m) * row_bytes);
    int w[8], next[8];
    const auto load = [&](int base, int (&to)[8]) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = base + 32 * u + lane;
        to[u] = r < n ? __ldg(row + r) : -1;
      }
    };
    load(kCheckNear, w);
    __syncwarp();
    for (int i = lane; i < row_bytes / 16; i += 32) srow[i] = __ldg(brow + i);
    __syncwarp();
    int found = -1;
    for (int base = kCheckNear; base < n && found < 0; base += 256) {
      load(base + 256, next);  // (all past n at the end)
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = base + 32 * u + lane;
        const unsigned hit = __ballot_sync(kFullMask, r < n && w[u] == wife);
        if (found < 0 && hit) found = base + 32 * u + __ffs(hit) - 1;
        if ((found < 0 || r < found) && static_cast<unsigned>(w[u]) < static_cast<unsigned>(n))
          blocking += (sbits[w[u] >> 5] >> (w[u] & 31)) & 1u;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) w[u] = next[u];
    }
    if (lane == 0) {
      if (found < 0)
        report(ctrl, kStatusInvalidInput, m);
      else
        props += static_cast<unsigned long long>(found + 1);
    }
  }
  check_sums(blocking, props, ctrl);
}

__global__ void k_check_prank(const int32_t *__restrict__ husband, const int32_t *__restrict__ rank,
                              int32_t *__restrict__ prank, int n, Control *ctrl) {
  const int stride = gridDim.x * blockDim.x;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += stride) {
    const int h = husband[w];
    if (h < 0) {
      report(ctrl, kStatusInvalidInput, w);
      prank[w] = -1;
      continue;
    }
    prank[w] = static_cast<int32_t>(rank[static_cast<size_t>(w) * n + h]);
  }
}

__global__ void k_check_scan_rank(const int32_t *__restrict__ pref_m, const int32_t *__restrict__ rank,
                             const int32_t *__restrict__ match, const int32_t *__restrict__ prank, int n,
                             Control *ctrl) {
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  unsigned long long blocking = 0, props = 0;
  for (int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < n; m += warps) {
    const int wife = match[m];
    const int32_t *row = pref_m + static_cast<size_t>(m) * n;
    bool found = false;
    for (int base = 0; base < n && !found; base += 32) {
      const int r = base + lane;
      const int w = r < n ? __ldg(row + r) : -1;
      const unsigned hit = __ballot_sync(kFullMask, r < n && w == wife);
      const int limit = hit ? (__ffs(hit) - 1) : 32;  // lanes before the wife
      if (lane < limit && r < n && static_cast<unsigned>(w) < static_cast<unsigned>(n)) {
        const int32_t pr = prank[w];
        if (pr >= 0 && static_cast<int32_t>(rank[static_cast<size_t>(w) * n + m]) < pr) blocking++;
      }
      if (hit) {
        found = true;
        if (lane == 0) props += static_cast<unsigned long long>(base + limit + 1);
      }
    }
    if (!found && lane == 0) report(ctrl, kStatusInvalidInput, m);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    blocking += __shfl_down_sync(kFullMask, blocking, off);
    props += __shfl_down_sync(kFullMask, props, off);
  }
  if (lane == 0) {
    if (blocking) atomicAdd(&ctrl->blocking, blocking);
    if (props) atomicAdd(&ctrl->check_proposals, props);
  }
}

}  // namespace smpb200
