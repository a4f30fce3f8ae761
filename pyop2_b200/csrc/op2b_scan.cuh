// Device-wide exclusive prefix sum of int32 counts, used by the plan, Sparsity,
// row block and partition builders: totals of 4096-item chunks, then every CTA
// scans its chunk from the sum of the totals before it (from 4 million items on
// these are scanned by one CTA in between).  In-place (out == in) is allowed:
// every CTA reads its chunk before it writes it.  Both passes move 16 bytes per
// lane, neighbouring lanes on neighbouring bytes: 1.0 million counts take 7 us,
// where a scan, its totals and a pass that adds them took 25 with 64 bytes
// between lanes.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "op2b_internal.h"

namespace op2b {

constexpr int kScanThreads = 256;
constexpr int kScanChunk = 16 * kScanThreads;

__device__ __forceinline__ int warp_incl_scan(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive scan of one value per thread across the CTA; returns the CTA total
// in *total.  blockDim.x must be a multiple of 32 and at most 1024.
__device__ __forceinline__ int block_excl_scan(int v, int *total) {
  __shared__ int warp_tot[33];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  int incl = warp_incl_scan(v);
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int w = lane < nw ? warp_tot[lane] : 0;
    int wi = warp_incl_scan(w);
    if (lane < nw) warp_tot[lane] = wi - w;
    if (lane == nw - 1) warp_tot[32] = wi;
  }
  __syncthreads();
  int res = incl - v + warp_tot[wid];
  int tot = warp_tot[32];
  __syncthreads();
  *total = tot;
  return res;
}

// The chunk's items 4 * (k * kScanThreads + thread) .. + 3 for k = 0 .. 3.
template <bool V4>
__device__ __forceinline__ void scan_load(const int *in, int64_t base, int64_t n, int (&v)[4][4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = base + 4 * (k * kScanThreads + (int)threadIdx.x);
    if (V4 && i + 4 <= n) {
      const int4 w = *reinterpret_cast<const int4 *>(in + i);
      v[k][0] = w.x, v[k][1] = w.y, v[k][2] = w.z, v[k][3] = w.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[k][j] = i + j < n ? in[i + j] : 0;
    }
  }
}

template <bool V4>
static __global__ void __launch_bounds__(kScanThreads) scan_totals_kernel(const int *in, int *sums, int64_t n) {
  int v[4][4], s = 0, total;
  scan_load<V4>(in, (int64_t)blockIdx.x * kScanChunk, n, v);
#pragma unroll
  for (int k = 0; k < 4; ++k) s += v[k][0] + v[k][1] + v[k][2] + v[k][3];
  block_excl_scan(s, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// scanned: sums holds the totals' exclusive scan (and *total is set), else the
// totals.
template <bool V4>
static __global__ void __launch_bounds__(kScanThreads)
scan_chunk_kernel(const int *in, int *out, const int *sums, int64_t n, bool scanned, int *total) {
  __shared__ int row_warp[4][kScanThreads / 32];
  const int64_t base = (int64_t)blockIdx.x * kScanChunk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int v[4][4], sum[4], incl[4];
  scan_load<V4>(in, base, n, v);
  int before = 0;
  if (scanned) {
    before = sums[blockIdx.x];
  } else {
    int s = 0;
    for (int j = threadIdx.x; j < (int)blockIdx.x; j += kScanThreads) s += sums[j];
    block_excl_scan(s, &before);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    sum[k] = v[k][0] + v[k][1] + v[k][2] + v[k][3];
    incl[k] = warp_incl_scan(sum[k]);
    if (lane == 31) row_warp[k][wid] = incl[k];
  }
  __syncthreads();
  int carry = before;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    int pre = carry + incl[k] - sum[k];
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
      const int r = row_warp[k][w];
      if (w < wid) pre += r;
      carry += r;
    }
    const int64_t i = base + 4 * (k * kScanThreads + (int)threadIdx.x);
    const int4 w = make_int4(pre, pre + v[k][0], pre + v[k][0] + v[k][1], pre + v[k][0] + v[k][1] + v[k][2]);
    if (V4 && i + 4 <= n) {
      *reinterpret_cast<int4 *>(out + i) = w;
    } else {
      if (i < n) out[i] = w.x;
      if (i + 1 < n) out[i + 1] = w.y;
      if (i + 2 < n) out[i + 2] = w.z;
      if (i + 3 < n) out[i + 3] = w.w;
    }
  }
  if (!scanned && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total = carry;
}

// One CTA: exclusive scan of the chunk totals in place; grand total to *total.
static __global__ void scan_sums_kernel(int *sums, int nchunks, int *total) {
  int carry = 0;
  for (int start = 0; start < nchunks; start += blockDim.x) {
    int i = start + threadIdx.x;
    int v = i < nchunks ? sums[i] : 0;
    int t;
    int pre = block_excl_scan(v, &t);
    if (i < nchunks) sums[i] = pre + carry;
    carry += t;
  }
  if (threadIdx.x == 0) *total = carry;
}

// out[i] = sum(in[0..i)); *d_total (device int) receives the grand total.
// Needs scratch of (n/4096 + 1) ints, allocated here stream-ordered.
inline int device_excl_scan(const int *in, int *out, int64_t n, int *d_total, cudaStream_t s) {
  if (n <= 0) {
    OP2B_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
    return OP2B_OK;
  }
  const int nchunks = (int)((n + kScanChunk - 1) / kScanChunk);
  int *sums = nullptr;
  int rc = dev_alloc((void **)&sums, sizeof(int) * (size_t)nchunks, s);
  if (rc) return rc;
  const bool v4 = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const bool scanned = nchunks > 1024;
  if (v4) scan_totals_kernel<true><<<nchunks, kScanThreads, 0, s>>>(in, sums, n);
  else scan_totals_kernel<false><<<nchunks, kScanThreads, 0, s>>>(in, sums, n);
  if (scanned) scan_sums_kernel<<<1, 1024, 0, s>>>(sums, nchunks, d_total);
  if (v4) scan_chunk_kernel<true><<<nchunks, kScanThreads, 0, s>>>(in, out, sums, n, scanned, d_total);
  else scan_chunk_kernel<false><<<nchunks, kScanThreads, 0, s>>>(in, out, sums, n, scanned, d_total);
  dev_free(sums, s);
  OP2B_CUDA(cudaGetLastError());
  return OP2B_OK;
}

}  // namespace op2b
