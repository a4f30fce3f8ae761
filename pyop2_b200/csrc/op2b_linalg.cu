// Linear algebra on the device CSR Mats and Dat vectors: sparse
// matrix-vector product, vector operations, reductions, and a
// Jacobi-preconditioned conjugate-gradient solve.
//
// Replaces the reference's PETSc KSP solve (pyop2/petsc_base.py:160-220,
// defaults linear_solver 'cg', preconditioner 'jacobi', pyop2/base.py:1591-
// 1601) and the Cusp CG of the CUDA backend (pyop2/cuda.py:445-600); the Dat
// arithmetic of pyop2/base.py:749-797 and Dat.norm (:836-839).
//
// Reductions are deterministic: each CTA reduces its share in a fixed order,
// and the partials are combined in CTA order by one CTA (or, inside the CG
// iteration, identically by every CTA that needs the total), so a result
// depends only on the data and the launch shape, never on scheduling.
//
// A CG solve is one cooperative launch: the iteration's scalars (alpha, beta,
// residual norms) are combined by every CTA from the same partials in the same
// order, so all of them take the same decisions, the solve stops at the exact
// iteration, and the host waits once.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "op2b_internal.h"

namespace op2b {

constexpr int kLinBlock = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the CTA in a fixed order; valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (wid == 0) {
    t = lane < nw ? scratch[lane] : 0.0;
    t = warp_sum(t);
  }
  return t;
}

// ------------------------------------------------------------------ SpMV
// One group of G lanes per row: strided partial products, then a shuffle
// tree inside the group (fixed order).
// Every lane of the warp must call it (the shuffles use the full mask): a
// lane past the last row passes live = false and contributes nothing.
template <int G>
__device__ __forceinline__ double row_dot(const int32_t *__restrict__ rowptr,
                                          const int32_t *__restrict__ colidx,
                                          const double *__restrict__ vals,
                                          const double *__restrict__ x, int row, int lane,
                                          bool live) {
  double s = 0.0;
  const int k0 = live ? rowptr[row] : 0, k1 = live ? rowptr[row + 1] : 0;
  for (int k = k0 + lane; k < k1; k += G) s += vals[k] * __ldg(x + colidx[k]);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
  return s;
}

// y = alpha * A x + beta * y (beta == 0: y is not read)
template <int G>
__global__ void __launch_bounds__(kLinBlock)
    spmv_kernel(const int32_t *__restrict__ rowptr, const int32_t *__restrict__ colidx,
                const double *__restrict__ vals, int nrows, const double *__restrict__ x,
                double *__restrict__ y, double alpha, double beta) {
  const int lane = threadIdx.x % G;
  const int groups = (gridDim.x * blockDim.x) / G;
  // every lane of a group walks the same rows (the row count padded to a
  // multiple of the groups), so the group shuffles stay converged
  const int rows_padded = ((nrows + groups - 1) / groups) * groups;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / G; row < rows_padded; row += groups) {
    const bool live = row < nrows;
    const double s = row_dot<G>(rowptr, colidx, vals, x, row, lane, live);
    if (live && lane == 0) y[row] = beta == 0.0 ? alpha * s : alpha * s + beta * y[row];
  }
}

// --------------------------------------------------------- vector kernels
constexpr int kVecUnroll = 4;    // 16-byte pieces a thread has in flight

template <typename T, int OP>
__device__ __forceinline__ T binop(T a, T b) {
  if constexpr (OP == 0) return a + b;
  else if constexpr (OP == 1) return a - b;
  else if constexpr (OP == 2) return a * b;
  else return a / b;
}

// out = x op y (y null: x op ys); out may be x or y.  Bound by HBM: W items of
// 16 bytes at a time, kVecUnroll of them loaded before the first store.  W = 1
// where a pointer is not 16-byte aligned.  4.2 M doubles out of HBM: scaling
// 12.7 us (5.3 TB/s; 14.8 with one item a thread per round), sum 18.8 (20.2).
template <typename T, int OP, int W>
__global__ void __launch_bounds__(kLinBlock) binop_kernel(T *out, const T *x, const T *y, T ys, int64_t n) {
  struct alignas(W * sizeof(T)) Piece {
    T v[W];
  };
  const int64_t pieces = n / W;
  const int64_t i0 = (int64_t)blockIdx.x * (kLinBlock * kVecUnroll) + threadIdx.x;
  Piece a[kVecUnroll], b[kVecUnroll];
#pragma unroll
  for (int u = 0; u < kVecUnroll; ++u) {
    const int64_t i = i0 + u * kLinBlock;
    if (i < pieces) {
      a[u] = reinterpret_cast<const Piece *>(x)[i];
      if (y) b[u] = reinterpret_cast<const Piece *>(y)[i];
    }
  }
#pragma unroll
  for (int u = 0; u < kVecUnroll; ++u) {
    const int64_t i = i0 + u * kLinBlock;
    if (i < pieces) {
#pragma unroll
      for (int w = 0; w < W; ++w) a[u].v[w] = binop<T, OP>(a[u].v[w], y ? b[u].v[w] : ys);
      reinterpret_cast<Piece *>(out)[i] = a[u];
    }
  }
  if (W > 1 && blockIdx.x == 0 && threadIdx.x < n - pieces * W) {
    const int64_t i = pieces * W + threadIdx.x;
    out[i] = binop<T, OP>(x[i], y ? y[i] : ys);
  }
}

// x . y in one launch: each CTA sums its share in a fixed order, and the last
// CTA to finish sums the CTAs' partials in CTA order into *result (host memory
// the device writes, its ticket last) and clears the counter for the next call.
// W as above.  The norm of 4.2 M doubles 26 us with the call and the wait
// (37.6 with a second launch, an allocation and a copy), of 1,000 15 (25).
struct DotResult {
  double value;
  unsigned long long ticket;
};

template <int W>
__global__ void __launch_bounds__(kLinBlock) dot_kernel(const double *__restrict__ x,
                                                        const double *__restrict__ y, int64_t n, double *part,
                                                        unsigned *counter, DotResult *result,
                                                        unsigned long long ticket) {
  __shared__ double scratch[32];
  __shared__ bool last;
  struct alignas(W * 8) Piece {
    double v[W];
  };
  const int64_t pieces = n / W, step = (int64_t)gridDim.x * kLinBlock;
  double s = 0.0;
  for (int64_t i0 = (int64_t)blockIdx.x * kLinBlock + threadIdx.x; i0 < pieces; i0 += step * kVecUnroll) {
    Piece a[kVecUnroll], b[kVecUnroll];
#pragma unroll
    for (int u = 0; u < kVecUnroll; ++u) {
      const int64_t i = i0 + u * step;
      if (i < pieces) {
        a[u] = reinterpret_cast<const Piece *>(x)[i];
        b[u] = x == y ? a[u] : reinterpret_cast<const Piece *>(y)[i];
      }
    }
#pragma unroll
    for (int u = 0; u < kVecUnroll; ++u)
      if (i0 + u * step < pieces)
#pragma unroll
        for (int w = 0; w < W; ++w) s += a[u].v[w] * b[u].v[w];
  }
  if (W > 1 && blockIdx.x == 0 && threadIdx.x < n - pieces * W)
    s += x[pieces * W + threadIdx.x] * y[pieces * W + threadIdx.x];
  s = block_sum(s, scratch);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  s = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kLinBlock) s += __ldcg(part + i);
  s = block_sum(s, scratch);
  if (threadIdx.x == 0) {
    *counter = 0u;
    result->value = s;
    __threadfence_system();
    *(volatile unsigned long long *)&result->ticket = ticket;
  }
}

// ------------------------------------------------------------------ CG
struct CgArgs {
  const int32_t *rowptr, *colidx;
  const double *vals, *b;
  double *x, *r, *p, *q, *dinv;
  double2 *part;                // [2][gridDim.x]: {p.q, 0} and {r.z, z.z} of each CTA
  double *hist;                 // [max_it + 1]: ||z|| of each iteration
  int *out;                     // reason (1 converged, 2 diverged, 3 breakdown, 4 limit), iterations
  int n, max_it, jacobi;
  double rtol, atol, dtol;
};

constexpr int kCgThreads = 512;
constexpr int kCgPerSm = 2;
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kCgChunk = 640;   // products a warp has in shared memory (80 KB per CTA)
constexpr int kCgAhead = 6;     // entries a lane has in flight

// A warp takes 32 consecutive rows: their entries, contiguous in the CSR
// arrays, are read by consecutive lanes, kCgAhead gathers each in flight, and
// the products kept in the warp's shared memory a chunk at a time; then every
// lane adds up its row in column order.  Warps do not wait for one another.
// row_done(row, sum) is called by the row's lane.
template <typename Done>
__device__ __forceinline__ void rows_by_warp(const int32_t *__restrict__ rowptr,
                                             const int32_t *__restrict__ colidx,
                                             const double *__restrict__ vals, const double *x, int n,
                                             double *prod, Done row_done) {
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * kCgThreads;
  int64_t row0 = ((int64_t)blockIdx.x * kCgThreads + threadIdx.x) & ~31ll;
  if (row0 >= n) return;
  int a = rowptr[min((int)row0 + lane, n)], e = rowptr[min((int)row0 + lane + 1, n)];
  while (row0 < n) {
    const int row = (int)row0 + lane;
    const int first = __shfl_sync(0xffffffffu, a, 0), last = __shfl_sync(0xffffffffu, e, 31);
    // the next group's row bounds, and its entries into L2
    const int64_t next0 = row0 + step;
    int an = 0, en = 0;
    if (next0 < n) {
      an = rowptr[min((int)next0 + lane, n)];
      en = rowptr[min((int)next0 + lane + 1, n)];
    }
    double s = 0.0;
    for (int base = first; base < last; base += kCgChunk) {
      const int m = min(kCgChunk, last - base);
      const int32_t *c = colidx + base;
      const double *v = vals + base;
      for (int k0 = lane; k0 < m; k0 += 32 * kCgAhead) {
        int cc[kCgAhead];
        double vv[kCgAhead];
#pragma unroll
        for (int u = 0; u < kCgAhead; ++u) {
          const int k = k0 + 32 * u;
          cc[u] = k < m ? __ldcs(c + k) : 0;
          vv[u] = k < m ? __ldcs(v + k) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kCgAhead; ++u)
          if (k0 + 32 * u < m) prod[k0 + 32 * u] = vv[u] * x[cc[u]];
      }
      if (base == first && next0 < n) {
        const int f = __shfl_sync(0xffffffffu, an, 0), l = min(__shfl_sync(0xffffffffu, en, 31), f + kCgChunk);
        for (int k = f + 32 * lane; k < l; k += 32 * 32)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(colidx + k));
        for (int k = f + 16 * lane; k < l; k += 16 * 32)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(vals + k));
      }
      __syncwarp();
      const int j1 = min(e - base, m);
      for (int j = max(a - base, 0); j < j1; ++j) s += prod[j];
      __syncwarp();
    }
    if (row < n) row_done(row, s);
    row0 = next0;
    a = an;
    e = en;
  }
}

// A group of G lanes per row, for rows too long for one thread.
template <int G, typename Done>
__device__ __forceinline__ void rows_by_group(const int32_t *__restrict__ rowptr,
                                              const int32_t *__restrict__ colidx,
                                              const double *__restrict__ vals, const double *x, int n,
                                              Done row_done) {
  const int lane = threadIdx.x % G;
  const int groups = (gridDim.x * blockDim.x) / G;
  const int rows_padded = ((n + groups - 1) / groups) * groups;
  for (int row = (blockIdx.x * blockDim.x + threadIdx.x) / G; row < rows_padded; row += groups) {
    double s = 0.0;
    if (row < n)
      for (int k = rowptr[row] + lane; k < rowptr[row + 1]; k += G) s += vals[k] * x[colidx[k]];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
    if (row < n && lane == 0) row_done(row, s);
  }
}

// Two sums over the CTA at once, in a fixed order; valid in every thread.
__device__ __forceinline__ double2 block_sum2(double2 v, double2 *scratch) {
  const int lane = threadIdx.x & 31;
  v.x = warp_sum(v.x);
  v.y = warp_sum(v.y);
  __syncthreads();
  if (lane == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  v = lane < kCgThreads / 32 ? scratch[lane] : make_double2(0.0, 0.0);
  return make_double2(warp_sum(v.x), warp_sum(v.y));
}

// The sums over CTAs of two partials, the same in every thread of the grid.
__device__ __forceinline__ double2 cg_total(const double2 *part, double2 *scratch) {
  double2 s = make_double2(0.0, 0.0);
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kCgThreads) {
    const double2 v = __ldcg(part + i);
    s.x += v.x;
    s.y += v.y;
  }
  return block_sum2(s, scratch);
}

// P2 mass matrix, 1.05 M rows of 11.5 entries, 25 steps to 1e-10: 1.39 ms
// (56 us a step, 34 of them the product: 150 MB of matrix from HBM at 4.4 TB/s,
// bound by the latency of 32 resident warps; vectors 14 us from L2, syncs 6)
// against 2.10 ms as three launches a step and a flag read every 16 steps.
// Products staged per CTA with block barriers measured 48 us, copied ahead to
// shared memory 48 us, four lanes a row 45 us.  2,401 rows: 0.31 against 0.57 ms.
//
// Per iteration: q = A p with p.q; r -= alpha q with r.z and z.z (z = D^-1 r is
// formed where it is needed, not stored); x += alpha p and p = z + beta p.
// Vectors are read with plain loads: other CTAs write them between two syncs.
// G lanes a row (1: rows_by_warp).
template <int G>
__global__ void __launch_bounds__(kCgThreads, kCgPerSm) cg_kernel(CgArgs s) {
  extern __shared__ double prod[];
  __shared__ double2 scratch[32];
  const auto grid = cooperative_groups::this_grid();
  const int tid = threadIdx.x, first = blockIdx.x * kCgThreads + tid, step = gridDim.x * kCgThreads;
  double2 *part_pq = s.part, *part_rz = part_pq + gridDim.x;
  double rz = 0.0, zz = 0.0;
  for (int i = first; i < s.n; i += step) {
    double d = 0.0;
    if (s.jacobi)
      for (int k = s.rowptr[i]; k < s.rowptr[i + 1]; ++k)
        if (s.colidx[k] == i) d = s.vals[k];
    // a missing or zero diagonal leaves that row unpreconditioned
    const double di = d != 0.0 ? 1.0 / d : 1.0, bi = s.b[i], zi = di * bi;
    s.dinv[i] = di;
    s.x[i] = 0.0;
    s.r[i] = bi;
    s.p[i] = zi;
    rz += bi * zi;
    zz += zi * zi;
  }
  auto publish = [&](double v, double w, double2 *part) {
    const double2 sum = block_sum2(make_double2(v, w), scratch);
    if (tid == 0) part[blockIdx.x] = sum;
  };
  publish(rz, zz, part_rz);
  grid.sync();
  double2 sums = cg_total(part_rz, scratch);
  rz = sums.x;
  const double rnorm0 = sqrt(sums.y);
  const double tol = fmax(s.rtol * rnorm0, s.atol), most = s.dtol * rnorm0;
  if (first == 0) s.hist[0] = rnorm0;
  int reason = rnorm0 <= tol ? 1 : isfinite(rnorm0) ? 0 : 3, k = 0;
  if (!reason && s.max_it == 0) reason = 4;
  while (!reason) {
    double pq = 0.0;
    auto done = [&](int row, double v) {
      s.q[row] = v;
      pq += s.p[row] * v;
    };
    if constexpr (G == 1)
      rows_by_warp(s.rowptr, s.colidx, s.vals, s.p, s.n, prod + (tid >> 5) * kCgChunk, done);
    else
      rows_by_group<G>(s.rowptr, s.colidx, s.vals, s.p, s.n, done);
    publish(pq, 0.0, part_pq);
    grid.sync();
    pq = cg_total(part_pq, scratch).x;
    const double alpha = (pq != 0.0 && isfinite(pq)) ? rz / pq : 0.0;
    double rz1 = 0.0;
    zz = 0.0;
    // the four work vectors and x are different memory: loads of several
    // elements may be in flight before their stores
    double *__restrict__ r = s.r, *__restrict__ p = s.p, *__restrict__ x = s.x;
    const double *__restrict__ q = s.q, *__restrict__ dinv = s.dinv;
#pragma unroll 4
    for (int i = first; i < s.n; i += step) {
      const double ri = r[i] - alpha * q[i], zi = dinv[i] * ri;
      r[i] = ri;
      rz1 += ri * zi;
      zz += zi * zi;
    }
    publish(rz1, zz, part_rz);
    grid.sync();
    sums = cg_total(part_rz, scratch);
    rz1 = sums.x;
    const double rnorm = sqrt(sums.y);
    const double beta = (rz != 0.0 && isfinite(rz)) ? rz1 / rz : 0.0;
#pragma unroll 4
    for (int i = first; i < s.n; i += step) {
      const double pi = p[i];
      x[i] += alpha * pi;
      p[i] = dinv[i] * r[i] + beta * pi;
    }
    rz = rz1;
    ++k;
    if (first == 0) s.hist[k] = rnorm;
    if (!isfinite(rnorm)) reason = 3;
    else if (rnorm <= tol) reason = 1;
    else if (rnorm >= most) reason = 2;
    else if (k >= s.max_it) reason = 4;
    if (!reason) grid.sync();
  }
  if (first == 0) {
    s.out[0] = reason;
    s.out[1] = k;
  }
}

// Lanes per row from the mean row length: on the P2 mass matrix (11.5
// entries per row) 4 lanes measured 0.150 ms per product, 2 lanes 0.152, 8
// lanes 0.221, 16 lanes 0.373 -- fewer lanes keep more rows in flight.
static int group_for(int64_t nnz, int nrows) {
  const double avg = nrows > 0 ? (double)nnz / nrows : 0.0;
  return avg <= 16 ? 4 : avg <= 48 ? 8 : avg <= 96 ? 16 : 32;
}

static int lin_grid(int64_t work) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((work + kLinBlock - 1) / kLinBlock,
                                                     (int64_t)sm_count() * 8));
}

template <typename T, int W>
static int launch_binop_as(uint64_t out, uint64_t x, uint64_t y, T ys, int64_t n, int op, cudaStream_t s) {
  const int64_t per = (int64_t)kLinBlock * kVecUnroll;
  const int64_t grid = std::max<int64_t>(1, (n / W + per - 1) / per);
  if (grid > INT32_MAX) return set_error(OP2B_ERR_ARG, "op2b_vec_binop: %lld items", (long long)n);
  T *o = (T *)out;
  const T *a = (const T *)x, *b = (const T *)y;
  switch (op) {
    case 0: binop_kernel<T, 0, W><<<(int)grid, kLinBlock, 0, s>>>(o, a, b, ys, n); break;
    case 1: binop_kernel<T, 1, W><<<(int)grid, kLinBlock, 0, s>>>(o, a, b, ys, n); break;
    case 2: binop_kernel<T, 2, W><<<(int)grid, kLinBlock, 0, s>>>(o, a, b, ys, n); break;
    default: binop_kernel<T, 3, W><<<(int)grid, kLinBlock, 0, s>>>(o, a, b, ys, n); break;
  }
  return check_cuda(cudaGetLastError(), "binop_kernel");
}

template <typename T>
static int launch_binop(uint64_t out, uint64_t x, uint64_t y, T ys, int64_t n, int op, cudaStream_t s) {
  return (out | x | y) % 16 ? launch_binop_as<T, 1>(out, x, y, ys, n, op, s)
                            : launch_binop_as<T, 16 / sizeof(T)>(out, x, y, ys, n, op, s);
}

// Scratch of op2b_vec_dot, one per host thread: a call waits for its result, so
// a thread never has two in flight, on whatever streams.  About 5 KB of device
// memory and one pinned word, given back when the thread ends.
struct DotScratch {
  int device = -1;
  double *part = nullptr;
  unsigned *counter = nullptr;
  DotResult *result = nullptr;
  unsigned long long ticket = 0;

  // The counter is cleared on the call's stream and waited for, once per thread
  // and device: later calls may come on any stream.
  int ready(int most, cudaStream_t s) {
    int dev = 0;
    OP2B_CUDA(cudaGetDevice(&dev));
    if (dev == device) return OP2B_OK;
    release();
    const size_t bytes = sizeof(double) * (most + 2);
    cudaError_t e = cudaMalloc((void **)&part, bytes);
    if (e == cudaSuccess) e = cudaHostAlloc((void **)&result, sizeof(DotResult), cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaMemsetAsync(part, 0, bytes, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      release();
      return check_cuda(e, "op2b_vec_dot scratch");
    }
    result->ticket = ticket = 0;
    counter = reinterpret_cast<unsigned *>(part + most);
    device = dev;
    return OP2B_OK;
  }
  void release() {
    if (part) cudaFree(part);
    if (result) cudaFreeHost(result);
    part = nullptr;
    result = nullptr;
    device = -1;
  }
  ~DotScratch() { release(); }
};

static thread_local DotScratch t_dot;

}  // namespace op2b

using namespace op2b;

extern "C" {

int op2b_csr_spmv(uint64_t rowptr, uint64_t colidx, uint64_t vals, int32_t nrows, int64_t nnz,
                  uint64_t x, uint64_t y, double alpha, double beta, int32_t group,
                  uint64_t stream) {
  OP2B_REQUIRE_INIT();
  if (nrows < 0 || nnz < 0) return set_error(OP2B_ERR_ARG, "op2b_csr_spmv: bad sizes");
  if (group != 0 && group != 1 && group != 2 && group != 4 && group != 8 && group != 16 &&
      group != 32)
    return set_error(OP2B_ERR_ARG, "op2b_csr_spmv: group %d (0 or a power of two up to 32)",
                     group);
  if (nrows == 0) return OP2B_OK;
  const int G = group ? group : group_for(nnz, nrows);
  const int grid = lin_grid((int64_t)nrows * G);
  cudaStream_t s = stream_of(stream);
  auto rp = (const int32_t *)rowptr;
  auto ci = (const int32_t *)colidx;
  auto v = (const double *)vals;
  switch (G) {
    case 1: spmv_kernel<1><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
    case 2: spmv_kernel<2><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
    case 4: spmv_kernel<4><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
    case 8: spmv_kernel<8><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
    case 16: spmv_kernel<16><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
    default: spmv_kernel<32><<<grid, kLinBlock, 0, s>>>(rp, ci, v, nrows, (const double *)x, (double *)y, alpha, beta); break;
  }
  return check_cuda(cudaGetLastError(), "spmv_kernel");
}

int op2b_vec_binop(uint64_t out, uint64_t x, uint64_t y, double yscalar, int64_t n, int32_t op,
                   int32_t dtype, uint64_t stream) {
  OP2B_REQUIRE_INIT();
  if (n < 0 || op < 0 || op > 3) return set_error(OP2B_ERR_ARG, "op2b_vec_binop: bad arguments");
  if (n == 0) return OP2B_OK;
  cudaStream_t s = stream_of(stream);
  int rc = OP2B_OK;
  switch (dtype) {
    case 0: rc = launch_binop<double>(out, x, y, yscalar, n, op, s); break;
    case 1: rc = launch_binop<float>(out, x, y, (float)yscalar, n, op, s); break;
    case 2: rc = launch_binop<int32_t>(out, x, y, (int32_t)yscalar, n, op, s); break;
    default: return set_error(OP2B_ERR_ARG, "op2b_vec_binop: dtype %d", dtype);
  }
  return rc;
}

int op2b_vec_dot(uint64_t x, uint64_t y, int64_t n, double *result, uint64_t stream) {
  OP2B_REQUIRE_INIT();
  if (n < 0 || !result) return set_error(OP2B_ERR_ARG, "op2b_vec_dot: bad arguments");
  cudaStream_t s = stream_of(stream);
  const int most = sm_count() * 4;
  DotScratch &w = t_dot;
  int rc = w.ready(most, s);
  if (rc) return rc;
  const int W = (x | y) % 16 ? 1 : 2;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n / W + kLinBlock - 1) / kLinBlock, most));
  const unsigned long long ticket = ++w.ticket;
  if (W == 2)
    dot_kernel<2><<<grid, kLinBlock, 0, s>>>((const double *)x, (const double *)y, n, w.part, w.counter, w.result,
                                             ticket);
  else
    dot_kernel<1><<<grid, kLinBlock, 0, s>>>((const double *)x, (const double *)y, n, w.part, w.counter, w.result,
                                             ticket);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return check_cuda(e, "dot_kernel");
  // the ticket shows up some microseconds before the stream reports its end;
  // past about a millisecond the stream is asked (it also reports errors)
  const volatile unsigned long long *seen = &w.result->ticket;
  bool in = false;
  for (int spin = 0; spin < 100000 && !in; ++spin) in = *seen == ticket;
  if (!in) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && !in && *seen != ticket) {
    w.release();       // no CTA saw itself as the last one: never a value of an earlier call
    return set_error(OP2B_ERR_CUDA, "op2b_vec_dot: the kernel left no result");
  }
  if (e == cudaSuccess) *result = *(const volatile double *)&w.result->value;
  return check_cuda(e, "op2b_vec_dot");
}

int op2b_cg_solve(uint64_t rowptr, uint64_t colidx, uint64_t vals, int32_t nrows, int64_t nnz,
                  uint64_t x, uint64_t b, int32_t jacobi, double rtol, double atol, double dtol,
                  int32_t max_it, int32_t *iterations, int32_t *reason, double *history,
                  uint64_t stream) {
  OP2B_REQUIRE_INIT();
  if (nrows < 0 || nnz < 0 || max_it < 0 || !iterations || !reason)
    return set_error(OP2B_ERR_ARG, "op2b_cg_solve: bad arguments");
  *iterations = 0;
  *reason = 1;
  if (nrows == 0) return OP2B_OK;
  cudaStream_t st = stream_of(stream);
  // rows of more than 48 entries on the mean take a group of lanes each
  const int G = nnz <= 48 * (int64_t)nrows ? 1 : group_for(nnz, nrows);
  const void *fn = G == 1 ? (const void *)cg_kernel<1> : G == 16 ? (const void *)cg_kernel<16>
                                                                : (const void *)cg_kernel<32>;
  const int smem = G == 1 ? kCgWarps * kCgChunk * (int)sizeof(double) : 0;
  int per_sm = 0;
  OP2B_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  OP2B_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kCgThreads, smem));
  const int grid = std::max(1, std::min(op2b_div_up(nrows, kCgThreads / G), per_sm * sm_count()));
  const size_t nv = (size_t)nrows;
  double *work = nullptr;
  int rc = dev_alloc((void **)&work, sizeof(double) * (4 * nv + 4 * (size_t)grid + (size_t)max_it + 1 + 1), st);
  if (rc) return rc;
  CgArgs s{};
  s.rowptr = (const int32_t *)rowptr;
  s.colidx = (const int32_t *)colidx;
  s.vals = (const double *)vals;
  s.b = (const double *)b;
  s.x = (double *)x;
  s.part = reinterpret_cast<double2 *>(work);
  s.r = work + 4 * (size_t)grid;
  s.p = s.r + nv;
  s.q = s.p + nv;
  s.dinv = s.q + nv;
  s.out = reinterpret_cast<int *>(s.dinv + nv);
  s.hist = s.dinv + nv + 1;
  s.n = nrows;
  s.max_it = max_it;
  s.jacobi = jacobi;
  s.rtol = rtol;
  s.atol = atol;
  s.dtol = dtol;
  void *args[] = {&s};
  cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kCgThreads), args, smem, st);
  // the outcome and, as a rule, the whole history in one copy
  constexpr int kFirst = 255;
  double got[1 + kFirst];
  const int head = std::min(max_it + 1, kFirst);
  if (e == cudaSuccess) e = cudaMemcpyAsync(got, s.out, sizeof(double) * (1 + head), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) {
    int out[2];
    memcpy(out, got, sizeof out);
    *reason = out[0];
    *iterations = out[1];
    if (history) {
      memcpy(history, got + 1, sizeof(double) * std::min(out[1] + 1, head));
      if (out[1] + 1 > head) {
        e = cudaMemcpyAsync(history + head, s.hist + head, sizeof(double) * (out[1] + 1 - head),
                            cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      }
    }
  }
  dev_free(work, st);
  return check_cuda(e, "op2b_cg_solve");
}

}  // extern "C"
