// Row blocks: Mat assembly run by the owners of the rows.
//
// A loop whose only writes are increments of scalar Mats through one (row Map,
// column Map) pair can be run by row instead of by element: a CTA owns a block
// of rows, evaluates every element that touches one of them into shared memory,
// and writes every stored entry of its rows once, adding the entry's
// contributions in element order (the order of pyop2/sequential.py:55-72).
// No add is atomic, there are no colours, and the result does not depend on
// scheduling; the price is that an element whose rows belong to several
// blocks is evaluated by each of them (about a third more elements for
// blocks of a hundred rows of a triangle mesh).  This file builds the tables
// such a stub walks:
//  * blocks: regions of elements are grown around hashed seeds by a
//    breadth-first search through the Map and ordered by sector (which of the
//    seed's targets an element was reached through), then level; the rows,
//    in order of first use along that order, are cut inside each region into
//    runs of nearly equal numbers of items ((element, map index) pairs), at
//    most `region` elements' worth: wedges, as compact as squares and of one
//    size, which is what the shared memory of a launch is sized by.  Which
//    region an element between two seeds joins may differ from build to build;
//    the loop's results do not depend on it;
//  * one packet per block, 16-byte aligned so that a CTA copies it to shared
//    memory while it still works on the block before:
//      header  int32 {elements NE, short entries, long entries, items NI},
//              int32 {targets of staged Map 0 .. 3}
//      elems   int32 [NE]: the elements the block evaluates (only where the
//              loop needs their ids: `ids` of the build)
//      items   uint16 [ra][NE]: the number of (element, map index) among those
//              that land in the block's rows, by map index then element; NI if
//              it lands in another block's row
//      per staged Map (the loop reads Dats through it): targets int32 [nt],
//              the block's distinct targets in order of first use, and
//              lidx uint16 [arity][NE], each element's targets in that list
//      longs   per entry of three or more contributions: {CSR position,
//              first | last + 1 << 16 of its contributions in list}
//      list    uint16: the long entries' contributions
//    and, which the CTA reads from where it lies,
//      shorts  per other entry, rows in order, columns in order: {CSR position,
//              first contribution | second << 16}; an entry of one has ca * NS
//              as its second, a place the stub fills with -0.0
//    A contribution is its place in the block's shared array [ca][NS], NS the
//    first odd number above NI: c * NS + item (column NI takes what other
//    blocks own); each part is padded to 16 bytes, and an entry's contributions
//    come in element order.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>

#include "op2b_internal.h"
#include "op2b_rowblk_room.h"
#include "op2b_scan.cuh"

namespace op2b {

constexpr int kRbThreads = 256;
constexpr int kRbStages = 4;
constexpr int kRbShort = 2;
constexpr int kRbMaxKeys = 8192;       // items of a block, and map entries of its elements
constexpr int kRbMaxContrib = 16384;   // contributions of a block

struct RowBlocks {
  int32_t nblocks = 0, max_items = 0;
  int32_t max_packet = 0;      // 16-byte units, without the short entries
  int32_t max_targets[kRbStages] = {0, 0, 0, 0};
  int2 *dir = nullptr;         // [nblocks] packet start, first | size << 16, 16-byte units
  uint4 *pkt = nullptr;
};

struct RbMaps {
  const int32_t *map[kRbStages];
  int32_t arity[kRbStages];
  int32_t n, rows;             // staged Maps, and their arities' sum
};

struct RbArgs {
  const int32_t *order, *rstart, *io, *eo, *list, *cmap, *rowptr, *colidx;
  int32_t ra, ca, max_items, max_rows, hash, ids;
  int64_t cap;                 // 16-byte units of pkt
  RbMaps st;
  int2 *dir;
  uint4 *pkt;
  int32_t *scal;               // see kS*
};

// device scalars; the cursor has 64 bits, since what the blocks take may be past
// what a directory entry can hold
enum {
  kSCursor,
  kSFlag = kSCursor + 2,
  kSMaxPacket,
  kSMaxTargets,
  kSScan = kSMaxTargets + kRbStages,
  kSBlocks = kSScan + 3,
  kSUsed,
  kSMaxItems,
  kSMaxRows,
  kSChanged,
  kSCount = kSChanged + 3
};

constexpr int kRbLevels = 32;          // levels told apart in a region's order

__device__ __forceinline__ uint32_t rb_hash(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  return x ^ (x >> 16);
}

// Element 0 and about one element in `mean` are seeds.
__global__ void rb_seed_kernel(int n, int mean, int32_t *__restrict__ seed) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e <= n; e += gridDim.x * blockDim.x)
    seed[e] = e < n && (e == 0 || rb_hash((uint32_t)e) % (uint32_t)mean == 0);
}

// Regions, in one cooperative launch: keys level << 32 | region << sbits |
// sector.  seed: the number of seeds before each element (regions are numbered
// in element order, so neighbouring blocks run together); a seed hands
// each of its targets its region and that target's own sector; then, level by
// level, every element without a key takes the smallest key of its targets,
// one level further, and hands it on.  Keys of the next level written during a
// pass are ignored by its readers.  tkey starts at all ones.
__global__ void rb_grow_kernel(int n, const int32_t *__restrict__ map, int arity,
                               const int32_t *__restrict__ seed, int most_seeds, int sbits, uint64_t *ekey,
                               unsigned long long *tkey, int32_t *scal) {
  const auto grid = cooperative_groups::this_grid();
  const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (int e = first; e < n; e += step) {
    uint64_t k = ~0ull;
    const int region = seed[e];
    if (seed[e + 1] != region && region < most_seeds) {
      k = (uint64_t)region << sbits;
      for (int r = 0; r < arity; ++r)
        atomicMin(&tkey[map[(int64_t)e * arity + r]], k | (uint64_t)(r & ((1 << sbits) - 1)));
    }
    ekey[e] = k;
  }
  grid.sync();
  volatile int32_t *changed = scal + kSChanged;
  for (uint64_t level = 0; level < (uint64_t)n; ++level) {
    int any = 0;
    const uint64_t limit = (level + 1) << 32;
    if (first == 0) changed[(level + 1) % 3] = 0;
    for (int e = first; e < n; e += step) {
      if (ekey[e] != ~0ull) continue;
      uint64_t best = ~0ull;
      for (int r = 0; r < arity; ++r) {
        const uint64_t k = ((volatile unsigned long long *)tkey)[map[(int64_t)e * arity + r]];
        if (k < limit && k < best) best = k;
      }
      if (best == ~0ull) continue;
      const uint64_t k = (level + 1) << 32 | (best & 0xffffffffull);
      ekey[e] = k;
      any = 1;
      for (int r = 0; r < arity; ++r) atomicMin(&tkey[map[(int64_t)e * arity + r]], (unsigned long long)k);
    }
    if (__syncthreads_or(any) && threadIdx.x == 0) changed[level % 3] = 1;
    grid.sync();
    if (!changed[level % 3]) break;
  }
}

// Bucket (region, sector, level) of every element, counted; elements the
// search did not reach form regions of consecutive elements.
__global__ void rb_bucket_kernel(int n, const uint64_t *__restrict__ ekey, int most_seeds, int part, int sbits,
                                 int32_t *__restrict__ bucket, int32_t *__restrict__ count) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint64_t k = ekey[e];
    const int rs = k == ~0ull ? (most_seeds + e / part) << sbits : (int)(k & 0xffffffffull);
    const int b = rs * kRbLevels + (k == ~0ull ? 0 : min((int)(k >> 32), kRbLevels - 1));
    bucket[e] = b;
    atomicAdd(&count[b], 1);
  }
}

// Elements in bucket order; cursor: the buckets' first places.
__global__ void rb_order_kernel(int n, const int32_t *__restrict__ bucket, int32_t *__restrict__ cursor,
                                int32_t *__restrict__ order) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    order[atomicAdd(&cursor[bucket[e]], 1)] = e;
}

// First use of every target along the elements' order (all ones: none), and
// the number of its uses.
__global__ void rb_first_kernel(int64_t tot, int ra, const int32_t *__restrict__ rmap,
                                const int32_t *__restrict__ eorder, unsigned *__restrict__ first,
                                int32_t *__restrict__ deg) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int t = rmap[(int64_t)eorder[q / ra] * ra + q % ra];
    atomicMin(&first[t], (unsigned)q);
    atomicAdd(&deg[t], 1);
  }
}

__global__ void rb_flag_kernel(int64_t tot, int ra, const int32_t *__restrict__ rmap,
                               const int32_t *__restrict__ eorder, const unsigned *__restrict__ first,
                               int32_t *__restrict__ flag) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q <= tot; q += (int64_t)gridDim.x * blockDim.x)
    flag[q] = q < tot && first[rmap[(int64_t)eorder[q / ra] * ra + q % ra]] == (unsigned)q;
}

// Rows in order of first use (those no element touches are in no block), with
// their items (element, map index) and entries, both to be summed up.
__global__ void rb_rows_kernel(int64_t tot, int ra, const int32_t *__restrict__ rmap,
                               const int32_t *__restrict__ eorder, const int32_t *__restrict__ ranks,
                               const int32_t *__restrict__ deg, const int32_t *__restrict__ rowptr,
                               int32_t *__restrict__ order, int32_t *__restrict__ rank, int32_t *__restrict__ io,
                               int32_t *__restrict__ eo) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < tot; q += (int64_t)gridDim.x * blockDim.x) {
    const int i = ranks[q];
    if (ranks[q + 1] == i) continue;
    const int t = rmap[(int64_t)eorder[q / ra] * ra + q % ra];
    order[i] = t;
    rank[t] = i;
    io[i] = deg[t];
    eo[i] = rowptr[t + 1] - rowptr[t];
  }
}

// Each row's items, in any order inside the row.  deg counts down to zero.
__global__ void rb_scatter_kernel(const int32_t *__restrict__ rmap, int64_t tot,
                                  const int32_t *__restrict__ rank, const int32_t *__restrict__ io,
                                  int32_t *__restrict__ deg, int32_t *__restrict__ list) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < tot;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int t = rmap[q];
    list[io[rank[t]] + atomicSub(&deg[t], 1) - 1] = (int32_t)q;
  }
}

// First row of region r: the first uses before its first element (bfirst: the
// buckets' first places).
__device__ __forceinline__ int rb_region_row(int r, int buckets, int ra, const int32_t *bfirst,
                                             const int32_t *ranks) {
  return ranks[(int64_t)bfirst[(int64_t)r * buckets] * ra];
}

// Runs each region's rows are cut into, of at most `most` items as a rule.
__global__ void rb_pieces_kernel(int nregions, int buckets, int ra, int most, const int32_t *__restrict__ bfirst,
                                 const int32_t *__restrict__ ranks, const int32_t *__restrict__ io,
                                 int32_t *__restrict__ pieces) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= nregions; r += gridDim.x * blockDim.x) {
    int m = 0;
    if (r < nregions) {
      const int a = rb_region_row(r, buckets, ra, bfirst, ranks),
                b = rb_region_row(r + 1, buckets, ra, bfirst, ranks);
      m = min(b - a, (io[b] - io[a] + most - 1) / most);
    }
    pieces[r] = m;
  }
}

// First row of every block, and the largest block's items and rows.
__global__ void rb_starts_kernel(int nregions, int buckets, int ra, const int32_t *__restrict__ bfirst,
                                 const int32_t *__restrict__ ranks, const int32_t *__restrict__ io,
                                 const int32_t *__restrict__ pieces, int32_t *__restrict__ rstart,
                                 int32_t *__restrict__ scal) {
  int mi = 0, mr = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nregions; r += gridDim.x * blockDim.x) {
    const int a = rb_region_row(r, buckets, ra, bfirst, ranks),
              b = rb_region_row(r + 1, buckets, ra, bfirst, ranks);
    const int first = pieces[r], m = pieces[r + 1] - first, total = io[b] - io[a];
    int from = a;
    for (int q = 1; q <= m; ++q) {
      // the first row at or past the q-th part of the items; every run has a row
      int lo = from + 1, hi = b - (m - q);
      if (q < m) {
        const int want = io[a] + (int)((int64_t)total * q / m);
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (io[mid] < want) lo = mid + 1;
          else hi = mid;
        }
      } else {
        lo = b;
      }
      rstart[first + q - 1] = from;
      mi = max(mi, io[lo] - io[from]);
      mr = max(mr, lo - from);
      from = lo;
    }
    if (r == nregions - 1) {
      rstart[pieces[nregions]] = b;
      scal[kSBlocks] = pieces[nregions];
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mi = max(mi, __shfl_xor_sync(0xffffffffu, mi, o));
    mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&scal[kSMaxItems], mi);
    atomicMax(&scal[kSMaxRows], mr);
  }
}

// Number the distinct values of n keys in order of first use: num[k] for each
// key, the values to out; returns how many.  tab, first: hash arrays of H
// slots (a power of two, H >= n, so probing ends); num doubles as the keys'
// slots.  The numbers do not depend on the order of the inserts.
template <typename Key, typename Num>
__device__ int rb_distinct(int n, int H, int *tab, int *first, Num *num, int *out, Key key) {
  const int tid = threadIdx.x;
  for (int h = tid; h < H; h += kRbThreads) {
    tab[h] = INT_MIN;
    first[h] = INT_MAX;
  }
  __syncthreads();
  for (int k = tid; k < n; k += kRbThreads) {
    const int v = key(k);
    int h = (int)(rb_hash((uint32_t)v) & (uint32_t)(H - 1));
    for (int probe = 0; probe < H; ++probe) {
      const int cur = atomicCAS(&tab[h], INT_MIN, v);
      if (cur == INT_MIN || cur == v) break;
      h = (h + 1) & (H - 1);
    }
    num[k] = (Num)h;
    atomicMin(&first[h], k);
  }
  __syncthreads();
  int carry = 0;
  for (int base = 0; base < n; base += kRbThreads) {
    const int k = base + tid;
    const int h = k < n ? (int)num[k] : 0;
    const int flag = k < n && first[h] == k;
    int tot;
    const int pos = block_excl_scan(flag, &tot);
    if (flag) {
      first[h] = -1 - (carry + pos);    // negative: no later key equals it
      out[carry + pos] = tab[h];
    }
    carry += tot;
    __syncthreads();
  }
  for (int k = tid; k < n; k += kRbThreads) num[k] = (Num)(-1 - first[(int)num[k]]);
  __syncthreads();
  return carry;
}

__device__ __forceinline__ int rb_units(int64_t bytes) { return (int)((bytes + 15) / 16); }

// One CTA per block.
__global__ void __launch_bounds__(kRbThreads) rb_build_kernel(const RbArgs A) {
  extern __shared__ int rb_smem[];
  const int blk = blockIdx.x, tid = threadIdx.x, ra = A.ra, ca = A.ca;
  const int row0 = A.rstart[blk], nr = A.rstart[blk + 1] - row0;
  const int i0 = A.io[row0], ni = A.io[row0 + nr] - i0;
  const int e0 = A.eo[row0], ne = A.eo[row0 + nr] - e0;
  const int ns = (ni + 1) | 1;              // columns of the contribution array
  int *it = rb_smem;                        // [max_items] flat positions, ascending inside a row
  int *elems = it + A.max_items;            // [max_items]
  int *ro = elems + A.max_items;            // [max_rows + 1] first item of each row
  int *re = ro + A.max_rows + 1;            // [max_rows + 1] first entry of each row
  int *rb = re + A.max_rows + 1;            // [max_rows] where a row's entries go
  int *tab = rb + A.max_rows;               // [hash]
  int *first = tab + A.hash;                // [hash]
  int *tl = first + A.hash;                 // [max_items * stage rows] targets of the staged Maps
  unsigned short *eloc = reinterpret_cast<unsigned short *>(tl + A.max_items * A.st.rows);  // [max_items]
  unsigned short *lidx = eloc + A.max_items;                                               // [max_items * stage rows]
  unsigned short *own = lidx + A.max_items * A.st.rows;                                    // [ra][max_items]
  for (int i = tid; i <= nr; i += kRbThreads) {
    ro[i] = A.io[row0 + i] - i0;
    re[i] = A.eo[row0 + i] - e0;
    if (i < nr) rb[i] = A.rowptr[A.order[row0 + i]];
  }
  __syncthreads();
  // row of item / entry k: the last row whose offset is <= k
  auto row_of = [&](const int *o, int k) {
    int lo = 0, hi = nr;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (o[mid] <= k) lo = mid;
      else hi = mid;
    }
    return lo;
  };
  for (int i = tid; i < ni; i += kRbThreads) {
    const int rl = row_of(ro, i), a = ro[rl], b = ro[rl + 1];
    const int v = A.list[i0 + i];
    int rank = 0;
    for (int j = a; j < b; ++j) rank += A.list[i0 + j] < v;
    it[a + rank] = v;
  }
  __syncthreads();
  const int NE = rb_distinct(ni, A.hash, tab, first, eloc, elems, [&](int k) { return it[k] / ra; });
  // items of the block's rows numbered by map index, then element
  for (int k = tid; k < ra * NE; k += kRbThreads) own[k] = (unsigned short)ni;
  __syncthreads();
  for (int i = tid; i < ni; i += kRbThreads) own[it[i] % ra * NE + eloc[i]] = 0;
  __syncthreads();
  for (int base = 0, carry = 0; base < ra * NE; base += kRbThreads) {
    const int k = base + tid;
    const bool mine = k < ra * NE && own[k] == 0;
    int tot;
    const int num = carry + block_excl_scan(mine, &tot);
    if (mine) own[k] = (unsigned short)num;
    carry += tot;
  }
  __syncthreads();
  int nt[kRbStages];
  {
    int at = 0;
    for (int s = 0; s < kRbStages; ++s) {
      nt[s] = 0;
      if (s >= A.st.n) continue;
      const int a = A.st.arity[s];
      const int32_t *m = A.st.map[s];
      nt[s] = rb_distinct(NE * a, A.hash, tab, first, lidx + A.max_items * at, tl + A.max_items * at,
                          [&](int k) { return m[(int64_t)elems[k / a] * a + k % a]; });
      at += a;
    }
  }
  // contributions of entry j of row rl; the elements' columns take the hash
  // arrays' place
  int *cols = tab;                          // [NE][ca]
  for (int k = tid; k < NE * ca; k += kRbThreads) cols[k] = A.cmap[(int64_t)elems[k / ca] * ca + k % ca];
  __syncthreads();
  auto entry_col = [&](int j, int rl) { return A.colidx[rb[rl] + j - re[rl]]; };
  auto count_of = [&](int j, int rl) {
    const int col = entry_col(j, rl);
    int cnt = 0;
    for (int i = ro[rl]; i < ro[rl + 1]; ++i) {
      const int *c = cols + eloc[i] * ca;
      for (int q = 0; q < ca; ++q) cnt += c[q] == col;
    }
    return cnt;
  };
  int nlong = 0, nempty = 0, nlids = 0;
  __shared__ int s_ids;
  if (tid == 0) s_ids = 0;
  __syncthreads();
  for (int base = 0; base < ne; base += kRbThreads) {
    const int j = base + tid;
    const int cnt = j < ne ? count_of(j, row_of(re, j)) : -1;
    nlong += __syncthreads_count(cnt > kRbShort);
    nempty += __syncthreads_count(cnt == 0);
    if (cnt > kRbShort) atomicAdd(&s_ids, cnt);
  }
  __syncthreads();
  nlids = s_ids;
  const int nshort = ne - nlong - nempty;
  __shared__ int64_t s_start;
  const int u_elems = A.ids ? rb_units(4 * NE) : 0, u_items = rb_units(2 * ra * NE);
  const int u_shorts = rb_units(8LL * nshort), u_longs = rb_units(8LL * nlong);
  int head = 2 + u_elems + u_items + u_longs + rb_units(2LL * nlids);
  for (int s = 0; s < A.st.n; ++s) head += rb_units(4 * nt[s]) + rb_units(2 * A.st.arity[s] * NE);
  const int total = head + u_shorts;
  if (tid == 0) {
    s_start = (int64_t)atomicAdd(reinterpret_cast<unsigned long long *>(A.scal + kSCursor),
                                 (unsigned long long)total);
    A.dir[blk] = make_int2((int)s_start, (int)((unsigned)head | (unsigned)total << 16));
    atomicMax(&A.scal[kSMaxPacket], head);
    for (int s = 0; s < A.st.n; ++s) atomicMax(&A.scal[kSMaxTargets + s], nt[s]);
    if ((int64_t)ns * ca > 65535 || total > 65535) atomicExch(&A.scal[kSFlag], 1);
  }
  __syncthreads();
  if (s_start + total > A.cap) return;    // the host allocates what the cursor says and repeats
  uint4 *P = A.pkt + s_start;
  if (tid == 0) {
    P[0] = make_uint4(NE, nshort, nlong, ni);
    P[1] = make_uint4(nt[0], nt[1], nt[2], nt[3]);
  }
  P += 2;
  if (A.ids)
    for (int i = tid; i < NE; i += kRbThreads) reinterpret_cast<int *>(P)[i] = elems[i];
  P += u_elems;
  for (int k = tid; k < ra * NE; k += kRbThreads) reinterpret_cast<unsigned short *>(P)[k] = own[k];
  P += u_items;
  for (int s = 0, at = 0; s < A.st.n; ++s) {
    const int a = A.st.arity[s];
    for (int i = tid; i < nt[s]; i += kRbThreads) reinterpret_cast<int *>(P)[i] = tl[A.max_items * at + i];
    P += rb_units(4 * nt[s]);
    for (int k = tid; k < NE * a; k += kRbThreads)
      reinterpret_cast<unsigned short *>(P)[(k % a) * NE + k / a] = lidx[A.max_items * at + k];
    P += rb_units(2 * a * NE);
    at += a;
  }
  uint2 *longs = reinterpret_cast<uint2 *>(P), *shorts = reinterpret_cast<uint2 *>(A.pkt + s_start + head);
  unsigned short *ids = reinterpret_cast<unsigned short *>(P + u_longs);
  int sc = 0, lc = 0, ic = 0, found = 0;
  for (int base = 0; base < ne; base += kRbThreads) {
    const int j = base + tid;
    const int rl = j < ne ? row_of(re, j) : 0;
    const int cnt = j < ne ? count_of(j, rl) : 0;
    int st, lt, idt;
    const int sa = sc + block_excl_scan(cnt > 0 && cnt <= kRbShort, &st);
    const int la = lc + block_excl_scan(cnt > kRbShort, &lt);
    int ia = ic + block_excl_scan(cnt > kRbShort ? cnt : 0, &idt);
    if (cnt > 0) {
      found += cnt;
      const unsigned pos = (unsigned)(rb[rl] + j - re[rl]);
      const int col = entry_col(j, rl);
      unsigned two[kRbShort] = {0u, (unsigned)(ca * ns)};
      if (cnt > kRbShort) longs[la] = make_uint2(pos, (unsigned)ia | (unsigned)(ia + cnt) << 16);
      int k = 0;
      for (int i = ro[rl]; i < ro[rl + 1]; ++i) {
        const int e = it[i] / ra, r = it[i] - e * ra;
        const int *c = cols + eloc[i] * ca;
        for (int q = 0; q < ca; ++q)
          if (c[q] == col) {
            const unsigned id = (unsigned)(q * ns + own[r * NE + eloc[i]]);
            if (cnt > kRbShort) ids[ia + k] = (unsigned short)id;
            else two[k] = id;
            ++k;
          }
      }
      if (cnt <= kRbShort) shorts[sa] = make_uint2(pos, two[0] | two[1] << 16);
    }
    sc += st;
    lc += lt;
    ic += idt;
  }
  __syncthreads();
  if (tid == 0) s_ids = 0;
  __syncthreads();
  if (found) atomicAdd(&s_ids, found);
  __syncthreads();
  if (tid == 0 && s_ids != ni * ca) atomicExch(&A.scal[kSFlag], 1);   // an entry the pattern lacks
}

}  // namespace op2b

using namespace op2b;

static void rowblk_release(RowBlocks *p, cudaStream_t s) {
  if (!p) return;
  dev_free(p->dir, s);
  dev_free(p->pkt, s);
  delete p;
}

extern "C" {

int op2b_row_blocks_build(uint64_t rmap_, uint64_t cmap_, int32_t nelem, int32_t ra, int32_t ca,
                          int32_t nrows, uint64_t rowptr_, uint64_t colidx_, int32_t region,
                          int32_t nstage, const uint64_t *stage_map, const int32_t *stage_arity,
                          int32_t ids, uint64_t stream, uint64_t *out) {
  OP2B_REQUIRE_INIT();
  if (nelem < 0 || ra <= 0 || ca <= 0 || nrows < 0 || region <= 0 || nstage < 0 || !out ||
      (nelem > 0 && (!rmap_ || !cmap_ || !rowptr_ || !colidx_)) || (nstage > 0 && (!stage_map || !stage_arity)))
    return set_error(OP2B_ERR_ARG, "row blocks: nelem %d arity %d/%d rows %d region %d", nelem, ra, ca, nrows,
                     region);
  *out = 0;
  const int64_t tot = (int64_t)nelem * ra;
  if (tot == 0 || nrows == 0 || tot * ca >= INT_MAX || nstage > kRbStages) return OP2B_OK;
  cudaStream_t s = stream_of(stream);
  const int32_t *rmap = reinterpret_cast<const int32_t *>(rmap_);
  RowBlocks *P = new RowBlocks();
  RbArgs A{};
  A.cmap = reinterpret_cast<const int32_t *>(cmap_);
  A.rowptr = reinterpret_cast<const int32_t *>(rowptr_);
  A.colidx = reinterpret_cast<const int32_t *>(colidx_);
  A.ra = ra;
  A.ca = ca;
  A.ids = ids ? 1 : 0;
  A.st.n = nstage;
  for (int q = 0; q < nstage; ++q) {
    A.st.map[q] = reinterpret_cast<const int32_t *>(stage_map[q]);
    A.st.arity[q] = stage_arity[q];
    A.st.rows += stage_arity[q];
  }
  int32_t *work = nullptr;
  auto done = [&](int rc, bool keep) {
    dev_free(work, s);
    if (!keep) rowblk_release(P, s);
    return rc;
  };
#define RB_TRY(call)                    \
  do {                                  \
    int _rc = (call);                   \
    if (_rc) return done(_rc, false);   \
  } while (0)
#define RB_CUDA(call) RB_TRY(check_cuda((call), #call))
  auto grid = [](int64_t n) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 8));
  };
  const int n = nelem, mean = 3 * region;
  int sbits = 0;
  while (sbits < 3 && (1 << sbits) < ra) ++sbits;
  const int most_seeds = n / mean * 2 + 32, nregions = most_seeds + n / region + 1;
  const int buckets = kRbLevels << sbits;
  const int64_t nbuckets = (int64_t)nregions * buckets, most_blocks = (int64_t)nregions + n / region + 1;
  if (nbuckets >= INT_MAX) return done(OP2B_OK, false);
  // one workspace; 64-bit keys first
  const int64_t words[] = {2LL * n, 2LL * nrows,                               // ekey, tkey
                           n, nbuckets + 1, nbuckets + 1, n + 1, nregions + 1,
                           nrows, nrows, tot + 1, nrows, nrows, nrows + 1, nrows + 1, tot, most_blocks + 1, kSCount};
  constexpr int kWords = sizeof words / sizeof words[0];
  int64_t at[kWords + 1] = {0};
  for (int k = 0; k < kWords; ++k) at[k + 1] = at[k] + (words[k] + 3) / 4 * 4;
  RB_TRY(dev_alloc((void **)&work, sizeof(int32_t) * (size_t)at[kWords], s));
  uint64_t *ekey = reinterpret_cast<uint64_t *>(work);
  unsigned long long *tkey = reinterpret_cast<unsigned long long *>(work + at[1]);
  int32_t *bucket = work + at[2], *bfirst = work + at[3], *cursor = work + at[4], *eorder = work + at[5],
          *pieces = work + at[6], *deg = work + at[8], *ranks = work + at[9], *order = work + at[10],
          *rank = work + at[11], *io = work + at[12], *eo = work + at[13], *list = work + at[14],
          *rstart = work + at[15], *scal = work + at[16];
  unsigned *first = reinterpret_cast<unsigned *>(work + at[7]);
  RB_CUDA(cudaMemsetAsync(scal, 0, sizeof(int32_t) * kSCount, s));
  RB_CUDA(cudaMemsetAsync(tkey, 0xff, sizeof(uint64_t) * nrows, s));
  RB_CUDA(cudaMemsetAsync(bfirst, 0, sizeof(int32_t) * (nbuckets + 1), s));
  RB_CUDA(cudaMemsetAsync(first, 0xff, sizeof(int32_t) * nrows, s));
  RB_CUDA(cudaMemsetAsync(deg, 0, sizeof(int32_t) * nrows, s));
  RB_CUDA(cudaMemsetAsync(io, 0, sizeof(int32_t) * (at[14] - at[12]), s));
  // regions of elements
  {
    int per_sm = 0, ra_ = ra, n_ = n, most = most_seeds, sb = sbits;
    RB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, rb_grow_kernel, 256, 0));
    int32_t *seed = eorder;      // the elements' order is written later
    rb_seed_kernel<<<grid(n + 1), 256, 0, s>>>(n, mean, seed);
    RB_TRY(device_excl_scan(seed, seed, (int64_t)n + 1, scal + kSScan, s));
    void *args[] = {&n_, &rmap, &ra_, &seed, &most, &sb, &ekey, &tkey, &scal};
    const int g = std::max(1, std::min(op2b_div_up(n, 256), sm_count() * per_sm));
    RB_CUDA(cudaLaunchCooperativeKernel((const void *)rb_grow_kernel, dim3(g), dim3(256), args, 0, s));
  }
  rb_bucket_kernel<<<grid(n), 256, 0, s>>>(n, ekey, most_seeds, region, sbits, bucket, bfirst);
  RB_TRY(device_excl_scan(bfirst, bfirst, nbuckets + 1, scal + kSScan, s));
  RB_CUDA(cudaMemcpyAsync(cursor, bfirst, sizeof(int32_t) * nbuckets, cudaMemcpyDeviceToDevice, s));
  rb_order_kernel<<<grid(n), 256, 0, s>>>(n, bucket, cursor, eorder);
  // rows, and the blocks they are cut into
  rb_first_kernel<<<grid(tot), 256, 0, s>>>(tot, ra, rmap, eorder, first, deg);
  rb_flag_kernel<<<grid(tot + 1), 256, 0, s>>>(tot, ra, rmap, eorder, first, ranks);
  RB_TRY(device_excl_scan(ranks, ranks, tot + 1, scal + kSUsed, s));
  rb_rows_kernel<<<grid(tot), 256, 0, s>>>(tot, ra, rmap, eorder, ranks, deg, A.rowptr, order, rank, io, eo);
  RB_TRY(device_excl_scan(io, io, (int64_t)nrows + 1, scal + kSScan, s));
  RB_TRY(device_excl_scan(eo, eo, (int64_t)nrows + 1, scal + kSScan + 1, s));
  rb_pieces_kernel<<<grid(nregions + 1), 256, 0, s>>>(nregions, buckets, ra, region * ra, bfirst, ranks, io, pieces);
  RB_TRY(device_excl_scan(pieces, pieces, nregions + 1, scal + kSScan + 2, s));
  rb_starts_kernel<<<grid(nregions), 256, 0, s>>>(nregions, buckets, ra, bfirst, ranks, io, pieces, rstart, scal);
  rb_scatter_kernel<<<grid(tot), 256, 0, s>>>(rmap, tot, rank, io, deg, list);
  RB_CUDA(cudaGetLastError());
  int32_t h[kSCount];
  RB_CUDA(cudaMemcpyAsync(h, scal, sizeof h, cudaMemcpyDeviceToHost, s));
  RB_CUDA(cudaStreamSynchronize(s));
  const int nblocks = h[kSBlocks];
  const int64_t mi = h[kSMaxItems], keys = mi * std::max((ca + 1) / 2, *std::max_element(A.st.arity, A.st.arity + kRbStages));
  // rows of too many elements for a block: the caller keeps its other form
  if (mi * ca > kRbMaxContrib || keys > kRbMaxKeys || mi * A.st.rows > 2 * kRbMaxKeys ||
      h[kSMaxRows] > 8192)
    return done(OP2B_OK, false);
  A.max_items = (int32_t)mi;
  A.max_rows = h[kSMaxRows];
  A.hash = 1;
  while (A.hash < keys) A.hash <<= 1;
  const int64_t smem = 4 * (2 * mi + 3LL * A.max_rows + 2 + 2LL * A.hash + mi * A.st.rows) +
                       2 * (mi + mi * A.st.rows + mi * ra);
  if (smem > smem_optin()) return done(OP2B_OK, false);
  A.order = order;
  A.rstart = rstart;
  A.io = io;
  A.eo = eo;
  A.list = list;
  A.scal = scal;
  RB_TRY(dev_alloc((void **)&P->dir, sizeof(int2) * (size_t)nblocks, s));
  A.dir = P->dir;
  A.cap = row_block_room(nelem, ra, ca, nrows, h[kSScan + 1], nblocks, A.ids, nstage, stage_arity);
  RB_CUDA(cudaFuncSetAttribute(rb_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (A.cap >= INT_MAX) return done(OP2B_OK, false);
    RB_TRY(dev_alloc((void **)&P->pkt, sizeof(uint4) * (size_t)A.cap, s));
    A.pkt = P->pkt;
    rb_build_kernel<<<nblocks, kRbThreads, smem, s>>>(A);
    RB_CUDA(cudaGetLastError());
    RB_CUDA(cudaMemcpyAsync(h, scal, sizeof h, cudaMemcpyDeviceToHost, s));
    RB_CUDA(cudaStreamSynchronize(s));
    if (h[kSFlag]) return done(OP2B_OK, false);
    int64_t taken;
    memcpy(&taken, h + kSCursor, sizeof taken);
    if (taken <= A.cap) break;
    A.cap = taken;
    dev_free(P->pkt, s);
    P->pkt = nullptr;
    RB_CUDA(cudaMemsetAsync(scal + kSCursor, 0, sizeof(int64_t), s));
  }
  P->nblocks = nblocks;
  P->max_items = A.max_items;
  P->max_packet = h[kSMaxPacket];
  memcpy(P->max_targets, h + kSMaxTargets, sizeof P->max_targets);
  *out = reinterpret_cast<uint64_t>(P);
  return done(OP2B_OK, true);
#undef RB_TRY
#undef RB_CUDA
}

int op2b_row_blocks_info(uint64_t rb, int32_t *nblocks, int32_t *max_items, int32_t *max_packet,
                         int32_t *max_targets, uint64_t *dir, uint64_t *packets) {
  RowBlocks *P = reinterpret_cast<RowBlocks *>(rb);
  if (!P) return set_error(OP2B_ERR_ARG, "null row blocks");
  if (nblocks) *nblocks = P->nblocks;
  if (max_items) *max_items = P->max_items;
  if (max_packet) *max_packet = P->max_packet;
  if (max_targets) memcpy(max_targets, P->max_targets, sizeof P->max_targets);
  if (dir) *dir = reinterpret_cast<uint64_t>(P->dir);
  if (packets) *packets = reinterpret_cast<uint64_t>(P->pkt);
  return OP2B_OK;
}

int op2b_row_blocks_free(uint64_t rb) {
  OP2B_REQUIRE_INIT();
  rowblk_release(reinterpret_cast<RowBlocks *>(rb), stream_of(0));
  return OP2B_OK;
}

}  // extern "C"
