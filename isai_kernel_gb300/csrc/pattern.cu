// Format conversions and sparsity patterns on the GPU (integer work,
// bit-exact with the reference's host builders).
//
//   csr_to_bsr5                            csr2bsr.h:14
//   bsr2csr_cusparse                       bsr2csr.h:19
//   build_bcsc_pattern_from_bsr_scalarILU  isai_bsr.h:246
//   build_triangular_bcsr_pattern_from_A   bcsc2bcsr.h:11
//   build_map_bcsc2bcsr_host               bcsc2bcsr.h:32
//   reorder_bcsc_val_to_bcsr_bs5           bcsc2bcsr.h:63
//   bcsc_to_bcsr                           bcsc2bcsrAndSpMV.h:76
//
// Transposes use atomic cursors for the scatter and then a warp-per-segment
// rank sort (rank = number of smaller keys in the segment), so the output
// order is ascending and independent of the atomic order.
#include <algorithm>

#include "common.cuh"
#include "scan.cuh"

namespace bilu {

namespace {

constexpr int kT = 256;

// err[0]: first offending block row (atomicMin), err[1]: kind (atomicMax)
// kind 1 = column out of range, 2 = columns not strictly ascending,
// 3 = missing diagonal block, 4 = row pointer decreasing
__device__ __forceinline__ void report(int* err, int row, int kind) {
  atomicMin(err, row);
  atomicMax(err + 1, kind);
}

__global__ void k_fill_int(int* p, long long n, int v) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// Per block row: validate and count qualifying off-diagonal entries into
// the column counters (ISAI pattern) -- cnt[] preset to 1 for the diagonal.
__global__ void k_isai_count(int nb, const int* __restrict__ row, const int* __restrict__ col,
                             int lower, int* cnt, int* err) {
  const int br = blockIdx.x * blockDim.x + threadIdx.x;
  int s = 0, e = 0;
  if (br < nb) {
    s = row[br];
    e = row[br + 1];
    if (e < s) report(err, br, 4);
  }
  for_row_entries(br, s, max(s, e), [&](int r, int p) {
    const int bc = col[p];
    if (bc < 0 || bc >= nb) { report(err, r, 1); return; }
    if (p > row[r] && bc <= col[p - 1]) { report(err, r, 2); return; }
    if (bc == r || (lower ? bc > r : bc < r)) return;
    atomicAdd(cnt + bc, 1);
  });
}

__global__ void k_isai_scatter(int nb, const int* __restrict__ row, const int* __restrict__ col,
                               int lower, const int* __restrict__ Mptr, int* cursor, int* tmp) {
  const int br = blockIdx.x * blockDim.x + threadIdx.x;
  int s = 0, e = 0;
  if (br < nb) {
    s = row[br];
    e = row[br + 1];
    tmp[Mptr[br] + atomicAdd(cursor + br, 1)] = br;
  }
  for_row_entries(br, s, max(s, e), [&](int r, int p) {
    const int bc = col[p];
    if (bc == r || bc < 0 || bc >= nb) return;
    if (lower ? (bc > r) : (bc < r)) return;
    tmp[Mptr[bc] + atomicAdd(cursor + bc, 1)] = r;
  });
}

// out[ptr[s] + rank(key)] = key (and payload), keys distinct inside a segment:
// L lanes per segment (8: most hold a handful of keys), the warp together on
// segments of more than kSharedRow keys.  A warp's segments are 8 apart, so that
// neighbouring hubs go to different warps (three dense columns beside one another,
// 5000 rows, the transposed product: 16.6 ms in one warp, 5.8 so).
__device__ __forceinline__ void rank_one(int i, int s, int e, const int* __restrict__ key,
                                         const int* __restrict__ pay, int* __restrict__ key_out,
                                         int* __restrict__ pay_out) {
  const int k = key[i];
  int rank = 0;
  for (int j = s; j < e; ++j) rank += key[j] < k;
  key_out[s + rank] = k;
  if (pay_out) pay_out[s + rank] = pay[i];
}

template <int L>
__global__ void __launch_bounds__(kT) k_segment_rank_sort(int nseg, const int* __restrict__ ptr,
                                                          const int* __restrict__ key,
                                                          const int* __restrict__ pay,
                                                          int* __restrict__ key_out,
                                                          int* __restrict__ pay_out) {
  constexpr int NW = kT / 32, PER = 32 / L;  // warps, segments of a warp
  const int lane = threadIdx.x & 31, l = lane % L;
  const long long sg =
      ((long long)blockIdx.x * PER + lane / L) * NW + (int)(threadIdx.x >> 5);
  const int s = sg < nseg ? ptr[sg] : 0, e = sg < nseg ? ptr[sg + 1] : 0;
  const bool shared = L < 32 && e - s > kSharedRow;
  if (!shared)
    for (int i = s + l; i < e; i += L) rank_one(i, s, e, key, pay, key_out, pay_out);
  unsigned todo = __ballot_sync(0xffffffffu, shared && l == 0);
  while (todo) {
    const int from = __ffs(todo) - 1;
    todo &= todo - 1;
    const int a = __shfl_sync(0xffffffffu, s, from), b = __shfl_sync(0xffffffffu, e, from);
    for (int i = a + lane; i < b; i += 32) rank_one(i, a, b, key, pay, key_out, pay_out);
  }
}

// A warp per segment while the chip holds as many warps.
int segment_rank_sort(int nseg, const int* ptr, const int* key, const int* pay, int* key_out,
                      int* pay_out, cudaStream_t st) {
  if (nseg <= 152 * 64)
    k_segment_rank_sort<32><<<ceil_div(nseg, kT / 32), kT, 0, st>>>(nseg, ptr, key, pay, key_out,
                                                                    pay_out);
  else
    k_segment_rank_sort<8><<<ceil_div(nseg, kT / 8), kT, 0, st>>>(nseg, ptr, key, pay, key_out,
                                                                  pay_out);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// Rows of the lower (upper) triangle in their stored order: a thread per row,
// the warp together on rows of more than kSharedRow entries (ballots keep the
// order).  FILL false: out[r] = entries; true: Tcol at out[r] (= Trow).
template <bool FILL>
__global__ void k_tri(int nb, const int* __restrict__ row, const int* __restrict__ col, int lower,
                      int* out, int* __restrict__ Tcol) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int s = r < nb ? row[r] : 0, e = r < nb ? row[r + 1] : 0;
  const bool shared = e - s > kSharedRow;
  if (r < nb && !shared) {
    int o = FILL ? out[r] : 0;
    for (int p = s; p < e; ++p) {
      const int c = col[p];
      if (!(lower ? (c <= r) : (c >= r))) continue;
      if (FILL) Tcol[o] = c;
      ++o;
    }
    if (!FILL) out[r] = o;
  }
  unsigned todo = __ballot_sync(0xffffffffu, shared);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int q = __shfl_sync(0xffffffffu, r, src);
    const int a = __shfl_sync(0xffffffffu, s, src), b = __shfl_sync(0xffffffffu, e, src);
    int o = FILL ? out[q] : 0;
    for (int p0 = a; p0 < b; p0 += 32) {
      const int c = p0 + lane < b ? col[p0 + lane] : 0;
      const bool in = p0 + lane < b && (lower ? (c <= q) : (c >= q));
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (FILL && in) Tcol[o + __popc(m & ((1u << lane) - 1u))] = c;
      o += __popc(m);
    }
    if (!FILL && lane == 0) out[q] = o;
  }
}

// Thread per BCSC column: binary search of each entry in its BCSR row.
__global__ void k_map(int nb, const int* __restrict__ cptr, const int* __restrict__ cind,
                      const int* __restrict__ rrow, const int* __restrict__ rcol,
                      int* __restrict__ map, unsigned long long* bad) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nb) return;
  for (int k = cptr[c]; k < cptr[c + 1]; ++k) {
    int r = cind[k];
    int lo = rrow[r], hi = rrow[r + 1] - 1, found = -1;
    while (lo <= hi) {
      int m = (lo + hi) >> 1, v = rcol[m];
      if (v == c) { found = m; break; }
      if (v < c) lo = m + 1; else hi = m - 1;
    }
    if (found < 0) {
      // first mismatch in the reference's visiting order (column-major)
      atomicMin(bad, ((unsigned long long)(unsigned)c << 32) | (unsigned)r);
      map[k] = -1;
    } else {
      map[k] = found;
    }
  }
}

// dst[map[k]] = src[k], blocks of bs2 doubles copied as double2 pairs when
// the block size allows it.
__global__ void k_reorder(long long nnzb, int bs2, const int* __restrict__ map,
                          const double* __restrict__ src, double* __restrict__ dst) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = nnzb * bs2;
  if (t >= total) return;
  long long k = t / bs2;
  int e = (int)(t - k * bs2);
  dst[(long long)map[k] * bs2 + e] = src[t];
}

__global__ void k_reorder_v2(long long nnzb, int half, const int* __restrict__ map,
                             const double2* __restrict__ src, double2* __restrict__ dst) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = nnzb * half;
  if (t >= total) return;
  long long k = t / half;
  int e = (int)(t - k * half);
  dst[(long long)map[k] * half + e] = src[t];
}

// bcsc -> bcsr: count blocks per row
__global__ void k_count_rows(long long nnzb, const int* __restrict__ ind, int mb, int* cnt,
                             int* err) {
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nnzb) return;
  int r = ind[k];
  if (r < 0 || r >= mb) { report(err, r, 1); return; }
  atomicAdd(cnt + r, 1);
}

__global__ void k_csc_scatter(int nbcol, const int* __restrict__ cptr,
                              const int* __restrict__ cind, const int* __restrict__ rptr,
                              int* cursor, int* key, int* src) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = c < nbcol ? cptr[c] : 0, e = c < nbcol ? cptr[c + 1] : 0;
  for_row_entries(c, s, max(s, e), [&](int q, int k) {
    const int r = cind[k];
    const int d = rptr[r] + atomicAdd(cursor + r, 1);
    key[d] = q;
    src[d] = k;
  });
}

// cnt[col[k]] += 1 over all blocks; words: 0 a column out of range, 1 the block
// count (read on the device, so that the host need not wait for it).
__global__ void __launch_bounds__(kT) k_count_cols(int mb, const int* __restrict__ row,
                                                   const int* __restrict__ col, int* cnt,
                                                   int* words) {
  const int nnzb = __ldg(row + mb);
  if (blockIdx.x == 0 && threadIdx.x == 0) words[1] = nnzb;
  for (long long k = (long long)blockIdx.x * kT + threadIdx.x; k < nnzb;
       k += (long long)gridDim.x * kT) {
    const int c = col[k];
    if (c < 0 || c >= mb) words[0] = 1;
    else atomicAdd(cnt + c, 1);
  }
}

// words[2] = the longest segment
__global__ void __launch_bounds__(kT) k_longest(int n, const int* __restrict__ ptr, int* words) {
  int m = 0;
  for (long long i = (long long)blockIdx.x * kT + threadIdx.x; i < n;
       i += (long long)gridDim.x * kT)
    m = max(m, ptr[i + 1] - ptr[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(words + 2, m);
}

__global__ void k_gather_blocks(long long nnzb, int bs2, const int* __restrict__ src,
                                const double* __restrict__ in, double* __restrict__ out) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nnzb * bs2) return;
  long long d = t / bs2;
  int e = (int)(t - d * bs2);
  out[t] = in[(long long)src[d] * bs2 + e];
}

// csr -> bsr.  A group of GW lanes per block row (4 lanes for block sizes up
// to 4, else 8; 8 or 4 block rows per warp), lane r walking scalar row r: the
// group merges its rows by block column -- the smallest block column any lane
// stands on is the next block, and the lanes standing on it consume their
// entries of that block.  Linear in the entries, with every entry read once
// per phase; the fill phase adds a lane's entries, in their order, into its
// row of the group's block in shared memory and the group writes the block
// out as one contiguous run.  What bounds it is the entries' traffic: 50^3
// 7-point grid of 5x5 blocks, 80% stored (17 M entries): 298 us for the whole
// conversion, 5897 us with the searches for every row.
//
// The merge needs block columns that never decrease along a scalar row.  A
// lane that sees one decrease marks its block row, which the whole warp then
// does over again with the searches below (up to cubic in the row's entries;
// only files with unsorted rows come here).
template <int BS>
struct C2b {
  static constexpr int GW = BS <= 4 ? 4 : 8;  // lanes per block row
  static constexpr int NG = 32 / GW;          // block rows per warp
};

// Count the distinct block columns of a block row with unsorted scalar rows,
// one warp: an entry counts if no earlier entry of the segment has the same
// block column.
__device__ __noinline__ int c2b_count_unsorted(int br, int bs, const int* __restrict__ crow,
                                               const int* __restrict__ ccol, int ncols) {
  const int lane = threadIdx.x & 31;
  const int s = crow[br * bs], e = crow[br * bs + bs];
  int c = 0;
  for (int i = s + lane; i < e; i += 32) {
    const int gc = ccol[i];
    if (gc < 0 || gc >= ncols) continue;  // reported by the merge
    const int bc = gc / bs;
    bool first = true;
    for (int j = s; j < i && first; ++j) first = (ccol[j] / bs) != bc;
    c += first;
  }
  return warp_sum(c);
}

__device__ __noinline__ void c2b_fill_unsorted(int br, int bs, const int* __restrict__ crow,
                                               const int* __restrict__ ccol,
                                               const double* __restrict__ cval,
                                               const int* __restrict__ brow, int* bcol,
                                               double* bval) {
  const int lane = threadIdx.x & 31;
  const int s = crow[br * bs], e = crow[br * bs + bs];
  const int base = brow[br], u = brow[br + 1] - base;
  // 1) distinct block columns in ascending order (column range checked by
  //    the count phase, which reports BILU_ERR_PATTERN)
  for (int i = s + lane; i < e; i += 32) {
    int bc = ccol[i] / bs;
    bool first = true;
    for (int j = s; j < i && first; ++j) first = (ccol[j] / bs) != bc;
    if (!first) continue;
    int rank = 0;
    for (int j = s; j < e; ++j) {
      int bj = ccol[j] / bs;
      if (bj < bc) {
        bool fj = true;
        for (int q = s; q < j && fj; ++q) fj = (ccol[q] / bs) != bj;
        rank += fj;
      }
    }
    if (rank < u) bcol[base + rank] = bc;
  }
  // 2) zero the blocks
  int bs2 = bs * bs;
  for (long long t = lane; t < (long long)u * bs2; t += 32) bval[(long long)base * bs2 + t] = 0.0;
  __syncwarp();
  // 3) lane per scalar row accumulates its entries in order (the reference's
  //    std::map accumulation order for a given position)
  if (lane < bs) {
    int rr = br * bs + lane;
    for (int p = crow[rr]; p < crow[rr + 1]; ++p) {
      int gc = ccol[p], bc = gc / bs, lc = gc - bc * bs;
      if (gc < 0) continue;
      int lo = 0, hi = u - 1, k = -1;
      while (lo <= hi) {
        int m = (lo + hi) >> 1, v = bcol[base + m];
        if (v == bc) { k = m; break; }
        if (v < bc) lo = m + 1; else hi = m - 1;
      }
      if (k >= 0) bval[((long long)(base + k) * bs + lane) * bs + lc] += cval[p];
    }
  }
}

// FILL false: out[br] = number of blocks.  FILL true: bcol / bval of the
// block rows at out[] (= bsrRowPtr).
template <int BS, bool FILL>
__global__ void __launch_bounds__(kT) k_c2b(int nb, const int* __restrict__ crow,
                                            const int* __restrict__ ccol,
                                            const double* __restrict__ cval, int ncols, int* out,
                                            int* bcol, double* bval, int* err) {
  constexpr int GW = C2b<BS>::GW, NG = C2b<BS>::NG, BS2 = BS * BS;
  constexpr int kNone = 0x7fffffff;
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ double tiles[FILL ? (kT / GW) * BS2 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / GW, r = lane - g * GW;
  const long long br0 = ((long long)blockIdx.x * (kT / 32) + warp) * NG;  // the warp's first
  const long long br = br0 + g;
  double* tile = tiles + (FILL ? (warp * NG + g) * BS2 : 0);
  int p = 0, e = 0, base = 0, u = 0;
  if (br < nb) {
    if (r < BS) {
      p = __ldg(crow + br * BS + r);
      e = __ldg(crow + br * BS + r + 1);
    }
    if (FILL) {
      base = out[br];
      u = out[br + 1] - base;
      for (int t = r; t < BS2; t += GW) tile[t] = 0.0;
    }
  }
  // the entry the lane stands on: its scalar and block column and its value
  int gc = 0, bc = kNone;
  double v = 0.0;
  auto fetch = [&]() {
    bc = kNone;
    for (; p < e; ++p) {
      gc = __ldg(ccol + p);
      if (gc >= 0 && gc < ncols) {
        bc = gc / BS;
        if (FILL) v = __ldg(cval + p);
        return;
      }
      if (!FILL) report(err, (int)br, 1);
    }
  };
  fetch();
  int k = 0;
  bool unsorted = false;
  while (true) {
    int m = bc;
#pragma unroll
    for (int o = GW / 2; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(kAll, m, o));
    if (__all_sync(kAll, m == kNone)) break;
    if (FILL) __syncwarp();  // the tile is zero again
    while (bc == m && m != kNone) {
      if (FILL) tile[r * BS + (gc - bc * BS)] += v;
      ++p;
      fetch();
      unsorted |= bc < m;
    }
    if (FILL) {
      __syncwarp();
      if (m != kNone && k < u) {
        double* dst = bval + (long long)(base + k) * BS2;
        if (r == 0) bcol[base + k] = m;
#pragma unroll
        for (int t0 = 0; t0 < BS2; t0 += GW) {
          const int t = t0 + r;
          if (t < BS2) {
            dst[t] = tile[t];
            tile[t] = 0.0;
          }
        }
      }
    }
    k += m != kNone;
  }
  const unsigned bad = __ballot_sync(kAll, unsorted);
  if (!FILL && br < nb && r == 0) out[br] = k;
  if (bad) {
    __syncwarp();
    for (int q = 0; q < NG; ++q) {
      if (!((bad >> (q * GW)) & ((1u << GW) - 1u))) continue;
      if (FILL) {
        c2b_fill_unsorted((int)(br0 + q), BS, crow, ccol, cval, out, bcol, bval);
      } else {
        const int n = c2b_count_unsorted((int)(br0 + q), BS, crow, ccol, ncols);
        if (lane == 0) out[br0 + q] = n;
      }
    }
  }
}

template <bool FILL>
int launch_c2b(int nb, int bs, const int* crow, const int* ccol, const double* cval, int ncols,
               int* out, int* bcol, double* bval, int* err, cudaStream_t st) {
#define BILU_C2B(B)                                                                           \
  case B:                                                                                     \
    k_c2b<B, FILL><<<ceil_div(nb, (kT / 32) * C2b<B>::NG), kT, 0, st>>>(nb, crow, ccol, cval, \
                                                                        ncols, out, bcol,     \
                                                                        bval, err);           \
    break;
  switch (bs) {
    BILU_C2B(1) BILU_C2B(2) BILU_C2B(3) BILU_C2B(4)
    BILU_C2B(5) BILU_C2B(6) BILU_C2B(7) BILU_C2B(8)
    default: return BILU_ERR_ARG;
  }
#undef BILU_C2B
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// bsr -> csr (row direction): thread per (block, row r) writes bs entries.
__global__ void k_b2c_rowptr(int mb, int bs, const int* __restrict__ brow, int* __restrict__ crow) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > (long long)mb * bs) return;
  if (t == (long long)mb * bs) { crow[t] = brow[mb] * bs * bs; return; }
  int br = (int)(t / bs), r = (int)(t - (long long)br * bs);
  int len = brow[br + 1] - brow[br];
  crow[t] = brow[br] * bs * bs + r * len * bs;
}

__global__ void k_b2c_fill(int mb, int bs, long long nnzb, const int* __restrict__ brow,
                           const int* __restrict__ bcol, const double* __restrict__ bval,
                           const int* __restrict__ crow, int* __restrict__ ccol,
                           double* __restrict__ cval) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nnzb * bs) return;
  long long p = t / bs;
  int r = (int)(t - p * bs);
  // block row of block p: last br with brow[br] <= p
  int lo = 0, hi = mb - 1;
  while (lo < hi) {
    int m = (lo + hi + 1) >> 1;
    if (brow[m] <= p) lo = m; else hi = m - 1;
  }
  int br = lo;
  int k = (int)(p - brow[br]);
  long long o = (long long)crow[(long long)br * bs + r] + (long long)k * bs;
  int bc = bcol[p];
  for (int c = 0; c < bs; ++c) {
    ccol[o + c] = bc * bs + c;
    cval[o + c] = bval[(p * bs + r) * bs + c];
  }
}

// Structure of both ISAI sides of a pattern in one pass each (the setup's form of
// k_isai_count / k_tri: the counts of M_L and M_U, of both triangles, and the
// longest rows together, so that the host waits once).  Column counters cL, cU,
// row counters tL, tU; words: 0 error kind, 1 longest row of the pattern, 2 / 3
// of its lower / upper triangle, 8 to 10 the blocks in long rows of the three.
__global__ void __launch_bounds__(kT) k_isai_both_count(int nb, const int* __restrict__ row,
                                                        const int* __restrict__ col, int* cL,
                                                        int* cU, int* __restrict__ tL,
                                                        int* __restrict__ tU, int* words) {
  const int br = blockIdx.x * blockDim.x + threadIdx.x;
  int s = 0, e = 0, nL = 0, nU = 0;
  if (br < nb) {
    s = row[br];
    e = row[br + 1];
    if (e < s) {
      atomicMax(words, 4);
      e = s;
    }
    int lo = s, hi = e;  // first column >= br (rows in order; checked below)
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      if (col[m] < br) lo = m + 1; else hi = m;
    }
    nL = lo - s + (lo < e && col[lo] == br);
    nU = e - lo;
    tL[br] = nL;
    tU[br] = nU;
    atomicAdd(cL + br, 1);  // the diagonal block of the column
    atomicAdd(cU + br, 1);
  }
  for_row_entries(br, s, e, [&](int r, int p) {
    const int bc = col[p];
    if (bc < 0 || bc >= nb) { atomicMax(words, 1); return; }
    if (p > row[r] && bc <= col[p - 1]) { atomicMax(words, 2); return; }
    if (bc < r) atomicAdd(cL + bc, 1);
    else if (bc > r) atomicAdd(cU + bc, 1);
  });
  const int a = __reduce_max_sync(0xffffffffu, e - s), b = __reduce_max_sync(0xffffffffu, nL),
            c = __reduce_max_sync(0xffffffffu, nU);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(words + 1, a);
    atomicMax(words + 2, b);
    atomicMax(words + 3, c);
  }
  if (a > kLongSpmvRow) {  // the triangles' rows are no longer than the pattern's
    auto add = [&](int n, int* to) {
      const int h = __reduce_add_sync(0xffffffffu, n > kLongSpmvRow ? n : 0);
      if ((threadIdx.x & 31) == 0 && h > 0) atomicAdd(to, h);
    };
    add(e - s, words + 8);
    add(nL, words + 9);
    add(nU, words + 10);
  }
}

// Both triangles' columns (BCSR order) and, per column, the rows of M_L / M_U
// with their BCSR positions (in any order: k_segment_rank_sort follows).  The
// BCSR position of an entry is known here, so the BCSC -> BCSR map is a payload
// of that sort instead of a search.
__global__ void __launch_bounds__(kT) k_isai_both_fill(
    int nb, const int* __restrict__ row, const int* __restrict__ col,
    const int* __restrict__ mL, const int* __restrict__ mU, const int* __restrict__ tL,
    const int* __restrict__ tU, int* curL, int* curU, int* __restrict__ tcolL,
    int* __restrict__ tcolU, int* __restrict__ keyL, int* __restrict__ payL,
    int* __restrict__ keyU, int* __restrict__ payU) {
  const int br = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = br < nb ? row[br] : 0, e = br < nb ? row[br + 1] : 0;
  for_row_entries(br, s, e, [&](int r, int p) {
    const int c = col[p];
    if (c <= r) {
      const int t = tL[r] + (p - row[r]);
      tcolL[t] = c;
      const int d = mL[c] + atomicAdd(curL + c, 1);
      keyL[d] = r;
      payL[d] = t;
    }
    if (c >= r) {
      const int t = tU[r + 1] - (row[r + 1] - p);
      tcolU[t] = c;
      const int d = mU[c] + atomicAdd(curU + c, 1);
      keyU[d] = r;
      payU[d] = t;
    }
  });
}

int read_err(int* d_err, int* h_err, cudaStream_t st) {
  BILU_TRY_CUDA(cudaMemcpyAsync(h_err, d_err, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaStreamSynchronize(st));
  return BILU_OK;
}

int init_err(int* d_err, cudaStream_t st) {
  int init[2] = {0x7fffffff, 0};
  BILU_TRY_CUDA(cudaMemcpyAsync(d_err, init, sizeof(init), cudaMemcpyHostToDevice, st));
  return BILU_OK;
}

}  // namespace

// --------------------------------------------------------------- ISAI pattern
size_t isai_pattern_ws(int nb, long long nnzb) {
  return carve_size(sizeof(int) * 2) + carve_size(sizeof(int) * (size_t)(nb + 1)) +
         carve_size(sizeof(int) * (size_t)(nnzb + nb)) + scan_ws_bytes(nb + 1);
}

int isai_pattern_colptr_impl(int nb, const int* row, const int* col, int lower, int* Mptr,
                             int* h_nnz, Carver& ws, cudaStream_t st) {
  int* err = ws.take<int>(2);
  if (!err) return BILU_ERR_WORKSPACE;
  BILU_TRY(init_err(err, st));
  if (nb > 0) {
    k_fill_int<<<ceil_div(nb, kT), kT, 0, st>>>(Mptr, nb, 1);
    BILU_LAUNCH_CHECK();
    k_isai_count<<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, lower, Mptr, err);
    BILU_LAUNCH_CHECK();
  }
  BILU_TRY(scan_exclusive(Mptr, Mptr, nb, h_nnz, ws, st));
  int h_err[2];
  BILU_TRY(read_err(err, h_err, st));
  if (h_err[1] != 0) return BILU_ERR_PATTERN;
  return BILU_OK;
}

int isai_pattern_fill_impl(int nb, const int* row, const int* col, int lower, const int* Mptr,
                           int* Mind, int mnnz, Carver& ws, cudaStream_t st) {
  int* cursor = ws.take<int>((size_t)nb + 1);
  int* tmp = ws.take<int>((size_t)mnnz + 1);
  if (!cursor || !tmp) return BILU_ERR_WORKSPACE;
  if (nb == 0) return BILU_OK;
  BILU_TRY_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int) * nb, st));
  k_isai_scatter<<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, lower, Mptr, cursor, tmp);
  BILU_LAUNCH_CHECK();
  return segment_rank_sort(nb, Mptr, tmp, nullptr, Mind, nullptr, st);
}

// --------------------------------------------------------------- both ISAI sides
size_t isai_both_ws(int nb, long long nnz) {
  return carve_size(sizeof(int) * 12) + scan_multi_ws_bytes(nb + 1) +
         2 * carve_size(sizeof(int) * ((size_t)nb + 1)) +
         4 * carve_size(sizeof(int) * (size_t)(nnz + 1));
}

// Column pointers of M_L and M_U and row pointers of the triangles of pattern
// (row, col); h_nnz: blocks of M_L, M_U, the lower and the upper triangle;
// h_longest: longest row of the pattern and of its triangles, then their blocks in
// long rows.  One host synchronisation.
int isai_both_count(int nb, const int* row, const int* col, int* mL, int* mU, int* tL, int* tU,
                    int* h_nnz, int* h_longest, Carver& ws, cudaStream_t st) {
  int* words = ws.take<int>(12);
  if (!words) return BILU_ERR_WORKSPACE;
  BILU_TRY_CUDA(cudaMemsetAsync(words, 0, sizeof(int) * 12, st));
  BILU_TRY_CUDA(cudaMemsetAsync(mL, 0, sizeof(int) * nb, st));
  BILU_TRY_CUDA(cudaMemsetAsync(mU, 0, sizeof(int) * nb, st));
  k_isai_both_count<<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, mL, mU, tL, tU, words);
  BILU_LAUNCH_CHECK();
  const ScanSets sets = {{mL, mU, tL, tU}, {nb, nb, nb, nb}};
  BILU_TRY(scan_exclusive_multi(4, sets, words + 4, ws, st));
  int h[12];
  BILU_TRY_CUDA(cudaMemcpyAsync(h, words, sizeof(h), cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaStreamSynchronize(st));
  if (h[0] != 0) return BILU_ERR_PATTERN;
  for (int i = 0; i < 4; ++i) h_nnz[i] = h[4 + i];
  for (int i = 0; i < 3; ++i) {
    h_longest[i] = h[1 + i];
    h_longest[3 + i] = h[8 + i];
  }
  return BILU_OK;
}

// Mind / Tcol / map of both sides (nL, nU blocks), after isai_both_count.
int isai_both_fill(int nb, const int* row, const int* col, const int* mL, const int* mU,
                   const int* tL, const int* tU, int nL, int nU, int* indL, int* indU,
                   int* tcolL, int* tcolU, int* mapL, int* mapU, Carver& ws, cudaStream_t st) {
  int* cur = ws.take<int>(2 * (size_t)nb);
  int* keyL = ws.take<int>((size_t)nL);
  int* payL = ws.take<int>((size_t)nL);
  int* keyU = ws.take<int>((size_t)nU);
  int* payU = ws.take<int>((size_t)nU);
  if (!cur || !keyL || !payL || !keyU || !payU) return BILU_ERR_WORKSPACE;
  BILU_TRY_CUDA(cudaMemsetAsync(cur, 0, sizeof(int) * 2 * nb, st));
  k_isai_both_fill<<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, mL, mU, tL, tU, cur, cur + nb,
                                                    tcolL, tcolU, keyL, payL, keyU, payU);
  BILU_LAUNCH_CHECK();
  BILU_TRY(segment_rank_sort(nb, mL, keyL, payL, indL, mapL, st));
  return segment_rank_sort(nb, mU, keyU, payU, indU, mapU, st);
}

// --------------------------------------------------------------- tri pattern
int tri_pattern_rowptr_impl(int nb, const int* row, const int* col, int lower, int* Trow,
                            int* h_nnz, Carver& ws, cudaStream_t st) {
  if (nb > 0) {
    k_tri<false><<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, lower, Trow, nullptr);
    BILU_LAUNCH_CHECK();
  }
  return scan_exclusive(Trow, Trow, nb, h_nnz, ws, st);
}

int tri_pattern_fill_impl(int nb, const int* row, const int* col, int lower, const int* Trow,
                          int* Tcol, cudaStream_t st) {
  if (nb == 0) return BILU_OK;
  k_tri<true><<<ceil_div(nb, kT), kT, 0, st>>>(nb, row, col, lower, const_cast<int*>(Trow), Tcol);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// --------------------------------------------------------------- map / reorder
int map_impl(int nb, const int* cptr, const int* cind, const int* rrow, const int* rcol, int* map,
             int* h_bad, Carver& ws, cudaStream_t st) {
  unsigned long long* bad = ws.take<unsigned long long>(1);
  if (!bad) return BILU_ERR_WORKSPACE;
  unsigned long long init = ~0ull, hb = 0;
  BILU_TRY_CUDA(cudaMemcpyAsync(bad, &init, sizeof(init), cudaMemcpyHostToDevice, st));
  if (nb > 0) {
    k_map<<<ceil_div(nb, kT), kT, 0, st>>>(nb, cptr, cind, rrow, rcol, map, bad);
    BILU_LAUNCH_CHECK();
  }
  BILU_TRY_CUDA(cudaMemcpyAsync(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaStreamSynchronize(st));
  if (hb != ~0ull) {
    if (h_bad) {
      h_bad[0] = (int)(hb & 0xffffffffu);
      h_bad[1] = (int)(hb >> 32);
    }
    return BILU_ERR_PATTERN;
  }
  return BILU_OK;
}

int reorder_impl(long long nnzb, int bs, const int* map, const double* src, double* dst,
                 cudaStream_t st) {
  if (nnzb == 0) return BILU_OK;
  int bs2 = bs * bs;
  if (bs2 % 2 == 0) {
    long long total = nnzb * (bs2 / 2);
    k_reorder_v2<<<ceil_div(total, kT), kT, 0, st>>>(nnzb, bs2 / 2, map, (const double2*)src,
                                                     (double2*)dst);
  } else {
    long long total = nnzb * bs2;
    k_reorder<<<ceil_div(total, kT), kT, 0, st>>>(nnzb, bs2, map, src, dst);
  }
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

// --------------------------------------------------------------- transpose
size_t transpose_ws(int mb, long long nnzb) {
  return carve_size(sizeof(int) * 2) + carve_size(sizeof(int) * (size_t)(mb + 1)) +
         3 * carve_size(sizeof(int) * (size_t)(nnzb + 1)) + scan_ws_bytes(mb + 1);
}

// The entries of a transposed pattern whose row pointer is known: rind
// ascending inside a row, src[d] = index of entry d in the given pattern.
int transpose_fill(int mb, int nbcol, const int* cptr, const int* cind, long long nnzb,
                   const int* rptr, int* rind, int* src, Carver& ws, cudaStream_t st) {
  int* cursor = ws.take<int>((size_t)mb + 1);
  int* key = ws.take<int>((size_t)nnzb + 1);
  int* pay = ws.take<int>((size_t)nnzb + 1);
  if (!cursor || !key || !pay) return BILU_ERR_WORKSPACE;
  if (mb == 0 || nnzb == 0) return BILU_OK;
  BILU_TRY_CUDA(cudaMemsetAsync(cursor, 0, sizeof(int) * mb, st));
  k_csc_scatter<<<ceil_div(nbcol, kT), kT, 0, st>>>(nbcol, cptr, cind, rptr, cursor, key, pay);
  BILU_LAUNCH_CHECK();
  return segment_rank_sort(mb, rptr, key, pay, rind, src, st);
}

// Row pointer of the transpose of a square pattern, its block count and longest
// row on the host (one synchronisation); BILU_ERR_PATTERN for a column out of
// range.
int transpose_count(int mb, const int* row, const int* col, int* trow, int* h_nnzb,
                    int* h_longest, Carver& ws, cudaStream_t st) {
  int* words = ws.take<int>(4);
  if (!words) return BILU_ERR_WORKSPACE;
  BILU_TRY_CUDA(cudaMemsetAsync(words, 0, sizeof(int) * 4, st));
  BILU_TRY_CUDA(cudaMemsetAsync(trow, 0, sizeof(int) * ((size_t)mb + 1), st));
  k_count_cols<<<152 * 8, kT, 0, st>>>(mb, row, col, trow, words);
  BILU_LAUNCH_CHECK();
  BILU_TRY(scan_exclusive(trow, trow, mb, nullptr, ws, st));
  k_longest<<<std::min<unsigned>(ceil_div(mb, kT), 152 * 8), kT, 0, st>>>(mb, trow, words);
  BILU_LAUNCH_CHECK();
  int h[4];
  BILU_TRY_CUDA(cudaMemcpyAsync(h, words, sizeof(h), cudaMemcpyDeviceToHost, st));
  BILU_TRY_CUDA(cudaStreamSynchronize(st));
  if (h[0]) return BILU_ERR_PATTERN;
  *h_nnzb = h[1];
  *h_longest = h[2];
  return BILU_OK;
}

// BCSC (cptr over nbcol columns) -> BCSR pattern with ascending columns and
// src[d] = BCSC index of BCSR entry d.
int transpose_pattern(int mb, int nbcol, const int* cptr, const int* cind, long long nnzb,
                      int* rptr, int* rind, int* src, Carver& ws, cudaStream_t st) {
  int* err = ws.take<int>(2);
  if (!err) return BILU_ERR_WORKSPACE;
  BILU_TRY(init_err(err, st));
  BILU_TRY_CUDA(cudaMemsetAsync(rptr, 0, sizeof(int) * (mb + 1), st));
  if (nnzb > 0) {
    k_count_rows<<<ceil_div(nnzb, kT), kT, 0, st>>>(nnzb, cind, mb, rptr, err);
    BILU_LAUNCH_CHECK();
  }
  BILU_TRY(scan_exclusive(rptr, rptr, mb, nullptr, ws, st));
  int h_err[2];
  BILU_TRY(read_err(err, h_err, st));
  if (h_err[1] != 0) return BILU_ERR_PATTERN;
  return transpose_fill(mb, nbcol, cptr, cind, nnzb, rptr, rind, src, ws, st);
}

int gather_blocks(long long nnzb, int bs, const int* src, const double* in, double* out,
                  cudaStream_t st) {
  if (nnzb == 0) return BILU_OK;
  long long total = nnzb * bs * bs;
  k_gather_blocks<<<ceil_div(total, kT), kT, 0, st>>>(nnzb, bs * bs, src, in, out);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}

}  // namespace bilu

using namespace bilu;

// --------------------------------------------------------------- C ABI
extern "C" size_t bilu_isai_pattern_ws_bytes(int nb, int nnzb) {
  return isai_pattern_ws(nb, nnzb);
}

extern "C" int bilu_isai_pattern_colptr(int nb, const int* d_Arow, const int* d_Acol, int lower,
                                        int* d_Mptr, int* h_nnz, void* d_ws, size_t ws_bytes,
                                        bilu_stream_t stream) {
  if (nb < 0 || !d_Mptr || (nb > 0 && (!d_Arow || !d_Acol))) return BILU_ERR_ARG;
  Carver ws(d_ws, ws_bytes);
  return isai_pattern_colptr_impl(nb, d_Arow, d_Acol, lower != 0, d_Mptr, h_nnz, ws, S(stream));
}

extern "C" int bilu_isai_pattern_fill(int nb, const int* d_Arow, const int* d_Acol, int lower,
                                      const int* d_Mptr, int* d_Mind, void* d_ws,
                                      size_t ws_bytes, bilu_stream_t stream) {
  if (nb < 0 || (nb > 0 && (!d_Arow || !d_Acol || !d_Mptr || !d_Mind))) return BILU_ERR_ARG;
  int mnnz = 0;  // bounded by nnzb(A) + nb, the size the workspace query used
  if (nb > 0)
    BILU_TRY_CUDA(cudaMemcpyAsync(&mnnz, d_Mptr + nb, sizeof(int), cudaMemcpyDeviceToHost,
                                  S(stream)));
  BILU_TRY_CUDA(cudaStreamSynchronize(S(stream)));
  Carver ws(d_ws, ws_bytes);
  if (!ws.take<int>(2)) return BILU_ERR_WORKSPACE;  // same layout as the count phase
  return isai_pattern_fill_impl(nb, d_Arow, d_Acol, lower != 0, d_Mptr, d_Mind, mnnz, ws,
                                S(stream));
}

extern "C" size_t bilu_tri_pattern_ws_bytes(int nb) { return scan_ws_bytes(nb + 1); }

extern "C" int bilu_tri_pattern_rowptr(int nb, const int* d_Arow, const int* d_Acol, int lower,
                                       int* d_Trow, int* h_nnz, void* d_ws, size_t ws_bytes,
                                       bilu_stream_t stream) {
  if (nb < 0 || !d_Trow || (nb > 0 && (!d_Arow || !d_Acol))) return BILU_ERR_ARG;
  Carver ws(d_ws, ws_bytes);
  return tri_pattern_rowptr_impl(nb, d_Arow, d_Acol, lower != 0, d_Trow, h_nnz, ws, S(stream));
}

extern "C" int bilu_tri_pattern_fill(int nb, const int* d_Arow, const int* d_Acol, int lower,
                                     const int* d_Trow, int* d_Tcol, bilu_stream_t stream) {
  if (nb < 0) return BILU_ERR_ARG;
  return tri_pattern_fill_impl(nb, d_Arow, d_Acol, lower != 0, d_Trow, d_Tcol, S(stream));
}

extern "C" size_t bilu_map_ws_bytes(void) { return carve_size(sizeof(unsigned long long)); }

extern "C" int bilu_map_bcsc2bcsr(int nb, const int* d_cscPtr, const int* d_cscInd,
                                  const int* d_csrRow, const int* d_csrCol, int* d_map,
                                  int* h_bad, void* d_ws, size_t ws_bytes,
                                  bilu_stream_t stream) {
  if (nb < 0) return BILU_ERR_ARG;
  Carver ws(d_ws, ws_bytes);
  return map_impl(nb, d_cscPtr, d_cscInd, d_csrRow, d_csrCol, d_map, h_bad, ws, S(stream));
}

extern "C" int bilu_reorder_bcsc_to_bcsr(int nnzb, int bs, const int* d_map, const double* d_src,
                                         double* d_dst, bilu_stream_t stream) {
  if (nnzb < 0 || bs < 1 || bs > 8) return BILU_ERR_ARG;
  return reorder_impl(nnzb, bs, d_map, d_src, d_dst, S(stream));
}

extern "C" size_t bilu_bcsc_to_bcsr_ws_bytes(int mb, int nnzb) {
  return transpose_ws(mb, nnzb) + carve_size(sizeof(int) * (size_t)(nnzb + 1));
}

extern "C" int bilu_bcsc_to_bcsr(int mb, int nbcol, int bs, const int* d_cscPtr,
                                 const int* d_cscInd, const double* d_cscVal, int* d_rowPtr,
                                 int* d_colInd, double* d_val, void* d_ws, size_t ws_bytes,
                                 bilu_stream_t stream) {
  if (mb < 0 || nbcol < 0 || bs < 1 || bs > 8) return BILU_ERR_ARG;
  int nnzb = 0;
  if (nbcol > 0)
    BILU_TRY_CUDA(cudaMemcpyAsync(&nnzb, d_cscPtr + nbcol, sizeof(int), cudaMemcpyDeviceToHost,
                                  S(stream)));
  BILU_TRY_CUDA(cudaStreamSynchronize(S(stream)));
  Carver ws(d_ws, ws_bytes);
  int* src = ws.take<int>((size_t)nnzb + 1);
  if (!src) return BILU_ERR_WORKSPACE;
  BILU_TRY(transpose_pattern(mb, nbcol, d_cscPtr, d_cscInd, nnzb, d_rowPtr, d_colInd, src, ws,
                             S(stream)));
  if (d_cscVal && d_val) BILU_TRY(gather_blocks(nnzb, bs, src, d_cscVal, d_val, S(stream)));
  return BILU_OK;
}

extern "C" size_t bilu_csr_to_bsr_ws_bytes(int n, int bs) {
  int nb = bs > 0 ? n / bs : 0;
  return carve_size(sizeof(int) * 2) + scan_ws_bytes(nb + 1);
}

extern "C" int bilu_csr_to_bsr_rowptr(int n, int bs, const int* d_csrRowPtr,
                                      const int* d_csrColInd, int* d_bsrRowPtr, int* h_nnzb,
                                      void* d_ws, size_t ws_bytes, bilu_stream_t stream) {
  if (n < 0 || bs < 1 || bs > 8 || n % bs) return BILU_ERR_ARG;
  int nb = n / bs;
  Carver ws(d_ws, ws_bytes);
  int* err = ws.take<int>(2);
  if (!err) return BILU_ERR_WORKSPACE;
  cudaStream_t st = S(stream);
  BILU_TRY(init_err(err, st));
  if (nb > 0) {
    BILU_TRY(launch_c2b<false>(nb, bs, d_csrRowPtr, d_csrColInd, nullptr, n, d_bsrRowPtr, nullptr,
                               nullptr, err, st));
  }
  BILU_TRY(scan_exclusive(d_bsrRowPtr, d_bsrRowPtr, nb, h_nnzb, ws, st));
  int h_err[2];
  BILU_TRY(read_err(err, h_err, st));
  return h_err[1] ? BILU_ERR_PATTERN : BILU_OK;
}

extern "C" int bilu_csr_to_bsr_fill(int n, int bs, const int* d_csrRowPtr, const int* d_csrColInd,
                                    const double* d_csrVal, const int* d_bsrRowPtr,
                                    int* d_bsrColInd, double* d_bsrVal, bilu_stream_t stream) {
  if (n < 0 || bs < 1 || bs > 8 || n % bs) return BILU_ERR_ARG;
  int nb = n / bs;
  if (nb == 0) return BILU_OK;
  return launch_c2b<true>(nb, bs, d_csrRowPtr, d_csrColInd, d_csrVal, n,
                          const_cast<int*>(d_bsrRowPtr), d_bsrColInd, d_bsrVal, nullptr,
                          S(stream));
}

extern "C" int bilu_bsr_to_csr(int mb, int bs, const int* d_bsrRowPtr, const int* d_bsrColInd,
                               const double* d_bsrVal, int* d_csrRowPtr, int* d_csrColInd,
                               double* d_csrVal, bilu_stream_t stream) {
  if (mb < 0 || bs < 1 || bs > 8) return BILU_ERR_ARG;
  cudaStream_t st = S(stream);
  int nnzb = 0;
  if (mb > 0) {
    BILU_TRY_CUDA(cudaMemcpyAsync(&nnzb, d_bsrRowPtr + mb, sizeof(int), cudaMemcpyDeviceToHost, st));
    BILU_TRY_CUDA(cudaStreamSynchronize(st));
  }
  long long nrow = (long long)mb * bs + 1;
  k_b2c_rowptr<<<ceil_div(nrow, kT), kT, 0, st>>>(mb, bs, d_bsrRowPtr, d_csrRowPtr);
  BILU_LAUNCH_CHECK();
  if (nnzb == 0) return BILU_OK;
  long long total = (long long)nnzb * bs;
  k_b2c_fill<<<ceil_div(total, kT), kT, 0, st>>>(mb, bs, nnzb, d_bsrRowPtr, d_bsrColInd,
                                                 d_bsrVal, d_csrRowPtr, d_csrColInd, d_csrVal);
  BILU_LAUNCH_CHECK();
  return BILU_OK;
}
