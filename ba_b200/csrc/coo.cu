// COO -> CSR on the device: CPU_CSR_lMatrix::TransformFromCOO
// (lmp/lmatrix_csr_cpu.cc:883-906), i.e. coo_2_csr (lmp/lmatrix_formats.h:
// 320-452), for matrices assembled as coordinate triplets.
//
// The reference counts the entries of each row, scatters them in input order
// and then sorts every row by column with a selection sort that keeps
// duplicates (and, being a selection sort with swaps, does not keep them in
// input order).  Here the same result comes from:
//   1. one pass over the triplets that checks every index (a bad triplet
//      fails the upload) and counts the rows with atomics, each entry keeping
//      the count it met as its place in the row,
//   2. the row pointer as the counts' prefix sum,
//   3. a scatter of (column, input position) pairs to their places, in windows
//      that fit in the L2 where the triplets come in no order; within a
//      row these come in the order the atomics ran in, which is never used:
//   4. the row sort, one warp per row: when the row's columns are distinct
//      the sorted row is unique, ranks come from shuffles and each value from
//      its input position; when a column repeats, the entries are first put
//      in input order (by the positions, which are distinct) and then sorted
//      by the reference's selection sort itself; rows above 32 entries go
//      through a worklist to a second kernel,
//   5. the diagonal positions and the longest row, as b200la_csr_upload does.
// What bounds it: random 32-byte sectors, one written (3) and one read (4)
// per entry, and the atomics.  A stable radix sort by row (four passes over
// 12-byte records) and a separate gather took 1.4 + 1.2 of 3.8 ms on 57 M
// triplets.
// The result is the reference's CSR bit for bit, duplicates included.
#include <algorithm>
#include <climits>
#include <cstring>

#include "internal.cuh"

namespace b200la {

// First bad triplet (smallest index), or all ones when every index is in
// range; place[i] = how many entries of its row were counted before entry i.
// Four entries in flight per thread.  With FAR one block in kFarBlocks
// counts, of one entry in four, the neighbours in the input whose rows lie
// span or more apart (far).
constexpr int kFarBlocks = 8;
template <bool FAR>
__global__ void __launch_bounds__(kBlock) coo_count_kernel(int64_t nnz, int nrow, int ncol,
                                                           const int *__restrict__ rows,
                                                           const int *__restrict__ cols, int *__restrict__ count,
                                                           int *__restrict__ place, unsigned long long *bad, int span,
                                                           int *far) {
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const bool sample = FAR && blockIdx.x % kFarBlocks == 0;
  int jumps = 0;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < nnz; i0 += U * stride) {
    int r[U], c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = i0 + u * stride < nnz;
      r[u] = in ? rows[i0 + u * stride] : 0;
      c[u] = in ? cols[i0 + u * stride] : 0;
    }
    if (sample && i0 + 1 < nnz) jumps += abs(rows[i0 + 1] - r[0]) >= span ? 1 : 0;
    int p[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride;
      if (i >= nnz) continue;
      if (r[u] < 0 || r[u] >= nrow || c[u] < 0 || c[u] >= ncol) {
        atomicMin(bad, (unsigned long long)i);
        p[u] = 0;
      } else {
        p[u] = atomicAdd(count + r[u], 1);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * stride < nnz) place[i0 + u * stride] = p[u];
  }
  if (sample) {
    jumps = (int)warp_sum((double)jumps);
    if ((threadIdx.x & 31) == 0 && jumps) atomicAdd(far, jumps);
  }
}

// ---- prefix sum of the row counts: a block's sum, the blocks' offsets, the
// row pointer (kScanRows rows a block, kScanEach a thread)
constexpr int kScanEach = 8;
constexpr int kScanRows = kBlock * kScanEach;

__device__ __forceinline__ int warp_scan(int v) {  // inclusive
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive prefix of v over the block's threads; *total = the block's sum.
__device__ __forceinline__ int block_scan(int v, int *total) {
  __shared__ int part[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  const int inc = warp_scan(v);
  if (lane == 31) part[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const int s = warp_scan(lane < nw ? part[lane] : 0);
    part[lane] = s;
  }
  __syncthreads();
  const int before = warp > 0 ? part[warp - 1] : 0;
  *total = part[nw - 1];
  __syncthreads();
  return before + inc - v;
}

__global__ void __launch_bounds__(kBlock) coo_block_sum_kernel(int nrow, const int *__restrict__ count,
                                                               int *__restrict__ sums) {
  const int64_t first = (int64_t)blockIdx.x * kScanRows + (int64_t)threadIdx.x * kScanEach;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanEach; ++k)
    if (first + k < nrow) s += count[first + k];
  int total;
  block_scan(s, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// sums -> their exclusive prefix, one block
__global__ void __launch_bounds__(1024) coo_scan_sums_kernel(int blocks, int *sums) {
  int carry = 0;
  for (int b0 = 0; b0 < blocks; b0 += (int)blockDim.x) {
    const int i = b0 + (int)threadIdx.x;
    const int v = i < blocks ? sums[i] : 0;
    int total;
    const int ex = block_scan(v, &total);
    if (i < blocks) sums[i] = carry + ex;
    carry += total;
  }
}

__global__ void __launch_bounds__(kBlock) coo_rowptr_kernel(int nrow, int nnz, const int *__restrict__ count,
                                                            const int *__restrict__ sums, int *__restrict__ rowptr) {
  const int64_t first = (int64_t)blockIdx.x * kScanRows + (int64_t)threadIdx.x * kScanEach;
  int c[kScanEach], s = 0;
#pragma unroll
  for (int k = 0; k < kScanEach; ++k) {
    c[k] = first + k < nrow ? count[first + k] : 0;
    s += c[k];
  }
  int total;
  int at = sums[blockIdx.x] + block_scan(s, &total);
#pragma unroll
  for (int k = 0; k < kScanEach; ++k) {
    if (first + k < nrow) rowptr[first + k] = at;
    at += c[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) rowptr[nrow] = nnz;
}

// Each triplet's column (high word) and input position (low word) to its
// place in its row; with PART only those of rows row0 .. row1 - 1.
// Triplets in random order write random 8 bytes of the pairs' array.  Beyond
// the L2 each write costs a sector of its own, so the array is then filled in
// windows that stay in the L2, one launch each, which re-reads the rows (4
// bytes an entry and launch) and lets a sector's entries meet.  us a
// conversion, one launch and windows (radix sort by row in brackets): 96^3,
// 24 M triplets, 193 MB of pairs 1,448 1,267 (1,591), 128^3, 57 M 4,173 3,510
// (3,796), 140^3, 75 M 5,704 4,960 (5,007); windows of half the size 3,580 on
// 128^3, of twice 3,535.
constexpr int kMaxWindows = 8;

template <bool PART>
__global__ void __launch_bounds__(kBlock) coo_scatter_kernel(int64_t nnz, int row0, int row1,
                                                             const int *__restrict__ rows,
                                                             const int *__restrict__ cols,
                                                             const int *__restrict__ place,
                                                             const int *__restrict__ rowptr,
                                                             unsigned long long *__restrict__ out) {
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < nnz; i0 += U * stride) {
    int at[U], c[U], r[U];
    bool mine[U];  // PART: the row decides; else the other loads need not wait for it
    if (PART) {
#pragma unroll
      for (int u = 0; u < U; ++u) r[u] = i0 + u * stride < nnz ? rows[i0 + u * stride] : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) mine[u] = PART ? r[u] >= row0 && r[u] < row1 : i0 + u * stride < nnz;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (mine[u]) {
        at[u] = __ldg(rowptr + (PART ? r[u] : rows[i0 + u * stride])) + place[i0 + u * stride];
        c[u] = cols[i0 + u * stride];
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (mine[u])
        out[at[u]] = ((unsigned long long)(unsigned)c[u] << 32) | (unsigned long long)(unsigned)(i0 + u * stride);
  }
}

// The reference's per-row selection sort (lmatrix_formats.h:405-431) on
// col[b, e) / val[b, e) in place, then the first diagonal entry; one lane.
template <typename T>
__device__ void row_selection_sort(int k, int b, int e, int *col, T *val, int *diag) {
  for (int i = b; i != e; ++i) {
    int mi = i, mc = col[i];
    for (int j = i + 1; j < e; ++j)
      if (col[j] < mc) {
        mi = j;
        mc = col[j];
      }
    const int tc = col[i];
    col[i] = col[mi];
    col[mi] = tc;
    const T tv = val[i];
    val[i] = val[mi];
    val[mi] = tv;
  }
  int d = -1;
  for (int i = b; i != e; ++i)
    if (col[i] == k) {
      d = i;
      break;
    }
  diag[k] = d;
}

// The same by a warp, which looks for each minimum together (long rows).
template <typename T>
__device__ void warp_selection_sort(int k, int b, int e, int *col, T *val, int *diag) {
  const int lane = threadIdx.x & 31;
  for (int i = b; i != e; ++i) {
    // the first of the smallest columns (columns are < ncol <= INT_MAX)
    int mi = INT_MAX, mc = INT_MAX;
    for (int j = i + lane; j < e; j += 32)
      if (col[j] < mc) {
        mi = j;
        mc = col[j];
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const int oi = __shfl_xor_sync(0xffffffffu, mi, o), oc = __shfl_xor_sync(0xffffffffu, mc, o);
      if (oc < mc || (oc == mc && oi < mi)) {
        mi = oi;
        mc = oc;
      }
    }
    if (lane == 0) {
      const int tc = col[i];
      col[i] = col[mi];
      col[mi] = tc;
      const T tv = val[i];
      val[i] = val[mi];
      val[mi] = tv;
    }
    __syncwarp();
  }
  int d = INT_MAX;
  for (int i = b + lane; i < e; i += 32)
    if (col[i] == k) {
      d = i;
      break;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) d = min(d, __shfl_xor_sync(0xffffffffu, d, o));
  if (lane == 0) diag[k] = d == INT_MAX ? -1 : d;
  __syncwarp();
}

// Row sort, one warp per row of up to 32 entries (lane l holds one of them).
// When the row's columns are distinct the sorted row is unique, so each entry
// goes straight to b + (number of smaller columns), ranks taken with shuffles;
// that equals the reference's selection sort.  A row with a repeated column
// (found by __match_any_sync) is first put in input order, then sorted by the
// selection sort itself, because there the order of equal columns depends on
// its swaps.  Longer rows are appended to a worklist for
// coo_long_rows_kernel.  Also the diagonal positions and the longest row.
template <typename T, typename S>
__global__ void __launch_bounds__(kBlock) coo_rowsort_kernel(int nrow, const int *__restrict__ rowptr,
                                                             const unsigned long long *__restrict__ packed,
                                                             const S *__restrict__ vals, int *col, T *val, int *diag,
                                                             int *max_row, int *long_rows, int *n_long) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int longest = 0;
  for (int64_t kk = warp; kk < nrow; kk += nwarps) {
    const int k = (int)kk;
    const int b = rowptr[k], e = rowptr[k + 1], L = e - b;
    longest = L > longest ? L : longest;
    if (L > 32) {
      if (lane == 0) long_rows[atomicAdd(n_long, 1)] = k;
      continue;
    }
    const bool valid = lane < L;
    const unsigned long long q = valid ? packed[b + lane] : 0ull;
    const int c = valid ? (int)(q >> 32) : INT_MAX;  // columns are < ncol <= INT_MAX
    const unsigned pos = (unsigned)q;
    T v = T(0);
    if (valid) v = (T)vals[pos];
    const unsigned same = __match_any_sync(0xffffffffu, c);
    if (__any_sync(0xffffffffu, valid && __popc(same) > 1)) {
      int r = 0;
      for (int j = 0; j < L; ++j) r += __shfl_sync(0xffffffffu, pos, j) < pos ? 1 : 0;
      if (valid) {
        col[b + r] = c;
        val[b + r] = v;
      }
      __syncwarp();
      if (lane == 0) row_selection_sort(k, b, e, col, val, diag);
      __syncwarp();
      continue;
    }
    int r = 0;
    for (int j = 0; j < L; ++j) r += __shfl_sync(0xffffffffu, c, j) < c ? 1 : 0;
    if (valid) {
      col[b + r] = c;
      val[b + r] = v;
    }
    // columns are distinct here, so at most one lane holds the diagonal
    const unsigned dm = __ballot_sync(0xffffffffu, valid && c == k);
    int rd = -1;
    if (dm) rd = __shfl_sync(0xffffffffu, r, __ffs(dm) - 1);
    if (lane == 0) diag[k] = dm ? b + rd : -1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  if (lane == 0 && longest > 0) atomicMax(max_row, longest);
}

// Rows longer than 32 entries (from coo_rowsort_kernel's worklist), one warp
// per row: lane l holds entries l, l + 32, ... (up to kMaxQ * 32 = 256) and the
// ranks come from shuffles as above.  A repeated column or a longer row takes
// the selection sort, after its entries were put in input order; only those
// rows pay for the ranks of the positions.  Measured, us for the conversion of
// shuffled triplets (every row's positions ranked and the selection sort on one
// lane in brackets): 100,000 rows of 100 entries 1,465 (1,641), 40,000 of 256
// 1,492 (1,820), 20,000 of 300 1,925 (5,490).
constexpr int kMaxQ = 8;

// Row b .. e of the pairs to col / val in input order: lane l ranks kMaxQ of
// its entries per pass over the row's positions.
template <typename T, typename S>
__device__ __forceinline__ void row_in_input_order(int b, int e, const unsigned long long *__restrict__ packed,
                                                   const S *__restrict__ vals, int *col, T *val) {
  const int lane = threadIdx.x & 31, L = e - b;
  for (int i0 = lane; i0 < L; i0 += 32 * kMaxQ) {
    unsigned long long own[kMaxQ];
    int rank[kMaxQ];
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) {
      own[q] = i0 + q * 32 < L ? packed[b + i0 + q * 32] : 0ull;
      rank[q] = 0;
    }
    for (int t = 0; t < L; ++t) {
      const unsigned pos = (unsigned)packed[b + t];
#pragma unroll
      for (int q = 0; q < kMaxQ; ++q) rank[q] += pos < (unsigned)own[q] ? 1 : 0;
    }
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q)
      if (i0 + q * 32 < L) {
        col[b + rank[q]] = (int)(own[q] >> 32);
        val[b + rank[q]] = (T)vals[(unsigned)own[q]];
      }
  }
  __syncwarp();
}

template <typename T, typename S>
__global__ void __launch_bounds__(kBlock) coo_long_rows_kernel(const int *__restrict__ rowptr,
                                                               const unsigned long long *__restrict__ packed,
                                                               const S *__restrict__ vals, int *col, T *val,
                                                               int *diag, const int *__restrict__ long_rows,
                                                               const int *__restrict__ n_long) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int count = *n_long;
  for (int64_t w = warp; w < count; w += nwarps) {
    const int k = long_rows[w];
    const int b = rowptr[k], e = rowptr[k + 1], L = e - b;
    if (L > kMaxQ * 32) {
      row_in_input_order<T, S>(b, e, packed, vals, col, val);
      warp_selection_sort(k, b, e, col, val, diag);
      continue;
    }
    const int nq = (L + 31) >> 5;
    int c[kMaxQ], rank[kMaxQ];
    T v[kMaxQ];
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) {
      const int i = q * 32 + lane;
      const bool ok = q < nq && i < L;
      const unsigned long long own = ok ? packed[b + i] : 0ull;
      c[q] = ok ? (int)(own >> 32) : INT_MAX;
      v[q] = ok ? (T)vals[(unsigned)own] : T(0);
      rank[q] = 0;
    }
    bool dup = false;
#pragma unroll
    for (int qj = 0; qj < kMaxQ; ++qj) {
      if (qj >= nq) break;
      const int jn = L - qj * 32 < 32 ? L - qj * 32 : 32;
      for (int jl = 0; jl < jn; ++jl) {
        const int cj = __shfl_sync(0xffffffffu, c[qj], jl);
#pragma unroll
        for (int q = 0; q < kMaxQ; ++q)
          if (q < nq && q * 32 + lane < L) {
            rank[q] += cj < c[q] ? 1 : 0;
            dup |= cj == c[q] && !(qj == q && jl == lane);
          }
      }
    }
    if (__any_sync(0xffffffffu, dup)) {
      row_in_input_order<T, S>(b, e, packed, vals, col, val);
      warp_selection_sort(k, b, e, col, val, diag);
      continue;
    }
    int d = INT_MAX;
#pragma unroll
    for (int q = 0; q < kMaxQ; ++q) {
      const int i = q * 32 + lane;
      if (q < nq && i < L) {
        col[b + rank[q]] = c[q];
        val[b + rank[q]] = v[q];
        if (c[q] == k) d = b + rank[q];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d = min(d, __shfl_xor_sync(0xffffffffu, d, o));
    if (lane == 0) diag[k] = d == INT_MAX ? -1 : d;
  }
}

static int grid_1d(b200la_ctx c, int64_t work) {
  int64_t g = (work + kBlock - 1) / kBlock;
  const int64_t cap = (int64_t)c->num_sms * 16;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

}  // namespace b200la

using namespace b200la;

extern "C" int b200la_coo_upload(b200la_ctx c, int nrow, int ncol, int64_t nnz, const int *rows, const int *cols,
                                 const void *val, int val_dtype, int dtype, int device_input, b200la_mat *out) {
  B_CHECK(c && out, B200LA_ERR_INVALID, "coo_upload: null argument");
  B_CHECK(nrow >= 0 && ncol >= 0, B200LA_ERR_INVALID, "coo_upload: negative size %d x %d", nrow, ncol);
  B_CHECK(nnz >= 0 && nnz <= INT_MAX, B200LA_ERR_INVALID, "coo_upload: nnz %lld not in [0, 2^31)", (long long)nnz);
  B_CHECK(dtype == B200LA_F64 || dtype == B200LA_F32, B200LA_ERR_DTYPE, "coo_upload: dtype %d", dtype);
  B_CHECK(val_dtype == B200LA_F64 || val_dtype == B200LA_F32, B200LA_ERR_DTYPE, "coo_upload: value dtype %d",
          val_dtype);
  B_CHECK(nnz == 0 || (rows && cols && val), B200LA_ERR_INVALID, "coo_upload: null triplet arrays");
  cudaStream_t s = c->stream;
  const size_t nz = (size_t)(nnz > 0 ? nnz : 1);
  const size_t vsz = dtype_size(val_dtype);
  // scratch: device triplets (when given host arrays), pairs by row, block sums
  int *d_rows = nullptr, *d_cols = nullptr, *sums = nullptr;
  unsigned long long *packed = nullptr;
  void *d_vals = nullptr;
  unsigned long long *bad = nullptr;
  int *max_row_d = nullptr, *n_long_d = nullptr, *long_rows = nullptr;
  b200la_mat m = new b200la_mat_s();
  m->ctx = c;
  m->nrow = nrow;
  m->ncol = ncol;
  m->nnz = nnz;
  m->dtype = dtype;
  int rc = B200LA_OK;
  auto cu = [&](cudaError_t e, const char *what) {
    if (e != cudaSuccess && rc == B200LA_OK)
      rc = fail(e == cudaErrorMemoryAllocation ? B200LA_ERR_NOMEM : B200LA_ERR_CUDA, "coo_upload: %s: %s", what,
                cudaGetErrorString(e));
    return rc == B200LA_OK;
  };
  do {
    if (!cu(cudaMallocAsync(&m->rowptr, sizeof(int) * ((size_t)nrow + 1), s), "allocation") ||
        !cu(cudaMallocAsync(&m->col, sizeof(int) * nz, s), "allocation") ||
        !cu(cudaMallocAsync(&m->val, dtype_size(dtype) * nz, s), "allocation") ||
        !cu(cudaMallocAsync(&m->diag, sizeof(int) * (size_t)(nrow > 0 ? nrow : 1), s), "allocation") ||
        !cu(cudaMallocAsync(&bad, sizeof(unsigned long long) + 4 * sizeof(int), s), "allocation"))
      break;
    max_row_d = reinterpret_cast<int *>(bad + 1);
    n_long_d = max_row_d + 1;
    int *far_d = max_row_d + 2;
    const unsigned long long none = ~0ull;
    if (!cu(cudaMemcpyAsync(bad, &none, sizeof(none), cudaMemcpyHostToDevice, s), "copy") ||
        !cu(cudaMemsetAsync(max_row_d, 0, 4 * sizeof(int), s), "memset"))
      break;
    if (nnz == 0) {
      if (!cu(cudaMemsetAsync(m->rowptr, 0, sizeof(int) * ((size_t)nrow + 1), s), "memset")) break;
      if (nrow > 0 && !cu(cudaMemsetAsync(m->diag, 0xff, sizeof(int) * (size_t)nrow, s), "memset")) break;
      break;
    }
    const int *r_in = rows, *c_in = cols;
    const void *v_in = val;
    if (!device_input) {
      if (!cu(cudaMallocAsync(&d_rows, sizeof(int) * nz, s), "allocation") ||
          !cu(cudaMallocAsync(&d_cols, sizeof(int) * nz, s), "allocation") ||
          !cu(cudaMallocAsync(&d_vals, vsz * nz, s), "allocation") ||
          !cu(cudaMemcpyAsync(d_rows, rows, sizeof(int) * nnz, cudaMemcpyHostToDevice, s), "copy") ||
          !cu(cudaMemcpyAsync(d_cols, cols, sizeof(int) * nnz, cudaMemcpyHostToDevice, s), "copy") ||
          !cu(cudaMemcpyAsync(d_vals, val, vsz * nnz, cudaMemcpyHostToDevice, s), "copy"))
        break;
      r_in = d_rows;
      c_in = d_cols;
      v_in = d_vals;
    }
    // the diagonal positions' buffer holds the row counts and the columns'
    // the entries' places until the row sort writes them
    int *count = m->diag, *place = m->col;
    const int g = grid_1d(c, (nnz + 3) / 4);
    if (nrow > 0 && !cu(cudaMemsetAsync(count, 0, sizeof(int) * (size_t)nrow, s), "memset")) break;
    // windows of the scatter (three quarters of the L2 each), where the order
    // of the triplets needs them: more than one neighbour in eight apart
    int l2 = 0;
    if (!cu(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, c->device), "L2 size")) break;
    const int64_t window = std::max<int64_t>(1, (int64_t)l2 / 4 * 3);
    int windows = (int)std::min<int64_t>(kMaxWindows, ((int64_t)sizeof(unsigned long long) * nnz + window - 1) / window);
    const int span = windows > 1 ? std::max(1, nrow / windows) : 0;
    const auto count_rows = span > 0 ? coo_count_kernel<true> : coo_count_kernel<false>;
    count_rows<<<g, kBlock, 0, s>>>(nnz, nrow, ncol, r_in, c_in, count, place, bad, span, far_d);
    struct {
      unsigned long long bad;
      int max_row, n_long, far, pad;
    } seen = {};
    if (!cu(cudaGetLastError(), "check") ||
        !cu(cudaMemcpyAsync(&seen, bad, sizeof(seen), cudaMemcpyDeviceToHost, s), "copy") ||
        !cu(cudaStreamSynchronize(s), "check"))
      break;
    if (seen.bad != ~0ull) {
      rc = fail(B200LA_ERR_MATRIX, "coo_upload: triplet %llu has an index out of range", seen.bad);
      break;
    }
    const int blocks = (int)(((int64_t)nrow + kScanRows - 1) / kScanRows);  // nrow > 0: every index is in range
    if (!cu(cudaMallocAsync(&sums, sizeof(int) * (size_t)blocks, s), "allocation") ||
        !cu(cudaMallocAsync(&packed, sizeof(unsigned long long) * nz, s), "allocation") ||
        !cu(cudaMallocAsync(&long_rows, sizeof(int) * (size_t)nrow, s), "allocation"))
      break;
    coo_block_sum_kernel<<<blocks, kBlock, 0, s>>>(nrow, count, sums);
    coo_scan_sums_kernel<<<1, 1024, 0, s>>>(blocks, sums);
    coo_rowptr_kernel<<<blocks, kBlock, 0, s>>>(nrow, (int)nnz, count, sums, m->rowptr);
    if (seen.far <= nnz / (8 * 4 * kFarBlocks)) windows = 1;
    for (int k = 0; k < windows; ++k) {
      const int row0 = (int)((int64_t)nrow * k / windows), row1 = (int)((int64_t)nrow * (k + 1) / windows);
      if (windows == 1)
        coo_scatter_kernel<false><<<g, kBlock, 0, s>>>(nnz, row0, row1, r_in, c_in, place, m->rowptr, packed);
      else
        coo_scatter_kernel<true><<<g, kBlock, 0, s>>>(nnz, row0, row1, r_in, c_in, place, m->rowptr, packed);
    }
    const int gr = grid_1d(c, (int64_t)nrow * 32);
    auto sort_rows = [&](auto t, auto u) {
      using T = decltype(t);
      using S = decltype(u);
      coo_rowsort_kernel<T, S><<<gr, kBlock, 0, s>>>(nrow, m->rowptr, packed, (const S *)v_in, m->col, (T *)m->val,
                                                     m->diag, max_row_d, long_rows, n_long_d);
      coo_long_rows_kernel<T, S><<<c->num_sms * 8, kBlock, 0, s>>>(m->rowptr, packed, (const S *)v_in, m->col,
                                                                   (T *)m->val, m->diag, long_rows, n_long_d);
    };
    if (dtype == B200LA_F64) {
      if (val_dtype == B200LA_F64) sort_rows(double(), double());
      else sort_rows(double(), float());
    } else {
      if (val_dtype == B200LA_F64) sort_rows(float(), double());
      else sort_rows(float(), float());
    }
    cu(cudaGetLastError(), "kernels");
  } while (false);
  int hmax = 0;
  if (rc == B200LA_OK && bad) {
    cu(cudaMemcpyAsync(&hmax, max_row_d, sizeof(int), cudaMemcpyDeviceToHost, s), "copy");
    cu(cudaStreamSynchronize(s), "sync");
  }
  void *scratch[] = {d_rows, d_cols, d_vals, sums, packed, bad, long_rows};
  for (void *p : scratch)
    if (p) cudaFreeAsync(p, s);
  if (rc != B200LA_OK) {
    cudaStreamSynchronize(s);
    b200la_mat_destroy(m);
    return rc;
  }
  m->max_row = hmax;
  const double avg = nrow ? (double)nnz / nrow : 0.0;
  m->format = B200LA_FMT_CSR;
  m->param = csr_start_lanes(nrow, avg, hmax, c->num_sms);
  *out = m;
  return B200LA_OK;
}

// CopyTo a host CSR: the uploaded (or built) CSR arrays as stored.
extern "C" int b200la_mat_download(b200la_mat m, int *rowptr, int *col, void *val) {
  B_CHECK(m && rowptr && (m->nnz == 0 || (col && val)), B200LA_ERR_INVALID, "mat_download: null argument");
  cudaStream_t s = m->ctx->stream;
  B_CUDA(cudaMemcpyAsync(rowptr, m->rowptr, sizeof(int) * ((size_t)m->nrow + 1), cudaMemcpyDeviceToHost, s));
  if (m->nnz) {
    B_CUDA(cudaMemcpyAsync(col, m->col, sizeof(int) * (size_t)m->nnz, cudaMemcpyDeviceToHost, s));
    B_CUDA(cudaMemcpyAsync(val, m->val, dtype_size(m->dtype) * (size_t)m->nnz, cudaMemcpyDeviceToHost, s));
  }
  B_CUDA(cudaStreamSynchronize(s));
  return B200LA_OK;
}
