// Conjugate gradients with the whole system on chip: one thread-block cluster
// holds a system's matrix and Krylov vectors in its SMs' shared memory and
// registers and iterates without touching HBM.
//
// What bounds the streamed form on such systems: an iteration re-reads the
// matrix and six to thirteen vectors from HBM or L2, or, when they are small,
// waits on three kernel launches and grid-wide reductions (15 us an iteration
// whatever the size).  Here an iteration reads shared memory only (18 words a
// row for a 9-point row) and meets at two cluster barriers (0.5 us for 8
// blocks), so it is bound by shared-memory bandwidth for large systems and by
// the barriers for small ones.
//
// Fits: symmetric matrices whose every row's columns are the row plus a
// subset of one symmetric set of offsets +-off[0..H) (structured-grid FE
// couplings), symmetric up to rows that hold only their diagonal (Dirichlet
// rows as identity rows), see sym_row_ok.  Only the diagonal and the upper
// entries are kept, v_k(i) = a(i, i + off[k]); the lower entry a(i, i-off[k])
// is v_k(i - off[k]), which halves the bytes on chip.  Where row i holds only
// its diagonal, v_k(i) is the value of the other row, and row i's product is
// its diagonal's alone.
//
// Layout: block `rank` of the cluster owns rows r0 = rank * rpc ... and keeps
//   vv[k][q]  k = 0 (diagonal) .. H, rows r0 - halo .. r0 + rpc (the halo rows
//             are those whose upper entries its own rows' lower entries are)
//   pw[q]     the direction p over rows r0 - halo .. r0 + rpc + halo
//   registers r, Ap, invD and the correction (or solution) c of its own rows:
//             thread t's row j is r0 + t + j * NT
// with halo = off[H-1].  After an update the owner pushes z = invD r of the
// rows other blocks' windows cover into their zh (distributed shared memory);
// the cluster barrier of the r.r / r.z sum publishes them, and every block
// then forms p = z + beta p over its whole window, with the owner's bits.
// Products are added in ascending column order, as every schedule adds them.
#pragma once

#include "internal.cuh"

namespace b200la {

// 16 warps, four per scheduler, so a thread may use 128 registers (17 would
// leave 96); 17 FP32 rows a thread hold 257 x 257 nodes in 8 blocks
constexpr int kClThreads = 512;
constexpr int kClWarps = kClThreads / 32;
constexpr int kClMaxBlocks = 16;  // largest cluster (non-portable size)
constexpr int kClMaxOff = 13;     // upper offsets: 4 (2D, 9-point) or 13 (3D, 27-point)
constexpr int kClSums = 3;

// The matrix as the kernels read it when they fill shared memory.
template <typename V> struct ClMatrix {
  int n, H, halo;
  int off[kClMaxOff];  // ascending positive offsets
  const int *rowptr, *col;
  const V *val;
};

// Upper offsets of a symmetric set (ascending, 0 in the middle); 0 if the
// set is not symmetric or has too many.
inline int cl_offsets(const int *off, int len, int *up) {
  if (len < 3 || !(len & 1) || len / 2 > kClMaxOff || off[len / 2] != 0) return 0;
  const int H = len / 2;
  for (int k = 1; k <= H; ++k) {
    if (off[H - k] != -off[H + k]) return 0;
    up[k - 1] = off[H + k];
  }
  return H;
}

// Dynamic shared memory of one block whose threads hold `held` rows each
// (the instance's count): p window, values, halo z, sum slots.  The product
// loop also reads, and discards, the held * kClThreads - rpc rows past the
// block's own (multiply()); what follows the values takes that, and where it
// would not, the block gets the difference.
constexpr size_t cl_smem_bytes(int rpc, int halo, int H, int held, size_t ts) {
  const size_t HP = H <= 4 ? 4 : kClMaxOff;
  const size_t values = ts * ((size_t)rpc + 2 * (size_t)halo) + ts * (HP + 1) * ((size_t)rpc + halo);
  size_t b = values + ts * 2 * (size_t)halo;
  b = (b + 15) & ~(size_t)15;
  b += sizeof(double) * 2 * kClSums * kClMaxBlocks * kClWarps;
  const size_t past = values + ts * ((size_t)held * kClThreads - (size_t)rpc);
  return b > past ? b : past;
}
// 3,104 FP64 rows on instances of 9: 1,504 values past the end; with rows of
// 1 a thread on instances of 4 the block is enlarged.
static_assert(cl_smem_bytes(3104, 1, 4, 9, 8) >= 8 * (3106 + 4 * 3105 + 9 * kClThreads + 1), "reads past the block");
static_assert(cl_smem_bytes(32, 1, 4, 4, 8) >= 8 * (34 + 4 * 33 + 4 * kClThreads + 1), "reads past the block");
inline int cl_rows_per_block(int n, int blocks) { return ((n + blocks - 1) / blocks + 31) & ~31; }

// Launch configuration of `systems` clusters of `blocks` blocks (attr must
// outlive the launch).
inline cudaLaunchConfig_t cl_config(int blocks, size_t smem, cudaStream_t st, cudaLaunchAttribute (&attr)[1],
                                    int systems = 1) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)blocks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)blocks * (unsigned)systems);
  cfg.blockDim = dim3(kClThreads);
  cfg.dynamicSmemBytes = smem;
  return cfg;
}

// Rows whose off-diagonal entries are all zero (Dirichlet rows).
template <typename V>
__device__ __forceinline__ bool diag_only_row(const int *__restrict__ rowptr, const int *__restrict__ col,
                                              const V *__restrict__ val, int i) {
  for (int j = rowptr[i]; j < rowptr[i + 1]; ++j)
    if (col[j] != i && !(val[j] == V(0))) return false;
  return true;
}

// Whether row i fits the halved storage: every off-diagonal entry equals its
// mirror bit for bit (or both are zero), unless one of the two rows holds
// only its diagonal.  The structure must have been checked before.
template <typename V>
__device__ __forceinline__ bool sym_row_ok(const int *__restrict__ rowptr, const int *__restrict__ col,
                                           const V *__restrict__ val, int i) {
  const int b = rowptr[i], e = rowptr[i + 1];
  for (int j = b; j < e; ++j) {
    const int c = col[j];
    if (c == i) continue;
    const V a = val[j];
    V m = V(0);
    for (int q = rowptr[c]; q < rowptr[c + 1]; ++q)
      if (col[q] == i) {
        m = val[q];
        break;
      }
    bool same = a == V(0) && m == V(0);
    if (sizeof(V) == 8) same |= __double_as_longlong((double)a) == __double_as_longlong((double)m);
    else same |= __float_as_int((float)a) == __float_as_int((float)m);
    if (!same && !diag_only_row(rowptr, col, val, i) && !diag_only_row(rowptr, col, val, c)) return false;
  }
  return true;
}

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cl_cluster_id() {
  unsigned r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
// All threads of the cluster; orders shared and global memory (release /
// acquire at cluster scope).
__device__ __forceinline__ void cl_barrier(unsigned blocks) {
  if (blocks == 1) {
    __syncthreads();
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cl_remote(const void *p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cl_store(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store_if(bool on, unsigned addr, double v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared::cluster.f64 [%0], %1;\n\t}" ::"r"(addr),
               "d"(v), "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ void cl_store_if(bool on, unsigned addr, float v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared::cluster.f32 [%0], %1;\n\t}" ::"r"(addr),
               "f"(v), "r"((unsigned)on)
               : "memory");
}

// Sums of one thread's products, in FP64 whatever T is: for FP32 a conversion
// and an addition instead of the seven operations of a compensated FP32 sum.
struct ClAcc {
  double s = 0.0;
  template <typename T> __device__ __forceinline__ void add(T v) { s += (double)v; }
};

template <typename T, int H, int R, bool PRE> struct ClCg {
  static constexpr int NT = kClThreads;
  T *pw, *vv, *zh;
  double *slots;
  int off[H];
  int n, r0, rows, rpc, halo, VW;
  unsigned rank, blocks;
  T r[R], ap[R], d[R], c[R];
  unsigned zh_prev, zh_next;  // zh of the neighbouring blocks (shared::cluster addresses)
  unsigned diag_only;  // bit j: own row j holds only its diagonal

  template <typename V> __device__ __forceinline__ void carve(unsigned char *dyn, const ClMatrix<V> &m) {
    rank = cl_rank();
    blocks = cl_size();
    n = m.n;
    halo = m.halo;
    rpc = ((n + (int)blocks - 1) / (int)blocks + 31) & ~31;
    r0 = (int)rank * rpc;
    rows = max(0, min(rpc, n - r0));
    VW = rpc + halo;
#pragma unroll
    for (int k = 0; k < H; ++k) off[k] = k < m.H ? m.off[k] : 0;
    pw = reinterpret_cast<T *>(dyn);
    vv = pw + rpc + 2 * halo;
    zh = vv + (size_t)(H + 1) * VW;
    size_t b = sizeof(T) * ((size_t)rpc + 2 * halo + (size_t)(H + 1) * VW + 2 * (size_t)halo);
    b = (b + 15) & ~(size_t)15;
    slots = reinterpret_cast<double *>(dyn + b);
    zh_prev = cl_remote(zh, rank > 0 ? rank - 1 : 0);
    zh_next = cl_remote(zh, rank + 1 < blocks ? rank + 1 : rank);
    // rows past the block's own stay zero in the loops below
#pragma unroll
    for (int j = 0; j < R; ++j) r[j] = d[j] = c[j] = ap[j] = T(0);
  }

  // Zeroes the window arrays, then every row that reaches this block's vv
  // writes its entries: upper ones at its own index, lower ones at the
  // mirror's.  Equal mirrors write the same bits; rows that hold only their
  // diagonal write only that.
  template <typename V> __device__ __forceinline__ void fill(const ClMatrix<V> &m) {
    const int total = rpc + 2 * halo + (H + 1) * VW + 2 * halo;
    for (int q = threadIdx.x; q < total; q += NT) pw[q] = T(0);
    __syncthreads();
    const int base = r0 - halo;
    const int hi = min(n, r0 + rpc + halo);
    for (int i = max(0, base) + (int)threadIdx.x; i < hi; i += NT) {
      const int b = m.rowptr[i], e = m.rowptr[i + 1];
      const bool only = diag_only_row(m.rowptr, m.col, m.val, i);
      for (int j = b; j < e; ++j) {
        const int o = m.col[j] - i;
        const T v = (T)m.val[j];
        if (o == 0) {
          if (i - base < VW) vv[i - base] = v;
        } else if (!only) {
          const int a = o > 0 ? o : -o;
          const int at = (o > 0 ? i : i + o) - base;  // the upper entry's row in this window
          if (at < 0 || at >= VW) continue;
#pragma unroll
          for (int k = 0; k < H; ++k)
            if (off[k] == a) vv[(k + 1) * VW + at] = v;
        }
      }
    }
    diag_only = 0;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int li = (int)threadIdx.x + j * NT;
      if (li < rows && diag_only_row(m.rowptr, m.col, m.val, r0 + li)) diag_only |= 1u << j;
    }
    __syncthreads();
  }

  // pw over the window from a global vector (rows outside [0, n) stay 0).
  __device__ __forceinline__ void load_window(const T *p) {
    const int base = r0 - halo;
    const int hi = min(n, r0 + rpc + halo);
    for (int i = max(0, base) + (int)threadIdx.x; i < hi; i += NT) pw[i - base] = __ldcg(p + i);
  }

  // f(j, li) for this thread's own rows
  template <typename F> __device__ __forceinline__ void each(F &&f) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int li = (int)threadIdx.x + j * NT;
      if (li < rows) f(j, li);
    }
  }

  // ap = A p; returns this thread's share of p.Ap.  Straight-line over the R
  // rows, so that the loads of one row overlap the sums of another: rows past
  // the block's own read what lies there in shared memory (R NT - rpc values
  // past an array's end at most, inside the block: cl_smem_bytes) and are
  // then set to zero, and rows that hold only their diagonal are selected.
  __device__ __forceinline__ double multiply() {
    ClAcc acc;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int li = (int)threadIdx.x + j * NT;
      const int i = li + halo;
      T y = T(0);
#pragma unroll
      for (int k = H - 1; k >= 0; --k) {
        const int q = i - off[k];
        y = fma(vv[(k + 1) * VW + q], pw[q], y);
      }
      const T v0 = vv[i], p0 = pw[i];
      y = fma(v0, p0, y);
#pragma unroll
      for (int k = 0; k < H; ++k) y = fma(vv[(k + 1) * VW + i], pw[i + off[k]], y);
      y = ((diag_only >> j) & 1u) ? v0 * p0 : y;
      const bool in = li < rows;
      ap[j] = in ? y : T(0);
      acc.add(in ? y * p0 : T(0));
    }
    return acc.s;
  }

  // Row li's z into the zh of every other block whose window covers the row.
  // Windows that reach only the neighbouring blocks (halo <= rpc) take two
  // predicated stores, so the callers' loops stay free of branches.
  __device__ __forceinline__ void push(int li, T z) {
    if (halo <= rpc) {
      cl_store_if(li < halo && li < rows && rank > 0, zh_prev + (unsigned)sizeof(T) * (unsigned)(halo + li), z);
      cl_store_if(li >= rpc - halo && li < rows && rank + 1 < blocks,
                  zh_next + (unsigned)sizeof(T) * (unsigned)(li - rpc + halo), z);
      return;
    }
    if (li >= rows) return;
    for (int dd = 1, first = 0; first < halo; ++dd, first += rpc) {
      if ((int)rank - dd >= 0 && li + first < halo)
        cl_store_if(true, cl_remote(zh + halo + li + first, rank - dd), z);
      if (rank + dd < blocks && li >= dd * rpc - halo)
        cl_store_if(true, cl_remote(zh + (li - dd * rpc + halo), rank + dd), z);
    }
  }

  // p = z + beta p over the window (own rows from r, halo rows from zh), or
  // p = z; `before(j, p_old)` sees each own row's p first.
  template <typename F> __device__ __forceinline__ void direction(T beta, bool keep, F &&before) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int li = (int)threadIdx.x + j * NT;
      const T z = PRE ? r[j] * d[j] : r[j];
      const T p = pw[li + halo];
      before(j, p);
      const T q = keep ? fma(beta, p, z) : z;
      if (li < rows) pw[li + halo] = q;
    }
    // halo rows outside [0, n) hold zeros in zh and stay zero
    for (int q = threadIdx.x; q < 2 * halo; q += NT) {
      const int w = q < halo ? q : rpc + q;
      const int row = r0 - halo + w;
      if (row < 0 || row >= n) continue;
      pw[w] = keep ? fma(beta, pw[w], zh[q]) : zh[q];
    }
    __syncthreads();
  }

  // Sums over the cluster, the same bits in every thread: each warp's partial
  // goes to every block's slots, one cluster barrier, then every warp adds
  // the slots in one order.  `set` alternates between consecutive sums.
  template <int NV> __device__ __forceinline__ void sum(double (&v)[NV], int set) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *s = slots + set * (kClSums * kClMaxBlocks * kClWarps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      v[k] = warp_sum(v[k]);
      double *at = s + k * (kClMaxBlocks * kClWarps) + (int)rank * kClWarps + warp;
      if (blocks == 1) {
        if (lane == 0) *at = v[k];
      } else if (lane < (int)blocks) {
        cl_store(cl_remote(at, lane), v[k]);
      }
    }
    cl_barrier(blocks);
    const int cnt = (int)blocks * kClWarps;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double a = 0.0;
      for (int q = lane; q < cnt; q += 32) a += s[k * (kClMaxBlocks * kClWarps) + q];
      v[k] = warp_sum(a);
    }
  }

  // One step's update after alpha: r -= alpha Ap, z pushed to the windows
  // that cover it; v = this thread's shares of r.r and r.z.
  __device__ __forceinline__ void update(T alpha, double (&v)[2]) {
    ClAcc rr, rz;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const T q = fma(-alpha, ap[j], r[j]);
      r[j] = q;
      const T z = PRE ? q * d[j] : q;
      rr.add(q * q);
      if (PRE) rz.add(q * z);
    }
    // the few rows other blocks' windows cover, out of the loop above
    if (blocks > 1) {
#pragma unroll
      for (int j = 0; j < R; ++j)
        if (j * NT < halo || (j + 1) * NT > rpc - halo) push((int)threadIdx.x + j * NT, PRE ? r[j] * d[j] : r[j]);
    }
    v[0] = rr.s;
    v[1] = rz.s;
  }
};

}  // namespace b200la
