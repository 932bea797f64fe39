// SpMV schedules (CSR lane groups, SELL-32 slices) shared by the plain
// VectorMult entry points, the autotuner and the fused CG kernels.
//
// A schedule is an "operator" type with run(x, emit): every thread block
// walks its share of the rows (grid-stride) and, on exactly one lane per row,
// calls emit.fetch(row) before the row's products and emit(row, y_row) after
// them (run_with: any block size and vector loader).  An emitter loads what
// it needs of other vectors in fetch, so that these loads overlap the row's
// own; loaded after the sum they cost each warp another round trip per row
// (FP64 128^3: the CG's product and dot 94 us where the product alone takes 78).  The fused kernels pass emitters that also
// accumulate dot products, so the SpMV result never makes an extra trip
// through HBM.
#pragma once

#include "internal.cuh"

namespace b200la {

// How a schedule reads the gathered vector: ld(column).  The plain form keeps
// it in the read-only path; a kernel that writes the vector while it runs
// brings its own.
// at(row) gives the loader of offsets from a row, so that a row's address is
// formed once and its entries' offsets are added to it.
template <typename X> struct KeepLoad {
  const X *__restrict__ x;
  __device__ __forceinline__ X operator()(int c) const { return ld_keep(x + c); }
  __device__ __forceinline__ KeepLoad at(int row) const { return KeepLoad{x + row}; }
  // x[c], x[c + 1] of a loader at an even row, c even
  __device__ __forceinline__ void pair(int c, X &a, X &b) const { ld_nc2(x + c, a, b); }
};

// ---- CSR, G lanes per row (G = 1..32) -------------------------------------
// Each warp covers 32/G consecutive rows, so a warp's loads of val/col fall
// in one contiguous span of the CSR arrays; x is gathered through L1/L2.
//
// Every schedule takes the stored value type T and the vector type X (x, y
// and the row sums; X = T except in the mixed-storage inner solve, where
// FP32 values meet FP64 vectors and each value is widened before its FMA).
template <typename T, int G, typename X = T> struct CsrOp {
  using XT = X;
  const int *__restrict__ rowptr;
  const int *__restrict__ col;
  const T *__restrict__ val;
  int n;
  static constexpr int kRowsPerBlock = kBlock / G;
  static constexpr int kLanes = G;  // threads per row
  __host__ __device__ int64_t work_items() const { return n; }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    constexpr int rpb = NT / G;
    for (int base = blockIdx.x * rpb; base < n; base += gridDim.x * rpb) {
      const int row = base + (int)threadIdx.x / G;
      const bool valid = row < n;
      if (valid && (threadIdx.x & (G - 1)) == 0) emit.fetch(row);
      X y = csr_row_group<T, G, X>(rowptr, col, val, x, row, valid);
      if (valid && (threadIdx.x & (G - 1)) == 0) emit(row, y);
    }
  }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  // the rows that run_with<NT> hands to this thread's emitter, in its order
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    constexpr int rpb = NT / G;
    if (threadIdx.x & (G - 1)) return;
    for (int base = blockIdx.x * rpb; base < n; base += gridDim.x * rpb)
      if (base + (int)threadIdx.x / G < n) f(base + (int)threadIdx.x / G);
  }
  // the most rows a block of NT threads owns in a grid of `blocks`
  template <int NT> int rows_per_block(int blocks) const {
    constexpr int rpb = NT / G;
    const int64_t tiles = ((int64_t)n + rpb - 1) / rpb;
    return (int)((tiles + blocks - 1) / blocks) * rpb;
  }
};

// ---- SELL-C-sigma ----------------------------------------------------------
// Rows are sorted by length, longest first, within windows of sigma rows
// (perm[position] = row; sigma = 1 keeps the order and perm is null), then
// cut into slices of C rows (C = 8, 16 or 32), each padded to its longest
// row rounded up to W entries.  Entry k of the row at position r of slice s
// sits at slice_ptr[s] + ((k/W)*C + r)*W + k%W: a row's W consecutive
// entries are one vector load, and the C rows of a slice read C*W contiguous
// values per step.  A warp handles 32/C slices at a time (lane = slice in
// the warp * C + r).  Padding entries hold value 0 and repeat a column the
// row already reads.  Every row's products are added in its stored order
// whatever C, sigma and W are, so all SELL variants give the same bits.
template <typename T, int W> struct VecW;
template <> struct VecW<double, 1> { using v = double; using i = int; };
template <> struct VecW<double, 2> { using v = double2; using i = int2; };
template <> struct VecW<double, 4> { using v = double4; using i = int4; };
template <> struct VecW<float, 1> { using v = float; using i = int; };
template <> struct VecW<float, 2> { using v = float2; using i = int2; };
template <> struct VecW<float, 4> { using v = float4; using i = int4; };

template <typename V, typename T, int W> __device__ __forceinline__ T lane_get(const V &v, int k) {
  return reinterpret_cast<const T *>(&v)[k];
}
template <typename I, int W> __device__ __forceinline__ int lane_geti(const I &v, int k) {
  return reinterpret_cast<const int *>(&v)[k];
}

template <typename T> __device__ __forceinline__ double4 ld_stream4(const double4 *p) {
  const double2 *q = reinterpret_cast<const double2 *>(p);
  double2 a = __ldcs(q), b = __ldcs(q + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

template <typename V> __device__ __forceinline__ V ld_vec_stream(const V *p) { return __ldcs(p); }
template <> __device__ __forceinline__ double4 ld_vec_stream<double4>(const double4 *p) {
  return ld_stream4<double>(p);
}

template <typename T, int W, typename X = T> struct SellOp {
  using XT = X;
  const int *__restrict__ slice_ptr;
  const int *__restrict__ slice_len;
  const int *__restrict__ col;
  const T *__restrict__ val;
  int n, nslices;
  int log2c;                 // C = 1 << log2c rows per slice
  const int *__restrict__ perm;  // row of each position, or null (identity)
  static constexpr int kRowsPerBlock = kBlock;
  static constexpr int kLanes = 1;
  __host__ __device__ int64_t work_items() const { return n; }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    const int lane = threadIdx.x & 31;
    const int C = 1 << log2c, spw = 32 >> log2c;
    const int r = lane & (C - 1), sub = lane >> log2c;
    for (int s0 = (blockIdx.x * (NT / 32) + ((int)threadIdx.x >> 5)) * spw; s0 < nslices;
         s0 += gridDim.x * (NT / 32) * spw) {
      const int s = s0 + sub, pos = s * C + r;
      if (s < nslices && pos < n) f(perm ? __ldg(perm + pos) : pos);
    }
  }
  template <int NT> int rows_per_block(int blocks) const {
    const int64_t tiles = ((int64_t)nslices * (1 << log2c) + NT - 1) / NT;
    return (int)((tiles + blocks - 1) / blocks) * NT;
  }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    using VV = typename VecW<T, W>::v;
    using VI = typename VecW<T, W>::i;
    const int lane = threadIdx.x & 31;
    constexpr int wpb = NT / 32;
    const int C = 1 << log2c, spw = 32 >> log2c;
    const int r = lane & (C - 1), sub = lane >> log2c;
    for (int s0 = (blockIdx.x * wpb + ((int)threadIdx.x >> 5)) * spw; s0 < nslices; s0 += gridDim.x * wpb * spw) {
      const int s = s0 + sub;
      const bool live = s < nslices;
      const int base = live ? __ldg(slice_ptr + s) : 0;
      const int chunks = live ? __ldg(slice_len + s) / W : 0;
      const VI *ci = reinterpret_cast<const VI *>(col + base) + r;
      const VV *vi = reinterpret_cast<const VV *>(val + base) + r;
      const int pos = s * C + r;
      const bool real = live && pos < n;
      const int row = real ? (perm ? __ldg(perm + pos) : pos) : 0;
      if (real) emit.fetch(row);
      X sum = X(0);
#pragma unroll 4
      for (int c = 0; c < chunks; ++c) {
        VI cc = ld_vec_stream(ci + c * C);
        VV vv = ld_vec_stream(vi + c * C);
#pragma unroll
        for (int k = 0; k < W; ++k)
          sum = fma((X)lane_get<VV, T, W>(vv, k), x(lane_geti<VI, W>(cc, k)), sum);
      }
      if (real) emit(row, sum);
    }
  }
};

// ---- SELL-32 with int16 column offsets -------------------------------------
// Same slices and value layout as SellOp; the stored column of entry k is
// (column - row) as int16, so a warp reads 2*W bytes of indices per lane and
// step instead of 4*W.  Products and their order are those of SellOp.
template <int W> struct VecS;
template <> struct VecS<1> { using i = short; };
template <> struct VecS<2> { using i = short2; };
template <> struct VecS<4> { using i = short4; };

template <typename I> __device__ __forceinline__ int lane_gets(const I &v, int k) {
  return (int)reinterpret_cast<const short *>(&v)[k];
}

template <typename T, int W, typename X = T> struct SellOp16 {
  using XT = X;
  const int *__restrict__ slice_ptr;
  const int *__restrict__ slice_len;
  const short *__restrict__ col;
  const T *__restrict__ val;
  int n, nslices;
  int log2c;                 // C = 1 << log2c rows per slice
  const int *__restrict__ perm;  // row of each position, or null (identity)
  static constexpr int kRowsPerBlock = kBlock;
  static constexpr int kLanes = 1;
  __host__ __device__ int64_t work_items() const { return n; }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    const int lane = threadIdx.x & 31;
    const int C = 1 << log2c, spw = 32 >> log2c;
    const int r = lane & (C - 1), sub = lane >> log2c;
    for (int s0 = (blockIdx.x * (NT / 32) + ((int)threadIdx.x >> 5)) * spw; s0 < nslices;
         s0 += gridDim.x * (NT / 32) * spw) {
      const int s = s0 + sub, pos = s * C + r;
      if (s < nslices && pos < n) f(perm ? __ldg(perm + pos) : pos);
    }
  }
  template <int NT> int rows_per_block(int blocks) const {
    const int64_t tiles = ((int64_t)nslices * (1 << log2c) + NT - 1) / NT;
    return (int)((tiles + blocks - 1) / blocks) * NT;
  }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    using VV = typename VecW<T, W>::v;
    using VI = typename VecS<W>::i;
    const int lane = threadIdx.x & 31;
    constexpr int wpb = NT / 32;
    const int C = 1 << log2c, spw = 32 >> log2c;
    const int r = lane & (C - 1), sub = lane >> log2c;
    for (int s0 = (blockIdx.x * wpb + ((int)threadIdx.x >> 5)) * spw; s0 < nslices; s0 += gridDim.x * wpb * spw) {
      const int s = s0 + sub;
      const bool live = s < nslices;
      const int base = live ? __ldg(slice_ptr + s) : 0;
      const int chunks = live ? __ldg(slice_len + s) / W : 0;
      const VI *ci = reinterpret_cast<const VI *>(col + base) + r;
      const VV *vi = reinterpret_cast<const VV *>(val + base) + r;
      const int pos = s * C + r;
      const bool real = live && pos < n;
      // the stored offsets are relative to the row itself; padding rows
      // past n (last slice) hold offset 0 and gather x[0]
      const int row = real ? (perm ? __ldg(perm + pos) : pos) : 0;
      const Ld xr = x.at(row);
      if (real) emit.fetch(row);
      X sum = X(0);
#pragma unroll 4
      for (int c = 0; c < chunks; ++c) {
        VI cc = __ldcs(ci + c * C);
        VV vv = ld_vec_stream(vi + c * C);
#pragma unroll
        for (int k = 0; k < W; ++k)
          sum = fma((X)lane_get<VV, T, W>(vv, k), xr(lane_gets(cc, k)), sum);
      }
      if (real) emit(row, sum);
    }
  }
};

// ---- values-only sliced ELL (a stencil of column offsets) -----------------
// Square matrices whose every row's columns are a subset of one ascending
// list of offsets (structured-grid FE matrices): 32-row slices, every row
// EP entries (the stencil, padded to a multiple of W with offset 0), entry k
// of the row at position r of slice s at s*EP*32 + ((k/W)*32 + r)*W + k%W,
// value 0 where the row has no entry.  The column of entry k is
// row + off[k] (a compile-time index into the operator's offsets, which sit
// in the kernel's parameter space); slices whose columns all fall inside
// [0, n) skip the clamp the border slices need.  No column bytes at all:
// an FP64 3D Q1 row moves 8 bytes per entry instead of 10 (SELL16) or 12.
// Products in ascending column order, the rows' stored order, so the bits
// are SELL's (absent entries add 0 * x).
template <typename T, int W, int EP, typename X = T> struct StencilOp {
  using XT = X;
  const T *__restrict__ val;
  int n, nslices;
  int lo, hi;  // smallest and largest offset
  int off[EP];
  static constexpr int kRowsPerBlock = kBlock;
  static constexpr int kLanes = 1;
  __host__ __device__ int64_t work_items() const { return n; }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    for (int s = blockIdx.x * (NT / 32) + ((int)threadIdx.x >> 5); s < nslices; s += gridDim.x * (NT / 32)) {
      const int row = s * 32 + (int)(threadIdx.x & 31);
      if (row < n) f(row);
    }
  }
  template <int NT> int rows_per_block(int blocks) const {
    const int64_t tiles = ((int64_t)nslices * 32 + NT - 1) / NT;
    return (int)((tiles + blocks - 1) / blocks) * NT;
  }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    using VV = typename VecW<T, W>::v;
    const int lane = threadIdx.x & 31;
    constexpr int wpb = NT / 32;
    for (int s = blockIdx.x * wpb + ((int)threadIdx.x >> 5); s < nslices; s += gridDim.x * wpb) {
      const int row = s * 32 + lane;
      const VV *vi = reinterpret_cast<const VV *>(val + (int64_t)s * EP * 32) + lane;
      if (row < n) emit.fetch(row);
      X sum = X(0);
      if (s * 32 + lo >= 0 && s * 32 + 31 + hi < n) {
        const Ld xr = x.at(row);
#pragma unroll
        for (int c = 0; c < EP / W; ++c) {
          const VV vv = ld_vec_stream(vi + c * 32);
#pragma unroll
          for (int k = 0; k < W; ++k) sum = fma((X)lane_get<VV, T, W>(vv, k), xr(off[c * W + k]), sum);
        }
      } else {
#pragma unroll
        for (int c = 0; c < EP / W; ++c) {
          const VV vv = ld_vec_stream(vi + c * 32);
#pragma unroll
          for (int k = 0; k < W; ++k)
            sum = fma((X)lane_get<VV, T, W>(vv, k), x(min(max(row + off[c * W + k], 0), n - 1)), sum);
        }
      }
      if (row < n) emit(row, sum);
    }
  }
};

template <typename Op> Op stencil_op(const void *val, int n, const SellData &s) {
  Op op;
  op.val = (decltype(op.val))val;
  op.n = n;
  op.nslices = s.nslices;
  op.lo = s.off_lo;
  op.hi = s.off_hi;
  for (int k = 0; k < (int)(sizeof(op.off) / sizeof(int)); ++k) op.off[k] = s.soff[k];
  return op;
}

// ---- values-only copy, symmetric half --------------------------------------
// The stencil copy of a matrix whose values are symmetric up to rows that
// hold only their diagonal (sym_row_ok in cluster_cg.cuh): the diagonal and
// the H upper diagonals, v_k(i) = a(i, i + off[k]) at (k * ld + pad + i); the
// lower entry a(i, i - off[k]) is v_k(i - off[k]), read from L2 where its row's
// own load left it.  DRAM moves 14 values a 27-point row instead of 27
// (FP64 128^3: product 74 -> 51 us; FP32 46 -> 40, where the requests in
// flight bind before the bytes do).  `only` holds a bit per row that stores
// only its diagonal; such a row's other values are taken as the zeros it
// stores.  Products in ascending column order: SELL's bits.
// A row's loads are issued kBatch entries at a time before their sums.
template <typename T, int E, typename X = T> struct SymStencilOp {
  using XT = X;
  static constexpr int H = E / 2, kBatch = 9;
  const T *__restrict__ val;           // v_0(0), after the front padding of the first diagonal
  const unsigned *__restrict__ only;   // [nslices]
  int n, nslices, ld;
  int hi;        // largest offset
  int off[E];    // all offsets, ascending
  static constexpr int kRowsPerBlock = kBlock;
  static constexpr int kLanes = 1;
  __host__ __device__ int64_t work_items() const { return n; }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    for (int s = blockIdx.x * (NT / 32) + ((int)threadIdx.x >> 5); s < nslices; s += gridDim.x * (NT / 32)) {
      const int row = s * 32 + (int)(threadIdx.x & 31);
      if (row < n) f(row);
    }
  }
  template <int NT> int rows_per_block(int blocks) const {
    const int64_t tiles = ((int64_t)nslices * 32 + NT - 1) / NT;
    return (int)((tiles + blocks - 1) / blocks) * NT;
  }
  // y of one row; IN: every column of the slice lies in [0, n); ONLY: the
  // slice has rows that hold only their diagonal (`diag` if this one does)
  template <bool IN, bool ONLY, typename Ld>
  __device__ __forceinline__ X row_sum(const Ld &x, int row, bool diag) const {
    const Ld xr = x.at(IN ? row : 0);
    X sum = X(0);
#pragma unroll
    for (int c = 0; c < E; c += kBatch) {
      T v[kBatch];
      X g[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (c + k < E) {
          const int e = c + k, q = e < H ? H - e : e - H;
          v[k] = ld_nc(val + (int64_t)q * ld + (e < H ? row + off[e] : row));
        }
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (c + k < E) g[k] = IN ? xr(off[c + k]) : xr(min(max(row + off[c + k], 0), n - 1));
#pragma unroll
      for (int k = 0; k < kBatch; ++k)
        if (c + k < E) sum = fma(ONLY && diag && c + k != H ? X(0) : (X)v[k], g[k], sum);
    }
    return sum;
  }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    const int lane = threadIdx.x & 31;
    constexpr int wpb = NT / 32;
    for (int s = blockIdx.x * wpb + ((int)threadIdx.x >> 5); s < nslices; s += gridDim.x * wpb) {
      const int row = s * 32 + lane;
      const unsigned word = __ldg(only + s);
      if (row < n) emit.fetch(row);
      const bool diag = (word >> lane) & 1u;
      X sum;
      if (s * 32 - hi >= 0 && s * 32 + 31 + hi < n) {
        sum = word == 0 ? row_sum<true, false>(x, row, false) : row_sum<true, true>(x, row, diag);
      } else {
        sum = row_sum<false, true>(x, row, diag);
      }
      if (row < n) emit(row, sum);
    }
  }
};

// The same copy, two consecutive rows a lane (64 rows a warp), for offsets
// in triples (o - 1, o, o + 1) whose middle ones follow one of two parity
// patterns (grids with m nodes an axis: multiples of m and m^2, all even when
// m is, else odd for odd multiples).  What bounds the one-row form in FP32 is
// not bytes but requests in flight: 54 four-byte loads a row, 128 bytes each,
// ~250 of them outstanding per SM (27% of the L1's request rate at 5 TB/s).
// Pairs halve the requests: own values are 8-byte (FP64: 16-byte) loads, two
// rows share four gathered values of a triple instead of loading six, and a
// lower value's pair is one load where its offset is even.  Products in
// ascending column order, so the bits do not change.
template <typename T, int E, bool ODD, typename X = T> struct SymPairOp {
  using XT = X;
  SymStencilOp<T, E, X> one;
  static constexpr int H = E / 2;
  static constexpr int kRowsPerBlock = 2 * kBlock;
  static constexpr int kLanes = 1;
  __host__ __device__ int64_t work_items() const { return one.n; }
  // whether the middle offset of triple t is odd
  __host__ __device__ static constexpr bool odd_triple(int t) {
    return ODD && (E == 9 ? t != 1 : (((t / 3 != 1) + (t % 3 != 1)) & 1) != 0);
  }
  template <typename Emit> __device__ __forceinline__ void run(const X *__restrict__ x, Emit &emit) const {
    run_with<kBlock>(KeepLoad<X>{x}, emit);
  }
  template <int NT, typename F> __device__ __forceinline__ void each_row(F &&f) const {
    for (int s = blockIdx.x * (NT / 32) + ((int)threadIdx.x >> 5); s * 2 < one.nslices; s += gridDim.x * (NT / 32)) {
      const int row = s * 64 + 2 * (int)(threadIdx.x & 31);
      if (row < one.n) f(row);
      if (row + 1 < one.n) f(row + 1);
    }
  }
  template <int NT> int rows_per_block(int blocks) const {
    const int64_t tiles = ((int64_t)one.nslices * 32 + 2 * NT - 1) / (2 * NT);
    return (int)((tiles + blocks - 1) / blocks) * 2 * NT;
  }
  template <bool ONLY, typename Ld>
  __device__ __forceinline__ void pair_sum(const Ld &x, int row, bool d0, bool d1, X &y0, X &y1) const {
    const Ld xr = x.at(row);
    X s0 = X(0), s1 = X(0);
#pragma unroll
    for (int p = 0; p < E; p += 9) {
      T v0[9], v1[9];
      X g[3][4];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const int e = p + k;
        if (e >= H) {
          ld_nc2(one.val + (int64_t)(e - H) * one.ld + row, v0[k], v1[k]);
        } else {
          const T *q = one.val + (int64_t)(H - e) * one.ld + (row + one.off[e]);
          if (odd_triple(e / 3) == (e % 3 == 1)) {  // odd offset
            v0[k] = ld_nc(q);
            v1[k] = ld_nc(q + 1);
          } else {
            ld_nc2(q, v0[k], v1[k]);
          }
        }
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const int o = one.off[p + 3 * t + 1];
        if (odd_triple(p / 3 + t)) {
          xr.pair(o - 1, g[t][0], g[t][1]);
          xr.pair(o + 1, g[t][2], g[t][3]);
        } else {
          g[t][0] = xr(o - 1);
          xr.pair(o, g[t][1], g[t][2]);
          g[t][3] = xr(o + 2);
        }
      }
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        s0 = fma(ONLY && d0 && p + k != H ? X(0) : (X)v0[k], g[k / 3][k % 3], s0);
        s1 = fma(ONLY && d1 && p + k != H ? X(0) : (X)v1[k], g[k / 3][k % 3 + 1], s1);
      }
    }
    y0 = s0;
    y1 = s1;
  }
  template <int NT, typename Ld, typename Emit>
  __device__ __forceinline__ void run_with(const Ld &x, Emit &emit) const {
    const int lane = threadIdx.x & 31;
    constexpr int wpb = NT / 32;
    const int n = one.n;
    for (int s = blockIdx.x * wpb + ((int)threadIdx.x >> 5); s * 2 < one.nslices; s += gridDim.x * wpb) {
      const int row = s * 64 + 2 * lane;
      const unsigned w0 = __ldg(one.only + 2 * s), w1 = 2 * s + 1 < one.nslices ? __ldg(one.only + 2 * s + 1) : 0u;
      // the second row's vectors lie in the lines the first row's fetch brings
      if (row < n) emit.fetch(row);
      const unsigned bits = (lane < 16 ? w0 >> (2 * lane) : w1 >> (2 * lane - 32)) & 3u;
      const bool d0 = bits & 1u, d1 = bits & 2u;
      X y0, y1;
      if (s * 64 - one.hi >= 0 && s * 64 + 63 + one.hi < n) {
        if ((w0 | w1) == 0) pair_sum<false>(x, row, false, false, y0, y1);
        else pair_sum<true>(x, row, d0, d1, y0, y1);
      } else {
        // rows past the last slice take the last row's place
        const int last = one.nslices * 32 - 1;
        y0 = one.template row_sum<false, true>(x, min(row, last), d0);
        y1 = one.template row_sum<false, true>(x, min(row + 1, last), d1);
      }
      if (row < n) emit(row, y0);
      if (row + 1 < n) {
        emit.fetch(row + 1);
        emit(row + 1, y1);
      }
    }
  }
};

template <typename Op> Op sym_stencil_op(const void *val, int n, const SellData &s) {
  Op op;
  op.val = (decltype(op.val))val + s.sym_pad;
  op.only = s.sym_only;
  op.n = n;
  op.nslices = s.nslices;
  op.ld = s.sym_ld;
  op.hi = s.off_hi;
  for (int k = 0; k < (int)(sizeof(op.off) / sizeof(int)); ++k) op.off[k] = s.soff[k];
  return op;
}

// ---- plain emitters --------------------------------------------------------
template <typename T> struct StoreEmit {
  T *__restrict__ y;
  __device__ __forceinline__ void fetch(int) {}
  __device__ __forceinline__ void operator()(int row, T v) { y[row] = v; }
};
template <typename T> struct AddEmit {
  T *__restrict__ y;
  T y0;
  __device__ __forceinline__ void fetch(int row) { y0 = y[row]; }
  __device__ __forceinline__ void operator()(int row, T v) { y[row] = y0 + v; }
};

template <typename Op, typename T, bool ADD>
__global__ void __launch_bounds__(kBlock) spmv_kernel(Op op, const T *__restrict__ x, T *__restrict__ y) {
  if (ADD) {
    AddEmit<T> e{y};
    op.run(x, e);
  } else {
    StoreEmit<T> e{y};
    op.run(x, e);
  }
}

// Calls f(op) with the schedule selected on the matrix (stored values T,
// vectors X).
template <typename T, typename X = T, typename F> int with_schedule(b200la_mat m, F &&f) {
  const T *val = (const T *)m->val;
  if (m->format == B200LA_FMT_SELL) {
    const SellData &s = m->sell;
    const T *sv = (const T *)s.val;
    switch (m->param) {
      case 1: return f(SellOp<T, 1, X>{s.slice_ptr, s.slice_len, s.col, sv, m->nrow, s.nslices, s.log2c, s.perm});
      case 2: return f(SellOp<T, 2, X>{s.slice_ptr, s.slice_len, s.col, sv, m->nrow, s.nslices, s.log2c, s.perm});
      case 4: return f(SellOp<T, 4, X>{s.slice_ptr, s.slice_len, s.col, sv, m->nrow, s.nslices, s.log2c, s.perm});
    }
    return fail(B200LA_ERR_INVALID, "SELL width %d", m->param);
  }
  if (m->format == B200LA_FMT_SELL16) {
    const SellData &s = m->sell;
    const T *sv = (const T *)s.val;
    switch (m->param) {
      case 1:
        return f(SellOp16<T, 1, X>{s.slice_ptr, s.slice_len, s.col16p, sv, m->nrow, s.nslices, s.log2c, s.perm});
      case 2:
        return f(SellOp16<T, 2, X>{s.slice_ptr, s.slice_len, s.col16p, sv, m->nrow, s.nslices, s.log2c, s.perm});
      case 4:
        return f(SellOp16<T, 4, X>{s.slice_ptr, s.slice_len, s.col16p, sv, m->nrow, s.nslices, s.log2c, s.perm});
    }
    return fail(B200LA_ERR_INVALID, "SELL16 width %d", m->param);
  }
  if (m->format == B200LA_FMT_STENCIL) {
    const SellData &s = m->sell;
    // FP64 requests are wide enough as they are (128^3 CG product 69 us with
    // one row a lane, 73 with two; FP32 Jacobi sweep 96^3 31 and 25)
    if constexpr (sizeof(T) == 4) {
      if (s.sym_pair && s.ell == 9) {
        const auto one = sym_stencil_op<SymStencilOp<T, 9, X>>(s.val, m->nrow, s);
        return s.sym_pair == 2 ? f(SymPairOp<T, 9, true, X>{one}) : f(SymPairOp<T, 9, false, X>{one});
      }
      if (s.sym_pair) {
        const auto one = sym_stencil_op<SymStencilOp<T, 27, X>>(s.val, m->nrow, s);
        return s.sym_pair == 2 ? f(SymPairOp<T, 27, true, X>{one}) : f(SymPairOp<T, 27, false, X>{one});
      }
    }
    if (s.sym) {
      if (s.ell == 9) return f(sym_stencil_op<SymStencilOp<T, 9, X>>(s.val, m->nrow, s));
      return f(sym_stencil_op<SymStencilOp<T, 27, X>>(s.val, m->nrow, s));
    }
    const int key = m->param * 100 + s.ell;
    switch (key) {
      case 109: return f(stencil_op<StencilOp<T, 1, 9, X>>(s.val, m->nrow, s));
      case 210: return f(stencil_op<StencilOp<T, 2, 10, X>>(s.val, m->nrow, s));
      case 412: return f(stencil_op<StencilOp<T, 4, 12, X>>(s.val, m->nrow, s));
      case 127: return f(stencil_op<StencilOp<T, 1, 27, X>>(s.val, m->nrow, s));
      case 228: return f(stencil_op<StencilOp<T, 2, 28, X>>(s.val, m->nrow, s));
      case 428: return f(stencil_op<StencilOp<T, 4, 28, X>>(s.val, m->nrow, s));
    }
    return fail(B200LA_ERR_INVALID, "STENCIL width %d with %d entries per row", m->param, s.ell);
  }
  switch (m->param) {
    case 1: return f(CsrOp<T, 1, X>{m->rowptr, m->col, val, m->nrow});
    case 2: return f(CsrOp<T, 2, X>{m->rowptr, m->col, val, m->nrow});
    case 4: return f(CsrOp<T, 4, X>{m->rowptr, m->col, val, m->nrow});
    case 8: return f(CsrOp<T, 8, X>{m->rowptr, m->col, val, m->nrow});
    case 16: return f(CsrOp<T, 16, X>{m->rowptr, m->col, val, m->nrow});
    case 32: return f(CsrOp<T, 32, X>{m->rowptr, m->col, val, m->nrow});
  }
  return fail(B200LA_ERR_INVALID, "CSR lanes per row %d", m->param);
}

int spmv_launch(b200la_mat m, const void *x, void *y, bool add, cudaStream_t s);
// y = (A - diag(A)) x from the CSR as uploaded (VectorMultNoDiag)
int spmv_nodiag_launch(b200la_mat m, const void *x, void *y, cudaStream_t s);
// Builds the sliced copy: `width` entries per vector load, int16 column
// offsets (col16), C rows per slice, rows sorted by length within windows of
// sigma rows (1 = no sorting; otherwise rounded up to a multiple of C).
int sell_build(b200la_mat m, int width, bool col16 = false, int C = 32, int sigma = 1);
// Builds the values-only copy (B200LA_FMT_STENCIL) with `width` entries per
// vector load; B200LA_ERR_UNSUPPORTED when the matrix has no stencil.
int stencil_build(b200la_mat m, int width);
// Looks once for the structure the cluster-resident solver needs (m->cl_*):
// rows that are subsets of one symmetric offset set, values symmetric up to
// rows that hold only their diagonal.  Waits for the stream.
int cl_detect(b200la_mat m);
inline bool is_sell(int format) { return format == B200LA_FMT_SELL || format == B200LA_FMT_SELL16; }
// any schedule with a sliced copy (rebuilt when the values change)
inline bool is_sliced(int format) { return is_sell(format) || format == B200LA_FMT_STENCIL; }
// frees the sliced copy and builds the one `format` / `param` name (C and
// sigma for SELL-C-sigma) from the CSR: after the values changed
int sliced_rebuild(b200la_mat m, int format, int param, int C, int sigma);
void sell_free(b200la_mat m);

}  // namespace b200la
