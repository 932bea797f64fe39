// Preconditioned CG on the device: CG<LAD>::SolvePrecond / SolveNoPrecond
// (linear_solver/cg.h:87-246) with PreconditionerBlockJacobiStand(Jacobi)
// (preconditioner_bjacobi_standard.cc:188-196, lmp/lpreconditioner.cc:184-200)
// and IterateControl::Check (common/iterate_control.cc:80-107).
//
// The reference runs the loop on the host: per iteration 1 SpMV, 3 blocking
// dot products and 6 more BLAS-1 passes, each its own launch.  Here one
// iteration is three kernels and no host round trip:
//   K1  Ap = A p, fused with the partial sums of p.Ap     (SpMV schedule)
//   K2  alpha = rz/pAp; x += alpha p; r -= alpha Ap; z = invD r;
//       fused sums r.r and r.z; its last block applies IterateControl
//   K3  beta = rz_new/rz_old; p = beta p + z  (z recomputed from r, invD)
// Where the system fits, the same loop runs in one launch instead, on one
// cluster (cg_cluster_kernel) or on resident blocks (cg_resident_kernel): an
// iteration of small systems is launches and reductions, not bytes.
// All scalars live in device memory.  The three kernels form the body of a
// CUDA-graph WHILE node, so one graph launch runs the whole solve; K3 clears
// the loop condition once the state leaves "iterate".  K3 also counts body
// passes and stops the loop after maxits + 2 passes whatever K2 reported, so
// the device loop ends even if a reduction misbehaves.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "cg_internal.cuh"
#include "cluster_cg.cuh"
#include "persist.cuh"
#include "spmv.cuh"

namespace b200la {

// IterateControl::Check; step 0 records the initial residual (res_init).
// Under the lmp cg() rule: no test before the first iteration, success once
// ||r|| <= max(rtol ||r0||, atol), no divergence test.
__device__ __forceinline__ int iterate_check(int step, double value, const CgScalars &s, double first) {
  if (s.stop_rule == B200LA_STOP_LMP_CG) {
    if (step > 0 && value <= fmax(s.rtol * first, s.atol)) return B200LA_SUCCESS_REL;
    if (step >= s.maxits) return B200LA_FAIL_MAXITS;
    return B200LA_ITERATE;
  }
  if (value <= s.atol) return B200LA_SUCCESS_ABS;
  if (value < s.rtol * first) return B200LA_SUCCESS_REL;
  if (value > s.dtol * first) return B200LA_FAIL_DIV;
  if (step >= s.maxits) return B200LA_FAIL_MAXITS;
  return B200LA_ITERATE;
}

template <typename T> struct CgVecs {
  T *x, *r, *p, *Ap;
  const T *invd;  // nullptr without preconditioner
  int64_t n;
};

// ---- init: r = b - A x0, z = invD r, p = z, rz = r.z, res_init -----------------
template <typename T, bool PRE> struct InitEmit {
  const T *__restrict__ b;
  const T *__restrict__ x_user;
  CgVecs<T> v;
  Acc<T> rr, rz;
  T br, xr, dr;
  __device__ __forceinline__ void fetch(int row) {
    br = b[row];
    xr = x_user[row];
    if (PRE) dr = v.invd[row];
  }
  __device__ __forceinline__ void operator()(int row, T y) {
    T r = br - y;  // r.ScaleAdd(b, -1): -1*(Ax) + b
    v.x[row] = xr;
    v.r[row] = r;
    T z = PRE ? r * dr : r;
    v.p[row] = z;
    rr.add(r * r);
    rz.add(r * z);
  }
};

template <typename Op, typename T, bool PRE>
__global__ void __launch_bounds__(kBlock) cg_init_kernel(Op op, const T *__restrict__ x_user, const T *__restrict__ b,
                                                         CgVecs<T> v, double *part, CgScalars *sc) {
  InitEmit<T, PRE> e{b, x_user, v};
  op.run(x_user, e);
  double s[2] = {e.rr.value(), e.rz.value()};
  if (grid_sum_last<2>(s, part, &sc->ticket[0]) && threadIdx.x == 0) {
    double res = sqrt(s[0]);
    sc->rr = s[0];
    sc->rz = PRE ? s[1] : s[0];
    sc->res = res;
    sc->res_init = res;
    sc->iter = 0;
    sc->guard = 0;
    sc->state = iterate_check(0, res, *sc, res);
  }
}

// Start from x0 = 0: r = b exactly (b - A*0), no SpMV needed.
template <typename T, bool PRE>
__global__ void __launch_bounds__(kBlock) cg_init_zero_kernel(const T *__restrict__ b, CgVecs<T> v, double *part,
                                                              CgScalars *sc) {
  Acc<T> rr, rz;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < v.n; i += stride) {
    const T r = b[i];
    v.x[i] = T(0);
    v.r[i] = r;
    const T z = PRE ? r * v.invd[i] : r;
    v.p[i] = z;
    rr.add(r * r);
    rz.add(r * z);
  }
  double s[2] = {rr.value(), rz.value()};
  if (grid_sum_last<2>(s, part, &sc->ticket[0]) && threadIdx.x == 0) {
    double res = sqrt(s[0]);
    sc->rr = s[0];
    sc->rz = PRE ? s[1] : s[0];
    sc->res = res;
    sc->res_init = res;
    sc->iter = 0;
    sc->guard = 0;
    sc->state = iterate_check(0, res, *sc, res);
  }
}

// ---- K1: Ap = A p and p.Ap --------------------------------------------------------
template <typename T> struct SpmvDotEmit {
  T *__restrict__ Ap;
  const T *__restrict__ p;
  Acc<T> acc;
  T pr;
  __device__ __forceinline__ void fetch(int row) { pr = __ldg(p + row); }
  __device__ __forceinline__ void operator()(int row, T y) {
    Ap[row] = y;
    acc.add(y * pr);
  }
};

template <typename Op, typename T>
__global__ void __launch_bounds__(kBlock) cg_spmv_kernel(Op op, CgVecs<T> v, double *part, CgScalars *sc) {
  if (__ldg(&sc->state) != B200LA_ITERATE) return;
  SpmvDotEmit<T> e{v.Ap, v.p};
  op.run(v.p, e);
  double s[1] = {e.acc.value()};
  if (grid_sum_last<1>(s, part, &sc->ticket[1]) && threadIdx.x == 0) {
    sc->pAp = s[0];
    double alpha = sc->rz / s[0];
    sc->alpha = alpha;
    if (!(s[0] != 0.0) || !isfinite(alpha)) sc->state = B200LA_FAIL_BREAKDOWN;
  }
}

// ---- K2: x += alpha p, r -= alpha Ap, sums r.r and r.z ----------------------------
template <typename T, bool PRE>
__global__ void __launch_bounds__(kBlock) cg_update_kernel(CgVecs<T> v, double *part, CgScalars *sc) {
  if (__ldg(&sc->state) != B200LA_ITERATE) return;
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::n;
  const T alpha = (T)sc->alpha;
  Acc<T> rr, rz;
  const int64_t n = v.n, nv = n / W;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride) {
    V xv = reinterpret_cast<V *>(v.x)[i];
    V pv = reinterpret_cast<const V *>(v.p)[i];
    V rv = reinterpret_cast<V *>(v.r)[i];
    V av = reinterpret_cast<const V *>(v.Ap)[i];
    V dv;
    if (PRE) dv = reinterpret_cast<const V *>(v.invd)[i];
    T *xs = reinterpret_cast<T *>(&xv);
    T *rs = reinterpret_cast<T *>(&rv);
    const T *ps = reinterpret_cast<const T *>(&pv);
    const T *as = reinterpret_cast<const T *>(&av);
    const T *ds = reinterpret_cast<const T *>(&dv);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      xs[k] = fma(alpha, ps[k], xs[k]);
      rs[k] = fma(-alpha, as[k], rs[k]);
      rr.add(rs[k] * rs[k]);
      if (PRE) rz.add(rs[k] * (rs[k] * ds[k]));
    }
    reinterpret_cast<V *>(v.x)[i] = xv;
    reinterpret_cast<V *>(v.r)[i] = rv;
  }
  for (int64_t i = nv * W + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    v.x[i] = fma(alpha, v.p[i], v.x[i]);
    T r = fma(-alpha, v.Ap[i], v.r[i]);
    v.r[i] = r;
    rr.add(r * r);
    if (PRE) rz.add(r * (r * v.invd[i]));
  }
  double s[2] = {rr.value(), rz.value()};
  if (grid_sum_last<2>(s, part, &sc->ticket[2]) && threadIdx.x == 0) {
    double res = sqrt(s[0]);
    int it = sc->iter + 1;
    sc->iter = it;
    sc->rr = s[0];
    sc->res = res;
    int st = iterate_check(it, res, *sc, sc->res_init);
    double rz_new = PRE ? s[1] : s[0];
    sc->beta = rz_new / sc->rz;
    sc->rz_prev = sc->rz;
    sc->rz = rz_new;
    sc->state = st;
  }
}

// ---- K3: p = beta p + z; ends the device loop ---------------------------------------
template <typename T, bool PRE, bool IN_GRAPH = true>
__global__ void __launch_bounds__(kBlock) cg_direction_kernel(CgVecs<T> v, CgScalars *sc,
                                                              cudaGraphConditionalHandle loop) {
  const int state = __ldg(&sc->state);
  if (IN_GRAPH && blockIdx.x == 0 && threadIdx.x == 0) {
    int g = sc->guard + 1;
    sc->guard = g;
    bool go = state == B200LA_ITERATE;
    if (go && g > sc->maxits + 2) {  // unreachable unless K2 failed to count
      sc->state = B200LA_FAIL_BREAKDOWN;
      go = false;
    }
    cudaGraphSetConditional(loop, go ? 1u : 0u);
  }
  if (state != B200LA_ITERATE) return;
  using V = typename Vec16<T>::type;
  constexpr int W = Vec16<T>::n;
  const T beta = (T)sc->beta;
  const int64_t n = v.n, nv = n / W;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += stride) {
    V pv = reinterpret_cast<V *>(v.p)[i];
    V rv = reinterpret_cast<const V *>(v.r)[i];
    V dv;
    if (PRE) dv = reinterpret_cast<const V *>(v.invd)[i];
    T *ps = reinterpret_cast<T *>(&pv);
    const T *rs = reinterpret_cast<const T *>(&rv);
    const T *ds = reinterpret_cast<const T *>(&dv);
#pragma unroll
    for (int k = 0; k < W; ++k) ps[k] = fma(beta, ps[k], PRE ? rs[k] * ds[k] : rs[k]);
    reinterpret_cast<V *>(v.p)[i] = pv;
  }
  for (int64_t i = nv * W + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    v.p[i] = fma(beta, v.p[i], PRE ? v.r[i] * v.invd[i] : v.r[i]);
}

// ---- the whole loop in one launch, vectors resident ------------------------------
// For systems whose iteration is bound by launches and not by bytes.  Every
// block owns the rows that the schedule gives it (grid-stride, as in K1) and
// keeps their x, r, p, Ap and invD in shared memory for the whole solve; one
// iteration is a gather phase and an update phase with one grid-wide sum
// (tag_sum) after each:
//   gather  p = z + beta p_old on the fly for every column read (the same
//           expression, so the same bits, as the owner's update of its own
//           p), Ap, p.Ap; the owner writes its p for the next iteration's
//           gathers
//   update  alpha; x += alpha p; r -= alpha Ap; z = invD r (written for the
//           gathers); r.r, r.z; every block then takes the same decision
// Two buffers of p by iteration parity: p_old of this iteration is read while
// p is written to the other.  z has one: a block rewrites its rows after the
// p.Ap sum, which every block has added to once its gathers are done.
// The first gather reads z = the given p and p_old = 0 with beta = 0.
template <typename T> struct CgGather {
  const T *z, *po;  // not read-only: rewritten between phases
  T beta;
  __device__ __forceinline__ T operator()(int c) const { return fma(beta, po[c], z[c]); }
  __device__ __forceinline__ CgGather at(int row) const { return CgGather{z + row, po + row, beta}; }
  __device__ __forceinline__ void pair(int c, T &a, T &b) const {
    a = (*this)(c);
    b = (*this)(c + 1);
  }
};

template <typename T> struct CgResidentBufs {
  T *z, *p0, *p1;
  int rows;  // shared-memory rows per block
};

template <typename T, bool PRE> struct CgGatherEmit {
  T *ps, *aps, *pn;
  const T *rs, *ds;
  T beta;
  bool first;
  int at, step;  // shared-memory index of this thread's next row
  Acc<T> acc;
  __device__ __forceinline__ void fetch(int) {}
  __device__ __forceinline__ void operator()(int row, T y) {
    T p = ps[at];
    if (!first) p = fma(beta, p, PRE ? rs[at] * ds[at] : rs[at]);
    ps[at] = p;
    aps[at] = y;
    pn[row] = p;
    acc.add(y * p);
    at += step;
  }
};

template <typename Op, typename T, bool PRE, int NT>
__global__ void __launch_bounds__(NT, 1) cg_resident_kernel(Op op, CgVecs<T> v, CgResidentBufs<T> rb, TagSync ts,
                                                            unsigned long long epoch, CgScalars *sc) {
  extern __shared__ __align__(16) unsigned char cg_dyn[];
  if (*(volatile int *)&sc->state != B200LA_ITERATE) return;
  constexpr int G = Op::kLanes;
  const int R = rb.rows;
  T *xs = reinterpret_cast<T *>(cg_dyn), *rs = xs + R, *ps = rs + R, *aps = ps + R, *ds = aps + R;
  int *row_of = reinterpret_cast<int *>(ds + (PRE ? R : 0));
  const int at0 = (int)threadIdx.x / G;
  constexpr int step = NT / G;
  int cnt = 0;
  op.template each_row<NT>([&](int row) {
    const int a = at0 + cnt * step;
    row_of[a] = row;
    xs[a] = v.x[row];
    rs[a] = v.r[row];
    const T p = v.p[row];
    ps[a] = p;
    if (PRE) ds[a] = v.invd[row];
    rb.z[row] = p;
    rb.p0[row] = T(0);
    ++cnt;
  });
  double rz = sc->rz, rz_prev = sc->rz_prev, rr = sc->rr, res = sc->res, beta_d = 0.0, alpha_d = 0.0, pap = 0.0;
  const double first_res = sc->res_init;
  const CgScalars lim = *sc;  // tolerances, maxits and the stop rule
  int iter = lim.iter, state = B200LA_ITERATE;
  if ((int)blockIdx.x == lim.stall_block) return;  // test hook: this block never joins a sum
  bool first = true;
  double s0[1] = {0.0};
  bool ok = tag_sum<1, true>(s0, ts, ++epoch);  // z and p0 are written
  // maxits ends the loop; the bound only guards against broken sums
  for (int k = 0; ok && state == B200LA_ITERATE && k < lim.maxits + 2; ++k) {
    T *pn = (k & 1) ? rb.p0 : rb.p1;
    const T beta = (T)beta_d;
    CgGatherEmit<T, PRE> e{ps, aps, pn, rs, ds, beta, first, at0, step};
    op.template run_with<NT>(CgGather<T>{rb.z, (k & 1) ? rb.p1 : rb.p0, beta}, e);
    first = false;
    double s1[1] = {e.acc.value()};
    ok = tag_sum<1, false>(s1, ts, ++epoch);
    if (!ok) break;
    pap = s1[0];
    alpha_d = rz / pap;
    if (!(pap != 0.0) || !isfinite(alpha_d)) {
      state = B200LA_FAIL_BREAKDOWN;
      break;
    }
    const T alpha = (T)alpha_d;
    Acc<T> arr, arz;
    for (int c = 0; c < cnt; ++c) {
      const int a = at0 + c * step;
      xs[a] = fma(alpha, ps[a], xs[a]);
      const T r = fma(-alpha, aps[a], rs[a]);
      rs[a] = r;
      const T z = PRE ? r * ds[a] : r;
      rb.z[row_of[a]] = z;
      arr.add(r * r);
      if (PRE) arz.add(r * z);
    }
    double s2[2] = {arr.value(), arz.value()};
    ok = tag_sum<2, true>(s2, ts, ++epoch);
    if (!ok) break;
    rr = s2[0];
    res = sqrt(rr);
    ++iter;
    state = iterate_check(iter, res, lim, first_res);
    const double rz_new = PRE ? s2[1] : rr;
    beta_d = rz_new / rz;
    rz_prev = rz;
    rz = rz_new;
  }
  if (ok && state == B200LA_ITERATE) state = B200LA_FAIL_BREAKDOWN;  // the guard
  for (int c = 0; c < cnt; ++c) {
    const int a = at0 + c * step, row = row_of[a];
    v.x[row] = xs[a];
    v.r[row] = rs[a];
    v.p[row] = ps[a];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->rz = rz;
    sc->rz_prev = rz_prev;
    sc->pAp = pap;
    sc->alpha = alpha_d;
    sc->beta = beta_d;
    sc->rr = rr;
    sc->res = res;
    sc->iter = iter;
    sc->state = ok ? state : B200LA_FAIL_BREAKDOWN;
  }
}

// ---- the whole loop on one cluster (cluster_cg.cuh) -------------------------------
// The same recurrence, decisions and outputs as the graph of three kernels;
// the matrix is read once, when shared memory is filled.
template <typename M, typename T, int H, int R, bool PRE>
__global__ void __launch_bounds__(kClThreads, 1) cg_cluster_kernel(ClMatrix<M> m, CgVecs<T> v, CgScalars *sc) {
  extern __shared__ __align__(16) unsigned char cl_dyn[];
  if (*(volatile int *)&sc->state != B200LA_ITERATE) return;
  ClCg<T, H, R, PRE> g;
  g.carve(cl_dyn, m);
  g.fill(m);
  g.load_window(v.p);
  g.each([&](int j, int li) {
    const int row = g.r0 + li;
    g.c[j] = v.x[row];
    g.r[j] = v.r[row];
    if (PRE) g.d[j] = v.invd[row];
  });
  const CgScalars lim = *sc;  // tolerances, maxits, the stop rule and the start
  double rz = lim.rz, rz_prev = lim.rz_prev, rr = lim.rr, res = lim.res, beta_d = 0.0, alpha_d = 0.0, pap = 0.0;
  int iter = lim.iter, state = B200LA_ITERATE;
  cl_barrier(g.blocks);  // every block of the cluster runs and has its window
  // maxits ends the loop; the bound only guards against broken sums
  for (int k = 0; state == B200LA_ITERATE && k < lim.maxits + 2; ++k) {
    double s1[1] = {g.multiply()};
    g.template sum<1>(s1, 0);
    pap = s1[0];
    alpha_d = rz / pap;
    if (!(pap != 0.0) || !isfinite(alpha_d)) {
      state = B200LA_FAIL_BREAKDOWN;
      break;
    }
    const T alpha = (T)alpha_d;
    double s2[2];
    g.update(alpha, s2);
    g.template sum<2>(s2, 1);
    rr = s2[0];
    res = sqrt(rr);
    ++iter;
    state = iterate_check(iter, res, lim, lim.res_init);
    const double rz_new = PRE ? s2[1] : rr;
    beta_d = rz_new / rz;
    rz_prev = rz;
    rz = rz_new;
    if (state == B200LA_ITERATE)
      g.direction((T)beta_d, true, [&](int j, T p) { g.c[j] = fma(alpha, p, g.c[j]); });
    else
      g.each([&](int j, int li) { g.c[j] = fma(alpha, g.pw[li + g.halo], g.c[j]); });
  }
  if (state == B200LA_ITERATE) state = B200LA_FAIL_BREAKDOWN;  // the guard
  g.each([&](int j, int li) {
    const int row = g.r0 + li;
    v.x[row] = g.c[j];
    v.r[row] = g.r[j];
    v.p[row] = g.pw[li + g.halo];
  });
  cl_barrier(g.blocks);  // no block leaves while another may still write to its shared memory
  if (g.rank == 0 && threadIdx.x == 0) {
    sc->rz = rz;
    sc->rz_prev = rz_prev;
    sc->pAp = pap;
    sc->alpha = alpha_d;
    sc->beta = beta_d;
    sc->rr = rr;
    sc->res = res;
    sc->iter = iter;
    sc->state = state;
  }
}

// ---- resume after a residual replacement: x = 0, p = z + beta p ------------------
// Every block derives beta from the same two scalars; block 0 then resets the
// solve's scalars for the new start (none of which the other blocks read).
template <typename T, bool PRE>
__global__ void __launch_bounds__(kBlock) cg_resume_kernel(CgVecs<T> v, const double *__restrict__ sums,
                                                           CgScalars *sc, int restart) {
  const double rr = sums[0], rz_new = PRE ? sums[1] : sums[0];
  const double beta_d = rz_new / __ldg(&sc->rz_prev);
  const bool keep = !restart && isfinite(beta_d);
  const T beta = keep ? (T)beta_d : T(0);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < v.n; i += stride) {
    const T r = v.r[i];
    const T z = PRE ? r * v.invd[i] : r;
    v.x[i] = T(0);
    v.p[i] = keep ? fma(beta, v.p[i], z) : z;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const double res = sqrt(rr);
    sc->rr = rr;
    sc->rz = rz_new;
    sc->res = res;
    sc->res_init = res;
    sc->iter = 0;
    sc->guard = 0;
    sc->state = iterate_check(0, res, *sc, res);
  }
}

}  // namespace b200la

using namespace b200la;

namespace b200la {

// One iteration: K1, K2, K3 on stream `st` (captured into the graph body,
// or launched from the host loop when graphs are off).
// M = stored matrix value type, T = vector type (M == T, or FP32 values over
// FP64 vectors).
template <typename M, typename T, bool PRE, bool IN_GRAPH>
static int cg_launch_body_t(b200la_cg s, cudaStream_t st, cudaGraphConditionalHandle h) {
  b200la_mat A = s->A;
  b200la_ctx c = A->ctx;
  CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  B_TRY((with_schedule<M, T>(A, [&](auto op) -> int {
    using Op = decltype(op);
    B_TRY(grid_for(c, (const void *)cg_spmv_kernel<Op, T>, op.work_items(), Op::kRowsPerBlock, &s->grid_spmv));
    cg_spmv_kernel<Op, T><<<s->grid_spmv, kBlock, 0, st>>>(op, v, s->part, s->sc);
    return B200LA_OK;
  })));
  cg_update_kernel<T, PRE><<<s->grid_ew, kBlock, 0, st>>>(v, s->part, s->sc);
  cg_direction_kernel<T, PRE, IN_GRAPH><<<s->grid_ew, kBlock, 0, st>>>(v, s->sc, h);
  return B200LA_OK;
}

// Calls f(M(), T(), std::bool_constant<PRE>()) with the solver's matrix value
// type M, vector type T and preconditioning.
template <typename F> static int cg_types(b200la_cg s, F &&f) {
  const bool pre = s->prm.precond != 0;
  auto go = [&](auto m, auto t) -> int { return pre ? f(m, t, std::true_type()) : f(m, t, std::false_type()); };
  if (s->A->dtype == B200LA_F64) return go(double(), double());
  if (s->vdtype == B200LA_F64) return go(float(), double());
  return go(float(), float());
}

template <typename M, typename T, bool PRE>
static int cg_build_graph_t(b200la_cg s) {
  b200la_mat A = s->A;
  b200la_ctx c = A->ctx;
  if (s->exec) { cudaGraphExecDestroy(s->exec); s->exec = nullptr; }
  if (s->graph) { cudaGraphDestroy(s->graph); s->graph = nullptr; }
  CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  B_TRY(grid_for(c, (const void *)cg_update_kernel<T, PRE>, (s->n + Vec16<T>::n - 1) / Vec16<T>::n, kBlock, &s->grid_ew));
  cudaGraph_t g;
  B_CUDA(cudaGraphCreate(&g, 0));
  s->graph = g;
  cudaGraphConditionalHandle h;
  B_CUDA(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
  cudaGraphNodeParams np = {};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = h;
  np.conditional.type = cudaGraphCondTypeWhile;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  B_CUDA(cudaGraphAddNode(&node, g, nullptr, 0, &np));
  cudaGraph_t body = np.conditional.phGraph_out[0];
  cudaStream_t cs;
  B_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  B_CUDA(cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  int rc = B200LA_OK;
  for (int k = 0; k < kWhileUnroll && rc == B200LA_OK; ++k) rc = cg_launch_body_t<M, T, PRE, true>(s, cs, h);
  cudaGraph_t captured;
  cudaError_t ce = cudaStreamEndCapture(cs, &captured);
  cudaStreamDestroy(cs);
  B_TRY(rc);
  B_CUDA(ce);
  B_CUDA(cudaGraphInstantiate(&s->exec, g, 0));
  s->g_format = A->format;
  s->g_param = A->param;
  s->g_gen = A->sched_gen;
  return B200LA_OK;
}

template <typename M, typename T, bool PRE> static int cg_size_cluster_t(b200la_cg s);
template <typename M, typename T, bool PRE> static int cg_size_resident_t(b200la_cg s);
static int cg_resident_buffers(b200la_cg s);
static int cg_build_graph(b200la_cg s);

// Picks the form for the matrix's current schedule: one cluster, the resident
// kernel, or the three kernels (whose graph is built here).
static int cg_select_form(b200la_cg s) {
  b200la_mat A = s->A;
  s->cl_blocks = s->res_blocks = 0;
  s->g_onchip = A->ctx->use_onchip;
  if (!s->g_onchip) return cg_build_graph(s);
  B_TRY(cg_types(s, [&](auto m, auto t, auto pre) -> int {
    using M = decltype(m);
    using T = decltype(t);
    constexpr bool PRE = decltype(pre)::value;
    B_TRY((cg_size_cluster_t<M, T, PRE>(s)));
    return s->cl_blocks > 0 ? B200LA_OK : cg_size_resident_t<M, T, PRE>(s);
  }));
  if (s->res_blocks > 0) B_TRY(cg_resident_buffers(s));
  if (s->cl_blocks == 0 && s->res_blocks == 0) return cg_build_graph(s);
  s->g_format = A->format;
  s->g_param = A->param;
  s->g_gen = A->sched_gen;
  return B200LA_OK;
}

static int cg_build_graph(b200la_cg s) {
  return cg_types(s, [&](auto m, auto t, auto pre) -> int {
    return cg_build_graph_t<decltype(m), decltype(t), decltype(pre)::value>(s);
  });
}

template <typename M, typename T, bool PRE>
static int cg_launch_init_t(b200la_cg s, const void *x_user, const void *b) {
  b200la_mat A = s->A;
  CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  cudaStream_t st = A->ctx->stream;
  if (!x_user) {
    int grid;
    B_TRY(grid_for(A->ctx, (const void *)cg_init_zero_kernel<T, PRE>, s->n, kBlock, &grid));
    cg_init_zero_kernel<T, PRE><<<grid, kBlock, 0, st>>>((const T *)b, v, s->part, s->sc);
    B_CUDA(cudaGetLastError());
    return B200LA_OK;
  }
  return with_schedule<M, T>(A, [&](auto op) -> int {
    using Op = decltype(op);
    int grid;
    B_TRY(grid_for(A->ctx, (const void *)cg_init_kernel<Op, T, PRE>, op.work_items(), Op::kRowsPerBlock, &grid));
    cg_init_kernel<Op, T, PRE><<<grid, kBlock, 0, st>>>(op, (const T *)x_user, (const T *)b, v, s->part, s->sc);
    B_CUDA(cudaGetLastError());
    return B200LA_OK;
  });
}

static int cg_launch_init(b200la_cg s, const void *x_user, const void *b) {
  return cg_types(s, [&](auto m, auto t, auto pre) -> int {
    return cg_launch_init_t<decltype(m), decltype(t), decltype(pre)::value>(s, x_user, b);
  });
}

int cg_start(b200la_cg s, const void *x_dev, const void *b_dev) { return cg_launch_init(s, x_dev, b_dev); }

int cg_resume(b200la_cg s, const double *sums, bool restart) {
  cudaStream_t st = s->A->ctx->stream;
  return cg_types(s, [&](auto m, auto t, auto pre) -> int {
    using T = decltype(t);
    constexpr bool PRE = decltype(pre)::value;
    CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
    int grid;
    B_TRY(grid_for(s->A->ctx, (const void *)cg_resume_kernel<T, PRE>, s->n, kBlock, &grid));
    cg_resume_kernel<T, PRE><<<grid, kBlock, 0, st>>>(v, sums, s->sc, restart ? 1 : 0);
    B_CUDA(cudaGetLastError());
    return B200LA_OK;
  });
}

template <typename M, typename T, bool PRE>
static int cg_host_loop_t(b200la_cg s) {
  cudaStream_t st = s->A->ctx->stream;
  // the kernels return at once when the state is no longer "iterate", so
  // checking the state every 16 iterations runs the same iterations
  for (int64_t it = 0;; it += 16) {
    for (int k = 0; k < 16; ++k) B_TRY((cg_launch_body_t<M, T, PRE, false>(s, st, 0)));
    B_CUDA(cudaGetLastError());
    CgScalars h;
    B_TRY(cg_fetch(s, &h));
    if (h.state != B200LA_ITERATE || it > (int64_t)s->prm.maxits + 32) break;
  }
  return B200LA_OK;
}

// Shared-memory bytes per owned row of the resident kernel: x, r, p, Ap (and
// invD) and the row's number.
template <typename T> static size_t cg_resident_row_bytes(bool pre) { return sizeof(T) * (pre ? 5 : 4) + sizeof(int); }

constexpr int kCgResThreads = 512;

// Blocks of the resident form: the sums cost 1.3 / 2.6 us (without / with
// published stores) up to 32 blocks and about twice that on more, so more
// blocks pay once a block's rows take longer than that.  Measured, us an
// iteration on 32 / 64 / 100 / 148 blocks: 2D 256^2 9.0 / 11.1 / 11.4 / 12.2,
// 400^2 15.5 / 12.9 / 12.7 / 14.2, 600^2 24 / 24 / 18.3 / 18.9; 3D 32^3
// 12.4 / 15.0 / 12.6 / 15.2, 48^3 24.6 / 18.2 / 16.5 / 16.0.
static int cg_resident_blocks(int64_t n, int max_row, int sms) {
  if (n <= 72000) return 32;
  return max_row <= 12 ? std::min(100, sms) : sms;
}
// Beyond this many rows the graph's three kernels win (their launches and
// the WHILE node cost ~8 us an iteration; the resident form gathers two
// vectors instead of one): 2D 600^2 18.3 against 23.7 us, 3D 48^3 16.0
// against 21.3, 64^3 26.0 against 27.6.
static int64_t cg_resident_limit(int max_row) { return max_row <= 12 ? 420000 : 280000; }

// Sizes the resident form, or leaves res_blocks = 0.
template <typename M, typename T, bool PRE> static int cg_size_resident_t(b200la_cg s) {
  s->res_blocks = 0;
  b200la_mat A = s->A;
  b200la_ctx c = A->ctx;
  int optin = 0;
  B_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  // CSR chains three dependent loads (row pointer, column, gather) behind
  // every grid-wide sum and was slower than the graph at every size tried
  if (!is_sliced(A->format) || s->n > cg_resident_limit(A->max_row)) return B200LA_OK;
  return with_schedule<M, T>(A, [&](auto op) -> int {
    using Op = decltype(op);
    constexpr int NT = kCgResThreads;
    const void *k = (const void *)cg_resident_kernel<Op, T, PRE, NT>;
    const int64_t threads = op.work_items() * Op::kLanes;
    int blocks = (int)std::min<int64_t>((threads + NT - 1) / NT, c->num_sms);
    blocks = std::max(1, std::min(blocks, cg_resident_blocks(s->n, A->max_row, c->num_sms)));
    const int rows = op.template rows_per_block<NT>(blocks);
    const size_t bytes = cg_resident_row_bytes<T>(PRE) * (size_t)rows;
    cudaFuncAttributes fa;
    B_CUDA(cudaFuncGetAttributes(&fa, k));
    if (bytes + fa.sharedSizeBytes > (size_t)optin) return B200LA_OK;
    B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
    int per_sm = 0;
    B_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, NT, bytes));
    if (per_sm < 1) return B200LA_OK;
    s->res_blocks = blocks;
    s->res_rows = rows;
    return B200LA_OK;
  });
}

constexpr int kCgClRows = 9;  // most rows a thread of the cluster form (257 x 257 nodes on 16 blocks)

// Rows a thread of the instance that holds `need` of them (<= kCgClRows).
static int cg_cluster_rows(int need) { return need <= 1 ? 1 : need <= 3 ? 3 : need <= 6 ? 6 : kCgClRows; }

// Calls f(H, R) (integral constants) for a cluster solve with `up` upper
// offsets and `regs` (a value of cg_cluster_rows) rows a thread.
template <typename T, typename F> static int cl_dispatch(int up, int regs, F &&f) {
  auto with_r = [&](auto h) -> int {
    if (regs == 1) return f(h, std::integral_constant<int, 1>());
    if (regs == 3) return f(h, std::integral_constant<int, 3>());
    if (regs == 6) return f(h, std::integral_constant<int, 6>());
    return f(h, std::integral_constant<int, kCgClRows>());
  };
  return up <= 4 ? with_r(std::integral_constant<int, 4>()) : with_r(std::integral_constant<int, kClMaxOff>());
}

static ClMatrix<char> cl_matrix_head(b200la_mat A) {
  ClMatrix<char> m{};
  m.n = A->nrow;
  m.H = A->cl_H;
  m.halo = A->cl_off[A->cl_H - 1];
  for (int k = 0; k < A->cl_H; ++k) m.off[k] = A->cl_off[k];
  m.rowptr = A->rowptr;
  m.col = A->col;
  return m;
}
template <typename M> static ClMatrix<M> cl_matrix(b200la_mat A) {
  const ClMatrix<char> h = cl_matrix_head(A);
  ClMatrix<M> m{h.n, h.H, h.halo, {}, h.rowptr, h.col, (const M *)A->val};
  for (int k = 0; k < kClMaxOff; ++k) m.off[k] = h.off[k];
  return m;
}

// Blocks of the cluster form: a block's rows take ~0.8 ns each (FP64, nine
// points), the two sums of an iteration 0.5 us more on 8 blocks than on one
// and 1.5 us on 16.  Measured, us an iteration on 1 / 2 / 4 / 8 / 16 blocks
// (the graph of three kernels 16-18): 289 rows 2.75 / 3.2 / 3.2 / 3.5 / 4.5,
// 2,401 rows 5.2 / 4.8 / 3.3 / 3.2 / 4.1, 10,201 rows - / - / 5.8 / 5.0 / 4.3,
// 25,921 rows 6.5 on 8, 6.2 on 16, 66,049 rows 8.4 on 16 (- : does not fit).
static int cg_cluster_blocks(int64_t n) { return n <= kClThreads ? 1 : n <= 6000 ? 8 : kClMaxBlocks; }

// Sizes the cluster form, or leaves cl_blocks = 0.
template <typename M, typename T, bool PRE> static int cg_size_cluster_t(b200la_cg s) {
  s->cl_blocks = 0;
  b200la_mat A = s->A;
  b200la_ctx c = A->ctx;
  if (s->n > (int64_t)kClMaxBlocks * kClThreads * kCgClRows) return B200LA_OK;
  B_TRY(cl_detect(A));
  if (A->cl_state != 1) return B200LA_OK;
  int optin = 0;
  B_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device));
  const int blocks = cg_cluster_blocks(s->n);
  const int rpc = cl_rows_per_block((int)s->n, blocks);
  const int need = (rpc + kClThreads - 1) / kClThreads;
  if (need > kCgClRows) return B200LA_OK;
  const int regs = cg_cluster_rows(need);
  const size_t smem = cl_smem_bytes(rpc, A->cl_off[A->cl_H - 1], A->cl_H, regs, sizeof(T));
  return cl_dispatch<T>(A->cl_H, regs, [&](auto h, auto r) -> int {
    auto k = cg_cluster_kernel<M, T, decltype(h)::value, decltype(r)::value, PRE>;
    cudaFuncAttributes fa;
    B_CUDA(cudaFuncGetAttributes(&fa, k));
    if (smem + fa.sharedSizeBytes > (size_t)optin) return B200LA_OK;
    B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
    B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cl_config(blocks, smem, c->stream, attr);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
      cudaGetLastError();  // a cluster of this size cannot be placed: another form
      return B200LA_OK;
    }
    s->cl_blocks = blocks;
    s->cl_regs = regs;
    s->cl_smem = smem;
    return B200LA_OK;
  });
}

template <typename M, typename T, bool PRE> static int cg_run_cluster_t(b200la_cg s) {
  b200la_mat A = s->A;
  cudaLaunchAttribute attr[1];
  const cudaLaunchConfig_t cfg = cl_config(s->cl_blocks, s->cl_smem, A->ctx->stream, attr);
  const CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  const ClMatrix<M> m = cl_matrix<M>(A);
  return cl_dispatch<T>(A->cl_H, s->cl_regs, [&](auto h, auto r) -> int {
    B_CUDA(cudaLaunchKernelEx(&cfg, cg_cluster_kernel<M, T, decltype(h)::value, decltype(r)::value, PRE>, m, v,
                              s->sc));
    return B200LA_OK;
  });
}

// Buffers of the resident form, made when it is first chosen.
static int cg_resident_buffers(b200la_cg s) {
  if (s->tag_slots) return B200LA_OK;
  cudaStream_t st = s->ctx->stream;
  const size_t vb = dtype_size(s->vdtype) * (size_t)s->n;
  if (cudaMallocAsync(&s->zg, vb, st) != cudaSuccess || cudaMallocAsync(&s->pg[0], vb, st) != cudaSuccess ||
      cudaMallocAsync(&s->pg[1], vb, st) != cudaSuccess ||
      cudaMallocAsync(&s->tag_slots, kTagSlotBytes, st) != cudaSuccess)
    return fail(B200LA_ERR_NOMEM, "cg: allocation of %zu-byte gather buffers failed", vb);
  B_CUDA(cudaMemsetAsync(s->tag_slots, 0, kTagSlotBytes, st));
  s->epoch = 0;
  return B200LA_OK;
}

template <typename M, typename T, bool PRE> static int cg_run_resident_t(b200la_cg s) {
  b200la_mat A = s->A;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = A->ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)s->res_blocks);
  cfg.blockDim = dim3(kCgResThreads);
  cfg.dynamicSmemBytes = cg_resident_row_bytes<T>(PRE) * (size_t)s->res_rows;
  const CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  const CgResidentBufs<T> rb{(T *)s->zg, (T *)s->pg[0], (T *)s->pg[1], s->res_rows};
  const TagSync ts{(TagSlot *)s->tag_slots, &s->sc->err};
  const unsigned long long epoch = s->epoch;
  s->epoch += 2ull * ((unsigned long long)s->prm.maxits + 4ull);
  return with_schedule<M, T>(A, [&](auto op) -> int {
    using Op = decltype(op);
    B_CUDA(cudaLaunchKernelEx(&cfg, cg_resident_kernel<Op, T, PRE, kCgResThreads>, op, v, rb, ts, epoch, s->sc));
    return B200LA_OK;
  });
}

int cg_run(b200la_cg s) {
  b200la_mat A = s->A;
  if (A->format != s->g_format || A->param != s->g_param || A->sched_gen != s->g_gen ||
      A->ctx->use_onchip != s->g_onchip)
    B_TRY(cg_select_form(s));
  if (s->cl_blocks > 0)
    return cg_types(s, [&](auto m, auto t, auto pre) -> int {
      return cg_run_cluster_t<decltype(m), decltype(t), decltype(pre)::value>(s);
    });
  if (s->res_blocks > 0)
    return cg_types(s, [&](auto m, auto t, auto pre) -> int {
      return cg_run_resident_t<decltype(m), decltype(t), decltype(pre)::value>(s);
    });
  if (!A->ctx->use_graphs) {
    return cg_types(s, [&](auto m, auto t, auto pre) -> int {
      return cg_host_loop_t<decltype(m), decltype(t), decltype(pre)::value>(s);
    });
  }
  B_CUDA(cudaGraphLaunch(s->exec, A->ctx->stream));
  return B200LA_OK;
}

int cg_fetch(b200la_cg s, CgScalars *out) {
  cudaStream_t st = s->A->ctx->stream;
  B_CUDA(cudaMemcpyAsync(s->sc_host, s->sc, sizeof(CgScalars), cudaMemcpyDeviceToHost, st));
  B_CUDA(cudaStreamSynchronize(st));
  *out = *s->sc_host;
  if (out->err != 0) {  // the blocks left at different epochs: fresh slots for the next solve
    B_CUDA(cudaMemsetAsync(&s->sc->err, 0, sizeof(unsigned), st));
    B_CUDA(cudaMemsetAsync(s->tag_slots, 0, kTagSlotBytes, st));
    return fail(B200LA_ERR_TIMEOUT, "cg: a wait of the resident kernel ran out");
  }
  return B200LA_OK;
}

// Runs the init kernel and then `iters` iterations as separate launches with
// CUDA events between the kernels; adds the mean time per launch of K1, K2
// and K3 to ms[0..2].  Same kernels as the graph body (K3 without the loop
// condition).
template <typename M, typename T, bool PRE>
static int cg_profile_t(b200la_cg s, const void *x_user, const void *b, int iters, double *ms) {
  b200la_mat A = s->A;
  cudaStream_t st = A->ctx->stream;
  CgVecs<T> v{(T *)s->x, (T *)s->r, (T *)s->p, (T *)s->Ap, (const T *)s->invd, s->n};
  // the grids of the three kernels on the matrix's present schedule, whatever
  // form the solves take; what the solver has selected stays untouched
  int grid_spmv = 0, grid_ew = 0;
  B_TRY(grid_for(A->ctx, (const void *)cg_update_kernel<T, PRE>, (s->n + Vec16<T>::n - 1) / Vec16<T>::n, kBlock,
                 &grid_ew));
  B_TRY((with_schedule<M, T>(A, [&](auto op) -> int {
    using Op = decltype(op);
    return grid_for(A->ctx, (const void *)cg_spmv_kernel<Op, T>, op.work_items(), Op::kRowsPerBlock, &grid_spmv);
  })));
  B_TRY((cg_launch_init_t<M, T, PRE>(s, x_user, b)));
  // every pass is queued before the first wait, after one untimed pass, so
  // the timed kernels run back to back and no host launch gap falls between
  // an event pair
  std::vector<cudaEvent_t> ev((size_t)(iters > 0 ? iters : 0) * 4);
  for (auto &e : ev) B_CUDA(cudaEventCreate(&e));
  int rc = B200LA_OK;
  auto pass = [&](cudaEvent_t *e) -> int {
    if (e) cudaEventRecord(e[0], st);
    B_TRY((with_schedule<M, T>(A, [&](auto op) -> int {
      using Op = decltype(op);
      cg_spmv_kernel<Op, T><<<grid_spmv, kBlock, 0, st>>>(op, v, s->part, s->sc);
      return B200LA_OK;
    })));
    if (e) cudaEventRecord(e[1], st);
    cg_update_kernel<T, PRE><<<grid_ew, kBlock, 0, st>>>(v, s->part, s->sc);
    if (e) cudaEventRecord(e[2], st);
    cg_direction_kernel<T, PRE, false><<<grid_ew, kBlock, 0, st>>>(v, s->sc, 0);
    if (e) cudaEventRecord(e[3], st);
    return B200LA_OK;
  };
  if (iters > 0) rc = pass(nullptr);
  for (int it = 0; it < iters && rc == B200LA_OK; ++it) rc = pass(&ev[(size_t)it * 4]);
  const cudaError_t se = cudaStreamSynchronize(st);
  float acc[3] = {0.f, 0.f, 0.f};
  for (int it = 0; it < iters && rc == B200LA_OK && se == cudaSuccess; ++it)
    for (int k = 0; k < 3; ++k) {
      float t = 0.f;
      cudaEventElapsedTime(&t, ev[(size_t)it * 4 + k], ev[(size_t)it * 4 + k + 1]);
      acc[k] += t;
    }
  for (auto &e : ev) cudaEventDestroy(e);
  B_CUDA(se);
  B_CUDA(cudaGetLastError());
  for (int k = 0; k < 3; ++k) ms[k] = iters > 0 ? acc[k] / iters : 0.0;
  return rc;
}

}  // namespace b200la

extern "C" {

int b200la_cg_form(b200la_cg s, int *form) {
  B_CHECK(s && form, B200LA_ERR_INVALID, "cg_form: null argument");
  *form = s->cl_blocks > 0 ? B200LA_FORM_CLUSTER : s->res_blocks > 0 ? B200LA_FORM_RESIDENT : B200LA_FORM_KERNELS;
  return B200LA_OK;
}

int b200la_cg_profile(b200la_cg s, b200la_vec b, b200la_vec x, int iters, double *ms) {
  B_CHECK(s && b && x && ms && iters >= 0, B200LA_ERR_INVALID, "cg_profile: bad argument");
  B_CHECK(b->n == s->n && x->n == s->n && s->n > 0, B200LA_ERR_INVALID, "cg_profile: sizes");
  B_CHECK(b->dtype == s->vdtype && x->dtype == s->vdtype, B200LA_ERR_DTYPE, "cg_profile: dtype");
  return cg_types(s, [&](auto m, auto t, auto pre) -> int {
    return cg_profile_t<decltype(m), decltype(t), decltype(pre)::value>(s, x->d, b->d, iters, ms);
  });
}

int b200la_cg_create(b200la_mat A, const b200la_cg_params *prm, b200la_cg *out) {
  B_CHECK(A, B200LA_ERR_INVALID, "cg_create: null argument");
  return cg_create_ex(A, prm, A->dtype, nullptr, out);
}

}  // extern "C"

int b200la::cg_create_ex(b200la_mat A, const b200la_cg_params *prm, int vdtype, b200la_mat invd_src,
                         b200la_cg *out) {
  B_CHECK(A && prm && out, B200LA_ERR_INVALID, "cg_create: null argument");
  B_CHECK(vdtype == A->dtype || (A->dtype == B200LA_F32 && vdtype == B200LA_F64), B200LA_ERR_DTYPE,
          "cg_create: vectors of dtype %d over a matrix of dtype %d", vdtype, A->dtype);
  B_CHECK(vdtype == A->dtype || !prm->precond ||
              (invd_src && invd_src->dtype == vdtype && invd_src->nrow == A->nrow && invd_src->nnz == A->nnz),
          B200LA_ERR_INVALID, "cg_create: mixed storage with Jacobi needs an FP64 matrix of the same structure");
  B_CHECK(A->nrow == A->ncol, B200LA_ERR_INVALID, "cg_create: matrix is %dx%d, not square", A->nrow, A->ncol);
  B_CHECK(prm->maxits >= 0 && prm->maxits <= kMaxIts, B200LA_ERR_INVALID, "cg_create: maxits %d not in [0, %d]",
          prm->maxits, kMaxIts);
  B_CHECK(prm->atol >= 0.0 && prm->rtol >= 0.0 && prm->dtol > 0.0, B200LA_ERR_INVALID,
          "cg_create: tolerances must be atol >= 0, rtol >= 0, dtol > 0");
  B_CHECK(prm->stop_rule == B200LA_STOP_ITERATE_CONTROL || (prm->stop_rule == B200LA_STOP_LMP_CG && !prm->precond),
          B200LA_ERR_INVALID, "cg_create: stop_rule %d (the lmp cg() rule takes no preconditioner)", prm->stop_rule);
  b200la_ctx c = A->ctx;
  cudaStream_t st = c->stream;
  b200la_cg s = new b200la_cg_s();
  s->A = A;
  s->ctx = c;
  s->prm = *prm;
  s->vdtype = vdtype;
  s->n = A->nrow;
  size_t es = dtype_size(vdtype);
  size_t vb = es * (size_t)(s->n > 0 ? s->n : 1);
  int rc = B200LA_OK;
  auto cleanup = [&](int code) { b200la_cg_destroy(s); return code; };
  if (cudaMallocAsync(&s->x, vb, st) != cudaSuccess || cudaMallocAsync(&s->r, vb, st) != cudaSuccess ||
      cudaMallocAsync(&s->p, vb, st) != cudaSuccess || cudaMallocAsync(&s->Ap, vb, st) != cudaSuccess ||
      cudaMallocAsync(&s->part, sizeof(double) * 2 * kMaxReduceBlocks, st) != cudaSuccess ||
      cudaMallocAsync(&s->sc, sizeof(CgScalars), st) != cudaSuccess ||
      cudaMallocHost(&s->sc_host, sizeof(CgScalars)) != cudaSuccess)
    return cleanup(fail(B200LA_ERR_NOMEM, "cg_create: allocation of %zu-byte work vectors failed", vb));
  CgScalars init = {};
  init.atol = prm->atol;
  init.rtol = prm->rtol;
  init.dtol = prm->dtol;
  init.maxits = prm->maxits;
  init.stop_rule = prm->stop_rule;
  init.state = B200LA_ITERATE;
  // B200LA_TEST_STALL_BARRIER=b makes block b of the resident kernel leave
  // before its first sum, so that the others' waits run out and the solve
  // ends with B200LA_ERR_TIMEOUT (as in GMRES; never set in normal use)
  const char *stall = getenv("B200LA_TEST_STALL_BARRIER");
  init.stall_block = stall && stall[0] ? atoi(stall) : -1;
  if (cudaMemcpyAsync(s->sc, &init, sizeof(init), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return cleanup(fail(B200LA_ERR_CUDA, "cg_create: scalar upload failed"));
  if (prm->precond) {
    if (cudaMallocAsync(&s->invd, vb, st) != cudaSuccess)
      return cleanup(fail(B200LA_ERR_NOMEM, "cg_create: allocation of the inverse diagonal failed"));
    b200la_vec_s dv{c, s->n, vdtype, s->invd, false};
    rc = b200la_mat_inv_diag(vdtype == A->dtype ? A : invd_src, &dv);
    if (rc != B200LA_OK) return cleanup(rc);
  }
  if (s->n > 0) {
    rc = cg_select_form(s);
    if (rc != B200LA_OK) return cleanup(rc);
  }
  *out = s;
  return B200LA_OK;
}

extern "C" {

int b200la_cg_destroy(b200la_cg s) {
  if (!s) return B200LA_OK;
  cudaStream_t st = s->ctx->stream;
  cudaStreamSynchronize(st);
  if (s->exec) cudaGraphExecDestroy(s->exec);
  if (s->graph) cudaGraphDestroy(s->graph);
  void *bufs[] = {s->x, s->r, s->p, s->Ap, s->invd, s->part, s->sc, s->zg, s->pg[0], s->pg[1], s->tag_slots};
  for (void *b : bufs)
    if (b) cudaFreeAsync(b, st);
  if (s->sc_host) cudaFreeHost(s->sc_host);
  delete s;
  return B200LA_OK;
}

int b200la_cg_solve(b200la_cg s, b200la_vec b, b200la_vec x, b200la_cg_result *res) {
  B_CHECK(s && b && x && res, B200LA_ERR_INVALID, "cg_solve: null argument");
  b200la_mat A = s->A;
  B_CHECK(b->n == s->n && x->n == s->n, B200LA_ERR_INVALID, "cg_solve: vector sizes %lld/%lld vs %lld",
          (long long)b->n, (long long)x->n, (long long)s->n);
  B_CHECK(b->dtype == s->vdtype && x->dtype == s->vdtype, B200LA_ERR_DTYPE, "cg_solve: dtype mismatch");
  memset(res, 0, sizeof(*res));
  if (s->n == 0) {
    res->state = B200LA_SUCCESS_ABS;
    return B200LA_OK;
  }
  cudaStream_t st = A->ctx->stream;
  B_TRY(cg_start(s, x->d, b->d));
  B_TRY(cg_run(s));
  B_CUDA(cudaMemcpyAsync(x->d, s->x, (size_t)s->n * dtype_size(s->vdtype), cudaMemcpyDeviceToDevice, st));
  CgScalars h;
  B_TRY(cg_fetch(s, &h));
  res->iters = h.iter;
  // the lmp cg() returns the 0-based index of the iteration that met its test
  if (s->prm.stop_rule == B200LA_STOP_LMP_CG && h.state == B200LA_SUCCESS_REL) res->iters = h.iter - 1;
  res->state = h.state;
  res->res = h.res;
  res->res_init = h.res_init;
  res->res_rel = h.res_init > 0.0 ? h.res / h.res_init : 0.0;
  if (h.state == B200LA_SUCCESS_ABS || h.state == B200LA_SUCCESS_REL)
    res->solver_state = B200LA_SOLVER_SUCCESS;
  else if (h.state == B200LA_FAIL_DIV || h.state == B200LA_FAIL_MAXITS)
    res->solver_state = B200LA_SOLVER_EXCEEDED;
  else
    res->solver_state = B200LA_SOLVER_ERROR;
  return B200LA_OK;
}

int b200la_pcg_solve(b200la_mat A, b200la_vec b, b200la_vec x, const b200la_cg_params *prm, b200la_cg_result *res) {
  b200la_cg s = nullptr;
  B_TRY(b200la_cg_create(A, prm, &s));
  int rc = b200la_cg_solve(s, b, x, res);
  b200la_cg_destroy(s);
  return rc;
}

}  // extern "C"
