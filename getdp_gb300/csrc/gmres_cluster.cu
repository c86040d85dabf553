// Batched GMRES / FGMRES with one thread-block cluster per system and the
// whole solve of every system in one launch.
//
// The systems of a batch (the diagonal blocks of one matrix, as in
// gmres_batch.cu) are independent, so nothing has to cross from one system
// to another while they iterate: a cluster of 1 to 16 CTAs (on as many SMs)
// takes a system from a queue (largest first), runs its restart cycles and
// Arnoldi steps to the end, and takes the next.  Within a cluster the rows
// are split between the CTAs; the steps that need rows of other CTAs (the
// ILU(0) sweeps level by level, the product with the preconditioned vector,
// the restart residual) follow a cluster barrier, and every sum (the
// Gram-Schmidt dot products, norms) is formed per CTA in a fixed order, left
// in the CTA's shared memory, and read by every CTA of the cluster through
// distributed shared memory in rank order, so that every CTA holds the same
// sums and runs the same scalar recurrences (Hessenberg column, Givens
// rotations, stopping tests) on its own copy: no launch per step, no
// grid-wide synchronisation, no host round trip.
//
// The iteration is the one of gmres_batch.cu and gmres.cu: right
// preconditioning, restart residual, classical Gram-Schmidt with the
// selective second pass (a second pass when the first removed more than
// 98 % of ||w||^2, mgsro's constant, iters.f:3475), Givens rotations
// (iters.f:3235-3273), Sparskit's stopping test on the rotated residual and
// its codes (iters.f:1912-2219 GMRES, :2522-2806 FGMRES).  The ILU(0)
// factor and its level schedule are the ones of gmres.cu, cut into the
// systems (ilu_sys_levels); a sweep's rows and arithmetic are those of
// lusol (ilut.F:2297-2347), in FP64 or with the FP32 factor.
//
// Cross-CTA data in global memory (vectors written by other CTAs of the
// cluster) is read through L2 (ld.global.cg) after a cluster barrier
// (barrier.cluster arrive.release / wait.acquire).  Every branch around a
// barrier depends only on values that all CTAs of the cluster hold alike,
// and every loop is bounded (restart cycles by the iteration cap, steps by
// the Krylov size, systems by the queue).
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "krylov.cuh"

namespace cg = cooperative_groups;

namespace gb {

// CTAs per cluster (one cluster per system): Batch_Kernel 1, 2, 4, 8 (the
// portable maximum) or 16 (a non-portable size this GPU allows); 512 threads
// each, two CTAs to an SM.  On 512 complex systems of 1,922..51,842 rows
// (ILU(0)-GMRES(40) in the multicolour order) four were the fastest: few CTAs
// leave the largest systems' steps to one or two SMs, many CTAs leave fewer
// systems running at once and make each cluster barrier dearer.  Fewer
// systems want larger clusters: the default, GB300_BATCH_AUTO, sizes them.  1024
// threads in one CTA per SM leave half as many clusters: 322 against 240 ms
// on 64 systems.
constexpr int kCMaxKrylov = 64;
// most levels of one system in either triangular sweep (one cluster
// barrier each); systems in GetDP's own order (~2n levels on an n x n grid)
// take the chunked batched solver
constexpr int kCMaxLevels = 64;

struct CState {
  double tol, res, res0, res6, scale, nrm0, rr;
  int its, status, active, cycle, first, k, did_cycle, breakdown, reorth;
};

struct CArgs {
  int nsys, m, maxit, flexible, precond;
  double rtol;
  const int *order, *off;
  int *queue;
  const int *rowptr, *col;
  const double *val, *rhs;
  double *x;
  const int *diag;
  const void *lu, *inv;
  const int *lrows, *urows, *llev, *ulev, *llb, *ulb;
  // multicolour order: system p's vertices of colour c are
  // [voff[p (ncol + 1) + c], voff[p (ncol + 1) + c + 1]), bs rows each
  // (ncol = 0: the level lists above)
  int ncol, bs;
  const int *voff;
  double *Vb, *Z, *zt, *u;
  float *t32;
  size_t ldv;
  int *out_status, *out_its;
  double *out_res, *out_rr, *out_bb;
};

// the sums over the cluster's CTAs, in rank order, of the nv partials each
// CTA left in buf: every CTA gets the same values in out
template <int CS, int NT>
__device__ __forceinline__ void cluster_sum(cg::cluster_group &cl, double *buf, int nv,
                                            double *out)
{
  cl.sync();
  for(int j = threadIdx.x; j < nv; j += NT) {
    // four chains over the ranks (an FP64 addition takes some 85 ns)
    double s[4] = {0., 0., 0., 0.};
#pragma unroll
    for(int r = 0; r < CS; r++) s[r & 3] += cl.map_shared_rank(buf, r)[j];
    out[j] = (s[0] + s[1]) + (s[2] + s[3]);
  }
  __syncthreads();
}

// s - sum_k a[k] x[col[k]] over k0 <= k < k1, in that order (lusol's
// accumulation order), with the column indices and values of four entries
// loaded before their gathers, so that a thread has four loads in flight
// instead of a chain of dependent ones
template <typename T, typename X>
__device__ __forceinline__ T row_acc(int k0, int k1, const int *__restrict__ col,
                                     const T *__restrict__ a, const X *x, T s)
{
  for(int kb = k0; kb < k1; kb += 4) {
    int c[4];
    T v[4];
    X xv[4];
#pragma unroll
    for(int u = 0; u < 4; u++) {
      int k = kb + u;
      c[u] = k < k1 ? col[k] : 0;
      v[u] = k < k1 ? a[k] : (T)0;
    }
#pragma unroll
    for(int u = 0; u < 4; u++)
      if(kb + u < k1) xv[u] = __ldcg(x + c[u]);
#pragma unroll
    for(int u = 0; u < 4; u++)
      if(kb + u < k1) s = s - v[u] * xv[u];
  }
  return s;
}

// the sum over the cluster's CTAs and their warps of the one partial per warp
// each CTA left in buf[0 .. NT / 32), in a fixed order (a tree over a CTA's
// warps, then one over the ranks: summing rank after rank cost 7 us on 16
// CTAs): every CTA gets the same value in out[0]
template <int CS, int NT>
__device__ __forceinline__ void cluster_sum_warps(cg::cluster_group &cl, double *buf,
                                                  double *out)
{
  __syncthreads();
  if(threadIdx.x < 32) {
    const double v = warp_sum(threadIdx.x < NT / 32 ? buf[threadIdx.x] : 0.);
    if(threadIdx.x == 0) buf[0] = v;
  }
  cl.sync();
  if(threadIdx.x < 32) {
    const double v = warp_sum(threadIdx.x < CS ? *cl.map_shared_rank(buf, threadIdx.x) : 0.);
    if(threadIdx.x == 0) out[0] = v;
  }
  __syncthreads();
}

// The three passes below run over some 2,000 rows per CTA from L2, so what
// paces them is how many loads a thread has in flight: each keeps 16 or more
// (with four, 64 systems of up to 50,562 rows took 243 ms instead of 230).

// w = A z on the rows [lo, hi), one thread per row, the next row's bounds
// loaded ahead; with RES, w = rhs - A z and the partial ||w||^2 (and
// ||rhs||^2 in bb)
template <int RES, int NT>
__device__ __noinline__ double c_spmv(const CArgs &P, int lo, int hi, const double *z,
                                         double *w, double *bb)
{
  constexpr int U = 8;
  double acc = 0., accb = 0.;
  int i = lo + threadIdx.x, k = 0, e = 0;
  if(i < hi) {
    k = P.rowptr[i];
    e = P.rowptr[i + 1];
  }
  while(i < hi) {
    const int in = i + NT;
    int kn = 0, en = 0;
    if(in < hi) {
      kn = P.rowptr[in];
      en = P.rowptr[in + 1];
    }
    double s = 0.;
    for(; k < e; k += U) {
      int c[U];
      double v[U], zv[U];
#pragma unroll
      for(int u = 0; u < U; u++) {
        c[u] = k + u < e ? P.col[k + u] : -1;
        v[u] = k + u < e ? P.val[k + u] : 0.;
      }
#pragma unroll
      for(int u = 0; u < U; u++) zv[u] = c[u] >= 0 ? __ldcg(z + c[u]) : 0.;
#pragma unroll
      for(int u = 0; u < U; u++)
        if(c[u] >= 0) s += v[u] * zv[u];
    }
    if(RES) {
      const double bi = P.rhs[i], ri = bi - s;
      if(w) w[i] = ri;
      acc += ri * ri;
      accb += bi * bi;
    }
    else
      w[i] = s;
    i = in;
    k = kn;
    e = en;
  }
  if(bb) *bb = accb;
  return acc;
}

// partial <V_j, w> over the rows [lo, hi) for j < kk, two columns per warp at
// a time (a fixed order per column), into buf[j]
template <int NT>
__device__ __noinline__ void c_dots(const CArgs &P, int lo, int hi, const double *w,
                                       int kk, double *buf)
{
  constexpr int U = 8, NW = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for(int j = warp; j < kk; j += 2 * NW) {
    const bool two = j + NW < kk;  // the same in the whole warp
    const double *va = P.Vb + (size_t)j * P.ldv;
    const double *vb = P.Vb + (size_t)(two ? j + NW : j) * P.ldv;
    double sa = 0., sb = 0.;
    for(int i = lo + lane; i < hi; i += 32 * U) {
      double a[U], b[U], x[U];
#pragma unroll
      for(int u = 0; u < U; u++) {
        const int r = i + 32 * u;
        x[u] = r < hi ? __ldcg(w + r) : 0.;
        a[u] = r < hi ? __ldcg(va + r) : 0.;
        b[u] = two && r < hi ? __ldcg(vb + r) : 0.;
      }
#pragma unroll
      for(int u = 0; u < U; u++) sa += a[u] * x[u];
      if(two)
#pragma unroll
        for(int u = 0; u < U; u++) sb += b[u] * x[u];
    }
    sa = warp_sum(sa);
    if(lane == 0) buf[j] = sa;
    if(two) {
      sb = warp_sum(sb);
      if(lane == 0) buf[j + NW] = sb;
    }
  }
}

// The previous rotations on column k (h, into Hc): they need the column only,
// so warp 0 runs them ahead of its share of the update, everything but their
// chain (one FMA each, some 85 ns) in parallel; k <= 64
__device__ __noinline__ void c_rotate(const double *h, const double *cs, const double *sn,
                                         int k, double *ra, double *Hc)
{
  const int lane = threadIdx.x;  // warp 0
  double t[2], q[2];
#pragma unroll
  for(int u = 0; u < 2; u++) {
    const int j = lane + 32 * u;
    const double b = j < k - 1 ? h[j + 1] : 0.;
    t[u] = j < k - 1 ? cs[j] * b : 0.;
    q[u] = j < k - 1 ? sn[j] * b : 0.;
    if(j < k - 1) ra[j] = t[u];
  }
  __syncwarp();
  if(lane == 0) {
    double a = h[0];
#pragma unroll 4
    for(int i = 0; i < k - 1; i++) {
      const double ti = ra[i];
      ra[i] = a;
      a = fma(-sn[i], a, ti);
    }
    ra[k - 1] = a;
  }
  __syncwarp();
#pragma unroll
  for(int u = 0; u < 2; u++) {
    const int j = lane + 32 * u;
    if(j < k) Hc[j] = j < k - 1 ? fma(cs[j], ra[j], q[u]) : ra[j];
  }
}

// w -= sum_{j<k} h_j V_j on the rows [lo, hi); the partial ||w||^2
template <int NT>
__device__ __noinline__ double c_update(const CArgs &P, int lo, int hi, double *w,
                                           const double *h, int k)
{
  // two rows at a time, one FMA chain each, k + 1 FP64 instructions per row
  // (they pace the kernel once the loads do not)
  constexpr int U = 8;
  double v = 0.;
  for(int i = lo + threadIdx.x; i < hi; i += 2 * NT) {
    const bool two = i + NT < hi;
    const double *va = P.Vb + i, *vb = va + (two ? NT : 0);
    double s0 = __ldcg(w + i), s1 = two ? __ldcg(w + i + NT) : 0.;
    for(int j = 0; j < k; j += U) {
      double a[U], b[U];
#pragma unroll
      for(int u = 0; u < U; u++) {
        a[u] = j + u < k ? __ldcg(va + (size_t)(j + u) * P.ldv) : 0.;
        b[u] = two && j + u < k ? __ldcg(vb + (size_t)(j + u) * P.ldv) : 0.;
      }
#pragma unroll
      for(int u = 0; u < U; u++)
        if(j + u < k) {
          s0 = fma(-h[j + u], a[u], s0);
          if(two) s1 = fma(-h[j + u], b[u], s1);
        }
    }
    w[i] = s0;
    v = fma(s0, s0, v);
    if(two) {
      w[i + NT] = s1;
      v = fma(s1, s1, v);
    }
  }
  return v;
}

// One row's strictly lower or upper entries: the first kAhead columns and
// values in registers, loaded before a cluster barrier so that only the
// gathers of x follow it, the rest read when they are needed
constexpr int kAhead = 4;
template <typename T> struct RowAhead {
  int k0, k1, c[kAhead];
  T v[kAhead];
  __device__ __forceinline__ void load(int a, int b, const int *__restrict__ col,
                                       const T *__restrict__ lu)
  {
    k0 = a;
    k1 = b;
#pragma unroll
    for(int u = 0; u < kAhead; u++) {
      c[u] = a + u < b ? col[a + u] : -1;
      v[u] = a + u < b ? lu[a + u] : (T)0;
    }
  }
  template <typename X> __device__ __forceinline__ void gather(const X *x, X (&xv)[kAhead]) const
  {
#pragma unroll
    for(int u = 0; u < kAhead; u++) xv[u] = c[u] >= 0 ? __ldcg(x + c[u]) : (X)0;
  }
  // s - sum over the entries, in their order
  template <typename X>
  __device__ __forceinline__ T apply(const int *__restrict__ col, const T *__restrict__ lu,
                                     const X *x, const X (&xv)[kAhead], T s) const
  {
#pragma unroll
    for(int u = 0; u < kAhead; u++)
      if(c[u] >= 0) s = s - v[u] * xv[u];
    return k0 + kAhead < k1 ? row_acc(k0 + kAhead, k1, col, lu, x, s) : s;
  }
};

// dst = M^-1 src colour by colour (the multicolour order): a colour's vertices
// share no entry, so its rows are independent but for the two real rows of a
// complex unknown (bs = 2), which sit in adjacent lanes and exchange their
// values by shuffles, the coupling entry l (row 2v + 1 on 2v) forward and u
// (2v on 2v + 1) backward.  The last colour's rows have no other upper
// entries, so both sweeps finish them at once: one barrier per colour and
// sweep but one.  A thread's first row of the next colour is loaded between
// the barrier's arrive and its wait: a colour costs a gather, a short FMA
// chain and the barrier (with the row's structure read after the barrier and
// a vertex's rows one after the other, 5 us a colour on 16 CTAs).
// src must be complete but for a cluster barrier; dst is complete on return.
template <typename T, int CS, int NT>
__device__ __noinline__ void c_colour_sweeps(const CArgs &P, cg::cluster_group &cl, int p, int rank,
                                const double *src, double *dst)
{
  const T *__restrict__ lu = (const T *)P.lu, *__restrict__ inv = (const T *)P.inv;
  const int *__restrict__ col = P.col;
  T *x = sizeof(T) == 8 ? (T *)dst : (T *)P.t32;
  const int *vo = P.voff + (size_t)p * (P.ncol + 1);
  const int bs = P.bs, C = P.ncol;
  const bool odd = bs == 2 && (threadIdx.x & 1), even = bs == 2 && !(threadIdx.x & 1);
  RowAhead<T> R;
  T cpl = (T)0, iv = (T)0;  // coupling entry with the partner row, pivot inverse
  int m0 = 0, m1 = 0;       // the entries' bounds, one colour further ahead
  auto bounds = [&](int c, int &r0, int &r1) {
    const int a = vo[c], cnt = vo[c + 1] - a;
    r0 = (a + (int)((long long)cnt * rank / CS)) * bs;
    r1 = (a + (int)((long long)cnt * (rank + 1) / CS)) * bs;
  };
  // bounds of row i's strictly lower or upper entries
  auto meta = [&](bool up, int i, bool in) {
    m0 = !in ? 0 : up ? P.diag[i] + 1 : P.rowptr[i];
    m1 = !in ? 0 : up ? P.rowptr[i + 1] : P.diag[i];
  };
  auto meta_first = [&](bool up, int c) {
    int r0, r1;
    bounds(c, r0, r1);
    meta(up, r0 + threadIdx.x, r0 + (int)threadIdx.x < r1);
  };
  // the entries within the bounds, the partner's taken out: the last of row
  // 2v + 1's lower ones, the first of row 2v's upper ones
  auto load = [&](bool up, int i, bool in) {
    cpl = (T)0;
    iv = up && in ? inv[i] : (T)0;
    if(up && even && m0 < m1 && col[m0] == i + 1) cpl = lu[m0++];
    if(!up && odd && m0 < m1 && col[m1 - 1] == i - 1) cpl = lu[--m1];
    R.load(m0, m1, col, lu);
  };
  auto put = [&](int i, T v, bool last) {
    x[i] = v;
    if(sizeof(T) == 4 && last) dst[i] = (double)v;
  };
  // v: this row's backward value before its partner's part and the pivot
  auto pivot = [&](T v, T u, T ivv) {
    const T w = ivv * v;
    const T wo = __shfl_down_sync(0xffffffffu, w, 1);
    return even ? ivv * (v - u * wo) : w;
  };
  cl.barrier_arrive();
  meta_first(false, 0);
  for(int c = 0; c < C; c++) {
    int r0, r1;
    bounds(c, r0, r1);
    int i = r0 + threadIdx.x;
    load(false, i, i < r1);
    if(c < C - 1)
      meta_first(false, c + 1);
    else if(C > 1)
      meta_first(true, C - 2);
    const int n0 = m0, n1 = m1;  // the next colour's
    cl.barrier_wait();
    for(int base = r0; base < r1; base += NT) {  // the same in every thread
      i = base + threadIdx.x;
      const bool in = i < r1;
      if(base > r0) {
        meta(false, i, in);
        load(false, i, in);
      }
      T s = in ? (T)__ldcg(src + i) : (T)0;
      T xv[kAhead];
      R.gather((const T *)x, xv);
      s = R.apply(col, lu, (const T *)x, xv, s);
      const T se = __shfl_up_sync(0xffffffffu, s, 1);
      if(odd) s = s - cpl * se;
      if(c == C - 1) {
        T u = (T)0, ivv = in ? inv[i] : (T)0;
        if(even && in) {
          const int k = P.diag[i] + 1;
          if(k < P.rowptr[i + 1] && col[k] == i + 1) u = lu[k];
        }
        s = pivot(s, u, ivv);
      }
      if(in) put(i, s, c == C - 1);
    }
    cl.barrier_arrive();
    m0 = n0;
    m1 = n1;
  }
  for(int c = C - 2; c >= 0; c--) {
    int r0, r1;
    bounds(c, r0, r1);
    int i = r0 + threadIdx.x;
    load(true, i, i < r1);
    if(c > 0) meta_first(true, c - 1);
    const int n0 = m0, n1 = m1;
    cl.barrier_wait();
    for(int base = r0; base < r1; base += NT) {
      i = base + threadIdx.x;
      const bool in = i < r1;
      if(base > r0) {
        meta(true, i, in);
        load(true, i, in);
      }
      T s = in ? __ldcg(x + i) : (T)0;
      T xv[kAhead];
      R.gather((const T *)x, xv);
      if(sizeof(T) == 8) {
        s = R.apply(col, lu, (const T *)x, xv, s);
        s = pivot(s, cpl, iv);
      }
      else {
        // FP32 sums in lusol's order, in which the partner comes first (the
        // FP64 ones put it last: no second FMA chain after the partner's)
        T w = (T)0;
        if(!even) w = iv * R.apply(col, lu, (const T *)x, xv, s);
        const T wo = __shfl_down_sync(0xffffffffu, w, 1);
        s = even ? iv * R.apply(col, lu, (const T *)x, xv, s - cpl * wo) : w;
      }
      if(in) put(i, s, true);
    }
    cl.barrier_arrive();
    m0 = n0;
    m1 = n1;
  }
  cl.barrier_wait();
}

// dst = M^-1 src for system p: the ILU(0) sweeps level by level, each
// level's rows split over the cluster (a barrier after each level), or a
// copy without a preconditioner.  src must be complete (all CTAs) on entry;
// dst is complete on return.
template <typename T, int CS, int NT>
__device__ __noinline__ void c_precond(const CArgs &P, cg::cluster_group &cl, int p, int rank, int lo,
                          int hi, const double *src, double *dst)
{
  if(!P.precond) {
    for(int i = lo + threadIdx.x; i < hi; i += NT) dst[i] = __ldcg(src + i);
    cl.sync();
    return;
  }
  const T *lu = (const T *)P.lu, *inv = (const T *)P.inv;
  if(P.ncol > 0) {
    c_colour_sweeps<T, CS, NT>(P, cl, p, rank, src, dst);
    return;
  }
  cl.sync();  // src written by every CTA
  for(int l = P.llb[p]; l + 1 < P.llb[p + 1]; l++) {
    const int a = P.llev[l], cnt = P.llev[l + 1] - a;
    const int t0 = a + (int)((long long)cnt * rank / CS);
    const int t1 = a + (int)((long long)cnt * (rank + 1) / CS);
    for(int t = t0 + threadIdx.x; t < t1; t += NT) {
      const int i = P.lrows[t];
      const int ke = P.diag[i];
      if constexpr(sizeof(T) == 8)
        dst[i] = row_acc(P.rowptr[i], ke, P.col, lu, (const double *)dst,
                                  __ldcg(src + i));
      else
        P.t32[i] = row_acc(P.rowptr[i], ke, P.col, lu, (const float *)P.t32,
                                    (float)__ldcg(src + i));
    }
    cl.sync();
  }
  for(int l = P.ulb[p]; l + 1 < P.ulb[p + 1]; l++) {
    const int a = P.ulev[l], cnt = P.ulev[l + 1] - a;
    const int t0 = a + (int)((long long)cnt * rank / CS);
    const int t1 = a + (int)((long long)cnt * (rank + 1) / CS);
    for(int t = t0 + threadIdx.x; t < t1; t += NT) {
      const int i = P.urows[t];
      const int ke = P.rowptr[i + 1];
      if constexpr(sizeof(T) == 8) {
        double s = row_acc(P.diag[i] + 1, ke, P.col, lu, (const double *)dst,
                                    __ldcg(dst + i));
        dst[i] = inv[i] * s;
      }
      else {
        float s = row_acc(P.diag[i] + 1, ke, P.col, lu, (const float *)P.t32,
                                   __ldcg(P.t32 + i));
        float v = inv[i] * s;
        P.t32[i] = v;
        dst[i] = (double)v;
      }
    }
    cl.sync();
  }
}

template <typename T, int CS, int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_c_solve(CArgs P)
{
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int tid = threadIdx.x;
  const int m = P.m;
  __shared__ double sH[(kCMaxKrylov + 1) * kCMaxKrylov];  // column-major, ld m + 1
  __shared__ double scs[kCMaxKrylov], ssn[kCMaxKrylov], sy[kCMaxKrylov];
  __shared__ double sg[kCMaxKrylov + 1], sh1[kCMaxKrylov + 1], sdot[kCMaxKrylov + 1];
  __shared__ double sra[kCMaxKrylov];
  __shared__ double xbuf[2][kCMaxKrylov + 2];  // partials read by the other CTAs
  __shared__ CState S;
  __shared__ int s_q;
  int xb = 0;

  for(int guard = 0; guard <= P.nsys; guard++) {
    if(rank == 0 && tid == 0) s_q = atomicAdd(P.queue, 1);
    cl.sync();
    const int q = *cl.map_shared_rank(&s_q, 0);
    cl.sync();  // every CTA has read the ticket before rank 0 takes the next
    if(q >= P.nsys) break;
    const int p = P.order[q];
    const int r0 = P.off[p], np = P.off[p + 1] - r0;
    const int lo = r0 + (int)((long long)np * rank / CS);
    const int hi = r0 + (int)((long long)np * (rank + 1) / CS);
    if(tid == 0) {
      memset(&S, 0, sizeof(S));
      S.active = 1;
      S.first = 1;
      S.status = 1;
    }
    __syncthreads();

    for(int cyc = 0; S.active && cyc <= P.maxit + 1; cyc++) {
      // restart: r = b - A x into V_0, ||r||
      cl.sync();  // x complete
      {
        double rr = warp_sum(c_spmv<1, NT>(P, lo, hi, P.x, P.Vb, nullptr));
        if((tid & 31) == 0) xbuf[xb][tid >> 5] = rr;
        cluster_sum_warps<CS, NT>(cl, xbuf[xb], sdot);
        xb ^= 1;
      }
      if(tid == 0) {
        S.its += 1;
        double alpha = sqrt(sdot[0]);
        if(S.first) {
          S.tol = P.rtol * alpha + 0.0;
          S.res0 = alpha;
          S.first = 0;
        }
        S.res = alpha;
        sg[0] = alpha;
        S.k = 0;
        S.did_cycle = 0;
        S.breakdown = 0;
        if(alpha <= S.tol) {
          S.status = 0;
          S.res6 = alpha;
          S.active = 0;
          S.cycle = 0;
        }
        else {
          S.scale = 1. / alpha;
          S.cycle = 1;
        }
      }
      __syncthreads();
      if(!S.cycle) break;  // converged at the restart
      for(int i = lo + tid; i < hi; i += NT) P.Vb[i] = S.scale * P.Vb[i];

      for(int k = 1; k <= m && S.cycle; k++) {
        double *vk = P.Vb + (size_t)(k - 1) * P.ldv;
        double *w = P.Vb + (size_t)k * P.ldv;
        double *z = P.flexible ? P.Z + (size_t)(k - 1) * P.ldv : P.zt;
        c_precond<T, CS, NT>(P, cl, p, rank, lo, hi, vk, z);
        c_spmv<0, NT>(P, lo, hi, z, w, nullptr);
        __syncthreads();
        // first Gram-Schmidt pass: <V_j, w> for j < k and <w, w>
        c_dots<NT>(P, lo, hi, w, k + 1, xbuf[xb]);
        cluster_sum<CS, NT>(cl, xbuf[xb], k + 1, sdot);
        xb ^= 1;
        if(tid == 0) {
          S.nrm0 = sdot[k];
          if(!(S.nrm0 > 0. && 1. / S.nrm0 > 0.)) {
            // mgsro's zero (-1) or abnormal (-2) norm: the cycle ends as a
            // break-down, the step's column unused
            S.breakdown = (S.nrm0 <= 0.) ? -1 : -2;
            S.its += 1;
            S.cycle = 0;
            S.reorth = 0;
          }
        }
        if(tid < k) sh1[tid] = sdot[tid];
        __syncthreads();
        if(!S.cycle) break;
        double *Hc = sH + (size_t)(k - 1) * (m + 1);
        if(tid < 32) c_rotate(sh1, scs, ssn, k, sra, Hc);
        {
          double v = warp_sum(c_update<NT>(P, lo, hi, w, sh1, k));
          if((tid & 31) == 0) xbuf[xb][tid >> 5] = v;
          cluster_sum_warps<CS, NT>(cl, xbuf[xb], sdot);
          xb ^= 1;
        }
        if(tid == 0) {
          S.rr = sdot[0];
          S.reorth = !(S.rr >= 0.02 * S.nrm0);
        }
        __syncthreads();
        if(S.reorth) {
          // second pass
          c_dots<NT>(P, lo, hi, w, k, xbuf[xb]);
          cluster_sum<CS, NT>(cl, xbuf[xb], k, sdot);
          xb ^= 1;
          if(tid < k) sh1[tid] += sdot[tid];
          __syncthreads();
          if(tid < 32) c_rotate(sh1, scs, ssn, k, sra, Hc);
          double v = warp_sum(c_update<NT>(P, lo, hi, w, sdot, k));
          if((tid & 31) == 0) xbuf[xb][tid >> 5] = v;
          cluster_sum_warps<CS, NT>(cl, xbuf[xb], sdot);
          xb ^= 1;
          if(tid == 0) S.rr = sdot[0];
          __syncthreads();
        }
        // end of the Arnoldi step: h(k+1,k), rotations, stopping test
        if(tid == 0) {
          S.its += 1;
          S.k = k;
          S.did_cycle = 1;
          if(!(S.rr > 0.)) {
            // the column without rotations, as the reference leaves it
            for(int j = 0; j < k; j++) Hc[j] = sh1[j];
            Hc[k] = sqrt(S.rr);
            S.breakdown = -3;
            S.cycle = 0;
          }
          else {
            const double rr = S.rr, hk = Hc[k - 1], r2 = fma(hk, hk, rr);
            double c, s;
            if(rr > 1e-280 && r2 < 1e280) {
              // the rotation by two independent reciprocal roots (as
              // k_gm_update: a third of the serial chain of givens)
              const double ri = rsqrt(rr), q = rsqrt(r2);
              S.scale = ri;
              c = hk * q;
              s = rr * ri * q;
              Hc[k - 1] = r2 * q;
            }
            else {
              double x = hk, y = sqrt(rr);
              S.scale = 1. / y;
              givens_dev(&x, &y, &c, &s);
              Hc[k - 1] = x;
            }
            scs[k - 1] = c;
            ssn[k - 1] = s;
            double alpha = -s * sg[k - 1];
            sg[k - 1] = c * sg[k - 1];
            sg[k] = alpha;
            alpha = fabs(alpha);
            S.res = alpha;
            if(!(k < m && !(alpha <= S.tol) && (P.maxit <= 0 || S.its < P.maxit)))
              S.cycle = 0;
          }
        }
        __syncthreads();
        if(S.cycle)
          for(int i = lo + tid; i < hi; i += NT) w[i] = S.scale * w[i];
      }

      // end of the cycle: H y = g (upper triangular), then the update.
      // Thread 0 changes S below: every thread takes what it branches on
      // first, and a barrier separates the two (a thread that read S after
      // the change would leave the cluster barriers of the others)
      const int dc = S.did_cycle;
      __syncthreads();
      if(dc) {
        if(tid == 0) {
          int k = S.k;
          while(k > 0 && sH[(k - 1) * (m + 1) + k - 1] == 0.) k--;
          if(k == 0) {
            S.status = -3;
            S.breakdown = -4;
            S.active = 0;
            S.did_cycle = 0;
          }
          else {
            S.k = k;
            for(int i = k - 1; i >= 0; i--) {
              double t = sg[i];
              for(int j = i + 1; j < k; j++) t -= sH[j * (m + 1) + i] * sy[j];
              sy[i] = t / sH[i * (m + 1) + i];
            }
          }
        }
        __syncthreads();
      }
      const int upd = S.active && S.did_cycle;
      __syncthreads();
      if(upd) {
        const int k = S.k;
        if(P.flexible) {
          for(int i = lo + tid; i < hi; i += NT) {
            double s = P.x[i];
            for(int j = 0; j < k; j++) s += sy[j] * __ldcg(P.Z + (size_t)j * P.ldv + i);
            P.x[i] = s;
          }
        }
        else {
          for(int i = lo + tid; i < hi; i += NT) {
            double s = 0.;
            for(int j = 0; j < k; j++) s += sy[j] * __ldcg(P.Vb + (size_t)j * P.ldv + i);
            P.u[i] = s;
          }
          c_precond<T, CS, NT>(P, cl, p, rank, lo, hi, P.u, P.zt);
          for(int i = lo + tid; i < hi; i += NT) P.x[i] += __ldcg(P.zt + i);
        }
      }
      __syncthreads();
      // the restart decision
      if(tid == 0 && S.active) {
        S.res6 = S.res;
        if(S.breakdown != 0) {
          S.status = -3;
          S.active = 0;
        }
        else {
          bool more = (S.its < P.maxit || P.maxit <= 0) && (S.res6 > S.tol);
          if(!more) {
            if(S.res6 <= S.tol)
              S.status = 0;
            else if(S.its >= P.maxit && P.maxit > 0)
              S.status = -1;
            else
              S.status = -10;
            S.active = 0;
          }
        }
      }
      __syncthreads();
    }

    // the system's true residual ||b - A x|| and ||b||
    cl.sync();
    {
      double bb = 0.;
      double rr = c_spmv<1, NT>(P, lo, hi, P.x, nullptr, &bb);
      rr = block_sum<double, NT>(rr);
      bb = block_sum<double, NT>(bb);
      if(tid == 0) {
        xbuf[xb][0] = rr;
        xbuf[xb][1] = bb;
      }
      cluster_sum<CS, NT>(cl, xbuf[xb], 2, sdot);
      xb ^= 1;
    }
    if(rank == 0 && tid == 0) {
      P.out_status[p] = S.active ? -1 : S.status;
      P.out_its[p] = S.its;
      P.out_res[p] = S.res6;
      P.out_rr[p] = sdot[0];
      P.out_bb[p] = sdot[1];
    }
    __syncthreads();
  }
}

template <typename T, int CS, int NT = 512>
static int launch_c(const CArgs &a, cudaStream_t st, int *nclusters)
{
  if(CS > 8 &&
     cudaFuncSetAttribute(k_c_solve<T, CS, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                          1) != cudaSuccess) {
    cudaGetLastError();
    *nclusters = 0;
    return GB300_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(NT, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.attrs = attr;
  // A cluster lies within a GPC, and the GPCs have fewer SMs here and there:
  // the policy that may place a cluster's CTAs unevenly keeps 15 clusters of
  // 16 CTAs resident instead of 14, 38 of 8 instead of 37 (as many of the
  // smaller ones).  64 systems of 1,922..50,562 rows on clusters of 16, twelve
  // draws of their values: 243 -> 231 ms on average, none slower.  (Clusters
  // of 12, of which 23 are resident: 232 on average, but 311 against 272 where
  // a system of many steps starts late.)
  attr[1].id = cudaLaunchAttributeClusterSchedulingPolicyPreference;
  attr[1].val.clusterSchedulingPolicyPreference = cudaClusterSchedulingPolicyLoadBalancing;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3(CS, 1, 1);
  int nc = 0;
  cudaError_t e = cudaOccupancyMaxActiveClusters(&nc, (void *)k_c_solve<T, CS, NT>, &cfg);
  if(e != cudaSuccess || nc < 1) {
    cudaGetLastError();
    *nclusters = 0;
    return GB300_OK;
  }
  if(nc > a.nsys) nc = a.nsys;
  *nclusters = nc;
  cfg.gridDim = dim3((unsigned)(nc * CS), 1, 1);
  if(cudaLaunchKernelEx(&cfg, k_c_solve<T, CS, NT>, a) != cudaSuccess) {
    // a launch the device refuses (nothing ran): the per-kernel form runs
    cudaGetLastError();
    *nclusters = 0;
  }
  return GB300_OK;
}

int gmres_solve_batch_cluster(gb300_matrix *A, const double *val, const double *rhs,
                              double *x, const gb300_solver_params *p, int nsys,
                              const int *off, gb300_solve_info *infos, Work &W,
                              bool *used, const Colouring *mc)
{
  *used = false;
  const bool sized = p->batch_kernel == GB300_BATCH_AUTO;  // here, by the batch
  int cs = sized ? 4 : p->batch_kernel;
  if(cs != 1 && cs != 2 && cs != 4 && cs != 8 && cs != 16) return GB300_OK;
  if((p->algorithm != 8 && p->algorithm != 9) ||
     (p->preconditioner != 0 && p->preconditioner != 6))
    return GB300_OK;
  const int m = p->krylov_size <= 1 ? 15 : p->krylov_size;
  // the restart cycles are bounded by the iteration cap inside the kernel
  // (Precision 2, the FP32 factor with FP64 sweeps, takes the per-kernel form)
  if(m > kCMaxKrylov || p->nb_iter_max <= 0 || p->nb_iter_max > 100000000 || nsys < 1 ||
     p->precision == 2)
    return GB300_OK;
  if(sized) {
    // larger clusters where a few systems would leave SMs idle,
    // while the largest system has a row per thread of its cluster.
    // Measured (ms, 4 / 8 / 16 CTAs): 64 systems of 1,922..50,562 rows 466 /
    // 231 / 230; 12 of 1,058..28,322 154 / 77 / 48; 32 of 450..6,962 20.4 /
    // 13.3 / 17.8; 200 of 1,922..19,602 124 / 130 / 213
    int most = 0;
    for(int q = 0; q < nsys; q++) most = std::max(most, off[q + 1] - off[q]);
    while(cs < 16 && (long long)nsys * cs < 768 && most / (2 * cs) >= 512) cs *= 2;
  }
  int dev = 0, can = 0;
  GB_CUDA(cudaGetDevice(&dev));
  if(cudaDeviceGetAttribute(&can, cudaDevAttrClusterLaunch, dev) != cudaSuccess || !can) {
    cudaGetLastError();
    return GB300_OK;
  }
  cudaStream_t st = A->ctx->stream;
  const int n = A->n;
  const bool precond = (p->preconditioner == 6);
  const bool fp32 = (p->precision != 0);
  const SysLevels *SL = nullptr;
  // the multicolour order's colour ranges, when A is its permuted copy and
  // they describe the same systems; else the level lists of the schedule
  const bool by_colour = precond && mc && mc->B == A &&
                         (int)mc->seg.size() == nsys + 1 &&
                         std::equal(off, off + nsys + 1, mc->seg.begin()) &&
                         (int)mc->voff.size() == nsys * (mc->ncolors + 1);
  DevBuf<int> dvoff;
  if(precond) {
    if(by_colour) {
      if(mc->ncolors > kCMaxLevels) return GB300_OK;
      GB_TRY(dvoff.alloc(mc->voff.size()));
      GB_CUDA(cudaMemcpyAsync(dvoff.p, mc->voff.data(), sizeof(int) * mc->voff.size(),
                              cudaMemcpyHostToDevice, st));
    }
    else {
      GB_TRY(ilu_sys_levels(A, nsys, off, &SL));
      if(SL->max_levels > kCMaxLevels) return GB300_OK;
    }
    int zr = 0;
    GB_TRY(ilu_factor(A, val, fp32, &zr));
    if(zr) {
      set_error("Zero pivot on line %d in ILU", zr);
      return GB300_ERR_ZERO_PIVOT;
    }
  }
  // the queue: systems by decreasing size (ties by index)
  std::vector<int> order(nsys);
  for(int q = 0; q < nsys; q++) order[q] = q;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return off[a + 1] - off[a] > off[b + 1] - off[b];
  });
  DevBuf<int> dorder, doff, ints;
  DevBuf<double> dbl;
  GB_TRY(dorder.alloc(nsys));
  GB_TRY(doff.alloc(nsys + 1));
  GB_TRY(ints.alloc(2 * (size_t)nsys + 1));
  GB_TRY(dbl.alloc(3 * (size_t)nsys));
  GB_CUDA(cudaMemcpyAsync(dorder.p, order.data(), sizeof(int) * nsys, cudaMemcpyHostToDevice, st));
  GB_CUDA(cudaMemcpyAsync(doff.p, off, sizeof(int) * (nsys + 1), cudaMemcpyHostToDevice, st));
  GB_CUDA(cudaMemsetAsync(ints.p, 0, sizeof(int) * ints.n, st));
  GB_CUDA(cudaMemsetAsync(dbl.p, 0, sizeof(double) * dbl.n, st));

  const bool flexible = (p->algorithm == 9);
  size_t ldv = (size_t)n;
  double *Vb = (double *)W.vec(0, sizeof(double) * ldv * (m + 1));
  double *Z = flexible ? (double *)W.vec(1, sizeof(double) * ldv * m) : nullptr;
  double *zt = (double *)W.vec(4, sizeof(double) * (n > 0 ? n : 1));
  double *u = (double *)W.vec(3, sizeof(double) * (n > 0 ? n : 1));
  float *t32 = fp32 ? (float *)W.vec(5, sizeof(float) * (n > 0 ? n : 1)) : nullptr;
  if(!Vb || (flexible && !Z) || !zt || !u || (fp32 && !t32)) return GB300_ERR_CUDA;
  GB_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * n, st));

  CArgs a = {};
  a.nsys = nsys;
  a.m = m;
  a.maxit = p->nb_iter_max;
  a.flexible = flexible;
  a.precond = precond;
  a.rtol = p->stopping_test;
  a.order = dorder.p;
  a.off = doff.p;
  a.queue = ints.p + 2 * nsys;
  a.rowptr = A->rowptr.p;
  a.col = A->col.p;
  a.val = val;
  a.rhs = rhs;
  a.x = x;
  if(precond) {
    ilu_factor_arrays(A, fp32, &a.lu, &a.inv, &a.diag);
    if(by_colour) {
      a.ncol = mc->ncolors;
      a.bs = mc->bs;
      a.voff = dvoff.p;
    }
    else {
      a.lrows = SL->lrows.p;
      a.urows = SL->urows.p;
      a.llev = SL->llev.p;
      a.ulev = SL->ulev.p;
      a.llb = SL->llb.p;
      a.ulb = SL->ulb.p;
    }
  }
  a.Vb = Vb;
  a.Z = Z;
  a.zt = zt;
  a.u = u;
  a.t32 = t32;
  a.ldv = ldv;
  a.out_status = ints.p;
  a.out_its = ints.p + nsys;
  a.out_res = dbl.p;
  a.out_rr = dbl.p + nsys;
  a.out_bb = dbl.p + 2 * (size_t)nsys;
  int nc = 0;
  const bool f32 = precond && fp32;
#define GB_LAUNCH_C(CSZ)                                                              \
  GB_TRY(f32 ? launch_c<float, CSZ>(a, st, &nc) : launch_c<double, CSZ>(a, st, &nc))
  for(;; cs /= 2) {
    switch(cs) {
    case 1: GB_LAUNCH_C(1); break;
    case 2: GB_LAUNCH_C(2); break;
    case 4: GB_LAUNCH_C(4); break;
    case 8: GB_LAUNCH_C(8); break;
    default: GB_LAUNCH_C(16); break;
    }
    // no cluster fits or the launch was refused: nothing ran, and of the sizes
    // chosen here the next smaller one may do (16 is not portable)
    if(nc > 0 || !sized || cs <= 4) break;
  }
#undef GB_LAUNCH_C
  // none (x was zeroed, as the per-kernel form does first): that form solves
  if(nc < 1) return GB300_OK;
  std::vector<int> hst(nsys), hits(nsys);
  std::vector<double> hres(nsys), hrr(nsys), hbb(nsys);
  GB_CUDA(cudaMemcpyAsync(hst.data(), a.out_status, sizeof(int) * nsys, cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaMemcpyAsync(hits.data(), a.out_its, sizeof(int) * nsys, cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaMemcpyAsync(hres.data(), a.out_res, sizeof(double) * nsys, cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaMemcpyAsync(hrr.data(), a.out_rr, sizeof(double) * nsys, cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaMemcpyAsync(hbb.data(), a.out_bb, sizeof(double) * nsys, cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  GB_CUDA(cudaGetLastError());
  for(int q = 0; q < nsys; q++) {
    gb300_solve_info &f = infos[q];
    memset(&f, 0, sizeof(f));
    f.status = hst[q];
    f.iterations = hits[q];
    f.residual_estimate = hres[q];
    f.true_residual = sqrt(hrr[q]);
    f.rhs_norm = sqrt(hbb[q]);
    f.ilu_factorized = precond ? 1 : 0;
    f.batch_form = 1;
  }
  *used = true;
  return GB300_OK;
}

}  // namespace gb
