// Two-level preconditioning on aggregates (Preconditioners 21 and 22; no
// counterpart in Sparskit, whose preconditioners are one-level).
//
// The unknowns are grouped into aggregates (gb300_matrix_set_aggregates:
// one aggregate number per row, given by the caller; geometric cells of the
// mesh, for instance).  P0 is the piecewise-constant prolongation (row i has
// a single 1 in column agg[i]); the coarse matrix Ac = P0^T A P0 sums A's
// entries by (aggregate of the row, aggregate of the column) and is inverted
// densely on the device.  One application of the preconditioner is the
// symmetric two-level cycle
//
//   z  = S v                          ILU(0) smoothing (+ the learned correction)
//   z += P0 Ac^-1 P0^T (v - A z)      exact coarse correction
//   z += S (v - A z)                  second smoothing
//
// ILU(0) alone removes the oscillating part of the error and leaves the
// smooth part, which costs one-level preconditioned Krylov methods a number
// of steps that grows with the mesh size; the coarse correction removes the
// smooth part on the aggregates.
//
// Everything here is deterministic:
//   * Ac is summed in 64-bit fixed point (integer atomic adds are exact and
//     associative), with a power-of-two quantum chosen from max|a_ij| and
//     the largest number of entries one coarse entry can receive, so that
//     no sum can overflow; each term is rounded once, by at most half a
//     quantum, 2^(h-62) of max|a_ij| with h - 1 the bits of the largest
//     number of entries one coarse entry receives (2^-51 for 1,000);
//   * the dense inverse is a blocked symmetric elimination without pivoting,
//     two launches per 32 pivots (Ac is symmetric positive definite when A is
//     and no aggregate is empty; a pivot <= 0 is reported as an error).  An Ac
//     that is not symmetric is found on the device and inverted by Gauss-Jordan
//     steps, one launch per pivot;
//   * restriction and the coarse product are warp sums in a fixed order.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "krylov.cuh"
#include "sparse.cuh"

namespace gb {

constexpr int kSwB = 32;  // block of the coarse inverse's elimination (below)

void coarse_free(Coarse *c) { delete c; }

void coarse_values_changed(gb300_matrix *A)
{
  if(A->coarse) A->coarse->ready = false;
}

bool coarse_valid(const gb300_matrix *A)
{
  return A->coarse && A->coarse->version == A->pattern_version && A->coarse->nc > 0 &&
         A->nnz > 0;
}

int coarse_set(gb300_matrix *A, const int *agg, int nc)
{
  const int n = A->n;
  if(nc < 1 || nc > kMaxCoarse) {
    set_error("aggregates: %d aggregates (1 to %d supported)", nc, kMaxCoarse);
    return GB300_ERR_ARG;
  }
  if(!A->csr_valid || A->nnz <= 0) {
    set_error("aggregates: the matrix has no assembled pattern");
    return GB300_ERR_ARG;
  }
  std::vector<int> cnt(nc + 1, 0);
  for(int i = 0; i < n; i++) {
    if(agg[i] < 0 || agg[i] >= nc) {
      set_error("aggregates: row %d has aggregate %d, outside 0..%d", i, agg[i], nc - 1);
      return GB300_ERR_ARG;
    }
    cnt[agg[i] + 1]++;
  }
  for(int k = 0; k < nc; k++)
    if(cnt[k + 1] == 0) {
      set_error("aggregates: aggregate %d has no row", k);
      return GB300_ERR_ARG;
    }
  for(int k = 0; k < nc; k++) cnt[k + 1] += cnt[k];
  std::vector<int> perm(n), pos(cnt.begin(), cnt.end() - 1);
  for(int i = 0; i < n; i++) perm[pos[agg[i]]++] = i;
  // headroom of the fixed-point sums: the entries summed into one coarse
  // entry come from the rows of one aggregate
  std::vector<int> rp(n + 1);
  cudaStream_t st = A->ctx->stream;
  GB_CUDA(cudaMemcpyAsync(rp.data(), A->rowptr.p, sizeof(int) * (n + 1),
                          cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  long long most = 0;
  for(int k = 0; k < nc; k++) {
    long long s = 0;
    for(int q = cnt[k]; q < cnt[k + 1]; q++) s += rp[perm[q] + 1] - rp[perm[q]];
    most = std::max(most, s);
  }
  int head = 1;
  while((1LL << (head - 1)) < most + 1) head++;
  if(!A->coarse) A->coarse = new Coarse();
  Coarse *c = A->coarse;
  c->n = n;
  c->nc = 0;  // not valid until all buffers are there
  c->headroom = head;
  c->stamp++;
  c->ready = false;
  GB_TRY(c->agg.alloc(n));
  GB_TRY(c->aperm.alloc(n));
  GB_TRY(c->aptr.alloc(nc + 1));
  GB_TRY(c->inv.alloc((size_t)nc * nc));
  GB_TRY(c->panel.alloc(2 * ((size_t)nc + kSwB) * kSwB));
  GB_TRY(c->rc.alloc(nc));
  GB_TRY(c->ec.alloc(nc));
  GB_TRY(c->err.alloc(1));
  GB_TRY(c->amax.alloc(1));
  GB_CUDA(cudaMemcpyAsync(c->agg.p, agg, sizeof(int) * n, cudaMemcpyHostToDevice, st));
  GB_CUDA(cudaMemcpyAsync(c->aperm.p, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice,
                          st));
  GB_CUDA(cudaMemcpyAsync(c->aptr.p, cnt.data(), sizeof(int) * (nc + 1),
                          cudaMemcpyHostToDevice, st));
  GB_CUDA(cudaStreamSynchronize(st));
  c->nc = nc;
  c->version = A->pattern_version;
  return GB300_OK;
}

// ---------------------------------------------------------------------------
// aggregates from A's graph alone (when the caller has no mesh to give):
// greedy breadth-first aggregation -- from the first row not yet taken,
// take rows breadth-first over A's pattern until the aggregate holds
// ceil(n / target) rows; then rows of aggregates below a quarter of that
// size join the neighbouring aggregate they have most entries with.  On
// the 2D nonlinear Jacobian at 128^2 (ILU(0) smoothing, GMRES(50) to
// 1e-10) these took 96 steps against 121 with square cells of the mesh.

int coarse_auto(gb300_matrix *A, int target)
{
  const int n = A->n;
  if(!A->csr_valid || A->nnz <= 0 || n <= 0) {
    set_error("aggregates: the matrix has no assembled pattern");
    return GB300_ERR_ARG;
  }
  target = std::max(1, std::min(target, kMaxCoarse));
  std::vector<int> rp(n + 1), ci(A->nnz);
  cudaStream_t st = A->ctx->stream;
  GB_CUDA(cudaMemcpyAsync(rp.data(), A->rowptr.p, sizeof(int) * (n + 1),
                          cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaMemcpyAsync(ci.data(), A->col.p, sizeof(int) * A->nnz,
                          cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  std::vector<int> agg(n), queue(n), cnt;
  long long size = (n + target - 1) / target;
  int nc = 0;
  for(;;) {
    std::fill(agg.begin(), agg.end(), -1);
    nc = 0;
    for(int seed = 0; seed < n; seed++) {
      if(agg[seed] >= 0) continue;
      int head = 0, tail = 0;
      long long got = 1;
      agg[seed] = nc;
      queue[tail++] = seed;
      while(head < tail && got < size) {
        const int i = queue[head++];
        for(int k = rp[i]; k < rp[i + 1] && got < size; k++) {
          const int j = ci[k];
          if(agg[j] < 0) {
            agg[j] = nc;
            queue[tail++] = j;
            got++;
          }
        }
      }
      nc++;
    }
    cnt.assign(nc, 0);
    for(int i = 0; i < n; i++) cnt[agg[i]]++;
    const long long small = size / 4;
    std::vector<std::pair<int, int>> seen;
    for(int i = 0; i < n; i++) {
      if(cnt[agg[i]] >= small) continue;
      seen.clear();
      for(int k = rp[i]; k < rp[i + 1]; k++) {
        const int a = agg[ci[k]];
        if(cnt[a] < small) continue;
        bool found = false;
        for(auto &pr : seen)
          if(pr.first == a) {
            pr.second++;
            found = true;
            break;
          }
        if(!found) seen.push_back({a, 1});
      }
      int best = -1, bc = 0;
      for(auto &pr : seen)
        if(pr.second > bc) {
          best = pr.first;
          bc = pr.second;
        }
      if(best >= 0) agg[i] = best;  // (counts stay those of the first pass)
    }
    // compact the numbering (aggregates emptied by the merge disappear)
    std::vector<int> id(nc, -1);
    int m = 0;
    for(int i = 0; i < n; i++) {
      if(id[agg[i]] < 0) id[agg[i]] = m++;
      agg[i] = id[agg[i]];
    }
    nc = m;
    if(nc <= kMaxCoarse) break;
    size *= 2;  // too many aggregates: grow them
  }
  return coarse_set(A, agg.data(), nc);
}

// ---------------------------------------------------------------------------
// a permuted copy of A (the multicolour ordering) follows A's aggregates

__global__ void k_follow_agg(int n, const int *__restrict__ old_of,
                             const int *__restrict__ agg, const int *__restrict__ new_of,
                             const int *__restrict__ aperm, int *__restrict__ bagg,
                             int *__restrict__ baperm)
{
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    bagg[i] = agg[old_of[i]];       // new row i is old row old_of[i]
    baperm[i] = new_of[aperm[i]];   // same aggregate order, rows renamed
  }
}

int coarse_follow(const gb300_matrix *A, gb300_matrix *B, const Colouring *C,
                  cudaStream_t st)
{
  const Coarse *a = A->coarse;
  if(!B->coarse) B->coarse = new Coarse();
  Coarse *c = B->coarse;
  if(c->followed == a->stamp && c->version == B->pattern_version && c->nc == a->nc)
    return GB300_OK;
  const int n = A->n, nc = a->nc;
  c->n = n;
  c->nc = 0;  // not valid until all buffers are there
  c->headroom = a->headroom;
  c->ready = false;
  GB_TRY(c->agg.alloc(n));
  GB_TRY(c->aperm.alloc(n));
  GB_TRY(c->aptr.alloc(nc + 1));
  GB_TRY(c->inv.alloc((size_t)nc * nc));
  GB_TRY(c->panel.alloc(2 * ((size_t)nc + kSwB) * kSwB));
  GB_TRY(c->rc.alloc(nc));
  GB_TRY(c->ec.alloc(nc));
  GB_TRY(c->err.alloc(1));
  GB_TRY(c->amax.alloc(1));
  k_follow_agg<<<grid_for(n, 256), 256, 0, st>>>(n, C->old_of.p, a->agg.p, C->new_of.p,
                                                 a->aperm.p, c->agg.p, c->aperm.p);
  GB_CUDA(cudaMemcpyAsync(c->aptr.p, a->aptr.p, sizeof(int) * (nc + 1),
                          cudaMemcpyDeviceToDevice, st));
  GB_CUDA(cudaGetLastError());
  c->nc = nc;
  c->followed = a->stamp;
  c->version = B->pattern_version;
  return GB300_OK;
}

// ---------------------------------------------------------------------------
// set-up: Ac = P0^T A P0 in fixed point, then its inverse

// max |val| (non-negative doubles order like their bit patterns; a NaN
// orders above +Inf and is caught by the scatter)
__global__ void k_abs_max(long long nnz, const double *__restrict__ val,
                          unsigned long long *out)
{
  unsigned long long m = 0;
  for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < nnz;
      k += (long long)gridDim.x * blockDim.x)
    m = max(m, (unsigned long long)__double_as_longlong(fabs(val[k])));
  for(int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
  if((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// every row's entries, summed by the aggregate of their column (one atomic
// add per run of equal aggregates), into acc[agg(row) * nc + agg(col)]
__global__ void k_coarse_scatter(int n, const int *__restrict__ rowptr,
                                 const int *__restrict__ col, const double *__restrict__ val,
                                 const int *__restrict__ agg, const int *__restrict__ aperm,
                                 int nc, int headroom, const unsigned long long *amax_bits,
                                 unsigned long long *acc, int *err)
{
  const double am = __longlong_as_double((long long)*amax_bits);
  if(!(am <= 1.7976931348623157e308) || am == 0.) {  // NaN, Inf or a zero matrix
    if(blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(err, 0, -1);
    return;
  }
  int e = 0;
  frexp(am, &e);  // am < 2^e
  const double s = ldexp(1.0, 62 - headroom - e);
  for(int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const int i = aperm[q];
    const size_t base = (size_t)agg[i] * nc;
    int run = -1;
    long long sum = 0;
    for(int k = rowptr[i]; k < rowptr[i + 1]; k++) {
      const int l = agg[col[k]];
      if(l != run) {
        if(run >= 0) atomicAdd(acc + base + run, (unsigned long long)sum);
        run = l;
        sum = 0;
      }
      sum += llrint(val[k] * s);
    }
    if(run >= 0) atomicAdd(acc + base + run, (unsigned long long)sum);
  }
}

__global__ void k_coarse_to_double(long long m, int headroom,
                                   const unsigned long long *amax_bits, double *a)
{
  const double am = __longlong_as_double((long long)*amax_bits);
  int e = 0;
  frexp(am, &e);
  const double qnt = ldexp(1.0, e + headroom - 62);
  unsigned long long *acc = reinterpret_cast<unsigned long long *>(a);
  for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < m;
      k += (long long)gridDim.x * blockDim.x) {
    const long long v = (long long)acc[k];
    a[k] = (double)v * qnt;
  }
}

// The inverse of the symmetric positive definite nc x nc matrix, in place, by
// the symmetric sweep operator on blocks of kSwB columns: for the block K
// with diagonal block D and panel P = A(:, K),
//
//   A(i, j) -= P(i) D^-1 P(j)^T   (i, j outside K)
//   A(i, K)  = P(i) D^-1,  A(K, K) = -D^-1,
//
// after which A holds -A^-1.  The matrix stays symmetric, so only the lower
// triangle is kept up: nc^3 / 2 FMAs.  GB300's FP64 pipe (two FMAs per SM
// per clock) bounds the update (1.0 ms at nc = 1024); a sweep of one pivot
// per launch read and wrote all nc^2 entries 1,024 times (8 GB each way
// through L2 and 1,024 launches, 14.6 ms).  32 columns: narrower blocks
// re-read the triangle more often, wider ones lengthen the serial inversion
// of D (32 pivots, each a division and an FMA deep: 27 us).  That inversion
// runs beside the update of the block before, in a CTA that computes its tile
// first: 45 us a block (panel 5, update 40) and 1.5 ms in all at nc = 1024,
// against 80 us and 2.4 ms with D inverted by every CTA of the panel.  No
// pivoting: the pivots met inside the blocks are those of the unblocked
// elimination, and one that is not positive is reported.
constexpr int kSwRows = 8;  // panel rows per CTA

// D^-1 by Gauss-Jordan steps, one barrier per pivot, for a block of 256
// threads with D in buf[0] (complete in every thread's sight, padded with the
// identity); thread t has entries (t / 8, t % 8 * 4 + 0..3).  False (in every
// thread) where a pivot is not positive and finite.
__device__ bool sweep_invert(double (*buf)[kSwB][kSwB + 1], double *rp, int k0, double *dinv,
                             int *err)
{
  const int t = threadIdx.x, i = t >> 3, j0 = (t & 7) * 4;
  if(t == 0) rp[0] = 1. / buf[0][0][0];
  __syncthreads();
  for(int k = 0; k < kSwB; k++) {
    const int cur = k & 1, nxt = cur ^ 1;
    const double piv = buf[cur][k][k];
    if(!(piv > 0.) || !(piv <= 1.7976931348623157e308)) {  // the same in every thread
      if(t == 0) atomicCAS(err, 0, k0 + k + 1);
      return false;
    }
    // one FMA per entry (FP64 instructions, not memory, pace the pivots):
    // row k is 0 + p R, column k is 0 + m 1, the rest D + m R
    const double p = rp[cur], m = i == k ? p : -buf[cur][i][k] * p;
#pragma unroll
    for(int u = 0; u < 4; u++) {
      const int j = j0 + u;
      const double r = j == k ? 1. : buf[cur][k][j];
      const double v = fma(m, r, (i == k || j == k) ? 0. : buf[cur][i][j]);
      buf[nxt][i][j] = v;
      if(i == k + 1 && j == k + 1) rp[nxt] = 1. / v;
    }
    __syncthreads();
  }
  static_assert(kSwB % 2 == 0, "the result is in buf[0]");
#pragma unroll
  for(int u = 0; u < 4; u++) dinv[i * kSwB + j0 + u] = buf[0][i][j0 + u];
  return true;
}

// D^-1 of the first block
__global__ void __launch_bounds__(256)
k_sweep_first(int nc, const double *__restrict__ a, double *__restrict__ dinv, int *err)
{
  if(*err) return;
  __shared__ double D[2][kSwB][kSwB + 1], rp[2];
  const int t = threadIdx.x, i = t >> 3, j0 = (t & 7) * 4;
#pragma unroll
  for(int u = 0; u < 4; u++) {
    const int j = j0 + u;
    const int hi = i > j ? i : j, lo = i > j ? j : i;
    D[0][i][j] = hi < nc ? a[(size_t)hi * nc + lo] : (i == j ? 1. : 0.);
  }
  __syncthreads();
  sweep_invert(D, rp, 0, dinv, err);
}

// W(i) = P(i) D^-1 for this CTA's kSwRows rows; P, W: nc x kSwB
__global__ void __launch_bounds__(128)
k_sweep_panel(int nc, int k0, const double *__restrict__ a, double *__restrict__ P,
              double *__restrict__ W, const double *__restrict__ dinv, const int *err)
{
  if(*err) return;
  __shared__ double D[kSwB][kSwB], sp[kSwRows][kSwB + 1];
  const int t = threadIdx.x;
  const int bw = nc - k0 < kSwB ? nc - k0 : kSwB;
  const int r0 = blockIdx.x * kSwRows;
#pragma unroll
  for(int q = t; q < kSwB * kSwB; q += 128) D[q / kSwB][q % kSwB] = dinv[q];
#pragma unroll
  for(int q = t; q < kSwRows * kSwB; q += 128) {
    // the panel's rows below K by row, those above K (stored transposed) by
    // column, so that both read runs of the lower triangle
    int r, c;
    if(r0 >= k0) {
      r = q / kSwB;
      c = q % kSwB;
    }
    else {
      r = q % kSwRows;
      c = q / kSwRows;
    }
    const int gi = r0 + r, gj = k0 + c;
    double v = 0.;
    if(gi < nc && c < bw)
      v = gi >= gj ? a[(size_t)gi * nc + gj] : a[(size_t)gj * nc + gi];
    sp[r][c] = v;
  }
  __syncthreads();
  const int r = t >> 4, c = (t & 15) * 2;
  double w0 = 0., w1 = 0.;
#pragma unroll 8
  for(int k = 0; k < kSwB; k++) {
    w0 = fma(sp[r][k], D[k][c], w0);
    w1 = fma(sp[r][k], D[k][c + 1], w1);
  }
  if(r0 + r < nc) {
    const size_t o = (size_t)(r0 + r) * kSwB + c;
    P[o] = sp[r][c];
    P[o + 1] = sp[r][c + 1];
    W[o] = w0;
    W[o + 1] = w1;
  }
}

// The lower triangle's 32 x 32 tiles after the sweep of block kb, four to a
// CTA (64 threads each); CTA 0 has tile (kb + 1, kb + 1) alone and inverts it
// for the next block.  Four tiles a CTA, not one: at nc = 1024 the 133 CTAs
// then lie on an SM each, and the inversion shares its FP64 pipe with none.
constexpr int kSwTiles = 4;
constexpr size_t kSwShared = sizeof(double) * kSwTiles * 2 * kSwB * (kSwB + 1);

__global__ void __launch_bounds__(64 * kSwTiles)
k_sweep_update(int nc, int nb, int kb, double *__restrict__ a, const double *__restrict__ P,
               const double *__restrict__ W, const double *__restrict__ dinv,
               double *__restrict__ dnext, int *err)
{
  // CTA 0 may set *err while this launch runs: one answer for the whole CTA
  // (its threads meet at barriers below)
  if(__syncthreads_or(*(volatile int *)err)) return;
  extern __shared__ double shared[];
  double (*buf)[kSwB][kSwB + 1] = reinterpret_cast<double (*)[kSwB][kSwB + 1]>(shared);
  __shared__ double rp[2];
  const int g = threadIdx.x >> 6, t = threadIdx.x & 63;
  const int nk = kb + 1;
  if(blockIdx.x == 0) {
    if(nk >= nb) return;
    const int k0 = nk * kSwB;
    for(int q = threadIdx.x; q < kSwB * kSwB; q += 256) {
      const int r = q / kSwB, c = q % kSwB;
      buf[0][c][r] = k0 + r < nc ? W[(size_t)(k0 + r) * kSwB + c] : 0.;
      buf[1][c][r] = k0 + r < nc ? P[(size_t)(k0 + r) * kSwB + c] : 0.;
    }
    __syncthreads();
    const int i = threadIdx.x >> 3, j0 = (threadIdx.x & 7) * 4;
    double acc[4];
#pragma unroll
    for(int u = 0; u < 4; u++)
      acc[u] = k0 + i < nc && k0 + j0 + u < nc ? a[(size_t)(k0 + i) * nc + k0 + j0 + u] : 0.;
#pragma unroll 8
    for(int k = 0; k < kSwB; k++)
#pragma unroll
      for(int u = 0; u < 4; u++)
        acc[u] = fma(-buf[0][k][i], buf[1][k][j0 + u], acc[u]);
#pragma unroll
    for(int u = 0; u < 4; u++) {
      const int j = j0 + u;
      const bool in = k0 + i < nc && k0 + j < nc;
      if(in) a[(size_t)(k0 + i) * nc + k0 + j] = acc[u];
      if(j <= i) {  // (the inversion takes the lower triangle for both)
        const double v = in ? acc[u] : (i == j ? 1. : 0.);
        buf[2][i][j] = v;
        buf[2][j][i] = v;
      }
    }
    __syncthreads();
    sweep_invert(buf + 2, rp, k0, dnext, err);
    return;
  }
  // tile number -> (ti, tj), tj <= ti
  const long long tile = (long long)(blockIdx.x - 1) * kSwTiles + g;
  int ti = (int)((sqrtf(8.f * (float)tile + 1.f) - 1.f) * 0.5f);
  while((long long)(ti + 1) * (ti + 2) / 2 <= tile) ti++;
  while((long long)ti * (ti + 1) / 2 > tile) ti--;
  const int tj = (int)(tile - (long long)ti * (ti + 1) / 2);
  const int i0 = ti * kSwB, j0 = tj * kSwB;
  const bool there = ti < nb && !(ti == nk && tj == nk);
  const bool inside = there && ti != kb && tj != kb;
  double (*sw)[kSwB + 1] = buf[2 * g], (*spt)[kSwB + 1] = buf[2 * g + 1];  // [k][row]
  if(there && !inside)
    for(int q = t; q < kSwB * kSwB; q += 64) {
      const int r = q / kSwB, c = q % kSwB;
      if(i0 + r >= nc || j0 + c >= nc) continue;
      double v;
      if(ti == tj)
        v = -dinv[q];
      else if(tj == kb)
        v = W[(size_t)(i0 + r) * kSwB + c];
      else
        v = W[(size_t)(j0 + c) * kSwB + r];
      a[(size_t)(i0 + r) * nc + j0 + c] = v;
    }
  // 4 x 4 entries per thread, rows and columns 8 apart (no bank conflicts,
  // coalesced columns)
  const int ty = t >> 3, tx = t & 7;
  double acc[4][4];
  if(inside) {
    for(int q = t; q < kSwB * kSwB; q += 64) {
      const int r = q / kSwB, c = q % kSwB;
      sw[c][r] = i0 + r < nc ? W[(size_t)(i0 + r) * kSwB + c] : 0.;
      spt[c][r] = j0 + r < nc ? P[(size_t)(j0 + r) * kSwB + c] : 0.;
    }
#pragma unroll
    for(int u = 0; u < 4; u++)
#pragma unroll
      for(int v = 0; v < 4; v++) {
        const int r = i0 + ty + 8 * u, c = j0 + tx + 8 * v;
        acc[u][v] = (r < nc && c < nc) ? a[(size_t)r * nc + c] : 0.;
      }
  }
  __syncthreads();
  if(!inside) return;
#pragma unroll 4
  for(int k = 0; k < kSwB; k++) {
    double wr[4], pc[4];
#pragma unroll
    for(int u = 0; u < 4; u++) {
      wr[u] = sw[k][ty + 8 * u];
      pc[u] = spt[k][tx + 8 * u];
    }
#pragma unroll
    for(int u = 0; u < 4; u++)
#pragma unroll
      for(int v = 0; v < 4; v++) acc[u][v] = fma(-wr[u], pc[v], acc[u][v]);
  }
#pragma unroll
  for(int u = 0; u < 4; u++)
#pragma unroll
    for(int v = 0; v < 4; v++) {
      const int r = i0 + ty + 8 * u, c = j0 + tx + 8 * v;
      if(r < nc && c < nc) a[(size_t)r * nc + c] = acc[u][v];
    }
}

// A^-1 = -(swept matrix), the upper triangle from the lower one
__global__ void __launch_bounds__(256)
k_sweep_finish(int nc, double *__restrict__ a, const int *err)
{
  if(*err) return;
  __shared__ double s[32][33];
  const int ti = blockIdx.y, tj = blockIdx.x;
  if(tj > ti) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for(int r = y; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + x;
    double v = 0.;
    if(i < nc && j <= i) {
      v = -a[(size_t)i * nc + j];
      a[(size_t)i * nc + j] = v;
    }
    s[r][x] = v;
  }
  __syncthreads();
  for(int r = y; r < 32; r += 8) {
    const int i = tj * 32 + r, j = ti * 32 + x;  // transposed tile
    if(j < nc && i < j) a[(size_t)i * nc + j] = s[x][r];
  }
}

// *err = kAsymmetric where two mirrored entries differ by more than rounding:
// than the fixed-point sums' own (2^(headroom - 1) terms, half a quantum each,
// in both) and 2^-44 of their rows' diagonals, for an A assembled in another
// order above and below its diagonal (the elimination's backward error, some
// nc 2^-53, is no smaller).  The symmetric sweep's kernels then do nothing.
constexpr int kAsymmetric = -2;

__global__ void __launch_bounds__(256)
k_coarse_symmetric(int nc, int headroom, const unsigned long long *amax_bits,
                   const double *__restrict__ a, int *err)
{
  __shared__ double s[32][33];
  const int ti = blockIdx.y, tj = blockIdx.x;
  if(tj > ti) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for(int r = y; r < 32; r += 8) {
    const int i = tj * 32 + r, j = ti * 32 + x;  // the transposed tile
    s[r][x] = i < nc && j < nc ? a[(size_t)i * nc + j] : 0.;
  }
  __syncthreads();
  int e = 0;
  frexp(__longlong_as_double((long long)*amax_bits), &e);
  const double sums = ldexp(1., e + 2 * headroom - 63);
  for(int r = y; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + x;
    if(i >= nc || j >= i) continue;
    const double d = fabs(a[(size_t)i * nc + j] - s[x][r]) - sums;
    if(d <= 0.) continue;
    const double di = a[(size_t)i * nc + i], dj = a[(size_t)j * nc + j];
    if(d > 0x1p-44 * sqrt(fabs(di)) * sqrt(fabs(dj))) atomicCAS(err, 0, kAsymmetric);
  }
}

// The inverse of any other Ac, by Gauss-Jordan steps without pivoting (14.6 ms
// at nc = 1024 against the sweep's 1.5: nc launches that read and write all
// nc^2 entries).
__global__ void k_gj_init(int nc, const double *__restrict__ a, double *rbuf, double *cbuf)
{
  for(int j = blockIdx.x * blockDim.x + threadIdx.x; j < nc; j += gridDim.x * blockDim.x) {
    rbuf[j] = a[j];                 // row 0
    cbuf[j] = a[(size_t)j * nc];    // column 0
  }
}

// pivot step k of the in-place Gauss-Jordan inversion; row k and column k of
// the matrix before the step come from the buffers of parity k, and the step
// writes row and column k + 1 of its result to the other parity
__global__ void k_gj_step(int nc, int k, double *a, double *rbuf, double *cbuf, int *err)
{
  if(*err) return;
  const double *R = rbuf + (size_t)(k & 1) * nc;
  const double *Cc = cbuf + (size_t)(k & 1) * nc;
  double *Rn = rbuf + (size_t)((k + 1) & 1) * nc;
  double *Cn = cbuf + (size_t)((k + 1) & 1) * nc;
  const double piv = R[k];
  if(!(piv > 0.) || !(piv <= 1.7976931348623157e308)) {
    if(blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(err, 0, k + 1);
    return;
  }
  const double p = 1.0 / piv;
  const long long m = (long long)nc * nc;
  for(long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < m;
      idx += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(idx / nc), j = (int)(idx - (long long)i * nc);
    double v;
    if(i == k)
      v = (j == k) ? p : R[j] * p;
    else if(j == k)
      v = -Cc[i] * p;
    else
      v = fma(-Cc[i] * p, R[j], a[idx]);
    a[idx] = v;
    if(i == k + 1) Rn[j] = v;
    if(j == k + 1) Cn[i] = v;
  }
}

static int coarse_invert_general(Coarse *c, cudaStream_t st)
{
  const int nc = c->nc;
  double *rbuf = c->panel.p, *cbuf = rbuf + 2 * (size_t)nc;  // (4 nc of 64 (nc + 32))
  GB_CUDA(cudaMemsetAsync(c->err.p, 0, sizeof(int), st));
  k_gj_init<<<grid_for(nc, 256), 256, 0, st>>>(nc, c->inv.p, rbuf, cbuf);
  const int g = grid_for((long long)nc * nc, 256, kReduceBlocks * 2);
  for(int k = 0; k < nc; k++)
    k_gj_step<<<g, 256, 0, st>>>(nc, k, c->inv.p, rbuf, cbuf, c->err.p);
  GB_CUDA(cudaGetLastError());
  return GB300_OK;
}

int coarse_setup(gb300_matrix *A, const double *val, bool reuse)
{
  Coarse *c = A->coarse;
  if(reuse && c->ready) return GB300_OK;
  cudaStream_t st = A->ctx->stream;
  const int nc = c->nc, n = A->n;
  const long long m = (long long)nc * nc;
  unsigned long long *amax = reinterpret_cast<unsigned long long *>(c->amax.p);
  GB_CUDA(cudaMemsetAsync(amax, 0, sizeof(unsigned long long), st));
  GB_CUDA(cudaMemsetAsync(c->err.p, 0, sizeof(int), st));
  GB_CUDA(cudaMemsetAsync(c->inv.p, 0, sizeof(double) * m, st));
  k_abs_max<<<grid_for(A->nnz, 256, kReduceBlocks), 256, 0, st>>>(A->nnz, val, amax);
  k_coarse_scatter<<<grid_for(n, 128), 128, 0, st>>>(
      n, A->rowptr.p, A->col.p, val, c->agg.p, c->aperm.p, nc, c->headroom, amax,
      reinterpret_cast<unsigned long long *>(c->inv.p), c->err.p);
  k_coarse_to_double<<<grid_for(m, 256, kReduceBlocks), 256, 0, st>>>(m, c->headroom, amax,
                                                                      c->inv.p);
  const int nb = (nc + kSwB - 1) / kSwB;
  k_coarse_symmetric<<<dim3(nb, nb), 256, 0, st>>>(nc, c->headroom, amax, c->inv.p, c->err.p);
  GB_CUDA(cudaGetLastError());
  const int tiles = nb * (nb + 1) / 2;
  double *P = c->panel.p, *Wp = P + (size_t)nc * kSwB, *dinv = Wp + (size_t)nc * kSwB;
  GB_CUDA(cudaFuncSetAttribute(k_sweep_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kSwShared));
  k_sweep_first<<<1, 256, 0, st>>>(nc, c->inv.p, dinv, c->err.p);
  for(int k = 0; k < nb; k++) {
    double *dnext = dinv + (k & 1 ? -1 : 1) * kSwB * kSwB;  // two, in turn
    k_sweep_panel<<<grid_for(nc, kSwRows), 128, 0, st>>>(nc, k * kSwB, c->inv.p, P, Wp, dinv,
                                                         c->err.p);
    k_sweep_update<<<1 + (tiles + kSwTiles - 1) / kSwTiles, 64 * kSwTiles, kSwShared, st>>>(
        nc, nb, k, c->inv.p, P, Wp, dinv, dnext, c->err.p);
    dinv = dnext;
  }
  k_sweep_finish<<<dim3(nb, nb), 256, 0, st>>>(nc, c->inv.p, c->err.p);
  GB_CUDA(cudaGetLastError());
  int err = 0;
  GB_CUDA(cudaMemcpyAsync(&err, c->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  if(err == kAsymmetric) {  // Ac is as it was
    GB_TRY(coarse_invert_general(c, st));
    GB_CUDA(cudaMemcpyAsync(&err, c->err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
  }
  if(err < 0) {
    set_error("coarse matrix: the matrix values are zero or not finite");
    return GB300_ERR_ARG;
  }
  if(err > 0) {
    set_error("coarse matrix P^T A P is not positive definite (pivot %d of %d)", err, nc);
    return GB300_ERR_ZERO_PIVOT;
  }
  c->ready = true;
  return GB300_OK;
}

// ---------------------------------------------------------------------------
// application

// rc = P0^T t: one CTA of kRestrictThreads per aggregate, its rows in a fixed
// order (a warp per aggregate had left a thousand gathers to 32 lanes)
constexpr int kRestrictThreads = 128;

__global__ void __launch_bounds__(kRestrictThreads)
k_restrict(const int *__restrict__ aptr, const int *__restrict__ aperm, const double *t,
           double *rc, const int *flag)
{
  constexpr int U = 4;
  const int k = blockIdx.x;
  const int q0 = aptr[k] + threadIdx.x, e = aptr[k + 1];
  int i[U];
#pragma unroll
  for(int u = 0; u < U; u++)
    i[u] = q0 + u * kRestrictThreads < e ? aperm[q0 + u * kRestrictThreads] : -1;
  chain_wait();
  if(flag && !*flag) return;
  double s = 0.;
#pragma unroll
  for(int u = 0; u < U; u++)
    if(i[u] >= 0) s += t[i[u]];
#pragma unroll 4
  for(int q = q0 + U * kRestrictThreads; q < e; q += kRestrictThreads) s += t[aperm[q]];
  s = block_sum<double, kRestrictThreads>(s);
  if(threadIdx.x == 0) rc[k] = s;
}

// ec = Ainv rc: one warp per row
__global__ void __launch_bounds__(256)
k_coarse_gemv(int nc, const double *__restrict__ inv, const double *rc, double *ec,
              const int *flag)
{
  constexpr int U = 8;
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const double *row = inv + (size_t)(i < nc ? i : 0) * nc;
  double a[U];
#pragma unroll
  for(int u = 0; u < U; u++) a[u] = lane + 32 * u < nc ? row[lane + 32 * u] : 0.;
  chain_wait();
  if(flag && !*flag) return;
  if(i >= nc) return;
  double s = 0.;
#pragma unroll
  for(int u = 0; u < U; u++)
    if(lane + 32 * u < nc) s = fma(a[u], rc[lane + 32 * u], s);
#pragma unroll 8
  for(int j = lane + 32 * U; j < nc; j += 32) s = fma(row[j], rc[j], s);
  s = warp_sum(s);
  if(lane == 0) ec[i] = s;
}

// out = z + P0 ec
__global__ void __launch_bounds__(256)
k_prolong_to(int n, const int *__restrict__ agg, const double *ec, const double *z, double *out,
             const int *flag)
{
  const int i = blockIdx.x * 256 + threadIdx.x;
  const int g = i < n ? agg[i] : 0;
  chain_wait();
  const int go = flag ? *flag : 1;
  if(i >= n || !go) return;
  out[i] = z[i] + ec[g];
}

static void coarse_solve(const Coarse *c, const double *t, int n, const int *flag,
                         cudaStream_t st)
{
  launch_chain(chain_early(n), k_restrict, c->nc, kRestrictThreads, st, c->aptr.p, c->aperm.p,
               t, c->rc.p, flag);
  launch_chain(chain_early(n), k_coarse_gemv, grid_for((long long)c->nc * 32, 256), 256, st,
               c->nc, c->inv.p, c->rc.p, c->ec.p, flag);
}

void coarse_correct(const gb300_matrix *A, const double *val, const double *v,
                    const double *z, double *out, double *t, const int *flag,
                    cudaStream_t st)
{
  const Coarse *c = A->coarse;
  product_chain(kChainRes, A, val, {z, v, t, nullptr, nullptr, nullptr, flag}, st);
  coarse_solve(c, t, A->n, flag, st);
  // the prolongation inside the residual saves a launch and a pass, but adds
  // an FP64 addition per matrix entry: 6.0 against 7.2 us at 65,025 rows, 45
  // against 31 at 1,046,529
  if(chain_early(A->n)) {
    product_chain(kChainProlong, A, val, {z, v, t, c->agg.p, c->ec.p, out, flag}, st);
    return;
  }
  launch_chain(false, k_prolong_to, grid_for(A->n, 256), 256, st, A->n, c->agg.p, c->ec.p, z,
               out, flag);
  product_chain(kChainRes, A, val, {out, v, t, nullptr, nullptr, nullptr, flag}, st);
}

// one block: out = rc . ec over the nc coarse entries, in a fixed order
__global__ void k_coarse_dot(int nc, const double *__restrict__ a,
                             const double *__restrict__ b, double *out)
{
  __shared__ double sh[32];
  double s = 0.;
  for(int k = threadIdx.x; k < nc; k += blockDim.x) s = fma(a[k], b[k], s);
  s = warp_sum(s);
  if((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if(threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.;
    s = warp_sum(s);
    if(threadIdx.x == 0) *out = s;
  }
}

__global__ void k_prolong_set(int n, const int *__restrict__ agg, const double *__restrict__ ec,
                              double *__restrict__ t)
{
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    t[i] = ec[agg[i]];
}

__global__ void k_sub_into(int n, const double *__restrict__ q, double *__restrict__ w)
{
  for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    w[i] -= q[i];
}

int coarse_energy_project(gb300_matrix *A, double *w, double *t, double *q, double *wcw,
                          cudaStream_t st)
{
  GB_TRY(coarse_setup(A, A->val.p, true));
  const Coarse *c = A->coarse;
  const int n = A->n, nc = c->nc;
  const int g = grid_for(n, 256, kReduceBlocks * 4);
  coarse_solve(c, w, n, nullptr, st);
  k_coarse_dot<<<1, 1024, 0, st>>>(nc, c->rc.p, c->ec.p, wcw);
  k_prolong_set<<<g, 256, 0, st>>>(n, c->agg.p, c->ec.p, t);
  spmv_plain(A, A->val.p, t, q, st);
  k_sub_into<<<g, 256, 0, st>>>(n, q, w);
  GB_CUDA(cudaGetLastError());
  return GB300_OK;
}

int coarse_energy(gb300_matrix *A, const double *u, double *ucu_dev, cudaStream_t st)
{
  GB_TRY(coarse_setup(A, A->val.p, true));
  const Coarse *c = A->coarse;
  const int nc = c->nc;
  coarse_solve(c, u, A->n, nullptr, st);
  k_coarse_dot<<<1, 1024, 0, st>>>(nc, c->rc.p, c->ec.p, ucu_dev);
  GB_CUDA(cudaGetLastError());
  return GB300_OK;
}

}  // namespace gb
