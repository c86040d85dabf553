// ILU(0) and the GMRES family on the GPU.
//
// ILU(0) (ilu0, contrib/Sparskit/ilut.F:1818-1941) keeps A's pattern; the
// factor is stored in a copy of A's values (L multipliers left of the
// diagonal, U right of it) plus the inverted pivots, as Sparskit's MSR
// layout does.  Rows are factored and solved level by level: a level holds
// rows whose lower (resp. upper) neighbours all belong to earlier levels,
// so its rows are independent.  Narrow levels (<= kNarrow rows) run back to
// back inside one thread block separated by __syncthreads; a wide level gets
// its own grid launch.  For the solves, each wide level also keeps its rows'
// L (resp. U) entries in a sliced-ELL copy (32 rows per slice, entry j of
// the slice's rows side by side), so that a warp reads them coalesced and
// without the row-pointer indirection; on a multicolour copy the sweeps are a
// chain of launches colour by colour over consecutive rows (k_colour_sweep),
// and a small system's whole step of sweeps and product is one CTA
// (k_small_step).  The triangular solves follow lusol (ilut.F:2297-2347) row
// by row in the same accumulation order.
//
// GMRES(m) and FGMRES(m) follow iters.f:1912-2219 / :2522-2806 with right
// preconditioning (Preconditioner_Position 2): restart residual, Arnoldi
// steps, Givens rotations (iters.f:3235-3273), the stopping test on the
// Givens residual estimate, and the triangular solve + update at the end of
// a cycle.  The orthogonalisation is classical Gram-Schmidt with block dot
// products, which parallelises over the basis, in place of the reference's
// sequential modified Gram-Schmidt; like mgsro (iters.f:3475) it
// re-orthogonalises selectively (a second pass when the first removed more
// than 98 % of ||w||^2), and both return an orthonormal basis to working
// precision.
#include <math.h>

#include <algorithm>
#include <memory>

#include "krylov.cuh"

namespace gb {

constexpr int kNarrow = 2048;
constexpr int kNarrowThreads = 1024;

struct Segment {
  int l0, l1;  // levels [l0, l1)
  bool narrow;
  int width;   // rows of the (single) wide level
  int r0;      // first index in the level-row list
};

// sliced-ELL copy of one triangular part, wide levels only: slice s holds
// 32 rows x width[s] entries at 32 * wscan[s], entry j of lane l at
// + 32 j + l; src is the entry's position in the CSR factor; padding has
// src = col = -1 and is skipped (a product of its zero with a vector entry
// not yet written would be NaN when that memory happens to hold one)
struct EllPart {
  std::vector<int> slice0;  // per segment: its first slice (wide segments)
  // per segment: the common width of its slices and the place of its first
  // entry, so that a kernel finds a row's entries without reading its slice's
  // width and offset (0: the widths differ)
  std::vector<int> common;
  std::vector<long long> first;
  int nslices = 0;
  long long entries = 0;
  DevBuf<int> width, col, src;
  DevBuf<long long> wscan;
  DevBuf<double> v64;
  DevBuf<float> v32;
};

struct ilu_data {
  int n = 0;
  EllPart lell, uell;
  DevBuf<int> diag;                 // position of a_ii in each row
  DevBuf<int> lrows, urows;         // rows grouped by level
  DevBuf<int> lptr, uptr;           // level offsets (device copies)
  std::vector<int> hlptr, huptr;    // level offsets (host)
  std::vector<Segment> lseg, useg;
  // a multicolour copy (one row per vertex): the levels are the colours, rows
  // in order (lrows and urows stay empty), the sweeps run as a chain
  bool by_colour = false;
  int n0 = 0;                       // rows of colour 0
  EllPart aell;                     // A's own rows, for the products
  const double *aell_of = nullptr;  // the values it holds (ilu_products)
  DevBuf<double> lu64, inv64;
  DevBuf<float> lu32, inv32;
  bool fact64 = false, fact32 = false;  // a factor of that precision is held
  unsigned version = ~0u;               // the matrix pattern it was set up for
  std::unique_ptr<SysLevels> sys;       // the schedule cut into a batch's blocks
};

void ilu_free(ilu_data *d) { delete d; }

// ---------------------------------------------------------------------------
// level schedule
// ---------------------------------------------------------------------------
__global__ void k_ilu_prep(int n, const int *__restrict__ rowptr,
                           const int *__restrict__ col, int *__restrict__ diag,
                           int *__restrict__ indl, int *__restrict__ indu,
                           int *__restrict__ err)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i >= n) return;
  int s = rowptr[i], e = rowptr[i + 1];
  int dpos = -1, nl = 0, nu = 0;
  for(int k = s; k < e; k++) {
    int c = col[k];
    if(c < i)
      nl++;
    else if(c > i)
      nu++;
    else
      dpos = k;
    // structural symmetry: (c, i) must exist
    if(c != i && find_col(col, rowptr[c], rowptr[c + 1], i) < 0)
      atomicOr(err, 2);
  }
  if(dpos < 0) atomicOr(err, 1);
  diag[i] = dpos;
  indl[i] = nl;
  indu[i] = nu;
}

__global__ void k_level0(int n, const int *__restrict__ indeg,
                         int *__restrict__ rows, int *__restrict__ cnt)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if(i < n && indeg[i] == 0) rows[atomicAdd(cnt, 1)] = i;
}

// release the dependants of one level; UPPER = 0 walks the lower
// triangular DAG (dependants of i are j > i in row i), UPPER = 1 the upper
template <int UPPER>
__global__ void k_level_next(int p0, int p1, const int *__restrict__ rowptr,
                             const int *__restrict__ col,
                             const int *__restrict__ diag,
                             int *__restrict__ indeg, int *__restrict__ rows,
                             int *__restrict__ cnt)
{
  int t = p0 + blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= p1) return;
  int i = rows[t];
  int s = UPPER ? rowptr[i] : diag[i] + 1;
  int e = UPPER ? diag[i] : rowptr[i + 1];
  for(int k = s; k < e; k++) {
    int j = col[k];
    if(atomicSub(&indeg[j], 1) == 1) rows[p1 + atomicAdd(cnt, 1)] = j;
  }
}

template <int UPPER>
static int make_levels(gb300_matrix *A, ilu_data *L, int *d_indeg,
                       DevBuf<int> &rows, DevBuf<int> &dptr,
                       std::vector<int> &hptr, std::vector<Segment> &seg)
{
  cudaStream_t st = A->ctx->stream;
  int n = A->n;
  DevBuf<int> cnt;
  GB_TRY(cnt.alloc(1));
  GB_TRY(rows.alloc(n));
  GB_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int), st));
  k_level0<<<grid_for(n, 256), 256, 0, st>>>(n, d_indeg, rows.p, cnt.p);
  int c = 0;
  GB_CUDA(cudaMemcpyAsync(&c, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  hptr.assign(1, 0);
  hptr.push_back(c);
  int p0 = 0, p1 = c;
  while(p1 < n) {
    if(p1 == p0) {
      set_error("ILU level schedule: dependency cycle");
      return GB300_ERR_ARG;
    }
    GB_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int), st));
    k_level_next<UPPER><<<grid_for(p1 - p0, 256), 256, 0, st>>>(
      p0, p1, A->rowptr.p, A->col.p, L->diag.p, d_indeg, rows.p, cnt.p);
    GB_CUDA(cudaMemcpyAsync(&c, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    p0 = p1;
    p1 += c;
    hptr.push_back(p1);
  }
  int nl = (int)hptr.size() - 1;
  GB_TRY(dptr.alloc(nl + 1));
  GB_CUDA(cudaMemcpyAsync(dptr.p, hptr.data(), sizeof(int) * (nl + 1),
                          cudaMemcpyHostToDevice, st));
  seg.clear();
  for(int l = 0; l < nl;) {
    int w = hptr[l + 1] - hptr[l];
    if(w > kNarrow) {
      seg.push_back({l, l + 1, false, w, hptr[l]});
      l++;
    }
    else {
      int l1 = l;
      while(l1 < nl && hptr[l1 + 1] - hptr[l1] <= kNarrow) l1++;
      seg.push_back({l, l1, true, 0, hptr[l]});
      l = l1;
    }
  }
  GB_CUDA(cudaStreamSynchronize(st));
  return GB300_OK;
}

// entries of row i's strictly lower (UPPER = 0) or upper (1) part, or of the
// whole row (2)
template <int UPPER>
__device__ __forceinline__ void part_range(int i, const int *rowptr, const int *diag,
                                           int &k0, int &cnt)
{
  k0 = UPPER == 1 ? diag[i] + 1 : rowptr[i];
  cnt = UPPER == 0 ? diag[i] - rowptr[i] : rowptr[i + 1] - (UPPER == 1 ? diag[i] + 1 : k0);
}

template <int UPPER>
__global__ void k_ell_width(int r0, int w, int nsl, int slice0, const int *__restrict__ rows,
                            const int *__restrict__ rowptr, const int *__restrict__ diag,
                            int *__restrict__ width)
{
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= nsl * 32) return;  // whole warps: nsl * 32 is a multiple of 32
  int cnt = 0;
  if(t < w) {
    int k0;
    part_range<UPPER>(rows ? rows[r0 + t] : r0 + t, rowptr, diag, k0, cnt);
  }
  cnt = __reduce_max_sync(0xffffffffu, cnt);
  if((t & 31) == 0) width[slice0 + (t >> 5)] = cnt;
}

template <int UPPER>
__global__ void k_ell_fill(int r0, int w, int nsl, int slice0, const int *__restrict__ rows,
                           const int *__restrict__ rowptr, const int *__restrict__ col,
                           const int *__restrict__ diag, const int *__restrict__ width,
                           const long long *__restrict__ wscan, int *__restrict__ ecol,
                           int *__restrict__ esrc)
{
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= nsl * 32) return;
  int s = slice0 + (t >> 5), lane = t & 31;
  long long base = 32 * wscan[s] + lane;
  int W = width[s];
  int k0 = 0, cnt = 0;
  if(t < w) part_range<UPPER>(rows ? rows[r0 + t] : r0 + t, rowptr, diag, k0, cnt);
  for(int j = 0; j < W; j++) {
    bool in = j < cnt;
    ecol[base + 32LL * j] = in ? col[k0 + j] : -1;
    esrc[base + 32LL * j] = in ? k0 + j : -1;
  }
}

template <typename T>
__global__ void k_ell_vals(long long m, const int *__restrict__ src, const T *__restrict__ lu,
                           T *__restrict__ v)
{
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if(e < m) v[e] = src[e] >= 0 ? lu[src[e]] : (T)0;
}

template <int UPPER>
static int build_ell(gb300_matrix *A, const std::vector<Segment> &seg, const int *rows,
                     const int *diag, EllPart &E, cudaStream_t st)
{
  E.slice0.assign(seg.size(), -1);
  E.nslices = 0;
  for(size_t q = 0; q < seg.size(); q++)
    if(!seg[q].narrow) {
      E.slice0[q] = E.nslices;
      E.nslices += (seg[q].width + 31) / 32;
    }
  E.entries = 0;
  E.common.assign(seg.size(), 0);
  E.first.assign(seg.size(), 0);
  if(E.nslices == 0) return GB300_OK;
  GB_TRY(E.width.alloc(E.nslices));
  GB_TRY(E.wscan.alloc(E.nslices));
  for(size_t q = 0; q < seg.size(); q++)
    if(!seg[q].narrow) {
      int nsl = (seg[q].width + 31) / 32;
      k_ell_width<UPPER><<<grid_for((long long)nsl * 32, 256), 256, 0, st>>>(
        seg[q].r0, seg[q].width, nsl, E.slice0[q], rows, A->rowptr.p, diag, E.width.p);
    }
  // slices of a segment padded to its widest where that adds at most a quarter
  std::vector<int> w(E.nslices);
  GB_CUDA(cudaMemcpyAsync(w.data(), E.width.p, sizeof(int) * E.nslices, cudaMemcpyDeviceToHost,
                          st));
  GB_CUDA(cudaStreamSynchronize(st));
  long long at = 0;
  bool padded = false;
  for(size_t q = 0; q < seg.size(); q++) {
    if(seg[q].narrow) continue;
    const int s0 = E.slice0[q], nsl = (seg[q].width + 31) / 32;
    long long sum = 0;
    int most = 0;
    for(int t = s0; t < s0 + nsl; t++) {
      sum += w[t];
      most = std::max(most, w[t]);
    }
    E.first[q] = 32 * at;
    if(most > 0 && 4LL * most * nsl <= 5 * sum) {
      E.common[q] = most;
      std::fill(w.begin() + s0, w.begin() + s0 + nsl, most);
      sum = (long long)most * nsl;
      padded = true;
    }
    at += sum;
  }
  if(padded)
    GB_CUDA(cudaMemcpyAsync(E.width.p, w.data(), sizeof(int) * E.nslices,
                            cudaMemcpyHostToDevice, st));
  DevBuf<long long> tmp;
  long long total = 0;
  GB_TRY(exclusive_scan(E.width.p, E.nslices, E.wscan.p, &total, tmp, st));
  GB_CUDA(cudaStreamSynchronize(st));  // (total; w goes out of scope)
  E.entries = 32 * total;
  GB_TRY(E.col.alloc(E.entries > 0 ? E.entries : 1));
  GB_TRY(E.src.alloc(E.entries > 0 ? E.entries : 1));
  for(size_t q = 0; q < seg.size(); q++)
    if(!seg[q].narrow) {
      int nsl = (seg[q].width + 31) / 32;
      k_ell_fill<UPPER><<<grid_for((long long)nsl * 32, 256), 256, 0, st>>>(
        seg[q].r0, seg[q].width, nsl, E.slice0[q], rows, A->rowptr.p, A->col.p, diag,
        E.width.p, E.wscan.p, E.col.p, E.src.p);
    }
  GB_CUDA(cudaGetLastError());
  GB_CUDA(cudaStreamSynchronize(st));
  return GB300_OK;
}

// the factor's values in the ELL copies (after each factorisation)
template <typename T>
static int ell_values(EllPart &E, const T *lu, DevBuf<T> &v, cudaStream_t st)
{
  if(E.entries == 0) return GB300_OK;
  GB_TRY(v.alloc(E.entries));
  k_ell_vals<T><<<grid_for(E.entries, 256), 256, 0, st>>>(E.entries, E.src.p, lu, v.p);
  GB_CUDA(cudaGetLastError());
  return GB300_OK;
}

// the level schedule, diagonal positions and sliced-ELL structure of A's pattern
static int ilu_schedule(gb300_matrix *A, ilu_data *L)
{
  cudaStream_t st = A->ctx->stream;
  int n = A->n;
  DevBuf<int> indl, indu, err;
  GB_TRY(L->diag.alloc(n));
  GB_TRY(indl.alloc(n));
  GB_TRY(indu.alloc(n));
  GB_TRY(err.alloc(1));
  GB_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), st));
  k_ilu_prep<<<grid_for(n, 256), 256, 0, st>>>(n, A->rowptr.p, A->col.p,
                                                L->diag.p, indl.p, indu.p, err.p);
  int herr = 0;
  GB_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  if(herr & 1) {
    set_error("ILU(0): a row has no diagonal entry");
    return GB300_ERR_ZERO_PIVOT;
  }
  if(herr & 2) {
    set_error("ILU(0): the level schedule needs a structurally symmetric pattern");
    return GB300_ERR_UNSUPPORTED;
  }
  const Colouring *C = A->order;
  if(C && C->kind == 0 && C->bs == 1 && C->seg.size() == 2) {
    // first-fit colours: a row of colour c has neighbours of every smaller
    // colour, so the colours are the forward sweep's levels; backwards they
    // are a valid schedule of the same length
    L->by_colour = true;
    L->n0 = C->voff[1];
    for(int c = 0; c < C->ncolors; c++)
      L->lseg.push_back({c, c + 1, false, C->voff[c + 1] - C->voff[c], C->voff[c]});
    L->useg.assign(L->lseg.rbegin(), L->lseg.rend());
  }
  else {
    GB_TRY(make_levels<0>(A, L, indl.p, L->lrows, L->lptr, L->hlptr, L->lseg));
    GB_TRY(make_levels<1>(A, L, indu.p, L->urows, L->uptr, L->huptr, L->useg));
  }
  GB_TRY(build_ell<0>(A, L->lseg, L->lrows.p, L->diag.p, L->lell, st));
  GB_TRY(build_ell<1>(A, L->useg, L->urows.p, L->diag.p, L->uell, st));
  if(L->by_colour)
    GB_TRY(build_ell<2>(A, {{0, 0, false, n, 0}}, nullptr, L->diag.p, L->aell, st));
  return GB300_OK;
}

static int ilu_setup(gb300_matrix *A)
{
  // it belongs to one pattern
  if(A->ilu && A->ilu->n == A->n && A->ilu->version == A->pattern_version) return GB300_OK;
  if(A->ilu) ilu_free(A->ilu);
  A->ilu = nullptr;
  // (held by A once it is whole: a set-up that ran out of memory half way must
  // not pass for one at the next call)
  auto L = std::make_unique<ilu_data>();
  L->n = A->n;
  L->version = A->pattern_version;
  GB_TRY(ilu_schedule(A, L.get()));
  A->ilu = L.release();
  return GB300_OK;
}

// ---------------------------------------------------------------------------
// per-row work of the three level-scheduled sweeps
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void row_fact(int i, const int *__restrict__ rowptr,
                                         const int *__restrict__ col,
                                         const int *__restrict__ diag, T *lu,
                                         T *inv, int *zero_row)
{
  int s = rowptr[i], e = rowptr[i + 1], di = diag[i];
  for(int k = s; k < di; k++) {
    int kr = col[k];
    T l = lu[k] * inv[kr];  // tl = alu(j) * alu(jrow)
    lu[k] = l;
    int ks = diag[kr] + 1, ke = rowptr[kr + 1];
    int lo = k + 1;  // columns of row i beyond kr
    for(int kk = ks; kk < ke; kk++) {
      int c = col[kk];
      int pos = find_col(col, lo, e, c);
      if(pos >= 0) {
        lu[pos] = lu[pos] - l * lu[kk];
        lo = pos + 1;
      }
    }
  }
  T piv = lu[di];
  if(piv == (T)0) {
    atomicMin(zero_row, i + 1);
    inv[i] = (T)0;
  }
  else
    inv[i] = (T)(1.0 / (double)piv);
}

// T: the factor's storage type; X: the vectors' (and the arithmetic's) type
template <typename T, typename X = T>
__device__ __forceinline__ void row_fwd(int i, const int *__restrict__ rowptr,
                                        const int *__restrict__ col,
                                        const int *__restrict__ diag,
                                        const T *__restrict__ lu, const X *src, X *x)
{
  X s = src[i];  // the right-hand side's entry (src may be x itself)
  for(int k = rowptr[i]; k < diag[i]; k++) s = s - (X)lu[k] * x[col[k]];
  x[i] = s;
}

template <typename T, typename X = T>
__device__ __forceinline__ void row_bwd(int i, const int *__restrict__ rowptr,
                                        const int *__restrict__ col,
                                        const int *__restrict__ diag,
                                        const T *__restrict__ lu,
                                        const T *__restrict__ inv, X *x)
{
  X s = x[i];
  for(int k = diag[i] + 1; k < rowptr[i + 1]; k++) s = s - (X)lu[k] * x[col[k]];
  x[i] = (X)inv[i] * s;
}

// MODE 0 factor, 1 forward solve, 2 backward solve
template <int MODE, typename T, typename X = T>
__global__ void __launch_bounds__(kNarrowThreads)
k_levels_narrow(int l0, int l1, const int *__restrict__ lptr,
                const int *__restrict__ rows, const int *__restrict__ rowptr,
                const int *__restrict__ col, const int *__restrict__ diag,
                T *lu, T *inv, X *x, int *zero_row, const int *flag,
                const unsigned char *__restrict__ rmask, const X *src)
{
  if(flag && !*flag) return;
  for(int l = l0; l < l1; l++) {
    int a = lptr[l], b = lptr[l + 1];
    for(int t = a + threadIdx.x; t < b; t += blockDim.x) {
      int i = rows[t];
      if(MODE != 0 && rmask && !rmask[i]) continue;
      if(MODE == 0)
        row_fact<T>(i, rowptr, col, diag, lu, inv, zero_row);
      else if(MODE == 1)
        row_fwd<T, X>(i, rowptr, col, diag, lu, src, x);
      else
        row_bwd<T, X>(i, rowptr, col, diag, lu, inv, x);
    }
    __syncthreads();
  }
}

template <int MODE, typename T, typename X = T>
__global__ void __launch_bounds__(256)
k_level_wide(int r0, int width, const int *__restrict__ rows,
             const int *__restrict__ rowptr, const int *__restrict__ col,
             const int *__restrict__ diag, T *lu, T *inv, X *x, int *zero_row,
             const int *flag, const unsigned char *__restrict__ rmask, const X *src)
{
  if(flag && !*flag) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= width) return;
  int i = rows ? rows[r0 + t] : r0 + t;
  if(MODE != 0 && rmask && !rmask[i]) return;
  if(MODE == 0)
    row_fact<T>(i, rowptr, col, diag, lu, inv, zero_row);
  else if(MODE == 1)
    row_fwd<T, X>(i, rowptr, col, diag, lu, src, x);
  else
    row_bwd<T, X>(i, rowptr, col, diag, lu, inv, x);
}

// one wide level of a triangular solve from the sliced-ELL copy: entry j
// of the warp's 32 rows is one coalesced load (the row's entries stay in
// CSR order, the accumulation order of lusol)
template <int MODE, typename T, typename X = T>
__global__ void __launch_bounds__(256)
k_level_ell(int r0, int w, int slice0, const int *__restrict__ rows,
            const int *__restrict__ width, const long long *__restrict__ wscan,
            const int *__restrict__ ecol, const T *__restrict__ ev,
            const T *__restrict__ inv, X *x, const int *flag,
            const unsigned char *__restrict__ rmask, const X *src)
{
  if(flag && !*flag) return;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if(t >= w) return;
  int i = rows ? rows[r0 + t] : r0 + t;
  if(rmask && !rmask[i]) return;
  int s = slice0 + (t >> 5);
  long long e = 32 * wscan[s] + (t & 31);
  int W = width[s];
  X acc = (MODE == 1) ? src[i] : x[i];
  for(int j = 0; j < W; j++, e += 32) {
    const int c = ecol[e];
    if(c >= 0) acc = acc - (X)ev[e] * x[c];
  }
  x[i] = (MODE == 2) ? (X)inv[i] * acc : acc;
}

template <typename T> const T *ell_vals(const EllPart &E);
template <> const double *ell_vals<double>(const EllPart &E) { return E.v64.p; }
template <> const float *ell_vals<float>(const EllPart &E) { return E.v32.p; }

// rmask (sweeps only): rows with rmask[i] == 0 are skipped (the rows of
// systems of a batch that have stopped)
template <int MODE, typename T, typename X = T>
// MODE 1 reads the right-hand side from src (x when null) and writes x
static void run_levels(const gb300_matrix *A, const ilu_data *L, T *lu, T *inv,
                       X *x, int *zero_row, const int *flag, cudaStream_t st,
                       const unsigned char *rmask = nullptr, const X *src = nullptr)
{
  if(!src) src = x;
  bool upper = (MODE == 2);
  const std::vector<Segment> &seg = upper ? L->useg : L->lseg;
  const int *rows = upper ? L->urows.p : L->lrows.p;
  const int *lptr = upper ? L->uptr.p : L->lptr.p;
  const EllPart &E = upper ? L->uell : L->lell;
  for(size_t q = 0; q < seg.size(); q++) {
    const Segment &s = seg[q];
    if(MODE != 0 && !s.narrow && E.entries > 0) {
      k_level_ell<MODE, T, X><<<grid_for(s.width, 256), 256, 0, st>>>(
        s.r0, s.width, E.slice0[q], rows, E.width.p, E.wscan.p, E.col.p,
        ell_vals<T>(E), inv, x, flag, rmask, src);
      continue;
    }
    if(s.narrow)
      k_levels_narrow<MODE, T, X><<<1, kNarrowThreads, 0, st>>>(
        s.l0, s.l1, lptr, rows, A->rowptr.p, A->col.p, L->diag.p, lu, inv, x,
        zero_row, flag, rmask, src);
    else
      k_level_wide<MODE, T, X><<<grid_for(s.width, 256), 256, 0, st>>>(
        s.r0, s.width, rows, A->rowptr.p, A->col.p, L->diag.p, lu, inv, x,
        zero_row, flag, rmask, src);
  }
}

template <typename TO, typename TI>
__global__ void k_cvt(long long n, const TI *__restrict__ in, TO *__restrict__ out,
                      const int *flag)
{
  if(flag && !*flag) return;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if(i < n) out[i] = (TO)in[i];
}

// factor A's values (val) into the ILU(0) of the requested precision; with
// reuse, a factor of that precision already held for A's pattern is kept
// (Re_Use_LU, as LinAlg_SolveAgain sets it: LinAlg_SPARSKIT.cpp:578-585)
int ilu_factor(gb300_matrix *A, const double *val, bool fp32, int *zero_row_out,
               bool reuse, int *factorized)
{
  GB_TRY(ilu_setup(A));
  ilu_data *L = A->ilu;
  if(factorized) *factorized = 0;
  if(reuse && (fp32 ? L->fact32 : L->fact64)) {
    *zero_row_out = 0;
    return GB300_OK;
  }
  if(factorized) *factorized = 1;
  L->fact32 = L->fact64 = false;
  cudaStream_t st = A->ctx->stream;
  int n = A->n;
  DevBuf<int> zr;
  GB_TRY(zr.alloc(1));
  int big = 0x7fffffff;
  GB_CUDA(cudaMemcpyAsync(zr.p, &big, sizeof(int), cudaMemcpyHostToDevice, st));
  if(!fp32) {
    GB_TRY(L->lu64.alloc(A->nnz));
    GB_TRY(L->inv64.alloc(n));
    GB_CUDA(cudaMemcpyAsync(L->lu64.p, val, sizeof(double) * A->nnz,
                            cudaMemcpyDeviceToDevice, st));
    run_levels<0, double>(A, L, L->lu64.p, L->inv64.p, (double *)nullptr, zr.p,
                          nullptr, st);
    GB_TRY(ell_values<double>(L->lell, L->lu64.p, L->lell.v64, st));
    GB_TRY(ell_values<double>(L->uell, L->lu64.p, L->uell.v64, st));
  }
  else {
    GB_TRY(L->lu32.alloc(A->nnz));
    GB_TRY(L->inv32.alloc(n));
    k_cvt<float, double><<<grid_for(A->nnz, 256), 256, 0, st>>>(A->nnz, val,
                                                                L->lu32.p, nullptr);
    run_levels<0, float>(A, L, L->lu32.p, L->inv32.p, (float *)nullptr, zr.p,
                         nullptr, st);
    GB_TRY(ell_values<float>(L->lell, L->lu32.p, L->lell.v32, st));
    GB_TRY(ell_values<float>(L->uell, L->lu32.p, L->uell.v32, st));
  }
  int hz = 0;
  GB_CUDA(cudaMemcpyAsync(&hz, zr.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  GB_CUDA(cudaGetLastError());
  *zero_row_out = (hz == big) ? 0 : hz;
  if(!*zero_row_out) (fp32 ? L->fact32 : L->fact64) = true;
  return GB300_OK;
}

// The sweeps on a multicolour copy, one launch per colour in a chain
// (launch_chain): forward through the colours, the last colour's rows
// finished at once (they have no upper entries), then backward to colour 0.
// Colour 0 has no lower entries, so its forward values are the right-hand
// side itself, which the other colours read in place: 2 C - 2 launches
// instead of 2 C, and no pass that converts the vector.  A row's first
// kSweepU entries and its pivot are loaded before the wait for the preceding
// colour, and the guard is tested once the gathers are on their way: one
// memory latency and a store remain of each colour.  kSweepU is 4 or 6 where all
// slices of the colour are that narrow (fewer registers, so more of a large
// colour's rows are in flight at once: 9.0 -> 5.8 us at 262,000 rows), else 8.
// Both sweeps at 1,046,529 rows, 4 colours: 94 us.  The accumulation order is
// that of lusol.
//   PART 0: forward, x = value          PART 1: last colour, both sweeps
//   PART 2: backward, from x            PART 3: backward, from src (colour 0)
// OUT 1: final values also to z as doubles; 2: added into z
template <int PART, int OUT, typename T, typename X, int kSweepU>
__global__ void __launch_bounds__(256)
k_colour_sweep(int r0, int w, int slice0, int common, long long first,
               const int *__restrict__ width,
               const long long *__restrict__ wscan, const int *__restrict__ ecol,
               const T *__restrict__ ev, const T *__restrict__ inv, int n0, const double *src,
               X *x, double *z, const int *flag)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = r0 + t;
  int W = 0;
  long long e = 0;
  T iv = (T)0, v[kSweepU];
  int c[kSweepU];
  if(t < w) {
    const int s = t >> 5;
    W = common > 0 ? common : width[slice0 + s];
    e = common > 0 ? first + 32LL * common * s : 32 * wscan[slice0 + s];
    e += t & 31;
    if(PART != 0) iv = inv[i];
  }
#pragma unroll
  for(int u = 0; u < kSweepU; u++) {
    c[u] = u < W ? ecol[e + 32 * u] : -1;
    v[u] = u < W ? ev[e + 32 * u] : (T)0;
  }
  chain_wait();
  if(t >= w) return;
  const int go = flag ? *flag : 1;
  X acc = PART == 2 ? x[i] : (X)src[i];
  auto gather = [&](int cc) -> X {
    if(PART < 2 && cc < n0) return (X)src[cc];
    return x[cc];
  };
  X xv[kSweepU];
#pragma unroll
  for(int u = 0; u < kSweepU; u++) xv[u] = c[u] >= 0 ? gather(c[u]) : (X)0;
  if(!go) return;
#pragma unroll
  for(int u = 0; u < kSweepU; u++)
    if(c[u] >= 0) acc = acc - (X)v[u] * xv[u];
  for(int j = kSweepU; j < W; j += kSweepU) {  // longer rows, as many at a time
    e += 32 * kSweepU;
#pragma unroll
    for(int u = 0; u < kSweepU; u++) {
      c[u] = j + u < W ? ecol[e + 32 * u] : -1;
      v[u] = j + u < W ? ev[e + 32 * u] : (T)0;
    }
#pragma unroll
    for(int u = 0; u < kSweepU; u++) xv[u] = c[u] >= 0 ? gather(c[u]) : (X)0;
#pragma unroll
    for(int u = 0; u < kSweepU; u++)
      if(c[u] >= 0) acc = acc - (X)v[u] * xv[u];
  }
  if(PART != 0) acc = (X)iv * acc;
  x[i] = acc;
  if(PART != 0 && OUT == 1) z[i] = (double)acc;
  if(PART != 0 && OUT == 2) z[i] += (double)acc;
}

template <int OUT, typename T, typename X>
static void colour_sweeps(const ilu_data *L, const T *inv, const double *src, X *x, double *z,
                          const int *flag, cudaStream_t st)
{
  const int C = (int)L->lseg.size();
  auto go = [&](auto u4, auto u6, auto u8, const EllPart &E, const std::vector<Segment> &seg,
                int q) {
    const Segment &g = seg[q];
    const int cw = E.common[q];
    launch_chain(chain_early(L->n), cw > 0 && cw <= 4 ? u4 : cw > 0 && cw <= 6 ? u6 : u8,
                 grid_for(g.width, 256), 256, st, g.r0, g.width, E.slice0[q], E.common[q],
                 E.first[q], E.width.p, E.wscan.p, E.col.p, ell_vals<T>(E), inv, L->n0, src, x,
                 z, flag);
  };
#define GB_SWEEP(PART, E, seg, q) \
  go(k_colour_sweep<PART, OUT, T, X, 4>, k_colour_sweep<PART, OUT, T, X, 6>,      \
     k_colour_sweep<PART, OUT, T, X, 8>, E, seg, q)
  for(int c = 1; c < C - 1; c++) GB_SWEEP(0, L->lell, L->lseg, c);
  GB_SWEEP(1, L->lell, L->lseg, C - 1);
  for(int q = 1; q < C; q++) {  // useg[q] is colour C - 1 - q
    if(q < C - 1)
      GB_SWEEP(2, L->uell, L->useg, q);
    else
      GB_SWEEP(3, L->uell, L->useg, q);
  }
#undef GB_SWEEP
}

// A multicolour copy's products, one thread per row of a sliced-ELL copy of
// A: GB300's FP64 pipe, not memory, bounds them from ~500,000 rows on (14 us
// for the 7.3 M FMAs at 1,046,529 rows), and a row shared by two lanes issues
// 10 FP64 instructions per 32 rows of 7 entries where a thread per row issues 7
template <int MODE, int U>
__global__ void __launch_bounds__(256)
k_ell_chain(int n, int common, const int *__restrict__ width,
            const long long *__restrict__ wscan,
            const int *__restrict__ ecol, const double *__restrict__ ev, ChainArgs a)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int W = 0, c[U], g[U], grow = 0;
  long long e = 0;
  double v[U];
  if(i < n) {
    W = common > 0 ? common : width[i >> 5];
    e = (common > 0 ? 32LL * common * (i >> 5) : 32 * wscan[i >> 5]) + (i & 31);
    if(MODE == kChainProlong) grow = a.agg[i];
  }
#pragma unroll
  for(int u = 0; u < U; u++) {
    c[u] = u < W ? ecol[e + 32 * u] : -1;
    v[u] = u < W ? ev[e + 32 * u] : 0.;
    if(MODE == kChainProlong) g[u] = c[u] >= 0 ? a.agg[c[u]] : 0;
  }
  chain_wait();
  if(i >= n) return;
  const int go = a.flag ? *a.flag : 1;
  double xv[U];
#pragma unroll
  for(int u = 0; u < U; u++) {
    xv[u] = c[u] >= 0 ? a.x[c[u]] : 0.;
    if(MODE == kChainProlong && c[u] >= 0) xv[u] += a.ec[g[u]];
  }
  if(!go) return;
  double sum = 0.;
#pragma unroll
  for(int u = 0; u < U; u++)
    if(c[u] >= 0) sum += v[u] * xv[u];
  for(int j = U; j < W; j += U) {
    e += 32 * U;
#pragma unroll
    for(int u = 0; u < U; u++) {
      c[u] = j + u < W ? ecol[e + 32 * u] : -1;
      v[u] = j + u < W ? ev[e + 32 * u] : 0.;
      if(MODE == kChainProlong) g[u] = c[u] >= 0 ? a.agg[c[u]] : 0;
    }
#pragma unroll
    for(int u = 0; u < U; u++) {
      xv[u] = c[u] >= 0 ? a.x[c[u]] : 0.;
      if(MODE == kChainProlong && c[u] >= 0) xv[u] += a.ec[g[u]];
    }
#pragma unroll
    for(int u = 0; u < U; u++)
      if(c[u] >= 0) sum += v[u] * xv[u];
  }
  chain_store<MODE>(a, i, grow, sum);
}

// Small systems: both sweeps and the product in one CTA, a row per thread and
// x in shared memory.  A launch per colour costs some 2 us whatever its rows
// (launch, guard, gather, store); a colour here costs a shared gather, a short
// FMA chain and a barrier, its entries loaded during the colour before: 5.4 us
// at 529 rows against 9 for the chain.  One SM's FP64 pipe sets the limit.
// Solve per GMRES step, set-up included, chain / this kernel: 65 / 48 us at 81
// rows, 38 / 34 at 529, 40 / 36 at 961; with two rows a thread 35.6 / 36.7 at
// 1,225 and 33 / 36 at 1,521, so the line lies at one.
constexpr int kSmallRows = 1024, kSmallColours = 12;
struct SmallStep {
  int n, C;
  int r0[kSmallColours + 1];                    // rows of colour c
  int lslice[kSmallColours], uslice[kSmallColours];
};

template <typename T, typename X>
__global__ void __launch_bounds__(kSmallRows)
k_small_step(SmallStep P, const int *__restrict__ lw, const long long *__restrict__ ls,
             const int *__restrict__ lc, const T *__restrict__ lv, const int *__restrict__ uw,
             const long long *__restrict__ us, const int *__restrict__ uc,
             const T *__restrict__ uv, const T *__restrict__ inv, const int *__restrict__ aw,
             const long long *__restrict__ as, const int *__restrict__ ac,
             const double *__restrict__ av, const double *src, double *z, double *y,
             const int *flag)
{
  constexpr int U = 6;
  __shared__ X x[kSmallRows];
  int c[U], W = 0;
  T v[U];
  long long e = 0;
  auto load = [&](int slice0, int t, bool in, const int *width, const long long *scan,
                  const int *col, const T *val) {
    W = in ? width[slice0 + (t >> 5)] : 0;
    e = in ? 32 * scan[slice0 + (t >> 5)] + (t & 31) : 0;
#pragma unroll
    for(int u = 0; u < U; u++) {
      c[u] = u < W ? col[e + 32 * u] : -1;
      v[u] = u < W ? val[e + 32 * u] : (T)0;
    }
  };
  auto apply = [&](X acc, const int *col, const T *val) {
#pragma unroll
    for(int u = 0; u < U; u++)
      if(c[u] >= 0) acc = acc - (X)v[u] * x[c[u]];
    for(int j = U; j < W; j++) {
      const int cc = col[e + 32LL * j];
      if(cc >= 0) acc = acc - (X)val[e + 32LL * j] * x[cc];
    }
    return acc;
  };
  const int t = threadIdx.x, C = P.C;
  auto rows = [&](int cc) { return P.r0[cc + 1] - P.r0[cc]; };
  if(C > 1) load(P.lslice[1], t, t < rows(1), lw, ls, lc, lv);
  chain_wait();
  if(flag && !*flag) return;  // the same in every thread
  if(t < P.n) x[t] = (X)src[t];
  __syncthreads();
  for(int cc = 1; cc < C; cc++) {
    const int i = P.r0[cc] + t;
    const bool in = t < rows(cc);
    X s = in ? apply(x[i], lc, lv) : (X)0;
    if(cc + 1 < C)
      load(P.lslice[cc + 1], t, t < rows(cc + 1), lw, ls, lc, lv);
    else {  // no upper entries
      load(P.uslice[C - 2], t, t < rows(C - 2), uw, us, uc, uv);
      if(in) s = (X)inv[i] * s;
    }
    if(in) x[i] = s;
    __syncthreads();
  }
  if(C == 1) {  // no sweeps: the copy is diagonal
    if(t < P.n) x[t] = (X)inv[t] * x[t];
    __syncthreads();
  }
  for(int cc = C - 2; cc >= 0; cc--) {
    const int i = P.r0[cc] + t;
    if(t < rows(cc)) x[i] = (X)inv[i] * apply(x[i], uc, uv);
    if(cc > 0) load(P.uslice[cc - 1], t, t < rows(cc - 1), uw, us, uc, uv);
    __syncthreads();
  }
  if(t >= P.n) return;
  z[t] = (double)x[t];
  if(!y) return;
  const int w = aw[t >> 5];
  const long long b = 32 * as[t >> 5] + (t & 31);
  double s = 0.;
#pragma unroll 8
  for(int j = 0; j < w; j++) {
    const int cc = ac[b + 32LL * j];
    if(cc >= 0) s += av[b + 32LL * j] * (double)x[cc];
  }
  y[t] = s;
}

// z = M^-1 v and, with y, y = A z for the plain ILU(0) of a small multicolour
// copy; false (nothing launched) where that form does not apply
static bool small_step(const gb300_matrix *A, const double *val, int mode, const double *v,
                       double *z, double *y, const int *flag, cudaStream_t st)
{
  const ilu_data *L = A->ilu;
  if(!L || !L->by_colour || L->aell_of != val || A->n > kSmallRows ||
     (int)L->lseg.size() > kSmallColours)
    return false;
  SmallStep P = {};
  P.n = A->n;
  P.C = (int)L->lseg.size();
  for(int c = 0; c < P.C; c++) {
    P.r0[c] = L->lseg[c].r0;
    P.lslice[c] = L->lell.slice0[c];
    P.uslice[c] = L->uell.slice0[P.C - 1 - c];  // useg[q] is colour C - 1 - q
  }
  P.r0[P.C] = P.n;
  auto go = [&](auto kernel, const auto *lv, const auto *uv, const auto *inv) {
    launch_chain(true, kernel, 1, (A->n + 31) / 32 * 32, st, P, L->lell.width.p, L->lell.wscan.p,
                 L->lell.col.p, lv, L->uell.width.p, L->uell.wscan.p, L->uell.col.p, uv, inv,
                 L->aell.width.p, L->aell.wscan.p, L->aell.col.p, L->aell.v64.p, v, z, y, flag);
  };
  if(mode == 0)
    go(k_small_step<double, double>, L->lell.v64.p, L->uell.v64.p, L->inv64.p);
  else if(mode == 2)
    go(k_small_step<float, double>, L->lell.v32.p, L->uell.v32.p, L->inv32.p);
  else
    go(k_small_step<float, float>, L->lell.v32.p, L->uell.v32.p, L->inv32.p);
  return true;
}

int ilu_products(gb300_matrix *A, const double *val)
{
  ilu_data *L = A->ilu;
  if(!L || !L->by_colour) return GB300_OK;
  L->aell_of = nullptr;
  GB_TRY(ell_values<double>(L->aell, val, L->aell.v64, A->ctx->stream));
  L->aell_of = val;
  return GB300_OK;
}

void product_chain(ChainMode mode, const gb300_matrix *A, const double *val,
                   const ChainArgs &a, cudaStream_t st)
{
  const ilu_data *L = A->ilu;
  if(!L || !L->by_colour || L->aell_of != val || L->aell.entries == 0) {
    spmv_chain(mode, A, val, a, st);
    return;
  }
  const EllPart &E = L->aell;
  auto go = [&](auto u7, auto u8) {  // (7: 2D meshes, fewer registers)
    launch_chain(chain_early(A->n), E.common[0] == 7 ? u7 : u8, grid_for(A->n, 256), 256, st,
                 A->n, E.common[0],
                 E.width.p, E.wscan.p, E.col.p, E.v64.p, a);
  };
  switch(mode) {
  case kChainMul: go(k_ell_chain<kChainMul, 7>, k_ell_chain<kChainMul, 8>); break;
  case kChainAdd: go(k_ell_chain<kChainAdd, 7>, k_ell_chain<kChainAdd, 8>); break;
  case kChainRes: go(k_ell_chain<kChainRes, 7>, k_ell_chain<kChainRes, 8>); break;
  case kChainProlong: go(k_ell_chain<kChainProlong, 7>, k_ell_chain<kChainProlong, 8>); break;
  case kChainAddBoth: go(k_ell_chain<kChainAddBoth, 7>, k_ell_chain<kChainAddBoth, 8>); break;
  }
}

// z = M^-1 v for the ILU(0) factor: mode 0 FP64 factor and sweeps; 1 FP32
// factor, sweeps on FP32 vectors in FP32 arithmetic; 2 FP32 factor, sweeps
// in FP64 (the reference built with HAVE_ILU_FLOAT: lusol's float alu
// against double x, ilut.F:2297-2347)
void ilu_apply(const gb300_matrix *A, int mode, const double *v, double *z,
               float *t32, const int *flag, cudaStream_t st,
               const unsigned char *rmask)
{
  const ilu_data *L = A->ilu;
  int n = A->n;
  if(mode == 0) {
    // the forward sweep reads v and writes z (no copy of v first); rows a
    // mask leaves out are not written
    run_levels<1, double>(A, L, (double *)L->lu64.p, (double *)L->inv64.p, z,
                          nullptr, flag, st, rmask, v);
    run_levels<2, double>(A, L, (double *)L->lu64.p, (double *)L->inv64.p, z,
                          nullptr, flag, st, rmask);
  }
  else if(mode == 2) {
    run_levels<1, float, double>(A, L, (float *)L->lu32.p, (float *)L->inv32.p, z, nullptr,
                                 flag, st, rmask, v);
    run_levels<2, float, double>(A, L, (float *)L->lu32.p, (float *)L->inv32.p, z, nullptr,
                                 flag, st, rmask);
  }
  else {
    k_cvt<float, double><<<grid_for(n, 256), 256, 0, st>>>(n, v, t32, flag);
    run_levels<1, float>(A, L, (float *)L->lu32.p, (float *)L->inv32.p, t32,
                         nullptr, flag, st, rmask);
    run_levels<2, float>(A, L, (float *)L->lu32.p, (float *)L->inv32.p, t32,
                         nullptr, flag, st, rmask);
    k_cvt<double, float><<<grid_for(n, 256), 256, 0, st>>>(n, t32, z, flag);
  }
}

// one sweep's levels cut into the diagonal blocks off[0..nsys]: the rows of
// each level go, in level order, to their system's range of out, and each
// system records where its levels begin (a system's rows occupy the same
// range [off[p], off[p+1]) in out as in the matrix)
static void cut_levels(int n, int nsys, const int *off, const std::vector<int> &rows,
                       const std::vector<int> &lptr, std::vector<int> &out,
                       std::vector<int> &lev, std::vector<int> &lb, int *max_levels)
{
  std::vector<int> sys_of(n), fill(nsys), last(nsys, -1);
  std::vector<std::vector<int>> starts(nsys);
  for(int q = 0; q < nsys; q++) {
    fill[q] = off[q];
    for(int i = off[q]; i < off[q + 1]; i++) sys_of[i] = q;
  }
  out.assign(n, 0);
  const int nl = (int)lptr.size() - 1;
  for(int l = 0; l < nl; l++)
    for(int t = lptr[l]; t < lptr[l + 1]; t++) {
      int i = rows[t], q = sys_of[i];
      if(last[q] != l) {
        starts[q].push_back(fill[q]);
        last[q] = l;
      }
      out[fill[q]++] = i;
    }
  lev.clear();
  lb.assign(nsys + 1, 0);
  for(int q = 0; q < nsys; q++) {
    lb[q] = (int)lev.size();
    lev.insert(lev.end(), starts[q].begin(), starts[q].end());
    lev.push_back(off[q + 1]);
    *max_levels = std::max(*max_levels, (int)starts[q].size());
  }
  lb[nsys] = (int)lev.size();
}

int ilu_sys_levels(gb300_matrix *A, int nsys, const int *off, const SysLevels **out)
{
  GB_TRY(ilu_setup(A));
  ilu_data *L = A->ilu;
  if(L->by_colour) {  // (its callers go by the colours)
    set_error("ILU(0): no level lists on a multicolour copy");
    return GB300_ERR_UNSUPPORTED;
  }
  if(L->sys && (int)L->sys->off.size() == nsys + 1 &&
     std::equal(off, off + nsys + 1, L->sys->off.begin())) {
    *out = L->sys.get();
    return GB300_OK;
  }
  cudaStream_t st = A->ctx->stream;
  const int n = A->n;
  std::vector<int> lr(n), ur(n);
  if(n > 0) {
    GB_CUDA(cudaMemcpyAsync(lr.data(), L->lrows.p, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaMemcpyAsync(ur.data(), L->urows.p, sizeof(int) * n, cudaMemcpyDeviceToHost, st));
  }
  GB_CUDA(cudaStreamSynchronize(st));
  auto S = std::make_unique<SysLevels>();
  S->off.assign(off, off + nsys + 1);
  std::vector<int> lo, uo, llev, ulev, llb, ulb;
  cut_levels(n, nsys, off, lr, L->hlptr, lo, llev, llb, &S->max_levels);
  cut_levels(n, nsys, off, ur, L->huptr, uo, ulev, ulb, &S->max_levels);
  auto up = [&](DevBuf<int> &d, const std::vector<int> &h) -> int {
    GB_TRY(d.alloc(h.size() > 0 ? h.size() : 1));
    if(!h.empty())
      GB_CUDA(cudaMemcpyAsync(d.p, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice, st));
    return GB300_OK;
  };
  GB_TRY(up(S->lrows, lo));
  GB_TRY(up(S->urows, uo));
  GB_TRY(up(S->llev, llev));
  GB_TRY(up(S->ulev, ulev));
  GB_TRY(up(S->llb, llb));
  GB_TRY(up(S->ulb, ulb));
  GB_CUDA(cudaStreamSynchronize(st));  // the host vectors go out of scope
  L->sys = std::move(S);
  *out = L->sys.get();
  return GB300_OK;
}

// the factor held for A (after ilu_factor): values, inverted pivots and the
// position of each diagonal entry
void ilu_factor_arrays(const gb300_matrix *A, bool fp32, const void **lu, const void **inv,
                       const int **diag)
{
  const ilu_data *L = A->ilu;
  *lu = fp32 ? (const void *)L->lu32.p : (const void *)L->lu64.p;
  *inv = fp32 ? (const void *)L->inv32.p : (const void *)L->inv64.p;
  *diag = L->diag.p;
}

// ---------------------------------------------------------------------------
// GMRES device state and kernels
// ---------------------------------------------------------------------------
constexpr int kMaxKrylov = 128;
constexpr int kDotCols = 8;  // columns of one group of dot products

struct GmState {
  int active;       // whole solve still running
  int cycle;        // current restart cycle still extending the basis
  int did_cycle;    // the cycle took >= 1 Arnoldi step (solution update due)
  int k;            // Arnoldi steps taken in the cycle
  int its;          // ipar(7)
  int maxit;        // ipar(6)
  int status;       // ipar(1)
  int breakdown;    // ipar(12) (-3: linear combination, -1/-2 bad vector)
  int first;        // first restart still to come
  double tol;       // fpar(4)
  double res0;      // fpar(3)
  double res;       // fpar(5)
  double res6;      // fpar(6)
  double rtol;
  double scale;     // 1 / ||r|| at a restart (V_0 is normalised)
  // vector j of the algorithm is sc[j] V_j: the basis vectors are left with
  // the norm h(j+1,j) they come out of the Gram-Schmidt step with, the
  // preconditioner and the product act on them as they are, and the scalars
  // carry the normalisation (no pass over the vector scales it)
  double sc[kMaxKrylov + 1];
  double H[(kMaxKrylov + 1) * kMaxKrylov];  // column-major, (m+1) x m
  double cs[kMaxKrylov], sn[kMaxKrylov], g[kMaxKrylov + 1], y[kMaxKrylov];
  double h1[kMaxKrylov + 1], h2[kMaxKrylov + 1];  // the column of each pass
  double nrm0;      // ||w||^2 before the Gram-Schmidt pass of this step
  int reorth;       // this step takes a second Gram-Schmidt pass
  // arrival counters of the kernels whose last CTA finishes a reduction
  unsigned tick_dots[2][kMaxKrylov / kDotCols + 1], tick_upd[2];
};

// restart: r = rhs - A x was computed with its partial norms
__global__ void k_gm_restart(GmState *S, const double *__restrict__ part, int m)
{
  if(!S->active) return;
  double rr = 0.;
  for(int i = threadIdx.x; i < kReduceBlocks; i += blockDim.x) rr += part[i];
  rr = block_sum<double, 256>(rr);
  if(threadIdx.x) return;
  S->its += 1;
  double alpha = sqrt(rr);
  if(S->first) {
    S->tol = S->rtol * alpha + 0.0;
    S->res0 = alpha;
    S->first = 0;
  }
  S->res = alpha;
  S->g[0] = alpha;
  S->k = 0;
  S->did_cycle = 0;
  S->breakdown = 0;
  // iters.f's restart test: converged when alpha <= tol (also for a zero
  // right-hand side); a NaN residual goes on to the Arnoldi step, where the
  // abnormal norm ends the solve as a break-down
  if(alpha <= S->tol) {
    S->status = 0;
    S->res6 = alpha;
    S->active = 0;
    S->cycle = 0;
    return;
  }
  S->scale = 1. / alpha;
  S->sc[0] = 1.;
  S->cycle = 1;
}

// y = x, or y = y2 = s x with s = *scale, guarded by *flag
__global__ void k_gm_scale(int n, const double *scale, const double *x, double *y, double *y2,
                           const int *flag)
{
  chain_wait();
  if(flag && !*flag) return;
  const double s = scale ? *scale : 1.;
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += (long long)gridDim.x * blockDim.x) {
    const double v = scale ? s * x[i] : x[i];
    y[i] = v;
    if(y2) y2[i] = v;
  }
}

__global__ void k_gm_add(int n, const double *t, double *z, const int *flag)
{
  chain_wait();
  if(flag && !*flag) return;
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += (long long)gridDim.x * blockDim.x)
    z[i] += t[i];
}

// The dot products <V_j, w>, j < k, of one Gram-Schmidt pass, k - 1 the steps
// taken in this cycle (read from the state, so that one captured step serves
// them all).  The CTAs are dealt to groups of at most kDotCols columns (the
// groups as even as they can be), which run side by side, and within a group
// to shares of the rows, the partial of column j and share b in
// part[j * kReduceBlocks + b]; CTAs left over return.  PASS 0 also forms <w, w> (column k:
// V_k is w), the norm the selective re-orthogonalisation compares with; PASS
// 1 runs only when this step takes the second pass.  The last CTA of each
// group sums its columns, one warp per column, in a fixed order (one CTA
// summing every group's had been 10 of 22 us at 65,025 rows and k = 49).
// Bound by the FP64 pipe: a warp's block sum costs as many FP64 instructions
// as two rows of a group, so the grid is one CTA per SM over all groups.
template <int CNT>
__device__ __forceinline__ void dots_group(int n, int j0, int k, int share, int shares,
                                           const double *V, size_t ldv, const double *w,
                                           double *part)
{
  double acc[kDotCols], x[CNT], wi = 0.;
#pragma unroll
  for(int u = 0; u < kDotCols; u++) acc[u] = 0.;
  const int stride = shares * blockDim.x;
  const double *Vj = V + (size_t)j0 * ldv;
  int i = share * blockDim.x + threadIdx.x;
  auto load = [&]() {
    wi = i < n ? w[i] : 0.;
#pragma unroll
    for(int u = 0; u < CNT; u++)  // column k is w
      x[u] = i < n ? (u == CNT - 1 && j0 + u == k ? wi : Vj[(size_t)u * ldv + i]) : 0.;
  };
  load();
  while(i < n) {
    double xc[CNT], wc = wi;
#pragma unroll
    for(int u = 0; u < CNT; u++) xc[u] = x[u];
    i += stride;
    load();  // the next row, in flight during this one's FMAs
#pragma unroll
    for(int u = 0; u < CNT; u++) acc[u] += xc[u] * wc;
  }
  const double s = block_sum8<256>(acc);
  if(threadIdx.x < CNT) part[(size_t)(j0 + threadIdx.x) * kReduceBlocks + share] = s;
}

template <int PASS>
__global__ void __launch_bounds__(256)
k_gm_dots(int n, const double *V, size_t ldv, const double *w, double *part, GmState *S)
{
  chain_wait();
  const int go = S->cycle, again = S->reorth, k = S->k + 1;
  if(!go || (PASS == 1 && !again)) return;  // the same in every CTA
  const int kk = PASS == 0 ? k + 1 : k;     // column k: V_k = w itself
  const int groups = (kk - 1) / kDotCols + 1;
  const int grp = (int)blockIdx.x % groups, share = (int)blockIdx.x / groups;
  const int rows256 = (n + 255) / 256, most = (int)gridDim.x / groups;
  const int shares = rows256 < most ? rows256 : most;
  if(share >= shares) return;
  const int j0 = grp * kk / groups;
  const int cnt = (grp + 1) * kk / groups - j0;
  switch(cnt) {
  case 1: dots_group<1>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 2: dots_group<2>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 3: dots_group<3>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 4: dots_group<4>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 5: dots_group<5>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 6: dots_group<6>(n, j0, k, share, shares, V, ldv, w, part); break;
  case 7: dots_group<7>(n, j0, k, share, shares, V, ldv, w, part); break;
  default: dots_group<8>(n, j0, k, share, shares, V, ldv, w, part); break;
  }
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31, j = j0 + wp;
  // (the scales, on their way while the ticket is drawn; after the first
  // pass w has its own scale)
  const double sw = PASS == 0 ? S->sc[k - 1] : 1.;
  const double sc = sw * (j < k ? S->sc[j] : sw);
  if(!arrive_last(&S->tick_dots[PASS][grp], shares)) return;
  static_assert(kDotCols == 256 / 32, "one warp per column");
  if(wp >= cnt) return;
  double v = 0.;
#pragma unroll 5
  for(int b = lane; b < shares; b += 32) v += __ldcg(part + (size_t)j * kReduceBlocks + b);
  v = warp_sum(v);
  if(lane) return;
  v *= sc;
  if(j < k)
    (PASS == 0 ? S->h1 : S->h2)[j] = v;
  else {
    // mgsro's checks on ||w||^2 before it orthogonalises (iters.f:3475-3600):
    // zero (ierr -1) or abnormal (-2) leaves the column unwritten and ends
    // the cycle; gmres then reports a break-down.  (k_gm_update clears
    // S->cycle: CTAs of the other groups may only now be reading it)
    S->nrm0 = v;
    if(!(v > 0. && 1. / v > 0.)) {
      S->its += 1;  // the Arnoldi step's product was formed
      S->breakdown = (v <= 0.) ? -1 : -2;
    }
  }
}

// V_k = cur = w - sum_j h_j V_j (h of pass `pass`; pass 1: w is cur) with the
// partials of ||V_k||^2 in pn.  cur is the copy of the newest basis vector
// that the next step's preconditioner reads at a fixed address; for FGMRES
// pass 0 also keeps the preconditioned vector zt as Z_{k-1}.
// CTA nb, beside the nb that do so, applies the previous Givens rotations to
// the new Hessenberg column: they need the column only, not the norm, and
// their serial chain (one FMA per rotation) hides behind the update (done
// by one thread at the end of the step it had cost 18 us at k = 49).  The
// last CTA to finish sums the partials.  After pass 0 it applies the
// selective re-orthogonalisation test with mgsro's constant (iters.f:
// 3475-3600, reorth = 0.98: mgsro repeats the projection on one basis vector
// when it removed more than 98 % of the squared norm left; here the second
// classical Gram-Schmidt pass runs when the first pass removed more than
// 98 % of ||w||^2, ||w'|| < 0.14 ||w||; the loss of orthogonality of one
// pass grows like eps ||w|| / ||w'||, so a pass that keeps more than 2 %
// leaves w' orthogonal to within ~10 eps); without a second pass, or after
// it, it ends the Arnoldi step: h(k+1,k), the new rotation, the stopping test.
__global__ void __launch_bounds__(256)
k_gm_update(int n, int m, double *V, size_t ldv, const double *w, double *cur,
            const double *zt, double *Z, double *pn, GmState *S, int pass)
{
  chain_wait();
  const int go = S->cycle, again = S->reorth, bad = S->breakdown, k = S->k + 1;
  if(!go || bad || (pass == 1 && !again)) {  // the same in every CTA
    if(bad && blockIdx.x == 0 && threadIdx.x == 0) S->cycle = 0;
    return;
  }
  const int nb = gridDim.x - 1;
  __shared__ double h[kMaxKrylov + 1];
  __shared__ double rc[kMaxKrylov], rs[kMaxKrylov], ra[kMaxKrylov];
  double *Hc = S->H + (size_t)(k - 1) * (kMaxKrylov + 1);  // column k
  if(blockIdx.x == nb) {
    // rotation i: (a, b) -> (c a + s b, c b - s a) with b = h(i+1), the second
    // the next rotation's a.  Everything but that chain in parallel.
    const int j = threadIdx.x;
    double c = 0., s = 0., b = 0.;
    if(j < k) {
      h[j] = S->h1[j] + (pass == 0 ? 0. : S->h2[j]);
      c = S->cs[j];
      s = S->sn[j];
    }
    __syncthreads();
    if(j < k - 1) {
      b = h[j + 1];
      rc[j] = c * b;
      rs[j] = s;
    }
    __syncthreads();
    if(j == 0) {
      double a = h[0];
#pragma unroll 4
      for(int i = 0; i < k - 1; i++) {
        ra[i] = a;
        a = fma(-rs[i], a, rc[i]);
      }
      ra[k - 1] = a;
    }
    __syncthreads();
    if(j < k) Hc[j] = j < k - 1 ? fma(c, ra[j], s * b) : ra[j];
  }
  else {
    for(int j = threadIdx.x; j < k; j += blockDim.x)
      h[j] = -S->sc[j] * (pass == 0 ? S->h1[j] : S->h2[j]);
    const double sw = pass == 0 ? S->sc[k - 1] : 1.;
    __syncthreads();
    double v = 0.;
    for(int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nb * blockDim.x) {
      // two chains of FMAs, k + 3 FP64 instructions per row in all (FP64
      // instructions pace the kernel; four chains and a separate subtraction
      // took k + 6)
      const double *Vi = V + i;
      double s0 = sw * w[i], s1 = 0.;
      int j = 0;
#pragma unroll 4
      for(; j + 1 < k; j += 2, Vi += 2 * ldv) {
        s0 = fma(h[j], Vi[0], s0);
        s1 = fma(h[j + 1], Vi[ldv], s1);
      }
      if(j < k) s0 = fma(h[j], Vi[0], s0);
      s0 += s1;
      V[(size_t)k * ldv + i] = s0;
      cur[i] = s0;
      if(Z && pass == 0) Z[(size_t)(k - 1) * ldv + i] = zt[i];
      v = fma(s0, s0, v);
    }
    const double s = block_sum<double, 256>(v);
    if(threadIdx.x == 0) pn[blockIdx.x] = s;
  }
  // what the end of the step reads, on its way while the ticket is drawn
  const double nrm0 = S->nrm0, tol = S->tol, g = S->g[k - 1];
  const int its = S->its, maxit = S->maxit;
  if(!arrive_last(&S->tick_upd[pass], gridDim.x)) return;
  const double hk = __ldcg(Hc + k - 1);
  double rr = 0.;
#pragma unroll 4
  for(int i = threadIdx.x; i < nb; i += blockDim.x) rr += __ldcg(pn + i);
  rr = block_sum<double, 256>(rr);
  if(threadIdx.x) return;
  if(pass == 0) {
    const bool more = !(rr >= 0.02 * nrm0);
    S->reorth = more;
    if(more) return;  // the step ends after the second pass
  }
  S->its = its + 1;
  S->k = k;
  S->did_cycle = 1;
  if(!(rr > 0.)) {
    // mgsro ierr -3: the new vector depends on the others; the reference
    // solves with the column as mgsro left it, no rotation applied
    for(int j = 0; j < k; j++) Hc[j] = S->h1[j] + (pass == 0 ? 0. : S->h2[j]);
    Hc[k] = sqrt(rr);
    S->breakdown = -3;
    S->cycle = 0;
    return;
  }
  // the rotation of (hk, nrm): givens (iters.f:3235-3273) in terms of two
  // independent reciprocal roots, a third of the serial chain of its root,
  // divisions and root (an FP64 division takes about 0.8 us here)
  const double r2 = fma(hk, hk, rr);
  double c, s;
  if(rr > 1e-280 && r2 < 1e280) {
    const double ri = rsqrt(rr), q = rsqrt(r2);
    S->sc[k] = ri;
    c = hk * q;
    s = rr * ri * q;
    Hc[k - 1] = r2 * q;
  }
  else {
    double x = hk, y = sqrt(rr);
    S->sc[k] = 1. / y;
    givens_dev(&x, &y, &c, &s);
    Hc[k - 1] = x;
  }
  S->cs[k - 1] = c;
  S->sn[k - 1] = s;
  S->g[k - 1] = c * g;
  S->g[k] = -s * g;
  const double alpha = fabs(-s * g);
  S->res = alpha;
  if(!(k < m && !(alpha <= tol) && (maxit <= 0 || its + 1 < maxit)))
    S->cycle = 0;  // the end of this cycle
}

// end of a cycle: solve H y = g (upper triangular, k x k) on one thread
__global__ void k_gm_solve_small(GmState *S)
{
  if(!S->active || !S->did_cycle || threadIdx.x) return;
  int k = S->k;
  const int ld = kMaxKrylov + 1;
  while(k > 0 && S->H[(size_t)(k - 1) * ld + (k - 1)] == 0.) k--;  // iters.f:2141-2155
  if(k == 0) {
    S->status = -3;
    S->breakdown = -4;
    S->active = 0;
    S->did_cycle = 0;
    return;
  }
  S->k = k;
  for(int i = k - 1; i >= 0; i--) {
    double t = S->g[i];
    for(int j = i + 1; j < k; j++) t -= S->H[(size_t)j * ld + i] * S->y[j];
    S->y[i] = t / S->H[(size_t)i * ld + i];
  }
}

// u = sum_j y_j Vj (GMRES) or x += sum_j y_j Z_j (FGMRES, ADD = 1)
template <int ADD>
__global__ void __launch_bounds__(256)
k_gm_combine(int n, const double *__restrict__ V, size_t ldv,
             double *__restrict__ out, const GmState *__restrict__ S)
{
  if(!S->active || !S->did_cycle) return;
  __shared__ double y[kMaxKrylov];
  int k = S->k;
  for(int j = threadIdx.x; j < k; j += blockDim.x)
    y[j] = S->y[j] * S->sc[j];
  __syncthreads();
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += (long long)gridDim.x * blockDim.x) {
    double s = ADD ? out[i] : 0.;
    for(int j = 0; j < k; j++) s += y[j] * V[(size_t)j * ldv + i];
    out[i] = s;
  }
}

__global__ void k_gm_addto(int n, const double *__restrict__ u,
                           double *__restrict__ x, const GmState *__restrict__ S)
{
  if(!S->active || !S->did_cycle) return;
  for(long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
      i += (long long)gridDim.x * blockDim.x)
    x[i] += u[i];
}

// after the update: the restart decision of iters.f:2196-2218
__global__ void k_gm_after(GmState *S)
{
  if(!S->active || threadIdx.x) return;
  S->res6 = S->res;
  if(S->breakdown != 0) {
    S->status = -3;
    S->active = 0;
    return;
  }
  bool more = (S->its < S->maxit || S->maxit <= 0) && (S->res6 > S->tol);
  if(!more) {
    if(S->res6 <= S->tol)
      S->status = 0;
    else if(S->its >= S->maxit && S->maxit > 0)
      S->status = -1;
    else
      S->status = -10;
    S->active = 0;
  }
}

__global__ void k_gm_apply_ok(GmState *S, int *ok)
{
  // the update's preconditioner runs when a solution update is due
  if(threadIdx.x == 0) *ok = (S->active && S->did_cycle) ? 1 : 0;
}

bool correction_valid(const gb300_matrix *A)
{
  return A->corr_version == A->pattern_version && A->corr.p && A->nnz > 0;
}

int PrecondScratch::alloc(const gb300_solver_params *p, int n,
                          const std::function<void *(int, size_t)> &get)
{
  const size_t b64 = sizeof(double) * (size_t)(n > 0 ? n : 1);
  bool ok = true;
  auto vec = [&](int slot) {
    double *q = (double *)get(slot, b64);
    ok = ok && q;
    return q;
  };
  if(p->precision != 0) {
    t32 = (float *)get(5, b64 / 2);
    ok = ok && t32;
  }
  if(precond_learned(p->preconditioner)) t1 = vec(8);
  if(precond_two_level(p->preconditioner)) {
    t3 = vec(13);
    t4 = vec(14);
    t5 = vec(15);
  }
  return ok ? GB300_OK : GB300_ERR_CUDA;
}

void precond_run(const gb300_matrix *A, const double *val, const gb300_solver_params *p,
                 const double *v, double *z, const PrecondScratch &s, const int *flag,
                 cudaStream_t st)
{
  const int n = A->n, pc = p->preconditioner;
  const bool learned = precond_learned(pc);
  const bool learned_post = learned && pc != kPrecondLearnedCoarsePre;
  const bool sai = (pc == kPrecondLearnedSai || pc == kPrecondSai);
  const bool ilu = (pc == 6 || learned || precond_two_level(pc)) && !sai;
  const ilu_data *L = ilu ? A->ilu : nullptr;
  const int gs = grid_for(n, 256, kReduceBlocks * 4);
  const bool early = chain_early(n);
  if(!ilu && !sai) {  // no preconditioner
    launch_chain(early, k_gm_scale, gs, 256, st, n, nullptr, v, z, nullptr, flag);
    return;
  }
  // out = S in (+ G (in - A out)), or added into out through tmp
  auto smooth = [&](const double *in, double *out, double *tmp, bool add, bool corr) {
    if(sai) {
      spmv_chain(add ? kChainAdd : kChainMul, A, A->corr.p,
                 {in, nullptr, out, nullptr, nullptr, nullptr, flag}, st);
      return;
    }
    double *x = add ? tmp : out;
    const bool sweep_adds = add && !corr;
    const int mode = ilu_mode(p);
    if(!L->by_colour) {
      ilu_apply(A, mode, in, x, s.t32, flag, st);
      if(sweep_adds) launch_chain(early, k_gm_add, gs, 256, st, n, (const double *)x, out, flag);
    }
    else if(mode == 0) {
      if(sweep_adds)
        colour_sweeps<2, double, double>(L, L->inv64.p, in, x, out, flag, st);
      else
        colour_sweeps<0, double, double>(L, L->inv64.p, in, x, nullptr, flag, st);
    }
    else if(mode == 2) {
      if(sweep_adds)
        colour_sweeps<2, float, double>(L, L->inv32.p, in, x, out, flag, st);
      else
        colour_sweeps<0, float, double>(L, L->inv32.p, in, x, nullptr, flag, st);
    }
    else {
      if(sweep_adds)
        colour_sweeps<2, float, float>(L, L->inv32.p, in, s.t32, out, flag, st);
      else
        colour_sweeps<1, float, float>(L, L->inv32.p, in, s.t32, x, flag, st);
    }
    if(corr) {
      // the learned correction: t1 = in - A x, then x += G t1 (or both added
      // into out)
      product_chain(kChainRes, A, val, {x, in, s.t1, nullptr, nullptr, nullptr, flag}, st);
      spmv_chain(add ? kChainAddBoth : kChainAdd, A, A->corr.p,
                 {s.t1, x, add ? out : x, nullptr, nullptr, nullptr, flag}, st);
    }
  };
  if(!precond_two_level(pc)) {
    smooth(v, z, nullptr, false, learned);
    return;
  }
  // z = S v;  z += P0 Ac^-1 P0^T (v - A z);  z += S (v - A z)
  smooth(v, s.t5, nullptr, false, learned && !sai);
  coarse_correct(A, val, v, s.t5, z, s.t3, flag, st);
  smooth(s.t3, z, s.t4, true, learned_post && !sai);
}

static int gmres_run(gb300_matrix *A, const double *val, const double *rhs, double *x,
                     const gb300_solver_params *p, gb300_solve_info *info, Work &W)
{
  cudaStream_t st = A->ctx->stream;
  int n = A->n;
  bool flexible = (p->algorithm == 9);
  if(p->algorithm != 8 && p->algorithm != 9) {
    set_error("Algorithm %d with Preconditioner %d is not supported", p->algorithm,
              p->preconditioner);
    return GB300_ERR_UNSUPPORTED;
  }
  int m = p->krylov_size <= 1 ? 15 : p->krylov_size;
  if(m > kMaxKrylov) {
    set_error("Krylov_Size %d exceeds this backend's maximum %d", m, kMaxKrylov);
    return GB300_ERR_UNSUPPORTED;
  }
  // 20: ILU(0) followed by the learned correction on A's pattern; 21, 22:
  // the two-level cycle on aggregates around ILU(0) (22: and the correction)
  const bool learned = precond_learned(p->preconditioner);
  const bool coarse = precond_two_level(p->preconditioner);
  // 24: G alone smooths, no ILU(0); 25: with G the SPAI-1 made here
  const bool sai = (p->preconditioner == kPrecondLearnedSai ||
                    p->preconditioner == kPrecondSai);
  if(p->preconditioner == kPrecondSai && !(p->re_use_lu && correction_valid(A)))
    GB_TRY(spai1(A, val));
  bool precond = ((p->preconditioner == 6) || learned || coarse) && !sai;
  if(p->preconditioner != 0 && p->preconditioner != 6 && p->preconditioner != 8 &&
     !learned && !coarse) {
    set_error("Preconditioner %d is not supported by this backend", p->preconditioner);
    return GB300_ERR_UNSUPPORTED;
  }
  if(learned && !correction_valid(A)) {
    set_error("Preconditioner %d needs a correction on the matrix pattern "
              "(gb300_matrix_set_correction)", p->preconditioner);
    return GB300_ERR_ARG;
  }
  if(coarse && !coarse_valid(A)) {
    set_error("Preconditioner %d needs aggregates on the matrix pattern "
              "(gb300_matrix_set_aggregates)", p->preconditioner);
    return GB300_ERR_ARG;
  }
  bool fp32 = (p->precision != 0);
  if(precond) {
    int zr = 0;
    // the factor is on A's values as given to the solver (scaled if needed)
    GB_TRY(ilu_factor(A, val, fp32, &zr, p->re_use_lu != 0, &info->ilu_factorized));
    if(zr) {
      info->status = zr;
      set_error("Zero pivot on line %d in ILU", zr);
      return GB300_ERR_ZERO_PIVOT;
    }
  }
  if(coarse) GB_TRY(coarse_setup(A, val, p->re_use_lu != 0));
  if(precond) GB_TRY(ilu_products(A, val));
  size_t ldv = (size_t)n;
  double *V = (double *)W.vec(0, sizeof(double) * ldv * (m + 1));
  double *Z = flexible ? (double *)W.vec(1, sizeof(double) * ldv * m) : nullptr;
  double *u = (double *)W.vec(3, sizeof(double) * n);
  double *cur = (double *)W.vec(2, sizeof(double) * n);
  double *w = (double *)W.vec(9, sizeof(double) * n);
  double *zt = (double *)W.vec(4, sizeof(double) * n);
  PrecondScratch ps;
  GB_TRY(ps.alloc(p, n, [&](int slot, size_t bytes) { return W.vec(slot, bytes); }));
  double *part = (double *)W.vec(6, sizeof(double) * kReduceBlocks * (m + 1));
  double *pn = (double *)W.vec(12, sizeof(double) * kReduceBlocks);
  GmState *S = (GmState *)W.state(sizeof(GmState));
  int *okflag = (int *)W.vec(7, sizeof(int));
  if(!V || (flexible && !Z) || !u || !cur || !w || !zt || !part || !pn || !S || !okflag)
    return GB300_ERR_CUDA;
  GmState h0;
  memset(&h0, 0, sizeof(h0));
  h0.active = 1;
  h0.first = 1;
  h0.maxit = p->nb_iter_max;
  h0.rtol = p->stopping_test;
  h0.status = 1;
  GB_CUDA(cudaMemcpyAsync(S, &h0, sizeof(GmState), cudaMemcpyHostToDevice, st));
  GB_CUDA(cudaMemsetAsync(x, 0, sizeof(double) * n, st));  // sol = 0

  int gs = grid_for(n, 256, kReduceBlocks * 4);
  // row shares of the Gram-Schmidt kernels, fixed for a given n and step, so
  // deterministic.  Dots: the groups' CTAs fill the SMs once (see k_gm_dots),
  // twice from 200,000 rows on, where the loads need more warps (304 against
  // 152 CTAs: 26 / 25 us at 261,121 rows, 39 / 50 at 434,281, k = 33).  Update:
  // every CTA that is resident at once, as far as there are rows: it reads k
  // vectors a row, and one CTA per SM leaves too few loads in flight (k = 33,
  // 152 / 456 / 760 CTAs: 35 / 32 / 31 us at 261,121 rows, 106 / 51 / 44 at
  // 434,281, 259 / 105 / 84 at 1,046,529; a second wave costs 15 % again)
  const int rows256 = (n + 255) / 256;
  const int nbd = std::min(152 * (n > 200000 ? 2 : 1), rows256 * (m / kDotCols + 1));
  const int nbu = std::min(rows256, resident_grid(k_gm_update, 256, 0));
  // The first pass's kernels start early where the grids leave most SMs idle;
  // elsewhere their waiting CTAs cost the kernel before more than the launch
  // (not / early, us per step: 53.9 / 51.8 at 81 rows, 34.0 / 33.6 at 529, 33.8
  // / 33.6 at 3,969, 33.8 / 35.2 at 7,921, 38.7 / 40.6 at 65,025, 335 / 362 at
  // 1,046,529).
  const bool gs_early = n <= 4096;
  const double *no_z = nullptr;

  // One graph holds a few Arnoldi steps (they find their place in the cycle
  // in the state) and is replayed through the cycle, another the end of the
  // cycle and the restart: a graph of all m steps had cost 1 to 3 ms per
  // solve to capture and instantiate, more than 50 steps of a small system.
  constexpr int kChunk = 5;
  auto restart = [&]() {  // V_0 = cur = (rhs - A x) / ||rhs - A x||
    residual64(A, val, x, rhs, V, part, st);
    k_gm_restart<<<1, 256, 0, st>>>(S, part, m);
    k_gm_scale<<<gs, 256, 0, st>>>(n, &S->scale, V, V, cur, &S->cycle);
  };
  auto step = [&]() {
    if(p->preconditioner != 6 || !small_step(A, val, ilu_mode(p), cur, zt, w, &S->cycle, st)) {
      precond_run(A, val, p, cur, zt, ps, &S->cycle, st);
      product_chain(kChainMul, A, val, {zt, nullptr, w, nullptr, nullptr, nullptr, &S->cycle},
                    st);
    }
    // classical Gram-Schmidt, a second pass only when the test after the
    // first asks for it; the reductions, the test and the end of the step
    // run in the last CTA of each kernel.  The second pass's kernels start
    // early (launch_chain): it seldom runs, and its launches then cost 0.3 to
    // 0.9 us a step less (38.0 / 37.1 us at 529 rows, 39.6 / 39.1 at 65,025).
    launch_chain(gs_early, k_gm_dots<0>, nbd, 256, st, n, V, ldv, w, part, S);
    launch_chain(gs_early, k_gm_update, nbu + 1, 256, st, n, m, V, ldv, w, cur, zt, Z, pn, S, 0);
    launch_chain(true, k_gm_dots<1>, nbd, 256, st, n, V, ldv, cur, part, S);
    launch_chain(true, k_gm_update, nbu + 1, 256, st, n, m, V, ldv, cur, cur, no_z, Z, pn, S, 1);
  };
  auto turn = [&]() {
    k_gm_solve_small<<<1, 32, 0, st>>>(S);
    if(flexible)
      k_gm_combine<1><<<gs, 256, 0, st>>>(n, Z, ldv, x, S);
    else {
      k_gm_combine<0><<<gs, 256, 0, st>>>(n, V, ldv, u, S);
      k_gm_apply_ok<<<1, 32, 0, st>>>(S, okflag);
      if(p->preconditioner != 6 || !small_step(A, val, ilu_mode(p), u, zt, nullptr, okflag, st))
        precond_run(A, val, p, u, zt, ps, okflag, st);
      k_gm_addto<<<gs, 256, 0, st>>>(n, zt, x, S);
    }
    k_gm_after<<<1, 32, 0, st>>>(S);
    restart();
  };
  struct Graph {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t e = nullptr;
    ~Graph()
    {
      if(e) cudaGraphExecDestroy(e);
      if(g) cudaGraphDestroy(g);
    }
  } steps, turns;
  auto capture = [&](Graph &G, auto body) -> int {
    auto capturing = hold_capture();
    GB_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    body();
    GB_CUDA(cudaStreamEndCapture(st, &G.g));
    capturing.unlock();
    GB_CUDA(cudaGraphInstantiate(&G.e, G.g, 0));
    return GB300_OK;
  };
  restart();
  GB_TRY(capture(steps, [&]() {
    for(int q = 0; q < std::min(m, kChunk); q++) step();
  }));
  GB_TRY(capture(turns, turn));
  const int replays = (m + kChunk - 1) / kChunk;
  int active = 1, launches = 0;
  int max_launches = p->nb_iter_max > 0 ? p->nb_iter_max + 2 : 1 << 30;
  while(active && launches < max_launches) {
    for(int q = 0; q < replays; q++) GB_CUDA(cudaGraphLaunch(steps.e, st));
    GB_CUDA(cudaGraphLaunch(turns.e, st));
    launches++;
    GB_CUDA(cudaMemcpyAsync(&active, &S->active, sizeof(int),
                            cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
  }
  GB_CUDA(cudaMemcpyAsync(&h0, S, sizeof(GmState), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  info->status = active ? -1 : h0.status;
  info->iterations = h0.its;
  info->residual_estimate = h0.res6;
  return GB300_OK;
}

// the largest |v_k| (non-negative doubles order like their bit patterns)
__global__ void k_max_abs(long long m, const double *__restrict__ v, unsigned long long *out)
{
  unsigned long long t = 0;
  for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < m;
      k += (long long)gridDim.x * blockDim.x)
    t = max(t, (unsigned long long)__double_as_longlong(fabs(v[k])));
  for(int o = 16; o > 0; o >>= 1) t = max(t, __shfl_down_sync(0xffffffffu, t, o));
  if((threadIdx.x & 31) == 0) atomicMax(out, t);
}

__global__ void k_times(long long m, double f, const double *v, double *out)
{
  for(long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < m;
      k += (long long)gridDim.x * blockDim.x)
    out[k] = f * v[k];
}

// The basis is left unnormalised, so the square of a product is of the order of
// ||A M^-1||^4.  With a preconditioner that is some power of one; without, a
// matrix whose largest entry is not within 2^+-64 is solved as
// (2^-e A) (2^e x) = b, which rounds nothing.  (Powers of two inside the step
// instead, where nothing has to be known in advance, cost every solve 1 %.)
int gmres_solve(gb300_matrix *A, const double *val, const double *rhs,
                double *x, const gb300_solver_params *p, gb300_solve_info *info,
                Work &W)
{
  if(p->preconditioner != 0 && p->preconditioner != 8)
    return gmres_run(A, val, rhs, x, p, info, W);
  cudaStream_t st = A->ctx->stream;
  DevBuf<unsigned long long> top;
  GB_TRY(top.alloc(1));
  GB_CUDA(cudaMemsetAsync(top.p, 0, sizeof(unsigned long long), st));
  k_max_abs<<<grid_for(A->nnz, 256, kReduceBlocks), 256, 0, st>>>(A->nnz, val, top.p);
  double most = 0.;
  GB_CUDA(cudaMemcpyAsync(&most, top.p, sizeof(most), cudaMemcpyDeviceToHost, st));
  GB_CUDA(cudaStreamSynchronize(st));
  int e = 0;
  if(most > 0. && most <= 1.7976931348623157e308) frexp(most, &e);
  if(e >= -64 && e <= 64) return gmres_run(A, val, rhs, x, p, info, W);
  const double f = ldexp(1., -std::max(e, -1000));
  DevBuf<double> sval;
  GB_TRY(sval.alloc(A->nnz));
  k_times<<<grid_for(A->nnz, 256, kReduceBlocks), 256, 0, st>>>(A->nnz, f, val, sval.p);
  GB_TRY(gmres_run(A, sval.p, rhs, x, p, info, W));
  k_times<<<grid_for(A->n, 256, kReduceBlocks), 256, 0, st>>>(A->n, f, x, x);
  GB_CUDA(cudaGetLastError());
  return GB300_OK;
}

}  // namespace gb
