// Shared infrastructure of the GB300 backend: error reporting, the context
// (one device, one stream), device buffers and small device helpers.
#pragma once

#include <nvtx3/nvToolsExt.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/getdp_gb300.h"
#include "pool.h"

namespace gb {

// NVTX range over a scope: the C ABI's phases (Generate, solve, batched
// solve, post-processing, network) show up by name in ncu / Nsight captures
// (ncu --nvtx --nvtx-include "gb300_solve/"); a no-op without a tool
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};


struct ilu_data;
struct Colouring;
struct Coarse;
// A's values changed: a coarse inverse made from the old ones is stale
void coarse_values_changed(gb300_matrix *A);

// last error message, per thread (read through gb300_last_error)
void set_error(const char *fmt, ...);

#define GB_CUDA(x)                                                           \
  do {                                                                       \
    cudaError_t e_ = (x);                                                    \
    if(e_ != cudaSuccess) {                                                  \
      ::gb::set_error("%s:%d: %s failed: %s", __FILE__, __LINE__, #x,        \
                      cudaGetErrorString(e_));                               \
      return GB300_ERR_CUDA;                                                 \
    }                                                                        \
  } while(0)

#define GB_TRY(...)                                                          \
  do {                                                                       \
    int r_ = (__VA_ARGS__);                                                  \
    if(r_ != GB300_OK) return r_;                                            \
  } while(0)

// number of SMs on GB300 and the partial-sum grid used by every
// deterministic reduction (fixed, so results do not depend on timing)
constexpr int kReduceBlocks = 1216;  // 152 SMs x 8
constexpr int kReduceThreads = 256;

template <typename T> struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  cudaStream_t from = nullptr;  // of the pool's context, null: cudaMalloc
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  ~DevBuf() { release(); }
  void release()
  {
    if(p) {
      if(from)
        cudaFreeAsync(p, from);
      else
        cudaFree(p);
    }
    p = nullptr;
    n = 0;
    from = nullptr;
  }
  int alloc(size_t count)
  {
    if(count <= n && p) return GB300_OK;
    release();
    if(count == 0) return GB300_OK;
    const cudaError_t e = device_alloc((void **)&p, count * sizeof(T), &from);
    if(e != cudaSuccess) {
      set_error("device allocation (%zu bytes) failed: %s", count * sizeof(T),
                cudaGetErrorString(e));
      p = nullptr;
      from = nullptr;
      return GB300_ERR_CUDA;
    }
    n = count;
    return GB300_OK;
  }
};

__device__ __forceinline__ double warp_sum(double v)
{
  for(int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v)
{
  for(int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Per-thread accumulator of a reduction over vector entries of type T:
// float for FP32 vectors (a thread sums a few dozen terms at most, FP64
// takes over at the block sum), double otherwise.  GB300's FP64 pipe
// retires about two FMAs (or conversions) per SM per clock, so FP64
// arithmetic on every entry of an FP32 vector costs more time than the
// entry's memory traffic.
template <typename T> struct Acc {
  using type = double;
};
template <> struct Acc<float> {
  using type = float;
};

// block-wide sum in a fixed order; result valid in thread 0
template <typename T, int NT> __device__ __forceinline__ T block_sum(T v)
{
  __shared__ T red[NT / 32];
  v = warp_sum(v);
  if((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  // the warps' sums in a tree as well (one after the other, eight FP64
  // additions of some 85 ns each stood at the end of every reduction)
  T s = 0;
  if(threadIdx.x < 32) s = warp_sum(threadIdx.x < NT / 32 ? red[threadIdx.x] : (T)0);
  __syncthreads();
  return s;
}

// Block-wide sums of eight per-thread accumulators, in a fixed order.
// Within a warp a transposing butterfly halves the accumulators a lane
// carries at each of the first three exchanges (offsets 16, 8, 4) and then
// adds across the remaining lane pairs: 9 FP64 additions per lane instead
// of 8 x 5 for eight separate warp sums (GB300's FP64 pipe makes the
// difference visible).  Afterwards lane l of each warp holds the warp total
// of accumulator (l >> 2) & 7.  out[j] is valid in thread j (j < 8).
template <int NT> __device__ __forceinline__ double block_sum8(const double (&a)[8])
{
  __shared__ double red[NT / 32][8];
  const int lane = threadIdx.x & 31;
  double b[4], c[2], d;
  {
    const bool hi = lane & 16;
#pragma unroll
    for(int m = 0; m < 4; m++) {
      double keep = hi ? a[m + 4] : a[m], send = hi ? a[m] : a[m + 4];
      b[m] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
  }
  {
    const bool hi = lane & 8;
#pragma unroll
    for(int m = 0; m < 2; m++) {
      double keep = hi ? b[m + 2] : b[m], send = hi ? b[m] : b[m + 2];
      c[m] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
  }
  {
    const bool hi = lane & 4;
    double keep = hi ? c[1] : c[0], send = hi ? c[0] : c[1];
    d = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  d += __shfl_xor_sync(0xffffffffu, d, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  if((lane & 3) == 0) red[threadIdx.x >> 5][lane >> 2] = d;
  __syncthreads();
  double s = 0.;
  if(threadIdx.x < 8)
    for(int w = 0; w < NT / 32; w++) s += red[w][threadIdx.x];
  __syncthreads();
  return s;
}

// Completion of a reduction inside the kernel that produces the partials:
// every block (of the grid, or of the group that shares the counter) calls
// arrive_last after its partials are stored; exactly one block, the last of
// `arrivals` to arrive, gets true and then sees every
// partial (read them with __ldcg).  It resets the counter for the next
// launch.  Needs no co-residency and never waits.
__device__ __forceinline__ bool arrive_last(unsigned *counter, unsigned arrivals)
{
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if(threadIdx.x == 0) {
    unsigned t = atomicAdd(counter, 1u);
    last = (t == arrivals - 1);
    if(last) *counter = 0u;
  }
  __syncthreads();
  if(last) __threadfence();
  return last != 0;
}

__device__ __forceinline__ bool arrive_last(unsigned *counter)
{
  return arrive_last(counter, gridDim.x * gridDim.y * gridDim.z);
}

// the first np partials summed in a fixed order (NT threads), read through L2
template <int NT>
__device__ __forceinline__ double sum_partials_l2(const double *part, int np)
{
  double s = 0.;
#pragma unroll 5
  for(int i = threadIdx.x; i < np; i += NT) s += __ldcg(part + i);
  return block_sum<double, NT>(s);
}

// streaming loads for data read once per pass (matrix values and indices)
template <typename T> __device__ __forceinline__ T ld_stream(const T *p)
{
  return __ldcs(p);
}

// Partial dot product of one CSR row with x for the TPR lanes that share
// the row: each lane first issues U independent (column, value) loads, then
// the U gathers of x, then the multiply-adds, so a warp keeps U memory
// requests in flight instead of one dependent chain.  READ_ONLY: x through the
// read-only path, for kernels in whose lifetime nothing writes it; a kernel
// that may start while x's writer runs (launch_chain) takes plain loads.
// Lanes past the row's end add nothing: the product of a zero with an entry of
// x that the row does not hold is NaN where that entry is not finite.
template <int TPR, int U, typename ACC, bool READ_ONLY = true, typename V, typename XT>
__device__ __forceinline__ ACC csr_row_dot(int s, int e, int lane,
                                           const int *__restrict__ col,
                                           const V *__restrict__ val, const XT *x)
{
  ACC sum = 0;
  for(int k0 = s + lane; k0 < e; k0 += TPR * U) {
    int c[U];
    V v[U];
#pragma unroll
    for(int u = 0; u < U; u++) {
      int k = k0 + u * TPR;
      bool in = k < e;
      c[u] = in ? __ldcs(col + k) : -1;
      v[u] = in ? __ldcs(val + k) : (V)0;
    }
    XT xv[U];
#pragma unroll
    for(int u = 0; u < U; u++)
      xv[u] = c[u] < 0 ? (XT)0 : READ_ONLY ? __ldg(x + c[u]) : x[c[u]];
#pragma unroll
    for(int u = 0; u < U; u++)
      if(c[u] >= 0) sum += (ACC)v[u] * (ACC)xv[u];
  }
  return sum;
}

// position of column c in the sorted row [lo, hi) of col[], or -1
__device__ __forceinline__ int find_col(const int *__restrict__ col, int lo,
                                        int hi, int c)
{
  const int end = hi;
  while(lo < hi) {
    int mid = (lo + hi) >> 1;
    int v = col[mid];
    if(v < c)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (lo < end && col[lo] == c) ? lo : -1;
}

// Programmatic dependent launch: a kernel launched with launch_chain and
// `early` may start while its predecessor in the stream still runs.
// chain_wait() returns when the predecessor has completed and its writes are
// visible; before it a kernel reads only data no kernel of the sequence
// writes (matrix structure and values, factors, permutations), so that those
// loads overlap the predecessor's tail.  The next kernel is released after
// the wait, so everything older than the direct predecessor is complete when
// a kernel starts.  Every CTA calls it (a CTA that skipped the wait could let
// the kernel after it overtake the predecessor); without `early` it returns
// at once.  Data written inside the sequence is read with plain loads (no
// __restrict__ const, no __ldg: the non-coherent path could return lines
// cached before the wait).
__device__ __forceinline__ void chain_wait()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... K, typename... A>
inline void launch_chain(bool early, void (*kernel)(K...), dim3 grid, dim3 block,
                         cudaStream_t st, A... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, K(args)...);  // errors: cudaGetLastError
}

// whether a sequence over n rows gains from the early start.  Measured on
// 2D meshes in the multicolour order, both sweeps / a product, early against
// not: 14.2 / 2.8 against 15.4 / 3.4 us at 65,025 rows, but 25.3 / 7.0
// against 19.3 / 7.6 at 261,121: the waiting CTAs of the next kernel take the
// free slots of whichever SMs have them, and its load is uneven from then on.
// (The FP64-bound Gram-Schmidt kernels lose by that at all but the smallest
// sizes and have a line of their own, in gmres_solve.)
inline bool chain_early(int n) { return n <= 131072; }

inline int grid_for(long long work, int threads, int max_blocks = 1 << 30)
{
  long long b = (work + threads - 1) / threads;
  if(b < 1) b = 1;
  if(b > max_blocks) b = max_blocks;
  return (int)b;
}

// CTAs of `kernel` that fit on the device at once (at most kReduceBlocks):
// a grid-stride kernel launched this wide runs in one wave
template <typename K> int resident_grid(K kernel, int threads, size_t smem)
{
  int dev = 0, sms = 0, per_sm = 0;
  if(cudaGetDevice(&dev) != cudaSuccess ||
     cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
     cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
       cudaSuccess ||
     per_sm < 1 || sms < 1)
    return kReduceBlocks;
  return per_sm * sms < kReduceBlocks ? per_sm * sms : kReduceBlocks;
}

}  // namespace gb

namespace gb {
struct GenCache;  // the pattern of the last Generate (assemble.cu)
void gen_cache_free(GenCache *c);
}  // namespace gb

// the objects behind the opaque handles of the C ABI
struct gb300_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 152;
  // scratch memory of the calls on this context; what is free in it beyond
  // kPoolKeep goes back to the device at the next synchronisation, all of it
  // with the context or when the device has no other memory left
  gb::MemPool mem;
  // CSR pattern, scatter positions and element colouring of the element
  // table last generated on this context: a Generate of the same table
  // (GetDP's ZeroMatrix recreates A before every Generate) reuses them
  gb::GenCache *gen = nullptr;
};

namespace gb {
// DevBuf allocates from this context's pool on this thread.  Entry points that
// make scratch buffers on each call set it for their duration: cudaMalloc and
// cudaFree cost some 10 to 200 us each and the latter waits for the device (a
// Generate at 513^2 spent 0.2 of its 0.3 ms in them).  Null: no pool, for
// buffers that may outlive the matrix's context.
struct PoolScope {
  MemPool *before;
  explicit PoolScope(gb300_ctx *c) : before(t_pool) { t_pool = c ? &c->mem : nullptr; }
  ~PoolScope() { t_pool = before; }
  PoolScope(const PoolScope &) = delete;
  PoolScope &operator=(const PoolScope &) = delete;
};
}  // namespace gb

struct gb300_vector {
  gb300_ctx *ctx = nullptr;
  int n = 0;
  gb::DevBuf<double> d;
};

struct gb300_matrix {
  gb300_ctx *ctx = nullptr;
  int n = 0;
  // host staging of LinAlg-style scalar adds, in call order
  std::vector<int> hr, hc;
  std::vector<double> hv;
  // bulk adds, staged on the device before the host's entries
  gb::DevBuf<int> sr, sc;
  gb::DevBuf<double> sv;
  long long staged = 0;
  void drop_staged_host()
  {
    hr.clear();
    hc.clear();
    hv.clear();
  }
  void drop_staged()
  {
    drop_staged_host();
    staged = 0;
    if(sv.n > (1u << 26)) {  // more than 1 GB is not kept for the next adds
      sr.release();
      sc.release();
      sv.release();
    }
  }
  // device CSR (0-based, rows sorted by column)
  gb::DevBuf<int> rowptr, col;
  gb::DevBuf<double> val;
  gb::DevBuf<float> val32;  // fp32 copy for mixed-precision inner solves
  long long nnz = 0;
  bool csr_valid = false;
  bool val32_valid = false;
  int tpr = 32;  // threads per row for the CSR kernels
  // three-component system in GetDP's component-major numbering (set by the
  // elasticity Generate hook): the CG may iterate on a 3x3-blocked copy
  bool block3 = false;
  // the pattern has been verified to hold 3 x 3 node blocks (elasticity
  // Generate: one search per node pair); reset by every pattern build
  bool node_blocks = false;
  int bsr_var32 = -1, bsr_var64 = -1;  // tuned SpMV launch shapes (-1: not yet)
  // ILU(0) state, created on demand by the solver
  gb::ilu_data *ilu = nullptr;
  // bumped whenever the pattern is rebuilt; the multicolour ordering of the
  // ILU solves (created on demand) remembers the version it was made for
  unsigned pattern_version = 0;
  unsigned diag_version = ~0u;  // the pattern known to hold every diagonal entry
  gb::Colouring *mc = nullptr;
  // on a permuted copy: the ordering it is the copy of (owned by the source)
  const gb::Colouring *order = nullptr;
  // rows per unknown (2: complex system in real form, harmonic-interleaved)
  int block_rows = 1;
  // learned preconditioner correction on the pattern (valid while
  // corr_version == pattern_version)
  gb::DevBuf<double> corr;
  unsigned corr_version = ~0u;
  // aggregates and coarse operator of the two-level preconditioners
  // (gb300_matrix_set_aggregates; valid while their version is pattern_version)
  gb::Coarse *coarse = nullptr;
  // the pattern came from the context's Generate cache entry gen_tag while
  // pattern_version was gen_pv (a later change of the pattern bumps the
  // version and so invalidates the link)
  unsigned gen_tag = 0, gen_pv = ~0u;
};
