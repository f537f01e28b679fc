// FP64 true residual r = b - A x and ||r||_2^2 for a CSR matrix on the GPU.
//
// The reference computes this residual before the PCG loop
// (src/solvers/pcg.F90:364-367) and, in doug_geom, after it
// (src/main/geom.F90:135-142).  The solver uses the same arithmetic
// internally; this file exposes it to callers that hold their own device
// CSR matrix (for example to check a solution written by dg_solve_device).
//
// The norm is reduced deterministically: each block of rows_per_block rows
// writes one partial sum, and one block adds the partials in order.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "../../include/doug_gpu.h"

namespace dg {
namespace resid {

constexpr int kThreads = 256;
constexpr int kMaxRowsPerBlock = 1024;            // rows per partial sum

// The products of entries e, e + W, .. below e1 with x, in that order; four
// entries are loaded before they are summed.
template <int W>
__device__ __forceinline__ double row_share(long long e, long long e1, const int *__restrict__ col,
                                            const double *__restrict__ val, const double *__restrict__ x) {
  double s = 0.0;
  for (; e + 3 * W < e1; e += 4 * W) {
    const int c0 = col[e], c1 = col[e + W], c2 = col[e + 2 * W], c3 = col[e + 3 * W];
    const double a0 = val[e], a1 = val[e + W], a2 = val[e + 2 * W], a3 = val[e + 3 * W];
    const double x0 = x[c0], x1 = x[c1], x2 = x[c2], x3 = x[c3];
    s = __fma_rn(a0, x0, s);
    s = __fma_rn(a1, x1, s);
    s = __fma_rn(a2, x2, s);
    s = __fma_rn(a3, x3, s);
  }
  for (; e < e1; e += W) s = __fma_rn(val[e], x[col[e]], s);
  return s;
}

// A block's rows [r0, r0 + nr) with L lanes per row; returns this thread's part
// of sum r_i^2.  Rows of more than kLongRow L entries are left to whole warps,
// after the others: their L lanes alone would hold up the block.  200,000 rows
// of 7 entries with one of 1,200: 143 us without this, 30 us with it; a million
// rows of 7 with 5 % of 100: 183 us, 121 us.  At the limit a lane makes 16
// rounds of loads; rows of 36 among rows of 2 are faster by lanes (168 us; 327
// with a limit of 32).
constexpr int kLongRow = 64;
template <int L>
__device__ __forceinline__ double block_rows(int r0, int nr, const long long *__restrict__ rp,
                                             const int *__restrict__ col, const double *__restrict__ val,
                                             const double *__restrict__ x, const double *__restrict__ b,
                                             double *__restrict__ r, int *any_long) {
  const int sub = threadIdx.x % L;
  double acc = 0.0;
  for (int q0 = 0; q0 < nr; q0 += kThreads / L) {
    const int q = q0 + threadIdx.x / L, i = r0 + q;
    double s = 0.0;
    bool on = q < nr;
    if (on) {
      const long long e0 = rp[i], e1 = rp[i + 1];
      on = L == 32 || e1 - e0 <= kLongRow * L;
      if (on) s = row_share<L>(e0 + sub, e1, col, val, x);
      else *any_long = 1;
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, L);
    if (on && sub == 0) {
      const double ri = __dsub_rn(b[i], s);
      r[i] = ri;
      acc += ri * ri;
    }
  }
  return acc;
}

// the rows of more than `limit` entries, a warp each in the rows' order
__device__ __noinline__ double long_rows(int r0, int nr, int limit, const long long *__restrict__ rp,
                                         const int *__restrict__ col, const double *__restrict__ val,
                                         const double *__restrict__ x, const double *__restrict__ b,
                                         double *__restrict__ r) {
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  for (int q0 = 0; q0 < nr; q0 += kThreads) {
    const int q = q0 + threadIdx.x;
    unsigned todo = __ballot_sync(0xffffffffu, q < nr && rp[r0 + q + 1] - rp[r0 + q] > limit);
    for (; todo; todo &= todo - 1) {
      const int i = r0 + q - lane + __ffs(todo) - 1;
      double s = row_share<32>(rp[i] + lane, rp[i + 1], col, val, x);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) {
        const double ri = __dsub_rn(b[i], s);
        r[i] = ri;
        acc += ri * ri;
      }
    }
  }
  return acc;
}

// r = b - A x for rows [blk*rpb, (blk+1)*rpb); partial[blk] = sum r_i^2.
// HBM bound: each block takes about 12 entries per lane for its own rows
// (rows of a 7-point stencil: one lane each).  Eight lanes for every row left
// one of eight idle, three shuffles per row and one load in flight.
__global__ void __launch_bounds__(kThreads)
residual_partials(int n, int rpb, const long long *__restrict__ rp, const int *__restrict__ col,
                  const double *__restrict__ val, const double *__restrict__ x,
                  const double *__restrict__ b, double *__restrict__ r, double *__restrict__ partial) {
  __shared__ double sh[kThreads / 32];
  __shared__ int any_long;
  const int r0 = blockIdx.x * rpb;
  const int nr = min(n - r0, rpb);
  const long long per = (rp[r0 + nr] - rp[r0]) / nr;
  if (threadIdx.x == 0) any_long = 0;
  __syncthreads();
  double acc;
  if (per <= 12) acc = block_rows<1>(r0, nr, rp, col, val, x, b, r, &any_long);
  else if (per <= 48) acc = block_rows<4>(r0, nr, rp, col, val, x, b, r, &any_long);
  else if (per <= 192) acc = block_rows<16>(r0, nr, rp, col, val, x, b, r, &any_long);
  else acc = block_rows<32>(r0, nr, rp, col, val, x, b, r, &any_long);
  __syncthreads();
  if (any_long) acc += long_rows(r0, nr, kLongRow * (per <= 12 ? 1 : per <= 48 ? 4 : 16), rp, col, val, x, b, r);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; w++) t += sh[w];
    partial[blockIdx.x] = t;
  }
}

// out = sum of partial[0..np) in a fixed order (one block)
__global__ void __launch_bounds__(kThreads)
sum_partials_ordered(int np, const double *__restrict__ partial, double *__restrict__ out) {
  __shared__ double sh[kThreads];
  double s = 0.0;
  for (int q = threadIdx.x; q < np; q += kThreads) s += partial[q];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = kThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// rows per block: 1,024 for large systems; a quarter of that keeps more SMs
// busy below about eight blocks per SM
int rows_per_block(int n) { return n >= 1200 * kMaxRowsPerBlock ? kMaxRowsPerBlock : kMaxRowsPerBlock / 4; }
int blocks_for(int n) {
  const int rpb = rows_per_block(n);
  return (int)(((long long)n + rpb - 1) / rpb);
}

// Scratch of dg_residual_csr: a memory pool of its own per device that keeps
// its memory between calls, up to kPoolKeep bytes.  The default pool gives
// everything back to the driver at each synchronisation, so that every call
// after one pays for a new mapping.  The threshold is compared with what the
// pool has reserved, which comes in chunks of 2 MB and more, not
// with what is in use: one of 1 MB kept nothing.  A
// call and a synchronisation: 24^3 185 -> 22 us, 128^3 224 -> 72 us (without a
// pool 203 and 393); back to back 10 and 61 us; a first call on new data, 128^3:
// 340 -> 110 us.
// Allocation and release stay stream ordered: any number of threads and
// streams may call at once.  The pool belongs to the context (its id is kept
// beside it) and goes with it.
constexpr unsigned long long kPoolKeep = 64ull << 20;
constexpr int kMaxDevices = 128;
cudaError_t current_context_id(unsigned long long *id);

struct ScratchPool {
  cudaMemPool_t pool = nullptr;
  unsigned long long ctx = 0;
};
ScratchPool g_pool[kMaxDevices];
std::mutex g_mu;  // this table, the fixed scratch's and the driver entry points below

cudaMemPool_t scratch_pool(int dev) {  // null: use the device's default pool
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(g_mu);
  unsigned long long ctx = 0;
  if (current_context_id(&ctx) != cudaSuccess || ctx == 0) return nullptr;
  ScratchPool &p = g_pool[dev];
  if (p.pool && p.ctx == ctx) return p.pool;
  p = ScratchPool{};
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  unsigned long long keep = kPoolKeep;
  // another stream of this thread may be under capture: creating the pool
  // counts as little as possible against it (the allocation itself is an
  // unsafe call beside a capture in the stricter modes, from any pool)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  const cudaError_t made = cudaMemPoolCreate(&pool, &props);
  if (made == cudaSuccess) cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  cudaThreadExchangeStreamCaptureMode(&mode);
  cudaGetLastError();
  if (made != cudaSuccess) return nullptr;
  p.pool = pool;
  p.ctx = ctx;
  return pool;
}

// stream-ordered scratch: from the kept pool of the stream's own device,
// which must be the current one; while the stream is captured (and anywhere
// else the pool cannot be had) from the default pool
cudaError_t alloc_scratch(double **p, size_t bytes, cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  int cur = -1, dev = -1;
  if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone &&
      cudaGetDevice(&cur) == cudaSuccess && cudaStreamGetDevice(s, &dev) == cudaSuccess && cur == dev) {
    cudaMemPool_t pool = scratch_pool(dev);
    if (pool) {
      if (cudaMallocFromPoolAsync(reinterpret_cast<void **>(p), bytes, pool, s) == cudaSuccess) return cudaSuccess;
      cudaGetLastError();
    }
  } else {
    cudaGetLastError();
  }
  return cudaMallocAsync(p, bytes, s);
}

}  // namespace resid
}  // namespace dg

extern "C" dg_status dg_residual_csr(int n, const long long *d_rowptr, const int *d_col,
                                     const double *d_val, const double *d_x, const double *d_b,
                                     double *d_r, double *d_norm2, void *cuda_stream) {
  using namespace dg::resid;
  if (n <= 0 || !d_rowptr || !d_col || !d_val || !d_x || !d_b || !d_r || !d_norm2) return DG_BAD_INPUT;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  const int nb = blocks_for(n);
  double *partial = nullptr;
  if (alloc_scratch(&partial, (size_t)nb * sizeof(double), s) != cudaSuccess) return DG_CUDA_ERROR;
  residual_partials<<<nb, kThreads, 0, s>>>(n, rows_per_block(n), d_rowptr, d_col, d_val, d_x, d_b, d_r, partial);
  sum_partials_ordered<<<1, kThreads, 0, s>>>(nb, partial, d_norm2);
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(partial, s);
  return e == cudaSuccess ? DG_OK : DG_CUDA_ERROR;
}

// ---------------------------------------------------------------------------
// Allocation-free variant.
//
// Some callers cannot allocate device memory at the point where they need
// the residual: an application that hands all device memory to its own pool
// and forbids other allocations, code that runs while another component is
// capturing the stream into a CUDA graph (where cudaMalloc is not allowed),
// or a latency-critical loop that must not pay for an allocation's implicit
// synchronisation.  dg_residual_csr_noalloc gives them the same result as
// dg_residual_csr without calling cudaMalloc, cudaFree or any allocating
// routine: its partial sums live in the fixed array below, which is part of
// the library image and stays resident on every GPU that loads the library
// until the process exits.
// ---------------------------------------------------------------------------
namespace dg {
namespace resid {

constexpr int kNoAllocMaxPartials = 65536;  // 512 KiB of doubles
constexpr long long kNoAllocMaxRows = (long long)kNoAllocMaxPartials * kMaxRowsPerBlock;  // 67,108,864

static __device__ __align__(256) double g_noalloc_partials[kNoAllocMaxPartials];

// Host code may not use g_noalloc_partials as an address: on the host the
// name refers to a stand-in variable, not to device memory.  The device
// address is looked up with the device current and cached per device,
// together with the id of the CUDA context it belongs to: after a
// cudaDeviceReset the device gets a new primary context, into which the
// library's module (and the array) is loaded again, possibly elsewhere, so a
// changed context id makes the next call look the address up again.
static double *g_noalloc_ptr[kMaxDevices];
static unsigned long long g_noalloc_ctx[kMaxDevices];

// cuCtxGetCurrent / cuCtxGetId through the runtime's driver entry points,
// so that the library does not link the driver library itself.
typedef int (*ctx_get_current_fn)(void **ctx);
typedef int (*ctx_get_id_fn)(void *ctx, unsigned long long *id);
static ctx_get_current_fn g_ctx_get_current;
static ctx_get_id_fn g_ctx_get_id;

// The id of the calling thread's current context (0: none yet).
cudaError_t current_context_id(unsigned long long *id) {
  *id = 0;
  if (!g_ctx_get_current || !g_ctx_get_id) {
    cudaDriverEntryPointQueryResult q1, q2;
    void *f1 = nullptr, *f2 = nullptr;
    cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1);
    if (e != cudaSuccess || q1 != cudaDriverEntryPointSuccess) return e != cudaSuccess ? e : cudaErrorNotSupported;
    e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2);
    if (e != cudaSuccess || q2 != cudaDriverEntryPointSuccess) return e != cudaSuccess ? e : cudaErrorNotSupported;
    g_ctx_get_current = reinterpret_cast<ctx_get_current_fn>(f1);
    g_ctx_get_id = reinterpret_cast<ctx_get_id_fn>(f2);
  }
  void *ctx = nullptr;
  if (g_ctx_get_current(&ctx) != 0) return cudaErrorUnknown;
  if (!ctx) return cudaSuccess;
  if (g_ctx_get_id(ctx, id) != 0) return cudaErrorUnknown;
  return cudaSuccess;
}

static cudaError_t noalloc_scratch(double **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_mu);
  unsigned long long ctx = 0;
  e = current_context_id(&ctx);
  if (e != cudaSuccess) return e;
  if (!g_noalloc_ptr[dev] || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
    double *p = nullptr;
    // loads the module into the device's primary context if it is not yet
    e = cudaGetSymbolAddress(reinterpret_cast<void **>(&p), g_noalloc_partials);
    if (e != cudaSuccess) return e;
    e = current_context_id(&ctx);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev] = p;
    g_noalloc_ctx[dev] = ctx;
  }
  *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

}  // namespace resid
}  // namespace dg

extern "C" dg_status dg_residual_csr_noalloc(int n, const long long *d_rowptr, const int *d_col,
                                             const double *d_val, const double *d_x, const double *d_b,
                                             double *d_r, double *d_norm2, void *cuda_stream) {
  using namespace dg::resid;
  if (n <= 0 || !d_rowptr || !d_col || !d_val || !d_x || !d_b || !d_r || !d_norm2) return DG_BAD_INPUT;
  if ((long long)n > kNoAllocMaxRows) return DG_BAD_INPUT;  // the fixed scratch holds 65,536 partials
  double *partial = nullptr;
  if (noalloc_scratch(&partial) != cudaSuccess) return DG_CUDA_ERROR;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  const int nb = blocks_for(n);
  // every partial of [0, nb) is written before it is read, so the contents
  // left by an earlier call need no clearing
  residual_partials<<<nb, kThreads, 0, s>>>(n, rows_per_block(n), d_rowptr, d_col, d_val, d_x, d_b, d_r, partial);
  sum_partials_ordered<<<1, kThreads, 0, s>>>(nb, partial, d_norm2);
  return cudaGetLastError() == cudaSuccess ? DG_OK : DG_CUDA_ERROR;
}
