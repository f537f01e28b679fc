// FP64 super-panel updates of the large fronts on the tensor cores.
//
// The update C -= A B^T (A, B: up to 128 columns of L, or of E) is a
// contraction whose FP64 multiply-adds the GPU issues at 2 per clock and SM.
// Here every row of A and B is written as integers of its own scale,
//     a = x 2^(e - 62),  |x| < 2^62,  x = sum_i q_i 2^(8 (7 - i)),
// e one above the exponent of the row's largest entry and q_i in [-128, 127]
// (q_0 in [-64, 64]): eight F16 slices that hold the digits exactly.  The
// tensor cores form the integer products
//     D_s = sum over i + j = s of Q_i Q_j^T,   s = 0 .. 7,
// in FP32 accumulators: |D_s| <= 8 * 128 * 2^14 = 2^24 for 128 columns, so
// every accumulator is exact, and the epilogue adds them as integers and
// rounds once.  What is dropped (s >= 8) is below 2^-58 (root mean square;
// 2^-53 at most) of the two rows' largest entries times each other, where a
// chain of 128 FP64 multiply-adds rounds by 2^-53 of its partial sums each
// time.  An entry more than nine binary orders below its row's largest keeps
// fewer bits than its own 53, so that a sum of such entries alone is not what
// the chain gives, entry by entry; the factor's error bound is in the rows'
// sizes (sqrt(c_ii c_jj) for the entry (i, j) of the Schur complement) either
// way.  Direct solves of one subdomain (3-D log-normal diffusion 14^3 .. 26^3,
// Poisson 65^2 .. 200^2, elasticity 6^3 .. 11^3, six seeds, four right-hand
// sides): residuals with this 0.95 to 1.01 times those of the CUDA cores, errors
// against 64 bits 0.84 to 1.16 times (geometric mean 0.99).  (Ozaki, Ogita, Oishi and Rump, error-free transformation of a matrix
// product by slices, Numer. Algorithms 59, 2012.)
//
// mf_split writes the slices once per super-panel, in the shared-memory
// layout of the MMA, so that mf_update_split only copies and multiplies:
// block b = 64 rows x 128 columns, as [2 chunks of 64 columns][8 slices]
// [64 rows x 128 bytes, SWIZZLE_128B], 128 KB; expo[64 b + r] is the row's
// biased largest exponent.
#pragma once
#include <cuda_fp16.h>

namespace dg {

constexpr int kSplit = 8;                                   // slices
constexpr int kSplitRows = 64;                              // rows of a block
constexpr uint32_t kSplitTile = kSplitRows * 64 * 2;        // bytes of one slice of a chunk: 8 KB
constexpr uint32_t kSplitBlock = 2 * kSplit * kSplitTile;   // bytes of a block: 128 KB
constexpr int kSplitK = 128;                                // largest K with exact accumulators
constexpr int kSplitNan = 1 << 20;                          // expo of a row with an infinity or a NaN
constexpr size_t kSplitSmem = kSplit * 3 * (size_t)kSplitTile + 1024;  // A (two blocks) and B of one chunk
constexpr int kSplitCtaRows = 32;                           // rows per CTA of mf_split

// 16 digits-of-a-slice bytes: byte s of eight integers (bias 128) as F16
__device__ __forceinline__ uint4 slice_f16(const uint32_t (&w)[8], int byte) {
  uint4 o;
  uint32_t *p = &o.x;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    // 1024 + d as F16 is 0x6400 | d for d < 1024; minus 1152 leaves d - 128
    const uint32_t b = __byte_perm(w[2 * u], w[2 * u + 1], (uint32_t)byte | (uint32_t)(byte + 4) << 8);
    const uint32_t h = __byte_perm(b, 0x64646464u, 0x4240u);
    __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&h), __half2half2(__ushort_as_half(0x6480)));
    p[u] = *reinterpret_cast<uint32_t *>(&v);
  }
  return o;
}

// task = {front, first row (rows of L below the super-panel) or ~first column
// (of E), 32-row half block, -}.  Eight lanes per row, 16 columns each: lane c
// the columns 8c.. of both chunks.  Rows past the matrix and columns past K
// are zero.  Bound by the loads of L and the stores of the slices (16 bytes
// per entry), both whole sectors: 10844 CTAs 82 us.
__global__ void __launch_bounds__(256)
mf_split(MfView v, const int4 *__restrict__ tasks, int jl, int kw, const double *__restrict__ arena,
         const double *__restrict__ E, unsigned char *__restrict__ slices, int *__restrict__ expo) {
  const int4 t = tasks[blockIdx.x];
  const int m = v.f_m[t.x], k = v.f_k[t.x], K = min(kw, k - jl);
  const bool ecol = t.y < 0;
  const int lane = threadIdx.x & 31, c = lane & 7;
  const int r = (threadIdx.x >> 5) * 4 + (lane >> 3);  // row of the half block
  const int row = (ecol ? ~t.y : t.y) + r;
  const bool on = row < (ecol ? jl + K : m);
  // entry (row, t) at p[t * st]
  const double *p = ecol ? E + v.e_off[t.x] + (int64_t)row * round4(m) + jl : arena + v.f_off[t.x] + (int64_t)jl * m + row;
  const int64_t st = ecol ? 1 : m;
  unsigned long long a[2][8];
  int e = 1;  // subnormal numbers have the exponent of the smallest normal ones
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int q = 64 * h + 8 * c + u;
      a[h][u] = on && q < K ? (unsigned long long)__double_as_longlong(p[q * st]) : 0ull;
    }
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int u = 0; u < 8; u++) e = max(e, (int)(a[h][u] >> 52) & 0x7ff);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  const int half = t.z, blk = half >> 1, br = (half & 1) * kSplitCtaRows + r;
  if (c == 0) expo[blk * kSplitRows + br] = e == 0x7ff ? kSplitNan : e;
  unsigned char *dst = slices + (size_t)blk * kSplitBlock + tc::sw128_chunk_f16(br, c);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (64 * h >= K) break;
    uint32_t lo[8], hi[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int eu = (int)(a[h][u] >> 52) & 0x7ff;
      const unsigned long long man = (a[h][u] & ((1ull << 52) - 1)) | (eu ? 1ull << 52 : 0ull);
      const int sh = e - (eu ? eu : 1);
      long long x = (long long)(sh < 63 ? (man << 9) >> sh : 0ull);
      if ((long long)a[h][u] < 0) x = -x;
      // balanced digits: after adding 128 to every digit the bytes are q + 128
      const unsigned long long b = (unsigned long long)x + 0x8080808080808080ull;
      lo[u] = (uint32_t)b;
      hi[u] = (uint32_t)(b >> 32);
    }
    unsigned char *d = dst + (size_t)h * kSplit * kSplitTile;
#pragma unroll
    for (int s = 0; s < kSplit; s++)
      *reinterpret_cast<uint4 *>(d + s * kSplitTile) = s < 4 ? slice_f16(hi, 3 - s) : slice_f16(lo, 7 - s);
  }
}

// top 2^-drop units of the last subnormal place, rounded to nearest (a call:
// the shifts in line cost the epilogue of every entry)
__device__ __noinline__ double split_subnormal(unsigned long long top, int drop) {
  if (drop > 64) return 0.0;
  return __longlong_as_double((long long)(((top >> 1) >> (drop - 1)) + ((top >> (drop - 1)) & 1)));
}

// sum_s d[s] 2^(8 (7 - s)) * 2^(ex - 2112), rounded to nearest (subnormal
// numbers too); the d[s] are integers of at most 2^24, ex the sum of the two
// rows' biased exponents
__device__ __forceinline__ double split_value(const int (&d)[kSplit], int ex) {
  long long h = ((long long)d[0] << 24) + ((long long)d[1] << 16) + ((long long)d[2] << 8) + d[3];
  const long long l = ((long long)d[4] << 24) + ((long long)d[5] << 16) + ((long long)d[6] << 8) + d[7];
  h += l >> 32;
  uint32_t lo = (uint32_t)l;
  const bool neg = h < 0;
  if (neg) {
    lo = 0u - lo;
    h = ~h + (lo == 0);
  }
  // |h| < 2^49: the value's 81 bits as 64 + 17
  const unsigned long long a = (unsigned long long)h << 15 | lo >> 17;
  const unsigned long long b = (unsigned long long)(lo & 0x1ffffu) << 47;
  const int n = a ? __clzll((long long)a) : 64 + __clzll((long long)b);
  const unsigned long long top = n == 0 ? a : n < 64 ? a << n | b >> (64 - n) : b << (n & 63);
  const int fe = 1023 + 80 - n + ex - 2112;  // biased exponent of the leading bit
  const unsigned long long bits = ((unsigned long long)(fe - 1) << 52) + (top >> 11) + ((top >> 10) & 1);
  double r = __longlong_as_double((long long)bits);
  if (fe > 2046) r = __longlong_as_double(0x7ff0000000000000ll);
  if ((a | b) == 0) r = 0.0;
  else if (fe < 1) r = split_subnormal(top, 12 - fe);
  if (ex >= kSplitNan) r = __longlong_as_double(0x7ff8000000000000ll);
  return neg ? -r : r;
}

// 128 x 64 tiles: task = {front, (ti << 16) | tj, first block of A (rows
// c0 + 128 ti ..), block of B}.  Trailing tiles (task < nupd):
// C[rows, cols] -= A B^T for the rows and columns from c0 = jl + K (lower
// part); E tiles: E[rows, cols] -= L E_J for the columns below c0 (block J's
// columns are assigned).  One persistent CTA per SM: shared memory holds the
// 16 slices of one 64-column chunk (192 KB), tensor memory the eight
// accumulators (all 512 columns).  The last warp copies the slices and
// issues the MMAs; the others read the tile's old values meanwhile and run the epilogue,
// under which the next tile's first slices arrive.  The first chunk is
// multiplied in the order in which its slices arrive (pairs by their larger
// index), which frees them from the middle outwards: slices 3 and 4 first,
// then 2 and 5, 1 and 6, 0 and 7; the second chunk's copies and products
// follow in that order.  Per tile of 128 columns 18.5 us, where the FP64 pipe
// takes 273 us for the same multiply-adds: about 7 us of it the MMAs (288 of
// 128 x 64 x 16), the rest the epilogue (eight conversions to integer and some
// hundred integer operations per entry; FP64 operations would take longer:
// one per entry is the subtraction), so 16 warps run it, and its loop is not
// unrolled: cold code costs a short launch 10 us.  64 subdomains of 96^3:
// all super-panel updates 72 ms -> 10 ms.  Every wait is bounded: whoever runs
// out of polls (the epilogue has epi_polls of them a tile) sets ERR_WAIT and
// tells the others, the copying warp waits once more for its copies and MMAs
// in flight, and the CTA frees its tensor memory.
constexpr int kSplitEpi = 512;  // threads of the epilogue
constexpr int kSplitThreads = kSplitEpi + 32;

// waits for a phase as tc::mbar_wait does, but not on after someone gave up
__device__ __forceinline__ bool split_wait(uint64_t *bar, uint32_t parity, long long polls, const volatile int *gave_up) {
  constexpr int kChunk = 1024;
  for (; polls > 0; polls -= kChunk) {
    if (tc::mbar_wait(bar, parity, polls < kChunk ? polls : kChunk)) return true;
    if (*gave_up) return false;
  }
  return false;
}

__global__ void __launch_bounds__(kSplitThreads, 1)
mf_update_split(MfView v, const int4 *__restrict__ tasks, int ntasks, int nupd, int jl, int kw,
                const unsigned char *__restrict__ slices, const int *__restrict__ expo, double *__restrict__ arena,
                double *__restrict__ E, int *__restrict__ status, long long epi_polls) {
  extern __shared__ unsigned char tc_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) &
                                                          ~static_cast<uintptr_t>(1023));
  constexpr int G = kSplit / 2;  // slice groups of the second chunk: {3,4} {2,5} {1,6} {0,7}
  __shared__ __align__(8) uint64_t full0[kSplit], full1[G], freed[G], done, empty, drain;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == kSplitEpi / 32) tc::tmem_alloc(&tmem_slot, 512);
  if (tid == 0) {
    gave_up = 0;
    for (int i = 0; i < kSplit; i++) tc::mbar_init_nofence(&full0[i], 1);
    for (int i = 0; i < G; i++) {
      tc::mbar_init_nofence(&full1[i], 1);
      tc::mbar_init_nofence(&freed[i], 1);
    }
    tc::mbar_init_nofence(&done, 1);
    tc::mbar_init_nofence(&empty, kSplitEpi / 32);
    tc::mbar_init_nofence(&drain, 1);
    tc::mbar_init_fence();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  const uint32_t sA = tc::smem_u32(base), sB = sA + kSplit * 2 * kSplitTile;
  bool ok = true;
  if (tid == kSplitEpi) {
    // copies and products: the barriers' phases are counted here and in the
    // epilogue, both of which pass each of them once per tile (full1 and
    // freed: once per tile of more than 64 columns)
    auto load = [&](const int4 &t, int i, int chunk, uint64_t *bar) {
      const unsigned char *a = slices + (size_t)t.z * kSplitBlock, *b = slices + (size_t)t.w * kSplitBlock;
      const size_t o = (size_t)(chunk * kSplit + i) * kSplitTile;
      tc::bulk_load(sA + i * 2 * kSplitTile, a + o, kSplitTile, bar);
      tc::bulk_load(sA + (i * 2 + 1) * kSplitTile, a + kSplitBlock + o, kSplitTile, bar);
      tc::bulk_load(sB + i * kSplitTile, b + o, kSplitTile, bar);
    };
    auto load_first = [&](const int4 &t) {
      for (int i = 0; i < kSplit; i++) {
        tc::mbar_expect(&full0[i], 3 * kSplitTile);
        load(t, i, 0, &full0[i]);
      }
    };
    constexpr uint32_t idesc = tc::idesc_f16(128, kSplitRows);
    // the loops over slices are unrolled: descriptors and accumulate flags are
    // constants apart from their bases, and one thread keeps up with the MMAs
    const uint64_t dA = tc::sw128_desc(sA), dB = tc::sw128_desc(sB);
    auto mul = [&](int i, int j, int ks, bool first) {
      const uint64_t a = dA + (uint32_t)(i * 2 * kSplitTile >> 4), b = dB + (uint32_t)(j * kSplitTile >> 4);
#pragma unroll
      for (int q = 0; q < 4; q++)  // 16 columns (32 bytes) per MMA
        if (q < ks) tc::mma_f16(tmem + 64 * (i + j), a + 2 * q, b + 2 * q, idesc, first && q == 0 ? 0u : 1u);
    };
    uint32_t p0 = 0, p1 = 0, pe = 0;  // phases of full0 and done, of full1 and freed, of empty
    int t = blockIdx.x, armed = 0;    // armed: full1 copies of this tile
    int4 task = tasks[t];
    load_first(task);
    for (;;) {
      const int K = min(kw, v.f_k[task.x] - jl);
      const bool two = K > 64;
      const int ks0 = (min(K, 64) + 15) / 16, ks1 = (K - 64 + 15) / 16;
      armed = 0;
      if (t != (int)blockIdx.x) {  // the epilogue has read the accumulators
        ok = split_wait(&empty, pe, kTcWaitPolls, &gave_up);
        pe ^= 1;
        if (!ok) break;
        tc::fence_after_sync();
      }
      // pairs (x, j) and (j, x), j <= min(x, 7 - x); the steps before x have
      // started the sums up to 2 x - 2 (all of them from x = 5 on)
#pragma unroll
      for (int x = 0; x < kSplit; x++) {
        if (ok) ok = tc::mbar_wait(&full0[x], p0, kTcWaitPolls);
        if (ok) {
          tc::fence_after_sync();
#pragma unroll
          for (int j = 0; j < G; j++)
            if (j <= x && j <= kSplit - 1 - x) {
              mul(x, j, ks0, x <= G && x + j > 2 * x - 2);
              if (j != x) mul(j, x, ks0, false);
            }
          if (two && x >= G) tc::mma_commit(tc::smem_u32(&freed[x - G]));
        }
      }
      for (int g = 0; two && g < G && ok; g++) {  // 48 KB each
        ok = tc::mbar_wait(&freed[g], p1, kTcWaitPolls);
        if (!ok) break;
        tc::mbar_expect(&full1[g], 6 * kSplitTile);
        load(task, G - 1 - g, 1, &full1[g]);
        load(task, G + g, 1, &full1[g]);
        armed = g + 1;
      }
#pragma unroll
      for (int g = 0; g < G; g++) {
        if (two && ok) ok = tc::mbar_wait(&full1[g], p1, kTcWaitPolls);
        if (two && ok) {
          tc::fence_after_sync();
          // pairs of the slices lo .. hi that involve lo or hi
          const int lo = G - 1 - g;
#pragma unroll
          for (int j = 0; j < kSplit; j++)
            if (j >= lo && j <= G + g) {
              mul(lo, j, ks1, false);
              if (j != lo) mul(j, lo, ks1, false);
            }
        }
      }
      if (!ok) break;
      tc::mma_commit(tc::smem_u32(&done));
      t += gridDim.x;
      if (t >= ntasks) {  // (the last tile's MMAs too use the tensor memory)
        ok = tc::mbar_wait(&done, p0, kTcWaitPolls);
        break;
      }
      task = tasks[t];
      ok = tc::mbar_wait(&done, p0, kTcWaitPolls);
      if (!ok) break;
      p0 ^= 1;
      if (two) p1 ^= 1;
      load_first(task);
    }
    if (!ok) {  // no copy and no MMA of this CTA may be left in flight
      gave_up = 1;
      atomicOr(status, ERR_WAIT);
      for (int i = 0; i < kSplit; i++) tc::mbar_wait(&full0[i], p0, kTcWaitPolls);
      for (int i = 0; i < armed; i++) tc::mbar_wait(&full1[i], p1, kTcWaitPolls);
      tc::mma_commit(tc::smem_u32(&drain));
      tc::mbar_wait(&drain, 0, kTcWaitPolls);
    }
  } else if (tid < kSplitEpi) {
    const int lg = warp & 3, cw = (warp >> 2) * 16, lrow = 32 * lg + lane;
    uint32_t ph = 0;
    for (int t = blockIdx.x; t < ntasks; t += gridDim.x) {
      const bool etile = t >= nupd;
      const int4 task = tasks[t];
      const int f = task.x, ti = task.y >> 16, tj = task.y & 0xffff;
      const int m = v.f_m[f], k = v.f_k[f];
      const int c0 = jl + min(kw, k - jl), row = c0 + ti * 128 + lrow;
      const int colb = (etile ? 0 : c0) + tj * kSplitRows + cw;
      double *C = etile ? E + v.e_off[f] : arena + v.f_off[f];
      const int64_t cs = etile ? round4(m) : m;
      // columns of this row that the tile writes, those that hold a value
      const int clim = row < m ? (etile ? c0 : min(m, row + 1)) - colb : 0;
      const int cold = etile && row < m ? jl - colb : clim;
      C += colb * cs + row;
      // the old values: the first while the tensor cores work, then two
      // columns ahead
      double cur[4];
#pragma unroll
      for (int c = 0; c < 4; c++) cur[c] = c < cold ? C[c * cs] : 0.0;
      const int ea = expo[task.z * kSplitRows + lrow], eb = expo[task.w * kSplitRows + cw + (lane & 15)];
      // a warp that gave up once waits no more, but meets the others below
      if (ok) {
        ok = __all_sync(0xffffffffu, split_wait(&done, ph, epi_polls, &gave_up));
        if (!ok && lane == 0) {
          gave_up = 1;
          atomicOr(status, ERR_WAIT);
        }
      }
      ph ^= 1;
      tc::fence_after_sync();
#pragma unroll 1
      for (int h = 0; h < (ok ? 8 : 0); h++) {
        float d[16];
        __syncwarp();
        tc::tmem_load_8x2(tmem + ((uint32_t)(32 * lg) << 16) + (uint32_t)(cw + 2 * h), d);
        if (h == 7) {  // the accumulators are read: the next tile's products may start
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(&empty);
        }
        double nxt[2];
#pragma unroll
        for (int c = 0; c < 2; c++) nxt[c] = 2 * h + 4 + c < min(cold, 16) ? C[(4 + c) * cs] : 0.0;
#pragma unroll
        for (int c = 0; c < 2; c++) {
          const int ex = ea + __shfl_sync(0xffffffffu, eb, 2 * h + c);
          int q[kSplit];
#pragma unroll
          for (int s = 0; s < kSplit; s++) q[s] = __float2int_rn(d[2 * s + c]);
          const double x = cur[c] - split_value(q, ex);  // (no branch: two columns at once)
          if (2 * h + c < clim) C[c * cs] = x;
          cur[c] = cur[2 + c];
          cur[2 + c] = nxt[c];
        }
        C += 2 * cs;
      }
      // trailing tile (0, 0) holds the next super-panel's first diagonal
      // block: this was its last update
      if (!etile && ti == 0 && tj == 0 && c0 < k) {
        asm volatile("bar.sync 2, %0;" ::"n"(kSplitEpi) : "memory");
        if (tid < kMfThreads) {
          factor_diag_block<double, true>(arena + v.f_off[f], m, c0, min(kNB, k - c0), status);
          diag_sync<true>();
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kSplitEpi / 32) tc::tmem_free(tmem, 512);
}

}  // namespace dg
