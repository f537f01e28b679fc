// sm_103a kernels of the GB300 solve path.
//
//   * batched multifrontal Cholesky (assembly + extend-add + partial
//     factorisation), one launch per assembly-tree level for all subdomains;
//   * multifrontal forward / backward solves, one launch per level;
//   * Schwarz gather and deterministic "pull" sum of subdomain solutions
//     (the reference adds subdomain solutions in subdomain order,
//     src/solvers/subsolvers.F90:68-73, then the coarse correction,
//     src/solvers/pcg.F90:191-193; the pull kernel adds in that same order);
//   * restriction / prolongation with R and P = R^T (src/solvers/pcg.F90:149,188);
//   * CSR SpMV fused with the CG direction update and the p.q partial sums;
//   * fused PCG vector updates with deterministic two-pass reductions.
//
// The level kernels wait only at hardware barriers (__syncthreads,
// __syncwarp, griddepcontrol.wait).  The optional dependency-driven solve
// schedule (mf_fwd_queue / mf_bwd_queue, option solve_schedule 1) polls the
// done flags of its producer tasks with clock64 + __nanosleep; every such
// wait is bounded, and on timeout it sets ERR_WAIT in the error word, skips
// the task's remaining waits and returns, and the host reports DG_CUDA_ERROR.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "dg_tc.cuh"

namespace dg {

constexpr int kRedBlocks = 1024;   // most partial sums of a reduction
constexpr int kVecThreads = 256;

// device error word bits
enum : int { ERR_NOT_SPD = 1, ERR_NAN = 2, ERR_BREAKDOWN = 4, ERR_WAIT = 8 };

// one entry of a front's child list (child ci of f_children): the child's
// relative-row map offset, update-vector offset and update-row count
struct ChildEdge {
  int64_t relmap, uoff;
  int rc, pad;
};

// What a solve reads about a front, in one load: beside each large-front
// task, and per front for the small ones.  tab: per row of the front its
// place in two children's update vectors (16 bits each, kNoChild: none), m
// words per pair of children, so that the right-hand side is gathered in one
// round of loads; cu0, cu1: the first two children's vectors, ch_edge[ch ..]:
// all nch children.  nch < 0: -nch children (more than kMostPairs, or one of
// 65,535 update rows and more) by lists instead, row i of the front the entries
// clist[cptr[tab + i] .. cptr[tab + i + 1]) of the update vectors, children in
// order: a row of a front with hundreds of children hears from a few of them.
struct __align__(16) SolveFront {
  int m, k;
  int64_t e_off;
  int64_t xo, xb;          // position of the first pivot, of the matrix's first row
  int64_t rows;            // offset into MfView::rows
  int64_t uoff;            // update vector
  int64_t tab;             // offset into the child table
  int64_t cu0, cu1;
  int nch, ch;
};
static_assert(sizeof(SolveFront) == 80, "five 16-byte loads");
constexpr unsigned kNoChild = 0xffffu;
constexpr int kMostPairs = 16;  // children in a table: what joined levels make of two each

struct MfView {  // device pointers of one multifrontal batch
  const int64_t *f_off;
  const int *f_m, *f_k;
  const int64_t *f_rows, *f_xoff;
  const int *f_p0;
  const int64_t *f_uoff, *f_woff;
  const int *f_child_ptr, *f_children;
  const int64_t *f_relmap, *f_asm;
  const int *rows, *relmap;
  const int64_t *asm_tgt, *asm_sp, *asm_src;
  const int64_t *e_off;        // offset of the front's elimination matrix E (m x k, ld round4(m))
  const ChildEdge *ch_edge;    // per child-list entry: see ChildEdge
  const SolveFront *sfront;    // per front: see SolveFront
  const unsigned *ctab;        // child tables
  const int64_t *cptr, *clist; // child lists
};

__host__ __device__ __forceinline__ int round4(int x) { return (x + 3) & ~3; }

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// block sum in a fixed order (result valid in thread 0)
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
  v = warp_sum(v);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  double s = 0.0;
  if (wid == 0) {
    s = lane < NT / 32 ? sh[lane] : 0.0;
    s = warp_sum(s);
  }
  __syncthreads();
  return s;
}

// Programmatic dependent launch of the level solves.  pdl_trigger (at the
// start of a CTA) lets the next kernel of the stream start its CTAs once
// every CTA of this one has started; pdl_wait returns once the previous
// kernel has completed and its writes are visible.  The solve bodies issue
// their first loads of E (written by the factorisation, before any of these
// kernels) and read their index lists, and only then wait, before they read a
// vector that the previous level wrote.  Without the launch attribute both
// instructions do nothing.  A kernel launched this way may find in an SM's L1
// what the kernel before it read there and other SMs have overwritten since:
// what both read and the earlier one writes is loaded past L1 (__ldcg), as the
// scalars and the ancestors' values are, or the launch is an ordinary one
// (the products after the direction p).  And a load through a const
// __restrict__ pointer may be moved above the wait: what the kernel before
// writes is not read through one (the gather before the first level does not
// trigger early for that reason).
__device__ __forceinline__ void pdl_trigger() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}
__device__ __forceinline__ void pdl_wait() {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 900
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// sum of np partials in a fixed order, by one warp; every lane gets the
// result.  (One FP64 addition of a warp takes 64 clocks, 1024 partials a
// microsecond: reductions over short vectors have fewer.)
__device__ __forceinline__ double sum_partials(const double *part, int np) {
  double s = 0.0;
  int lane = threadIdx.x & 31;
  for (int q0 = lane; q0 < np; q0 += 32 * 8) {  // eight loads in flight
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = q0 + 32 * u < np ? __ldcg(part + q0 + 32 * u) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (q0 - lane + 32 * u >= np) break;
      s += v[u];
    }
  }
  s = warp_sum(s);
  return __shfl_sync(0xffffffffu, s, 0);
}

// ---------------------------------------------------------------------------
// multifrontal numeric factorisation, one CTA per front of a level
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T tsqrt(T x);
template <>
__device__ __forceinline__ double tsqrt<double>(double x) { return sqrt(x); }
template <>
__device__ __forceinline__ float tsqrt<float>(float x) { return sqrtf(x); }

constexpr int kMfThreads = 256;
constexpr int kNB = 32;      // panel width
// Tile of mf_update: FP32 64 x 64 (4 x 4 per thread).  FP64 32 x 32: its pipe
// is the limit at any tile size, small tiles leave less padding and spread a
// short update over more SMs (one 64 x 64 x 32 tile took 32 us on its SM).
template <typename T> struct UpdTile { static constexpr int N = sizeof(T) == 8 ? 32 : 64; };

// Every factorisation kernel also produces the front's elimination matrix
//     E = [ L11^-1 ; -L21 L11^-1 ]     (m x k, column-major, ld = round4(m)),
// the partial forward elimination applied to the identity columns [I ; 0]:
// pivot j scales row j of E by 1/L(j,j) and subtracts L(i,j) times it from
// the rows i > j.  A forward solve of the front is then the product
// [y ; u] = E b1 + [0 ; b2] and a backward solve x1 = E^T [y ; x2]; neither
// has a dependency chain inside the front.  E needs L only while the panel
// that produced it is current, so the factor columns of the arena are dead
// once E is formed; the update (Schur complement) block stays in the arena
// for the parent's extend-add.

// 1 / d of a pivot d > 0.  FP64: the division of the language is a chain of
// some ten dependent FP64 operations, each 64 clocks and more on this pipe,
// between one pivot and the next.  Here the single-precision reciprocal of the
// significand (relative error below 2^-21) and one step of Chebyshev's
// third-order iteration (r (1 + e + e^2), e = 1 - x r; Traub, Iterative Methods
// for the Solution of Equations, 1964): three dependent FP64 operations,
// error e^3 < 2^-63 before the last rounding.
__device__ __forceinline__ double normal_inverse(double d) {  // d and 1 / d normal numbers
  const int hi = __double2hiint(d), lo = __double2loint(d), ex = hi >> 20;
  const double x = __hiloint2double((hi & 0xfffff) | 0x3ff00000, lo);  // in [1, 2)
  const float f = __int_as_float(0x3f800000 | (hi & 0xfffff) << 3 | (int)((unsigned)lo >> 29));
  const unsigned g = (unsigned)__float_as_int(__frcp_rn(f));  // in (1/2, 1]
  const double r = __hiloint2double((int)(g >> 3) + (896 << 20), (int)(g << 29));
  const double e = __fma_rn(-x, r, 1.0);
  const double y = __fma_rn(r, __fma_rn(e, e, e), r);
  return __hiloint2double(__double2hiint(y) + ((1023 - ex) << 20), __double2loint(y));
}
__device__ __forceinline__ float normal_inverse(float d) { return 1.0f / d; }

// The largest and smallest powers of two between which d and 1 / d are normal
// numbers, tested by the exponent (d > 0).
__device__ __forceinline__ bool plain_pivot(float d) { return (unsigned)((__float_as_int(d) >> 23) - 1) < 252u; }
__device__ __forceinline__ bool plain_pivot(double d) { return (unsigned)((__double2hiint(d) >> 20) - 1) < 2044u; }
template <typename T>
__device__ __forceinline__ T pivot_inverse(T d) { return plain_pivot(d) ? normal_inverse(d) : T(1) / d; }

// A pivot as the factorisations keep it: 1 / d, or a negative number where d
// or 1 / d is no normal number.  FP64: -d, and those divide; the sign is the
// same for a whole CTA and read in an integer operation (as in the reciprocal,
// FP64 operations beside the one product would show: 129^2 1.035 ms with a
// division that is never reached, 1.115 with products by a power of two).
// FP32: -1 / (d 2^64) or -1 / (d 2^-64), which the magnitude tells apart, and a
// product by that power or by one (48 grids 2.42 ms, with the division 2.49).
template <typename T> struct KeptPivot;
template <> struct KeptPivot<double> {
  double v;
  __device__ explicit KeptPivot(double kept) : v(kept) {}
  __device__ static double keep(double d) { return plain_pivot(d) ? normal_inverse(d) : -d; }
  __device__ bool whole() const { return __double2hiint(v) < 0; }
  __device__ double divide(double c) const {  // c / d
    if (whole()) return c / -v;
    return c * v;
  }
  __device__ double inverse_root() const {  // d^-1/2
    if (whole()) return 1.0 / sqrt(-v);
    return sqrt(v);
  }
};
template <> struct KeptPivot<float> {
  float v, up;
  __device__ explicit KeptPivot(float kept) : v(fabsf(kept)), up(kept >= 0.f ? 1.f : kept < -1.f ? 0x1p64f : 0x1p-64f) {}
  __device__ static float keep(float d) {
    if (plain_pivot(d)) return normal_inverse(d);
    return -1.f / (d * (d < 1.f ? 0x1p64f : 0x1p-64f));
  }
  __device__ float divide(float c) const { return c * up * v; }
  __device__ float inverse_root() const { return sqrtf(v) * (up == 1.f ? 1.f : up > 1.f ? 0x1p32f : 0x1p-32f); }
};

// Extend-add of column b of a child's update block into column pb of the
// parent (Dst = the parent's column base; row r of the column at
// Dst[r * stride]): rows a >= b, by the lanes of one warp.  kEaBatch rows
// per lane are loaded (child values, target rows, old target values) before
// any is stored, so a warp keeps many independent loads in flight; the
// targets of one child column are distinct.
constexpr int kEaBatch = 4;

template <typename T>
__device__ __forceinline__ void extend_add_column(T *__restrict__ Dst, const int *__restrict__ rel,
                                                  const T *__restrict__ Ucol, int b, int rc, int lane,
                                                  int stride = 1) {
  for (int a0 = b + lane; a0 < rc; a0 += 32 * kEaBatch) {
    int row[kEaBatch];
    T val[kEaBatch], old[kEaBatch];
#pragma unroll
    for (int u = 0; u < kEaBatch; u++) {
      const int a = a0 + 32 * u;
      row[u] = a < rc ? rel[a] * stride : 0;
      val[u] = a < rc ? Ucol[a] : T(0);
    }
#pragma unroll
    for (int u = 0; u < kEaBatch; u++)
      if (a0 + 32 * u < rc) old[u] = Dst[row[u]];
#pragma unroll
    for (int u = 0; u < kEaBatch; u++)
      if (a0 + 32 * u < rc) Dst[row[u]] = old[u] + val[u];
  }
}

// 16-byte vectors of T in shared memory
template <typename T> struct SVec;
template <> struct SVec<float> {
  static constexpr int N = 4;
  using V = float4;
  __device__ static __forceinline__ float get(const V &v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }
  __device__ static __forceinline__ void set(V &v, int q, float x) {
    if (q == 0) v.x = x; else if (q == 1) v.y = x; else if (q == 2) v.z = x; else v.w = x;
  }
};
template <> struct SVec<double> {
  static constexpr int N = 2;
  using V = double2;
  __device__ static __forceinline__ double get(const V &v, int q) { return q == 0 ? v.x : v.y; }
  __device__ static __forceinline__ void set(V &v, int q, double x) { if (q == 0) v.x = x; else v.y = x; }
};

// Row stride (elements) of the one-CTA kernel's panel in shared memory: whole
// 16-byte vectors, an odd number of them, so that the vectors of 8
// consecutive rows fall into 8 different bank groups.
template <typename T> __host__ __device__ constexpr int pan_ld(int k) {
  const int vn = 16 / (int)sizeof(T);
  int nv = (k + vn - 1) / vn;
  if ((nv & 1) == 0) nv++;
  return nv * vn;
}
// shared memory of one front: panel (m rows), unit lower factor (k rows), two
// multiplier rows, reciprocal pivots and their square roots
template <typename T> __host__ __device__ constexpr size_t pan_smem(int m, int k) {
  return ((size_t)m + k + 4) * pan_ld<T>(k) * sizeof(T);
}

// Fronts whose panel (m x k) and factor (k x k) fit in shared memory: one CTA
// per front.
//
//   1. The pivot columns are assembled into shared memory (row-major), the
//      update block in the arena.
//   2. A11 = Lt D Lt^T and Lt^-1, in place, one barrier per pivot: step j
//      subtracts li = P(i, j) / d_j times a multiplier row from row i, whose
//      columns left of j hold Lt^-1 so far and right of j the Schur
//      complement.  The multiplier row (row j of Lt^-1, 1, column j of the
//      Schur complement) is written by the threads of the step before.
//   3. Rows of L21 by substitution with Lt, four lanes per row, no barrier;
//      E11 = D^-1/2 Lt^-1.
//   4. E21 = -L21 E11, four lanes per row; E to global; the update block
//      receives -L21 L21^T in 4x4 register blocks.
//
// Only the k x k part walks the pivots one after the other; the m - k rows
// below (most of the work) take part in two products.  Updating all m rows of
// panel and E at every pivot instead, with two barriers, a square root and a
// division per row each time, took: 705 FP64 fronts of up to 56 x 24 123 us
// (now 77), 18 of up to 145 x 61 241 us (167), all one-CTA fronts of a 128^3
// problem in FP32 9.9 ms (8.9).  FP64 is bound by its pipe from there on.
constexpr int kPanThreads = 128;       // fronts of up to kPanWideRows rows
constexpr int kPanThreadsWide = 256;   // larger fronts
constexpr int kPanWideRows = 160;

template <typename T>
__global__ void __launch_bounds__(kPanThreadsWide)
mf_factor_panel(MfView v, const int *__restrict__ fronts, const double *__restrict__ vals,
                T *__restrict__ arena, T *__restrict__ E, int *__restrict__ status) {
  using SV = SVec<T>;
  using V = typename SV::V;
  constexpr int VN = SV::N;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int f = fronts[blockIdx.x];
  const int m = v.f_m[f], k = v.f_k[f], r = m - k;
  const int ldk = pan_ld<T>(k), nv = ldk / VN;
  T *P = reinterpret_cast<T *>(smem_raw);   // m x k panel, row-major, row stride ldk
  T *L = P + (size_t)m * ldk;               // k x k unit lower factor, likewise
  T *mul = L + (size_t)k * ldk;             // multiplier rows of even and odd steps
  T *inv = mul + 2 * ldk;                   // 1 / d_j
  T *rs = inv + ldk;                        // d_j^-1/2
  const int64_t off = v.f_off[f];
  T *F = arena + off;
  const int tid = threadIdx.x, nt = blockDim.x;
  // 1. zero: panel and factor in shared memory, update block in the arena
  {
    V z;
#pragma unroll
    for (int u = 0; u < VN; u++) SV::set(z, u, T(0));
    V *p = reinterpret_cast<V *>(P);
    for (int q = tid; q < (m + k + 2) * nv; q += nt) p[q] = z;
  }
  for (int c = 0; c < r; c++)
    for (int i = c + tid; i < r; i += nt) F[(int64_t)(k + c) * m + k + i] = T(0);
  __syncthreads();
  // original entries (each target once, duplicates summed in order)
  for (int64_t e = v.f_asm[f] + tid; e < v.f_asm[f + 1]; e += nt) {
    double sv = 0.0;
    for (int64_t q = v.asm_sp[e]; q < v.asm_sp[e + 1]; q++) sv += vals[v.asm_src[q]];
    const int64_t t = v.asm_tgt[e] - off;
    if (t < (int64_t)m * k) {
      const int col = (int)(t / m), row = (int)(t - (int64_t)col * m);
      P[(size_t)row * ldk + col] = (T)sv;
    } else {
      F[t] = (T)sv;
    }
  }
  __syncthreads();
  // extend-add of the children's update matrices, children in order
  for (int ci = v.f_child_ptr[f]; ci < v.f_child_ptr[f + 1]; ci++) {
    const int c = v.f_children[ci];
    const int mc = v.f_m[c], kc = v.f_k[c], rc = mc - kc;
    const T *U = arena + v.f_off[c] + (int64_t)kc * mc + kc;
    const int *rel = v.relmap + v.f_relmap[c];
    const int lane = tid & 31, wid = tid >> 5, nw = nt / 32;
    for (int b = wid; b < rc; b += nw) {
      const int col = rel[b];
      if (col < k) extend_add_column<T>(P + col, rel, U + (int64_t)b * mc, b, rc, lane, ldk);
      else extend_add_column<T>(F + (int64_t)col * m, rel, U + (int64_t)b * mc, b, rc, lane);
    }
    __syncthreads();
  }
  // 2. the pivots
  auto pivot = [&](T d, int j) {
    if (!(d > T(0))) {
      atomicOr(status, ERR_NOT_SPD);
      d = T(1);
    }
    inv[j] = KeptPivot<T>::keep(d);
  };
  for (int c = tid; c < k; c += nt) {
    const T x = P[(size_t)c * ldk];
    mul[c] = c == 0 ? T(1) : x;
    if (c == 0) pivot(x, 0);
  }
  __syncthreads();
  constexpr int TX = 4;  // threads per row
  const int tx = tid & (TX - 1), ty = tid / TX, ny = nt / TX;
  for (int j = 0; j < k - 1; j++) {
    const T *cur = mul + (j & 1) * ldk;
    T *nxt = mul + ((j + 1) & 1) * ldk;
    const KeptPivot<T> piv(inv[j]);
    for (int i = j + 1 + ty; i < k; i += ny) {
      const T li = piv.divide(cur[i]);
      if (tx == 0) L[(size_t)i * ldk + j] = li;
      V *row = reinterpret_cast<V *>(P + (size_t)i * ldk);
      // (entries right of the diagonal take garbage; nothing reads them)
      for (int q = tx; q * VN <= i; q += TX) {
        const V a = row[q], w = reinterpret_cast<const V *>(cur)[q];
        V o;
#pragma unroll
        for (int u = 0; u < VN; u++) SV::set(o, u, SV::get(a, u) - li * SV::get(w, u));
        if (q == j / VN)
#pragma unroll
          for (int u = 0; u < VN; u++)
            if (u == j % VN) SV::set(o, u, -li);
        row[q] = o;
        if (i == j + 1) {  // the next pivot's row
#pragma unroll
          for (int u = 0; u < VN; u++) {
            const int c = q * VN + u;
            if (c <= j) nxt[c] = SV::get(o, u);
            else if (c == i) {
              nxt[c] = T(1);
              pivot(SV::get(o, u), i);
            }
          }
        } else if (q == (j + 1) / VN) {  // and its column
#pragma unroll
          for (int u = 0; u < VN; u++)
            if (u == (j + 1) % VN) nxt[i] = SV::get(o, u);
        }
      }
    }
    __syncthreads();
  }
  for (int j = tid; j < k; j += nt) rs[j] = KeptPivot<T>(inv[j]).inverse_root();
  __syncthreads();
  // 3. E11: rows of Lt^-1 scaled (its unit diagonal and the zeros above it)
  for (int q = tid; q < k * nv; q += nt) {
    const int i = q / nv, c0 = (q % nv) * VN;
    V a = reinterpret_cast<V *>(P + (size_t)i * ldk)[q % nv];
    const T sc = rs[i];
#pragma unroll
    for (int u = 0; u < VN; u++) SV::set(a, u, c0 + u < i ? SV::get(a, u) * sc : c0 + u == i ? sc : T(0));
    reinterpret_cast<V *>(P + (size_t)i * ldk)[q % nv] = a;
  }
  //    L21, LW lanes per row and CL columns per lane (FP64 four lanes: the
  //    pipe of one SM sub-partition would walk a row alone; FP32 two, for more
  //    multiplications per shared-memory read): z = A21 Lt^-T block
  //    by block of 8 columns, then scaled by D^-1/2
  constexpr int LW = sizeof(T) == 8 ? 4 : 2, CL = 8 / LW;
  const int sub = tid % LW, g0 = (tid & 31) / LW * LW;  // lane in the row's group, group's first lane
  for (int i0 = k; i0 < m; i0 += nt / LW) {
    const int i = min(i0 + tid / LW, m - 1);  // (rows past m repeat the last one)
    const bool on = i0 + tid / LW < m;
    T *pr = P + (size_t)i * ldk;
    for (int b0 = 0; b0 < k; b0 += 8) {
      const int c0 = b0 + CL * sub;
      T a[CL];
      const T *l[CL];
#pragma unroll
      for (int h = 0; h < CL; h++) {
        a[h] = c0 + h < k ? pr[c0 + h] : T(0);
        l[h] = L + (size_t)min(c0 + h, k - 1) * ldk;
      }
      for (int q = 0; q < b0; q += VN) {
        const V z = *reinterpret_cast<const V *>(pr + q);
#pragma unroll
        for (int h = 0; h < CL; h++) {
          const V x = *reinterpret_cast<const V *>(l[h] + q);
#pragma unroll
          for (int u = 0; u < VN; u++) a[h] -= SV::get(z, u) * SV::get(x, u);
        }
      }
#pragma unroll
      for (int t = 0; t < 7; t++) {
        T z = a[t % CL];
        if constexpr (LW > 1) z = __shfl_sync(0xffffffffu, z, g0 + t / CL);
        if (b0 + t < k - 1)
#pragma unroll
          for (int h = 0; h < CL; h++)
            if (CL * sub + h > t) a[h] -= z * l[h][b0 + t];
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < CL; h++)
        if (on && c0 + h < k) pr[c0 + h] = a[h];
      __syncwarp();
    }
    if (on)
      for (int c = sub; c < k; c += LW) pr[c] *= rs[c];
    __syncwarp();
  }
  __syncthreads();
  // 4. E -> global (column-major, ld round4(m)); the padding rows stay zero
  {
    const int ld = round4(m);
    T *Eg = E + v.e_off[f];
    for (int c = 0; c < k; c++)
      for (int i = tid; i < k; i += nt) Eg[(int64_t)c * ld + i] = P[(size_t)i * ldk + c];
    for (int i = k + tid / LW; i < m; i += nt / LW) {
      const T *pr = P + (size_t)i * ldk;
      for (int b0 = 0; b0 < k; b0 += 8) {
        const int c0 = b0 + CL * sub;
        T a[CL];
#pragma unroll
        for (int h = 0; h < CL; h++) a[h] = T(0);
        for (int q = b0; q < k; q += VN) {
          const V z = *reinterpret_cast<const V *>(pr + q);
#pragma unroll
          for (int u = 0; u < VN; u++) {
            if (q + u < k) {
              // (a row's vectors past column k: the next row's first, unused)
              const T *e = P + (size_t)(q + u) * ldk + c0;
#pragma unroll
              for (int h = 0; h < CL; h += VN) {
                const V x = *reinterpret_cast<const V *>(e + h);
#pragma unroll
                for (int w = 0; w < VN; w++) a[h + w] -= SV::get(z, u) * SV::get(x, w);
              }
            }
          }
        }
#pragma unroll
        for (int h = 0; h < CL; h++)
          if (c0 + h < k) Eg[(int64_t)(c0 + h) * ld + i] = a[h];
      }
    }
  }
  //    update block: F[k:m, k:m] -= L21 L21^T (lower), 4x4 blocks per thread
  //    over the lower block triangle; L21 rows read VN columns at a time
  const int nb4 = (r + 3) / 4, nblk = nb4 * (nb4 + 1) / 2;
  for (int q = tid; q < nblk; q += nt) {
    // q-th block of the lower triangle, column by column (consecutive threads
    // share a column block and update consecutive rows): t columns from the
    // last one, counted from its end
    const int e = nblk - 1 - q;
    int t = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while (t * (t + 1) / 2 > e) t--;
    while ((t + 1) * (t + 2) / 2 <= e) t++;
    const int bc = nb4 - 1 - t, bi = nb4 - 1 - (e - t * (t + 1) / 2);
    const int i0 = k + 4 * bi, c0 = k + 4 * bc;
    T acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) acc[a][b] = T(0);
    const V *li[4], *lc[4];
#pragma unroll
    for (int a = 0; a < 4; a++) {
      li[a] = reinterpret_cast<const V *>(P + (size_t)min(i0 + a, m - 1) * ldk);
      lc[a] = reinterpret_cast<const V *>(P + (size_t)min(c0 + a, m - 1) * ldk);
    }
    const int qk = (k + VN - 1) / VN;
    for (int qq = 0; qq < qk; qq++) {
      V xi[4], xc[4];
#pragma unroll
      for (int a = 0; a < 4; a++) {
        xi[a] = li[a][qq];
        xc[a] = lc[a][qq];
      }
#pragma unroll
      for (int u = 0; u < VN; u++) {
        if (qq * VN + u < k) {
#pragma unroll
          for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] += SV::get(xi[a], u) * SV::get(xc[b], u);
        }
      }
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const int col = c0 + b;
      if (col >= m) continue;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int row = i0 + a;
        if (row < m && row >= col) F[(int64_t)col * m + row] -= acc[a][b];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// large fronts: assembly by column chunks, then for every panel step one
// launch that factors the panels and one that applies the trailing update
// tile by tile, so that one front occupies many SMs.
// ---------------------------------------------------------------------------
constexpr int kAsmCols = 64;

__device__ __forceinline__ int64_t lower_bound64(const int64_t *a, int64_t lo, int64_t hi, int64_t key) {
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ int lower_bound32(const int *a, int lo, int hi, int key) {
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Right-looking Cholesky of the lower triangle of D[0..jb)[0..jb) by one
// warp: lane i keeps row i in registers, column j of L is broadcast by
// shuffles.  Per element the same operations in the same order as the
// column-by-column algorithm (scale by the pivot's square root, then
// D[i][c] -= D[i][j] D[c][j] for j = 0, 1, ...).
template <typename T>
__device__ __forceinline__ void chol_warp(T (*D)[kNB + 1], int jb, int *status) {
  const int lane = threadIdx.x & 31;
  T a[kNB];
#pragma unroll
  for (int c = 0; c < kNB; c++) a[c] = D[lane][c];
#pragma unroll
  for (int j = 0; j < kNB; j++) {
    if (j < jb) {
      T d = __shfl_sync(0xffffffffu, a[j], j);
      if (!(d > T(0))) {
        if (lane == 0) atomicOr(status, ERR_NOT_SPD);
        d = T(1);
      }
      const T p = tsqrt<T>(d);
      if (lane == j) a[j] = p;
      else if (lane > j) a[j] /= p;
      const T lij = a[j];
#pragma unroll
      for (int c = j + 1; c < kNB; c++) {
        const T lcj = __shfl_sync(0xffffffffu, lij, c);
        if (c < jb && lane >= c) a[c] -= lij * lcj;
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kNB; c++) D[lane][c] = a[c];
}

// The Cholesky factor by a whole CTA in shared memory as L D L^T with the
// columns scaled at the end, one barrier and one division per pivot: for
// FP64, whose square roots and divisions are too slow for one warp's chain
// on the FP64 pipe.  NAMED: the first kMfThreads threads of a larger CTA.
template <bool NAMED>
__device__ __forceinline__ void diag_sync() {
  if constexpr (NAMED) asm volatile("bar.sync 1, %0;" ::"n"(kMfThreads) : "memory");
  else __syncthreads();
}
template <typename T, bool NAMED = false>
__device__ __forceinline__ void chol_cta(T (*D)[kNB + 1], int jb, int *status) {
  __shared__ T inv[kNB];
  const int tid = threadIdx.x;
  auto pivot = [&](T d, int j) {
    if (!(d > T(0))) {
      atomicOr(status, ERR_NOT_SPD);
      d = T(1);
    }
    D[j][j] = d;
    inv[j] = KeptPivot<T>::keep(d);
  };
  if (tid == 0) pivot(D[0][0], 0);
  diag_sync<NAMED>();
  constexpr int TX = kMfThreads / kNB;  // threads per row
  const int i = tid / TX, tx = tid % TX;
  for (int j = 0; j < jb - 1; j++) {
    if (i > j && i < jb) {
      const T li = KeptPivot<T>(inv[j]).divide(D[i][j]);
      for (int c = j + 1 + tx; c <= i; c += TX) {
        const T x = D[i][c] - li * D[c][j];
        if (c == i && i == j + 1) pivot(x, i);
        else D[i][c] = x;
      }
    }
    diag_sync<NAMED>();
  }
  for (int q = tid; q < jb * jb; q += kMfThreads) {
    const int c = q / jb, k = q % jb;
    if (k > c) D[k][c] *= KeptPivot<T>(inv[c]).inverse_root();
  }
  diag_sync<NAMED>();
  if (tid < jb) D[tid][tid] = tsqrt<T>(D[tid][tid]);
}

// FP32: one warp per front (chol_warp); FP64: kMfThreads per front (chol_cta)
template <typename T> __host__ __device__ constexpr int diag_threads() { return sizeof(T) == 4 ? 32 : kMfThreads; }

// Factor the jb x jb diagonal block at column j0 of a front in place (F: the
// front's arena block, ld m): its lower part into shared memory, FP32 by one
// warp in registers, FP64 by the whole CTA; every thread of the CTA calls it,
// after a barrier that makes the block's final values visible.
template <typename T, bool NAMED = false>
__device__ __forceinline__ void factor_diag_block(T *__restrict__ F, int m, int j0, int jb, int *status) {
  __shared__ T D[kNB][kNB + 1];
  const int tid = threadIdx.x, nt = NAMED ? kMfThreads : blockDim.x;
  for (int q = tid; q < kNB * kNB; q += nt) {  // lower part, zeros elsewhere
    const int c = q / kNB, i = q % kNB;  // column-major walk: coalesced over rows
    D[i][c] = (i >= c && i < jb) ? F[(int64_t)(j0 + c) * m + j0 + i] : T(0);
  }
  diag_sync<NAMED>();
  if constexpr (sizeof(T) == 4) {
    if (tid < 32) chol_warp<T>(D, jb, status);
  } else {
    chol_cta<T, NAMED>(D, jb, status);
  }
  diag_sync<NAMED>();
  for (int q = tid; q < jb * jb; q += nt) {
    const int c = q / jb, i = q % jb;
    if (i >= c) F[(int64_t)(j0 + c) * m + j0 + i] = D[i][c];
  }
}

// The diagonal block of a panel step in a launch of its own: only where no
// earlier kernel of the chain finishes the block (the first step of an FP32
// super-panel after the mma.sync trailing update, tensor_update 0)
template <typename T>
__global__ void __launch_bounds__(diag_threads<T>())
mf_diag(MfView v, const int *__restrict__ fronts, int j0, T *__restrict__ arena, int *__restrict__ status) {
  const int f = fronts[blockIdx.x];
  const int m = v.f_m[f], k = v.f_k[f];
  factor_diag_block<T>(arena + v.f_off[f], m, j0, min(kNB, k - j0), status);
}

// task = {front, first column of the chunk}.  The CTA of chunk 0 then
// factors the front's first diagonal block (the first panel step's).
template <typename T>
__global__ void __launch_bounds__(kMfThreads)
mf_assemble_large(MfView v, const int2 *__restrict__ tasks, const double *__restrict__ vals,
                  T *__restrict__ arena, int *__restrict__ status) {
  const int f = tasks[blockIdx.x].x, c0 = tasks[blockIdx.x].y;
  const int m = v.f_m[f];
  const int c1 = min(c0 + kAsmCols, m);
  const int64_t off = v.f_off[f];
  T *F = arena + off;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = kMfThreads / 32;
  for (int c = c0 + wid; c < c1; c += nw)
    for (int i = c + lane; i < m; i += 32) F[(int64_t)c * m + i] = T(0);
  __syncthreads();
  const int64_t lo = lower_bound64(v.asm_tgt, v.f_asm[f], v.f_asm[f + 1], off + (int64_t)c0 * m);
  const int64_t hi = lower_bound64(v.asm_tgt, lo, v.f_asm[f + 1], off + (int64_t)c1 * m);
  for (int64_t e = lo + tid; e < hi; e += kMfThreads) {
    double s = 0.0;
    for (int64_t q = v.asm_sp[e]; q < v.asm_sp[e + 1]; q++) s += vals[v.asm_src[q]];
    arena[v.asm_tgt[e]] = (T)s;
  }
  __syncthreads();
  for (int ci = v.f_child_ptr[f]; ci < v.f_child_ptr[f + 1]; ci++) {
    const int c = v.f_children[ci];
    const int mc = v.f_m[c], kc = v.f_k[c], rc = mc - kc;
    const T *U = arena + v.f_off[c] + (int64_t)kc * mc + kc;
    const int *rel = v.relmap + v.f_relmap[c];
    const int blo = lower_bound32(rel, 0, rc, c0), bhi = lower_bound32(rel, blo, rc, c1);
    for (int b = blo + wid; b < bhi; b += nw)
      extend_add_column<T>(F + (int64_t)rel[b] * m, rel, U + (int64_t)b * mc, b, rc, lane);
    __syncthreads();
  }
  if (c0 == 0) factor_diag_block<T>(F, m, 0, min(kNB, v.f_k[f]), status);
}

// Panel at column j0 of a large front: its diagonal block was factored by
// the kernel that finished it (factor_diag_block: the assembly, the previous
// step's update tile (0, 0) or the super-panel's trailing-update tile (0, 0));
// mf_panel solves L21 = A21 L11^-T for row chunks of kPanelRows rows (task =
// {front, first row of the chunk}), many CTAs per front, or forms E rows of
// the panel (escale tasks, below).
constexpr int kPanelRows = 256;

// E rows of the panel (escale task = {front, first column}): E_J <- L_JJ^-1 E_J
// on kEscCols columns of [0, j0 + jb); the columns of block J start as the
// identity, so block J of E becomes L_JJ^-1
template <typename T> struct EscCols { static constexpr int N = 1024 / sizeof(T); };

template <typename T>
__global__ void __launch_bounds__(kMfThreads)
mf_panel(MfView v, const int2 *__restrict__ tasks, int npanel, const int2 *__restrict__ esc, int j0,
         T *__restrict__ arena, T *__restrict__ E) {
  __shared__ T D[kNB][kNB + 1];
  const bool escale = (int)blockIdx.x >= npanel;
  const int2 task = escale ? esc[blockIdx.x - npanel] : tasks[blockIdx.x];
  const int f = task.x;
  const int m = v.f_m[f], k = v.f_k[f];
  const int jb = min(kNB, k - j0);
  T *F = arena + v.f_off[f];
  const int tid = threadIdx.x;
  for (int q = tid; q < jb * jb; q += kMfThreads) {  // the factored diagonal block
    int c = q / jb, i = q % jb;
    D[i][c] = i >= c ? F[(int64_t)(j0 + c) * m + j0 + i] : T(0);
  }
  __shared__ T rd[kNB];  // FP64: reciprocals of its diagonal, no division per row
  if (sizeof(T) == 8 && tid < jb) rd[tid] = pivot_inverse(F[(int64_t)(j0 + tid) * m + j0 + tid]);
  if (escale) {
    constexpr int NC = EscCols<T>::N;
    __shared__ T Eb[NC][kNB + 1];
    const int ld = round4(m);
    T *Eg = E + v.e_off[f];
    const int c0 = task.y, nc = min(NC, j0 + jb - c0);
    for (int q = tid; q < nc * kNB; q += kMfThreads) {
      const int cc = q / kNB, t = q % kNB, c = c0 + cc;
      T e = T(0);
      if (t < jb) e = c < j0 ? Eg[(int64_t)c * ld + j0 + t] : (c - j0 == t ? T(1) : T(0));
      Eb[cc][t] = e;
    }
    __syncthreads();
    for (int cc = tid; cc < nc; cc += kMfThreads) {
      for (int t = 0; t < jb; t++) {
        T s = Eb[cc][t];
        for (int q = 0; q < t; q++) s -= D[t][q] * Eb[cc][q];
        Eb[cc][t] = sizeof(T) == 8 ? s * rd[t] : s / D[t][t];
      }
    }
    __syncthreads();
    for (int q = tid; q < nc * kNB; q += kMfThreads) {
      const int cc = q / kNB, t = q % kNB;
      if (t < jb) Eg[(int64_t)(c0 + cc) * ld + j0 + t] = Eb[cc][t];
    }
    return;
  }
  __syncthreads();
  const int r0 = task.y;
  const int rb = max(r0, j0 + jb), re = min(r0 + kPanelRows, m);
  // one row per thread (no row loop: the diagonal block is read inside the
  // solve instead of being held in registers across rows)
  static_assert(kPanelRows == kMfThreads, "a row chunk has one row per thread");
  const int i = rb + tid;
  if (i < re) {
    T x[kNB];
#pragma unroll
    for (int t = 0; t < kNB; t++) x[t] = t < jb ? F[(int64_t)(j0 + t) * m + i] : T(0);
#pragma unroll
    for (int t = 0; t < kNB; t++) {
      if (t < jb) {
        T s = x[t];
#pragma unroll
        for (int q = 0; q < t; q++) s -= x[q] * D[t][q];
        x[t] = sizeof(T) == 8 ? s * rd[t] : s / D[t][t];
      }
    }
#pragma unroll
    for (int t = 0; t < kNB; t++)
      if (t < jb) F[(int64_t)(j0 + t) * m + i] = x[t];
  }
}

// The same for levels with few rows: four lanes per row (of L21, or column of
// E), eight columns each, kThinRows rows per CTA.  One thread per row walks
// 528 multiply-adds on its own, and a warp's FP64 multiply-add takes its
// sub-partition 64 clocks: 18 us at least, 35 us for the eight warps of a
// 256-row CTA, however few CTAs there are; this way 16 us (33 rows), with the
// columns in the order as above.
constexpr int kThinRows = 32, kThinLanes = 4;

template <typename T>
__global__ void __launch_bounds__(kThinRows * kThinLanes)
mf_panel_thin(MfView v, const int2 *__restrict__ tasks, int npanel, const int2 *__restrict__ esc, int j0,
              T *__restrict__ arena, T *__restrict__ E) {
  constexpr int LW = kThinLanes, NC = kNB / LW, NT = kThinRows * LW;
  __shared__ T D[kNB][kNB + 1], rd[kNB];
  const bool escale = (int)blockIdx.x >= npanel;
  const int2 task = escale ? esc[blockIdx.x - npanel] : tasks[blockIdx.x];
  const int f = task.x, m = v.f_m[f], k = v.f_k[f], jb = min(kNB, k - j0);
  T *F = arena + v.f_off[f];
  const int tid = threadIdx.x, lane = tid & 31;
  // eight rows per warp, a row's lanes eight apart: consecutive lanes read consecutive rows
  const int g = lane & 7, l = lane >> 3, i = task.y + (tid >> 5) * 8 + g;
  const bool on = escale ? i < j0 + jb : i < m;
  // entry t of the row at p[t * st]
  T *p = escale ? E + v.e_off[f] + (int64_t)i * round4(m) + j0 : F + (int64_t)j0 * m + i;
  const int64_t st = escale ? 1 : m;
  T x[NC];  // entries LW * q + l
#pragma unroll
  for (int q = 0; q < NC; q++) {
    const int t = LW * q + l;
    x[q] = T(0);
    if (on && t < jb) x[q] = escale && i >= j0 ? (i - j0 == t ? T(1) : T(0)) : p[t * st];
  }
  for (int q = tid; q < kNB * kNB; q += NT) {
    const int c = q / kNB, r = q % kNB;
    D[r][c] = r >= c && r < jb ? F[(int64_t)(j0 + c) * m + j0 + r] : T(0);
  }
  __syncthreads();
  if (tid < jb) rd[tid] = sizeof(T) == 8 ? pivot_inverse(D[tid][tid]) : D[tid][tid];
  __syncthreads();
#pragma unroll
  for (int t = 0; t < kNB; t++) {
    if (t >= jb) break;
    const T own = sizeof(T) == 8 ? x[t / LW] * rd[t] : x[t / LW] / rd[t];
    const T xt = __shfl_sync(0xffffffffu, own, t % LW * 8 + g);
    if (l == t % LW) x[t / LW] = xt;
#pragma unroll
    for (int q = t / LW; q < NC; q++)
      if (LW * q + l > t) x[q] -= xt * D[LW * q + l][t];
  }
#pragma unroll
  for (int q = 0; q < NC; q++)
    if (on && LW * q + l < jb) p[(LW * q + l) * st] = x[q];
}

// One tile (UpdTile) of an update with the L columns [jl, jl + K), K = min(kw, k - jl).
// Trailing-update tiles (task = {front, (ti << 16) | tj}, ti >= tj) cover rows
// and columns from c0 = jl + K: C -= L[rows, J] L[cols, J]^T (lower part),
// only columns below cend = min(cend_base, k) when cend_base > 0 (the update
// inside a 128-column super-panel), all columns otherwise (the trailing update
// of the whole super-panel, K up to 128, staged 32 columns at a time).  For
// blockIdx.x >= nupd the tile belongs to the E update
// E[c0:m, 0:c0] -= L[c0:m, J] E_J (task = {front, (ti << 16) | tc}, columns
// from 0; J = [jl, c0)); the columns of block J are assigned, the earlier
// ones accumulated.  A panel step (cend_base > 0) updates the E rows below
// cend only, the rest of its super-panel; the super-panel's own launch
// (cend_base 0, J = the super-panel) updates the rows below it.
template <typename T>
__global__ void __launch_bounds__(kMfThreads)
mf_update(MfView v, const int2 *__restrict__ tasks, int nupd, const int2 *__restrict__ etasks, int jl, int kw,
          int cend_base, T *__restrict__ arena, T *__restrict__ E, int *__restrict__ status) {
  constexpr int kTile = UpdTile<T>::N, R = kTile / 16;
  __shared__ T As[kNB][kTile];
  __shared__ T Bs[kNB][kTile + 1];
  const bool etile = (int)blockIdx.x >= nupd;
  const int2 task = etile ? etasks[blockIdx.x - nupd] : tasks[blockIdx.x];
  const int f = task.x;
  const int ti = task.y >> 16, tj = task.y & 0xffff;
  const int m = v.f_m[f], k = v.f_k[f];
  const int K = min(kw, k - jl);
  T *F = arena + v.f_off[f];
  const int c0 = jl + K;
  const int r0 = c0 + ti * kTile;
  const int cc0 = etile ? tj * kTile : c0 + tj * kTile;
  const bool diag = !etile && ti == tj;
  const int cend = cend_base > 0 ? min(cend_base, k) : m;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int ld = round4(m);
  T *Eg = E + v.e_off[f];
  T acc[R][R];
#pragma unroll
  for (int a = 0; a < R; a++)
#pragma unroll
    for (int b = 0; b < R; b++) acc[a][b] = T(0);
  for (int t0 = 0; t0 < K; t0 += kNB) {
    const int tb = min(kNB, K - t0);
    if (t0 > 0) __syncthreads();  // the previous chunk is consumed
    for (int q = tid; q < kNB * kTile; q += kMfThreads) {
      int t = q / kTile, r = q % kTile;
      As[t][r] = (t < tb && r0 + r < m) ? F[(int64_t)(jl + t0 + t) * m + r0 + r] : T(0);
    }
    if (etile) {
      for (int q = tid; q < kNB * kTile; q += kMfThreads) {
        const int r = q / kNB, t = q % kNB;
        Bs[t][r] = (t < tb && cc0 + r < c0) ? Eg[(int64_t)(cc0 + r) * ld + jl + t0 + t] : T(0);
      }
    } else {
      for (int q = tid; q < kNB * kTile; q += kMfThreads) {
        int t = q / kTile, r = q % kTile;
        Bs[t][r] = (t < tb && cc0 + r < cend) ? F[(int64_t)(jl + t0 + t) * m + cc0 + r] : T(0);
      }
    }
    __syncthreads();
    for (int t = 0; t < tb; t++) {
      T ra[R], rb[R];
#pragma unroll
      for (int a = 0; a < R; a++) ra[a] = As[t][tx + 16 * a];
#pragma unroll
      for (int b = 0; b < R; b++) rb[b] = Bs[t][ty + 16 * b];
      // (16-row blocks above the diagonal of a diagonal tile are not stored)
#pragma unroll
      for (int a = 0; a < R; a++)
#pragma unroll
        for (int b = 0; b < R; b++)
          if (a >= b || !diag) acc[a][b] += ra[a] * rb[b];
    }
  }
  const int j0 = jl;
  if (etile) {
    const int rend = cend_base > 0 ? cend : m;
#pragma unroll
    for (int b = 0; b < R; b++) {
      const int col = cc0 + ty + 16 * b;
      if (col >= c0) continue;
#pragma unroll
      for (int a = 0; a < R; a++) {
        const int row = r0 + tx + 16 * a;
        if (row >= rend) continue;
        T *dst = Eg + (int64_t)col * ld + row;
        *dst = col >= j0 ? -acc[a][b] : *dst - acc[a][b];
      }
    }
    return;
  }
#pragma unroll
  for (int b = 0; b < R; b++) {
    const int col = cc0 + ty + 16 * b;
    if (col >= cend) continue;
#pragma unroll
    for (int a = 0; a < R; a++) {
      const int row = r0 + tx + 16 * a;
      if (row < m && row >= col) F[(int64_t)col * m + row] -= acc[a][b];
    }
  }
  // tile (0, 0) holds the next panel step's diagonal block (columns c0 ..,
  // inside the super-panel for a panel step): this was its last update
  if (ti == 0 && tj == 0 && c0 < (cend_base > 0 ? min(cend_base, k) : k)) {
    __syncthreads();
    factor_diag_block<T>(F, m, c0, min(kNB, k - c0), status);
  }
}

// Trailing update of a super-panel with 128 x 128 tiles (FP32): C -= L_rows L_cols^T
// for the L columns [jl, jl + K), K = min(kw, k - jl), rows and columns from
// c0 = jl + K (task = {front, (ti << 16) | tj}, ti >= tj, 128-row units).
constexpr int kBT = 128, kBK = 8;

// It runs on the tensor cores (C -= L_I L_J^T, 128 x 128 per CTA, K walked
// in chunks of 8 columns, double-buffered in shared memory with the next
// chunk's global loads issued before the current chunk is consumed), each product as three TF32 products (split 3xTF32:
// a = a_hi + a_lo with a_hi, a_lo TF32; a b ~ a_lo b_hi + a_hi b_lo + a_hi b_hi,
// FP32 accumulation), which keeps the FP32 accuracy of the factorisation.
// 8 warps, warp w owns rows 64*(w%2) .. +63 and columns 32*(w/2) .. +31 of the
// tile: 4 x 4 mma.m16n8k8 tiles.  Operands are split when they are staged.
__device__ __forceinline__ uint32_t tf32_of(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int kTcPad = kBT + 8;  // row stride of the staged operands (conflict-free fragment loads)

__global__ void __launch_bounds__(256, 2)
mf_update_big_tf32(MfView v, const int2 *__restrict__ tasks, int jl, int kw, float *__restrict__ arena) {
  __shared__ __align__(16) uint32_t Ah[2][kBK][kTcPad], Al[2][kBK][kTcPad];
  __shared__ __align__(16) uint32_t Bh[2][kBK][kTcPad], Bl[2][kBK][kTcPad];
  const int f = tasks[blockIdx.x].x;
  const int ti = tasks[blockIdx.x].y >> 16, tj = tasks[blockIdx.x].y & 0xffff;
  const int m = v.f_m[f], k = v.f_k[f];
  const int K = min(kw, k - jl);
  const int c0 = jl + K, r0 = c0 + ti * kBT, cc0 = c0 + tj * kBT;
  float *F = arena + v.f_off[f];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lt = tid >> 5, lr = (tid & 31) * 4;  // chunk column and first of 4 rows this thread stages
  const int wm = (warp & 1) * 64, wn = (warp >> 1) * 32;
  const int gid = lane >> 2, tig = lane & 3;
  float pa[4], pb[4];
  auto fetch = [&](int kc) {
    const int t = kc + lt;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int ra = r0 + lr + u, rb = cc0 + lr + u;
      pa[u] = (t < K && ra < m) ? F[(int64_t)(jl + t) * m + ra] : 0.f;
      pb[u] = (t < K && rb < m) ? F[(int64_t)(jl + t) * m + rb] : 0.f;
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t ah = tf32_of(pa[u]), bh = tf32_of(pb[u]);
      Ah[buf][lt][lr + u] = ah;
      Al[buf][lt][lr + u] = tf32_of(pa[u] - __uint_as_float(ah));
      Bh[buf][lt][lr + u] = bh;
      Bl[buf][lt][lr + u] = tf32_of(pb[u] - __uint_as_float(bh));
    }
  };
  float acc[4][4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[a][b][q] = 0.f;
  fetch(0);
  stash(0);
  __syncthreads();
  int buf = 0;
  for (int kc = 0; kc < K; kc += kBK) {
    const bool more = kc + kBK < K;
    if (more) fetch(kc + kBK);
    // B fragments (hi and lo) of the warp's 4 column tiles
    uint32_t bh[4][2], bl[4][2];
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int col = wn + nt * 8 + gid;
      bh[nt][0] = Bh[buf][tig][col];
      bh[nt][1] = Bh[buf][tig + 4][col];
      bl[nt][0] = Bl[buf][tig][col];
      bl[nt][1] = Bl[buf][tig + 4][col];
    }
#pragma unroll
    for (int mt = 0; mt < 4; mt++) {
      const int row = wm + mt * 16 + gid;
      const uint32_t ah[4] = {Ah[buf][tig][row], Ah[buf][tig][row + 8], Ah[buf][tig + 4][row],
                              Ah[buf][tig + 4][row + 8]};
      const uint32_t al[4] = {Al[buf][tig][row], Al[buf][tig][row + 8], Al[buf][tig + 4][row],
                              Al[buf][tig + 4][row + 8]};
#pragma unroll
      for (int nt = 0; nt < 4; nt++) {  // small terms first
        mma_tf32(acc[mt][nt], al, bh[nt]);
        mma_tf32(acc[mt][nt], ah, bl[nt]);
        mma_tf32(acc[mt][nt], ah, bh[nt]);
      }
    }
    if (more) stash(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int mt = 0; mt < 4; mt++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int row = r0 + wm + mt * 16 + gid + (q >= 2 ? 8 : 0);
        const int col = cc0 + wn + nt * 8 + tig * 2 + (q & 1);
        if (row < m && col < m && row >= col) F[(int64_t)col * m + row] -= acc[mt][nt][q];
      }
}

// The same update on the fifth-generation tensor cores: tcgen05.mma
// kind::tf32 with the 128 x 128 FP32 accumulator in tensor memory.  The CTA
// (8 warps) stages K in chunks of 32 columns: every thread loads rows of the
// two column blocks of L (coalesced along the column), splits them into
// TF32 hi and lo parts and writes them into four 16 KB shared-memory tiles
// in the 128-byte-swizzled K-major layout (dg_tc.cuh); one thread issues the
// 3 x 4 MMAs of the chunk (lo*hi, hi*lo, hi*hi per K step of 8) and commits
// them to an mbarrier that all threads wait on (bounded: on a timeout the
// CTA sets ERR_WAIT, waits once more and frees its tensor memory) before
// the tiles are refilled.  The epilogue reads the accumulator back with
// tcgen05.ld (warp w: lanes 32 (w % 4) .., columns 64 (w / 4) ..) and
// subtracts it from the lower part of the front.  A diagonal tile (ti == tj)
// stages one block and uses it as both operands.
constexpr int kTcChunk = 32;
constexpr size_t kTcTileBytes = 128 * kTcChunk * sizeof(float);  // 16 KB
constexpr size_t kTcSmem = 4 * kTcTileBytes + 1024;                // + alignment to 1024 bytes
constexpr long long kTcWaitPolls = 1LL << 24;

__global__ void __launch_bounds__(256, 3)
mf_update_big_tc(MfView v, const int2 *__restrict__ tasks, int nupd, const int2 *__restrict__ etasks, int jl,
                 int kw, float *__restrict__ arena, float *__restrict__ E, int *__restrict__ status,
                 int fuse_diag) {
  extern __shared__ unsigned char tc_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) &
                                                          ~static_cast<uintptr_t>(1023));
  unsigned char *Ahi = base, *Alo = base + kTcTileBytes, *Bhi = base + 2 * kTcTileBytes,
                *Blo = base + 3 * kTcTileBytes;
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  const bool etile = (int)blockIdx.x >= nupd;
  const int2 task = etile ? etasks[blockIdx.x - nupd] : tasks[blockIdx.x];
  const int f = task.x;
  const int ti = task.y >> 16, tj = task.y & 0xffff;
  const int m = v.f_m[f], k = v.f_k[f];
  const int K = min(kw, k - jl);
  const int c0 = jl + K, r0 = c0 + ti * kBT, cc0 = etile ? tj * kBT : c0 + tj * kBT;
  const bool diag = !etile && ti == tj;
  float *F = arena + v.f_off[f];
  const int ld = round4(m);
  float *Eg = E + v.e_off[f];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 128);
  if (tid == 0) tc::mbar_init(&bar, 1);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  constexpr uint32_t idesc = tc::idesc_tf32(128, 128);
  // this thread stages rows (tid & 127) and columns kk = (tid >> 7) + 2 q of
  // every chunk: 16 values of each operand, loaded together
  constexpr int NQ = 128 * kTcChunk / 256;
  const int r = tid & 127, kk0 = tid >> 7;
  const int ra = r0 + r, rb = cc0 + r;
  // E tiles: B row rr is E column cc0 + rr, 16 consecutive K values of it
  // (E rows jl + kc + te ..), read as four 16-byte vectors
  const int rr = tid >> 1, te = (tid & 1) * 16;
  const bool eok = etile && cc0 + rr < c0;
  float pa[NQ], pb[NQ];
  auto fetch = [&](int kc) {
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const int t = kc + kk0 + 2 * q;
      pa[q] = (t < K && ra < m) ? F[(int64_t)(jl + t) * m + ra] : 0.f;
      if (!etile) pb[q] = (!diag && t < K && rb < m) ? F[(int64_t)(jl + t) * m + rb] : 0.f;
    }
    if (etile) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int t = kc + te + 4 * u;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (eok && t < K) x = *reinterpret_cast<const float4 *>(Eg + (int64_t)(cc0 + rr) * ld + jl + t);
        pb[4 * u] = x.x;
        pb[4 * u + 1] = t + 1 < K ? x.y : 0.f;
        pb[4 * u + 2] = t + 2 < K ? x.z : 0.f;
        pb[4 * u + 3] = t + 3 < K ? x.w : 0.f;
      }
    }
  };
  auto stash = [&]() {
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const uint32_t off = tc::sw128_offset(r, kk0 + 2 * q);
      const uint32_t ah = tf32_of(pa[q]);
      *reinterpret_cast<uint32_t *>(Ahi + off) = ah;
      *reinterpret_cast<uint32_t *>(Alo + off) = tf32_of(pa[q] - __uint_as_float(ah));
      if (!diag && !etile) {
        const uint32_t bh = tf32_of(pb[q]);
        *reinterpret_cast<uint32_t *>(Bhi + off) = bh;
        *reinterpret_cast<uint32_t *>(Blo + off) = tf32_of(pb[q] - __uint_as_float(bh));
      }
    }
    if (etile) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t off = tc::sw128_offset(rr, te + 4 * u);  // 4 values in one 16-byte chunk
        uint4 h, l;
        h.x = tf32_of(pb[4 * u]);     l.x = tf32_of(pb[4 * u] - __uint_as_float(h.x));
        h.y = tf32_of(pb[4 * u + 1]); l.y = tf32_of(pb[4 * u + 1] - __uint_as_float(h.y));
        h.z = tf32_of(pb[4 * u + 2]); l.z = tf32_of(pb[4 * u + 2] - __uint_as_float(h.z));
        h.w = tf32_of(pb[4 * u + 3]); l.w = tf32_of(pb[4 * u + 3] - __uint_as_float(h.w));
        *reinterpret_cast<uint4 *>(Bhi + off) = h;
        *reinterpret_cast<uint4 *>(Blo + off) = l;
      }
    }
  };
  uint32_t parity = 0;
  bool bad = false;
  fetch(0);
  for (int kc = 0; kc < K; kc += kTcChunk) {
    stash();
    tc::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
      const uint64_t dAh = tc::sw128_desc(tc::smem_u32(Ahi)), dAl = tc::sw128_desc(tc::smem_u32(Alo));
      const uint64_t dBh = diag ? dAh : tc::sw128_desc(tc::smem_u32(Bhi));
      const uint64_t dBl = diag ? dAl : tc::sw128_desc(tc::smem_u32(Blo));
#pragma unroll
      for (int ks = 0; ks < kTcChunk / 8; ks++) {  // 8 TF32 values (32 bytes) per MMA
        const uint64_t o = (uint64_t)((ks * 32) >> 4);
        tc::mma_tf32(tmem, dAl + o, dBh + o, idesc, (kc > 0 || ks > 0) ? 1u : 0u);
        tc::mma_tf32(tmem, dAh + o, dBl + o, idesc, 1u);
        tc::mma_tf32(tmem, dAh + o, dBh + o, idesc, 1u);
      }
      tc::mma_commit(tc::smem_u32(&bar));
    }
    // the next chunk's loads are in flight while the tensor cores work
    if (kc + kTcChunk < K) fetch(kc + kTcChunk);
    const bool ok = tc::mbar_wait(&bar, parity, kTcWaitPolls);
    parity ^= 1;
    if (__syncthreads_or(!ok)) { bad = true; break; }
  }
  if (bad) {
    if (tid == 0) atomicOr(status, ERR_WAIT);
    tc::mbar_wait(&bar, parity ^ 1, kTcWaitPolls);  // its MMAs in flight, once more (bounded)
  } else {
    tc::fence_after_sync();
    const int lg = warp & 3, ch = warp >> 2;
    const int row = r0 + 32 * lg + lane;
#pragma unroll 1
    for (int h = 0; h < 4; h++) {
      float d[16];
      tc::tmem_load16(tmem + ((uint32_t)(32 * lg) << 16) + (uint32_t)(ch * 64 + 16 * h), d);
      if (etile) {
        // E[row, col] for col < c0: the super-panel's own columns (>= jl)
        // are assigned, the earlier ones accumulated
        if (row < m) {
          const int colb = cc0 + ch * 64 + 16 * h;
          float cur[16];
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const int col = colb + c;
            cur[c] = (col < jl) ? Eg[(int64_t)col * ld + row] : 0.f;
          }
#pragma unroll
          for (int c = 0; c < 16; c++) {
            const int col = colb + c;
            if (col < c0) Eg[(int64_t)col * ld + row] = cur[c] - d[c];
          }
        }
      } else if (row < m) {
        const int colb = cc0 + ch * 64 + 16 * h;
        float cur[16];
#pragma unroll
        for (int c = 0; c < 16; c++) {
          const int col = colb + c;
          cur[c] = (col < m && row >= col) ? F[(int64_t)col * m + row] : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 16; c++) {
          const int col = colb + c;
          if (col < m && row >= col) F[(int64_t)col * m + row] = cur[c] - d[c];
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, 128);
  // trailing-update tile (0, 0) holds the next super-panel's first diagonal
  // block: this was its last update
  if (fuse_diag && !bad && !etile && ti == 0 && tj == 0 && c0 < k)
    factor_diag_block<float>(F, m, c0, min(kNB, k - c0), status);
}

}  // namespace dg
#include "dg_split.cuh"  // FP64 super-panel updates on the tensor cores
namespace dg {

// ---------------------------------------------------------------------------
// multifrontal solves with the elimination matrices E
//
// Forward, one level:  the front's right-hand side is b = [xl(pivots) ; 0]
// plus the children's update vectors (extend-add, children in order); then
//     y = E[0:k, :] b1   -> yl (pivots)      u = b2 + E[k:m, :] b1 -> uvec.
// Backward, one level: v = [yl(pivots) ; xl(ancestor rows)], x1 = E^T v -> xl.
// The forward writes y to a second local vector so that the CTAs of one front
// never overwrite the right-hand side another CTA still reads.
//
// E is read with 16-byte vector loads: ld = round4(m) and every E block starts
// on a multiple of 4 elements, and the padding rows m..ld-1 are zero.
// ---------------------------------------------------------------------------
template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int N = 4;
  __device__ static __forceinline__ void load(const float *p, float *o) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  }
  __device__ static __forceinline__ void lds(const float *p, float *o) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  }
};
template <> struct Vec16<double> {
  static constexpr int N = 2;
  __device__ static __forceinline__ void load(const double *p, double *o) {
    const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
    o[0] = t.x; o[1] = t.y;
  }
  __device__ static __forceinline__ void lds(const double *p, double *o) {
    const double2 t = *reinterpret_cast<const double2 *>(p);
    o[0] = t.x; o[1] = t.y;
  }
};

constexpr int kSolveSmall = 128;   // fronts of at most this many rows: one warp each

// Small fronts are solved by groups of G lanes (G = 8, 16 or 32; 32 / G
// fronts per warp): a front of at most 4G rows, lane l of its group holding
// the rows VN*l + G*VN*p.  Levels put their small fronts into three buckets
// by size so that tiny fronts do not leave most of a warp idle.
constexpr int kSmallUnroll = 4;   // E columns per load batch of a small-front group
template <typename T> struct SmallMinBlocks { static constexpr int N = sizeof(T) == 8 ? 3 : 6; };

template <int G>
__device__ __forceinline__ unsigned group_mask(int lane) {
  return G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane / G * G));
}

// E loads of one batch of kSmallUnroll columns [j0, j0 + kSmallUnroll) for the rows
// of one group lane; vectors wholly above the diagonal (r + VN <= j) are zero
template <typename T, int PASS, int G>
__device__ __forceinline__ void load_e_batch(const T *Ef, int ld, int m, int k, int sl, int j0,
                                             T (&e)[PASS][kSmallUnroll][Vec16<T>::N]) {
  constexpr int VN = Vec16<T>::N;
#pragma unroll
  for (int p = 0; p < PASS; p++) {
    const int r = VN * sl + G * VN * p;
#pragma unroll
    for (int u = 0; u < kSmallUnroll; u++) {
      const int j = j0 + u;
      if (r < m && j < k && r + VN > j) Vec16<T>::load(Ef + (int64_t)j * ld + r, e[p][u]);
      else {
#pragma unroll
        for (int q = 0; q < VN; q++) e[p][u][q] = T(0);
      }
    }
  }
}

// x + the first two children's updates at a row (t: the row's child table
// entry), children in order
template <typename T>
__device__ __forceinline__ T add_children(T x, unsigned t, const T *__restrict__ u, int64_t cu0, int64_t cu1) {
  const unsigned t0 = t & 0xffffu, t1 = t >> 16;
  const T a = t0 != kNoChild ? __ldcg(u + cu0 + t0) : T(0);
  const T b = t1 != kNoChild ? __ldcg(u + cu1 + t1) : T(0);
  if (t0 != kNoChild) x += a;
  if (t1 != kNoChild) x += b;
  return x;
}

// and the children from the pair cp on (w: the row's table entry of pair 0)
template <typename T>
__device__ __forceinline__ T add_more_children(T x, const MfView &v, int64_t w, int m, int nch, int ch, int cp,
                                               const T *__restrict__ u) {
  for (; 2 * cp < nch; cp++)
    x = add_children(x, v.ctab[w + (int64_t)cp * m], u, v.ch_edge[ch + 2 * cp].uoff,
                     2 * cp + 1 < nch ? v.ch_edge[ch + 2 * cp + 1].uoff : 0);
  return x;
}

// and the listed updates of a row (row: tab + its place in the front)
template <typename T>
__device__ __forceinline__ T add_listed(T x, const MfView &v, int64_t row, const T *__restrict__ u) {
  int64_t e = v.cptr[row];
  const int64_t e1 = v.cptr[row + 1];
  for (; e + 3 < e1; e += 4) {
    T a[4];
#pragma unroll
    for (int q = 0; q < 4; q++) a[q] = __ldcg(u + v.clist[e + q]);
#pragma unroll
    for (int q = 0; q < 4; q++) x += a[q];
  }
  for (; e < e1; e++) x += __ldcg(u + v.clist[e]);
  return x;
}

// small fronts, forward: the first batch of E is loaded before the
// right-hand side is assembled.  cta: this CTA's index within its bucket.
// MORE: 1 fronts of more than two children as well, 2 and of listed children
template <typename T, int G, int MORE>
__device__ __forceinline__ void fwd_small_body(const MfView &v, const int *__restrict__ fronts, int nf,
                                               const T *__restrict__ E, const T *__restrict__ xl,
                                               T *__restrict__ yl, T *__restrict__ uvec, int cta,
                                               T *wsh) {
  constexpr int VN = Vec16<T>::N, M = 4 * G, PASS = M / (G * VN), FPW = 32 / G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int grp = lane / G, sl = lane % G;
  const unsigned gm = group_mask<G>(lane);
  const int gf = (cta * 8 + wid) * FPW + grp;
  if (gf >= nf) return;  // group-level work: no block barriers below
  T *w = wsh + (wid * FPW + grp) * M;
  const SolveFront &f = v.sfront[fronts[gf]];
  const int m = f.m, k = f.k, ld = round4(m), nch = f.nch;
  const int64_t xo = f.xo, cu0 = f.cu0, cu1 = f.cu1;
  const T *Ef = E + f.e_off;
  T e[PASS][kSmallUnroll][VN];
  load_e_batch<T, PASS, G>(Ef, ld, m, k, sl, 0, e);
  // the child table is static: read before the wait (a lane has at most 4 rows)
  unsigned t[4];
#pragma unroll
  for (int q = 0; q < 4; q++) t[q] = nch > 0 && sl + q * G < m ? v.ctab[f.tab + sl + q * G] : ~0u;
  pdl_wait();
#pragma unroll
  for (int h = 0; h < 4; h += 2) {  // two rows at once: more do not fit the registers
    T x[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = sl + (h + q) * G;
      x[q] = add_children(i < k ? __ldcg(xl + xo + i) : T(0), t[h + q], uvec, cu0, cu1);
    }
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (sl + (h + q) * G < m) w[sl + (h + q) * G] = x[q];
    asm volatile("" ::: "memory");
  }
  if constexpr (MORE == 2)
    if (nch < 0)
      for (int i = sl; i < m; i += G) w[i] = add_listed(w[i], v, f.tab + i, uvec);
  __syncwarp(gm);
  if constexpr (MORE > 0)  // children beyond the second, in order
    for (int ci = 2; ci < nch; ci++) {
      const ChildEdge ed = v.ch_edge[f.ch + ci];
      const int *rel = v.relmap + ed.relmap;
      for (int a = sl; a < ed.rc; a += G) w[rel[a]] += __ldcg(uvec + ed.uoff + a);
      __syncwarp(gm);
    }
  T acc[PASS][VN];
#pragma unroll
  for (int p = 0; p < PASS; p++)
#pragma unroll
    for (int q = 0; q < VN; q++) acc[p][q] = T(0);
  for (int j0 = 0; j0 < k; j0 += kSmallUnroll) {
    if (j0 > 0) load_e_batch<T, PASS, G>(Ef, ld, m, k, sl, j0, e);
#pragma unroll
    for (int u = 0; u < kSmallUnroll; u++) {
      if (j0 + u >= k) break;
      const T bj = w[j0 + u];
#pragma unroll
      for (int p = 0; p < PASS; p++)
        if (VN * sl + G * VN * p < m)  // (FP64: the pipe is the limit; no rows of padding)
#pragma unroll
          for (int q = 0; q < VN; q++) acc[p][q] += e[p][u][q] * bj;
    }
  }
  T *uf = uvec + f.uoff;
#pragma unroll
  for (int p = 0; p < PASS; p++)
#pragma unroll
    for (int q = 0; q < VN; q++) {
      const int row = VN * sl + G * VN * p + q;
      if (row < k) yl[xo + row] = acc[p][q];
      else if (row < m) uf[row - k] = w[row] + acc[p][q];
    }
}

// the sums over G lanes of four values per lane: every step halves the
// values a lane still holds (5 additions a lane for G = 16, not 16); lane
// G/4 * c .. of the group holds the sum of value c
template <typename T, int G>
__device__ __forceinline__ T reduce4(const T (&s)[4], int sl, unsigned gm) {
  const bool hi = (sl & (G / 2)) != 0;
  const T a0 = (hi ? s[2] : s[0]) + __shfl_xor_sync(gm, hi ? s[0] : s[2], G / 2);
  const T a1 = (hi ? s[3] : s[1]) + __shfl_xor_sync(gm, hi ? s[1] : s[3], G / 2);
  const bool h2 = (sl & (G / 4)) != 0;
  T t = (h2 ? a1 : a0) + __shfl_xor_sync(gm, h2 ? a0 : a1, G / 4);
#pragma unroll
  for (int o = G / 8; o > 0; o >>= 1) t += __shfl_xor_sync(gm, t, o);
  return t;
}

// small fronts, backward: the first batch of E is loaded before v is gathered
template <typename T, int G>
__device__ __forceinline__ void bwd_small_body(const MfView &v, const int *__restrict__ fronts, int nf,
                                               const T *__restrict__ E, const T *__restrict__ yl,
                                               T *__restrict__ xl, int cta, T *wsh) {
  constexpr int VN = Vec16<T>::N, M = 4 * G, PASS = M / (G * VN), FPW = 32 / G;
  static_assert(kSmallUnroll == 4, "four column sums are reduced together");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int grp = lane / G, sl = lane % G;
  const unsigned gm = group_mask<G>(lane);
  const int gf = (cta * 8 + wid) * FPW + grp;
  if (gf >= nf) return;
  T *w = wsh + (wid * FPW + grp) * M;
  const SolveFront &f = v.sfront[fronts[gf]];
  const int m = f.m, k = f.k, ld = round4(m);
  const int64_t xo = f.xo;
  const T *Ef = E + f.e_off;
  T e[PASS][kSmallUnroll][VN];
  load_e_batch<T, PASS, G>(Ef, ld, m, k, sl, 0, e);
  // the ancestor rows' positions are static: read before the wait (a lane
  // has at most 4 of the front's ld <= 4G rows)
  const int *rows = v.rows + f.rows;
  int rw[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int i = sl + q * G;
    rw[q] = (i >= k && i < m) ? rows[i] : 0;
  }
  pdl_wait();
  const T *xb = xl + f.xb;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int i = sl + q * G;
    if (i < ld) w[i] = i < k ? __ldcg(yl + xo + i) : (i < m ? __ldcg(xb + rw[q]) : T(0));
  }
  __syncwarp(gm);
  T wr[PASS][VN];
#pragma unroll
  for (int p = 0; p < PASS; p++)
#pragma unroll
    for (int q = 0; q < VN; q++) {
      const int i = VN * sl + G * VN * p + q;
      wr[p][q] = i < ld ? w[i] : T(0);
    }
  for (int c0 = 0; c0 < k; c0 += kSmallUnroll) {
    if (c0 > 0) load_e_batch<T, PASS, G>(Ef, ld, m, k, sl, c0, e);
    T s[kSmallUnroll];
#pragma unroll
    for (int u = 0; u < kSmallUnroll; u++) {
      s[u] = T(0);
      if (c0 + u < k)
#pragma unroll
        for (int p = 0; p < PASS; p++)
          if (VN * sl + G * VN * p < m)
#pragma unroll
            for (int q = 0; q < VN; q++) s[u] += e[p][u][q] * wr[p][q];
    }
    const T t = reduce4<T, G>(s, sl, gm);
    const int c = c0 + sl / (G / 4);
    if (sl % (G / 4) == 0 && c < k) xl[xo + c] = t;
  }
}

// One launch per level for the three small-front buckets: the first
// nb.x CTAs take the fronts of <= 32 rows (8 lanes each), the next nb.y those
// of <= 64 rows (16 lanes), the rest those of <= 128 rows (32 lanes).
// fronts: the level's small fronts, bucket after bucket; cnt: bucket sizes.
struct SmallBuckets {
  int cnt0, cnt1, cnt2;   // fronts per bucket
  int nb0, nb1;           // CTAs of buckets 0 and 1
};


// Several right-hand sides (nrhs > 1): CTA x serves right-hand side x % nrhs
// of the work unit x / nrhs, so the CTAs that read the same E are adjacent;
// the vectors of right-hand side k start at k * xs (xl, yl) and k * us (u).
template <typename T, int MORE>
__global__ void __launch_bounds__(256, SmallMinBlocks<T>::N)
mf_fwd_small(MfView v, const int *__restrict__ fronts, SmallBuckets sb, const T *__restrict__ E,
             const T *__restrict__ xl, T *__restrict__ yl, T *__restrict__ uvec, int nrhs = 1, int64_t xs = 0,
             int64_t us = 0) {
  __shared__ __align__(16) T wsh[8 * kSolveSmall];
  pdl_trigger();
  const int b = blockIdx.x / nrhs, rk = blockIdx.x % nrhs;
  xl += rk * xs;
  yl += rk * xs;
  uvec += rk * us;
  if (b < sb.nb0) fwd_small_body<T, 8, MORE>(v, fronts, sb.cnt0, E, xl, yl, uvec, b, wsh);
  else if (b < sb.nb0 + sb.nb1)
    fwd_small_body<T, 16, MORE>(v, fronts + sb.cnt0, sb.cnt1, E, xl, yl, uvec, b - sb.nb0, wsh);
  else
    fwd_small_body<T, 32, MORE>(v, fronts + sb.cnt0 + sb.cnt1, sb.cnt2, E, xl, yl, uvec, b - sb.nb0 - sb.nb1, wsh);
}

template <typename T>
__global__ void __launch_bounds__(256, SmallMinBlocks<T>::N)
mf_bwd_small(MfView v, const int *__restrict__ fronts, SmallBuckets sb, const T *__restrict__ E,
             const T *__restrict__ yl, T *__restrict__ xl, int nrhs = 1, int64_t xs = 0) {
  __shared__ __align__(16) T wsh[8 * kSolveSmall];
  pdl_trigger();
  const int b = blockIdx.x / nrhs, rk = blockIdx.x % nrhs;
  yl += rk * xs;
  xl += rk * xs;
  if (b < sb.nb0) bwd_small_body<T, 8>(v, fronts, sb.cnt0, E, yl, xl, b, wsh);
  else if (b < sb.nb0 + sb.nb1)
    bwd_small_body<T, 16>(v, fronts + sb.cnt0, sb.cnt1, E, yl, xl, b - sb.nb0, wsh);
  else
    bwd_small_body<T, 32>(v, fronts + sb.cnt0 + sb.cnt1, sb.cnt2, E, yl, xl, b - sb.nb0 - sb.nb1, wsh);
}

// Large fronts, forward: task = {front, (first chunk << 16) | chunk count}; a
// chunk is LPR * VN rows.  The CTA assembles the part of the right-hand side
// b that its chunks need (the pivots up to their last row, and their own
// update rows) once, then per chunk every warp takes CW = 32 / LPR columns
// of E at a time, LPR lanes of VN rows each; the warps' sums are added in a
// fixed order.  Pivot-row chunks need the columns below their last row only,
// and a vector of rows wholly above the diagonal of E is zero and not loaded.
//
// Variants (kFwdVariants, chosen per level): threads, E loads in flight per
// thread and lanes per column.  The loads of one batch are issued together,
// the first batch before the dependency wait; each further batch costs
// another round to memory, so levels with few tasks take more threads and
// shorter chunks until one batch holds a task, and levels with many take
// 128-thread CTAs at high occupancy.
struct FwdVariant { int nt, un, lpr, ctas; };  // ctas per SM (launch bounds)
constexpr FwdVariant kFwdVariants[4] = {{128, 4, 32, 12}, {256, 8, 32, 4}, {256, 8, 16, 4}, {128, 8, 32, 7}};
template <typename T, int LPR> __host__ __device__ constexpr int fwd_rows() { return LPR * Vec16<T>::N; }

// the task body; b: shared memory for the right-hand side (at most the
// front's rows), red: the warp sums of one chunk
// (MORE: as for the small ones)
template <typename T, int NT, int UN, int LPR, int MORE>
__device__ __forceinline__ void fwd_big_body(const MfView &v, int2 tk, const SolveFront &f, const T *__restrict__ E,
                                             const T *__restrict__ xl, T *__restrict__ yl, T *__restrict__ uvec,
                                             T *b, T *red) {
  constexpr int VN = Vec16<T>::N, RC = LPR * VN, NW = NT / 32, CW = 32 / LPR, STEP = NW * CW;
  const int ch0 = tk.y >> 16, nch = tk.y & 0xffff;
  const int m = f.m, k = f.k, ld = round4(m), nc = f.nch;
  const int64_t xo = f.xo, cu0 = f.cu0, cu1 = f.cu1, tab = f.tab;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int sl = lane % LPR, j0 = wid * CW + lane / LPR;
  const T *Ef = E + f.e_off;
  // one batch: columns j + u*STEP (u < UN) of the chunk's rows of this lane;
  // a vector wholly above E's diagonal (rb + VN <= column) is zero
  T e[UN][VN];
  auto load_batch = [&](int r0, int K, int j) {
    const int rb = r0 + sl * VN;
#pragma unroll
    for (int u = 0; u < UN; u++) {
      const int jj = j + u * STEP;
      if (rb < m && jj < K && rb + VN > jj) Vec16<T>::load(Ef + (int64_t)jj * ld + rb, e[u]);
      else {
#pragma unroll
        for (int q = 0; q < VN; q++) e[u][q] = T(0);
      }
    }
  };
  auto chunk_cols = [&](int r0) { return r0 < k ? min(k, r0 + RC) : k; };
  load_batch(ch0 * RC, chunk_cols(ch0 * RC), j0);  // in flight while b is assembled
  // rows of b: pivots [0, kn), then update rows [rlo, rhi); the child table
  // is static, its entries of this thread's first rows are read before the wait
  const int kn = min(k, (ch0 + nch) * RC), rlo = max(k, ch0 * RC), rhi = min(m, (ch0 + nch) * RC);
  const int nrow = kn + max(0, rhi - rlo);
  constexpr int NP = NT == 128 && UN == 4 ? 2 : 4;
  unsigned t[NP];
#pragma unroll
  for (int q = 0; q < NP; q++) {
    const int i = tid + q * NT;
    t[q] = nc > 0 && i < nrow ? v.ctab[tab + (i < kn ? i : rlo + i - kn)] : ~0u;
  }
  // A front of more than two children (MORE): the first four together, RB rows
  // of a thread at once.  (The branch is the CTA's: predicated FP64 additions
  // cost the pipe as much as others.)
  constexpr bool kPairs = MORE > 0;
  constexpr int RB = NP == 2 ? 1 : 2;
  unsigned t2[NP];
  int64_t cu2 = 0, cu3 = 0;
  if (kPairs && nc > 2) {
    cu2 = v.ch_edge[f.ch + 2].uoff;
    if (nc > 3) cu3 = v.ch_edge[f.ch + 3].uoff;
#pragma unroll
    for (int q = 0; q < NP; q++) {
      const int i = tid + q * NT;
      t2[q] = i < nrow ? v.ctab[tab + m + (i < kn ? i : rlo + i - kn)] : ~0u;
    }
  }
  pdl_wait();
  if (kPairs && nc > 2) {
#pragma unroll
    for (int h = 0; h < NP; h += RB) {
      if (h * NT >= nrow) break;
      T x[RB], c[RB][4];
#pragma unroll
      for (int q = 0; q < RB; q++) {
        const int i = tid + (h + q) * NT;
        const unsigned w0 = t[h + q], w1 = t2[h + q];
        x[q] = i < kn ? __ldcg(xl + xo + i) : T(0);
        c[q][0] = (w0 & 0xffffu) != kNoChild ? __ldcg(uvec + cu0 + (w0 & 0xffffu)) : T(0);
        c[q][1] = w0 >> 16 != kNoChild ? __ldcg(uvec + cu1 + (w0 >> 16)) : T(0);
        c[q][2] = (w1 & 0xffffu) != kNoChild ? __ldcg(uvec + cu2 + (w1 & 0xffffu)) : T(0);
        c[q][3] = w1 >> 16 != kNoChild ? __ldcg(uvec + cu3 + (w1 >> 16)) : T(0);
      }
#pragma unroll
      for (int q = 0; q < RB; q++)
        if (tid + (h + q) * NT < nrow) b[tid + (h + q) * NT] = ((x[q] + c[q][0]) + c[q][1] + c[q][2]) + c[q][3];
    }
    if (nc > 4)
#pragma unroll 1
      for (int i = tid; i < min(nrow, NP * NT); i += NT)
        b[i] = add_more_children(b[i], v, tab + (i < kn ? i : rlo + i - kn), m, nc, f.ch, 2, uvec);
  } else {
    T x[NP];
#pragma unroll
    for (int q = 0; q < NP; q++) {
      const int i = tid + q * NT;
      x[q] = add_children(i < kn ? __ldcg(xl + xo + i) : T(0), t[q], uvec, cu0, cu1);
    }
#pragma unroll
    for (int q = 0; q < NP; q++)
      if (tid + q * NT < nrow) b[tid + q * NT] = x[q];
  }
#pragma unroll 1
  for (int i = tid + NP * NT; i < nrow; i += NT) {
    const int64_t w = tab + (i < kn ? i : rlo + i - kn);
    const T s = add_children(i < kn ? __ldcg(xl + xo + i) : T(0), nc > 0 ? v.ctab[w] : ~0u, uvec, cu0, cu1);
    b[i] = kPairs ? add_more_children(s, v, w, m, nc, f.ch, 1, uvec) : s;
  }
  if constexpr (MORE == 2)
    if (nc < 0)
#pragma unroll 1
      for (int i = tid; i < nrow; i += NT) b[i] = add_listed(b[i], v, tab + (i < kn ? i : rlo + i - kn), uvec);
  __syncthreads();
  for (int ch = ch0; ch < ch0 + nch; ch++) {
    const int r0 = ch * RC;
    const int K = chunk_cols(r0);
    T acc[VN];
#pragma unroll
    for (int q = 0; q < VN; q++) acc[q] = T(0);
    for (int jw = wid * CW; jw < K; jw += UN * STEP) {
      const int j = jw + lane / LPR;
      if (jw != wid * CW) load_batch(r0, K, j);  // every chunk's first batch was loaded ahead
#pragma unroll
      for (int u = 0; u < UN; u++) {
        if (jw + u * STEP >= K) break;  // (warp-uniform: no multiplications of padding columns)
        const T bj = j + u * STEP < K ? b[j + u * STEP] : T(0);
#pragma unroll
        for (int q = 0; q < VN; q++) acc[q] += e[u][q] * bj;
      }
    }
    // the next chunk's first batch is in flight during this chunk's reduction
    if (ch + 1 < ch0 + nch) load_batch((ch + 1) * RC, chunk_cols((ch + 1) * RC), j0);
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < VN; q++) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
    if (lane < LPR)
#pragma unroll
      for (int q = 0; q < VN; q++) red[wid * RC + sl * VN + q] = acc[q];
    __syncthreads();
    const int nw = min(NW, (K + CW - 1) / CW);  // warps that had columns
    for (int i = tid; i < RC; i += NT) {
      const int row = r0 + i;
      T s = red[i];
      for (int w = 1; w < nw; w++) s += red[w * RC + i];
      if (row < k) yl[xo + row] = s;
      else if (row < m) uvec[f.uoff + row - k] = b[kn + row - rlo] + s;
    }
    __syncthreads();
  }
}

template <typename T, int V, int MORE>
__global__ void __launch_bounds__(kFwdVariants[V].nt, kFwdVariants[V].ctas)
mf_fwd_big(MfView v, const int2 *__restrict__ tasks, const SolveFront *__restrict__ tmeta, const T *__restrict__ E,
           const T *__restrict__ xl, T *__restrict__ yl, T *__restrict__ uvec, int nrhs = 1, int64_t xs = 0,
           int64_t us = 0) {
  constexpr FwdVariant fv = kFwdVariants[V];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T red[fv.nt / 32 * fwd_rows<T, fv.lpr>()];
  pdl_trigger();
  const int task = blockIdx.x / nrhs, rk = blockIdx.x % nrhs;
  fwd_big_body<T, fv.nt, fv.un, fv.lpr, MORE>(v, tasks[task], tmeta[task], E, xl + rk * xs, yl + rk * xs, uvec + rk * us,
                                        reinterpret_cast<T *>(smem_raw), red);
}

// Large fronts, backward: task = {front, column block J} of CB columns; x of
// the block from rows [CB J, m) of E.  LPC lanes per column, NT / LPC columns
// at once.  Variants as in the forward: threads, loads in flight, columns.
struct BwdVariant { int nt, un, cb, ctas; };
constexpr BwdVariant kBwdVariants[4] = {{128, 4, 32, 12}, {256, 8, 32, 4}, {256, 8, 16, 4}, {128, 8, 16, 7}};

template <typename T, int NT, int UN, int CB>
__device__ __forceinline__ void bwd_big_body(const MfView &v, int2 tk, const SolveFront &f, const T *__restrict__ E,
                                             const T *__restrict__ yl, T *__restrict__ xl, T *w) {
  constexpr int VN = Vec16<T>::N;
  // lanes per column: a 32-row vector's worth, twice that where the CTA has
  // more lanes than the block's columns need
  constexpr int LPC = NT / CB > 32 ? 32 : NT / CB > 32 / VN ? NT / CB : 32 / VN, NCS = NT / LPC, RS = LPC * VN;
  const int J = tk.y;
  const int m = f.m, k = f.k, ld = round4(m);
  const int c0 = CB * J, jb = min(CB, k - c0);
  const int64_t xo = f.xo;
  const T *xb = xl + f.xb;
  const int *rows = v.rows + f.rows;
  const int tid = threadIdx.x;
  const int rq = tid % LPC, cs = tid / LPC;
  // one batch: rows i + RS*u (u < UN) of column c for this lane; a vector
  // wholly above E's diagonal (i + VN <= c) is zero
  T e[UN][VN];
  const T *E0 = E + f.e_off;
  auto load_batch = [&](int c, int i) {
    const T *Ec = E0 + (int64_t)c * ld;
#pragma unroll
    for (int u = 0; u < UN; u++) {
      const int ii = i + u * RS;
      if (c - c0 < jb && ii < m && ii + VN > c) Vec16<T>::load(Ec + ii, e[u]);
      else {
#pragma unroll
        for (int q = 0; q < VN; q++) e[u][q] = T(0);
      }
    }
  };
  load_batch(c0 + cs, c0 + rq * VN);  // in flight while v is gathered
  // the ancestor rows' positions are static: the first kRowsAhead of this
  // thread are read before the wait
  constexpr int kRowsAhead = 4;
  int rw[kRowsAhead];
#pragma unroll
  for (int q = 0; q < kRowsAhead; q++) {
    const int i = c0 + tid + q * NT;
    rw[q] = (i >= k && i < m) ? rows[i] : 0;
  }
  pdl_wait();
#pragma unroll
  for (int q = 0; q < kRowsAhead; q++) {
    const int i = c0 + tid + q * NT;
    if (i < ld) w[i - c0] = i < k ? __ldcg(yl + xo + i) : (i < m ? __ldcg(xb + rw[q]) : T(0));
  }
  for (int i = c0 + tid + kRowsAhead * NT; i < ld; i += NT)
    w[i - c0] = i < k ? __ldcg(yl + xo + i) : (i < m ? __ldcg(xb + rows[i]) : T(0));
  __syncthreads();
  // the column sums of all passes are reduced together: FP64 additions across
  // lanes cost as much as the multiplications (16 of a lane's 56 operations
  // with 150 rows and a reduction per pass)
  constexpr int NP = CB / NCS;
  static_assert(NP == 1 || NP == 2 || NP == 4, "passes over the columns");
  T s[4];
#pragma unroll
  for (int h = 0; h < 4; h++) s[h] = T(0);
#pragma unroll
  for (int h = 0; h < NP; h++) {
    const int cc = cs + h * NCS, c = c0 + cc;
    if (cc < jb) {
      for (int i = c0 + rq * VN; i < m; i += UN * RS) {
        if (i != c0 + rq * VN) load_batch(c, i);  // every column's first batch was loaded ahead
#pragma unroll
        for (int u = 0; u < UN; u++) {
          const int ii = i + u * RS;  // w holds rows [c0, ld): rows past m are not read
          if (ii < m) {
            T x[VN];
            Vec16<T>::lds(w + ii - c0, x);
#pragma unroll
            for (int q = 0; q < VN; q++) s[h] += e[u][q] * x[q];
          }
        }
      }
    }
    if (h + 1 < NP) load_batch(c + NCS, c0 + rq * VN);
  }
  // h of this lane's sum, which lane of its group writes it
  int h = 0;
  T t;
  if constexpr (NP == 4) {
    t = reduce4<T, LPC>(s, rq, 0xffffffffu);
    h = rq / (LPC / 4);
  } else {
    t = s[0];
    if constexpr (NP == 2) {
      const bool hi = (rq & (LPC / 2)) != 0;
      t = (hi ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, hi ? s[0] : s[1], LPC / 2);
      h = hi;
    }
#pragma unroll
    for (int o = LPC / (2 * NP); o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  if (rq % (LPC / NP) == 0 && cs + h * NCS < jb) xl[xo + c0 + cs + h * NCS] = t;
}

template <typename T, int V>
__global__ void __launch_bounds__(kBwdVariants[V].nt, kBwdVariants[V].ctas)
mf_bwd_big(MfView v, const int2 *__restrict__ tasks, const SolveFront *__restrict__ tmeta, const T *__restrict__ E,
           const T *__restrict__ yl, T *__restrict__ xl, int nrhs = 1, int64_t xs = 0) {
  constexpr BwdVariant bv = kBwdVariants[V];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pdl_trigger();
  const int task = blockIdx.x / nrhs, rk = blockIdx.x % nrhs;
  bwd_big_body<T, bv.nt, bv.un, bv.cb>(v, tasks[task], tmeta[task], E, yl + rk * xs, xl + rk * xs,
                                       reinterpret_cast<T *>(smem_raw));
}

// ---------------------------------------------------------------------------
// Dependency-driven solve (solve_schedule 1): one launch per direction.  The
// tasks of all levels form one list (forward: leaves first; backward: roots
// first; the level kernels' tasks and small-front CTAs, unchanged); a CTA
// takes the next task with an atomic counter, waits until the tasks that
// produce its fronts' inputs have published their done flags (forward: the
// children's tasks, backward: the parent's), runs the task and publishes its
// own flag.  A task's dependencies come earlier in the list, so they were
// taken by CTAs that were running when they took them: no CTA waits on work
// that has not started, whether or not all CTAs are resident.  The waits are
// bounded (kQueueWaitCycles); on a timeout the CTA records ERR_WAIT and goes
// on, and the host reports the error.  Data written by other CTAs of the same
// launch (update vectors, ancestors' solutions) is read past L1 (__ldcg).
// With nrhs right-hand sides, list entry g is task g / nrhs for right-hand
// side g % nrhs and waits for the same right-hand side's producers.
// ---------------------------------------------------------------------------
constexpr long long kQueueWaitCycles = 1000000000LL;  // default wait limit, about 0.5 s at 2 GHz

struct QueueView {
  const int4 *tasks;   // {kind (0 small CTA, 1 large-front task), level, index, 0}
  const int *dep_ptr;  // dependencies of task t: dep[dep_ptr[t] .. dep_ptr[t+1])
  const int *dep;
  int ntasks;
  long long wait_cycles;  // limit of one dependency wait (clock64 cycles)
  int skip_publish;       // list entry whose done flag is never published (-1: none; failure tests)
};

__device__ __forceinline__ int ld_volatile(const int *p) { return *(const volatile int *)p; }

__device__ __forceinline__ void queue_wait(const QueueView &q, int t, int rk, int nrhs, const int *done,
                                           int *status) {
  for (int i = q.dep_ptr[t]; i < q.dep_ptr[t + 1]; i++) {
    const int *flag = done + (int64_t)q.dep[i] * nrhs + rk;
    const long long t0 = clock64();
    while (ld_volatile(flag) == 0) {
      if (clock64() - t0 > q.wait_cycles || (ld_volatile(status) & ERR_WAIT)) {
        atomicOr(status, ERR_WAIT);  // after one timeout no CTA waits any more
        return;
      }
      __nanosleep(100);
    }
  }
  __threadfence();
}

template <typename T>
__device__ __forceinline__ void queue_publish(const QueueView &q, int *done, int64_t idx) {
  __threadfence();
  if (idx == q.skip_publish) return;  // a producer that never finishes (failure tests)
  atomicExch(done + idx, 1);
}

// forward; small tasks: level lv, CTA index c of the level's small-front
// launch (fronts small_fronts + lvl_small_off[lv], buckets lvl_sb[lv])
template <typename T>
__global__ void __launch_bounds__(256, 4)
mf_fwd_queue(MfView v, QueueView q, const int *__restrict__ small_fronts, const int *__restrict__ lvl_small_off,
             const SmallBuckets *__restrict__ lvl_sb, const int2 *__restrict__ fwd_tasks,
             const SolveFront *__restrict__ fwd_tmeta, const T *__restrict__ E,
             const T *__restrict__ xl, T *__restrict__ yl, T *__restrict__ uvec, int *counter, int *done,
             int *status, int nrhs = 1, int64_t xs = 0, int64_t us = 0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T red[8 * fwd_rows<T, 32>()];
  __shared__ int s_g;
  T *sm = reinterpret_cast<T *>(smem_raw);
  const int total = q.ntasks * nrhs;
  for (;;) {
    if (threadIdx.x == 0) s_g = atomicAdd(counter, 1);
    __syncthreads();
    const int g = s_g;
    if (g >= total) return;
    const int t = g / nrhs, rk = g % nrhs;
    if (threadIdx.x == 0) queue_wait(q, t, rk, nrhs, done, status);
    __syncthreads();
    const int4 tk = q.tasks[t];
    const T *xk = xl + rk * xs;
    T *yk = yl + rk * xs, *uk = uvec + rk * us;
    if (tk.x == 0) {
      const SmallBuckets sb = lvl_sb[tk.y];
      const int *fr = small_fronts + lvl_small_off[tk.y];
      const int b = tk.z;
      if (b < sb.nb0) fwd_small_body<T, 8, 2>(v, fr, sb.cnt0, E, xk, yk, uk, b, sm);
      else if (b < sb.nb0 + sb.nb1)
        fwd_small_body<T, 16, 2>(v, fr + sb.cnt0, sb.cnt1, E, xk, yk, uk, b - sb.nb0, sm);
      else fwd_small_body<T, 32, 2>(v, fr + sb.cnt0 + sb.cnt1, sb.cnt2, E, xk, yk, uk, b - sb.nb0 - sb.nb1, sm);
    } else {
      fwd_big_body<T, 256, 8, 32, 2>(v, fwd_tasks[tk.z], fwd_tmeta[tk.z], E, xk, yk, uk, sm, red);
    }
    __syncthreads();
    if (threadIdx.x == 0) queue_publish<T>(q, done, g);
  }
}

template <typename T>
__global__ void __launch_bounds__(256, 4)
mf_bwd_queue(MfView v, QueueView q, const int *__restrict__ small_fronts, const int *__restrict__ lvl_small_off,
             const SmallBuckets *__restrict__ lvl_sb, const int2 *__restrict__ bwd_tasks,
             const SolveFront *__restrict__ bwd_tmeta, const T *__restrict__ E,
             const T *__restrict__ yl, T *__restrict__ xl, int *counter, int *done, int *status, int nrhs = 1,
             int64_t xs = 0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_g;
  T *sm = reinterpret_cast<T *>(smem_raw);
  const int total = q.ntasks * nrhs;
  for (;;) {
    if (threadIdx.x == 0) s_g = atomicAdd(counter, 1);
    __syncthreads();
    const int g = s_g;
    if (g >= total) return;
    const int t = g / nrhs, rk = g % nrhs;
    if (threadIdx.x == 0) queue_wait(q, t, rk, nrhs, done, status);
    __syncthreads();
    const int4 tk = q.tasks[t];
    const T *yk = yl + rk * xs;
    T *xk = xl + rk * xs;
    if (tk.x == 0) {
      const SmallBuckets sb = lvl_sb[tk.y];
      const int *fr = small_fronts + lvl_small_off[tk.y];
      const int b = tk.z;
      if (b < sb.nb0) bwd_small_body<T, 8>(v, fr, sb.cnt0, E, yk, xk, b, sm);
      else if (b < sb.nb0 + sb.nb1)
        bwd_small_body<T, 16>(v, fr + sb.cnt0, sb.cnt1, E, yk, xk, b - sb.nb0, sm);
      else bwd_small_body<T, 32>(v, fr + sb.cnt0 + sb.cnt1, sb.cnt2, E, yk, xk, b - sb.nb0 - sb.nb1, sm);
    } else {
      bwd_big_body<T, 256, 8, 32>(v, bwd_tasks[tk.z], bwd_tmeta[tk.z], E, yk, xk, sm);
    }
    __syncthreads();
    if (threadIdx.x == 0) queue_publish<T>(q, done, g);
  }
}

// ---------------------------------------------------------------------------
// Symmetric Gauss-Seidel subdomain preconditioner (fine_method 2).  The
// reference runs, per subdomain, forward and backward Gauss-Seidel sweeps in
// global row order on the entries of A inside the subdomain, from x = 0
// (FinePreconditioner_sgs.F90:69-86, stationary.F90:33-88).  Here one CTA owns
// one subdomain; its rows are grouped into dependency levels of the
// (symmetrised) subdomain graph, so every row of a level depends only on rows
// of earlier levels in the sweep direction, and the result equals the
// sequential sweep (same entry order, separate multiply and subtract,
// division by the diagonal).  Levels are separated by __syncthreads.
// ---------------------------------------------------------------------------
struct SgsView {
  const int64_t *rp;        // local CSR over arena positions (entries inside the subdomain)
  const int *ci;            // column as arena position
  const double *va, *dg;    // values; diagonal (0 = row skipped, as in the reference)
  const int *gidx;          // global row of every arena position
  const int *sd_lev_f, *sd_lev_b;    // per subdomain: its range of levels
  const int *lev_f, *lev_b;          // per level: its range of rows
  const int *rows_f, *rows_b;        // rows (arena positions) grouped by level
};

constexpr int kSgsThreads = 256;

__device__ __forceinline__ void sgs_sweep(const SgsView &g, const int *sd_lev, const int *lev, const int *rows,
                                          int sd, const double *__restrict__ r, double *__restrict__ x) {
  for (int L = sd_lev[sd]; L < sd_lev[sd + 1]; L++) {
    for (int t = lev[L] + threadIdx.x; t < lev[L + 1]; t += kSgsThreads) {
      const int q = rows[t];
      const double d = g.dg[q];
      if (d == 0.0) continue;
      double xi = r[g.gidx[q]];
      for (int64_t e = g.rp[q]; e < g.rp[q + 1]; e++) {
        const int c = g.ci[e];
        if (c != q) xi = __dsub_rn(xi, __dmul_rn(g.va[e], x[c]));
      }
      x[q] = __ddiv_rn(xi, d);
    }
    __syncthreads();
  }
}

// one CTA per subdomain: x (arena, subdomain block) = SGS(iters) applied to r
__global__ void __launch_bounds__(kSgsThreads)
sgs_subdomains(SgsView g, const int64_t *__restrict__ sd_ptr, int iters, const double *__restrict__ r,
               double *__restrict__ x) {
  const int sd = blockIdx.x;
  for (int64_t q = sd_ptr[sd] + threadIdx.x; q < sd_ptr[sd + 1]; q += kSgsThreads) x[q] = 0.0;
  __syncthreads();
  for (int it = 0; it < iters; it++) {
    sgs_sweep(g, g.sd_lev_f, g.lev_f, g.rows_f, sd, r, x);
    sgs_sweep(g, g.sd_lev_b, g.lev_b, g.rows_b, sd, r, x);
  }
}

// ---------------------------------------------------------------------------
// Gradients of a loss L(x) through x = A^-1 b, given the adjoint solution
// lambda = A^-1 dL/dx (A symmetric): dL/db = lambda, dL/dA_ij = -lambda_i x_j.
// ---------------------------------------------------------------------------
// one value per input triplet (row gi, column gj, 0-based)
__global__ void grad_coo(int64_t nnz, const int *__restrict__ gi, const int *__restrict__ gj,
                         const double *__restrict__ lam, const double *__restrict__ x, double *__restrict__ g) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
    g[k] = -(lam[gi[k]] * x[gj[k]]);
}

// one value per element: the derivative with respect to a factor s_e that
// scales the element's matrix, -sum_ij lambda[f_j] A_e(i,j) x[f_i] (the
// element assembly stores A_e(i,j) at row f_j, column f_i); one warp per
// element, the element's terms summed in a fixed order
__global__ void grad_elements(int nell, const int *__restrict__ eptr, const int *__restrict__ efl,
                              const int64_t *__restrict__ eoff, const double *__restrict__ emat,
                              const double *__restrict__ lam, const double *__restrict__ x, double *__restrict__ g) {
  const int lane = threadIdx.x & 31;
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (e >= nell) return;
  const int f0 = eptr[e], nf = eptr[e + 1] - f0;
  const double *Ae = emat + eoff[e];
  double s = 0.0;
  for (int q = lane; q < nf * nf; q += 32) {
    const int j = q / nf, i = q % nf;  // column j, row i of the element matrix
    s += lam[efl[f0 + j]] * Ae[q] * x[efl[f0 + i]];
  }
  s = warp_sum(s);
  if (lane == 0) g[e] = -s;
}

// ---------------------------------------------------------------------------
// Matrix-free product with stored element matrices (elemental input, option
// elemental_matvec 1): q = A p with A = sum_e of element e's matrix placed at
// its freedoms (A_e(i,j) at row f_j, column f_i, as the element assembly puts
// it).  Pass 1 stages a run of element matrices in shared memory with
// coalesced loads and forms every element's column products
// c[e, j] = sum_i A_e(i,j) p[f_i]; pass 2 sums, for every row, its element
// contributions in element order (no atomics: the result is deterministic)
// and the p.q partial sums.
// ---------------------------------------------------------------------------
constexpr int kElemChunk = 4096;  // matrix values per CTA stage (32 KB)
constexpr int kElemFree = 512;    // element freedoms per CTA stage
constexpr int kElemRun = 512;     // elements per CTA stage

// A(i, j) of an element matrix in shared memory: full column-major storage,
// or (SYM) the lower triangle column by column, column c starting at
// c*nf - c(c-1)/2 (for bitwise symmetric element matrices: the same values)
template <bool SYM>
__device__ __forceinline__ double elem_entry(const double *Me, int nf, int i, int j) {
  if (!SYM) return Me[j * nf + i];
  const int r = i >= j ? i : j, c = i >= j ? j : i;
  return Me[c * nf - (c * (c - 1)) / 2 + (r - c)];
}

// task t = elements [erun[t], erun[t+1]); the CTA stages their matrices, their
// offsets and the p values of their freedoms in shared memory (coalesced
// loads; the p gathers all in flight at once), then one thread per
// (element, column): c = sum_i A_e(i, j) p[f_i] in increasing i
template <bool SYM>
__global__ void __launch_bounds__(256)
elem_contrib(const int *__restrict__ erun, const int *__restrict__ eptr, const int *__restrict__ efl,
             const int64_t *__restrict__ eoff, const double *__restrict__ emat, const double *__restrict__ p,
             double *__restrict__ c) {
  __shared__ double Ms[kElemChunk];
  __shared__ double ps[kElemFree];
  __shared__ int ep[kElemRun + 1], eo[kElemRun + 1];
  const int e0 = erun[blockIdx.x], e1 = erun[blockIdx.x + 1], ne = e1 - e0;
  const int f0 = eptr[e0], nfr = eptr[e1] - f0;
  const int64_t m0 = eoff[e0];
  const int len = (int)(eoff[e1] - m0);
  for (int q = threadIdx.x; q < len; q += blockDim.x) Ms[q] = emat[m0 + q];
  for (int q = threadIdx.x; q <= ne; q += blockDim.x) {
    ep[q] = eptr[e0 + q] - f0;
    eo[q] = (int)(eoff[e0 + q] - m0);
  }
  for (int q = threadIdx.x; q < nfr; q += blockDim.x) ps[q] = p[efl[f0 + q]];
  __syncthreads();
  for (int t = threadIdx.x; t < nfr; t += blockDim.x) {
    int lo = 0, hi = ne - 1;  // element of item t: the last e with ep[e] <= t
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (ep[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const int fe = ep[lo], nf = ep[lo + 1] - fe, j = t - fe;
    const double *Me = Ms + eo[lo];
    const double *pe = ps + fe;
    double s = 0.0;
    // fused multiply-adds: FP64 issue, not DRAM, bounds this product on GB300
    for (int i = 0; i < nf; i++) s = __fma_rn(elem_entry<SYM>(Me, nf, i, j), pe[i], s);
    c[f0 + t] = s;
  }
}

// q[r] = sum of r's element contributions (element order); partial p.q.
// Four contributions of a row are loaded before they are added.
__global__ void __launch_bounds__(kVecThreads)
elem_pull_pq(int n, const int64_t *__restrict__ rptr, const int *__restrict__ ridx, const double *__restrict__ c,
             const double *__restrict__ p, double *__restrict__ q, double *__restrict__ part_pq) {
  __shared__ double sh[32];
  double spq = 0.0;
  for (int r = blockIdx.x * kVecThreads + threadIdx.x; r < n; r += gridDim.x * kVecThreads) {
    const int64_t t0 = rptr[r], t1 = rptr[r + 1];
    const double pr = p[r];
    double s = 0.0;
    int64_t t = t0;
    for (; t + 4 <= t1; t += 4) {
      const int i0 = ridx[t], i1 = ridx[t + 1], i2 = ridx[t + 2], i3 = ridx[t + 3];
      const double c0 = c[i0], c1 = c[i1], c2 = c[i2], c3 = c[i3];
      s = __dadd_rn(s, c0);
      s = __dadd_rn(s, c1);
      s = __dadd_rn(s, c2);
      s = __dadd_rn(s, c3);
    }
    for (; t < t1; t++) s = __dadd_rn(s, c[ridx[t]]);
    q[r] = s;
    spq += pr * s;
  }
  double b = block_sum<kVecThreads>(spq, sh);
  if (threadIdx.x == 0) part_pq[blockIdx.x] = b;
}

// ---------------------------------------------------------------------------
// Schwarz gather / pull sum and coarse transfer
// ---------------------------------------------------------------------------
// Conversions between FP32 and FP64 (exact, and round to nearest even), in
// integer operations: a conversion instruction takes the FP64 pipe as long as
// a multiply-add (64 clocks of a sub-partition), and the mixed pull sum makes
// seven a node beside five additions (by count 43 of its 71 us at 128^3).
// Zeros and numbers normal in both formats; others by the instruction.  Per
// iteration: 128^3 1108 -> 1092 us, 32 right-hand sides of 513^2 1508 -> 1448,
// 48 grids 255 -> 243.
__device__ __forceinline__ double to_f64(double x) { return x; }
__device__ __forceinline__ double to_f64(float x) {
  const unsigned b = (unsigned)__float_as_int(x), a = b & 0x7fffffffu;
  if (a != 0u && a - 0x00800000u >= 0x7f000000u) return (double)x;  // subnormal, infinity, NaN
  const unsigned hi = (b & 0x80000000u) | (a ? (a >> 3) + (896u << 20) : 0u);
  return __hiloint2double((int)hi, (int)(b << 29));
}
template <typename T>
__device__ __forceinline__ T from_f64(double x);
template <>
__device__ __forceinline__ double from_f64<double>(double x) { return x; }
template <>
__device__ __forceinline__ float from_f64<float>(double x) {
  const unsigned h = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), a = h & 0x7fffffffu;
  if ((a | lo) != 0u && a - (897u << 20) >= (253u << 20)) return (float)x;  // subnormal or too large for FP32, NaN
  unsigned f = (a << 3 | lo >> 29) - (896u << 23);
  const unsigned rem = lo << 3;  // the dropped bits
  f += rem > 0x80000000u || (rem == 0x80000000u && (f & 1u));
  return __int_as_float((int)((h & 0x80000000u) | ((a | lo) ? f : 0u)));
}

// nrhs right-hand sides: vector k at r + k * rs, local vector k at xl + k * len
template <typename T>
__global__ void gather_subdomains(const double *__restrict__ r, const int *__restrict__ gidx,
                                  T *__restrict__ xl, int64_t len, int nrhs = 1, int64_t rs = 0) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < len;
       p += (int64_t)gridDim.x * blockDim.x) {
    const int g = gidx[p];
    for (int k = 0; k < nrhs; k++) xl[k * len + p] = from_f64<T>(r[k * rs + g]);
  }
}

// crhs (in the coarse batch's local numbering) = R r
// nrhs right-hand sides: r_k at r + k * rs, the coarse vector k at xc + k * xcs.
// L lanes per coarse row (chosen for about 12 entries per lane), four loads
// in flight per lane, the lane sums added by a shuffle tree; G right-hand
// sides at once share the entries and their conversions to FP64 (blockIdx.y:
// groups of them).
template <typename TR, int L, int G>
__global__ void __launch_bounds__(kVecThreads)
restrict_to_coarse(const int64_t *__restrict__ Rp, const int *__restrict__ Rc, const TR *__restrict__ Rv,
                   const double *__restrict__ r, const int *__restrict__ cpos, double *__restrict__ xc, int nc,
                   int nrhs = 1, int64_t rs = 0, int64_t xcs = 0) {
  const int sub = threadIdx.x % L;
  const int rows_per_grid = gridDim.x * (kVecThreads / L);
  constexpr int U = G > 1 ? 2 : 4;
  for (int a0 = blockIdx.x * (kVecThreads / L); a0 < nc; a0 += rows_per_grid) {
    const int a = a0 + threadIdx.x / L;
    const bool on = a < nc;
    const int64_t e0 = on ? Rp[a] : 0, e1 = on ? Rp[a + 1] : 0;
    for (int k0 = blockIdx.y * G; k0 < nrhs; k0 += gridDim.y * G) {
      const double *rk = r + k0 * rs;
      double s[G];
#pragma unroll
      for (int g = 0; g < G; g++) s[g] = 0.0;
      int64_t e = e0 + sub;
      for (; e + (U - 1) * L < e1; e += U * L) {
        int c[U];
        double w[U], x[U][G];
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = Rc[e + u * L];
#pragma unroll
        for (int u = 0; u < U; u++) w[u] = to_f64(Rv[e + u * L]);
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int g = 0; g < G; g++) x[u][g] = k0 + g < nrhs ? rk[g * rs + c[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int g = 0; g < G; g++) s[g] += w[u] * x[u][g];
      }
      for (; e < e1; e += L) {
        const int c = Rc[e];
        const double w = to_f64(Rv[e]);
#pragma unroll
        for (int g = 0; g < G; g++)
          if (k0 + g < nrhs) s[g] += w * rk[g * rs + c];
      }
#pragma unroll
      for (int g = 0; g < G; g++) {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) s[g] += __shfl_down_sync(0xffffffffu, s[g], o, L);
        if (on && sub == 0 && k0 + g < nrhs) xc[(k0 + g) * xcs + cpos[a]] = s[g];
      }
    }
  }
}

// z_g = (sum of subdomain solutions at g, in subdomain order) + (P x_c)_g ;
// partial sums of r.z (and of r.z_old for the flexible variant).  One thread
// per node; Pcp holds coarse-vector positions (composed at setup).  The loads
// of a node are issued in three dependent rounds (row pointers, r and z_old;
// the first two pull positions and the first four P entries; the gathers),
// the rare longer rows finish in loops; the sums keep the entries' order.
template <typename T, typename TP>
__global__ void __launch_bounds__(kVecThreads)
pull_prolong_dot(int n, const int *__restrict__ pull_ptr, const int *__restrict__ pull_idx,
                 const T *__restrict__ xl, const int64_t *__restrict__ Pp, const int *__restrict__ Pcp,
                 const TP *__restrict__ Pv, const double *__restrict__ xc,
                 int mode, const double *__restrict__ r, double *__restrict__ z,
                 double *__restrict__ zold, double *__restrict__ part_rz, double *__restrict__ part_rzo,
                 const int *__restrict__ cb = nullptr, const int *__restrict__ csys = nullptr,
                 int64_t vs = 0, int64_t xls = 0, int64_t xcs = 0) {
  // mode bit 0: fine subdomains on; bit 1: coarse on; bit 2: identity fine (z=r);
  // bit 3: keep z_old and produce r.z_old.  cb (batched systems / right-hand
  // sides): CTA b owns the positions [cb[b], cb[b+1]) of the stacked vectors
  // and its partial sums are that chunk's; with csys, the chunk belongs to
  // right-hand side k = csys[b]: rows g - k*vs of the matrix and the local
  // vectors at k*xls (subdomains) and k*xcs (coarse).
  __shared__ double sh[32];
  pdl_trigger();
  double srz = 0.0, srzo = 0.0;
  const int g0 = cb ? cb[blockIdx.x] + threadIdx.x : blockIdx.x * kVecThreads + threadIdx.x;
  const int gend = cb ? cb[blockIdx.x + 1] : n;
  const int gstep = cb ? kVecThreads : gridDim.x * kVecThreads;
  const int64_t rk = csys ? csys[blockIdx.x] : 0;
  const int64_t voff = rk * vs;
  if (xl) xl += rk * xls;
  if (xc) xc += rk * xcs;
  const bool pull = (mode & 5) == 1, prol = (mode & 2) != 0, flex = (mode & 8) != 0;
  for (int gg = g0; gg < gend; gg += gstep) {
    const int64_t g = gg;              // position in the stacked vectors
    const int gl = (int)(g - voff);    // row of the matrix / pull lists
    // round 1
    const double rg = r[g];
    const double zo = flex ? zold[g] : 0.0;
    int q0 = 0, q1 = 0;
    int64_t e0 = 0, e1 = 0;
    if (pull) { q0 = pull_ptr[gl]; q1 = pull_ptr[gl + 1]; }
    if (prol) { e0 = Pp[gl]; e1 = Pp[gl + 1]; }
    // round 2
    const int i0 = q0 < q1 ? pull_idx[q0] : -1;
    const int i1 = q0 + 1 < q1 ? pull_idx[q0 + 1] : -1;
    int pc[4];
    TP pv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const bool on = e0 + u < e1;
      pc[u] = on ? Pcp[e0 + u] : -1;
      pv[u] = on ? Pv[e0 + u] : TP(0);
    }
    // round 3
    const T x0 = i0 >= 0 ? xl[i0] : T(0);
    const T x1 = i1 >= 0 ? xl[i1] : T(0);
    TP xv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) xv[u] = pc[u] >= 0 ? from_f64<TP>(xc[pc[u]]) : TP(0);
    double sv = 0.0;
    if (mode & 4) {
      sv = rg;
    } else if (pull) {
      if (i0 >= 0) sv = sv + to_f64(x0);
      if (i1 >= 0) sv = sv + to_f64(x1);
      for (int q = q0 + 2; q < q1; q++) sv = sv + to_f64(xl[pull_idx[q]]);
    }
    if (prol) {
      TP t = TP(0);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (pc[u] >= 0) t += pv[u] * xv[u];
      for (int64_t e = e0 + 4; e < e1; e++) t += Pv[e] * from_f64<TP>(xc[Pcp[e]]);
      sv = sv + to_f64(t);
    }
    if (flex) {
      srzo += rg * zo;
      zold[g] = sv;
    }
    z[g] = sv;
    srz += rg * sv;
  }
  double b = block_sum<kVecThreads>(srz, sh);
  if (threadIdx.x == 0) part_rz[blockIdx.x] = b;
  if (flex) {
    b = block_sum<kVecThreads>(srzo, sh);
    if (threadIdx.x == 0) part_rzo[blockIdx.x] = b;
  }
}

// ---------------------------------------------------------------------------
// CG steps.  sc[] holds device scalars:
//   0 rho_prev, 1 rho, 2 alpha, 3 res_norm (r.r), 4 init_norm, 5 beta, 6 p.q
// ---------------------------------------------------------------------------
enum { SC_RHO_PREV = 0, SC_RHO = 1, SC_ALPHA = 2, SC_RES = 3, SC_INIT = 4, SC_BETA = 5, SC_PQ = 6 };

// beta of the iteration from the r.z partials: Fletcher-Reeves (DOUG) or
// flexible Polak-Ribiere
__device__ __forceinline__ double cg_beta(const double *part_rz, const double *part_rzo,
                                          const double *sc, int first, int flexible, int np, double *rho_out) {
  const double rho = sum_partials(part_rz, np);
  *rho_out = rho;
  if (first) return 0.0;
  if (flexible) {
    const double rzo = sum_partials(part_rzo, np);
    return __ddiv_rn(__dsub_rn(rho, rzo), __ldcg(sc + SC_RHO_PREV));
  }
  return __ddiv_rn(rho, __ldcg(sc + SC_RHO_PREV));
}

// p = z + beta p (p = z on the first step); beta from the r.z partials
__global__ void __launch_bounds__(kVecThreads)
cg_direction(int n, const double *z, double *p,
             const double *part_rz, const double *part_rzo,
             double *sc, int first, int flexible, int np) {
  __shared__ double s_beta;
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x < 32) {
    double rho;
    double beta = cg_beta(part_rz, part_rzo, sc, first, flexible, np, &rho);
    if (threadIdx.x == 0) {
      s_beta = beta;
      if (blockIdx.x == 0) { sc[SC_RHO] = rho; sc[SC_BETA] = beta; }
    }
  }
  __syncthreads();
  const double beta = s_beta;
  for (int i = blockIdx.x * kVecThreads + threadIdx.x; i < n; i += gridDim.x * kVecThreads)
    p[i] = first ? z[i] : __fma_rn(beta, p[i], z[i]);
}

// q = A p with LANES lanes per row; partial sums of p.q
template <int LANES>
__global__ void __launch_bounds__(kVecThreads)
spmv_pq(int n, const int64_t *__restrict__ Ap, const int *__restrict__ Ac, const double *__restrict__ Av,
        const double *__restrict__ p, double *__restrict__ q, double *__restrict__ part_pq) {
  __shared__ double sh[32];
  const int sub = threadIdx.x % LANES;
  const int rows_per_block = kVecThreads / LANES;
  double spq = 0.0;
  pdl_trigger();
  for (int row0 = blockIdx.x * rows_per_block; row0 < n; row0 += gridDim.x * rows_per_block) {
    const int i = row0 + threadIdx.x / LANES;
    double s = 0.0;
    if (i < n) {
      int64_t e = Ap[i] + sub;
      const int64_t e1 = Ap[i + 1];
      // four entries of this lane's share loaded before they are summed
      for (; e + 3 * LANES < e1; e += 4 * LANES) {
        const int c0 = Ac[e], c1 = Ac[e + LANES], c2 = Ac[e + 2 * LANES], c3 = Ac[e + 3 * LANES];
        const double a0 = Av[e], a1 = Av[e + LANES], a2 = Av[e + 2 * LANES], a3 = Av[e + 3 * LANES];
        const double p0 = p[c0], p1 = p[c1], p2 = p[c2], p3 = p[c3];
        s = __fma_rn(a0, p0, s);
        s = __fma_rn(a1, p1, s);
        s = __fma_rn(a2, p2, s);
        s = __fma_rn(a3, p3, s);
      }
      for (; e < e1; e += LANES) s = __fma_rn(Av[e], p[Ac[e]], s);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
    if (i < n && sub == 0) {
      q[i] = s;
      spq += p[i] * s;
    }
  }
  double b = block_sum<kVecThreads>(spq, sh);
  if (threadIdx.x == 0) part_pq[blockIdx.x] = b;
}

// end of an iteration: res = r.r, rho_prev = rho, and what the host reads
__device__ __forceinline__ void cg_publish(double *sc, double rr, int init, volatile double *host_out,
                                           const int *status, volatile int *host_status) {
  // init: 1 = initial residual, 0 = end of an iteration, 2 = report only
  if (init == 1) sc[SC_INIT] = rr;
  else if (init == 0) { sc[SC_RES] = rr; sc[SC_RHO_PREV] = __ldcg(sc + SC_RHO); }
  host_out[0] = rr;
  host_out[1] = __ldcg(sc + SC_INIT);
  host_out[2] = __ldcg(sc + SC_ALPHA);
  host_out[3] = __ldcg(sc + SC_BETA);
  host_out[4] = __ldcg(sc + SC_RHO);
  host_out[5] = __ldcg(sc + SC_PQ);
  *host_status = __ldcg(status);
}

// x += alpha p; r -= alpha q; partial r.r  (alpha = rho / p.q).  With a
// ticket the last CTA ends the iteration (a launch of its own takes 3 us).
__global__ void __launch_bounds__(kVecThreads)
cg_update(int n, const double *p, const double *q,
          double *x, double *r, double *sc,
          const double *part_pq, double *part_rr, int np,
          int *ticket = nullptr, volatile double *host_out = nullptr,
          const int *status = nullptr, volatile int *host_status = nullptr) {
  __shared__ double sh[32];
  __shared__ double s_alpha;
  __shared__ bool s_last;
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x < 32) {
    const double pq = sum_partials(part_pq, np);
    if (threadIdx.x == 0) {
      const double alpha = __ddiv_rn(__ldcg(sc + SC_RHO), pq);
      s_alpha = alpha;
      if (blockIdx.x == 0) { sc[SC_ALPHA] = alpha; sc[SC_PQ] = pq; }
    }
  }
  __syncthreads();
  const double alpha = s_alpha;
  double srr = 0.0;
  for (int i = blockIdx.x * kVecThreads + threadIdx.x; i < n; i += gridDim.x * kVecThreads) {
    x[i] = __fma_rn(alpha, p[i], x[i]);
    const double ri = __fma_rn(-alpha, q[i], r[i]);
    r[i] = ri;
    srr += ri * ri;
  }
  double b = block_sum<kVecThreads>(srr, sh);
  if (threadIdx.x == 0) {
    part_rr[blockIdx.x] = b;
    if (ticket) {
      __threadfence();
      s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
  }
  if (!ticket) return;
  __syncthreads();
  if (s_last && threadIdx.x < 32) {
    __threadfence();
    const double rr = sum_partials(part_rr, gridDim.x);
    if (threadIdx.x == 0) {
      *ticket = 0;
      cg_publish((double *)sc, rr, 0, host_out, status, host_status);
    }
  }
}

// r = b - A x (FP64 true residual), partial r.r
template <int LANES>
__global__ void __launch_bounds__(kVecThreads)
residual(int n, const int64_t *__restrict__ Ap, const int *__restrict__ Ac, const double *__restrict__ Av,
         const double *__restrict__ x, const double *__restrict__ b, double *__restrict__ r,
         double *__restrict__ part_rr) {
  __shared__ double sh[32];
  const int sub = threadIdx.x % LANES;
  const int rows_per_block = kVecThreads / LANES;
  double srr = 0.0;
  for (int row0 = blockIdx.x * rows_per_block; row0 < n; row0 += gridDim.x * rows_per_block) {
    const int i = row0 + threadIdx.x / LANES;
    double s = 0.0;
    if (i < n)
      for (int64_t e = Ap[i] + sub; e < Ap[i + 1]; e += LANES) s = __fma_rn(Av[e], x[Ac[e]], s);
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
    if (i < n && sub == 0) {
      const double ri = __dsub_rn(b[i], s);
      r[i] = ri;
      srr += ri * ri;
    }
  }
  double t = block_sum<kVecThreads>(srr, sh);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = t;
}

// the same after a residual in full (init: see cg_publish)
__global__ void cg_finish(double *__restrict__ sc, const double *__restrict__ part_rr, int np, int init,
                          volatile double *__restrict__ host_out, const int *__restrict__ status,
                          volatile int *__restrict__ host_status) {
  const double rr = sum_partials(part_rr, np);
  if (threadIdx.x == 0) cg_publish(sc, rr, init, host_out, status, host_status);
}

// ---------------------------------------------------------------------------
// Batched independent systems (dg_set_systems).  The systems are the diagonal
// blocks of one matrix; every CTA of these vector kernels owns one chunk
// [cb[c], cb[c+1]) of the rows of system csys[c], so partial sums are per
// chunk and the CG scalars per system (bsc[k * BS_N + ...]).  A system leaves
// the iteration when its own residual test passes: its x, r and p are then
// frozen while the others go on, which makes each system's iterates those of
// its own PCG.
// ---------------------------------------------------------------------------
constexpr int kBatchChunk = 1024;  // rows per CTA of the batched vector kernels (or a multiple)
enum { BS_RHO_PREV = 0, BS_RHO = 1, BS_ALPHA = 2, BS_RES = 3, BS_INIT = 4, BS_BETA = 5, BS_PQ = 6,
       BS_TRUE = 7, BS_N = 8 };
// per-system state
enum { BT_DONE = 0, BT_ACTIVE = 1, BT_CHECK = 2, BT_BREAKDOWN = 3 };
// bt_scalars steps
enum { BT_INIT = 2, BT_FINISH = 3, BT_CONFIRM = 4, BT_REPORT = 5 };

// sum of a system's chunk partials, by one warp, in a fixed order
__device__ __forceinline__ double bt_sum(const double *part, const int *sys_cptr, int k) {
  return sum_partials(part + sys_cptr[k], sys_cptr[k + 1] - sys_cptr[k]);
}

// p = z + beta p; every CTA forms its system's beta from the chunk partials,
// the system's first one keeps rho and beta (a launch of one CTA for all
// systems' scalars takes 8 us)
__global__ void __launch_bounds__(kVecThreads)
bt_direction(const int *cb, const int *csys, const int *sys_cptr,
             const int *state, double *bsc, const double *part_rz,
             const double *part_rzo, const double *z, double *p, int first,
             int flexible) {
  __shared__ double s_beta;
  pdl_trigger();
  pdl_wait();
  const int k = csys[blockIdx.x];
  if (__ldcg(state + k) != BT_ACTIVE) return;
  if (threadIdx.x < 32) {
    double *sc = bsc + (size_t)k * BS_N;
    const double rho = bt_sum(part_rz, sys_cptr, k);
    double beta = 0.0;
    if (!first) {
      const double rzo = flexible ? bt_sum(part_rzo, sys_cptr, k) : 0.0;
      beta = __ddiv_rn(flexible ? __dsub_rn(rho, rzo) : rho, __ldcg(sc + BS_RHO_PREV));
    }
    if (threadIdx.x == 0) {
      s_beta = beta;
      if ((int)blockIdx.x == sys_cptr[k]) { sc[BS_RHO] = rho; sc[BS_BETA] = beta; }
    }
  }
  __syncthreads();
  const double beta = s_beta;
  const int i1 = cb[blockIdx.x + 1];
  for (int i = cb[blockIdx.x] + threadIdx.x; i < i1; i += kVecThreads)
    p[i] = first ? z[i] : __fma_rn(beta, p[i], z[i]);
}

// q = A p on the chunk's rows (LANES lanes per row), partial p.q
template <int LANES>
__global__ void __launch_bounds__(kVecThreads)
bt_spmv_pq(const int *__restrict__ cb, const int *__restrict__ csys, const int *__restrict__ state,
           const int64_t *__restrict__ Ap, const int *__restrict__ Ac, const double *__restrict__ Av,
           const double *__restrict__ p, double *__restrict__ q, double *__restrict__ part_pq) {
  __shared__ double sh[32];
  pdl_trigger();
  if (state[csys[blockIdx.x]] != BT_ACTIVE) {
    if (threadIdx.x == 0) part_pq[blockIdx.x] = 0.0;
    return;
  }
  const int sub = threadIdx.x % LANES;
  const int rows_per_block = kVecThreads / LANES;
  const int i1 = cb[blockIdx.x + 1];
  double spq = 0.0;
  for (int row0 = cb[blockIdx.x]; row0 < i1; row0 += rows_per_block) {
    const int i = row0 + threadIdx.x / LANES;
    double s = 0.0;
    if (i < i1) {
      int64_t e = Ap[i] + sub;
      const int64_t e1 = Ap[i + 1];
      for (; e + 3 * LANES < e1; e += 4 * LANES) {
        const int c0 = Ac[e], c1 = Ac[e + LANES], c2 = Ac[e + 2 * LANES], c3 = Ac[e + 3 * LANES];
        const double a0 = Av[e], a1 = Av[e + LANES], a2 = Av[e + 2 * LANES], a3 = Av[e + 3 * LANES];
        const double p0 = p[c0], p1 = p[c1], p2 = p[c2], p3 = p[c3];
        s = __fma_rn(a0, p0, s);
        s = __fma_rn(a1, p1, s);
        s = __fma_rn(a2, p2, s);
        s = __fma_rn(a3, p3, s);
      }
      for (; e < e1; e += LANES) s = __fma_rn(Av[e], p[Ac[e]], s);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
    if (i < i1 && sub == 0) {
      q[i] = s;
      spq += p[i] * s;
    }
  }
  double b = block_sum<kVecThreads>(spq, sh);
  if (threadIdx.x == 0) part_pq[blockIdx.x] = b;
}

// q = A p for G right-hand sides of one matrix at once: a row's entries are
// read once for them (one right-hand side per CTA spent 250 us at 32 right-hand
// sides of 513^2 unknowns on entries that a warp's lanes read 56 bytes apart).
// CTA b: chunk b % nch of `chunk` rows, right-hand sides G * (b / nch) ..; the
// partial sum of right-hand side k at k * nch + chunk.  Right-hand sides that
// left the iteration are not read.  174 us: FP64 issue takes 110.
template <int LANES, int G>
__global__ void __launch_bounds__(kVecThreads)
bt_spmv_pq_multi(int n, int nrhs, int nch, int chunk, const int *__restrict__ state, const int64_t *__restrict__ Ap,
                 const int *__restrict__ Ac, const double *__restrict__ Av, const double *__restrict__ p,
                 double *__restrict__ q, double *__restrict__ part_pq, int64_t vs) {
  __shared__ double sh[32];
  pdl_trigger();
  const int cc = blockIdx.x % nch, k0 = blockIdx.x / nch * G;
  bool on[G], any = false;
#pragma unroll
  for (int g = 0; g < G; g++) {
    on[g] = k0 + g < nrhs && state[k0 + g] == BT_ACTIVE;
    any |= on[g];
    if (k0 + g < nrhs && !on[g] && threadIdx.x == 0) part_pq[(k0 + g) * nch + cc] = 0.0;
  }
  if (!any) return;
  p += k0 * vs;
  q += k0 * vs;
  const int sub = threadIdx.x % LANES;
  constexpr int rows_per_block = kVecThreads / LANES, U = 4;
  const int i1 = min(n, (cc + 1) * chunk);
  double spq[G];
#pragma unroll
  for (int g = 0; g < G; g++) spq[g] = 0.0;
  for (int row0 = cc * chunk; row0 < i1; row0 += rows_per_block) {
    const int i = row0 + threadIdx.x / LANES;
    double s[G];
#pragma unroll
    for (int g = 0; g < G; g++) s[g] = 0.0;
    if (i < i1) {
      const int64_t e1 = Ap[i + 1];
      for (int64_t e = Ap[i] + sub; e < e1; e += U * LANES) {
        int c[U];
        double a[U], x[U][G];
#pragma unroll
        for (int u = 0; u < U; u++) c[u] = e + u * LANES < e1 ? Ac[e + u * LANES] : -1;
#pragma unroll
        for (int u = 0; u < U; u++) a[u] = c[u] >= 0 ? Av[e + u * LANES] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int g = 0; g < G; g++) x[u][g] = on[g] && c[u] >= 0 ? p[g * vs + c[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (e - sub + u * LANES >= e1) break;  // (no multiplications of a whole group's padding)
#pragma unroll
          for (int g = 0; g < G; g++)
            if (c[u] >= 0) s[g] = __fma_rn(a[u], x[u][g], s[g]);
        }
      }
    }
#pragma unroll
    for (int g = 0; g < G; g++) {
#pragma unroll
      for (int o = LANES / 2; o > 0; o >>= 1) s[g] += __shfl_down_sync(0xffffffffu, s[g], o, LANES);
      if (on[g] && i < i1 && sub == 0) {
        q[g * vs + i] = s[g];
        spq[g] += p[g * vs + i] * s[g];
      }
    }
  }
#pragma unroll
  for (int g = 0; g < G; g++) {
    if (!on[g]) continue;
    const double b = block_sum<kVecThreads>(spq[g], sh);
    if (threadIdx.x == 0) part_pq[(k0 + g) * nch + cc] = b;
  }
}

// x += alpha_k p; r -= alpha_k q; partial r.r; alpha as beta above.  A system
// with p.q <= 0 or NaN leaves the iteration.
__global__ void __launch_bounds__(kVecThreads)
bt_update(const int *cb, const int *csys, const int *sys_cptr,
          int *state, double *bsc, const double *part_pq,
          int *iters, const int *dit, const double *p,
          const double *q, double *x, double *r,
          double *part_rr) {
  __shared__ double sh[32];
  __shared__ double s_alpha;
  __shared__ bool s_on;
  pdl_trigger();
  pdl_wait();
  const int k = csys[blockIdx.x];
  if (threadIdx.x < 32) {
    double *sc = bsc + (size_t)k * BS_N;
    const double pq = bt_sum(part_pq, sys_cptr, k);
    if (threadIdx.x == 0) {
      // (the system's first CTA may set the state to BT_BREAKDOWN meanwhile:
      // then this one finds the same p.q)
      const bool on = __ldcg(state + k) == BT_ACTIVE;
      const double alpha = __ddiv_rn(__ldcg(sc + BS_RHO), pq);
      s_alpha = alpha;
      s_on = on && pq > 0.0;
      if (on && (int)blockIdx.x == sys_cptr[k]) {
        sc[BS_PQ] = pq;
        sc[BS_ALPHA] = alpha;
        if (!(pq > 0.0)) {
          state[k] = BT_BREAKDOWN;
          iters[k] = *dit + 1;
        }
      }
    }
  }
  __syncthreads();
  if (!s_on) {
    if (threadIdx.x == 0) part_rr[blockIdx.x] = 0.0;
    return;
  }
  const double alpha = s_alpha;
  const int i1 = cb[blockIdx.x + 1];
  double srr = 0.0;
  for (int i = cb[blockIdx.x] + threadIdx.x; i < i1; i += kVecThreads) {
    x[i] = __fma_rn(alpha, p[i], x[i]);
    const double ri = __fma_rn(-alpha, q[i], r[i]);
    r[i] = ri;
    srr += ri * ri;
  }
  double b = block_sum<kVecThreads>(srr, sh);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = b;
}

// r = b - A x on the chunks of the systems in state `want` (all when want < 0)
template <int LANES>
__global__ void __launch_bounds__(kVecThreads)
bt_residual(const int *__restrict__ cb, const int *__restrict__ csys, const int *__restrict__ state, int want,
            const int64_t *__restrict__ Ap, const int *__restrict__ Ac, const double *__restrict__ Av,
            const double *__restrict__ x, const double *__restrict__ b, double *__restrict__ r,
            double *__restrict__ part_rr, int64_t vs = 0) {
  __shared__ double sh[32];
  const int64_t voff = (int64_t)csys[blockIdx.x] * vs;
  const double *xc = x + voff;  // xc[c]: column c of this right-hand side
  if (want >= 0 && state[csys[blockIdx.x]] != want) {
    if (threadIdx.x == 0) part_rr[blockIdx.x] = 0.0;
    return;
  }
  const int sub = threadIdx.x % LANES;
  const int rows_per_block = kVecThreads / LANES;
  const int i1 = cb[blockIdx.x + 1];
  double srr = 0.0;
  for (int row0 = cb[blockIdx.x]; row0 < i1; row0 += rows_per_block) {
    const int i = row0 + threadIdx.x / LANES;
    double s = 0.0;
    if (i < i1)
      for (int64_t e = Ap[i - voff] + sub; e < Ap[i - voff + 1]; e += LANES) s = __fma_rn(Av[e], xc[Ac[e]], s);
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, LANES);
    if (i < i1 && sub == 0) {
      const double ri = __dsub_rn(b[i], s);
      r[i] = ri;
      srr += ri * ri;
    }
  }
  double t = block_sum<kVecThreads>(srr, sh);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = t;
}

// Per-system CG scalars from the chunk partials (one warp per system, chunks
// summed in a fixed order), the state machine and the counts the host reads.
// One CTA of 1024 threads.  dit: the device iteration counter (incremented by
// BT_FINISH), so that a captured graph needs no per-iteration argument.
__global__ void __launch_bounds__(1024)
bt_scalars(int nsys, const int *sys_cptr, int step, int mixed, double tol2,
           const double *part_rr, double *bsc,
           int *state, int *iters, int *dit,
           volatile int *host_counts) {
  __shared__ int cnt[3];
  pdl_wait();
  if (threadIdx.x < 3) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int it = __ldcg(dit) + (step == BT_FINISH ? 1 : 0);
  for (int k = wid; k < nsys; k += nw) {
    double *sc = bsc + (size_t)k * BS_N;
    const double a = bt_sum(part_rr, sys_cptr, k);
    int stt = __ldcg(state + k);
    if (lane == 0) {
      switch (step) {
        case BT_INIT:
          sc[BS_RES] = a;
          sc[BS_INIT] = a == 0.0 ? 1.0 : a;
          sc[BS_TRUE] = a;
          sc[BS_RHO_PREV] = 0.0;
          stt = BT_ACTIVE;
          iters[k] = 0;
          break;
        case BT_FINISH:
          if (stt == BT_ACTIVE) {
            sc[BS_RES] = a;
            sc[BS_RHO_PREV] = __ldcg(sc + BS_RHO);
            iters[k] = it;
            if (a != a) stt = BT_BREAKDOWN;
            else if (!(a / __ldcg(sc + BS_INIT) > tol2)) stt = mixed ? BT_CHECK : BT_DONE;
          }
          break;
        case BT_CONFIRM:  // the FP64 true residual decides; r now holds it
          if (stt == BT_CHECK) {
            sc[BS_RES] = a;
            stt = a / __ldcg(sc + BS_INIT) > tol2 ? BT_ACTIVE : BT_DONE;
          }
          break;
        default:  // BT_REPORT
          sc[BS_TRUE] = a;
          break;
      }
      state[k] = stt;
      if (stt == BT_ACTIVE) atomicAdd(&cnt[0], 1);
      else if (stt == BT_CHECK) atomicAdd(&cnt[1], 1);
      else if (stt == BT_BREAKDOWN) atomicAdd(&cnt[2], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (step == BT_FINISH) *dit = it;
    if (step == BT_INIT) *dit = 0;
    host_counts[0] = cnt[0];
    host_counts[1] = cnt[1];
    host_counts[2] = cnt[2];
  }
}

}  // namespace dg
