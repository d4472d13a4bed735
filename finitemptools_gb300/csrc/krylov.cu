// Krylov solvers on device-resident vectors: the reference's plain Lanczos
// for the lowest eigenpair and a Krylov exponential for TDVP.
//
// Vectors stay in HBM for the whole solve; only the small matrices and scalars
// that steer the host loop come back to the host (beta for the Lanczos stopping
// test; the Krylov exponential's Hessenberg matrix, whose small exponential and
// step-size control run on the host).  All reductions are deterministic
// two-level sums (warp shuffles inside a block, a fixed-order sum over the block
// partials, recomputed by every consumer block so that no separate
// finalisation launch is needed).
#include <algorithm>
#include <cmath>
#include <complex>
#include <mutex>
#include <vector>

#include "tc_planes.cuh"

namespace fmpt {
namespace {

constexpr int KT = 256;

// a kernel of KT threads per block, overlapping its launch with the kernel before it
#define CHAIN(kernel, grid, stream, ...) \
  FMPT_CUDA(h, launch_chain(kernel, grid, KT, 0, stream, __VA_ARGS__))

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Warp sums of K values at once (K a power of two <= 32).  GB300 issues an FP64 warp
// instruction at about 2 lanes per clock per SM, so the adds of a reduction cost more than
// the shuffles: plain xor-sums take 5 K adds per lane, this takes K - 1 + (5 - log2 K).
// Recursive halving: at each butterfly step (lane offsets 16, 8, ...) a lane keeps one half
// of its values, the partner lane the other half, and each adds the partner's copy of the
// half it keeps; then a plain xor-sum over the remaining lane bits.  a[0] ends up holding
// the warp sum of value (lane >> (5 - log2 K)); the order of the adds is fixed.
template <int K>
__device__ __forceinline__ void warp_sum_many(double (&a)[K]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int cnt = K; cnt > 1; cnt >>= 1, o >>= 1) {
    const int half = cnt >> 1;
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const double send = upper ? a[i] : a[i + half];
      const double keep = upper ? a[i + half] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
}

// Sum over the lanes and over the first nw <= 8 of 8 rows a[w] (rows past nw are exact zeros),
// by one warp: the rows' warp sums, then their sum in the order of a warp sum over lanes 0..7.
// The adds of rows that do not exist are left out (x + 0 = x).  All lanes get the result.
__device__ __forceinline__ double rows_sum(double (&a)[8], int nw) {
  if (nw <= 1) return warp_sum(a[0]);
  if (nw <= 2) {
    double b[2] = {a[0], a[1]};
    warp_sum_many<2>(b);
    return b[0] + __shfl_xor_sync(0xffffffffu, b[0], 16);
  }
  if (nw <= 4) {
    double b[4] = {a[0], a[1], a[2], a[3]};
    warp_sum_many<4>(b);
    b[0] += __shfl_xor_sync(0xffffffffu, b[0], 16);
    return b[0] + __shfl_xor_sync(0xffffffffu, b[0], 8);
  }
  warp_sum_many<8>(a);
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 16);
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 8);
  return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 4);
}

// Sum over the block, in warp order.  One warp adds all of it: the adds of eight warp sums
// (45 FP64 warp instructions of 64 to 77 cycles each) become 12, and with four blocks on an
// SM that is most of what the short vector kernels below do.
__device__ double block_sum(double v) {
  __shared__ double red[KT];
  __shared__ double total;
  red[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double a[8];
#pragma unroll
    for (int w = 0; w < 8; w++) a[w] = red[32 * w + threadIdx.x];
    const double t = rows_sum(a, 8);
    if (threadIdx.x == 0) total = t;
  }
  __syncthreads();
  const double r = total;
  __syncthreads();
  return r;
}

// Fixed-order sum of G partials, or its square root (every block computes the same value): by
// one warp, with the sums of 256 threads striding over the partials.
__device__ double sum_parts(const double* part, int G, bool root = false) {
  __shared__ double total;
  if (threadIdx.x < 32) {
    const int nw = G >= KT ? 8 : (G + 31) / 32;
    double a[8];
#pragma unroll
    for (int w = 0; w < 8; w++) {
      const int i = 32 * w + (int)threadIdx.x;
      a[w] = i < G ? part[i] : 0.0;
    }
    for (int k = KT; k < G; k += KT) {
      double b[8];
#pragma unroll
      for (int w = 0; w < 8; w++) {
        const int i = k + 32 * w + (int)threadIdx.x;
        b[w] = i < G ? part[i] : 0.0;
      }
#pragma unroll
      for (int w = 0; w < 8; w++)
        if (k + 32 * w < G) a[w] += b[w];
    }
    double t = rows_sum(a, nw);
    if (root) t = sqrt(t);
    if (threadIdx.x == 0) total = t;
  }
  __syncthreads();
  const double r = total;
  __syncthreads();
  return r;
}

// part[b] = sum x*y over a grid-stride slice (real view of length n)
__global__ void rdot_partial(int64_t n, const double* __restrict__ x, const double* __restrict__ y,
                             double* __restrict__ part, const int* gate = nullptr) {
  chain_begin();
  if (gate && *gate) return;
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
    s = fma(x[i], y[i], s);
  s = block_sum(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// x = v / ||v|| with ||v||^2 = sum(part); stores the norm in *nrm
__global__ void normalize_from_parts(int64_t n, const double* __restrict__ v, double* __restrict__ x,
                                     const double* __restrict__ part, int G, double* nrm) {
  chain_begin();
  const double s = sum_parts(part, G, true);
  if (blockIdx.x == 0 && threadIdx.x == 0) *nrm = s;
  double inv = s > 0.0 ? 1.0 / s : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
    x[i] = v[i] * inv;
}

// a = sum(part_a); alpha_out = a; y -= (q*a + qm1*b_old); part_b = partial |y|^2
__global__ void lanczos_axpy(int64_t n, double* __restrict__ y, const double* __restrict__ q,
                             const double* __restrict__ qm1, const double* __restrict__ part_a,
                             int G, const double* b_old, double* alpha_out,
                             double* __restrict__ part_b, const int* gate = nullptr) {
  chain_begin();
  if (gate && *gate) return;
  const double a = sum_parts(part_a, G);
  const double b = (qm1 != nullptr) ? *b_old : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) *alpha_out = a;
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT) {
    double t = q[i] * a;
    if (qm1) t += qm1[i] * b;
    double v = y[i] - t;
    y[i] = v;
    s = fma(v, v, s);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) part_b[blockIdx.x] = s;
}

// b = sqrt(sum(part_b)); beta_out = b; vnext = y / b (y itself if b is 0); alpha and b also
// go to pinned host memory, ab[0] and ab[1], and stop (if given) is raised where the host's test
// of b ends the solve.  MODE >= 0: vnext also goes, rounded, to the operand
// planes of the tensor-core operator that is applied to it next, which saves that operator's
// conversion pass (5.7 us of a step at D = 256).
template <int MODE>
__global__ void lanczos_scale(int64_t n, const double* __restrict__ y,
                              const double* __restrict__ part_b, int G, const double* alpha,
                              double* beta_out, double* __restrict__ vnext, double* ab,
                              double btol, int* stop, void* hi, void* lo) {
  chain_begin();
  const double b = sum_parts(part_b, G, true);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *beta_out = b;
    ab[0] = *alpha;
    ab[1] = b;
    if (stop && (!(b >= btol) || isinf(b))) *stop = 1;
  }
  // Julia's qi /= b divides element-wise; so does this (no reciprocal).  b >= 0 or NaN; the test
  // is on its words, an FP64 comparison otherwise.
  const bool zero = (__double2hiint(b) | __double2loint(b)) == 0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT) {
    const double v = zero ? y[i] : y[i] / b;
    vnext[i] = v;
    if constexpr (MODE >= 0) put<MODE>(hi, lo, i, v);
  }
}

// ---- multi-vector kernels over the Krylov basis V (j vectors of length n,
// complex split planes when cplx: V_i re at V + i*2n, im at V + i*2n + n)
// partial dots h_i = <V_i, z> ; part layout [j][2][G].  Chunks of MD_CH vectors per pass
// over z: every thread keeps MD_CH running sums (re, im), reduced by warp shuffles; the warps'
// sums meet in shared memory once per MD_MAX vectors (a pass and two barriers per chunk kept
// the block from loading the next chunk: 22 us at n = 262144 and 10 vectors, now 17).  Fixed
// summation order throughout (deterministic).
constexpr int MD_CH = 8, MD_MAX = 64;         // vectors per chunk, per pass over shared memory
template <bool CPLX>
__global__ void __launch_bounds__(KT, CPLX ? 2 : 4) multidot_partial(int64_t n, int j,
                                                       const double* __restrict__ V,
                                                       int64_t vstride,
                                                       const double* __restrict__ z,
                                                       double* __restrict__ part,
                                                       const int* gate = nullptr) {
  chain_begin();
  if (gate && *gate) return;
  __shared__ double red[KT / 32][(CPLX ? 2 : 1) * MD_MAX];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int g0 = 0; g0 < j; g0 += MD_MAX) {
    const int g1 = min(j, g0 + MD_MAX);
    for (int i0 = g0; i0 < g1; i0 += MD_CH) {
      double sr[MD_CH], si[MD_CH];
#pragma unroll
      for (int c = 0; c < MD_CH; c++) {
        sr[c] = 0.0;
        si[c] = 0.0;
      }
      for (int64_t e = (int64_t)blockIdx.x * KT + threadIdx.x; e < n; e += (int64_t)gridDim.x * KT) {
        const double zr = z[e], zi = CPLX ? z[n + e] : 0.0;
        double vr[MD_CH], vi[MD_CH];
#pragma unroll
        for (int c = 0; c < MD_CH; c++) {
          const double* v = V + (int64_t)(i0 + c) * vstride;
          vr[c] = i0 + c < g1 ? v[e] : 0.0;
          vi[c] = CPLX && i0 + c < g1 ? v[n + e] : 0.0;
        }
#pragma unroll
        for (int c = 0; c < MD_CH; c++) {
          if (i0 + c < g1) {
            sr[c] = fma(vr[c], zr, sr[c]);
            if constexpr (CPLX) {
              sr[c] = fma(vi[c], zi, sr[c]);
              si[c] = fma(vr[c], zi, si[c]);
              si[c] = fma(-vi[c], zr, si[c]);
            }
          }
        }
      }
      if constexpr (CPLX) {
        double v[2 * MD_CH];
#pragma unroll
        for (int c = 0; c < MD_CH; c++) {
          v[2 * c] = sr[c];
          v[2 * c + 1] = si[c];
        }
        warp_sum_many<2 * MD_CH>(v);
        if ((lane & 1) == 0) red[wid][2 * (i0 - g0) + (lane >> 1)] = v[0];      // 2 MD_CH = 16 values
      } else if (g1 - i0 > 2) {
        warp_sum_many<MD_CH>(sr);                             // no imaginary parts to add
        if ((lane & 3) == 0) red[wid][i0 - g0 + (lane >> 2)] = sr[0];
      } else {                                                // fewer values, the same order
        double v[2] = {sr[0], sr[1]};
        warp_sum_many<2>(v);
        if ((lane & 15) == 0) red[wid][i0 - g0 + (lane >> 4)] = v[0];
      }
    }
    __syncthreads();
    const int nv = (g1 - g0) * (CPLX ? 2 : 1);
    const int t = threadIdx.x;
    if (t < nv) {
      double s = 0.0;
      for (int w = 0; w < KT / 32; w++) s += red[w][t];
      double* p = part + (2 * (int64_t)g0 + (CPLX ? t : 2 * t)) * gridDim.x + blockIdx.x;
      *p = s;
      if (!CPLX) p[gridDim.x] = 0.0;
    }
    __syncthreads();                                        // red is written again
  }
}

// coef[t] (t = 2 i + re/im) = the sum over the G partials [2 j][G] (accum[t] += it when
// given): one warp per value, a lane adds its partials g = lane, lane + 32, .. in order, then
// the warp sums; real data has no odd values.  Launched with (2 j + 7) / 8 blocks: one block
// for all values took 12 us at G = 608, 20 partials per lane one after the other on one SM.
__global__ void multidot_finalize(int cplx, int j, int G, const double* __restrict__ part,
                                  double* __restrict__ coef, double* __restrict__ accum,
                                  const int* gate = nullptr) {
  chain_begin();
  if (gate && *gate) return;
  const int t = blockIdx.x * (KT / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= 2 * j) return;
  double s = 0.0;
  if (cplx || !(t & 1)) {
    for (int g0 = 0; g0 < G; g0 += 32 * 8) {
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int g = g0 + 32 * q + lane;
        v[q] = g < G ? part[(int64_t)t * G + g] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (g0 + 32 * q < G) s += v[q];
    }
    s = warp_sum(s);
  }
  if (lane == 0) {
    coef[t] = s;
    if (accum) accum[t] += s;
  }
}

__global__ void multi_axpy_sub(int cplx, int64_t n, int j, const double* __restrict__ V,
                               int64_t vstride, const double* __restrict__ coef,
                               double* __restrict__ z, double* __restrict__ part,
                               const int* gate = nullptr) {
  chain_begin();
  if (gate && *gate) return;
  double s = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * KT + threadIdx.x; e < n; e += (int64_t)gridDim.x * KT) {
    double zr = z[e], zi = cplx ? z[n + e] : 0.0;
    // MD_CH vectors' elements are loaded together (their L2 latencies overlap), then
    // subtracted in vector order
    for (int i0 = 0; i0 < j; i0 += MD_CH) {
      double vr[MD_CH], vi[MD_CH];
#pragma unroll
      for (int c = 0; c < MD_CH; c++) {
        vr[c] = 0.0;
        vi[c] = 0.0;
        if (i0 + c < j) {
          const double* v = V + (int64_t)(i0 + c) * vstride;
          vr[c] = v[e];
          if (cplx) vi[c] = v[n + e];
        }
      }
#pragma unroll
      for (int c = 0; c < MD_CH; c++) {
        if (i0 + c < j) {
          const double cr = coef[2 * (i0 + c)], ci = coef[2 * (i0 + c) + 1];
          if (cplx) {
            zr -= cr * vr[c] - ci * vi[c];
            zi -= cr * vi[c] + ci * vr[c];
          } else {
            zr -= cr * vr[c];
          }
        }
      }
    }
    z[e] = zr;
    if (cplx) z[n + e] = zi;
    s = fma(zr, zr, s);
    if (cplx) s = fma(zi, zi, s);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out_q = scale sum_i c_qi V_i for q = blockIdx.y (coefficients (re, im) pairs, cq = their
// stride per q; scale a device scalar, or 1).  Eight vectors' elements are loaded together:
// one at a time the sum is a chain of L2 latencies (21 us at 30 vectors, now 5).
__global__ void combine_basis(int cplx, int64_t n, int j, const double* __restrict__ V,
                              int64_t vstride, const double* __restrict__ c, int64_t cq,
                              const double* scale, double* __restrict__ out, int64_t oq) {
  chain_begin();
  constexpr int U = 8;
  c += blockIdx.y * cq;
  out += blockIdx.y * oq;
  const double f = scale ? *scale : 1.0;
  for (int64_t e = (int64_t)blockIdx.x * KT + threadIdx.x; e < n; e += (int64_t)gridDim.x * KT) {
    double r = 0.0, im = 0.0;
    for (int i0 = 0; i0 < j; i0 += U) {
      double vr[U], vi[U], cr[U], ci[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const bool in = i0 + u < j;
        const double* v = V + (int64_t)(i0 + u) * vstride;
        vr[u] = in ? v[e] : 0.0;
        vi[u] = in && cplx ? v[n + e] : 0.0;
        cr[u] = in ? c[2 * (i0 + u)] : 0.0;
        ci[u] = in && cplx ? c[2 * (i0 + u) + 1] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (i0 + u >= j) break;
        r = fma(cr[u], vr[u], r);
        if (cplx) {
          r = fma(-ci[u], vi[u], r);
          im = fma(cr[u], vi[u], im);
          im = fma(ci[u], vr[u], im);
        }
      }
    }
    out[e] = r * f;
    if (cplx) out[n + e] = im * f;
  }
}

// ---- orthogonalisation step of one Arnoldi vector: two Gram-Schmidt passes of z against
// V_0..V_j and the normalisation V_{j+1} = z / s.
//
// On GB300 an FP64 warp instruction occupies its SM sub-partition for about 60 cycles and a
// dependent one waits about 200, so the step is bound by its chains of dependent FP64
// instructions and by its grid-wide waits, not by the loads.  Hence
// - a warp's unit is a chunk of 32 elements of ONE component (real or imaginary plane): two
//   multiply-adds per lane and vector instead of four, twice as many warps at work;
// - a block of 8 working warps holds cpb chunks (1, 2, 4 or 8), and 8 / cpb warps share a
//   chunk, each taking every (8 / cpb)-th vector;
// - sums run as independent chains or trees, over the values that exist;
// - |z|^2 is one more value of each pass's dots: s^2 = |z|^2 - sum |c2|^2 after the second
//   (c2 is of rounding size), which saves a third grid-wide wait;
// - s and 1 / s are found by a ninth warp while the others form sum c_i V_i.
// One step at n = 8192 complex, 16 vectors (D = 64, 128 blocks of 4 chunks): 26 us, half of it
// the FP64 pipe, 1.4 us in each grid-wide wait; the form it replaces (both components of an
// element per thread, a plain warp sum per block, three waits) took 38 us, and 45 on any
// small vector, now about 15.
constexpr int GS_T = 288;                      // 8 working warps and the closing one
constexpr int GS_NV = 64;                      // values per pass: (re, im) per vector, |z|^2
struct GsArgs {
  int cplx, j;                                 // orthogonalise against V_0..V_j
  int64_t n;                                   // elements (complex ones if cplx)
  int cpb;                                     // chunks per block: 1, 2, 4, 8
  const double* V;
  int64_t vstride;
  double* z;
  double* part;                                // [2][GS_NV][G] block sums
  double* Hcol;
  double* vnext;
};

struct GsWarp {
  int lane, wid, cs, vg, VG;
  int64_t nch, S, step;
  __device__ GsWarp(const GsArgs& a) {
    lane = threadIdx.x & 31;
    wid = threadIdx.x >> 5;
    cs = wid % a.cpb;
    vg = wid / a.cpb;
    VG = 8 / a.cpb;
    nch = (a.n + 31) / 32;
    S = a.cplx ? 2 * nch : nch;
    step = (int64_t)gridDim.x * a.cpb;
  }
  // this warp's first chunk
  __device__ int64_t first(const GsArgs& a) const { return (int64_t)blockIdx.x * a.cpb + cs; }
  __device__ void locate(const GsArgs& a, int64_t ch, int& comp, int64_t& e, bool& in) const {
    comp = ch >= nch ? 1 : 0;
    e = (ch - (comp ? nch : 0)) * 32 + lane;
    in = ch < S && e < a.n;
  }
};

// r[0] + r[stride] + .. (n = 1, 2, 4, 8 terms) as a tree
__device__ __forceinline__ double gs_tree(const double* r, int stride, int n) {
  double x[8];
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = k < n ? r[k * stride] : 0.0;
  if (n == 1) return x[0];
  x[0] += x[1];
  if (n == 2) return x[0];
  x[2] += x[3];
  x[0] += x[2];
  if (n == 4) return x[0];
  x[4] += x[5];
  x[6] += x[7];
  x[4] += x[6];
  return x[0] + x[4];
}

// Block sums bp[2 i], bp[2 i + 1] of conj(V_i) z over the block's chunks, bp[2 j + 2] of
// |z|^2 (the dot with z itself, i = j + 1).  SINGLE: every warp has one chunk, zv is this
// lane's element; otherwise the warps loop over chunks and read a.z.
template <bool SINGLE>
__device__ void gs_dots(const GsArgs& a, const GsWarp& w, double zv, double* bp) {
  __shared__ double red[8][GS_NV];
  constexpr int U = 8;
  const int nvec = a.j + 2;
  for (int i0 = w.vg; i0 < nvec && w.wid < 8; i0 += U * w.VG) {
    double v[2 * U];
#pragma unroll
    for (int u = 0; u < 2 * U; u++) v[u] = 0.0;
    for (int64_t ch = w.first(a); ch < w.S; ch += w.step) {
      int comp;
      int64_t e;
      bool in;
      w.locate(a, ch, comp, e, in);
      const double z = SINGLE ? zv : (in ? a.z[comp * a.n + e] : 0.0);
      double vs[U], vo[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int i = i0 + u * w.VG;
        const double* p = a.V + (int64_t)i * a.vstride;
        vs[u] = in && i <= a.j ? p[comp * a.n + e] : (i == a.j + 1 ? z : 0.0);
        vo[u] = in && i <= a.j && a.cplx ? p[(1 - comp) * a.n + e] : 0.0;
      }
      // Re: vr zr + vi zi; Im: vr zi - vi zr
      const double zo = comp ? z : -z;
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (i0 + u * w.VG < nvec) {
          v[2 * u] = fma(vs[u], z, v[2 * u]);
          if (a.cplx) v[2 * u + 1] = fma(vo[u], zo, v[2 * u + 1]);
        }
      }
    }
    // few vectors: fewer values to sum
    const int left = (nvec - i0 + w.VG - 1) / w.VG;
    if (left > 4) {
      warp_sum_many<16>(v);
    } else if (left > 1) {
      double v8[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v8[u] = v[u];
      warp_sum_many<8>(v8);
      v[0] = v8[0];
    } else {
      double v2[2] = {v[0], v[1]};
      warp_sum_many<2>(v2);
      v[0] = v2[0];
    }
    const int sh = left > 4 ? 1 : (left > 1 ? 2 : 4);
    const int q = w.lane >> sh;                // value index: 2 u + component
    const int i = i0 + (q >> 1) * w.VG;
    if ((w.lane & ((1 << sh) - 1)) == 0 && i < nvec) red[w.cs][2 * i + (q & 1)] = v[0];
  }
  __syncthreads();
  if ((int)threadIdx.x < 2 * nvec - 1) bp[threadIdx.x] = gs_tree(&red[0][threadIdx.x], GS_NV, a.cpb);
  __syncthreads();
}

template <int K>
__device__ __forceinline__ void gs_total_k(const double* part, int G, int nv, double* c) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double x[K][4];
#pragma unroll
  for (int u = 0; u < K; u++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int t = wid + 8 * u, g = lane + 32 * q;
      x[u][q] = t < nv && g < G ? __ldcg(part + (int64_t)t * G + g) : 0.0;
    }
  double v[K];
#pragma unroll
  for (int u = 0; u < K; u++) v[u] = x[u][0];
  if (G > 32) {
#pragma unroll
    for (int u = 0; u < K; u++) v[u] += x[u][1];
  }
  if (G > 64) {
#pragma unroll
    for (int u = 0; u < K; u++) x[u][2] += x[u][3];
#pragma unroll
    for (int u = 0; u < K; u++) v[u] += x[u][2];
  }
  warp_sum_many<K>(v);
  constexpr int sh = K == 8 ? 2 : (K == 4 ? 3 : (K == 2 ? 4 : 5));
  const int t = wid + 8 * (lane >> sh);
  if ((lane & ((1 << sh) - 1)) == 0 && t < nv) c[t] = v[0];
}

// sums over the G <= 128 blocks: c[t] for t < nv; warp w < 8 takes t = w + 8 u
__device__ __forceinline__ void gs_total(const double* part, int G, int nv, double* c) {
  const int wid = threadIdx.x >> 5;
  const int mine = wid < 8 ? (nv - wid + 7) / 8 : 0;
  if (mine > 4) gs_total_k<8>(part, G, nv, c);
  else if (mine > 2) gs_total_k<4>(part, G, nv, c);
  else if (mine > 1) gs_total_k<2>(part, G, nv, c);
  else if (mine == 1) gs_total_k<1>(part, G, nv, c);
}

// sum over the vectors of this warp of -c_i V_i at its element of one component
__device__ __forceinline__ double gs_correction(const GsArgs& a, const GsWarp& w, const double* c,
                                                int comp, int64_t e, bool in) {
  constexpr int U = 8;
  const int jj = a.j + 1;
  double p[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i0 = w.vg; i0 < jj; i0 += U * w.VG) {
    double vs[U], vo[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * w.VG;
      const double* q = a.V + (int64_t)i * a.vstride;
      vs[u] = in && i < jj ? q[comp * a.n + e] : 0.0;
      vo[u] = in && i < jj && a.cplx ? q[(1 - comp) * a.n + e] : 0.0;
    }
    // Re: - (cr vr - ci vi); Im: - (cr vi + ci vr)
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * w.VG;
      if (i < jj) {
        p[u & 1] = fma(-c[2 * i], vs[u], p[u & 1]);
        if (a.cplx) p[2 + (u & 1)] = fma(comp ? -c[2 * i + 1] : c[2 * i + 1], vo[u], p[2 + (u & 1)]);
      }
    }
  }
  if (!a.cplx) return p[0] + p[1];
  return (p[0] + p[1]) + (p[2] + p[3]);
}

// The step's closure by one warp: hc = c1 + c2 into H's column, s from the second pass's
// |z|^2.  If s is below 1e-12 of the norm before the step the Krylov space is exhausted
// (happy breakdown) and V_{j+1}, H[j+1][j] are zero.  Returns 1 / s or 0.
__device__ double gs_close(const GsArgs& a, const double* c1, const double* c2, bool write) {
  const int lane = threadIdx.x & 31, jj = a.j + 1;
  double q2 = 0.0;
  for (int t = lane; t < 2 * jj; t += 32) {
    q2 = fma(c2[t], c2[t], q2);
    if (write) a.Hcol[t] = c1[t] + c2[t];
  }
  q2 = warp_sum(q2);
  const double d = c2[2 * jj] - q2;
  const double s2 = d < 0.0 ? 0.0 : d;                         // NaN stays
  const bool breakdown = s2 <= 1e-24 * c1[2 * jj];
  const double s = sqrt(s2);
  if (write && lane == 0) {
    a.Hcol[2 * jj] = breakdown ? 0.0 : s;
    a.Hcol[2 * jj + 1] = 0.0;
  }
  return breakdown ? 0.0 : 1.0 / s;
}

// z - sum c_i V_i: SINGLE returns this lane's new element (the same in all warps of a
// chunk), otherwise z is updated in place.  After the second pass (last) the result is
// scaled by 1 / s and goes to V_{j+1}; close() runs on the ninth warp meanwhile and returns
// 1 / s.
template <bool SINGLE, class Close>
__device__ double gs_axpy(const GsArgs& a, const GsWarp& w, const double* c, double zv, bool last,
                          Close close) {
  __shared__ double ps[8][32], s_inv;
  int comp = 0;
  int64_t e = 0;
  bool in = false;
  if (w.wid == 8) {
    if (last) {
      const double inv = close();
      if (w.lane == 0) s_inv = inv;
    }
  } else if (SINGLE) {
    w.locate(a, w.first(a), comp, e, in);
    ps[w.wid][w.lane] = gs_correction(a, w, c, comp, e, in);
  }
  __syncthreads();
  const double inv = last ? s_inv : 1.0;
  if (w.wid == 8) return 0.0;
  if constexpr (SINGLE) {
    zv += gs_tree(&ps[w.cs][w.lane], 32 * a.cpb, w.VG);
    if (last) zv *= inv;
    if (last && w.vg == 0 && in) a.vnext[comp * a.n + e] = zv;
    return zv;
  } else {
    for (int64_t ch = w.first(a); ch < w.S; ch += w.step) {    // cpb = 8: VG = 1
      w.locate(a, ch, comp, e, in);
      const double p = gs_correction(a, w, c, comp, e, in);
      if (in) {
        const double z = a.z[comp * a.n + e] + p;
        if (last) a.vnext[comp * a.n + e] = z * inv;
        else a.z[comp * a.n + e] = z;
      }
    }
    return 0.0;
  }
}

// this lane's element when every warp has one chunk
__device__ __forceinline__ double gs_load(const GsArgs& a, const GsWarp& w) {
  int comp;
  int64_t e;
  bool in;
  w.locate(a, w.first(a), comp, e, in);
  return in && w.wid < 8 ? a.z[comp * a.n + e] : 0.0;
}

// ---- the step as ONE cooperative launch.  Its grid-wide waits are bounded (2 s on
// %globaltimer): a timeout sets the abort flag and the handle's status word and every block
// returns.  The arrival counter runs on from step to step (target; zeroed once per basis).
struct CoopBar {
  int* count;        // arrivals
  int* abort_flag;
  int* status;       // handle status word
  uint64_t wait_ns;
  int hold;          // arrivals waited for beyond the grid: 0, or 1 only to test the bound
};

__device__ __forceinline__ int ld_acquire_i(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ uint64_t now_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Every block has written its sums.  False: given up.  The block barriers order the block's
// writes before its release and its reads after the acquire (cumulativity); the readers go
// to L2 (__ldcg).
__device__ bool gs_grid_wait(const CoopBar& b, int target) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(b.count) : "memory");
    int ok = 1;
    const uint64_t t0 = now_ns();
    // the count alone is polled; every 32nd poll also looks at the abort flag, the status
    // word (this launch gave up, or an earlier one of the same solve did: the word stays
    // set until the host reads it) and the clock
    for (unsigned polls = 1; ld_acquire_i(b.count) < target + b.hold; polls++) {
      if ((polls & 31u) != 0) continue;
      if (ld_acquire_i(b.abort_flag) || ld_acquire_i(b.status)) { ok = 0; break; }
      if (now_ns() - t0 > b.wait_ns) {
        atomicExch(b.abort_flag, 1);
        atomicExch(b.status, 1);
        ok = 0;
        break;
      }
    }
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

template <bool SINGLE>
__global__ void __launch_bounds__(GS_T) arnoldi_gs_fused(GsArgs a, CoopBar bar) {
  chain_begin();
  __shared__ double bp[GS_NV], c[2][GS_NV];
  const GsWarp w(a);
  const int G = gridDim.x, nv = 2 * a.j + 3;
  double zv = SINGLE ? gs_load(a, w) : 0.0;
  for (int pass = 0; pass < 2; pass++) {
    double* part = a.part + (int64_t)pass * GS_NV * G;
    if (G == 1) {
      gs_dots<SINGLE>(a, w, zv, c[pass]);
    } else {
      gs_dots<SINGLE>(a, w, zv, bp);
      if ((int)threadIdx.x < nv) part[(int64_t)threadIdx.x * G + blockIdx.x] = bp[threadIdx.x];
      if (!gs_grid_wait(bar, (2 * a.j + pass + 1) * G)) return;
      gs_total(part, G, nv, c[pass]);
      __syncthreads();
    }
    zv = gs_axpy<SINGLE>(a, w, c[pass], zv, pass == 1,
                         [&]() { return gs_close(a, c[0], c[1], blockIdx.x == 0); });
  }
}

// The step of a short vector (gs_geometry) as one block or one cluster: the blocks meet at the
// cluster's hardware barrier, and as the launch is not a cooperative one it overlaps the kernel
// before it.  The same device functions on the same grid, so the same sums.
__global__ void __launch_bounds__(GS_T) arnoldi_gs_cluster(GsArgs a) {
  chain_begin();
  __shared__ double bp[GS_NV], c[2][GS_NV];
  const GsWarp w(a);
  const int G = gridDim.x, nv = 2 * a.j + 3;
  double zv = gs_load(a, w);
  for (int pass = 0; pass < 2; pass++) {
    double* part = a.part + (int64_t)pass * GS_NV * G;
    if (G == 1) {
      gs_dots<true>(a, w, zv, c[pass]);
    } else {
      gs_dots<true>(a, w, zv, bp);
      if ((int)threadIdx.x < nv) part[(int64_t)threadIdx.x * G + blockIdx.x] = bp[threadIdx.x];
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
      gs_total(part, G, nv, c[pass]);
      __syncthreads();
    }
    zv = gs_axpy<true>(a, w, c[pass], zv, pass == 1,
                       [&]() { return gs_close(a, c[0], c[1], blockIdx.x == 0); });
  }
}

// ---- the same step as six launches (fmpt_set_fused_krylov off): the same device functions
// on the same grid, so the same sums
template <bool SINGLE>
__global__ void __launch_bounds__(GS_T) arnoldi_gs_dots(GsArgs a, int pass) {
  __shared__ double bp[GS_NV];
  const GsWarp w(a);
  gs_dots<SINGLE>(a, w, SINGLE ? gs_load(a, w) : 0.0, bp);
  double* part = a.part + (int64_t)pass * GS_NV * gridDim.x;
  if ((int)threadIdx.x < 2 * a.j + 3)
    part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = bp[threadIdx.x];
}

// one block: totals c[pass], after the second pass also H's column and 1 / s
__global__ void __launch_bounds__(GS_T) arnoldi_gs_sums(GsArgs a, int pass, int G, double* coef) {
  __shared__ double c[2][GS_NV];
  const int nv = 2 * a.j + 3;
  gs_total(a.part + (int64_t)pass * GS_NV * G, G, nv, c[1]);
  __syncthreads();
  for (int t = threadIdx.x; t < nv; t += GS_T) {
    coef[pass * GS_NV + t] = c[1][t];
    c[0][t] = coef[t];
  }
  __syncthreads();
  if (pass == 1 && threadIdx.x < 32) {
    const double inv = gs_close(a, c[0], c[1], true);
    if (threadIdx.x == 0) coef[2 * GS_NV] = inv;
  }
}

template <bool SINGLE>
__global__ void __launch_bounds__(GS_T) arnoldi_gs_axpy(GsArgs a, int pass, const double* coef) {
  const GsWarp w(a);
  const double zv = gs_axpy<SINGLE>(a, w, coef + pass * GS_NV, SINGLE ? gs_load(a, w) : 0.0,
                                    pass == 1, [&]() { return coef[2 * GS_NV]; });
  if (SINGLE && pass == 0 && w.wid < 8 && w.vg == 0) {
    int comp;
    int64_t e;
    bool in;
    w.locate(a, w.first(a), comp, e, in);
    if (in) a.z[comp * a.n + e] = zv;
  }
}

// acc *= v (device scalars)
__global__ void mul_scalar(double* acc, const double* v) { *acc *= *v; }

// x *= *a (device scalar)
__global__ void scale_by(int64_t n, double* __restrict__ x, const double* a) {
  chain_begin();
  const double f = *a;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    x[e] *= f;
}

// Lowest eigenpair of the symmetric tridiagonal (alpha[0..k-1], beta[0..k-2])
// by Sturm-sequence bisection and inverse iteration with a partially pivoted
// tridiagonal solve (the LAPACK dgtsv elimination), k <= 128, on the host: about 1400
// dependent FP64 divisions at k = 20, which one GPU thread ran in 640 us (a quarter of a
// D = 64 solve) and a host core runs in about 10, while alpha and beta are on the host for
// the stopping test anyway.  The multiply-adds are fused explicitly, as the device compiler
// fuses them: the eigenvector's sign hangs on the last bit of the eigenvalue, so another
// rounding would flip it.
void tridiag_lowest(int k, const double* alpha, const double* beta, double* eval_out,
                    double* evec_out) {
  double lo = alpha[0], hi = alpha[0];
  for (int i = 0; i < k; i++) {
    double r = (i > 0 ? std::fabs(beta[i - 1]) : 0.0) + (i < k - 1 ? std::fabs(beta[i]) : 0.0);
    lo = std::fmin(lo, alpha[i] - r);
    hi = std::fmax(hi, alpha[i] + r);
  }
  const double tiny = 1e-300;
  for (int it = 0; it < 200; it++) {
    double mid = 0.5 * (lo + hi);
    if (mid <= lo || mid >= hi) break;
    int cnt = 0;
    double q = alpha[0] - mid;
    if (q < 0) cnt++;
    for (int i = 1; i < k; i++) {
      if (q == 0.0) q = tiny;
      q = (alpha[i] - mid) - beta[i - 1] * beta[i - 1] / q;
      if (q < 0) cnt++;
    }
    if (cnt >= 1) hi = mid; else lo = mid;
  }
  const double lam = 0.5 * (lo + hi);
  *eval_out = lam;
  if (k == 1) { evec_out[0] = 1.0; return; }
  double dl[128], dd[128], du[128], du2[128], x[128];
  for (int i = 0; i < k; i++) x[i] = 1.0 / std::sqrt((double)k) * std::fma(0.01, (double)i, 1.0);
  // a zero pivot is replaced by eps*|T| (the LAPACK dlagts perturbation idea)
  const double pert = 2.2e-16 * (std::fmax(std::fabs(lo), std::fabs(hi)) + 1e-300);
  for (int iter = 0; iter < 3; iter++) {
    for (int i = 0; i < k; i++) {
      dd[i] = alpha[i] - lam;
      if (i < k - 1) { dl[i] = beta[i]; du[i] = beta[i]; }
      du2[i] = 0.0;
    }
    // forward elimination with row interchanges
    for (int i = 0; i < k - 1; i++) {
      if (std::fabs(dd[i]) >= std::fabs(dl[i])) {
        if (dd[i] == 0.0) dd[i] = pert;
        double f = dl[i] / dd[i];
        dd[i + 1] = std::fma(-f, du[i], dd[i + 1]);
        x[i + 1] = std::fma(-f, x[i], x[i + 1]);
        dl[i] = 0.0;
      } else {
        double f = dd[i] / dl[i];
        dd[i] = dl[i];
        double t = dd[i + 1];
        dd[i + 1] = std::fma(-f, t, du[i]);
        if (i < k - 2) {
          du2[i] = du[i + 1];
          du[i + 1] = -f * du2[i];
        }
        du[i] = t;
        double xt = x[i];
        x[i] = x[i + 1];
        x[i + 1] = std::fma(-f, x[i + 1], xt);
      }
    }
    if (dd[k - 1] == 0.0) dd[k - 1] = pert;
    // back substitution
    x[k - 1] = x[k - 1] / dd[k - 1];
    x[k - 2] = std::fma(-du[k - 2], x[k - 1], x[k - 2]) / dd[k - 2];
    for (int i = k - 3; i >= 0; i--)
      x[i] = std::fma(-du2[i], x[i + 2], std::fma(-du[i], x[i + 1], x[i])) / dd[i];
    // normalise without overflow: scale by the largest entry first
    double mx = 0.0;
    for (int i = 0; i < k; i++) mx = std::fmax(mx, std::fabs(x[i]));
    if (!(mx > 0.0) || !std::isfinite(mx)) { for (int i = 0; i < k; i++) x[i] = (i == 0); mx = 1.0; }
    double nrm = 0.0;
    for (int i = 0; i < k; i++) { x[i] /= mx; nrm = std::fma(x[i], x[i], nrm); }
    nrm = std::sqrt(nrm);
    for (int i = 0; i < k; i++) x[i] /= nrm;
  }
  for (int i = 0; i < k; i++) evec_out[i] = x[i];
}

// Ritz coefficients by value
struct RitzCoef {
  double c[128];
};

// out = sum_i c_i V_i in the order of lanczos_linear_transformation_single
// (simple_lanczos.jl:70-78), which adds the last basis vector first
__global__ void combine_ritz(int64_t n, int k, const double* __restrict__ V, int64_t vstride,
                             const __grid_constant__ RitzCoef c, double* __restrict__ out) {
  chain_begin();
  for (int64_t e = (int64_t)blockIdx.x * KT + threadIdx.x; e < n; e += (int64_t)gridDim.x * KT) {
    double r = c.c[k - 1] * V[(int64_t)(k - 1) * vstride + e];
    for (int i = 0; i < k - 1; i++) r = fma(c.c[i], V[(int64_t)i * vstride + e], r);
    out[e] = r;
  }
}

// Graph-driven Lanczos step closure.  ctl: [0] stop (converged or failed),
// [1] Krylov dimension k, [2] beta was not finite, [3] converged (beta < btol).
// Step j has produced alpha_j and the partial norms of the new residual y:
// beta_j = ||y||; k = j + 1; stop when beta_j < btol (or is not finite),
// otherwise V_{j+1} = y / beta_j.
__global__ void lanczos_close(int64_t n, const double* __restrict__ y,
                              const double* __restrict__ part_b, int G, double* beta_out,
                              int* ctl, double btol, int j, double* __restrict__ vnext) {
  chain_begin();
  if (ctl[0]) return;
  const double b = sum_parts(part_b, G, true);
  const bool bad = !isfinite(b);
  const bool conv = !bad && b < btol;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *beta_out = b;
    ctl[1] = j + 1;
    if (bad) ctl[2] = 1;
    if (conv) ctl[3] = 1;
    if (bad || conv) ctl[0] = 1;
  }
  if (bad || conv) return;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT)
    vnext[i] = y[i] / b;
}

// exp(A) e_1 for the small complex matrix A = t * H_m of a Krylov exponential (m <= 31,
// column-major (re, im) pairs), on the host: the m x m problem is a few hundred thousand
// flops, which a host core runs in tens of microseconds while one SM's FP64 pipe (about
// 2 DFMA per clock) needs a millisecond -- and the step-size control reads the result on
// the host anyway.  Taylor scaling and squaring (Moler & Van Loan, method 3): s halvings
// bring ||A||_1 to <= 1, where the degree-kDeg Taylor polynomial T is exact to rounding
// (remainder < e / 19! ~ 2e-17); exp(A) e_1 = T(A / 2^s)^(2^s) e_1, applied to the vector
// when 2^s applications of T cost less than s squarings of the matrix, else by squaring.
constexpr int kDeg = 18;
constexpr double kTheta = 1.0;     // ||A / 2^s||_1 <= 1: the Taylor remainder is < 1 / 19!
using cplx = std::complex<double>;

// y = a x for an m x m complex matrix in split planes (ar, ai column-major) whose column c
// is zero below row rows[c] - 1 (an upper Hessenberg matrix has rows[c] = c + 2); plain
// double arithmetic (std::complex products take a slow special-value path without
// fast-math)
void cmatvec(int m, const double* ar, const double* ai, const int* rows, const double* xr,
             const double* xi, double* yr, double* yi) {
  for (int r = 0; r < m; r++) { yr[r] = 0.0; yi[r] = 0.0; }
  for (int c = 0; c < m; c++) {
    const double br = xr[c], bi = xi[c];
    const double* cr = ar + (size_t)m * c;
    const double* ci = ai + (size_t)m * c;
    const int nr = rows[c];
    for (int r = 0; r < nr; r++) {
      yr[r] += cr[r] * br - ci[r] * bi;
      yi[r] += cr[r] * bi + ci[r] * br;
    }
  }
}

void host_expm_col(int m, const double* A, std::vector<cplx>& out) {
  const size_t mm = (size_t)m * m;
  std::vector<double> ar(mm), ai(mm);
  std::vector<int> rows(m, 0), full(m, m);
  double nrm = 0.0;
  for (int c = 0; c < m; c++) {
    double col = 0.0;
    for (int r = 0; r < m; r++) {
      const size_t e = r + (size_t)m * c;
      ar[e] = A[2 * e];
      ai[e] = A[2 * e + 1];
      col += std::hypot(ar[e], ai[e]);
      if (ar[e] != 0.0 || ai[e] != 0.0) rows[c] = r + 1;
    }
    nrm = std::max(nrm, col);
  }
  int sq = 0;
  while (nrm > kTheta && sq < 60) { nrm *= 0.5; sq++; }
  const double sc = std::ldexp(1.0, -sq);
  for (size_t e = 0; e < mm; e++) { ar[e] *= sc; ai[e] *= sc; }
  out.assign(m, cplx(0.0, 0.0));
  const bool by_vector = sq < 20 && (double)(1 << sq) * kDeg < (double)(kDeg + sq) * m;
  if (by_vector) {
    // Horner: T(A) w = w + A (w + A / 2 (w + ... (w + A w / kDeg)))
    std::vector<double> wr(m, 0.0), wi(m, 0.0), ur(m), ui(m), tr(m), ti(m);
    wr[0] = 1.0;
    for (int round = 0; round < (1 << sq); round++) {
      ur = wr;
      ui = wi;
      for (int k = kDeg; k >= 1; k--) {
        cmatvec(m, ar.data(), ai.data(), rows.data(), ur.data(), ui.data(), tr.data(),
                ti.data());
        const double inv = 1.0 / (double)k;
        for (int r = 0; r < m; r++) {
          ur[r] = wr[r] + tr[r] * inv;
          ui[r] = wi[r] + ti[r] * inv;
        }
      }
      wr.swap(ur);
      wi.swap(ui);
    }
    for (int r = 0; r < m; r++) out[r] = cplx(wr[r], wi[r]);
    return;
  }
  // matrix form: E = T(A) by the powers A^k / k!, then s squarings; column 0 out
  std::vector<double> er(mm, 0.0), ei(mm, 0.0), pr(mm, 0.0), pi(mm, 0.0), qr(mm), qi(mm);
  for (int r = 0; r < m; r++) { er[r + (size_t)m * r] = 1.0; pr[r + (size_t)m * r] = 1.0; }
  // Z = X Y, column by column as matrix-vector products
  auto matmul = [&](const std::vector<double>& xr, const std::vector<double>& xi,
                    const std::vector<double>& yr, const std::vector<double>& yi,
                    std::vector<double>& zr, std::vector<double>& zi) {
    for (int c = 0; c < m; c++)
      cmatvec(m, xr.data(), xi.data(), full.data(), yr.data() + (size_t)m * c,
              yi.data() + (size_t)m * c, zr.data() + (size_t)m * c, zi.data() + (size_t)m * c);
  };
  for (int k = 1; k <= kDeg; k++) {
    matmul(pr, pi, ar, ai, qr, qi);
    const double inv = 1.0 / (double)k;
    for (size_t e = 0; e < mm; e++) {
      pr[e] = qr[e] * inv;
      pi[e] = qi[e] * inv;
      er[e] += pr[e];
      ei[e] += pi[e];
    }
  }
  for (int t = 0; t < sq; t++) {
    matmul(er, ei, er, ei, qr, qi);
    er.swap(qr);
    ei.swap(qi);
  }
  for (int r = 0; r < m; r++) out[r] = cplx(er[r], ei[r]);
}


int grid_for(fmpt_handle* h, int64_t n) {
  int64_t g = (n + KT - 1) / KT;
  int64_t cap = (int64_t)h->sm_count * 4;
  if (cap < 1) cap = 1;
  return (int)std::max<int64_t>(1, std::min(g, cap));
}

// Lanczos on a block-sparse operator as ONE CUDA graph: every step of the
// reference recurrence (simple_lanczos.jl:27-68) for j = 0..kmax-1 is
// captured; the step closure (lanczos_close) raises a device stop flag when
// beta < btol, and every later node of the graph -- the grouped H_eff launch
// included -- reads it and returns at once.  One host synchronisation per
// solve.  Any capture or instantiation failure sets *fallback and leaves the
// stream as it was, so the caller runs the host-driven loop instead.
int lanczos_graph(fmpt_op* op, const double* x0, int kmax, double btol, int reorth,
                  double* eigval, double* xout, int* info, int* niter, bool* fallback) {
  fmpt_handle* h = op->h;
  *fallback = true;
  cudaStreamCaptureStatus cap0 = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(h->stream, &cap0) != cudaSuccess ||
      cap0 != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return FMPT_OK;   // the caller is capturing already: no nested capture
  }
  const int64_t n = op->n;   // real data
  const int G = grid_for(h, n);
  DevBuf Vb, Yb, scal, partA, partB, partM, coef, ctlb;
  FMPT_TRY(Vb.alloc(h, (size_t)(kmax + 1) * n * sizeof(double)));
  FMPT_TRY(Yb.alloc(h, (size_t)n * sizeof(double)));
  FMPT_TRY(scal.alloc(h, (size_t)(3 * kmax + 8) * sizeof(double)));
  FMPT_TRY(partA.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(partB.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(partM.alloc(h, (size_t)G * (kmax + 1) * 2 * sizeof(double)));
  FMPT_TRY(coef.alloc(h, (size_t)(kmax + 1) * 2 * sizeof(double)));
  FMPT_TRY(ctlb.alloc(h, 4 * sizeof(int)));
  FMPT_TRY(gp_prepare(h));
  FMPT_TRY(ensure_pinned(h, (size_t)2 * kmax + 2));
  double* V = Vb.d();
  double* y = Yb.d();
  double* s_vm = scal.d();
  double* s_alpha = scal.d() + 1;
  double* s_beta = scal.d() + 1 + kmax;
  int* ctl = static_cast<int*>(ctlb.p);
  auto V_ = [&](int i) { return V + (int64_t)i * n; };
  cudaStream_t st = h->stream;
  auto record = [&]() -> int {
    FMPT_CUDA(h, cudaMemsetAsync(ctl, 0, 4 * sizeof(int), st));
    CHAIN(rdot_partial, G, st, n, x0, x0, partA.d(), nullptr);
    FMPT_LAUNCHED(h);
    CHAIN(normalize_from_parts, G, st, n, x0, V_(0), partA.d(), G, s_vm);
    FMPT_LAUNCHED(h);
    for (int j = 0; j < kmax; j++) {
      FMPT_TRY(op_u1_apply(op, V_(j), y, ctl));
      FMPT_TRY(op_project(op, y, ctl));
      CHAIN(rdot_partial, G, st, n, V_(j), y, partA.d(), ctl);
      FMPT_LAUNCHED(h);
      CHAIN(lanczos_axpy, G, st, n, y, V_(j), j ? V_(j - 1) : nullptr, partA.d(), G,
                                     j ? s_beta + (j - 1) : nullptr, s_alpha + j, partB.d(), ctl);
      FMPT_LAUNCHED(h);
      if (reorth) {
        CHAIN(multidot_partial<false>, G, st, n, j + 1, V, n, y, partM.d(), ctl);
        FMPT_LAUNCHED(h);
        CHAIN(multidot_finalize, (2 * (j + 1) + 7) / 8, st, 0, j + 1, G, partM.d(), coef.d(),
                                                                nullptr, ctl);
        FMPT_LAUNCHED(h);
        CHAIN(multi_axpy_sub, G, st, 0, n, j + 1, V, n, coef.d(), y, partB.d(), ctl);
        FMPT_LAUNCHED(h);
      }
      CHAIN(lanczos_close, G, st, n, y, partB.d(), G, s_beta + j, ctl, btol, j, V_(j + 1));
      FMPT_LAUNCHED(h);
    }
    // alpha and beta are adjacent
    FMPT_CUDA(h, cudaMemcpyAsync(h->pinned, s_alpha, (size_t)2 * kmax * sizeof(double),
                                 cudaMemcpyDeviceToHost, st));
    FMPT_CUDA(h, cudaMemcpyAsync(h->pinned + 2 * kmax, ctl, 4 * sizeof(int),
                                 cudaMemcpyDeviceToHost, st));
    return FMPT_OK;
  };
  if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return FMPT_OK;
  }
  const int rst = record();
  cudaGraph_t graph = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(st, &graph);
  if (rst != FMPT_OK || ce != cudaSuccess || !graph) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    return FMPT_OK;
  }
  bool ready = false;
  if (h->lanczos_exec) {
    cudaGraphExecUpdateResultInfo ri;
    if (cudaGraphExecUpdate(h->lanczos_exec, graph, &ri) == cudaSuccess) {
      ready = true;
    } else {
      cudaGetLastError();
      cudaGraphExecDestroy(h->lanczos_exec);
      h->lanczos_exec = nullptr;
    }
  }
  if (!ready && cudaGraphInstantiate(&h->lanczos_exec, graph, 0) != cudaSuccess) {
    cudaGetLastError();
    h->lanczos_exec = nullptr;
    cudaGraphDestroy(graph);
    return FMPT_OK;
  }
  cudaGraphDestroy(graph);
  *fallback = false;
  FMPT_CUDA(h, cudaGraphLaunch(h->lanczos_exec, st));
  h->graph_launches++;
  FMPT_CUDA(h, cudaStreamSynchronize(st));
  // read the staged results before anything else reuses the pinned buffer
  const int* c = reinterpret_cast<const int*>(h->pinned + 2 * kmax);
  const int k = c[1], bad = c[2], conv = c[3];
  double ev = 0.0;
  RitzCoef rc;
  if (!bad && k > 0) tridiag_lowest(k, h->pinned, h->pinned + kmax, &ev, rc.c);
  FMPT_TRY(gp_check_status(h));
  if (bad) return set_error(h, FMPT_ERR_NONFINITE, "lanczos: beta is not finite");
  CHAIN(combine_ritz, G, st, n, k, V, n, rc, xout);
  FMPT_LAUNCHED(h);
  *eigval = ev;
  if (info) *info = conv ? 0 : -1;
  if (niter) *niter = k;
  return FMPT_OK;
}

// part[2b], part[2b+1] = Re, Im of a grid-stride slice of dot(y, p) = sum conj(y) p
// (Julia's dot, as in _project!); split planes at offset n when cplx
__global__ void proj_dot_partial(int cplx, int64_t n, const double* __restrict__ y,
                                 const double* __restrict__ p, double* __restrict__ part,
                                 const int* gate) {
  if (gate && *gate) return;
  double sr = 0.0, si = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT) {
    sr = fma(y[i], p[i], sr);
    if (cplx) {
      sr = fma(y[n + i], p[n + i], sr);
      si = fma(y[i], p[n + i], si);
      si = fma(-y[n + i], p[i], si);
    }
  }
  sr = block_sum(sr);
  if (cplx) si = block_sum(si);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sr;
    part[2 * blockIdx.x + 1] = si;
  }
}

// c = sum of the G partials (same fixed order in every block); y -= c p
__global__ void proj_axpy(int cplx, int64_t n, double* __restrict__ y, const double* __restrict__ p,
                          const double* __restrict__ part, int G, const int* gate) {
  if (gate && *gate) return;
  double ar = 0.0, ai = 0.0;
  for (int i = threadIdx.x; i < G; i += KT) {
    ar += part[2 * i];
    ai += part[2 * i + 1];
  }
  const double cr = block_sum(ar);
  const double ci = cplx ? block_sum(ai) : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * KT + threadIdx.x; i < n; i += (int64_t)gridDim.x * KT) {
    if (cplx) {
      const double pr = p[i], pi = p[n + i];
      y[i] -= cr * pr - ci * pi;
      y[n + i] -= cr * pi + ci * pr;
    } else {
      y[i] -= cr * p[i];
    }
  }
}

// ---- several eigenpairs: thick-restart Lanczos (exact diagonalisation)

// Symmetric eigendecomposition of a small dense matrix by cyclic Jacobi
// rotations (the two-sided rotation of Golub & Van Loan, Matrix Computations,
// sec. 8.5): A (column-major m x m) is destroyed, w receives the eigenvalues in
// ascending order and Z the matching orthonormal columns.
void jacobi_eigh(int m, std::vector<double>& A, std::vector<double>& w, std::vector<double>& Z) {
  std::vector<double> R((size_t)m * m, 0.0);
  for (int i = 0; i < m; i++) R[i + (size_t)i * m] = 1.0;
  auto a = [&](int i, int j) -> double& { return A[i + (size_t)j * m]; };
  double fro = 0.0;
  for (double v : A) fro += v * v;
  for (int sweep = 0; sweep < 64; sweep++) {
    double off = 0.0;
    for (int q = 1; q < m; q++)
      for (int p = 0; p < q; p++) off += a(p, q) * a(p, q);
    if (off <= 1e-32 * fro) break;
    for (int p = 0; p < m - 1; p++)
      for (int q = p + 1; q < m; q++) {
        const double apq = a(p, q);
        if (apq == 0.0) continue;
        const double theta = (a(q, q) - a(p, p)) / (2.0 * apq);
        const double t = (theta >= 0.0 ? 1.0 : -1.0) /
                         (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), sn = t * c;
        for (int k = 0; k < m; k++) {          // A J
          const double akp = a(k, p), akq = a(k, q);
          a(k, p) = c * akp - sn * akq;
          a(k, q) = sn * akp + c * akq;
        }
        for (int k = 0; k < m; k++) {          // J^T (A J)
          const double apk = a(p, k), aqk = a(q, k);
          a(p, k) = c * apk - sn * aqk;
          a(q, k) = sn * apk + c * aqk;
        }
        for (int k = 0; k < m; k++) {          // Z J
          double* zp = &R[k + (size_t)p * m];
          double* zq = &R[k + (size_t)q * m];
          const double zkp = *zp, zkq = *zq;
          *zp = c * zkp - sn * zkq;
          *zq = sn * zkp + c * zkq;
        }
      }
  }
  std::vector<int> ord(m);
  for (int i = 0; i < m; i++) ord[i] = i;
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return a(x, x) < a(y, y); });
  w.resize(m);
  Z.assign((size_t)m * m, 0.0);
  for (int i = 0; i < m; i++) {
    w[i] = a(ord[i], ord[i]);
    for (int k = 0; k < m; k++) Z[k + (size_t)i * m] = R[k + (size_t)ord[i] * m];
  }
}

// C (nr x c) = V (nr x mm, real view, ld nr) * Y (mm x c, host) on the stream
int basis_times(fmpt_handle* h, const double* V, int64_t nr, int mm, const std::vector<double>& Y,
                int c, DevBuf& Yd, double* C) {
  FMPT_CUDA(h, cudaMemcpyAsync(Yd.d(), Y.data(), (size_t)mm * c * sizeof(double),
                               cudaMemcpyHostToDevice, h->stream));
  GemmArgs g{};
  g.cplx = 0; g.ta = FMPT_N; g.tb = FMPT_N;
  g.m = (int)nr; g.n = c; g.k = mm;
  g.alpha[0] = 1.0; g.beta[0] = 0.0;
  g.A = V; g.lda = nr; g.planeA = 0;
  g.B = Yd.d(); g.ldb = mm; g.planeB = 0;
  g.C = C; g.ldc = nr; g.planeC = 0;
  g.batch = 1;
  return gemm_f64(h, g);
}

// Thick-restart Lanczos (Wu & Simon, SIAM J. Matrix Anal. Appl. 22 (2000) 602)
// with full reorthogonalisation (two classical Gram-Schmidt passes) for the
// ``num`` eigenvalues of a Hermitian operator at one end of the spectrum
// (which 0: smallest, 1: largest).  The basis lives on the device; the
// Rayleigh quotient (at most krylovdim x krylovdim, real symmetric: the
// Lanczos coefficients of a Hermitian operator are real) is solved on the host.
// A Ritz pair has converged when its residual norm |beta_m y_m| <= tol.
int eigsolve_impl(fmpt_op* op, const double* x0, int num, int kdim, int maxiter, double tol,
                  int which, double* evals, double* evecs, double* resid, int* nconv,
                  int* napply) {
  fmpt_handle* h = op->h;
  const int cp = op->dtype == FMPT_C128;
  const int64_t n = op->n;
  const int64_t nr = n * (cp ? 2 : 1);
  const int m = (int)std::min<int64_t>(kdim, n);
  if (num > m) return set_error(h, FMPT_ERR_ARG, "eigsolve: num %d exceeds the space", num);
  if (m < n && m < num + 2)
    return set_error(h, FMPT_ERR_ARG, "eigsolve: krylovdim must be at least num + 2");
  const int G = grid_for(h, n);
  DevBuf Vb, zb, partA, partM, coef, acc, Yd, tmp, snrm;
  FMPT_TRY(Vb.alloc(h, (size_t)(m + 1) * nr * sizeof(double)));
  FMPT_TRY(zb.alloc(h, (size_t)nr * sizeof(double)));
  FMPT_TRY(partA.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(partM.alloc(h, (size_t)G * (m + 1) * 2 * sizeof(double)));
  FMPT_TRY(coef.alloc(h, (size_t)(m + 1) * 2 * sizeof(double)));
  FMPT_TRY(acc.alloc(h, (size_t)(m + 1) * 2 * sizeof(double)));
  FMPT_TRY(Yd.alloc(h, (size_t)m * m * sizeof(double)));
  FMPT_TRY(snrm.alloc(h, sizeof(double)));
  FMPT_TRY(ensure_pinned(h, (size_t)2 * (m + 1) + G + 1));
  double* V = Vb.d();
  double* z = zb.d();
  auto V_ = [&](int i) { return V + (int64_t)i * nr; };
  cudaStream_t st = h->stream;
  CHAIN(rdot_partial, G, st, nr, x0, x0, partA.d(), nullptr);
  FMPT_LAUNCHED(h);
  CHAIN(normalize_from_parts, G, st, nr, x0, V_(0), partA.d(), G, snrm.d());
  FMPT_LAUNCHED(h);
  FMPT_CUDA(h, cudaMemcpyAsync(h->pinned, snrm.d(), sizeof(double), cudaMemcpyDeviceToHost, st));
  FMPT_CUDA(h, cudaStreamSynchronize(st));
  if (!(h->pinned[0] > 0.0) || !std::isfinite(h->pinned[0]))
    return set_error(h, FMPT_ERR_ARG, "eigsolve: the start vector is zero or not finite");
  std::vector<double> H((size_t)(m + 1) * (m + 1), 0.0);
  auto Hx = [&](int i, int j) -> double& { return H[i + (size_t)j * (m + 1)]; };
  std::vector<double> theta, Y, A;
  int k = 0, applies = 0;
  for (int it = 0;; it++) {
    bool breakdown = false;
    int j = k;
    for (; j < m; j++) {
      FMPT_TRY(fmpt_op_apply(op, V_(j), z));
      applies++;
      FMPT_CUDA(h, cudaMemsetAsync(acc.d(), 0, (size_t)2 * (j + 1) * sizeof(double), st));
      for (int pass = 0; pass < 2; pass++) {
        if (cp) CHAIN(multidot_partial<true>, G, st, n, j + 1, V, nr, z, partM.d(), nullptr);
        else CHAIN(multidot_partial<false>, G, st, n, j + 1, V, nr, z, partM.d(), nullptr);
        FMPT_LAUNCHED(h);
        CHAIN(multidot_finalize, (2 * (j + 1) + 7) / 8, st, cp, j + 1, G, partM.d(), coef.d(),
                                                                acc.d(), nullptr);
        FMPT_LAUNCHED(h);
        CHAIN(multi_axpy_sub, G, st, cp, n, j + 1, V, nr, coef.d(), z, partA.d(), nullptr);
        FMPT_LAUNCHED(h);
      }
      double* hp = h->pinned;
      FMPT_CUDA(h, cudaMemcpyAsync(hp, acc.d(), (size_t)2 * (j + 1) * sizeof(double),
                                   cudaMemcpyDeviceToHost, st));
      FMPT_CUDA(h, cudaMemcpyAsync(hp + 2 * (j + 1), partA.d(), (size_t)G * sizeof(double),
                                   cudaMemcpyDeviceToHost, st));
      FMPT_CUDA(h, cudaStreamSynchronize(st));
      double b2 = 0.0;
      for (int g = 0; g < G; g++) b2 += hp[2 * (j + 1) + g];
      double ref = b2;
      for (int i = 0; i <= j; i++) {
        Hx(i, j) = Hx(j, i) = hp[2 * i];
        ref += hp[2 * i] * hp[2 * i] + hp[2 * i + 1] * hp[2 * i + 1];
      }
      if (!std::isfinite(b2)) return set_error(h, FMPT_ERR_NONFINITE, "eigsolve: not finite");
      const double beta = std::sqrt(b2);
      if (!(beta > 1e-12 * std::sqrt(ref))) {     // invariant subspace: exact Ritz pairs
        breakdown = true;
        j++;
        break;
      }
      CHAIN(normalize_from_parts, G, st, nr, z, V_(j + 1), partA.d(), G, snrm.d());
      FMPT_LAUNCHED(h);
      Hx(j + 1, j) = Hx(j, j + 1) = beta;
    }
    const int mm = j;
    const double beta_last = breakdown ? 0.0 : Hx(mm, mm - 1);
    A.assign((size_t)mm * mm, 0.0);
    for (int c = 0; c < mm; c++)
      for (int r = 0; r < mm; r++) A[r + (size_t)c * mm] = Hx(r, c);
    jacobi_eigh(mm, A, theta, Y);
    std::vector<int> idx(mm);
    for (int i = 0; i < mm; i++) idx[i] = which == 1 ? mm - 1 - i : i;
    std::vector<double> res(mm);
    int conv = 0;
    for (int i = 0; i < mm; i++) res[i] = std::fabs(beta_last * Y[(mm - 1) + (size_t)idx[i] * mm]);
    while (conv < num && res[conv] <= tol) conv++;
    if (conv >= num || breakdown || it + 1 >= maxiter) {
      if (mm < num)
        return set_error(h, FMPT_ERR_ARG,
                         "eigsolve: the start vector lies in an invariant subspace of "
                         "dimension %d < num", mm);
      std::vector<double> Ys((size_t)mm * num);
      for (int i = 0; i < num; i++)
        for (int r = 0; r < mm; r++) Ys[r + (size_t)i * mm] = Y[r + (size_t)idx[i] * mm];
      FMPT_TRY(basis_times(h, V, nr, mm, Ys, num, Yd, evecs));
      for (int i = 0; i < num; i++) {
        evals[i] = theta[idx[i]];
        if (resid) resid[i] = res[i];
      }
      if (nconv) *nconv = breakdown ? num : conv;
      if (napply) *napply = applies;
      FMPT_CUDA(h, cudaStreamSynchronize(st));
      return FMPT_OK;
    }
    // keep the ``keep`` best Ritz vectors and the residual direction
    const int keep = std::min(mm - 1, num + (mm - num) / 2);
    std::vector<double> Ys((size_t)mm * keep);
    for (int i = 0; i < keep; i++)
      for (int r = 0; r < mm; r++) Ys[r + (size_t)i * mm] = Y[r + (size_t)idx[i] * mm];
    if (!tmp.p) {
      FMPT_TRY(tmp.alloc(h, (size_t)m * nr * sizeof(double)));
    }
    FMPT_TRY(basis_times(h, V, nr, mm, Ys, keep, Yd, tmp.d()));
    FMPT_CUDA(h, cudaMemcpyAsync(V, tmp.d(), (size_t)keep * nr * sizeof(double),
                                 cudaMemcpyDeviceToDevice, st));
    FMPT_CUDA(h, cudaMemcpyAsync(V_(keep), V_(mm), (size_t)nr * sizeof(double),
                                 cudaMemcpyDeviceToDevice, st));
    std::fill(H.begin(), H.end(), 0.0);
    for (int i = 0; i < keep; i++) {
      Hx(i, i) = theta[idx[i]];
      Hx(i, keep) = Hx(keep, i) = beta_last * Y[(mm - 1) + (size_t)idx[i] * mm];
    }
    k = keep;
  }
}

}  // namespace

// _project! (algorithms/dmrgexcited.jl:1-6): y = y - dot(y, p) p for every
// projector in turn, on the handle's stream with the scalars kept on the device
int op_project(fmpt_op* op, double* y, const int* gate) {
  if (op->proj.empty()) return FMPT_OK;
  fmpt_handle* h = op->h;
  const int cp = op->dtype == FMPT_C128;
  for (const double* p : op->proj) {
    proj_dot_partial<<<op->proj_G, KT, 0, h->stream>>>(cp, op->n, y, p, op->proj_part, gate);
    FMPT_LAUNCHED(h);
    proj_axpy<<<op->proj_G, KT, 0, h->stream>>>(cp, op->n, y, p, op->proj_part, op->proj_G,
                                                 gate);
    FMPT_LAUNCHED(h);
  }
  return FMPT_OK;
}

// Workspace and launch shape of the Arnoldi orthogonalisation step.
struct GsWork {
  int G, cpb;
  bool single;        // every warp has one chunk
  bool fused;         // one launch per step
  bool cluster;       // .. of one block or one cluster, otherwise cooperative
  double* part;       // [2][GS_NV][G]
  double* coef;       // [2 GS_NV + 1] (separate launches)
  int* bar;
  int* status;
  uint64_t wait_ns;
  int hold;
};

// Blocks of the step and chunks per block for S chunks: one block, without grid-wide waits, up
// to 4 chunks; one cluster of 4, 8 or 16 blocks up to GS_CLUSTER_S chunks (complex exponential of
// 20 vectors, cooperative -> cluster: D = 8 649 -> 592 us, D = 16 754 -> 706, D = 22, the last
// one, 832 -> 810; D = 27 would take 978 instead of 904: 16 SMs are too few for it); then as few
// chunks per block as keep it within 128 blocks (n = 8192 complex: 4 chunks, one per SM
// sub-partition); beyond 1024 chunks the warps loop.
constexpr int GS_CLUSTER_S = 64;
void gs_geometry(int64_t S, int& G, int& cpb, bool& single) {
  single = true;
  if (S <= 4) {
    G = 1;
    cpb = S <= 1 ? 1 : (S <= 2 ? 2 : 4);
    return;
  }
  if (S <= GS_CLUSTER_S) {
    cpb = 1;
    while ((S + cpb - 1) / cpb > 16) cpb *= 2;
    G = 4;
    while ((int64_t)G * cpb < S) G *= 2;
    return;
  }
  for (cpb = 1; cpb <= 8; cpb *= 2)
    if ((S + cpb - 1) / cpb <= 128) {
      G = (int)((S + cpb - 1) / cpb);
      return;
    }
  cpb = 8;
  G = 128;
  single = false;
}

// Whether G blocks of the fused step are co-resident on this device (the cooperative launch
// needs it); measured once per device.
bool gs_fused_fits(fmpt_handle* h, int G) {
  static std::mutex mu;
  static int occ[64] = {};
  static bool done[64] = {};
  const int dev = h->device;
  if (dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (!done[dev]) {
    int a = 0, b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, arnoldi_gs_fused<true>, GS_T, 0) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, arnoldi_gs_fused<false>, GS_T, 0) !=
            cudaSuccess) {
      cudaGetLastError();
      a = b = 0;
    }
    occ[dev] = std::min(a, b);
    done[dev] = true;
  }
  return (int64_t)occ[dev] * h->sm_count >= G;
}

void gs_cluster_config(fmpt_handle* h, int G, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(GS_T);
  cfg.stream = h->stream;
  cfg.attrs = attr;
  chain_attr(attr[0]);
  cfg.numAttrs = 1;
  if (G > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = G;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
}
// Whether a cluster of G blocks (up to 16: beyond the portable 8) fits this device.
bool gs_cluster_fits(fmpt_handle* h, int G) {
  if (G == 1) return true;
  static std::mutex mu;
  static signed char fits[64][5] = {};                      // 0 unknown, 1 yes, -1 no; by log2 G
  const int dev = h->device, l = G == 4 ? 2 : (G == 8 ? 3 : 4);
  if (dev < 0 || dev >= 64) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (!fits[dev][l]) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    gs_cluster_config(h, G, cfg, attr);
    std::swap(attr[0], attr[1]);                            // the cluster attribute alone
    cfg.numAttrs = 1;
    int n = 0;
    const bool ok = cudaFuncSetAttribute(arnoldi_gs_cluster,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                        cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, arnoldi_gs_cluster, &cfg) == cudaSuccess &&
                    n > 0;
    if (!ok) cudaGetLastError();
    fits[dev][l] = ok ? 1 : -1;
  }
  return fits[dev][l] > 0;
}

int gs_setup(fmpt_handle* h, int cp, int64_t n, int M, DevBuf& buf, GsWork& w) {
  const int64_t nch = (n + 31) / 32;
  gs_geometry(cp ? 2 * nch : nch, w.G, w.cpb, w.single);
  w.fused = h->fused_gs && gs_fused_fits(h, w.G);
  // (the test of the bounded grid waits needs the launch that has them)
  w.cluster = w.fused && (cp ? 2 * nch : nch) <= GS_CLUSTER_S && h->wait_test_hold == 0 &&
              gs_cluster_fits(h, w.G);
  const size_t parts = (size_t)2 * GS_NV * w.G;
  FMPT_TRY(buf.alloc(h, (parts + 2 * GS_NV + 2 + 2) * sizeof(double)));
  w.part = buf.d();
  w.coef = w.part + parts;
  w.bar = reinterpret_cast<int*>(w.coef + 2 * GS_NV + 2);
  FMPT_TRY(gp_status_word(h, &w.status));
  w.wait_ns = h->wait_test_ns > 0 ? (uint64_t)h->wait_test_ns : 2000000000ull;
  w.hold = h->wait_test_hold;
  return FMPT_OK;
}

// V_{j+1} and H's column j from z = op(V_j)
int gs_step(fmpt_handle* h, const GsWork& w, int cp, int64_t n, int64_t nr, int j, double* V,
            double* z, double* Hcol) {
  cudaStream_t st = h->stream;
  GsArgs a{};
  a.cplx = cp;
  a.j = j;
  a.n = n;
  a.cpb = w.cpb;
  a.V = V;
  a.vstride = nr;
  a.z = z;
  a.part = w.part;
  a.Hcol = Hcol;
  a.vnext = V + (int64_t)(j + 1) * nr;
  if (w.cluster) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    gs_cluster_config(h, w.G, cfg, attr);
    FMPT_CUDA(h, cudaLaunchKernelEx(&cfg, arnoldi_gs_cluster, a));
    FMPT_LAUNCHED(h);
    return FMPT_OK;
  }
  if (w.fused) {
    const CoopBar bar{w.bar, w.bar + 1, w.status, w.wait_ns, w.hold};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(w.G);
    cfg.blockDim = dim3(GS_T);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FMPT_CUDA(h, w.single ? cudaLaunchKernelEx(&cfg, arnoldi_gs_fused<true>, a, bar)
                          : cudaLaunchKernelEx(&cfg, arnoldi_gs_fused<false>, a, bar));
    FMPT_LAUNCHED(h);
    return FMPT_OK;
  }
  for (int pass = 0; pass < 2; pass++) {
    if (w.single) arnoldi_gs_dots<true><<<w.G, GS_T, 0, st>>>(a, pass);
    else arnoldi_gs_dots<false><<<w.G, GS_T, 0, st>>>(a, pass);
    FMPT_LAUNCHED(h);
    arnoldi_gs_sums<<<1, GS_T, 0, st>>>(a, pass, w.G, w.coef);
    FMPT_LAUNCHED(h);
    if (w.single) arnoldi_gs_axpy<true><<<w.G, GS_T, 0, st>>>(a, pass, w.coef);
    else arnoldi_gs_axpy<false><<<w.G, GS_T, 0, st>>>(a, pass, w.coef);
    FMPT_LAUNCHED(h);
  }
  return FMPT_OK;
}

// The Arnoldi basis V_1..V_M of fmpt_exponentiate / fmpt_expm_nodes (two-pass classical
// Gram-Schmidt; the columns of H into Hdev), device launches only.  Launched one by one: a
// vector's four or five kernels take the device 25 us and the host 10, while recording them into
// a graph and updating its executable kept the device waiting (TDVP1 gradient of 8 sites, 116
// bases: 109 ms recorded, 104 launched).
int arnoldi_basis(fmpt_op* op, int cp, int64_t n, int64_t nr, int M, int ldh, double* V,
                  double* z, DevBuf& Hdev, const GsWork& gs) {
  fmpt_handle* h = op->h;
  struct KPieces {
    fmpt_handle* h;
    explicit KPieces(fmpt_handle* hh) : h(hh) { h->k_pieces = 1; }
    ~KPieces() { h->k_pieces = 0; }
  } pieces(h);
  FMPT_CUDA(h, cudaMemsetAsync(Hdev.p, 0, Hdev.bytes, h->stream));
  if (gs.fused && !gs.cluster)
    FMPT_CUDA(h, cudaMemsetAsync(gs.bar, 0, 2 * sizeof(int), h->stream));
  for (int j = 0; j < M; j++) {
    FMPT_TRY(fmpt_op_apply(op, V + (int64_t)j * nr, z));
    FMPT_TRY(gs_step(h, gs, cp, n, nr, j, V, z, Hdev.d() + (size_t)2 * ldh * j));
  }
  return FMPT_OK;
}

}  // namespace fmpt

using namespace fmpt;

extern "C" {

int fmpt_eigsolve(fmpt_op* op, const double* x0, int num, int krylovdim, int maxiter, double tol,
                  int which, double* evals, double* evecs, double* resid, int* nconv,
                  int* napply) {
  if (!op) return FMPT_ERR_ARG;
  fmpt_handle* h = op->h;
  if (!x0 || !evals || !evecs) return set_error(h, FMPT_ERR_ARG, "eigsolve: null pointer");
  if (num < 1 || krylovdim < 2 || krylovdim > 256 || maxiter < 1 || !(tol >= 0.0) ||
      (which != 0 && which != 1))
    return set_error(h, FMPT_ERR_ARG, "eigsolve: bad num/krylovdim/maxiter/tol/which");
  return eigsolve_impl(op, x0, num, krylovdim, maxiter, tol, which, evals, evecs, resid, nconv,
                       napply);
}

int fmpt_op_set_projectors(fmpt_op* op, int nproj, const double* const* p) {
  if (!op) return FMPT_ERR_ARG;
  fmpt_handle* h = op->h;
  if (nproj < 0 || (nproj > 0 && !p))
    return set_error(h, FMPT_ERR_ARG, "set_projectors: bad projector list");
  for (int i = 0; i < nproj; i++)
    if (!p[i]) return set_error(h, FMPT_ERR_ARG, "set_projectors: null projector %d", i);
  if (nproj > 0 && !op->proj_part) {
    const int G = grid_for(h, op->n);
    void* q = nullptr;
    cudaError_t e = cudaMallocAsync(&q, 2 * (size_t)G * sizeof(double), h->stream);
    if (e != cudaSuccess)
      return set_error(h, e == cudaErrorMemoryAllocation ? FMPT_ERR_NOMEM : FMPT_ERR_CUDA,
                       "set_projectors: %s", cudaGetErrorString(e));
    op->proj_part = static_cast<double*>(q);
    op->proj_G = G;
  }
  op->proj.assign(p, p + nproj);
  return FMPT_OK;
}

// fmpt_lanczos_ground, its last launches (among them the one that writes xout) still queued
static int lanczos_ground(fmpt_op* op, const double* x0, int kmax, double btol, int reorth,
                          double* eigval, double* xout, int* info, int* niter) {
  fmpt_handle* h = op->h;
  // the solve's tensor-core FP64 GEMMs are the digit products (ozaki_digits.cu says why)
  struct DigitEngine {
    fmpt_handle* h;
    explicit DigitEngine(fmpt_handle* hh) : h(hh) { h->oz_digits = 1; }
    ~DigitEngine() { h->oz_digits = 0; }
  } digit_engine(h);
  if (op->u1 && h->graphs) {
    bool fallback = false;
    const int st = lanczos_graph(op, x0, kmax, btol, reorth, eigval, xout, info, niter, &fallback);
    if (!fallback) return st;
  }
  const int cp = op->dtype == FMPT_C128;
  const int64_t n = op->n * (cp ? 2 : 1);   // real view of the vector
  const int G = grid_for(h, n);
  DevBuf Vb, Yb, scal, partA, partB, partM, coef;
  FMPT_TRY(Vb.alloc(h, (size_t)(kmax + 1) * n * sizeof(double)));
  FMPT_TRY(Yb.alloc(h, (size_t)n * sizeof(double)));
  FMPT_TRY(scal.alloc(h, (size_t)(2 * kmax + 2) * sizeof(double)));   // vm, alpha, beta, stop
  FMPT_TRY(partA.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(partB.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(partM.alloc(h, (size_t)G * (kmax + 1) * 2 * sizeof(double)));
  FMPT_TRY(coef.alloc(h, (size_t)(kmax + 1) * 2 * sizeof(double)));
  if (!h->step_host) FMPT_CUDA(h, cudaMallocHost((void**)&h->step_host, 256 * sizeof(double)));
  for (cudaEvent_t& e : h->step_event)
    if (!e) FMPT_CUDA(h, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  double* V = Vb.d();
  double* y = Yb.d();
  double* s_vm = scal.d();
  double* s_alpha = scal.d() + 1;
  double* s_beta = scal.d() + 1 + kmax;
  auto V_ = [&](int i) { return V + (int64_t)i * n; };

  // reorthogonalise y against V_0..V_{j-1} (classical Gram-Schmidt, one pass)
  auto reorthogonalise = [&](int j) -> int {
    CHAIN(multidot_partial<false>, G, h->stream, n, j, V, n, y, partM.d(), nullptr);
    FMPT_LAUNCHED(h);
    CHAIN(multidot_finalize, (2 * j + 7) / 8, h->stream, 0, j, G, partM.d(), coef.d(), nullptr,
          nullptr);
    FMPT_LAUNCHED(h);
    CHAIN(multi_axpy_sub, G, h->stream, 0, n, j, V, n, coef.d(), y, partB.d(), nullptr);
    FMPT_LAUNCHED(h);
    return FMPT_OK;
  };

  // Step j + 1 is queued before beta_j is looked at, so that the device does not wait for the
  // host's test (10 us per step); one step past convergence is thrown away.  Where its GEMMs
  // take more than about 50 us they look at a flag that the step before raises, and do nothing
  // (a solve that ends with its first step: FP64 D = 256 195 -> 127 us, D = 512 1005 -> 551;
  // the looks are 1% of a D = 128 step); below, the step is cheaper than the looks.
  double flops = 0.0;
  FMPT_TRY(fmpt_op_flops(op, &flops));
  int* stop = nullptr;
  if (flops > 50e-6 * (prec_is_f64(op->precision) ? 1.1e12 : 1e14)) {
    stop = reinterpret_cast<int*>(s_beta + kmax);
    FMPT_CUDA(h, cudaMemsetAsync(stop, 0, sizeof(int), h->stream));
  }
  struct Gate {
    fmpt_handle* h;
    Gate(fmpt_handle* hh, const int* g) : h(hh) { h->gate = g; }
    ~Gate() { h->gate = nullptr; }
  };

  // step j: lanczos_make_first_step / lanczos_make_step (simple_lanczos.jl:27-68), from V_j
  // to alpha_j, beta_j and V_{j+1}; alpha_j and beta_j are in step_host[2 j], [2 j + 1] once
  // step_event[j & 1] has passed
  double* ab = h->step_host;
  const TcPlanes px = op_tc_planes(op);        // V_1, V_2, .. are written there as well
  auto launch_step = [&](int j) -> int {
    {
      Gate closed(h, j > 0 ? stop : nullptr);
      FMPT_TRY(j > 0 && px.mode >= 0 ? op_apply_planes(op, y) : fmpt_op_apply(op, V_(j), y));
    }
    CHAIN(rdot_partial, G, h->stream, n, V_(j), y, partA.d(), nullptr);
    FMPT_LAUNCHED(h);
    CHAIN(lanczos_axpy, G, h->stream, n, y, V_(j), j ? V_(j - 1) : nullptr, partA.d(), G,
                                          j ? s_beta + (j - 1) : nullptr, s_alpha + j, partB.d(), nullptr);
    FMPT_LAUNCHED(h);
    if (reorth) FMPT_TRY(reorthogonalise(j + 1));
    auto scale = px.mode == M_TF32     ? lanczos_scale<M_TF32>
                 : px.mode == M_TF32X3 ? lanczos_scale<M_TF32X3>
                 : px.mode == M_BF16   ? lanczos_scale<M_BF16>
                                       : lanczos_scale<-1>;
    CHAIN(scale, G, h->stream, n, y, partB.d(), G, s_alpha + j, s_beta + j, V_(j + 1), ab + 2 * j,
          btol, stop, px.hi, px.lo);
    FMPT_LAUNCHED(h);
    FMPT_CUDA(h, cudaEventRecord(h->step_event[j & 1], h->stream));
    return FMPT_OK;
  };
  CHAIN(rdot_partial, G, h->stream, n, x0, x0, partA.d(), nullptr);
  FMPT_LAUNCHED(h);
  CHAIN(normalize_from_parts, G, h->stream, n, x0, V_(0), partA.d(), G, s_vm);
  FMPT_LAUNCHED(h);
  double al[128], be[128];
  int k = 0;
  bool converged = false;
  FMPT_TRY(launch_step(0));
  while (k < kmax && !converged) {
    if (k + 1 < kmax) FMPT_TRY(launch_step(k + 1));
    FMPT_CUDA(h, cudaEventSynchronize(h->step_event[k & 1]));
    al[k] = ab[2 * k];
    be[k] = ab[2 * k + 1];
    if (!std::isfinite(be[k]))
      return set_error(h, FMPT_ERR_NONFINITE, "lanczos: beta is not finite");
    converged = be[k] < btol;
    k++;
  }
  if (converged && k == 1) {
    // converged after the first step: Rayleigh quotient and the start vector
    FMPT_CUDA(h, cudaMemcpyAsync(xout, V_(0), n * sizeof(double), cudaMemcpyDeviceToDevice,
                                 h->stream));
    *eigval = al[0];
  } else {
    // eigen(Symmetric(T[1:k,1:k])), lowest pair (find_lanczos "SR")
    RitzCoef rc;
    tridiag_lowest(k, al, be, eigval, rc.c);
    CHAIN(combine_ritz, G, h->stream, n, k, V, n, rc, xout);
    FMPT_LAUNCHED(h);
  }
  if (!prec_is_f64(op->precision)) FMPT_TRY(op_tc_check(op));
  if (op->u1) FMPT_TRY(gp_check_status(op->h));
  if (info) *info = converged ? 0 : -1;
  if (niter) *niter = k;
  return FMPT_OK;
}

int fmpt_lanczos_ground(fmpt_op* op, const double* x0, int kmax, double btol, int reorth,
                        double* eigval, double* xout, int* info, int* niter) {
  if (!op) return FMPT_ERR_ARG;
  fmpt_handle* h = op->h;
  if (!x0 || !xout || !eigval) return set_error(h, FMPT_ERR_ARG, "lanczos: null pointer");
  if (kmax < 1 || kmax > 128) return set_error(h, FMPT_ERR_ARG, "lanczos: kmax must be 1..128");
  const int st = lanczos_ground(op, x0, kmax, btol, reorth, eigval, xout, info, niter);
  // A call that returns host scalars synchronises: xout may be read on any stream, and nothing
  // that is still queued (a step thrown away, after an error too) reads the caller's data.
  const cudaError_t e = cudaStreamSynchronize(h->stream);
  if (st != FMPT_OK) return st;
  FMPT_CUDA(h, e);
  return FMPT_OK;
}

int fmpt_exponentiate(fmpt_op* op, double t_re, double t_im, const double* x, double* xout,
                      int krylovdim, double tol, int* info) {
  if (!op) return FMPT_ERR_ARG;
  fmpt_handle* h = op->h;
  if (!x || !xout) return set_error(h, FMPT_ERR_ARG, "exponentiate: null pointer");
  if (krylovdim < 1 || krylovdim > 31)
    return set_error(h, FMPT_ERR_ARG, "exponentiate: krylovdim must be 1..31");
  const int cp = op->dtype == FMPT_C128;
  if (!cp && t_im != 0.0)
    return set_error(h, FMPT_ERR_ARG, "exponentiate: complex time step needs dtype C128");
  const int64_t n = op->n;                     // elements (complex for C128)
  const int64_t nr = n * (cp ? 2 : 1);         // real view
  const int G = grid_for(h, nr);
  // the Krylov space cannot be larger than the vector space
  const int M = (int)std::min<int64_t>(krylovdim, n);
  const int ldh = M + 1;
  DevBuf Vb, zb, part, Hdev, Ed, nrm, acc;
  FMPT_TRY(Vb.alloc(h, (size_t)(M + 1) * nr * sizeof(double)));
  FMPT_TRY(zb.alloc(h, (size_t)nr * sizeof(double)));
  FMPT_TRY(part.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(Hdev.alloc(h, (size_t)ldh * M * 2 * sizeof(double)));
  FMPT_TRY(Ed.alloc(h, (size_t)M * 2 * sizeof(double)));
  std::vector<double> colbuf((size_t)2 * M);
  FMPT_TRY(nrm.alloc(h, 2 * sizeof(double)));
  FMPT_TRY(acc.alloc(h, 2 * sizeof(double)));
  FMPT_TRY(ensure_pinned(h, (size_t)ldh * M * 2 + 8));
  DevBuf gsbuf;
  GsWork gs{};
  FMPT_TRY(gs_setup(h, cp, n, M, gsbuf, gs));
  double* V = Vb.d();
  auto V_ = [&](int i) { return V + (int64_t)i * nr; };
  const double tabs = std::hypot(t_re, t_im);
  if (tabs == 0.0) {
    FMPT_CUDA(h, cudaMemcpyAsync(xout, x, nr * sizeof(double), cudaMemcpyDeviceToDevice,
                                 h->stream));
    if (info) *info = 0;
    return FMPT_OK;
  }
  const double sg_r = t_re / tabs, sg_i = t_im / tabs;
  // w = x / ||x||, acc = ||x|| (the running norm stays on the device)
  CHAIN(rdot_partial, G, h->stream, nr, x, x, part.d(), nullptr);
  FMPT_LAUNCHED(h);
  CHAIN(normalize_from_parts, G, h->stream, nr, x, V_(0), part.d(), G, acc.d());
  FMPT_LAUNCHED(h);
  double tau_done = 0.0, dtau = tabs;
  int steps = 0;
  std::vector<double> Hh((size_t)ldh * M * 2);
  std::vector<double> Hs;
  while (tau_done < tabs * (1.0 - 1e-15)) {
    if (++steps > 1000) return set_error(h, FMPT_ERR_NOCONV, "exponentiate: too many steps");
    // ---- Arnoldi (two-pass classical Gram-Schmidt) entirely on the device
    FMPT_TRY(arnoldi_basis(op, cp, n, nr, M, ldh, V, zb.d(), Hdev, gs));
    FMPT_CUDA(h, cudaMemcpyAsync(h->pinned, Hdev.p, Hdev.bytes, cudaMemcpyDeviceToHost,
                                 h->stream));
    FMPT_CUDA(h, cudaStreamSynchronize(h->stream));
    if (gs.fused) FMPT_TRY(gp_check_status(h));     // a fused step that gave up left H invalid
    std::copy(h->pinned, h->pinned + Hh.size(), Hh.begin());
    for (double v : Hh)
      if (!std::isfinite(v)) return set_error(h, FMPT_ERR_NONFINITE, "exponentiate: NaN");
    // happy breakdown: the first zero subdiagonal closes the Krylov space
    int m = M;
    bool happy = M == n;
    for (int j = 0; j < M; j++)
      if (Hh[2 * (j + 1 + (size_t)ldh * j)] == 0.0) { m = j + 1; happy = true; break; }
    dtau = happy ? (tabs - tau_done) : std::min(dtau, tabs - tau_done);
    Hs.assign((size_t)m * m * 2, 0.0);
    std::vector<cplx> col;
    for (int tries = 0; tries < 200; tries++) {
      const double fr = sg_r * dtau, fi = sg_i * dtau;
      for (int c = 0; c < m; c++)
        for (int r = 0; r < m; r++) {
          const double hr = Hh[2 * (r + (size_t)ldh * c)], hi = Hh[2 * (r + (size_t)ldh * c) + 1];
          Hs[2 * (r + (size_t)m * c)] = fr * hr - fi * hi;
          Hs[2 * (r + (size_t)m * c) + 1] = fr * hi + fi * hr;
        }
      host_expm_col(m, Hs.data(), col);
      if (happy) break;
      // error estimate |h_{m+1,m} dtau [exp(dtau H)]_{m,1}|
      const double hlast = Hh[2 * (m + (size_t)ldh * (m - 1))];
      const double err = std::abs(hlast * dtau) * std::abs(col[m - 1]);
      if (err <= 0.9 * tol * dtau) break;
      dtau *= 0.5;
    }
    // pageable source: the copy has left colbuf when cudaMemcpyAsync returns
    for (int r = 0; r < m; r++) {
      colbuf[2 * r] = col[r].real();
      colbuf[2 * r + 1] = col[r].imag();
    }
    FMPT_CUDA(h, cudaMemcpyAsync(Ed.d(), colbuf.data(), (size_t)2 * m * sizeof(double),
                                 cudaMemcpyHostToDevice, h->stream));
    // w = sum_i E[i, 0] V_i, renormalised into V_0; acc *= ||w||
    CHAIN(combine_basis, G, h->stream, cp, n, m, V, nr, Ed.d(), 0, nullptr, zb.d(), 0);
    FMPT_LAUNCHED(h);
    CHAIN(rdot_partial, G, h->stream, nr, zb.d(), zb.d(), part.d(), nullptr);
    FMPT_LAUNCHED(h);
    CHAIN(normalize_from_parts, G, h->stream, nr, zb.d(), V_(0), part.d(), G, nrm.d());
    FMPT_LAUNCHED(h);
    mul_scalar<<<1, 1, 0, h->stream>>>(acc.d(), nrm.d());
    FMPT_LAUNCHED(h);
    tau_done += dtau;
    if (!happy && tau_done < tabs) dtau = std::min(2.0 * dtau, tabs - tau_done);
  }
  // xout = acc * V_0
  FMPT_CUDA(h, cudaMemcpyAsync(xout, V_(0), nr * sizeof(double), cudaMemcpyDeviceToDevice,
                               h->stream));
  CHAIN(scale_by, G, h->stream, nr, xout, acc.d());
  FMPT_LAUNCHED(h);
  if (!prec_is_f64(op->precision)) FMPT_TRY(op_tc_check(op));
  if (op->u1 || gs.fused) FMPT_TRY(gp_check_status(op->h));
  if (info) *info = steps;
  return FMPT_OK;
}

// exp(s_j t H) x for several s_j from ONE Krylov space of x (the quadrature
// nodes of the exponential's adjoint).  Arnoldi as in fmpt_exponentiate;
// no step-size control: err_est (host) gets max_j |h_{m+1,m} [exp(s_j t H_m)]_{m,1}|,
// the usual a-posteriori estimate relative to ||x||.
int fmpt_expm_nodes(fmpt_op* op, double t_re, double t_im, const double* x, int krylovdim,
                    int nnodes, const double* nodes, double* out, double* err_est) {
  if (!op) return FMPT_ERR_ARG;
  fmpt_handle* h = op->h;
  if (!x || !out || !nodes || nnodes < 1)
    return set_error(h, FMPT_ERR_ARG, "expm_nodes: null pointer or no nodes");
  if (krylovdim < 1 || krylovdim > 31)
    return set_error(h, FMPT_ERR_ARG, "expm_nodes: krylovdim must be 1..31");
  const int cp = op->dtype == FMPT_C128;
  if (!cp && t_im != 0.0)
    return set_error(h, FMPT_ERR_ARG, "expm_nodes: complex time needs dtype C128");
  const int64_t n = op->n;
  const int64_t nr = n * (cp ? 2 : 1);
  const int G = grid_for(h, nr);
  const int M = (int)std::min<int64_t>(krylovdim, n);
  const int ldh = M + 1;
  DevBuf Vb, zb, part, Hdev, Ed, acc;
  FMPT_TRY(Vb.alloc(h, (size_t)(M + 1) * nr * sizeof(double)));
  FMPT_TRY(zb.alloc(h, (size_t)nr * sizeof(double)));
  FMPT_TRY(part.alloc(h, (size_t)G * sizeof(double)));
  FMPT_TRY(Hdev.alloc(h, (size_t)ldh * M * 2 * sizeof(double)));
  FMPT_TRY(Ed.alloc(h, (size_t)nnodes * M * 2 * sizeof(double)));
  FMPT_TRY(acc.alloc(h, 2 * sizeof(double)));
  FMPT_TRY(ensure_pinned(h, (size_t)ldh * M * 2 + 8));
  DevBuf gsbuf;
  GsWork gs{};
  FMPT_TRY(gs_setup(h, cp, n, M, gsbuf, gs));
  double* V = Vb.d();
  auto V_ = [&](int i) { return V + (int64_t)i * nr; };
  CHAIN(rdot_partial, G, h->stream, nr, x, x, part.d(), nullptr);
  FMPT_LAUNCHED(h);
  CHAIN(normalize_from_parts, G, h->stream, nr, x, V_(0), part.d(), G, acc.d());
  FMPT_LAUNCHED(h);
  FMPT_TRY(arnoldi_basis(op, cp, n, nr, M, ldh, V, zb.d(), Hdev, gs));
  std::vector<double> Hh((size_t)ldh * M * 2);
  FMPT_CUDA(h, cudaMemcpyAsync(h->pinned, Hdev.p, Hdev.bytes, cudaMemcpyDeviceToHost, h->stream));
  FMPT_CUDA(h, cudaStreamSynchronize(h->stream));
  if (gs.fused) FMPT_TRY(gp_check_status(h));       // a fused step that gave up left H invalid
  std::copy(h->pinned, h->pinned + Hh.size(), Hh.begin());
  for (double v : Hh)
    if (!std::isfinite(v)) return set_error(h, FMPT_ERR_NONFINITE, "expm_nodes: NaN");
  int m = M;
  bool happy = M == n;
  for (int j = 0; j < M; j++)
    if (Hh[2 * (j + 1 + (size_t)ldh * j)] == 0.0) { m = j + 1; happy = true; break; }
  // every node's exp(s_q t H_m) e_1 on the host, uploaded in one copy (pageable source:
  // the copy has left it when cudaMemcpyAsync returns)
  std::vector<double> Hs((size_t)m * m * 2), cols((size_t)nnodes * m * 2);
  std::vector<cplx> col;
  double e = 0.0;
  const double hlast = happy ? 0.0 : std::abs(Hh[2 * (m + (size_t)ldh * (m - 1))]);
  for (int q = 0; q < nnodes; q++) {
    const double fr = nodes[q] * t_re, fi = nodes[q] * t_im;
    for (int c = 0; c < m; c++)
      for (int r = 0; r < m; r++) {
        const double hr = Hh[2 * (r + (size_t)ldh * c)], hi = Hh[2 * (r + (size_t)ldh * c) + 1];
        Hs[2 * (r + (size_t)m * c)] = fr * hr - fi * hi;
        Hs[2 * (r + (size_t)m * c) + 1] = fr * hi + fi * hr;
      }
    host_expm_col(m, Hs.data(), col);
    for (int r = 0; r < m; r++) {
      cols[2 * (r + (size_t)m * q)] = col[r].real();
      cols[2 * (r + (size_t)m * q) + 1] = col[r].imag();
    }
    if (!happy) e = std::max(e, hlast * std::abs(col[m - 1]));
  }
  FMPT_CUDA(h, cudaMemcpyAsync(Ed.d(), cols.data(), cols.size() * sizeof(double),
                               cudaMemcpyHostToDevice, h->stream));
  for (int q0 = 0; q0 < nnodes; q0 += 65535) {               // the nodes are the grid's y axis
    CHAIN(combine_basis, dim3(G, std::min(65535, nnodes - q0)), h->stream, cp, n, m, V, nr,
          Ed.d() + (int64_t)2 * m * q0, 2 * m, acc.d(), out + nr * q0, nr);
    FMPT_LAUNCHED(h);
  }
  if (err_est) *err_est = e;
  if (!prec_is_f64(op->precision)) FMPT_TRY(op_tc_check(op));
  if (op->u1 || gs.fused) FMPT_TRY(gp_check_status(op->h));
  return FMPT_OK;
}

}  // extern "C"
