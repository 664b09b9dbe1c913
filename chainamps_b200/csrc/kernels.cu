// Memory-bound kernels of the hot path: block AXPY lists (LeftPart /
// RightPart formation) and the FP64 vector kernels of the device Krylov
// solver.  These are grid-stride loops over a few CTAs per SM.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "internal.h"
#include "kernels.h"

namespace cmps {

namespace {

int grid_for(int64_t n, int threads) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int64_t want = (n + threads - 1) / threads;
  int64_t cap = (int64_t)sms * 8;
  if (want < 1) want = 1;
  return (int)(want < cap ? want : cap);
}

// One CTA per destination block; dst = sum_t w_t src_t (dst += ... when
// `accumulate`).
__global__ void k_block_axpy(const AxpyBlock* __restrict__ blocks, const AxpyTerm* __restrict__ terms,
                             const double* __restrict__ sr, const double* __restrict__ si,
                             double* __restrict__ dr, double* __restrict__ di, int accumulate) {
  const AxpyBlock b = blocks[blockIdx.x];
  for (int64_t e = threadIdx.x; e < b.len; e += blockDim.x) {
    double xr = 0.0, xi = 0.0;
    for (int t = b.t0; t < b.t1; ++t) {
      const AxpyTerm tm = terms[t];
      double vr = sr[tm.src_off + e], vi = si[tm.src_off + e];
      xr += tm.wr * vr - tm.wi * vi;
      xi += tm.wr * vi + tm.wi * vr;
    }
    if (accumulate) {
      xr += dr[b.dst_off + e];
      xi += di[b.dst_off + e];
    }
    dr[b.dst_off + e] = xr;
    di[b.dst_off + e] = xi;
  }
}

// ---- Krylov vector kernels (planar FP64 vectors of length n) ----------------
constexpr int RED_THREADS = 256;

// partial[j][blk] = sum_i conj(V_j[i]) * w[i] over this CTA's slice, j < k.
__global__ void k_multidot(const double* __restrict__ Vr, const double* __restrict__ Vi, int64_t ldv,
                           int k, const double* __restrict__ wr, const double* __restrict__ wi, int64_t n,
                           double* __restrict__ partial) {
  extern __shared__ double red[];
  for (int j = 0; j < k; ++j) {
    double sr = 0.0, si = 0.0;
    const double* vr = Vr + (int64_t)j * ldv;
    const double* vi = Vi + (int64_t)j * ldv;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
      double ar = vr[i], ai = vi[i], br = wr[i], bi = wi[i];
      sr += ar * br + ai * bi;
      si += ar * bi - ai * br;
    }
    red[threadIdx.x] = sr;
    red[threadIdx.x + blockDim.x] = si;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        red[threadIdx.x] += red[threadIdx.x + s];
        red[threadIdx.x + blockDim.x] += red[threadIdx.x + s + blockDim.x];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      partial[(2 * j) * gridDim.x + blockIdx.x] = red[0];
      partial[(2 * j + 1) * gridDim.x + blockIdx.x] = red[blockDim.x];
    }
    __syncthreads();
  }
}

// out[r] = sum_b partial[r][b], r < rows (one warp-per-row, deterministic order).
__global__ void k_reduce_rows(const double* __restrict__ partial, int nb, int rows, double* __restrict__ out) {
  int r = blockIdx.x;
  if (r >= rows) return;
  __shared__ double red[RED_THREADS];
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[(int64_t)r * nb + b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[r] = red[0];
}

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33;
  return x;
}

__global__ void k_random(double* __restrict__ re, double* __restrict__ im, int64_t n, uint64_t seed) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t a = mix64(seed ^ (2 * (uint64_t)i + 1));
    uint64_t b = mix64(a + 0x9e3779b97f4a7c15ULL);
    re[i] = ((double)(a >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
    im[i] = ((double)(b >> 11) * (1.0 / 9007199254740992.0)) - 0.5;
  }
}

// per-CTA max |x| and its index
__global__ void k_absmax(const double* __restrict__ re, const double* __restrict__ im, int64_t n,
                         double* __restrict__ pval, int64_t* __restrict__ pidx) {
  __shared__ double sv[RED_THREADS];
  __shared__ int64_t si[RED_THREADS];
  double best = -1.0;
  int64_t bi = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double a = re[i] * re[i] + im[i] * im[i];
    if (a > best) { best = a; bi = i; }
  }
  sv[threadIdx.x] = best;
  si[threadIdx.x] = bi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      double o = sv[threadIdx.x + s];
      int64_t oi = si[threadIdx.x + s];
      if (o > sv[threadIdx.x] || (o == sv[threadIdx.x] && oi < si[threadIdx.x])) {
        sv[threadIdx.x] = o;
        si[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    pval[blockIdx.x] = sv[0];
    pidx[blockIdx.x] = si[0];
  }
}

// x *= phase; drop |x| <= thr; FixComplexPrecision (sparse_interface.cpp:28-32)
__global__ void k_phase_drop(double* __restrict__ re, double* __restrict__ im, int64_t n, double pr, double pi,
                             double thr) {
  const double eps = 2.220446049250313e-16;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double a = re[i], b = im[i];
    double xr = a * pr - b * pi, xi = a * pi + b * pr;
    if (sqrt(xr * xr + xi * xi) > thr) {
      if (fabs(xi / xr) < eps) xi = 0.0;
      else if (fabs(xr / xi) < eps) xr = 0.0;
    } else {
      xr = 0.0;
      xi = 0.0;
    }
    re[i] = xr;
    im[i] = xi;
  }
}

// y = sum_j c_j V_j (c real)
__global__ void k_combine(const double* __restrict__ Vr, const double* __restrict__ Vi, int64_t ldv, int k,
                          const double* __restrict__ c, double* __restrict__ yr, double* __restrict__ yi, int64_t n) {
  __shared__ double cs[128];
  for (int j = threadIdx.x; j < k; j += blockDim.x) cs[j] = c[j];
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double xr = 0.0, xi = 0.0;
    for (int j = 0; j < k; ++j) {
      xr += cs[j] * Vr[(int64_t)j * ldv + i];
      xi += cs[j] * Vi[(int64_t)j * ldv + i];
    }
    yr[i] = xr;
    yi[i] = xi;
  }
}

// ---- Krylov kernels with device-resident coefficients ----------------------
// The Lanczos loop keeps its coefficients on the device: a projection's
// coefficients are reduced into device memory and read back by the update
// kernel, so one iteration needs no host round trip.
constexpr int KR_THREADS = 256;
constexpr int KR_E = 8;  // elements per thread per tile: w is read once, into registers

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// partial[r][blk]: r = 2j, 2j+1 -> <V_j, w> (re, im) for j < k; r = 2k -> |w|^2.
// One pass over w (held in registers per tile) and one over each V_j.
__global__ void __launch_bounds__(KR_THREADS)
k_mdot(const double* __restrict__ Vr, const double* __restrict__ Vi, int64_t ldv, int k,
       const double* __restrict__ wr, const double* __restrict__ wi, int64_t n, double* __restrict__ partial) {
  extern __shared__ double acc[];  // [warps][2k + 1], one row per warp: no shared-memory atomics
  const int nw = KR_THREADS / 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = 2 * k + 1;
  for (int t = threadIdx.x; t < nw * rows; t += blockDim.x) acc[t] = 0.0;
  __syncthreads();
  const int64_t tile = (int64_t)KR_THREADS * KR_E;
  for (int64_t base = (int64_t)blockIdx.x * tile; base < n; base += (int64_t)gridDim.x * tile) {
    double xr[KR_E], xi[KR_E];
    double s = 0.0;
#pragma unroll
    for (int e = 0; e < KR_E; ++e) {
      const int64_t i = base + (int64_t)e * KR_THREADS + threadIdx.x;
      xr[e] = i < n ? wr[i] : 0.0;
      xi[e] = i < n ? wi[i] : 0.0;
      s += xr[e] * xr[e] + xi[e] * xi[e];
    }
    s = warp_sum(s);
    if (lane == 0) acc[warp * rows + 2 * k] += s;
    for (int j = 0; j < k; ++j) {
      const double* vr = Vr + (int64_t)j * ldv;
      const double* vi = Vi + (int64_t)j * ldv;
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int e = 0; e < KR_E; ++e) {
        const int64_t i = base + (int64_t)e * KR_THREADS + threadIdx.x;
        if (i < n) {
          const double ar = vr[i], ai = vi[i];
          sr += ar * xr[e] + ai * xi[e];
          si += ar * xi[e] - ai * xr[e];
        }
      }
      sr = warp_sum(sr);
      si = warp_sum(si);
      if (lane == 0) {
        acc[warp * rows + 2 * j] += sr;
        acc[warp * rows + 2 * j + 1] += si;
      }
    }
  }
  __syncthreads();
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += acc[w * rows + r];
    partial[(int64_t)r * gridDim.x + blockIdx.x] = t;
  }
}

// w -= sum_j h_j V_j (h complex, on the device); partial[blk] = |w|^2 over
// this CTA's elements afterwards.
__global__ void __launch_bounds__(KR_THREADS)
k_maxpy_norm(const double* __restrict__ Vr, const double* __restrict__ Vi, int64_t ldv, int k,
             const double* __restrict__ h, double* __restrict__ wr, double* __restrict__ wi, int64_t n,
             double* __restrict__ partial) {
  __shared__ double hs[2 * 128];
  __shared__ double red[KR_THREADS / 32];
  for (int j = threadIdx.x; j < 2 * k; j += blockDim.x) hs[j] = h[j];
  __syncthreads();
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double xr = wr[i], xi = wi[i];
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
      const double hr = hs[2 * j], hi = hs[2 * j + 1];
      const double vr = Vr[(int64_t)j * ldv + i], vi = Vi[(int64_t)j * ldv + i];
      xr -= hr * vr - hi * vi;
      xi -= hr * vi + hi * vr;
    }
    wr[i] = xr;
    wi[i] = xi;
    s += xr * xr + xi * xi;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < KR_THREADS / 32; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// ---- One Lanczos step in three passes ---------------------------------------
// The basis is kept unnormalised: vector i is U_i = V_i / s_i with the scale
// s_i = 1 / |U_i| on the device (LanczosCoef::scale), so that no pass only
// rescales.  With w = s_j y, y = H U_j, or w = y, y = H V_j (`unit`),
//   dot     a = <V_j, w>
//   mdot    w' = w - beta_{j-1} V_{j-1} - a V_j;  h_i = <V_i, w'>, i <= j
//   update  U_{j+1} = w' - sum_i h_i V_i;  beta_j = |U_{j+1}|, alpha_j = a + h_j
// w' is formed again in `update` from the same operands by the same
// operations (local_step: explicit fused multiply-adds), so it is never
// stored.  Per step the passes read 2 + (j + 2) + (j + 2) vectors and write
// one: 16 (2 j + 7) n bytes.
// These passes are bound by HBM.  Each CTA works on tiles of 512 P elements in
// 16-byte loads (8-byte ones where n is odd and the imaginary plane starts
// between two 16-byte boundaries), eight of them in flight per thread and
// vector; `mdot` keeps one partial sum per thread and vector in shared memory,
// because a warp reduction per tile and vector took as long as the loads.
// The partial sums are added by the last CTA to finish, in a fixed order.
// Before (five passes, 8-byte loads): 3.0 to 4.2 TB/s of 16 (2 j + 13) n bytes,
// 90 ms of a ladder step at chi = 512 and 121 ms of an Ising step at chi = 64.
// In three passes with the basis in ascending order: 54 and 75 ms.  U_j and
// U_{j-1}, read for w', are first in the sums over the basis too, while the
// CTA's tile of them is in L1 or L2, and `update` walks the tiles from the end,
// where `mdot` stopped: 5.5 to 6 TB/s, mdot + update 47.7 -> 43.9 ms of the
// ladder step and 0.588 -> 0.557 ms per step of the Ising one.
template <bool V2>
__device__ __forceinline__ double2 load2(const double* __restrict__ p, int64_t i, int64_t n) {
  if (V2) return i < n ? *reinterpret_cast<const double2*>(p + i) : double2{0.0, 0.0};
  return double2{i < n ? p[i] : 0.0, i + 1 < n ? p[i + 1] : 0.0};
}
template <bool V2>
__device__ __forceinline__ void store2(double* __restrict__ p, int64_t i, int64_t n, double2 v) {
  if (V2) {
    if (i < n) *reinterpret_cast<double2*>(p + i) = v;
  } else {
    if (i < n) p[i] = v.x;
    if (i + 1 < n) p[i + 1] = v.y;
  }
}

// x + i y of one element: w' = s y - b p - (ar + i ai) v
__device__ __forceinline__ void local_step(double& xr, double& xi, double s, double b, double pr, double pi, double ar,
                                           double ai, double vr, double vi) {
  xr = __fma_rn(-b, pr, __dmul_rn(s, xr));
  xi = __fma_rn(-b, pi, __dmul_rn(s, xi));
  xr = __fma_rn(ai, vi, __fma_rn(-ar, vr, xr));
  xi = __fma_rn(-ai, vr, __fma_rn(-ar, vi, xi));
}

// The rows of partial sums of a launch (partial[row][CTA]), added up by the
// CTA that finishes last; true in its threads, with out[row] visible to them.
__device__ __forceinline__ bool add_partials(const double* __restrict__ partial, int rows, double* __restrict__ out,
                                             unsigned* __restrict__ count) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int r = threadIdx.x >> 5; r < rows; r += KR_THREADS / 32) {
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < (int)gridDim.x; b += 32) s += __ldcg(partial + (int64_t)r * gridDim.x + b);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) out[r] = s;
  }
  if (threadIdx.x == 0) *count = 0u;  // for the next launch on the stream
  __syncthreads();
  return true;
}

// a = <s_j U_j, w>, scaled before the products: U_j and y have H's size, and
// their squares are as large as a double needs to hold
template <bool V2, int P>
__global__ void __launch_bounds__(KR_THREADS, 2)
k_lanczos_dot(const double* __restrict__ ur, const double* __restrict__ ui, const double* __restrict__ yr,
              const double* __restrict__ yi, int64_t n, bool unit, int j, LanczosCoef c,
              double* __restrict__ partial, unsigned* __restrict__ count) {
  __shared__ double red[2][KR_THREADS / 32];
  grid_wait();
  const double su = c.scale[j], sy = unit ? 1.0 : su;
  double sr = 0.0, si = 0.0;
  const int64_t tile = (int64_t)KR_THREADS * 2 * P;
  for (int64_t base = (int64_t)blockIdx.x * tile; base < n; base += (int64_t)gridDim.x * tile) {
    double2 a[P], b[P], x[P], y[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int64_t i = base + (int64_t)(p * KR_THREADS + threadIdx.x) * 2;
      a[p] = load2<V2>(ur, i, n);
      b[p] = load2<V2>(ui, i, n);
      x[p] = load2<V2>(yr, i, n);
      y[p] = load2<V2>(yi, i, n);
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      a[p].x *= su, a[p].y *= su, b[p].x *= su, b[p].y *= su;
      x[p].x *= sy, x[p].y *= sy, y[p].x *= sy, y[p].y *= sy;
      sr += a[p].x * x[p].x + b[p].x * y[p].x + a[p].y * x[p].y + b[p].y * y[p].y;
      si += a[p].x * y[p].x - b[p].x * x[p].x + a[p].y * y[p].y - b[p].y * x[p].y;
    }
  }
  sr = warp_sum(sr);
  si = warp_sum(si);
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = sr;
    red[1][threadIdx.x >> 5] = si;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double t = 0.0;
    for (int w = 0; w < KR_THREADS / 32; ++w) t += red[threadIdx.x][w];
    partial[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
  add_partials(partial, 2, c.a, count);
}

// h_i = s_i <U_i, w'> for c0 <= i < c1; U_i at U + i ldv (re; im n further)
template <bool V2, int P>
__global__ void __launch_bounds__(KR_THREADS, 2)
k_lanczos_mdot(const double* __restrict__ U, int64_t ldv, const double* __restrict__ yr,
               const double* __restrict__ yi, int64_t n, bool unit, int j, int c0, int c1, LanczosCoef c,
               double* __restrict__ partial, unsigned* __restrict__ count) {
  extern __shared__ double2 dots[];  // [c1 - c0][KR_THREADS]
  const int tid = threadIdx.x;
  grid_wait();
  for (int i = 0; i < c1 - c0; ++i) dots[i * KR_THREADS + tid] = double2{0.0, 0.0};
  const double s = unit ? 1.0 : c.scale[j], b = j > 0 ? c.beta[j - 1] * c.scale[j - 1] : 0.0;
  const double ar = c.a[0] * c.scale[j], ai = c.a[1] * c.scale[j];
  const double* uj = U + (int64_t)j * ldv;
  const double* up = j > 0 ? uj - ldv : uj;
  const int64_t tile = (int64_t)KR_THREADS * 2 * P;
  for (int64_t base = (int64_t)blockIdx.x * tile; base < n; base += (int64_t)gridDim.x * tile) {
    double2 x[P], y[P];
    const int64_t i0 = base + (int64_t)tid * 2;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
      x[p] = load2<V2>(yr, i, n);
      y[p] = load2<V2>(yi, i, n);
    }
    double2 v[P], u[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
      v[p] = load2<V2>(uj, i, n);
      u[p] = load2<V2>(uj + n, i, n);
      const double2 pr = load2<V2>(up, i, n), pi = load2<V2>(up + n, i, n);
      local_step(x[p].x, y[p].x, s, b, pr.x, pi.x, ar, ai, v[p].x, u[p].x);
      local_step(x[p].y, y[p].y, s, b, pr.y, pi.y, ar, ai, v[p].y, u[p].y);
    }
#pragma unroll 2
    for (int q = c1 - 1; q >= c0; --q) {
      const double* vq = U + (int64_t)q * ldv;
      double2 t{0.0, 0.0};
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
        v[p] = load2<V2>(vq, i, n);
        u[p] = load2<V2>(vq + n, i, n);
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        t.x += v[p].x * x[p].x + u[p].x * y[p].x + v[p].y * x[p].y + u[p].y * y[p].y;
        t.y += v[p].x * y[p].x - u[p].x * x[p].x + v[p].y * y[p].y - u[p].y * x[p].y;
      }
      double2& a = dots[(q - c0) * KR_THREADS + tid];
      a.x += t.x;
      a.y += t.y;
    }
  }
  __syncthreads();
  for (int q = tid >> 5; q < c1 - c0; q += KR_THREADS / 32) {
    double2 t{0.0, 0.0};
    for (int l = tid & 31; l < KR_THREADS; l += 32) {
      const double2 a = dots[q * KR_THREADS + l];
      t.x += a.x;
      t.y += a.y;
    }
    t.x = warp_sum(t.x);
    t.y = warp_sum(t.y);
    if ((tid & 31) == 0) {
      partial[(int64_t)(2 * q) * gridDim.x + blockIdx.x] = t.x;
      partial[(int64_t)(2 * q + 1) * gridDim.x + blockIdx.x] = t.y;
    }
  }
  if (add_partials(partial, 2 * (c1 - c0), c.h + 2 * c0, count))
    for (int r = tid; r < 2 * (c1 - c0); r += KR_THREADS) c.h[2 * c0 + r] *= c.scale[c0 + r / 2];
}

// U_{j+1} = w' - sum_{i <= j} h_i s_i U_i into (outr, outi), or nowhere if null
// (a cycle's last step needs its norm only); then the step's coefficients,
// which the host reads from `host` (pinned) after the stream has come this far.
template <bool V2, int P>
__global__ void __launch_bounds__(KR_THREADS, 2)
k_lanczos_update(const double* __restrict__ U, int64_t ldv, const double* __restrict__ yr,
                 const double* __restrict__ yi, int64_t n, bool unit, int j, double* __restrict__ outr,
                 double* __restrict__ outi, LanczosCoef c, double* __restrict__ partial,
                 unsigned* __restrict__ count, double* __restrict__ host) {
  __shared__ double2 hs[128];
  __shared__ double red[KR_THREADS / 32];
  const int tid = threadIdx.x;
  grid_wait();
  for (int i = tid; i <= j; i += KR_THREADS)
    hs[i] = double2{c.h[2 * i] * c.scale[i], c.h[2 * i + 1] * c.scale[i]};
  const double s = unit ? 1.0 : c.scale[j], b = j > 0 ? c.beta[j - 1] * c.scale[j - 1] : 0.0;
  const double ar = c.a[0] * c.scale[j], ai = c.a[1] * c.scale[j];
  __syncthreads();
  const double* uj = U + (int64_t)j * ldv;
  const double* up = j > 0 ? uj - ldv : uj;
  double nrm = 0.0;
  const int64_t tile = (int64_t)KR_THREADS * 2 * P;
  // from the end: what `mdot` read last may still be in L2
  for (int64_t base = (n - 1) / tile * tile - (int64_t)blockIdx.x * tile; base >= 0; base -= (int64_t)gridDim.x * tile) {
    double2 x[P], y[P];
    const int64_t i0 = base + (int64_t)tid * 2;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
      x[p] = load2<V2>(yr, i, n);
      y[p] = load2<V2>(yi, i, n);
      const double2 v = load2<V2>(uj, i, n), u = load2<V2>(uj + n, i, n);
      const double2 pr = load2<V2>(up, i, n), pi = load2<V2>(up + n, i, n);
      local_step(x[p].x, y[p].x, s, b, pr.x, pi.x, ar, ai, v.x, u.x);
      local_step(x[p].y, y[p].y, s, b, pr.y, pi.y, ar, ai, v.y, u.y);
    }
#pragma unroll 2
    for (int q = j; q >= 0; --q) {
      const double* vq = U + (int64_t)q * ldv;
      const double2 h = hs[q];
      double2 v[P], u[P];
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
        v[p] = load2<V2>(vq, i, n);
        u[p] = load2<V2>(vq + n, i, n);
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        x[p].x -= h.x * v[p].x - h.y * u[p].x;
        y[p].x -= h.x * u[p].x + h.y * v[p].x;
        x[p].y -= h.x * v[p].y - h.y * u[p].y;
        y[p].y -= h.x * u[p].y + h.y * v[p].y;
      }
    }
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const int64_t i = i0 + (int64_t)p * KR_THREADS * 2;
      if (outr) {
        store2<V2>(outr, i, n, x[p]);
        store2<V2>(outi, i, n, y[p]);
      }
      nrm += x[p].x * x[p].x + y[p].x * y[p].x + x[p].y * x[p].y + y[p].y * y[p].y;
    }
  }
  nrm = warp_sum(nrm);
  if ((tid & 31) == 0) red[tid >> 5] = nrm;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < KR_THREADS / 32; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
  if (add_partials(partial, 1, c.nrm2, count) && tid == 0) {
    const double a = c.a[0] + c.h[2 * j];
    const double be = sqrt(fmax(0.0, *c.nrm2));
    c.beta[j] = be;
    // an exhausted Krylov space: the next basis vector counts as zero
    c.scale[j + 1] = be > 1e-14 * fmax(1.0, fabs(a)) ? 1.0 / be : 0.0;
    host[0] = a;
    host[1] = be;
    __threadfence_system();
  }
}

// y = x / sqrt(*p), 0 when *p is not positive.
__global__ void k_scale_dev(const double* __restrict__ xr, const double* __restrict__ xi,
                            const double* __restrict__ p, double* __restrict__ yr, double* __restrict__ yi,
                            int64_t n) {
  const double v = *p;
  const double s = v > 0.0 ? 1.0 / sqrt(v) : 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    yr[i] = s * xr[i];
    yi[i] = s * xi[i];
  }
}

}  // namespace

int launch_block_axpy(const AxpyBlock* d_blocks, int nblocks, const AxpyTerm* d_terms, const Planar& src,
                      Planar& dst, cudaStream_t st, bool accumulate) {
  if (nblocks == 0) return CMPS_OK;
  k_block_axpy<<<nblocks, 256, 0, st>>>(d_blocks, d_terms, src.re(), src.im(), dst.re(), dst.im(), accumulate ? 1 : 0);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

// ---- Krylov helpers ---------------------------------------------------------
int VecOps::init(int64_t n_, cudaStream_t st) {
  n = n_;
  nb = grid_for(n, RED_THREADS);
  if (nb > 1024) nb = 1024;
  CMPS_CUDA(dmalloc(&d_partial, sizeof(double) * (2 * 128 + 2) * nb));
  CMPS_CUDA(dmalloc(&d_coef, sizeof(double) * kCoefDoubles));
  CMPS_CUDA(dmalloc(&d_small, sizeof(double) * 2 * 128 * 2));
  CMPS_CUDA(dmalloc(&d_pidx, sizeof(int64_t) * nb));
  CMPS_CUDA(dmalloc(&d_count, sizeof(unsigned)));
  return zero_wait(d_count, sizeof(unsigned), st);
}

void VecOps::release() {
  if (d_partial) dfree(d_partial);
  if (d_small) dfree(d_small);
  if (d_pidx) dfree(d_pidx);
  if (d_coef) dfree(d_coef);
  if (d_count) dfree(d_count);
  d_count = nullptr;
  d_partial = d_small = d_coef = nullptr;
  d_pidx = nullptr;
}

int VecOps::multidot(const double* Vr, const double* Vi, int64_t ldv, int k, const double* wr, const double* wi,
                     double* h_host, cudaStream_t st) {
  if (k > 128) return fail(CMPS_ERR_ARG, "krylov dimension above 128");
  k_multidot<<<nb, RED_THREADS, 2 * RED_THREADS * sizeof(double), st>>>(Vr, Vi, ldv, k, wr, wi, n, d_partial);
  CMPS_CUDA(cudaGetLastError());
  k_reduce_rows<<<2 * k, RED_THREADS, 0, st>>>(d_partial, nb, 2 * k, d_small);
  CMPS_CUDA(cudaGetLastError());
  if (h_host) {
    CMPS_CUDA(cudaMemcpyAsync(h_host, d_small, sizeof(double) * 2 * k, cudaMemcpyDeviceToHost, st));
    CMPS_CUDA(cudaStreamSynchronize(st));
  }
  return CMPS_OK;
}

int VecOps::norm2(const double* xr, const double* xi, double* out, cudaStream_t st) {
  double h[2];
  CMPS_TRY(multidot(xr, xi, 0, 1, xr, xi, h, st));
  *out = h[0];
  return CMPS_OK;
}

int VecOps::random(double* re, double* im, uint64_t seed, cudaStream_t st) {
  k_random<<<grid_for(n, 256), 256, 0, st>>>(re, im, n, seed);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

int VecOps::combine(const double* Vr, const double* Vi, int64_t ldv, int k, const double* c_host, double* yr,
                    double* yi, cudaStream_t st) {
  if (k > 128) return fail(CMPS_ERR_ARG, "krylov dimension above 128");
  CMPS_CUDA(cudaMemcpyAsync(d_small + 256, c_host, sizeof(double) * k, cudaMemcpyHostToDevice, st));
  k_combine<<<grid_for(n, 256), 256, 0, st>>>(Vr, Vi, ldv, k, d_small + 256, yr, yi, n);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

int VecOps::absmax(const double* re, const double* im, double* val, int64_t* idx, cudaStream_t st) {
  k_absmax<<<nb, RED_THREADS, 0, st>>>(re, im, n, d_partial, d_pidx);
  CMPS_CUDA(cudaGetLastError());
  std::vector<double> pv(nb);
  std::vector<int64_t> pi(nb);
  CMPS_CUDA(cudaMemcpyAsync(pv.data(), d_partial, sizeof(double) * nb, cudaMemcpyDeviceToHost, st));
  CMPS_CUDA(cudaMemcpyAsync(pi.data(), d_pidx, sizeof(int64_t) * nb, cudaMemcpyDeviceToHost, st));
  CMPS_CUDA(cudaStreamSynchronize(st));
  double best = -1.0;
  int64_t bi = 0;
  for (int b = 0; b < nb; ++b)
    if (pv[b] > best || (pv[b] == best && pi[b] < bi)) {
      best = pv[b];
      bi = pi[b];
    }
  *val = best;
  *idx = bi;
  return CMPS_OK;
}

int VecOps::phase_drop(double* re, double* im, double pr, double pi, double thr, cudaStream_t st) {
  k_phase_drop<<<grid_for(n, 256), 256, 0, st>>>(re, im, n, pr, pi, thr);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

int VecOps::mdot_dev(const double* Vr, const double* Vi, int64_t ldv, int k, const double* wr, const double* wi,
                     double* d_out, cudaStream_t st) {
  if (k < 0 || k > 128) return fail(CMPS_ERR_ARG, "krylov dimension above 128");
  const int64_t tile = (int64_t)KR_THREADS * KR_E;
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(nb, (n + tile - 1) / tile));
  const int rows = 2 * k + 1;
  const size_t smem = sizeof(double) * (KR_THREADS / 32) * rows;
  k_mdot<<<g, KR_THREADS, smem, st>>>(Vr, Vi, ldv, k, wr, wi, n, d_partial);
  CMPS_CUDA(cudaGetLastError());
  k_reduce_rows<<<rows, RED_THREADS, 0, st>>>(d_partial, g, rows, d_out);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

int VecOps::maxpy_norm_dev(const double* Vr, const double* Vi, int64_t ldv, int k, const double* d_h, double* wr,
                           double* wi, double* d_nrm2, cudaStream_t st) {
  if (k < 0 || k > 128) return fail(CMPS_ERR_ARG, "krylov dimension above 128");
  const int g = std::min(nb, grid_for(n, KR_THREADS));
  k_maxpy_norm<<<g, KR_THREADS, 0, st>>>(Vr, Vi, ldv, k, d_h, wr, wi, n, d_partial);
  CMPS_CUDA(cudaGetLastError());
  k_reduce_rows<<<1, RED_THREADS, 0, st>>>(d_partial, g, 1, d_nrm2);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

LanczosCoef VecOps::lanczos_coef() const {
  double* p = d_coef;
  return LanczosCoef{p, p + 8, p + 280, p + 408, p + 544};
}

// Tiles of 512 or 2048 elements: the small ones spread a short vector (the
// XXZ chain's few thousand entries) over more CTAs; two CTAs per SM at most.
template <bool V2, int P>
static int lanczos_step(const VecOps& o, const double* U, int64_t ldv, const double* yr, const double* yi, bool unit,
                        int j, double* outr, double* outi, double* host, cudaStream_t st) {
  const LanczosCoef c = o.lanczos_coef();
  const int64_t tiles = (o.n + (int64_t)KR_THREADS * 2 * P - 1) / ((int64_t)KR_THREADS * 2 * P);
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(std::min(o.nb, 296), tiles));
  const double* uj = U + (int64_t)j * ldv;
  CMPS_CUDA(launch_chained(k_lanczos_dot<V2, P>, dim3(g), dim3(KR_THREADS), 0, st, uj, uj + o.n, yr, yi, o.n, unit, j, c,
                           o.d_partial, o.d_count));
  constexpr int kChunk = 24;  // vectors per launch of the products: 96 KB of partial sums
  CMPS_TRY(ensure_smem_optin((const void*)k_lanczos_mdot<V2, P>, kChunk * KR_THREADS * (int)sizeof(double2)));
  for (int c0 = 0; c0 <= j; c0 += kChunk) {
    const int c1 = std::min(j + 1, c0 + kChunk);
    CMPS_CUDA(launch_chained(k_lanczos_mdot<V2, P>, dim3(g), dim3(KR_THREADS),
                             (size_t)(c1 - c0) * KR_THREADS * sizeof(double2), st, U, ldv, yr, yi, o.n, unit, j, c0, c1, c,
                             o.d_partial, o.d_count));
  }
  CMPS_CUDA(launch_chained(k_lanczos_update<V2, P>, dim3(g), dim3(KR_THREADS), 0, st, U, ldv, yr, yi, o.n, unit, j, outr,
                           outi, c, o.d_partial, o.d_count, host));
  return CMPS_OK;
}

int VecOps::lanczos(const double* U, int64_t ldv, const double* yr, const double* yi, bool unit, int j, double* outr,
                    double* outi, double* host, cudaStream_t st) {
  if (j < 0 || j > 126) return fail(CMPS_ERR_ARG, "krylov dimension above 127");
  const bool even = n % 2 == 0 && ldv % 2 == 0 &&
                    (((uintptr_t)U | (uintptr_t)yr | (uintptr_t)yi | (uintptr_t)outr | (uintptr_t)outi) & 15) == 0;
  const bool wide = n >= (int64_t)148 * 2 * 2048;
  if (even && wide) return lanczos_step<true, 4>(*this, U, ldv, yr, yi, unit, j, outr, outi, host, st);
  if (even) return lanczos_step<true, 1>(*this, U, ldv, yr, yi, unit, j, outr, outi, host, st);
  if (wide) return lanczos_step<false, 4>(*this, U, ldv, yr, yi, unit, j, outr, outi, host, st);
  return lanczos_step<false, 1>(*this, U, ldv, yr, yi, unit, j, outr, outi, host, st);
}

int VecOps::scale_dev(const double* xr, const double* xi, const double* d_sq, double* yr, double* yi, cudaStream_t st) {
  k_scale_dev<<<grid_for(n, 256), 256, 0, st>>>(xr, xi, d_sq, yr, yi, n);
  CMPS_CUDA(cudaGetLastError());
  return CMPS_OK;
}

}  // namespace cmps
