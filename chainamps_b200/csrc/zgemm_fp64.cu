// Grouped complex-double GEMM on the FP64 tensor path (DMMA, mma.sync
// m8n8k4 f64) for sm_100a.
//
// One launch runs a whole list of independent output tiles.  Each output
// region ("task") is C = sum over its terms of op(A_t) op(B_t), where every
// term has its own A block, B block and K -- the K-concatenation that turns
// the charge-sector structure of H_eff (sum over MPO indices and physical
// states) into a single accumulation.  Complex operands are stored as two
// planes (re, im) of one allocation.  op(A) is A or A^H (A stored K x M),
// op(B) is B or B^H (B stored N x K), all row-major with leading dimensions.
// NSPLIT: the N index of B and C is two-level (GemmTask::n_in), so one task
// can run over several equally strided column ranges, e.g. the rows of
// every state of one charge class, or one column class of every row.
//
// The FP64 pipe (36.6 TFLOP/s measured for DMMA alone) is the bound of every
// plan whose blocks are not tiny: a DMMA holds its sub-core's pipe for 16
// cycles, so what counts is how many DMMAs are issued, and that there is
// always a warp ready to issue one.
//  * Trimmed tiles.  Charge sectors have any size (2, 9, 27, 61, 99, 117 on
//    the ladder at chi = 512), so whole 64 x 64 tiles did 1.40 x the useful
//    work there, 2.5 x on 40 uneven sectors and 4.5 x on the XXZ chain.  A
//    tile therefore carries its own number of 8-row and 8-column slices, a
//    task is cut into tiles of equal slice counts, K is run in steps of 4,
//    and the slices of a tile are dealt out evenly over its four warps in
//    the best of the arrangements 4 x 1, 2 x 2, 1 x 4 (GemmTile::cut).  The
//    work then is 1.07 x, 1.13 x and 1.09 x the useful one.
//  * Four products per complex one, Re = Ar Br - Ai Bi and Im = Ar Bi + Ai Br,
//    each component from its own terms alone.  Three multiplications (Im from
//    (Ar + Ai)(Br + Bi) less the other two) would be a quarter fewer DMMAs, but
//    leave the rounding error of the real products in an imaginary part that
//    may be many orders smaller: with Im / Re = 1e-8 in both operands its
//    relative error is 1e-7 instead of 1e-15, and eigenvectors whose phase is
//    fixed are nearly real.  The sums are folded into the result every kFold
//    values of K, so that rounding errors do not grow along all of K.
//  * AREAL: a plan whose A operand has no imaginary part (the MPO blocks of
//    real operators) needs two products, Ar Br and Ar Bi, and no folding.
//  * Four CTAs of four warps per SM, each with a ring of three 16 KB stages
//    filled by 8-byte cp.async (block offsets and leading dimensions have any
//    parity) and one barrier per 16 values of K.
// Against whole 64 x 64 tiles with two CTAs per SM, per matvec: ladder at chi =
// 512 11.9 and 8.7 ms (the zero parts of T, which the plans leave out, are a
// fifth of that), Ising chains at chi = 64 10.9 and 6.1 ms, 40 uneven sectors 3.4
// and 1.56 ms.  The same kernel with three multiplications took 7.7, 5.8 and
// 1.43 ms.  A loop of this shape on registers reaches 36.9 TFLOP/s, with
// fragment reads from shared memory 36.1; the rest goes to operand loads,
// their addresses and the slices that the busiest warp has more.
//
// An element's value does not depend on the tile shape or on how tasks are
// cut: the order of its DMMAs and folds is fixed by its terms alone.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "internal.h"

namespace cmps {

namespace {

// Output tile of up to BM x BN, a warp holds at most WI x WJ slices of 8 x 8.
// An operand is staged as it is stored, unpadded: rows of 16 values of K, or
// rows of BM / BN elements per value of K.  The position inside a row is
// XORed with 4 * (row mod 4), which makes the 8-byte fragment reads free of
// bank conflicts and keeps four 48 KB rings on an SM.
constexpr int BK = 16;
constexpr int NTHREADS = 128;
constexpr int STAGES = 3;
constexpr int kFold = 128;  // values of K between two folds of the products
template <int BM_, int BN_, int WI_, int WJ_, int CTAS_>
struct Tile {
  static constexpr int BM = BM_, BN = BN_, WI = WI_, WJ = WJ_, CTAS = CTAS_;
  static constexpr int PLANE_A = BM * BK, PLANE_B = BN * BK;  // doubles per plane per stage
  static constexpr int STAGE_DOUBLES = 2 * PLANE_A + 2 * PLANE_B;  // A re, A im, B re, B im
  static constexpr size_t SMEM_BYTES = (size_t)STAGES * STAGE_DOUBLES * sizeof(double);
};
using TileQ = Tile<32, 32, 2, 2, 4>;
using TileS = Tile<32, 16, 2, 1, 4>;  // plans with too few tiles to fill the GPU

__device__ __forceinline__ void cp_async8(unsigned s, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async8z(unsigned s, const double* gmem, bool pred) {
  int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_wait1() { asm volatile("cp.async.wait_group 1;\n" ::); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Offset of column n under the two-level N index (NSPLIT), else n.
template <bool NSPLIT>
__device__ __forceinline__ int64_t ncol(int n, int n_in, int ld_out) {
  if (!NSPLIT) return n;
  const int q = n / n_in;
  return (int64_t)q * ld_out + (n - q * n_in);
}

// One thread's part of an operand's loads into a stage buffer, one element
// of each plane per pass.  KLANE: the lanes of a 16-thread group run along K
// and the passes along the other index, 8 apart (A as stored, B^H); else the
// lanes run along the other index (EXT of them) and the passes along K.
// Elements of rows or columns outside the block are not loaded: they only
// reach outputs that are not stored.  K past the term's end, up to the next
// multiple of 4, is filled with zeros.
template <int EXT, bool KLANE, bool REAL>
struct Loader {
  static constexpr int PASSES = KLANE ? EXT / 8 : BK * EXT / NTHREADS;
  static constexpr int APART = KLANE ? 8 : NTHREADS / EXT;
  static constexpr unsigned PLANE = EXT * BK * sizeof(double);
  static constexpr unsigned SSTEP = APART * (KLANE ? BK : EXT) * sizeof(double);
  const double *re, *im;
  int ld;       // leading dimension of the current term
  int n;        // passes that this thread loads: all whose element exists
  unsigned s;   // where pass 0 lands in the stage buffer
  static __device__ __forceinline__ int lane() { return threadIdx.x % (KLANE ? BK : EXT); }
  static __device__ __forceinline__ int row() { return threadIdx.x / (KLANE ? BK : EXT); }
  // slices: of this tile along the operand's other index; left: elements there
  __device__ __forceinline__ void open_tile(unsigned ring, int slices, int left) {
    const int l = lane(), r = row();
    n = KLANE ? min(slices, (left - r + 7) >> 3) : (l < left && l < 8 * slices ? PASSES : 0);
    s = ring + (r * (KLANE ? BK : EXT) + (l ^ (r & 3) << 2)) * (unsigned)sizeof(double);
  }
  // origin: element (0, 0) of this tile in the term's block; at: this
  // thread's offset from it along the other index when the lanes run there
  __device__ __forceinline__ void open_term(const double* origin, int64_t plane, int ld_, int64_t at) {
    ld = ld_;
    re = origin + (int64_t)row() * ld + (KLANE ? lane() : at);
    if (!REAL) im = re + plane;
  }
  __device__ __forceinline__ void load(unsigned stage, int kl) {
    const unsigned d = s + stage;
    if (kl == BK) {
#pragma unroll
      for (int j = 0; j < PASSES; ++j)
        if (j < n) {
          cp_async8(d + j * SSTEP, re + (int64_t)ld * (APART * j));
          if (!REAL) cp_async8(d + j * SSTEP + PLANE, im + (int64_t)ld * (APART * j));
        }
    } else {
      const int kl4 = (kl + 3) & ~3;
#pragma unroll
      for (int j = 0; j < PASSES; ++j) {
        const int k = KLANE ? lane() : row() + APART * j;
        if (j < n && k < kl4) {
          const int64_t o = k < kl ? (int64_t)ld * (APART * j) : 0;
          cp_async8z(d + j * SSTEP, re + o, k < kl);
          if (!REAL) cp_async8z(d + j * SSTEP + PLANE, im + o, k < kl);
        }
      }
    }
    re += KLANE ? (int64_t)BK : (int64_t)ld * BK;
    if (!REAL) im += KLANE ? (int64_t)BK : (int64_t)ld * BK;
  }
};

// The arrangement of the four warps over a tile of sm x sn slices, 2^wml of
// them along M, with the fewest slice pairs hm x hn on the busiest warp.
template <class T>
__host__ __device__ __forceinline__ void arrange(int sm, int sn, int& hm, int& hn, int& wml) {
  int best = 1 << 20;
  hm = hn = wml = 0;
#pragma unroll
  for (int x = 0; x <= 2; ++x) {
    const int a = (sm + (1 << x) - 1) >> x, b = (sn + (4 >> x) - 1) >> (2 - x);
    if (a <= T::WI && b <= T::WJ && a * b < best) {
      best = a * b;
      hm = a;
      hn = b;
      wml = x;
    }
  }
}

// A warp's accumulators: the result and, unless AREAL, the sums since the last
// fold, Ar Br, Ai Bi and Ar Bi + Ai Br.
template <class T>
struct Acc {
  double cr[T::WI][T::WJ][2], ci[T::WI][T::WJ][2];
  double rr[T::WI][T::WJ][2], ii[T::WI][T::WJ][2], ri[T::WI][T::WJ][2];
};

// One stage of kl values of K for a warp's NI x NJ slices, straight-line.
// WHOLE: kl is BK, without a test per 4 values; the body of nearly all
// stages (chi = 512 ladder: 4.18 + 4.49 -> 4.13 + 4.45 ms per matvec stage,
// chi = 96 sectors 0.804 + 0.772 -> 0.796 + 0.759 ms).
template <class T, bool AH, bool BH, bool AREAL, int NI, int NJ, bool WHOLE = false>
__device__ __forceinline__ void mma_stage(Acc<T>& c, const double* buf, int i0, int j0, int kl) {
  const int lane = threadIdx.x & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const double* sA = buf + (AH ? tig * T::BM : (i0 * 8 + gid) * BK + tig);
  const double* sB = buf + 2 * T::PLANE_A + (BH ? (j0 * 8 + gid) * BK + tig : tig * T::BN);
  const int xk = (gid & 3) << 2, xt = tig << 2;  // the rows' XOR patterns
#pragma unroll
  for (int kk = 0; kk < BK; kk += 4) {
    if (!WHOLE && kk >= kl) break;
    double ar[NI], ai[NI], br[NJ], bi[NJ];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int o = AH ? kk * T::BM + (((i0 + i) * 8 + gid) ^ xt) : 8 * i * BK + (kk ^ xk);
      ar[i] = sA[o];
      if (!AREAL) ai[i] = AH ? -sA[o + T::PLANE_A] : sA[o + T::PLANE_A];
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int o = BH ? 8 * j * BK + (kk ^ xk) : kk * T::BN + (((j0 + j) * 8 + gid) ^ xt);
      br[j] = sB[o];
      bi[j] = BH ? -sB[o + T::PLANE_B] : sB[o + T::PLANE_B];
    }
    // one product of all slice pairs after the other, the two that share an
    // accumulator apart (pair by pair: chi = 512 ladder 8.78 ms instead of 8.69).
    // One accumulator for Re (with -Ai) instead of two makes its chain twice as
    // long: 40 sectors 1.65 ms instead of 1.56; four, one per product, spill.
    auto products = [](double (&d)[T::WI][T::WJ][2], const double (&a)[NI], const double (&b)[NJ]) {
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < NI; ++i) dmma(d[i][j][0], d[i][j][1], a[i], b[j]);
    };
    if constexpr (AREAL) {
      products(c.cr, ar, br);
      products(c.ci, ar, bi);
    } else {
      products(c.rr, ar, br);
      products(c.ri, ar, bi);
      products(c.ii, ai, bi);
      products(c.ri, ai, br);
    }
  }
}

template <class T, bool AH, bool BH, bool NSPLIT, bool AREAL>
__global__ void __launch_bounds__(NTHREADS, T::CTAS)
zgemm_grouped_fp64(const GemmTile* __restrict__ tiles, const GemmTask* __restrict__ tasks,
                   const GemmTerm* __restrict__ terms, const double* __restrict__ Ar, int64_t planeA,
                   const double* __restrict__ Br, int64_t planeB, double* __restrict__ Cr, int64_t planeC) {
  extern __shared__ double smem[];
  const GemmTile tile = tiles[blockIdx.x];
  const GemmTask task = tasks[tile.task];
  const int lane = threadIdx.x & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const int m0 = tile.m0, n0 = tile.n0, sm = tile.cut & 63, sn = tile.cut >> 6 & 63;
  Loader<T::BM, !AH, AREAL> la;
  Loader<T::BN, BH, false> lb;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(smem);
  la.open_tile(ring, sm, task.m - m0);
  lb.open_tile(ring + 2 * T::PLANE_A * (unsigned)sizeof(double), sn, task.n - n0);
  int nq = 0, nr = 0;  // two-level index of this thread's B column
  if (NSPLIT) {
    const int gn = n0 + (int)threadIdx.x % T::BN;
    nq = gn / task.n_in;
    nr = gn - nq * task.n_in;
  }
  // this warp's share of the tile's slices; the warps' roles rotate with the
  // block, so that the larger shares of resident CTAs do not meet on one
  // sub-core
  const int wml = tile.cut >> 12 & 3, hm = tile.cut >> 14 & 63, hn = tile.cut >> 20;
  const int role = ((threadIdx.x >> 5) + blockIdx.x) & 3;
  const int i0 = (role & ((1 << wml) - 1)) * hm, j0 = (role >> wml) * hn;
  const int ni = min(hm, sm - i0), nj = ni > 0 ? min(hn, sn - j0) : 0;

  Acc<T> c;
#pragma unroll
  for (int i = 0; i < T::WI; ++i)
#pragma unroll
    for (int j = 0; j < T::WJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        c.cr[i][j][e] = c.ci[i][j][e] = c.rr[i][j][e] = c.ii[i][j][e] = c.ri[i][j][e] = 0.0;

  // issue cursor over (term, k): fills stage buffer b and returns its values of K
  int it = task.t0, left = 0;
  auto issue = [&](int b) -> int {
    if (left <= 0 && it < task.t1) {
      const GemmTerm t = terms[it++];
      left = t.k;
      la.open_term(Ar + t.a_off + (AH ? (int64_t)m0 : (int64_t)m0 * t.lda), planeA, t.lda, la.lane());
      lb.open_term(Br + t.b_off + (NSPLIT ? 0 : BH ? (int64_t)n0 * t.ldb : (int64_t)n0), planeB, t.ldb,
                   NSPLIT ? (int64_t)nq * t.ldb_out + nr : (int64_t)lb.lane());
    }
    const int kl = max(0, min(BK, left));
    if (kl) {
      const unsigned stage = (unsigned)(b * T::STAGE_DOUBLES * sizeof(double));
      la.load(stage, kl);
      lb.load(stage, kl);
      left -= BK;
    }
    cp_commit();
    return kl;
  };
  grid_wait();  // up to here only the plan was read
  int len0 = issue(0), len1 = issue(1);
  int buf = 0, since = 0;
  while (len0 > 0) {
    cp_wait1();
    __syncthreads();  // stage `buf` has landed for every thread, and the stage refilled below has been read by all
    const int len2 = issue(buf == 0 ? 2 : buf - 1);
    const double* sbuf = smem + buf * T::STAGE_DOUBLES;
    // at most WI x WJ slices, one straight-line body each
    if (nj == 2) {
      if constexpr (T::WJ >= 2) {
        if (ni == 2 && len0 == BK) mma_stage<T, AH, BH, AREAL, 2, 2, true>(c, sbuf, i0, j0, len0);
        else if (ni == 2) mma_stage<T, AH, BH, AREAL, 2, 2>(c, sbuf, i0, j0, len0);
        else mma_stage<T, AH, BH, AREAL, 1, 2>(c, sbuf, i0, j0, len0);
      }
    } else if (nj == 1) {
      if (ni == 2 && len0 == BK) mma_stage<T, AH, BH, AREAL, 2, 1, true>(c, sbuf, i0, j0, len0);
      else if (ni == 2) mma_stage<T, AH, BH, AREAL, 2, 1>(c, sbuf, i0, j0, len0);
      else mma_stage<T, AH, BH, AREAL, 1, 1>(c, sbuf, i0, j0, len0);
    }
    since += len0;
    if (!AREAL && (since >= kFold || len1 == 0)) {
      since = 0;
#pragma unroll
      for (int i = 0; i < T::WI; ++i)
#pragma unroll
        for (int j = 0; j < T::WJ; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            c.cr[i][j][e] += c.rr[i][j][e] - c.ii[i][j][e];
            c.ci[i][j][e] += c.ri[i][j][e];
            c.rr[i][j][e] = c.ii[i][j][e] = c.ri[i][j][e] = 0.0;
          }
    }
    len0 = len1;
    len1 = len2;
    buf = buf == STAGES - 1 ? 0 : buf + 1;
  }
  // epilogue
  const int gm0 = m0 + i0 * 8 + gid, gn0 = n0 + j0 * 8 + 2 * tig;
  const int rows = task.m - gm0, cols = task.n - gn0;
  double* row = Cr + task.c_off + (int64_t)gm0 * task.ldc;
  int64_t col[T::WJ][2];
#pragma unroll
  for (int j = 0; j < T::WJ; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) col[j][e] = ncol<NSPLIT>(gn0 + 8 * j + e, task.n_in, task.ldc_out);
#pragma unroll
  for (int i = 0; i < T::WI; ++i) {
    if (i < ni && 8 * i < rows) {
#pragma unroll
      for (int j = 0; j < T::WJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (j < nj && 8 * j + e < cols) {
            row[col[j][e]] = c.cr[i][j][e];
            row[col[j][e] + planeC] = c.ci[i][j][e];
          }
    }
    row += (int64_t)8 * task.ldc;
  }
}

template <class T, bool AH, bool BH, bool NSPLIT, bool AREAL>
int launch_variant(const GemmPlan& p, const Planar& A, const Planar& B, Planar& C, cudaStream_t st) {
  CMPS_TRY(ensure_smem_optin((const void*)zgemm_grouped_fp64<T, AH, BH, NSPLIT, AREAL>, (int)T::SMEM_BYTES));
  if (p.t64.n <= 0) return CMPS_OK;
  if (p.t64.n > 0x7fffffff) return fail(CMPS_ERR_ARG, "too many GEMM tiles");
  CMPS_CUDA(launch_chained(zgemm_grouped_fp64<T, AH, BH, NSPLIT, AREAL>, dim3((unsigned)p.t64.n), dim3(NTHREADS),
                           T::SMEM_BYTES, st, p.t64.d, p.d_tasks, p.d_terms, A.re(), A.im() - A.re(), B.re(),
                           B.im() - B.re(), C.re(), C.im() - C.re()));
  return CMPS_OK;
}

template <class T>
int launch_shape(const GemmPlan& p, bool a_h, bool b_h, const Planar& A, const Planar& B, Planar& C,
                 cudaStream_t st) {
  if (p.nsplit || p.a_real) {
    if (a_h || b_h) return fail(CMPS_ERR_STATE, "two-level N index or real A with a conjugate-transposed operand");
    if (p.nsplit && p.a_real) return launch_variant<T, false, false, true, true>(p, A, B, C, st);
    if (p.a_real) return launch_variant<T, false, false, false, true>(p, A, B, C, st);
    return launch_variant<T, false, false, true, false>(p, A, B, C, st);
  }
  if (!a_h && !b_h) return launch_variant<T, false, false, false, false>(p, A, B, C, st);
  if (a_h && !b_h) return launch_variant<T, true, false, false, false>(p, A, B, C, st);
  if (!a_h && b_h) return launch_variant<T, false, true, false, false>(p, A, B, C, st);
  return launch_variant<T, true, true, false, false>(p, A, B, C, st);
}

constexpr int kNumShapes64 = 2;
constexpr int kShapes32[3][2] = {{64, 64}, {32, 128}, {128, 32}};

// Tiles of at most `most` slices of 8 along an extent of n.
int parts(int64_t n, int most) { return (int)(((n + 7) / 8 + most - 1) / most); }

}  // namespace

int launch_zgemm_fp64(const GemmPlan& p, bool a_h, bool b_h, const Planar& A, const Planar& B, Planar& C,
                      cudaStream_t st) {
  switch (p.t64.shape) {
    case 0: return launch_shape<TileQ>(p, a_h, b_h, A, B, C, st);
    case 1: return launch_shape<TileS>(p, a_h, b_h, A, B, C, st);
    default: return fail(CMPS_ERR_STATE, "GEMM plan not uploaded (no tile shape)");
  }
}

// A tile's cost in SM cycles: its busiest warp's DMMAs (16 cycles each; two
// or four per slice pair and 4 values of K) or the issue of its loads and
// fragment reads, whichever is more, plus what its epilogue takes.
template <class T>
static double tile_cost(int sm, int sn, double k4, double k16, bool a_real) {
  int hm, hn, wml;
  arrange<T>(sm, sn, hm, hn, wml);
  return std::max(k4 * hm * hn * (a_real ? 32 : 64), 300.0 * k16) + 500.0;
}

template <class T>
static double task_cost(const GemmPlan& p, const GemmTask& t, int64_t* ntiles, double* longest) {
  if (t.m <= 0 || t.n <= 0) return 0.0;
  double k4 = 0.0, k16 = 0.0;
  for (int q = t.t0; q < t.t1; ++q) {
    k4 += (p.terms[q].k + 3) / 4;
    k16 += (p.terms[q].k + BK - 1) / BK;
  }
  const int pm = parts(t.m, T::BM / 8), pn = parts(t.n, T::BN / 8);
  const int sm = ((t.m + 7) / 8 + pm - 1) / pm, sn = ((t.n + 7) / 8 + pn - 1) / pn;
  const double c = tile_cost<T>(sm, sn, k4, k16, p.a_real);
  *ntiles += (int64_t)pm * pn;
  if (c > *longest) *longest = c;
  return c;
}

// Tile shape of a plan in FP64: 32 x 32, or 32 x 16 where the 32 x 32 tiles
// are too few to fill the GPU evenly -- a launch takes the larger of the
// tiles' summed cost over 148 SMs and the longest tile beside the others on
// its SM.  32 x 16 reads each element of A more often, which costs it up to 23%
// on plans of many tiles: both stages in 32 x 32 and in 32 x 16, ladder at chi =
// 512 4.13 + 4.44 and 4.42 + 4.34 ms, 40 uneven sectors 0.79 + 0.91 and 0.82 +
// 0.75 ms, XXZ chain at chi = 250 21 + 51 and 17 + 33 us.  Larger tiles (64 x 32,
// 32 x 64) leave room for two CTAs per SM only and lost to 32 x 32 on nearly
// every plan.
template <class T>
static double launch_cost(const GemmPlan& p) {
  double sum = 0.0, longest = 0.0;
  for (const GemmTask& t : p.tasks) {
    int64_t n = 0;
    const double c = task_cost<T>(p, t, &n, &longest);
    sum += c * (double)n;
  }
  return std::max(sum / 148.0, longest * T::CTAS);
}
static int pick_shape64(const GemmPlan& p) { return launch_cost<TileQ>(p) <= 1.1 * launch_cost<TileS>(p) ? 0 : 1; }

// One block per listed task writes the task's tiles, rows of tiles first: a
// plan has a few thousand tasks and up to some 10^5 tiles.
struct TaskTiles {
  int32_t task, pm, pn, pad;
  int64_t first;
};
template <class T>
__global__ void k_expand_tiles(const TaskTiles* __restrict__ list, const GemmTask* __restrict__ tasks,
                               GemmTile* __restrict__ tiles) {
  const TaskTiles tt = list[blockIdx.x];
  const GemmTask t = tasks[tt.task];
  // slice counts differ by at most one over a task's tiles
  const int64_t sM = (t.m + 7) / 8, sN = (t.n + 7) / 8;
  for (int64_t i = threadIdx.x; i < (int64_t)tt.pm * tt.pn; i += blockDim.x) {
    const int64_t a = i / tt.pn, b = i - a * tt.pn;
    const int64_t ma = sM * a / tt.pm, nb = sN * b / tt.pn;
    const int sm = (int)(sM * (a + 1) / tt.pm - ma), sn = (int)(sN * (b + 1) / tt.pn - nb);
    int hm, hn, wml;
    arrange<T>(sm, sn, hm, hn, wml);
    tiles[tt.first + i] = GemmTile{tt.task, (int32_t)(8 * ma), (int32_t)(8 * nb),
                                   sm | sn << 6 | wml << 12 | hm << 14 | hn << 20};
  }
}

// The plan's tasks in the order of their tiles; returns the number of tiles.
// Tasks with long K come first (in octaves of K, so that tasks sharing operands
// stay neighbours): the launch's last wave is then made of short tiles.
template <class T>
static int64_t tile_list(const GemmPlan& p, std::vector<TaskTiles>& list) {
  std::vector<std::pair<int, TaskTiles>> order;
  order.reserve(p.tasks.size());
  for (size_t i = 0; i < p.tasks.size(); ++i) {
    const GemmTask& t = p.tasks[i];
    if (t.m <= 0 || t.n <= 0) continue;
    int64_t k = 1;
    for (int q = t.t0; q < t.t1; ++q) k += (p.terms[q].k + BK - 1) / BK;
    int oct = 0;
    while (k >>= 1) ++oct;
    order.push_back({-oct, TaskTiles{(int32_t)i, parts(t.m, T::BM / 8), parts(t.n, T::BN / 8), 0, 0}});
  }
  std::stable_sort(order.begin(), order.end(), [](auto& a, auto& b) { return a.first < b.first; });
  list.clear();
  list.reserve(order.size());
  int64_t total = 0;
  for (auto& o : order) {
    o.second.first = total;
    total += (int64_t)o.second.pm * o.second.pn;
    list.push_back(o.second);
  }
  return total;
}
static int64_t tile_list(const GemmPlan& p, int shape, std::vector<TaskTiles>& list) {
  return shape == 0 ? tile_list<TileQ>(p, list) : tile_list<TileS>(p, list);
}

// Writes the tiles of the listed tasks on the device and waits for them: a
// launch may read its tiles before the kernel ahead of it is done (grid_wait).
static int expand_tiles(int shape, const std::vector<TaskTiles>& list, TaskTiles* d_list, const GemmTask* d_tasks,
                        GemmTile* d_tiles, cudaStream_t st) {
  CMPS_CUDA(cudaMemcpyAsync(d_list, list.data(), list.size() * sizeof(TaskTiles), cudaMemcpyHostToDevice, st));
  if (shape == 0) k_expand_tiles<TileQ><<<(unsigned)list.size(), 128, 0, st>>>(d_list, d_tasks, d_tiles);
  else k_expand_tiles<TileS><<<(unsigned)list.size(), 128, 0, st>>>(d_list, d_tasks, d_tiles);
  CMPS_CUDA(cudaGetLastError());
  CMPS_CUDA(cudaStreamSynchronize(st));
  return CMPS_OK;
}

// Tile shape of a plan in FP32 (cgemm_fp32.cu, whole tiles): the shape whose
// padded work (every task rounded up to whole tiles, times its K) plus a
// fixed cost per tile (prologue, epilogue, scheduling: the work of 16 k-steps
// of a 32 x 32 quarter tile) is least.  Ties keep 64 x 64.
static int pick_shape32(const GemmPlan& p) {
  double best = 0.0;
  int shape = 0;
  for (int s = 0; s < 3; ++s) {
    const int bm = kShapes32[s][0], bn = kShapes32[s][1];
    double cost = 0.0;
    for (const GemmTask& t : p.tasks) {
      if (t.m <= 0 || t.n <= 0) continue;
      int64_t k = 0;
      for (int q = t.t0; q < t.t1; ++q) k += p.terms[q].k;
      const double tm = (double)((t.m + bm - 1) / bm), tn = (double)((t.n + bn - 1) / bn);
      cost += tm * tn * ((double)bm * bn * (double)std::max<int64_t>(k, BK) + 16.0 * 32 * 32 * BK);
    }
    if (s == 0 || cost < 0.97 * best) {
      best = cost;
      shape = s;
    }
  }
  return shape;
}

int GemmPlan::retile(bool fp32, int s, cudaStream_t st) {
  if (s < 0 || s >= (fp32 ? 3 : kNumShapes64)) return fail(CMPS_ERR_ARG, "GEMM plan: unknown tile shape");
  if (!d_tasks && !tasks.empty()) return fail(CMPS_ERR_STATE, "GEMM plan not uploaded");
  GemmTiles nt;
  nt.shape = s;
  int rc = CMPS_OK;
  if (!fp32) {
    std::vector<TaskTiles> list;
    nt.n = tile_list(*this, s, list);
    if (nt.n) {
      TaskTiles* d_list = nullptr;
      CMPS_CUDA(dmalloc((void**)&nt.d, (size_t)nt.n * sizeof(GemmTile)));
      if (dmalloc((void**)&d_list, list.size() * sizeof(TaskTiles)) != cudaSuccess)
        rc = fail(CMPS_ERR_CUDA, "GEMM plan: tile list");
      if (rc == CMPS_OK) rc = expand_tiles(s, list, d_list, d_tasks, nt.d, st);
      dfree(d_list);
    }
  } else {
    const int bm = kShapes32[s][0], bn = kShapes32[s][1];
    std::vector<GemmTile> v;
    for (size_t i = 0; i < tasks.size(); ++i)
      for (int m0 = 0; m0 < tasks[i].m; m0 += bm)
        for (int n0 = 0; n0 < tasks[i].n; n0 += bn) v.push_back(GemmTile{(int32_t)i, m0, n0, 0});
    nt.n = (int64_t)v.size();
    if (nt.n) {
      CMPS_CUDA(dmalloc((void**)&nt.d, v.size() * sizeof(GemmTile)));
      rc = copy_wait(nt.d, v.data(), v.size() * sizeof(GemmTile), cudaMemcpyHostToDevice, st);
    }
  }
  if (rc != CMPS_OK) {
    if (nt.d) dfree(nt.d);
    return rc;
  }
  GemmTiles& to = fp32 ? t32 : t64;
  if (to.d && to.d != d_tiles0) dfree(to.d);
  to = nt;
  return CMPS_OK;
}

int GemmPlan::tile_fp32(cudaStream_t st) { return retile(true, pick_shape32(*this), st); }

namespace {
std::mutex g_tune_mu;
std::map<std::vector<int64_t>, int> g_tune_cache;  // plan signature -> measured best shape
}  // namespace

int autotune_plan(GemmPlan& p, int role, bool fp32, const std::function<int()>& run, cudaStream_t st,
                  TuneStats* stats) {
  if (p.tasks.empty()) return CMPS_OK;
  const int heuristic = (fp32 ? p.t32 : p.t64).shape;
  // signature: the role, the task and term counts, the flops to 3 digits and
  // the modelled choice -- plans of the same shape population share it
  double fl = 0.0;
  for (const GemmTask& t : p.tasks)
    for (int q = t.t0; q < t.t1; ++q) fl += 8.0 * t.m * (double)t.n * p.terms[q].k;
  const int64_t fq = fl > 0.0 ? (int64_t)std::llround(std::log10(fl) * 300.0) : 0;
  const std::vector<int64_t> sig{role, (int64_t)p.tasks.size(), (int64_t)p.terms.size(), fq, heuristic};
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tune_cache.find(sig);
    if (it != g_tune_cache.end()) {
      if (stats) ++stats->cached;
      return it->second == heuristic ? CMPS_OK : p.retile(fp32, it->second, st);
    }
  }
  float best = 0.0f, heur = 0.0f;
  int pick = heuristic;
  cudaEvent_t e0, e1;
  CMPS_CUDA(cudaEventCreate(&e0));
  CMPS_CUDA(cudaEventCreate(&e1));
  int rc = CMPS_OK;
  for (int s = 0; s < (fp32 ? 3 : kNumShapes64) && rc == CMPS_OK; ++s) {
    rc = p.retile(fp32, s, st);
    if (rc == CMPS_OK) rc = run();  // warm-up
    if (rc != CMPS_OK) break;
    cudaEventRecord(e0, st);
    for (int r = 0; r < 3 && rc == CMPS_OK; ++r) rc = run();
    cudaEventRecord(e1, st);
    if (rc != CMPS_OK || cudaEventSynchronize(e1) != cudaSuccess) {
      if (rc == CMPS_OK) rc = fail(CMPS_ERR_CUDA, "autotune: timing failed");
      break;
    }
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (s == heuristic) heur = ms;
    if (s == 0 || ms < best) {
      best = ms;
      pick = s;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  CMPS_TRY(rc);
  CMPS_TRY(p.retile(fp32, pick, st));
  if (std::getenv("CMPS_TUNE_TRACE"))
    std::fprintf(stderr, "autotune role %d: tasks %zu, heuristic shape %d %.3f ms, best shape %d %.3f ms\n", role,
                 p.tasks.size(), heuristic, heur / 3, pick, best / 3);
  if (stats) {
    ++stats->tuned;
    stats->ms_heuristic += heur / 3;
    stats->ms_best += best / 3;
  }
  std::lock_guard<std::mutex> lock(g_tune_mu);
  g_tune_cache[sig] = pick;
  return CMPS_OK;
}

// Tasks, terms, tiles and the list that these are written from in one
// allocation, with one wait at the end: plans are made anew for every operator
// and environment update (XXZ chain at chi = 100: 40 us a plan less than with an
// allocation and a wait for each of them).
int GemmPlan::upload(cudaStream_t st) {
  release();
  const int shape = pick_shape64(*this);
  std::vector<TaskTiles> list;
  t64.shape = shape;
  t64.n = tile_list(*this, shape, list);
  if (tasks.empty()) return CMPS_OK;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t b_tasks = al(tasks.size() * sizeof(GemmTask)), b_terms = al(terms.size() * sizeof(GemmTerm)),
               b_list = al(list.size() * sizeof(TaskTiles)), b_tiles = (size_t)t64.n * sizeof(GemmTile);
  char* p = nullptr;
  CMPS_CUDA(dmalloc((void**)&p, b_tasks + b_terms + b_list + b_tiles));
  d_tasks = (GemmTask*)p;
  d_terms = (GemmTerm*)(p + b_tasks);
  CMPS_CUDA(cudaMemcpyAsync(d_tasks, tasks.data(), tasks.size() * sizeof(GemmTask), cudaMemcpyHostToDevice, st));
  if (!terms.empty())
    CMPS_CUDA(cudaMemcpyAsync(d_terms, terms.data(), terms.size() * sizeof(GemmTerm), cudaMemcpyHostToDevice, st));
  if (!t64.n) {
    CMPS_CUDA(cudaStreamSynchronize(st));
    return CMPS_OK;
  }
  t64.d = d_tiles0 = (GemmTile*)(p + b_tasks + b_terms + b_list);
  return expand_tiles(shape, list, (TaskTiles*)(p + b_tasks + b_terms), d_tasks, t64.d, st);
}

int GemmPlan::validate(bool a_h, bool b_h, int64_t a_len, int64_t b_len, int64_t c_len, const char* what) const {
  for (const GemmTask& t : tasks) {
    if (t.m < 0 || t.n < 0 || t.t0 < 0 || t.t1 < t.t0 || t.t1 > (int32_t)terms.size())
      return fail(CMPS_ERR_STATE, std::string(what) + ": malformed task");
    if (t.m == 0 || t.n == 0) continue;
    if ((t.n_in > 0) != nsplit || (nsplit && (a_h || b_h || t.ldc_out < t.n_in)))
      return fail(CMPS_ERR_STATE, std::string(what) + ": malformed two-level N index");
    // extent of one row of C or B along N: the last column's offset + 1
    const int64_t nspan = nsplit ? (int64_t)((t.n - 1) / t.n_in) * t.ldc_out + (t.n - 1) % t.n_in + 1 : t.n;
    if (t.c_off < 0 || t.c_off + (int64_t)(t.m - 1) * t.ldc + nspan > c_len || (!nsplit && t.ldc < t.n))
      return fail(CMPS_ERR_STATE, std::string(what) + ": output range outside its buffer");
    for (int q = t.t0; q < t.t1; ++q) {
      const GemmTerm& tm = terms[q];
      if (tm.k <= 0) return fail(CMPS_ERR_STATE, std::string(what) + ": empty term");
      // A is M x K (row-major, lda >= K) or stored K x M (lda >= M)
      int64_t arows = a_h ? tm.k : t.m, acols = a_h ? t.m : tm.k;
      int64_t brows = b_h ? t.n : tm.k, bcols = b_h ? tm.k : t.n;
      if (tm.lda < acols || tm.a_off < 0 || tm.a_off + (arows - 1) * tm.lda + acols > a_len)
        return fail(CMPS_ERR_STATE, std::string(what) + ": A operand range outside its buffer");
      if (nsplit) {
        const int64_t bspan = (int64_t)((t.n - 1) / t.n_in) * tm.ldb_out + (t.n - 1) % t.n_in + 1;
        if (tm.ldb_out < t.n_in || tm.b_off < 0 || tm.b_off + (int64_t)(tm.k - 1) * tm.ldb + bspan > b_len)
          return fail(CMPS_ERR_STATE, std::string(what) + ": B operand range outside its buffer");
      } else if (tm.ldb < bcols || tm.b_off < 0 || tm.b_off + (brows - 1) * tm.ldb + bcols > b_len) {
        return fail(CMPS_ERR_STATE, std::string(what) + ": B operand range outside its buffer");
      }
    }
  }
  return CMPS_OK;
}

void GemmPlan::release() {
  for (GemmTiles* t : {&t64, &t32}) {
    if (t->d && t->d != d_tiles0) dfree(t->d);
    *t = GemmTiles{};
  }
  if (d_tasks) dfree(d_tasks);
  d_tasks = nullptr;
  d_terms = nullptr;
  d_tiles0 = nullptr;
}

}  // namespace cmps
