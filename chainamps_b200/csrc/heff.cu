// Host side of the device-resident effective Hamiltonian: parsing of the
// reference's MPX tensors, charge-sector structure, LeftPart / RightPart
// formation, the two grouped-GEMM stages of the matvec and the Krylov
// ground-state solver.
//
// Matvec (TwoVertexMPOMPSMultiply, DMRG_routines.cpp:898-945):
//   LeftPart^{b1}[(s1', a0'), (s1, a0)]  = sum_b0 W[s1', b0, s1, b1] L^{b0}[a0', a0]
//   RightPart^{b1}[(s2, a2), (s2', a2')] = sum_b2 W[s2', b1, s2, b2] R^{b2}[a2', a2]
//   T^{b1}  = LeftPart^{b1} . Theta                       (stage 1)
//   Theta'  = sum_b1 T^{b1} . RightPart^{b1}               (stage 2)
// exactly the reference's (LeftPart . V) . RightPart order
// (DMRG_routines.cpp:779, :943), with every operand held as dense
// charge-sector blocks instead of CSC.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <numeric>
#include <set>

#include "heff.h"

namespace cmps {

// ---------------------------------------------------------------------------
QKey Rules::add(const QKey& a, const QKey& b) const {
  QKey o = zero();
  for (int i = 0; i < nq; ++i) {
    int v = (int)a[i] + (int)b[i];
    if (n[i] > 0) v = ((v % n[i]) + n[i]) % n[i];
    o[i] = (int16_t)v;
  }
  return o;
}
QKey Rules::sub(const QKey& a, const QKey& b) const {
  QKey o = zero();
  for (int i = 0; i < nq; ++i) {
    int v = (int)a[i] - (int)b[i];
    if (n[i] > 0) v = ((v % n[i]) + n[i]) % n[i];
    o[i] = (int16_t)v;
  }
  return o;
}

void Bond::build(const std::vector<QKey>& charges) {
  sq.clear(); sdim.clear(); esec.assign(charges.size(), 0); epos.assign(charges.size(), 0);
  selem.clear(); lookup.clear();
  for (size_t e = 0; e < charges.size(); ++e) {
    auto it = lookup.find(charges[e]);
    int s;
    if (it == lookup.end()) {
      s = (int)sq.size();
      lookup[charges[e]] = s;
      sq.push_back(charges[e]);
      sdim.push_back(0);
      selem.emplace_back();
    } else {
      s = it->second;
    }
    esec[e] = s;
    epos[e] = sdim[s]++;
    selem[s].push_back((int64_t)e);
  }
}

std::vector<QKey> Bond::element_charges() const {
  std::vector<QKey> out(esec.size());
  for (size_t e = 0; e < esec.size(); ++e) out[e] = sq[esec[e]];
  return out;
}

int Planar::alloc(int64_t n) {
  release();
  len = n;
  if (n == 0) return CMPS_OK;
  cudaError_t e = dmalloc(&d, sizeof(double) * 2 * (size_t)n);
  if (e != cudaSuccess) {
    d = nullptr;
    len = 0;
    return fail(CMPS_ERR_NOMEM, std::string("device allocation of ") + std::to_string(16.0 * n / 1e9) +
                                    " GB failed: " + cudaGetErrorString(e));
  }
  return CMPS_OK;
}

void Planar::release() {
  if (d) dfree(d);
  d = nullptr;
  len = 0;
}

int64_t Env::block_rows(int b, int s) const {
  int sp = partner[(size_t)b * a.nsec() + s];
  return right ? a.sdim[s] : a.sdim[sp];
}
int64_t Env::block_cols(int b, int s) const {
  int sp = partner[(size_t)b * a.nsec() + s];
  return right ? a.sdim[sp] : a.sdim[s];
}

// ---------------------------------------------------------------------------
// desc helpers
static int check_desc(const cmps_mpx_desc* d, int nidx, const char* what) {
  if (!d) return fail(CMPS_ERR_ARG, std::string(what) + ": null descriptor");
  if (d->num_indices != nidx)
    return fail(CMPS_ERR_ARG, std::string(what) + ": expected " + std::to_string(nidx) + " indices, got " +
                                  std::to_string(d->num_indices));
  if (d->num_row_indices < 0 || d->num_row_indices > d->num_indices)
    return fail(CMPS_ERR_ARG, std::string(what) + ": bad num_row_indices");
  int64_t r = 1, c = 1;
  for (int i = 0; i < d->num_indices; ++i) {
    if (d->sizes[i] < 1) return fail(CMPS_ERR_ARG, std::string(what) + ": empty index");
    (i < d->num_row_indices ? r : c) *= d->sizes[i];
  }
  if (r != d->rows || c != d->cols)
    return fail(CMPS_ERR_ARG, std::string(what) + ": matrix shape does not match index sizes");
  if (d->colptr[0] != 0) return fail(CMPS_ERR_ARG, std::string(what) + ": colptr[0] != 0");
  for (int64_t j = 0; j < d->cols; ++j)
    if (d->colptr[j + 1] < d->colptr[j]) return fail(CMPS_ERR_ARG, std::string(what) + ": colptr not monotone");
  int64_t nnz = d->colptr[d->cols];
  for (int64_t p = 0; p < nnz; ++p)
    if (d->rowind[p] < 0 || d->rowind[p] >= d->rows)
      return fail(CMPS_ERR_ARG, std::string(what) + ": row index out of range");
  return CMPS_OK;
}

int parse_index_charges(const Rules& r, const cmps_mpx_desc* d, int idx, std::vector<QKey>& out) {
  int64_t off = 0;
  for (int i = 0; i < idx; ++i) off += d->sizes[i];
  out.assign(d->sizes[idx], r.zero());
  for (int64_t e = 0; e < d->sizes[idx]; ++e) {
    QKey q = r.zero();
    for (int c = 0; c < r.nq; ++c) {
      int v = d->charges[(off + e) * r.nq + c];
      if (r.n[c] > 0) v = ((v % r.n[c]) + r.n[c]) % r.n[c];
      q[c] = (int16_t)v;
    }
    out[e] = q;
  }
  return CMPS_OK;
}

// Visit every stored entry with its multi-index (first index fastest).
template <typename F>
static void for_each_entry(const cmps_mpx_desc* d, F&& f) {
  int k = d->num_indices, nr = d->num_row_indices;
  std::vector<int64_t> mi(k, 0);
  for (int64_t c = 0; c < d->cols; ++c) {
    int64_t cc = c;
    for (int i = nr; i < k; ++i) {
      mi[i] = cc % d->sizes[i];
      cc /= d->sizes[i];
    }
    for (int64_t p = d->colptr[c]; p < d->colptr[c + 1]; ++p) {
      int64_t rr = d->rowind[p];
      for (int i = 0; i < nr; ++i) {
        mi[i] = rr % d->sizes[i];
        rr /= d->sizes[i];
      }
      f(mi.data(), d->values[2 * p], d->values[2 * p + 1]);
    }
  }
}

// L: a' = 1, b = 3, a = 5.  R: a' = 0, b = 2, a = 4.  Blocks are allocated
// for every (b, sector) with a charge-consistent partner sector.
int build_env_from_desc(const Rules& r, const cmps_mpx_desc* d, bool right, Env& env, int D,
                        const std::vector<QKey>& bq, cudaStream_t st) {
  const char* what = right ? "right block" : "left block";
  CMPS_TRY(check_desc(d, 6, what));
  const int ia = right ? 4 : 5, iap = right ? 0 : 1, ib = right ? 2 : 3;
  for (int i = 0; i < 6; ++i)
    if (i != ia && i != iap && i != ib && d->sizes[i] != 1)
      return fail(CMPS_ERR_ARG, std::string(what) + ": index " + std::to_string(i) + " must be a size-1 dummy");
  if (d->sizes[ib] != D) return fail(CMPS_ERR_ARG, std::string(what) + ": MPO index size differs from W");
  std::vector<QKey> qa, qap, qb;
  parse_index_charges(r, d, ia, qa);
  parse_index_charges(r, d, iap, qap);
  parse_index_charges(r, d, ib, qb);
  if (qa.size() != qap.size() || qa != qap)
    return fail(CMPS_ERR_ARG, std::string(what) + ": bra and ket bond indices differ");
  if (qb != bq) return fail(CMPS_ERR_ARG, std::string(what) + ": MPO index charges differ from W");
  env.right = right;
  env.a.build(qa);
  env.D = D;
  env.bq = bq;
  const int ns = env.a.nsec();
  env.off.assign((size_t)D * ns, -1);
  env.partner.assign((size_t)D * ns, -1);
  int64_t total = 0;
  for (int b = 0; b < D; ++b)
    for (int s = 0; s < ns; ++s) {
      int sp = env.a.find(r.add(env.a.sq[s], bq[b]));
      if (sp < 0) continue;
      env.partner[(size_t)b * ns + s] = sp;
      env.off[(size_t)b * ns + s] = total;
      total += env.a.sdim[s] * env.a.sdim[sp];
    }
  std::vector<double> h(2 * (size_t)total, 0.0);
  int status = CMPS_OK;
  for_each_entry(d, [&](const int64_t* mi, double re, double im) {
    if (status != CMPS_OK) return;
    int64_t a = mi[ia], ap = mi[iap], b = mi[ib];
    int s = env.a.esec[a], sp = env.a.esec[ap];
    if (env.partner[(size_t)b * ns + s] != sp) {
      if (re != 0.0 || im != 0.0) status = fail(CMPS_ERR_CHARGE, std::string(what) + ": entry violates charge conservation");
      return;
    }
    int64_t o = env.off[(size_t)b * ns + s];
    int64_t p = env.a.epos[a], pp = env.a.epos[ap];
    int64_t e = right ? o + p * env.a.sdim[sp] + pp : o + pp * env.a.sdim[s] + p;
    h[e] += re;
    h[total + e] += im;
  });
  if (status != CMPS_OK) return status;
  CMPS_TRY(env.data.alloc(total));
  CMPS_TRY(copy_wait(env.data.d, h.data(), sizeof(double) * 2 * total, cudaMemcpyHostToDevice, st));
  return CMPS_OK;
}

// ---------------------------------------------------------------------------
Heff::~Heff() {
  release_split(this);
  release_canonical(this);
  L.data.release();
  R.data.release();
  LP.release();
  RP.release();
  T.release();
  x.release();
  y.release();
  theta.release();
  kv.release();
  proj.release();
  if (d_proj) dfree(d_proj);
  d_proj = nullptr;
  stage1.release();
  stage2.release();
  ops.release();
  if (d_pack) dfree(d_pack);
  if (d_io) dfree(d_io);
  if (h_ab) cudaFreeHost(h_ab);
  if (d_lp_blocks) dfree(d_lp_blocks);
  if (d_lp_terms) dfree(d_lp_terms);
  if (d_rp_blocks) dfree(d_rp_blocks);
  if (d_rp_terms) dfree(d_rp_terms);
}

template <typename T>
static int upload_vec(const std::vector<T>& v, T** d, cudaStream_t st) {
  if (*d) dfree(*d);
  *d = nullptr;
  if (v.empty()) return CMPS_OK;
  CMPS_CUDA(dmalloc((void**)d, sizeof(T) * v.size()));
  return copy_wait(*d, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, st);
}

int Heff::build(cmps_context* c, const Rules& r, const cmps_mpx_desc* Ld, const cmps_mpx_desc* Wd,
                const cmps_mpx_desc* Rd) {
  ctx = c;
  device = c->device;
  rules = r;
  CMPS_TRY(parse_mpo(Wd));
  CMPS_TRY(build_env_from_desc(r, Ld, false, L, D, bq, c->stream));
  CMPS_TRY(build_env_from_desc(r, Rd, true, R, D, bq, c->stream));
  return finish();
}

int copy_env(const Env& src, Env& dst, cudaStream_t st) {
  dst.a = src.a;
  dst.D = src.D;
  dst.bq = src.bq;
  dst.off = src.off;
  dst.partner = src.partner;
  dst.right = src.right;
  CMPS_TRY(dst.data.alloc(src.data.len));
  CMPS_TRY(copy_wait(dst.data.d, src.data.d, sizeof(double) * 2 * src.data.len, cudaMemcpyDeviceToDevice, st));
  return CMPS_OK;
}

int Heff::build_from_envs(cmps_context* c, const Rules& r, const Env& Lsrc, const cmps_mpx_desc* Wd,
                          const Env& Rsrc) {
  ctx = c;
  device = c->device;
  rules = r;
  CMPS_TRY(parse_mpo(Wd));
  if (Lsrc.right || !Rsrc.right) return fail(CMPS_ERR_ARG, "block handedness: need a left and a right block");
  if (Lsrc.D != D || Rsrc.D != D || Lsrc.bq != bq || Rsrc.bq != bq)
    return fail(CMPS_ERR_ARG, "block MPO index differs from W");
  CMPS_TRY(copy_env(Lsrc, L, c->stream));
  CMPS_TRY(copy_env(Rsrc, R, c->stream));
  return finish();
}

int Heff::parse_mpo(const cmps_mpx_desc* Wd) {
  const Rules& r = rules;
  CMPS_TRY(check_desc(Wd, 4, "MPO"));
  d = (int)Wd->sizes[0];
  D = (int)Wd->sizes[1];
  if (Wd->sizes[2] != d || Wd->sizes[3] != D) return fail(CMPS_ERR_ARG, "MPO: index sizes inconsistent");
  std::vector<QKey> sig2, bq3;
  parse_index_charges(r, Wd, 0, sigq);
  parse_index_charges(r, Wd, 2, sig2);
  parse_index_charges(r, Wd, 1, bq);
  parse_index_charges(r, Wd, 3, bq3);
  if (sigq != sig2 || bq != bq3) return fail(CMPS_ERR_ARG, "MPO: row and column index charges differ");
  W.clear();
  int status = CMPS_OK;
  for_each_entry(Wd, [&](const int64_t* mi, double re, double im) {
    if (re == 0.0 && im == 0.0) return;
    int sp = (int)mi[0], bl = (int)mi[1], s = (int)mi[2], br = (int)mi[3];
    if (r.add(sigq[sp], bq[bl]) != r.add(sigq[s], bq[br])) {
      status = fail(CMPS_ERR_CHARGE, "MPO: entry violates charge conservation");
      return;
    }
    W.push_back(WEntry{sp, bl, s, br, re, im});
  });
  if (status != CMPS_OK) return status;
  return CMPS_OK;
}

// One CTA per ARPACK column: out[start + i] for the i-th allowed row of the
// column's sector block (mode 0: theta offset, mode 1: full linear index).
__global__ void k_arpack_map(const Heff::MapCol* __restrict__ cols, const Heff::MapSec* __restrict__ secs,
                             const int64_t* __restrict__ rowlin, const int64_t* __restrict__ rowth, int64_t dchiL,
                             int mode, int64_t* __restrict__ out) {
  const Heff::MapCol c = cols[blockIdx.x];
  const Heff::MapSec s = secs[c.m];
  for (int64_t i = threadIdx.x; i < s.nrows; i += blockDim.x) {
    const int64_t r = s.rowstart + i;
    out[c.start + i] = mode == 0 ? s.base + rowth[r] * s.ncols + c.colth : rowlin[r] + dchiL * c.colpart;
  }
}

int Heff::arpack_map(int mode, int64_t* d_out, cudaStream_t st) const {
  if (map_cols.empty() || n_allowed == 0) return CMPS_OK;
  if (map_cols.size() > 0x7fffffffull) return fail(CMPS_ERR_ARG, "too many wavefunction columns");
  MapCol* dc = nullptr;
  MapSec* ds = nullptr;
  int64_t *drl = nullptr, *drt = nullptr;
  int rc = CMPS_OK;
  auto up = [&](auto& v, auto** d) -> int {
    const size_t bytes = sizeof(v[0]) * std::max<size_t>(1, v.size());
    CMPS_CUDA(dmalloc((void**)d, bytes));
    return copy_wait(*d, v.data(), sizeof(v[0]) * v.size(), cudaMemcpyHostToDevice, st);
  };
  if ((rc = up(map_cols, &dc)) == CMPS_OK && (rc = up(map_secs, &ds)) == CMPS_OK &&
      (rc = up(map_rowlin, &drl)) == CMPS_OK && (rc = up(map_rowth, &drt)) == CMPS_OK) {
    const int64_t dchiL = (int64_t)d * L.a.size();
    k_arpack_map<<<(unsigned)map_cols.size(), 256, 0, st>>>(dc, ds, drl, drt, dchiL, mode, d_out);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = fail(CMPS_ERR_CUDA, std::string("ARPACK index map: ") + cudaGetErrorString(e));
  }
  if (dc) dfree(dc);
  if (ds) dfree(ds);
  if (drl) dfree(drl);
  if (drt) dfree(drt);
  return rc;
}

int Heff::allowed_indices(int64_t* host_out) const {
  if (n_allowed == 0) return CMPS_OK;
  int64_t* tmp = nullptr;
  CMPS_CUDA(dmalloc(&tmp, sizeof(int64_t) * n_allowed));
  int rc = arpack_map(1, tmp, ctx->stream);
  if (rc == CMPS_OK) rc = copy_wait(host_out, tmp, sizeof(int64_t) * n_allowed, cudaMemcpyDeviceToHost, ctx->stream);
  dfree(tmp);
  return rc;
}

// ARPACK order <-> sector blocks: CTA = (group of <= 32 columns, 64 rows in the
// gather, 32 in the scatter).
// Reads run down each ARPACK column (contiguous), writes along theta rows
// (the group's columns are consecutive theta columns).
// HBM bound (16 bytes in, 16 out per entry).  Two dependent reads of
// descriptors stand before the data: gather 0.207 ms and scatter 0.190 ms at
// 33.5M entries, 0.27 and 0.26 with four.  The gather takes the tile's 64 rows in
// one CTA, so that more reads are in flight; the scatter, which reads short runs,
// gives each half of them a CTA of its own.
template <bool PACK>
__global__ void __launch_bounds__(256) k_pack_tiles(const Heff::PackTile* __restrict__ tiles,
                                                    const Heff::PackGroup* __restrict__ groups,
                                                    const int64_t* __restrict__ starts,
                                                    const int64_t* __restrict__ rowth, double2* __restrict__ arp,
                                                    double* __restrict__ re, double* __restrict__ im) {
  constexpr int ROWS = PACK ? 64 : 32, LD = ROWS + 1, E = ROWS / 8;  // E elements per thread
  __shared__ double2 t[32 * LD];  // [column j][row r]
  const Heff::PackTile tl = tiles[PACK ? blockIdx.x : blockIdx.x >> 1];
  const Heff::PackGroup g = groups[tl.group];
  const int64_t r0 = tl.r0 + (PACK ? 0 : 32 * (int)(blockIdx.x & 1));
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int nr = (int)min((int64_t)ROWS, g.nrows - r0), nc = (int)g.cnt;
  if (nr <= 0) {
    grid_wait();
    return;
  }
  const int64_t* rows = rowth + g.rowstart + r0;
  const int64_t* col = starts + g.off;
  grid_wait();  // up to here only descriptors were read
  // along an ARPACK column: column j, row r of element k; along a theta row: row ty + 8 k, column tx
  auto j_of = [&](int k) { return ty + 8 * (k / (ROWS / 32)); };
  auto r_of = [&](int k) { return tx + 32 * (k % (ROWS / 32)); };
  if (PACK) {
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (j_of(k) < nc && r_of(k) < nr) t[j_of(k) * LD + r_of(k)] = arp[col[j_of(k)] + r0 + r_of(k)];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int r = ty + 8 * k;
      if (tx < nc && r < nr) {
        const int64_t p = g.base + rows[r] * g.ncols + tx;
        const double2 w = t[tx * LD + r];
        re[p] = w.x;
        im[p] = w.y;
      }
    }
  } else {
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int r = ty + 8 * k;
      if (tx < nc && r < nr) {
        const int64_t p = g.base + rows[r] * g.ncols + tx;
        t[tx * LD + r] = make_double2(re[p], im[p]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (j_of(k) < nc && r_of(k) < nr) arp[col[j_of(k)] + r0 + r_of(k)] = t[j_of(k) * LD + r_of(k)];
  }
}

int Heff::build_pack(cudaStream_t st) {
  // ARPACK column index of (a2, s2), then groups per (m, s2) in a2-sector order
  const Bond& A2 = R.a;
  std::vector<int32_t> col_of((size_t)A2.size() * d, -1);
  for (size_t c = 0; c < map_cols.size(); ++c) {
    const int64_t s2 = map_cols[c].colpart % d, a2 = map_cols[c].colpart / d;
    col_of[(size_t)a2 * d + s2] = (int32_t)c;
  }
  std::vector<std::vector<int64_t>> elems(A2.nsec());
  for (int64_t a2 = 0; a2 < A2.size(); ++a2) elems[A2.esec[a2]].push_back(a2);
  std::vector<int64_t> starts;
  std::vector<PackGroup> groups;
  std::vector<PackTile> tiles;
  for (int m = 0; m < (int)th.mq.size(); ++m)
    for (int s2 = 0; s2 < d; ++s2) {
      if (th.coloff[m][s2] < 0) continue;
      const int t = A2.find(rules.add(th.mq[m], sigq[s2]));
      const std::vector<int64_t>& el = elems[t];
      for (size_t e0 = 0; e0 < el.size(); e0 += 32) {
        PackGroup g{(int64_t)starts.size(), th.base[m] + th.coloff[m][s2] + (int64_t)e0, th.ncols[m],
                    map_secs[m].rowstart,   th.nrows[m], (int64_t)std::min<size_t>(32, el.size() - e0)};
        for (int j = 0; j < g.cnt; ++j) {
          const int32_t c = col_of[(size_t)el[e0 + j] * d + s2];
          if (c < 0 || map_cols[c].m != m || map_cols[c].colth != th.coloff[m][s2] + (int64_t)(e0 + j))
            return fail(CMPS_ERR_STATE, "internal: pack group columns not consecutive");
          starts.push_back(map_cols[c].start);
        }
        for (int64_t r0 = 0; r0 < th.nrows[m]; r0 += 64) tiles.push_back(PackTile{(int32_t)groups.size(), (int32_t)r0});
        groups.push_back(g);
      }
    }
  if (tiles.size() > 0x3fffffffull) return fail(CMPS_ERR_ARG, "too many pack tiles");
  n_pack_tiles = 0;
  if (tiles.empty()) return CMPS_OK;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t b_rowth = al(sizeof(int64_t) * map_rowth.size()), b_starts = al(sizeof(int64_t) * starts.size()),
               b_groups = al(sizeof(PackGroup) * groups.size()), b_tiles = al(sizeof(PackTile) * tiles.size());
  if (d_pack) dfree(d_pack);
  d_pack = nullptr;
  CMPS_CUDA(dmalloc(&d_pack, b_rowth + b_starts + b_groups + b_tiles));
  char* p = (char*)d_pack;
  d_map_rowth = (const int64_t*)p;
  CMPS_TRY(copy_wait(p, map_rowth.data(), sizeof(int64_t) * map_rowth.size(), cudaMemcpyHostToDevice, st));
  p += b_rowth;
  d_pack_starts = (const int64_t*)p;
  CMPS_TRY(copy_wait(p, starts.data(), sizeof(int64_t) * starts.size(), cudaMemcpyHostToDevice, st));
  p += b_starts;
  d_pack_groups = (const PackGroup*)p;
  CMPS_TRY(copy_wait(p, groups.data(), sizeof(PackGroup) * groups.size(), cudaMemcpyHostToDevice, st));
  p += b_groups;
  d_pack_tiles = (const PackTile*)p;
  CMPS_TRY(copy_wait(p, tiles.data(), sizeof(PackTile) * tiles.size(), cudaMemcpyHostToDevice, st));
  n_pack_tiles = (int64_t)tiles.size();
  return CMPS_OK;
}

int Heff::pack(const double* in, const Planar& out, cudaStream_t st) const {
  if (n_pack_tiles == 0) return CMPS_OK;
  CMPS_CUDA(launch_chained(k_pack_tiles<true>, dim3((unsigned)n_pack_tiles), dim3(256), 0, st, d_pack_tiles,
                           d_pack_groups, d_pack_starts, d_map_rowth, (double2*)in, out.re(), out.im()));
  return CMPS_OK;
}

int Heff::unpack(const Planar& in, double* out, cudaStream_t st) const {
  if (n_pack_tiles == 0) return CMPS_OK;
  CMPS_CUDA(launch_chained(k_pack_tiles<false>, dim3((unsigned)(2 * n_pack_tiles)), dim3(256), 0, st, d_pack_tiles,
                           d_pack_groups, d_pack_starts, d_map_rowth, (double2*)out, in.re(), in.im()));
  return CMPS_OK;
}

// Phase timer of Heff::finish for CMPS_BUILD_TRACE (host wall ms to stderr).
struct BuildTrace {
  bool on = std::getenv("CMPS_BUILD_TRACE") != nullptr;
  std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
  void mark(const char* what) {
    if (!on) return;
    const auto now = std::chrono::steady_clock::now();
    std::fprintf(stderr, "build %-22s %8.2f ms\n", what, std::chrono::duration<double, std::milli>(now - t).count());
    t = now;
  }
};

int Heff::finish() {
  BuildTrace bt;
  const Rules& r = rules;
  const Bond& A0 = L.a;
  const Bond& A2 = R.a;
  // ---- theta space ----
  // middle charges ordered by first appearance over columns c = s2 + d*a2
  // ascending (the block order of GetAllBlockColumns, MPX_matrix.cpp:365-385)
  std::set<QKey> rowm;
  for (int s1 = 0; s1 < d; ++s1)
    for (int s = 0; s < A0.nsec(); ++s) rowm.insert(r.add(sigq[s1], A0.sq[s]));
  th = ThetaSpace();
  for (int64_t a2 = 0; a2 < A2.size(); ++a2)
    for (int s2 = 0; s2 < d; ++s2) {
      QKey m = r.sub(A2.sq[A2.esec[a2]], sigq[s2]);
      if (!rowm.count(m) || th.mfind.count(m)) continue;
      th.mfind[m] = (int)th.mq.size();
      th.mq.push_back(m);
    }
  const int nm = (int)th.mq.size();
  // charge classes of the physical states; blocks list states class by class
  cls_mem.clear();
  cls_of.assign(d, -1);
  cls_pos.assign(d, -1);
  {
    std::map<QKey, int> cfind;
    for (int s = 0; s < d; ++s) {
      auto it = cfind.find(sigq[s]);
      int c = it == cfind.end() ? -1 : it->second;
      if (c < 0) {
        c = (int)cls_mem.size();
        cfind[sigq[s]] = c;
        cls_mem.emplace_back();
      }
      cls_of[s] = c;
      cls_pos[s] = (int)cls_mem[c].size();
      cls_mem[c].push_back(s);
    }
  }
  std::vector<int> sig_order;
  for (const auto& mem : cls_mem) sig_order.insert(sig_order.end(), mem.begin(), mem.end());
  th.nrows.assign(nm, 0);
  th.ncols.assign(nm, 0);
  th.base.assign(nm, 0);
  th.rowoff.assign(nm, std::vector<int64_t>(d, -1));
  th.coloff.assign(nm, std::vector<int64_t>(d, -1));
  for (int m = 0; m < nm; ++m) {
    for (int s1 : sig_order) {
      int s = A0.find(r.sub(th.mq[m], sigq[s1]));
      if (s < 0) continue;
      th.rowoff[m][s1] = th.nrows[m];
      th.nrows[m] += A0.sdim[s];
    }
    for (int s2 : sig_order) {
      int t = A2.find(r.add(th.mq[m], sigq[s2]));
      if (t < 0) continue;
      th.coloff[m][s2] = th.ncols[m];
      th.ncols[m] += A2.sdim[t];
    }
    th.base[m] = th.total;
    th.total += th.nrows[m] * th.ncols[m];
  }
  default_windows();
  bt.mark("theta space");
  // ---- allowed indices, ARPACK order (DMRG_routines.cpp:808-824) ----
  // ARPACK order = ascending s1 + d a0 + d chiL (s2 + d a2).  Every entry of
  // sector block m is allowed, so a column (s2, a2) holds exactly the rows of
  // block m = q(a2) - q(s2), in ascending s1 + d a0 order: the maps follow
  // from one row list per block and one descriptor per column.
  full_length = (int64_t)d * A0.size() * d * A2.size();
  const int64_t chiL = A0.size();
  map_secs.assign(nm, MapSec{0, 0, 0, 0});
  map_rowlin.clear();
  map_rowth.clear();
  for (int m = 0; m < nm; ++m) {
    map_secs[m].rowstart = (int64_t)map_rowlin.size();
    for (int64_t a0 = 0; a0 < chiL; ++a0)
      for (int s1 = 0; s1 < d; ++s1) {
        if (r.add(sigq[s1], A0.sq[A0.esec[a0]]) != th.mq[m]) continue;
        map_rowlin.push_back(s1 + (int64_t)d * a0);
        map_rowth.push_back(th.rowoff[m][s1] + A0.epos[a0]);
      }
    map_secs[m].nrows = (int64_t)map_rowlin.size() - map_secs[m].rowstart;
    map_secs[m].base = th.base[m];
    map_secs[m].ncols = th.ncols[m];
    if (map_secs[m].nrows != th.nrows[m]) return fail(CMPS_ERR_STATE, "internal: sector row count mismatch");
  }
  map_cols.clear();
  n_allowed = 0;
  for (int64_t a2 = 0; a2 < A2.size(); ++a2) {
    const QKey qa2 = A2.sq[A2.esec[a2]];
    for (int s2 = 0; s2 < d; ++s2) {
      const int im = th.find(r.sub(qa2, sigq[s2]));
      if (im < 0) continue;
      map_cols.push_back(MapCol{s2 + (int64_t)d * a2, th.coloff[im][s2] + A2.epos[a2], n_allowed, im});
      n_allowed += th.nrows[im];
    }
  }
  if (n_allowed != th.total) return fail(CMPS_ERR_STATE, "internal: allowed count differs from sector total");

  bt.mark("ARPACK maps");
  // ---- LeftPart blocks: key (b1, s1', s1, a0-sector s), RightPart blocks: key (b1, s2, s2', a2-sector t) ----
  // One term per (MPO entry, sector) that has an environment block and a
  // middle charge on both sides; sorted by key, terms of one key in W order.
  // The charges are looked up once per (state, sector) and (middle charge, MPO
  // index), not per term, and the keys are dense integers, so a radix sort in
  // steps of 11 bits orders them: 19.4 -> 7.6 ms on the Ising chains (64 states,
  // 100 thousand terms a side), where this was a third of an operator's build.
  std::vector<int> mplus((size_t)nm * D);  // middle charge m + q(b), or -1
  for (int m = 0; m < nm; ++m)
    for (int b = 0; b < D; ++b) mplus[(size_t)m * D + b] = th.find(r.add(th.mq[m], bq[b]));
  auto form = [&](bool right, BlockOffsets& off, std::vector<AxpyBlock>& blocks, std::vector<AxpyTerm>& terms) {
    const Bond& A = right ? A2 : A0;
    const Env& E = right ? R : L;
    const int nsec = A.nsec();
    std::vector<int> mid((size_t)d * nsec);  // middle charge of (state, sector), or -1
    for (int s = 0; s < d; ++s)
      for (int a = 0; a < nsec; ++a)
        mid[(size_t)s * nsec + a] = th.find(right ? r.sub(A.sq[a], sigq[s]) : r.add(sigq[s], A.sq[a]));
    struct KeyTerm {
      uint64_t key;
      AxpyTerm t;
    };
    std::vector<KeyTerm> v, w2;
    v.reserve(W.size() * (size_t)std::min(nsec, 8));
    for (const WEntry& w : W) {
      const int be = right ? w.br : w.bl, bk = right ? w.bl : w.br;  // the environment's MPO index, the key's
      const int s0 = right ? w.s : w.sp, s1 = right ? w.sp : w.s;
      for (int a = 0; a < nsec; ++a) {
        const int64_t lo = E.off[(size_t)be * nsec + a];
        if (lo < 0) continue;
        const int m = mid[(size_t)w.s * nsec + a];
        if (m < 0 || mplus[(size_t)m * D + bk] < 0) continue;
        v.push_back(KeyTerm{(((uint64_t)bk * d + s0) * d + s1) * nsec + a, AxpyTerm{lo, w.wr, w.wi}});
      }
    }
    const uint64_t top = (uint64_t)D * d * d * nsec;
    w2.resize(v.size());
    std::vector<size_t> at(2049);
    for (int shift = 0; shift < 64 && top >> shift; shift += 11) {
      std::fill(at.begin(), at.end(), 0);
      for (const KeyTerm& k : v) ++at[(k.key >> shift & 2047) + 1];
      for (int i = 0; i < 2048; ++i) at[i + 1] += at[i];
      for (const KeyTerm& k : v) w2[at[k.key >> shift & 2047]++] = k;
      v.swap(w2);
    }
    off.clear();
    blocks.clear();
    terms.clear();
    terms.reserve(v.size());
    int64_t total = 0;
    for (size_t i = 0, j = 0; i < v.size(); i = j) {
      for (j = i; j < v.size() && v[j].key == v[i].key; ++j) {
      }
      uint64_t k = v[i].key;
      const int a = (int)(k % nsec), s1 = (int)((k /= nsec) % d), s0 = (int)((k /= d) % d), b1 = (int)(k / d);
      // partner sector, left: q(s') = q(s) + q(b0) = q(s) + q(s1) + q(b1) - q(s1');
      // right: q(t') = q(t) + q(b2) = q(t) + q(s2') + q(b1) - q(s2)
      const int ap = A.find(r.sub(r.add(r.add(A.sq[a], sigq[s1]), bq[b1]), sigq[s0]));
      if (ap < 0) continue;
      const int64_t len = A.sdim[ap] * A.sdim[a];
      off.push_back({{b1, s0, s1, a}, total});
      blocks.push_back(AxpyBlock{total, len, (int32_t)terms.size(), (int32_t)(terms.size() + (j - i))});
      for (size_t q = i; q < j; ++q) terms.push_back(v[q].t);
      total += len;
    }
    return total;
  };
  const int64_t lp_total = form(false, lp_off, lp_blocks, lp_terms);
  const int64_t rp_total = form(true, rp_off, rp_blocks, rp_terms);
  bt.mark("LP/RP block lists");
  CMPS_TRY(LP.alloc(lp_total));
  CMPS_TRY(RP.alloc(rp_total));
  CMPS_TRY(upload_vec(lp_blocks, &d_lp_blocks, ctx->stream));
  CMPS_TRY(upload_vec(lp_terms, &d_lp_terms, ctx->stream));
  CMPS_TRY(upload_vec(rp_blocks, &d_rp_blocks, ctx->stream));
  CMPS_TRY(upload_vec(rp_terms, &d_rp_terms, ctx->stream));

  bt.mark("LP/RP alloc+upload");
  owned.assign(nm, 1);
  CMPS_TRY(build_plans());
  for (const AxpyBlock& b : lp_blocks)
    for (int q = b.t0; q < b.t1; ++q)
      if (b.dst_off + b.len > lp_total || lp_terms[q].src_off + b.len > L.data.len)
        return fail(CMPS_ERR_STATE, "LeftPart block range outside its buffer");
  for (const AxpyBlock& b : rp_blocks)
    for (int q = b.t0; q < b.t1; ++q)
      if (b.dst_off + b.len > rp_total || rp_terms[q].src_off + b.len > R.data.len)
        return fail(CMPS_ERR_STATE, "RightPart block range outside its buffer");
  // pack map: every column and row index inside its sector block
  for (const MapCol& c : map_cols)
    if (c.m < 0 || c.m >= nm || c.colth < 0 || c.colth >= th.ncols[c.m])
      return fail(CMPS_ERR_STATE, "pack map column outside the sector blocks");
  for (int m = 0; m < nm; ++m)
    for (int64_t i = 0; i < map_secs[m].nrows; ++i) {
      const int64_t rt = map_rowth[map_secs[m].rowstart + i];
      if (rt < 0 || rt >= th.nrows[m]) return fail(CMPS_ERR_STATE, "pack map row outside the sector blocks");
    }
  bt.mark("folded plans");
  CMPS_TRY(build_pack(ctx->stream));
  cudaStream_t st = ctx->stream;
  CMPS_TRY(launch_block_axpy(d_lp_blocks, (int)lp_blocks.size(), d_lp_terms, L.data, LP, st));
  CMPS_TRY(launch_block_axpy(d_rp_blocks, (int)rp_blocks.size(), d_rp_terms, R.data, RP, st));

  bt.mark("pack + LP/RP formation");
  // ---- canonical four-stage flop count ----
  {
    double f = 0.0;
    std::set<int> usedbl, usedbr;
    for (const WEntry& w : W) { usedbl.insert(w.bl); usedbr.insert(w.br); }
    std::vector<std::vector<const WEntry*>> by_state(d);
    for (const WEntry& w : W) by_state[w.s].push_back(&w);
    for (int m = 0; m < nm; ++m)
      for (int s1 = 0; s1 < d; ++s1) {
        if (th.rowoff[m][s1] < 0) continue;
        int s = A0.find(r.sub(th.mq[m], sigq[s1]));
        for (int b0 : usedbl) {
          int64_t lo = L.off[(size_t)b0 * A0.nsec() + s];
          if (lo < 0) continue;
          int sp = L.partner[(size_t)b0 * A0.nsec() + s];
          f += 8.0 * A0.sdim[sp] * (double)A0.sdim[s] * th.ncols[m];            // L . theta
        }
        for (const WEntry* p : by_state[s1]) {
          const WEntry& w = *p;
          int64_t lo = L.off[(size_t)w.bl * A0.nsec() + s];
          if (lo < 0) continue;
          int sp = L.partner[(size_t)w.bl * A0.nsec() + s];
          f += 8.0 * A0.sdim[sp] * (double)th.ncols[m];                          // W1
        }
      }
    for (int m = 0; m < nm; ++m)
      for (int s2 = 0; s2 < d; ++s2) {
        if (th.coloff[m][s2] < 0) continue;
        int t = A2.find(r.add(th.mq[m], sigq[s2]));
        for (const WEntry* p : by_state[s2]) {
          const int mp = mplus[(size_t)m * D + p->bl];
          if (mp < 0) continue;
          f += 8.0 * th.nrows[mp] * (double)A2.sdim[t];                         // W2
        }
        for (int b2 : usedbr) {
          int64_t ro = R.off[(size_t)b2 * A2.nsec() + t];
          if (ro < 0) continue;
          int tp = R.partner[(size_t)b2 * A2.nsec() + t];
          f += 8.0 * th.nrows[m] * (double)A2.sdim[t] * A2.sdim[tp];             // . R
        }
      }
    flops_canonical = f;
  }
  bt.mark("flop count");
  CMPS_TRY(x.alloc(th.total));
  CMPS_TRY(y.alloc(th.total));
  CMPS_CUDA(dmalloc(&d_io, sizeof(double) * 2 * std::max<int64_t>(1, n_allowed)));
  CMPS_TRY(ops.init(th.total, st));
  bt.mark("work vectors");
  CMPS_TRY(select_order());
  CMPS_CUDA(cudaStreamSynchronize(st));
  bt.mark("contraction order");
  return CMPS_OK;
}

// The FP64 matvec's contraction order: the one requested, or with
// CMPS_ORDER_AUTO the canonical order when it executes at most half the
// flops of the folded order over whole T blocks (it moves three intermediates through HBM where the
// folded order moves one, so a small flop advantage does not pay).
int Heff::select_order() {
  flops_folded = flops_executed;
  std::vector<uint8_t> cneed;
  CMPS_TRY(canonical_flops(*this, &flops_canon, &cneed));
  // the input sectors of either order (the windows must hold both)
  for (size_t m = 0; m < cneed.size() && m < in_need.size(); ++m) in_need[m] |= cneed[m];
  int want = order_req;
  if (want == CMPS_ORDER_AUTO) want = flops_canon <= 0.5 * flops_folded_full ? CMPS_ORDER_CANONICAL : CMPS_ORDER_FOLDED;
  // the canonical plans are rebuilt (or dropped), and the split-precision
  // operator, whose form follows the order, is prepared again
  release_split(this);
  if (want == CMPS_ORDER_CANONICAL) {
    CMPS_TRY(build_canonical(*this));
  } else {
    release_canonical(this);
  }
  order = want;
  if (is_split(precision)) CMPS_TRY(prepare_precision(this, precision));
  return CMPS_OK;
}

// The two grouped-GEMM plans of the matvec and the intermediate T, for the
// output sectors marked in `owned` (all of them unless the matvec is
// sharded): stage-2 tasks of owned output sectors only, and stage-1 tasks
// only for the blocks T^{b1}_m those read (m + q(b1) owned).
int Heff::build_plans() {
  const Rules& r = rules;
  const Bond& A0 = L.a;
  const Bond& A2 = R.a;
  const int nm = (int)th.mq.size();
  if ((int)owned.size() != nm) return fail(CMPS_ERR_STATE, "owned-sector mask size");
  stage1.release();
  stage2.release();
  T.release();
  if ((int)in_base.size() != nm || (int)out_base.size() != nm) return fail(CMPS_ERR_STATE, "window size");
  in_need.assign(nm, 0);
  // Dense (b, sigma', sigma, sector) -> block offset tables of lp_off /
  // rp_off for the plan loops below (several lookups per (b, m, sigma',
  // sigma)), when they stay small; searched otherwise.
  const int64_t nlp = (int64_t)D * d * d * A0.nsec(), nrp = (int64_t)D * d * d * A2.nsec();
  constexpr int64_t kDenseMax = int64_t(1) << 24;
  std::vector<int64_t> lp_tab, rp_tab;
  if (nlp <= kDenseMax) {
    lp_tab.assign(nlp, -1);
    for (auto& kv2 : lp_off)
      lp_tab[(((int64_t)kv2.first[0] * d + kv2.first[1]) * d + kv2.first[2]) * A0.nsec() + kv2.first[3]] = kv2.second;
  }
  if (nrp <= kDenseMax) {
    rp_tab.assign(nrp, -1);
    for (auto& kv2 : rp_off)
      rp_tab[(((int64_t)kv2.first[0] * d + kv2.first[1]) * d + kv2.first[2]) * A2.nsec() + kv2.first[3]] = kv2.second;
  }
  auto lp_at = [&](int b, int sp, int sg, int sec) -> int64_t {
    if (!lp_tab.empty()) return lp_tab[(((int64_t)b * d + sp) * d + sg) * A0.nsec() + sec];
    auto it = lp_off.find({b, sp, sg, sec});
    return it == lp_off.end() ? -1 : it->second;
  };
  auto rp_at = [&](int b, int sg, int sp, int sec) -> int64_t {
    if (!rp_tab.empty()) return rp_tab[(((int64_t)b * d + sg) * d + sp) * A2.nsec() + sec];
    auto it = rp_off.find({b, sg, sp, sec});
    return it == rp_off.end() ? -1 : it->second;
  };
  // T^{b1}_m = LeftPart^{b1} . Theta_m holds only what the second stage can
  // use: the rows of states sigma1' that some LeftPart block of b1 produces
  // (live) and the columns of states sigma2 that some RightPart block of b1
  // reads.  A raising or lowering operator of one chain of a spin ladder
  // connects half of the vertex's states, so over all b1 a third of T's rows
  // are zero and half of T is zero or unread; stored and multiplied in full,
  // as one [L(m')] x [R(m)] block per (b1, m), the two stages at chi = 512
  // moved 2.1 x the bytes and did 1.25 x the work (9.6 against 7.9 ms in FP64,
  // with three multiplications per complex product).
  std::vector<int> by_off;  // states in the order of theta's rows and columns (class by class)
  for (const std::vector<int>& c : cls_mem) by_off.insert(by_off.end(), c.begin(), c.end());
  // sector of a0 / a2 that a state of a theta row / column carries, -1 if none
  std::vector<int> rsec((size_t)nm * d, -1), csec = rsec;
  for (int m = 0; m < nm; ++m)
    for (int q = 0; q < d; ++q) {
      if (th.rowoff[m][q] >= 0) rsec[(size_t)m * d + q] = A0.find(r.sub(th.mq[m], sigq[q]));
      if (th.coloff[m][q] >= 0) csec[(size_t)m * d + q] = A2.find(r.add(th.mq[m], sigq[q]));
    }
  std::set<int> b1s;
  for (auto& kv2 : lp_off) b1s.insert(kv2.first[0]);
  std::set<int> b1r;
  for (auto& kv2 : rp_off) b1r.insert(kv2.first[0]);
  t_base.assign((size_t)D * nm, -1);
  t_reads.assign((size_t)D * nm, {});
  struct TBlock {
    std::vector<int64_t> row, col;  // per state: first row / column in the block, -1 if absent
    int64_t rows = 0, cols = 0;
  };
  std::vector<TBlock> tb((size_t)D * nm);
  stage1 = GemmPlan();
  int64_t t_total = 0;
  t_full = 0;
  flops_executed = flops_folded_full = 0.0;
  std::vector<double> fl(nm, 0.0);  // executed flops per output sector
  for (int b1 : b1s) {
    if (!b1r.count(b1)) continue;
    for (int m = 0; m < nm; ++m) {
      int mp = th.find(r.add(th.mq[m], bq[b1]));
      if (mp < 0 || !owned[mp]) continue;  // T^{b1}_m only feeds output sector mp
      TBlock& B = tb[(size_t)b1 * nm + m];
      B.row.assign(d, -1);
      B.col.assign(d, -1);
      double k_dim = 0.0;
      for (int s1p : by_off) {
        const int sp = rsec[(size_t)mp * d + s1p];
        if (sp < 0) continue;
        bool live = false;
        for (int s1 = 0; s1 < d; ++s1) {
          const int s = rsec[(size_t)m * d + s1];
          if (s < 0 || lp_at(b1, s1p, s1, s) < 0) continue;
          live = true;
          k_dim += (double)A0.sdim[sp] * A0.sdim[s];
        }
        if (!live) continue;
        B.row[s1p] = B.rows;
        B.rows += A0.sdim[sp];
      }
      if (!B.rows) continue;
      in_need[m] = 1;
      t_full += th.nrows[mp] * th.ncols[m];
      flops_folded_full += 8.0 * k_dim * (double)th.ncols[m];
      for (int s2 : by_off) {
        const int t = csec[(size_t)m * d + s2];
        if (t < 0) continue;
        bool read = false;
        for (int s2p = 0; s2p < d; ++s2p) {
          const int tp = csec[(size_t)mp * d + s2p];
          if (tp < 0 || rp_at(b1, s2, s2p, t) < 0) continue;
          read = true;
          flops_folded_full += 8.0 * (double)th.nrows[mp] * A2.sdim[t] * (double)A2.sdim[tp];
        }
        if (!read) continue;
        B.col[s2] = B.cols;
        B.cols += A2.sdim[t];
      }
      if (!B.cols) continue;
      // ---- stage 1: one task per live state and run of neighbouring read states ----
      if (in_base[m] < 0) return fail(CMPS_ERR_ARG, "input window lacks a sector the owned outputs read");
      t_base[(size_t)b1 * nm + m] = t_total;
      std::vector<uint8_t>& rd = t_reads[(size_t)b1 * nm + m];
      for (int s2 = 0; s2 < d; ++s2) rd.push_back(B.col[s2] >= 0);
      for (int s1p : by_off) {
        if (B.row[s1p] < 0) continue;
        const int sp = rsec[(size_t)mp * d + s1p];
        for (size_t i = 0; i < by_off.size();) {
          const int s2 = by_off[i];
          if (B.col[s2] < 0) {
            ++i;
            continue;
          }
          int64_t n = 0;
          for (; i < by_off.size() && B.col[by_off[i]] == B.col[s2] + n && th.coloff[m][by_off[i]] == th.coloff[m][s2] + n; ++i)
            n += A2.sdim[csec[(size_t)m * d + by_off[i]]];
          GemmTask task{};
          task.c_off = t_total + B.row[s1p] * B.cols + B.col[s2];
          task.m = (int32_t)A0.sdim[sp];
          task.n = (int32_t)n;
          task.ldc = (int32_t)B.cols;
          task.t0 = (int32_t)stage1.terms.size();
          for (int s1 = 0; s1 < d; ++s1) {
            const int s = rsec[(size_t)m * d + s1];
            const int64_t lo = s < 0 ? -1 : lp_at(b1, s1p, s1, s);
            if (lo < 0) continue;
            GemmTerm tm{};
            tm.a_off = lo;
            tm.lda = (int32_t)A0.sdim[s];
            tm.k = (int32_t)A0.sdim[s];
            tm.b_off = in_base[m] + th.rowoff[m][s1] * th.ncols[m] + th.coloff[m][s2];
            tm.ldb = (int32_t)th.ncols[m];
            stage1.terms.push_back(tm);
            flops_executed += 8.0 * task.m * (double)task.n * tm.k;
            fl[mp] += 8.0 * task.m * (double)task.n * tm.k;
          }
          task.t1 = (int32_t)stage1.terms.size();
          stage1.tasks.push_back(task);
        }
      }
      t_total += B.rows * B.cols;
    }
  }
  t_len = t_total;  // T itself is allocated by the first folded FP64 matvec
  // ---- stage 2: Theta'_m' = sum_b1 T^{b1}_{m'-q(b1)} . RightPart^{b1} ----
  // one task per output state sigma2' and group of neighbouring states
  // sigma1' that are live for the same b1 (their rows are then neighbours in
  // every T block as well)
  stage2 = GemmPlan();
  for (int mp = 0; mp < nm; ++mp) {
    if (!owned[mp]) continue;
    if (out_base[mp] < 0) return fail(CMPS_ERR_ARG, "output window lacks an owned sector");
    std::vector<int> mof(D, -1);  // b1 -> m of its T block
    for (int b1 = 0; b1 < D; ++b1) {
      const int m = th.find(r.sub(th.mq[mp], bq[b1]));
      if (m >= 0 && t_base[(size_t)b1 * nm + m] >= 0) mof[b1] = m;
    }
    auto live_row = [&](int b1, int s1p) { return mof[b1] < 0 ? int64_t(-1) : tb[(size_t)b1 * nm + mof[b1]].row[s1p]; };
    // RightPart blocks by output state, in the order of (b1, sigma2)
    struct Read {
      int b1, s2;
      int64_t ro;
    };
    std::vector<std::vector<Read>> reads(d);
    for (int b1 = 0; b1 < D; ++b1) {
      if (mof[b1] < 0) continue;
      for (int s2 = 0; s2 < d; ++s2) {
        const int t = csec[(size_t)mof[b1] * d + s2];
        if (t < 0) continue;
        for (int s2p = 0; s2p < d; ++s2p) {
          const int64_t ro = rp_at(b1, s2, s2p, t);
          if (ro >= 0) reads[s2p].push_back(Read{b1, s2, ro});
        }
      }
    }
    for (size_t i = 0; i < by_off.size();) {
      const int first = by_off[i];
      if (th.rowoff[mp][first] < 0) {
        ++i;
        continue;
      }
      int64_t rows = 0;
      for (; i < by_off.size(); ++i) {
        const int s1p = by_off[i];
        if (th.rowoff[mp][s1p] < 0) continue;  // no rows: does not part its neighbours
        bool same = true;
        for (int b1 = 0; b1 < D && same; ++b1) same = (live_row(b1, s1p) < 0) == (live_row(b1, first) < 0);
        if (!same) break;
        rows += A0.sdim[rsec[(size_t)mp * d + s1p]];
      }
      for (int s2p = 0; s2p < d; ++s2p) {
        const int tp = csec[(size_t)mp * d + s2p];
        if (tp < 0) continue;
        GemmTask task{};
        task.c_off = out_base[mp] + th.rowoff[mp][first] * th.ncols[mp] + th.coloff[mp][s2p];
        task.m = (int32_t)rows;
        task.n = (int32_t)A2.sdim[tp];
        task.ldc = (int32_t)th.ncols[mp];
        task.t0 = (int32_t)stage2.terms.size();
        for (const Read& q : reads[s2p]) {
          const int64_t row = live_row(q.b1, first);
          if (row < 0) continue;
          const int m = mof[q.b1];
          const TBlock& B = tb[(size_t)q.b1 * nm + m];
          GemmTerm tm{};
          tm.a_off = t_base[(size_t)q.b1 * nm + m] + row * B.cols + B.col[q.s2];
          tm.lda = (int32_t)B.cols;
          tm.k = (int32_t)A2.sdim[csec[(size_t)m * d + q.s2]];
          tm.b_off = q.ro;
          tm.ldb = (int32_t)A2.sdim[tp];
          stage2.terms.push_back(tm);
          flops_executed += 8.0 * task.m * (double)task.n * tm.k;
          fl[mp] += 8.0 * task.m * (double)task.n * tm.k;
        }
        task.t1 = (int32_t)stage2.terms.size();
        stage2.tasks.push_back(task);  // a task without terms writes zeros
      }
    }
  }
  CMPS_TRY(stage1.validate(false, false, LP.len, in_len, t_total, "stage 1"));
  CMPS_TRY(stage2.validate(false, false, t_total, RP.len, out_len, "stage 2"));
  if (all_owned()) sector_flops = fl;
  CMPS_TRY(stage1.upload(ctx->stream));
  CMPS_TRY(stage2.upload(ctx->stream));
  return CMPS_OK;
}

int Heff::autotune(TuneStats* stats) {
  cudaStream_t st = ctx->stream;
  if (is_split(precision) && !low_canonical) return CMPS_OK;
  CMPS_TRY(zero_wait(x.d, sizeof(double) * 2 * x.len, st));
  if (low_canonical && ctc) return CMPS_OK;  // tcgen05 stages: fixed tiles
  if (low_canonical) return autotune_canonical(*this, true, st, stats);
  if (order == CMPS_ORDER_CANONICAL) return autotune_canonical(*this, false, st, stats);
  CMPS_TRY(ensure_T());
  Planar in, out;
  in.d = x.d;
  in.len = in_len;
  out.d = y.d;
  out.len = out_len;
  int rc = autotune_plan(stage1, 1, false, [&] { return launch_zgemm_fp64(stage1, false, false, LP, in, T, st); }, st, stats);
  if (rc == CMPS_OK)
    rc = autotune_plan(stage2, 2, false, [&] { return launch_zgemm_fp64(stage2, false, false, T, RP, out, st); }, st, stats);
  in.d = out.d = nullptr;
  return rc;
}

void Heff::default_windows() {
  in_base = th.base;
  out_base = th.base;
  in_len = out_len = th.total;
  windowed = false;
}

int Heff::set_windows(const int64_t* ib, int64_t il, const int64_t* ob, int64_t ol) {
  const int nm = (int)th.mq.size();
  if (proj_np) return fail(CMPS_ERR_STATE, "windows: the projector term needs whole vectors");
  if (il < 0 || ol < 0) return fail(CMPS_ERR_ARG, "windows: negative length");
  for (int m = 0; m < nm; ++m) {
    const int64_t sz = th.nrows[m] * th.ncols[m];
    if (in_need[m] && (ib[m] < 0 || ib[m] + sz > il)) return fail(CMPS_ERR_ARG, "input window: a read sector is outside it");
    if (owned[m] && (ob[m] < 0 || ob[m] + sz > ol)) return fail(CMPS_ERR_ARG, "output window: an owned sector is outside it");
  }
  CMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  in_base.assign(ib, ib + nm);
  out_base.assign(ob, ob + nm);
  for (int m = 0; m < nm; ++m) {
    if (!in_need[m]) in_base[m] = -1;
    if (!owned[m]) out_base[m] = -1;
  }
  in_len = il;
  out_len = ol;
  windowed = true;
  release_split(this);
  CMPS_TRY(build_plans());
  CMPS_TRY(select_order());
  if (is_split(precision)) CMPS_TRY(prepare_precision(this, precision));
  return CMPS_OK;
}

int Heff::set_owned(const uint8_t* mask) {
  const int nm = (int)th.mq.size();
  CMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  default_windows();
  for (int m = 0; m < nm; ++m) owned[m] = mask[m] ? 1 : 0;
  release_split(this);
  CMPS_TRY(build_plans());
  CMPS_TRY(select_order());
  if (is_split(precision)) CMPS_TRY(prepare_precision(this, precision));
  return CMPS_OK;
}

bool Heff::all_owned() const {
  return std::all_of(owned.begin(), owned.end(), [](uint8_t o) { return o != 0; });
}

// The folded order's intermediate T: a canonical-order or split-precision
// handle never runs the folded FP64 stages, so T (about D x the wavefunction)
// is only allocated when they first run.
int Heff::ensure_T() {
  if (T.d && T.len == t_len) return CMPS_OK;
  return T.alloc(t_len);
}

// which = 1: the first half of the matvec (folded: T = LeftPart . in;
// canonical: stages L and W1), 2: the second half.
int Heff::apply_stage(int which, const Planar& in, Planar& out, cudaStream_t st) {
  if (is_split(precision)) return apply_split_stage(*this, which, in, out, st);
  if (order == CMPS_ORDER_CANONICAL) return apply_canonical(*this, which, in, out, st);
  CMPS_TRY(ensure_T());
  if (which == 1) return launch_zgemm_fp64(stage1, false, false, LP, in, T, st);
  return launch_zgemm_fp64(stage2, false, false, T, RP, out, st);
}

int Heff::apply_theta(const Planar& in, Planar& out, cudaStream_t st) {
  if (is_split(precision)) return apply_split(*this, in, out, st);
  CMPS_TRY(apply_stage(1, in, out, st));
  CMPS_TRY(apply_stage(2, in, out, st));
  return add_projectors(in, out, st);
}

int Heff::apply_fp64_stages(const Planar& in, Planar& out, cudaStream_t st) {
  if (order == CMPS_ORDER_CANONICAL) return apply_canonical(*this, 0, in, out, st);
  return apply_folded_fp64(in, out, st);
}

int Heff::apply_folded_fp64(const Planar& in, Planar& out, cudaStream_t st) {
  CMPS_TRY(ensure_T());
  CMPS_TRY(launch_zgemm_fp64(stage1, false, false, LP, in, T, st));
  CMPS_TRY(launch_zgemm_fp64(stage2, false, false, T, RP, out, st));
  return CMPS_OK;
}

int Heff::apply_theta_fp64(const Planar& in, Planar& out, cudaStream_t st) {
  CMPS_TRY(apply_fp64_stages(in, out, st));
  return add_projectors(in, out, st);
}

namespace {
// h[2p], h[2p+1] = -w_p * c_p (c_p = <phi_p, x>, times *scale unless null), for
// the subtracting multi-axpy
__global__ void k_proj_coef(const double* __restrict__ c, const double* __restrict__ w, int np,
                            const double* __restrict__ scale, double* __restrict__ h) {
  const int p = threadIdx.x;
  if (p < np) {
    const double f = scale ? -w[p] * *scale : -w[p];
    h[2 * p] = f * c[2 * p];
    h[2 * p + 1] = f * c[2 * p + 1];
  }
}
}  // namespace

int Heff::set_projectors(int np, const double* host_arpack, const double* weights) {
  CMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  proj.release();
  if (d_proj) dfree(d_proj);
  d_proj = nullptr;
  proj_np = 0;
  proj_w.clear();
  if (np == 0) return CMPS_OK;
  if (np < 0 || np > 64) return fail(CMPS_ERR_ARG, "projectors: between 0 and 64 of them");
  if (!host_arpack || !weights) return fail(CMPS_ERR_ARG, "projectors: null argument");
  if (windowed) return fail(CMPS_ERR_STATE, "projectors: the matvec has vector windows (sharded)");
  const int64_t n = th.total;
  CMPS_TRY(proj.alloc((int64_t)np * n));
  CMPS_CUDA(dmalloc(&d_proj, sizeof(double) * (3 * (size_t)np + 4)));
  cudaStream_t st = ctx->stream;
  std::vector<double> buf(2 * (size_t)n_allowed);
  for (int p = 0; p < np; ++p) {
    const double* src = host_arpack + 2 * (size_t)n_allowed * p;
    for (int64_t i = 0; i < n_allowed; ++i) {  // phi = conj(P)
      buf[2 * i] = src[2 * i];
      buf[2 * i + 1] = -src[2 * i + 1];
    }
    CMPS_TRY(copy_wait(d_io, buf.data(), sizeof(double) * 2 * n_allowed, cudaMemcpyHostToDevice, st));
    Planar v;
    v.d = proj.d + 2 * n * p;
    v.len = n;
    const int rc = pack(d_io, v, st);
    v.d = nullptr;
    CMPS_TRY(rc);
  }
  proj_w.assign(weights, weights + np);
  CMPS_TRY(copy_wait(d_proj, proj_w.data(), sizeof(double) * np, cudaMemcpyHostToDevice, st));
  CMPS_CUDA(cudaStreamSynchronize(st));
  proj_np = np;
  return CMPS_OK;
}

int Heff::set_projectors_device(int np, const double* d_phi_arpack, const double* weights) {
  CMPS_CUDA(cudaStreamSynchronize(ctx->stream));
  proj.release();
  if (d_proj) dfree(d_proj);
  d_proj = nullptr;
  proj_np = 0;
  proj_w.clear();
  if (np == 0) return CMPS_OK;
  if (np < 0 || np > 64) return fail(CMPS_ERR_ARG, "projectors: between 0 and 64 of them");
  if (!d_phi_arpack || !weights) return fail(CMPS_ERR_ARG, "projectors: null argument");
  const int64_t n = th.total;
  CMPS_TRY(proj.alloc((int64_t)np * n));
  CMPS_CUDA(dmalloc(&d_proj, sizeof(double) * (3 * (size_t)np + 4)));
  cudaStream_t st = ctx->stream;
  for (int p = 0; p < np; ++p) {
    Planar v;
    v.d = proj.d + 2 * n * p;
    v.len = n;
    const int rc = pack(d_phi_arpack + 2 * (size_t)n_allowed * p, v, st);
    v.d = nullptr;
    CMPS_TRY(rc);
  }
  proj_w.assign(weights, weights + np);
  CMPS_TRY(copy_wait(d_proj, proj_w.data(), sizeof(double) * np, cudaMemcpyHostToDevice, st));
  CMPS_CUDA(cudaStreamSynchronize(st));
  proj_np = np;
  return CMPS_OK;
}

int Heff::add_projectors(const Planar& in, Planar& out, cudaStream_t st, const double* scale) {
  if (!proj_np) return CMPS_OK;
  const int64_t n = th.total;
  // d_proj: weights [0, np), then c = <phi_p, x> (2 np) and |x|^2, then one
  // scratch norm; the coefficients are turned into -w_p c_p in place
  double* c = d_proj + proj_np;
  CMPS_TRY(ops.mdot_dev(proj.d, proj.d + n, 2 * n, proj_np, in.re(), in.im(), c, st));
  k_proj_coef<<<1, 64, 0, st>>>(c, d_proj, proj_np, scale, c);
  CMPS_CUDA(cudaGetLastError());
  return ops.maxpy_norm_dev(proj.d, proj.d + n, 2 * n, proj_np, c, out.re(), out.im(), c + 2 * proj_np + 1, st);
}

int Heff::apply_device(const double* din, double* dout, cudaStream_t st) {
  if (!whole()) return fail(CMPS_ERR_STATE, "matvec is sharded: use the theta-layout entry point");
  if (is_split(precision) && split_reads_arpack(*this)) {
    CMPS_TRY(apply_split_arpack(*this, din, y, st));
    return unpack(y, dout, st);
  }
  CMPS_TRY(pack(din, x, st));
  if (is_split(precision)) {
    CMPS_TRY(apply_split_stage(*this, 1, x, y, st));
    CMPS_TRY(apply_split_stage(*this, 2, x, y, st));
    CMPS_TRY(add_projectors(x, y, st));
  } else {
    CMPS_TRY(apply_theta(x, y, st));
  }
  CMPS_TRY(unpack(y, dout, st));
  return CMPS_OK;
}

int Heff::apply_host(const double* in, double* out) {
  cudaStream_t st = ctx->stream;
  size_t bytes = sizeof(double) * 2 * n_allowed;
  CMPS_CUDA(cudaMemcpyAsync(d_io, in, bytes, cudaMemcpyHostToDevice, st));
  CMPS_TRY(apply_device(d_io, d_io, st));
  CMPS_CUDA(cudaMemcpyAsync(out, d_io, bytes, cudaMemcpyDeviceToHost, st));
  CMPS_CUDA(cudaStreamSynchronize(st));
  if (is_split(precision)) CMPS_TRY(split_error(*this));
  return CMPS_OK;
}

// ---------------------------------------------------------------------------
// Lowest eigenpair of the symmetric tridiagonal matrix with diagonal a[0..k)
// and off-diagonal b[0..k-1): the eigenvalue by Sturm-sequence bisection,
// the vector by two steps of inverse iteration with a row-pivoted
// tridiagonal LU.  O(k) per bisection step, so it runs after every Lanczos
// step.
static void tridiag_lowest(int k, const double* a, const double* b, double* lam, std::vector<double>& y) {
  y.assign(k, 0.0);
  if (k == 1) {
    *lam = a[0];
    y[0] = 1.0;
    return;
  }
  double lo = a[0], hi = a[0];
  for (int i = 0; i < k; ++i) {
    const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < k ? std::fabs(b[i]) : 0.0);
    lo = std::min(lo, a[i] - r);
    hi = std::max(hi, a[i] + r);
  }
  const double eps = 2.220446049250313e-16;
  const double scale = std::max({std::fabs(lo), std::fabs(hi), 1e-300});
  const double pivmin = eps * scale;
  // number of eigenvalues below x (signs of the LDL^T pivots of T - x)
  auto below = [&](double x) {
    int c = 0;
    double d = 1.0;
    for (int i = 0; i < k; ++i) {
      double q = a[i] - x - (i > 0 ? b[i - 1] * b[i - 1] / d : 0.0);
      if (std::fabs(q) < pivmin) q = -pivmin;
      if (q < 0.0) ++c;
      d = q;
    }
    return c;
  };
  lo -= pivmin;
  hi += pivmin;
  for (int it = 0; it < 200 && hi - lo > 2.0 * eps * scale; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (below(mid) >= 1) hi = mid;
    else lo = mid;
  }
  *lam = 0.5 * (lo + hi);
  // inverse iteration: (T - lam) z = r
  std::vector<double> d(k), dl(k), du(k), du2(k), z(k, 1.0);
  std::vector<char> swapped(k, 0);
  for (int i = 0; i < k; ++i) d[i] = a[i] - *lam;
  for (int i = 0; i + 1 < k; ++i) dl[i] = du[i] = b[i];
  for (int i = 0; i + 1 < k; ++i) {
    du2[i] = 0.0;
    if (std::fabs(d[i]) >= std::fabs(dl[i])) {
      if (d[i] == 0.0) d[i] = pivmin;
      const double f = dl[i] / d[i];
      dl[i] = f;
      d[i + 1] -= f * du[i];
    } else {
      // exchange rows i and i+1
      const double f = d[i] / dl[i];
      d[i] = dl[i];
      dl[i] = f;
      const double t = du[i];
      du[i] = d[i + 1];
      d[i + 1] = t - f * d[i + 1];
      if (i + 2 < k) {
        du2[i] = du[i + 1];
        du[i + 1] = -f * du[i + 1];
      }
      swapped[i] = 1;
    }
  }
  if (d[k - 1] == 0.0) d[k - 1] = pivmin;
  for (int pass = 0; pass < 2; ++pass) {
    for (int i = 0; i + 1 < k; ++i) {
      if (!swapped[i]) {
        z[i + 1] -= dl[i] * z[i];
      } else {
        const double t = z[i] - dl[i] * z[i + 1];
        z[i] = z[i + 1];
        z[i + 1] = t;
      }
    }
    z[k - 1] /= d[k - 1];
    z[k - 2] = (z[k - 2] - du[k - 2] * z[k - 1]) / d[k - 2];
    for (int i = k - 3; i >= 0; --i) z[i] = (z[i] - du[i] * z[i + 1] - du2[i] * z[i + 2]) / d[i];
    double nz = 0.0;
    for (double v : z) nz += v * v;
    nz = std::sqrt(nz);
    for (double& v : z) v /= nz;
  }
  y = z;
}

// Steps that take less than this on the device are issued one ahead of the
// host.  That hides the host's turn, 5 us of a step with the split operator and
// 25 us of an FP64 one, but a cycle's end wastes a step.
// Eigensolve of a growth step with never, short and all steps ahead, ms: XXZ
// chain at chi = 100, mixed, 2.76, 2.45, 2.46; ladder, mixed, chi = 64 7.20, 6.92,
// 6.93, chi = 125 16.18, 16.04, 16.23, chi = 165 24.19, 24.21, 24.38; Ising chains,
// chi = 6, mixed (1.4 ms a step) 137.8, 138.0, 140.4.
constexpr float kStepAheadMs = 0.2f;

// Restarted Lanczos with full re-orthogonalisation (the local three-term
// step, then one classical Gram-Schmidt pass against the whole basis),
// coefficients kept on the device and a convergence check after every step.
//
// FP64 operator: every step uses the FP64 matvec; the run ends when the Ritz
// residual estimate |beta_j y_j| falls below tol |lambda|.
//
// Split-TF32 operator (accurate to ~1e-5 relative): every restart cycle
// opens with an FP64 matvec of its start vector x, which gives the FP64
// Rayleigh quotient alpha_0 and the true residual beta_0 = |H x - alpha_0 x|;
// the run ends there once beta_0 <= tol |alpha_0|, with energy alpha_0.  The
// remaining steps of a cycle use the split operator and stop once the Ritz
// estimate has dropped by the cycle's factor eta_c below beta_0 (adapted
// from cycle to cycle, as described where it is declared).  A cycle therefore
// contracts the error of x by about max(eta, |dH| / gap) at the cost of one
// FP64 matvec, as in mixed-precision iterative refinement; if two cycles in a
// row fail to halve beta_0, the remaining cycles run in FP64.
int Heff::eigs(const double* guess, double tol, int max_restarts, int kdim, double* eval, double* evec,
               int* matvecs, bool start_in_x) {
  cudaStream_t st = ctx->stream;
  const int64_t n = th.total;
  if (n == 0) return fail(CMPS_ERR_STATE, "empty effective Hamiltonian");
  if (!whole()) return fail(CMPS_ERR_STATE, "matvec is sharded: the single-GPU eigensolver needs every sector");
  if (kdim < 2) kdim = 2;
  if (kdim > 96) kdim = 96;
  if ((int64_t)kdim > n) kdim = (int)n;
  if (kv_dim != kdim || kv.len != (int64_t)kdim * n) {
    CMPS_TRY(kv.alloc((int64_t)kdim * n));
    kv_dim = kdim;
  }
  if (!h_ab) CMPS_CUDA(cudaMallocHost(&h_ab, sizeof(double) * 8));
  const int64_t ldv = 2 * n;
  auto vre = [&](int j) { return kv.d + (int64_t)j * ldv; };
  auto view = [&](int j) {
    Planar p;
    p.d = vre(j);
    p.len = n;
    return p;
  };
  double* nrm = ops.d_coef + 900;  // clear of the Lanczos coefficients
  eig_stats = EigStats{};
  // per step in flight (two at most): matvec begin and end, step done; and the
  // whole solve
  cudaEvent_t ev[8] = {};
  struct EvGuard {
    cudaEvent_t* e;
    ~EvGuard() {
      for (int i = 0; i < 8; ++i)
        if (e[i]) cudaEventDestroy(e[i]);
    }
  } ev_guard{ev};
  for (auto& e : ev) CMPS_CUDA(cudaEventCreate(&e));
  CMPS_CUDA(cudaEventRecord(ev[6], st));
  // start vector into x
  if (guess) {
    CMPS_CUDA(cudaMemcpyAsync(d_io, guess, sizeof(double) * 2 * n_allowed, cudaMemcpyHostToDevice, st));
    CMPS_TRY(pack(d_io, x, st));
  }
  double nrm0 = 0.0;
  const bool have_start = guess || start_in_x;
  if (have_start) CMPS_TRY(ops.norm2(x.re(), x.im(), &nrm0, st));
  if (!have_start || !(nrm0 > 1e-300)) CMPS_TRY(ops.random(x.re(), x.im(), 0x5eed1234ULL, st));
  CMPS_TRY(ops.mdot_dev(nullptr, nullptr, 0, 0, x.re(), x.im(), nrm, st));
  CMPS_TRY(ops.scale_dev(x.re(), x.im(), nrm, x.re(), x.im(), st));
  h_ab[4] = 1.0;  // a cycle's first basis vector is normalised
  CMPS_CUDA(cudaMemcpyAsync(ops.lanczos_coef().scale, h_ab + 4, sizeof(double), cudaMemcpyHostToDevice, st));

  const bool mixed = is_split(precision);
  if (mixed) CMPS_TRY(split_reset_error(*this, st));
  bool all_fp64 = !mixed;
  const int max_cycles = std::max(1, max_restarts) * (mixed ? 4 : 1);
  // Per-cycle contraction asked of the split steps.  A cycle's FP64 residual
  // shows what the previous cycle's split steps achieved: if they reached
  // their request, the next request is 30x stronger; if not, they met the
  // floor |dH|/gap of the split operator (or the Krylov cap), and the next
  // request is what they achieved.  No cycle asks for more than the
  // tolerance still needs (with a margin of 10).
  double eta = 1e-3;
  double eta_c = eta, prev_eta_c = eta;
  double prev_beta0 = HUGE_VAL;
  int stalls = 0, nmv = 0;
  double lam = 0.0;
  bool converged = false;
  std::vector<double> al, be, ycoef;
  // the last step's device time, FP64 and split; before the first one, short
  // for vectors whose passes are
  float step_ms[2] = {n <= 32768 ? 0.f : HUGE_VALF, HUGE_VALF};
  for (int cycle = 0; cycle < max_cycles && !converged; ++cycle) {
    ++eig_stats.cycles;
    CMPS_CUDA(cudaMemcpyAsync(vre(0), x.d, sizeof(double) * 2 * n, cudaMemcpyDeviceToDevice, st));
    al.clear();
    be.clear();
    int k = 0;
    double beta0 = -1.0;
    bool split_used = false;
    // Step j: y = H U_j, or y = H V_j in split precision, whose operands have
    // the range of 32 bits while U_j is of H's own size; then the three passes
    // of VecOps::lanczos.  The vector after the last step's is not part of the
    // basis and not stored.
    auto issue = [&](int j) -> int {
      cudaEvent_t* e = ev + 3 * (j & 1);
      Planar vj = view(j);
      CMPS_CUDA(cudaEventRecord(e[0], st));
      const bool split = !all_fp64 && j > 0;
      if (split) {
        CMPS_TRY(apply_split_async(*this, vj, y, st, ops.lanczos_coef().scale + j));
        split_used = true;
      } else {
        CMPS_TRY(apply_theta_fp64(vj, y, st));
      }
      CMPS_CUDA(cudaEventRecord(e[1], st));
      double* out = j + 1 < kdim ? vre(j + 1) : nullptr;
      CMPS_TRY(ops.lanczos(kv.d, ldv, y.re(), y.im(), split, j, out, out ? out + n : nullptr, h_ab + 2 * (j & 1), st));
      CMPS_CUDA(cudaEventRecord(e[2], st));
      return CMPS_OK;
    };
    // the matvec of step j, which has run
    auto count_matvec = [&](int j) -> int {
      float ms = 0.f;
      CMPS_CUDA(cudaEventElapsedTime(&ms, ev[3 * (j & 1)], ev[3 * (j & 1) + 1]));
      const bool fp64 = all_fp64 || j == 0;
      ++(fp64 ? eig_stats.mv_fp64 : eig_stats.mv_split);
      (fp64 ? eig_stats.ms_fp64 : eig_stats.ms_split) += ms;
      return CMPS_OK;
    };
    int issued = 0;
    for (int j = 0; j < kdim; ++j) {
      const int kind = all_fp64 || j == 0 ? 0 : 1;
      // Short steps: the next one is issued before this one's coefficients are
      // read (it needs them on the device only).  A cycle that ends at this step
      // drops the extra one: its vector lies past the basis.
      const int upto = (all_fp64 || j > 0) && step_ms[kind] < kStepAheadMs ? std::min(j + 1, kdim - 1) : j;
      while (issued <= upto) CMPS_TRY(issue(issued++));
      cudaEvent_t* e = ev + 3 * (j & 1);
      CMPS_CUDA(cudaEventSynchronize(e[2]));
      ++nmv;
      CMPS_TRY(count_matvec(j));
      CMPS_CUDA(cudaEventElapsedTime(&step_ms[kind], e[0], e[2]));
      const double a = h_ab[2 * (j & 1)], b = h_ab[2 * (j & 1) + 1];
      al.push_back(a);
      be.push_back(b);
      k = j + 1;
      const bool exhausted = !(b > 1e-14 * std::max(1.0, std::fabs(a)));
      tridiag_lowest(k, al.data(), be.data(), &lam, ycoef);
      const double resid = exhausted ? 0.0 : std::fabs(b * ycoef[k - 1]);
      if (all_fp64) {
        if (resid <= tol * std::max(1.0, std::fabs(lam))) {
          converged = true;
          break;
        }
        continue;
      }
      if (j == 0) {
        beta0 = b;
        if (exhausted || b <= tol * std::max(1.0, std::fabs(a))) {
          converged = true;  // x is the eigenvector; alpha_0 its FP64 energy
          lam = a;
          break;
        }
        if (prev_beta0 < HUGE_VAL) {
          const double got = b / prev_beta0;
          if (got > 0.5) {
            if (++stalls >= 2) all_fp64 = true;
          } else {
            stalls = 0;
          }
          eta = got <= 2.0 * prev_eta_c ? std::max(1e-10, prev_eta_c * 0.03) : std::min(0.1, got);
        }
        eta_c = std::min(0.5, std::max(eta, 0.1 * tol * std::max(1.0, std::fabs(a)) / b));
        prev_beta0 = b;
        prev_eta_c = eta_c;
      } else if (exhausted || resid <= eta_c * beta0) {
        break;
      }
    }
    if (split_used) CMPS_TRY(split_error(*this));
    if (converged && !all_fp64 && k == 1) break;
    // Ritz vector x = sum_j y_j V_j, V_j = U_j / beta_{j-1}, normalised
    for (int j = 1; j < k; ++j)
      ycoef[j] *= be[j - 1] > 1e-14 * std::max(1.0, std::fabs(al[j - 1])) ? 1.0 / be[j - 1] : 0.0;
    CMPS_TRY(ops.combine(kv.d, kv.d + n, ldv, k, ycoef.data(), x.re(), x.im(), st));
    CMPS_TRY(ops.mdot_dev(nullptr, nullptr, 0, 0, x.re(), x.im(), nrm, st));
    CMPS_TRY(ops.scale_dev(x.re(), x.im(), nrm, x.re(), x.im(), st));
    if (issued > k) {  // a step issued ahead and dropped: its matvec has run all the same
      CMPS_CUDA(cudaEventSynchronize(ev[3 * (k & 1) + 1]));
      CMPS_TRY(count_matvec(k));
    }
  }
  CMPS_CUDA(cudaEventRecord(ev[7], st));
  // HED post-processing (DMRG_routines.cpp:870-889)
  double mx2 = 0.0;
  int64_t imx = 0;
  CMPS_TRY(ops.absmax(x.re(), x.im(), &mx2, &imx, st));
  double mr = 0.0, mi = 0.0;
  CMPS_CUDA(cudaMemcpyAsync(&mr, x.re() + imx, sizeof(double), cudaMemcpyDeviceToHost, st));
  CMPS_CUDA(cudaMemcpyAsync(&mi, x.im() + imx, sizeof(double), cudaMemcpyDeviceToHost, st));
  CMPS_CUDA(cudaStreamSynchronize(st));
  double mabs = std::sqrt(mx2);
  // phase = |max| / max = conj(max) / |max|
  double pr = mr / mabs, pi = -mi / mabs;
  CMPS_TRY(ops.phase_drop(x.re(), x.im(), pr, pi, 2.220446049250313e-16 * mabs, st));
  if (theta.len != n) CMPS_TRY(theta.alloc(n));
  CMPS_CUDA(cudaMemcpyAsync(theta.d, x.d, sizeof(double) * 2 * n, cudaMemcpyDeviceToDevice, st));
  have_theta = true;
  if (evec) {
    CMPS_TRY(unpack(theta, d_io, st));
    CMPS_CUDA(cudaMemcpyAsync(evec, d_io, sizeof(double) * 2 * n_allowed, cudaMemcpyDeviceToHost, st));
  }
  CMPS_CUDA(cudaStreamSynchronize(st));
  float total_ms = 0.f;
  CMPS_CUDA(cudaEventElapsedTime(&total_ms, ev[6], ev[7]));
  eig_stats.ms_total = total_ms;
  *eval = lam;
  if (matvecs) *matvecs = nmv;
  if (!converged) return fail(CMPS_ERR_SOLVER, "Lanczos did not reach the requested residual");
  return CMPS_OK;
}

}  // namespace cmps
