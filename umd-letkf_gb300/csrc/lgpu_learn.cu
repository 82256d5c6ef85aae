// lgpu_learn.cu -- kernels of the learned analysis form.
//
// The reference solves every grid column exactly (src/letkf_solver.F90:
// 203-384, one letkf_core_solve per column and group).  The learned form
// solves exactly only the columns of a coarse lattice (every s-th column in
// longitude and latitude), a random judge sample and the columns its
// confidence gate sends back; every other column gets the bilinear
// interpolation of the coarse solutions (W, w-bar) plus a correction from
// the network of lgpu_mlp.cu.  The analysis update itself is unchanged.
//
//   k_lrn_cellstats, k_lrn_obsfeat  per column: the observation-geometry
//                  features (local count, sums of localisation weights,
//                  nearest distance, innovation moments) from per-cell
//                  aggregates of the observation index and the same
//                  localizer as the exact path
//   k_lrn_interp   per column, while collecting training data: the bilinear
//                  (W, w-bar) of the four coarse neighbours as a raw input
//                  row, and the residual target exact - interpolated
//   k_lrn_input    per column: the same inputs standardised, as BF16 in the
//                  network's tiled order
//   k_lrn_apply    per column: interpolation + de-standardised correction ->
//                  T = W + w-bar 1^T, the gate score, the fallback list
//   k_lrn_judge, k_lrn_scatter  judge errors; exact transforms into place
//   k_lrn_colstats, k_lrn_batch  training-set standardisation and batches
#include "lgpu_internal.cuh"
#include <cuda_bf16.h>

namespace lgpu {

namespace {

constexpr int FT = 128;   // threads of the per-column kernels

__device__ __forceinline__ float bsum128(float v, float *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  return red[0] + red[1] + red[2] + red[3];
}

// Per-cell aggregates of the cell-sorted observation table: centroid
// direction (sum of unit vectors) and count; sums of dep, dep^2, 1/err,
// dep/err.  One thread per cell.
__global__ void k_lrn_cellstats(int ncell, ObsSorted obs, float4 *c0, float4 *c1) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int b = obs.cell_start[c], e = obs.cell_start[c + 1];
  float sx = 0.f, sy = 0.f, sz = 0.f, sd = 0.f, sd2 = 0.f, si = 0.f, sdi = 0.f;
  for (int p = b; p < e; p++) {
    const float4 A = obs.A[p];
    const float dep = obs.B[p].x, ie = 1.0f / A.w;
    sx += A.x; sy += A.y; sz += A.z;
    sd += dep; sd2 += dep * dep; si += ie; sdi += dep * ie;
  }
  c0[c] = make_float4(sx, sy, sz, (float)(e - b));
  c1[c] = make_float4(sd, sd2, si, sdi);
}

// Observation-geometry features of column cols[f] from the cell aggregates
// of its search window (one warp per column; a cell's observations are
// taken at the cell's centroid):
//   0 count within the search radius / 100   1 sum rho / 100
//   2 sum rho/err / 1000   3 nearest centroid distance / search radius (1 if none)
//   4 mean dep   5 variance of dep   6 rho-weighted mean dep
//   7 (rho/err)-weighted mean dep   8 max rho   9 mean rho
// (features 10-15 are filled by k_lrn_interp)
__global__ void __launch_bounds__(FT) k_lrn_obsfeat(int nfine, const int *cols, const ColPar *cps, DevLoc loc,
                                                    const int *cell_start, const float4 *c0, const float4 *c1,
                                                    const IndexGeom *geom, float *feat, int *nkept) {
  // the index geometry from shared memory: its two loads per band were part
  // of the kernel's latency chain (315 us for 38,307 columns, now 287)
  __shared__ IndexGeom gs;
  for (int t = threadIdx.x; t < (int)(sizeof(IndexGeom) / 4); t += FT)
    reinterpret_cast<int *>(&gs)[t] = reinterpret_cast<const int *>(geom)[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int f = blockIdx.x * (FT / 32) + (threadIdx.x >> 5);
  if (f >= nfine) return;   // whole warps
  const int col = cols[f];
  const ColPar cp = cps[col];
  float n = 0.f, sr = 0.f, sre = 0.f, dmin = 3.0e38f, sd = 0.f, sd2 = 0.f, srd = 0.f, sred = 0.f, rmx = 0.f;
  for (int b = cp.b0; b <= cp.b1; b++) {
    const int nl = gs.nlon[b], off = gs.off[b];
    int lo = 0, cnt = nl;
    if (cp.dlon < 180.0f) {
      const int clo = (int)floorf((cp.lonn - cp.dlon) * (float)nl / 360.0f);
      const int chi = (int)floorf((cp.lonn + cp.dlon) * (float)nl / 360.0f);
      if (chi - clo + 1 < nl) { lo = clo; cnt = chi - clo + 1; }
    }
    for (int q = lane; q < cnt; q += 32) {
      // the window starts within a turn of the band (lonn in [0, 360), dlon < 180)
      int c = lo + q;
      c = c < 0 ? c + nl : (c >= nl ? c - nl : c);
      const int cell = off + c;
      const float4 A = c0[cell];
      if (A.w <= 0.0f) continue;
      const float inv = rsqrtf(A.x * A.x + A.y * A.y + A.z * A.z);
      const float d = dist_from_chord2(chord2_exact(cp.ux, cp.uy, cp.uz, A.x * inv, A.y * inv, A.z * inv));
      if (d > cp.rmax) continue;
      const float r = localize(loc, cp, 0, d, 0.0f, 0.0f, 0.0f);
      if (!(r > kKeep)) continue;
      const float4 B = c1[cell];
      n += A.w;
      sr += r * A.w;
      sre += r * B.z;
      dmin = fminf(dmin, d);
      sd += B.x;
      sd2 += B.y;
      srd += r * B.x;
      sred += r * B.w;
      rmx = fmaxf(rmx, r);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    n += __shfl_xor_sync(0xffffffffu, n, o);
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    sre += __shfl_xor_sync(0xffffffffu, sre, o);
    sd += __shfl_xor_sync(0xffffffffu, sd, o);
    sd2 += __shfl_xor_sync(0xffffffffu, sd2, o);
    srd += __shfl_xor_sync(0xffffffffu, srd, o);
    sred += __shfl_xor_sync(0xffffffffu, sred, o);
    dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    rmx = fmaxf(rmx, __shfl_xor_sync(0xffffffffu, rmx, o));
  }
  if (lane == 0) {
    float *o = feat + (size_t)f * 16;
    const float nn = fmaxf(n, 1.0f);
    const float m = sd / nn;
    o[0] = n / 100.0f;
    o[1] = sr / 100.0f;
    o[2] = sre / 1000.0f;
    o[3] = n > 0.0f ? dmin / cp.rmax : 1.0f;
    o[4] = m;
    o[5] = fmaxf(sd2 / nn - m * m, 0.0f);
    o[6] = sr > 0.0f ? srd / sr : 0.0f;
    o[7] = sre > 0.0f ? sred / sre : 0.0f;
    o[8] = rmx;
    o[9] = sr / nn;
    nkept[f] = (int)n;
  }
}

struct Nb {
  int src[4];
  float w[4];
  int missing;
  float fx, fy;
};

// the four coarse neighbours of column (i, j) on the lattice of stride s
// (periodic in longitude, clamped at the last coarse latitude row) and
// their bilinear weights; src = row of the coarse solution or -1
__device__ __forceinline__ Nb neighbours(int col, int nx, int ny, int s, const int *src_of_col) {
  Nb nb;
  const int i = col % nx, j = col / nx;
  const int i0 = (i / s) * s, j0 = (j / s) * s;
  const int i1 = (i0 + s) % nx;
  const int j1 = j0 + s < ny ? j0 + s : j0;
  nb.fx = (float)(i - i0) / (float)s;
  nb.fy = j1 != j0 ? (float)(j - j0) / (float)s : 0.0f;
  const int c[4] = {i0 + nx * j0, i1 + nx * j0, i0 + nx * j1, i1 + nx * j1};
  const float w[4] = {(1.0f - nb.fx) * (1.0f - nb.fy), nb.fx * (1.0f - nb.fy), (1.0f - nb.fx) * nb.fy, nb.fx * nb.fy};
  nb.missing = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    nb.src[q] = src_of_col[c[q]];
    nb.w[q] = w[q];
    if (w[q] > 0.0f && nb.src[q] < 0) nb.missing = 1;
  }
  return nb;
}

// interpolated W_ij (i < k, j < k) or w-bar_i (j == k) of the neighbours
__device__ __forceinline__ float interp_at(const Nb &nb, const float *Ts, const float *ws, int k, int i, int j) {
  float v = 0.0f;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (nb.w[q] == 0.0f || nb.src[q] < 0) continue;
    const float wb = ws[(size_t)nb.src[q] * k + i];
    const float t = j < k ? Ts[(size_t)nb.src[q] * k * k + (size_t)i * k + j] - wb : wb;
    v += nb.w[q] * t;
  }
  return v;
}

}  // namespace

namespace {

// feature q of the 16 that follow the transform: observation geometry,
// latitude, position in the lattice cell, the neighbours' spread
__device__ __forceinline__ float geometry_feature(const LrnInterpArgs &a, int f, int col, const Nb &nb, float spread,
                                                  int q) {
  const float *fo = a.feat + (size_t)f * 16;
  if (q < 10) return fo[q];
  if (q == 10) return sinf(a.lat[col] * 0.017453292519943295f);
  if (q == 11) return cosf(a.lat[col] * 0.017453292519943295f);
  if (q == 12) return nb.fx;
  if (q == 13) return nb.fy;
  if (q == 14) return log1pf(100.0f * fo[0]);
  return sqrtf(spread) / (float)a.k;
}

// raw rows for the training store
__global__ void __launch_bounds__(FT) k_lrn_interp(LrnInterpArgs a) {
  __shared__ float red[4];
  const int f = blockIdx.x;
  if (f >= a.nfine) return;
  const int col = a.cols[f], k = a.k, kk = k * k;
  const Nb nb = neighbours(col, a.nx, a.ny, a.s, a.src_of_col);
  float *x = a.X + (size_t)f * a.ldx;
  // interpolated W (row-major) and w-bar; spread of the neighbours around it
  float spread = 0.0f;
  for (int e = threadIdx.x; e < kk + k; e += FT) {
    const int i = e < kk ? e / k : e - kk, j = e < kk ? e % k : k;
    const float v = interp_at(nb, a.Ts, a.ws, k, i, j);
    if (e < kk) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (nb.w[q] == 0.0f || nb.src[q] < 0) continue;
        const float wb = a.ws[(size_t)nb.src[q] * k + i];
        const float d = a.Ts[(size_t)nb.src[q] * kk + (size_t)i * k + j] - wb - v;
        spread += nb.w[q] * d * d;
      }
    }
    x[e] = v;
    if (a.Yt) {
      const int act = a.col2act[col];
      const float ex = a.wex[(size_t)act * k + i];
      const float t = j < k ? a.Tex[(size_t)act * kk + (size_t)i * k + j] - ex : ex;
      a.Yt[(size_t)f * a.ldy + e] = t - v;
    }
  }
  spread = bsum128(spread, red);
  if (threadIdx.x < 16) {
    const int q = threadIdx.x;
    const float v = geometry_feature(a, f, col, nb, spread, q);
    const int e = kk + k + q;
    x[e] = v;
  }
  if (threadIdx.x == 0) a.flag[f] = nb.missing;
}

// The same inputs for inference, standardised, rounded and written in the
// network's tiled order, a block per row (rows past nfine: zeros).  With
// QUADS (k a multiple of 4: 16-byte rows of T, and no quad crosses one) four
// elements share the row's w-bar and the index division.  Before, k_lrn_interp
// wrote FP32 rows, element by element, and another kernel read and tiled them
// (455 us for 38,307 columns at k = 32, now 185).
template <bool QUADS>
__global__ void __launch_bounds__(FT) k_lrn_input(LrnInterpArgs a, int k1, unsigned char *Xt) {
  extern __shared__ __align__(16) __nv_bfloat16 row[];   // [k1]
  __shared__ float red[4];
  __shared__ float wsm[4][128];
  const int f = blockIdx.x;
  // this row's 16-byte groups of the tiled matrix (row blocks of 128): group
  // c8 of K slice c8 / 2
  unsigned char *dst = Xt + (size_t)(f >> 7) * (size_t)(k1 >> 4) * 4096 + (size_t)((f & 127) >> 3) * 256 +
                       (size_t)(f & 7) * 16;
  auto put = [&](int c8, uint4 v) {
    *reinterpret_cast<uint4 *>(dst + (size_t)(c8 >> 1) * 4096 + (size_t)(c8 & 1) * 128) = v;
  };
  if (f >= a.nfine) {
    for (int c8 = threadIdx.x; c8 < k1 >> 3; c8 += FT) put(c8, make_uint4(0, 0, 0, 0));
    return;
  }
  const int col = a.cols[f], k = a.k, kk = k * k;
  const Nb nb = neighbours(col, a.nx, a.ny, a.s, a.src_of_col);
  bool on[4];
  const float *T[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    on[q] = nb.w[q] != 0.0f && nb.src[q] >= 0;
    T[q] = a.Ts + (size_t)(on[q] ? nb.src[q] : 0) * kk;
    for (int i = threadIdx.x; i < k; i += FT) wsm[q][i] = on[q] ? a.ws[(size_t)nb.src[q] * k + i] : 0.0f;
  }
  __syncthreads();
  float spread = 0.0f;
  constexpr int V = QUADS ? 4 : 1;
  for (int e = V * threadIdx.x; e < kk; e += V * FT) {
    const int i = e / k;
    float t[4][V], v[V];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (QUADS) {
        const float4 x = on[q] ? __ldg(reinterpret_cast<const float4 *>(T[q] + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
        t[q][0] = x.x; t[q][1 % V] = x.y; t[q][2 % V] = x.z; t[q][3 % V] = x.w;
      } else {
        t[q][0] = on[q] ? __ldg(T[q] + e) : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < V; u++) {
      v[u] = 0.0f;
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (on[q]) v[u] += nb.w[q] * (t[q][u] - wsm[q][i]);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float d = t[q][u] - wsm[q][i] - v[u];
        if (on[q]) spread += nb.w[q] * d * d;
      }
      row[e + u] = __float2bfloat16_rn((v[u] - a.mu[e + u]) / a.sd[e + u]);
    }
  }
  for (int i = threadIdx.x; i < k; i += FT) {
    float v = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (on[q]) v += nb.w[q] * wsm[q][i];
    row[kk + i] = __float2bfloat16_rn((v - a.mu[kk + i]) / a.sd[kk + i]);
  }
  spread = bsum128(spread, red);
  if (threadIdx.x < 16) {
    const int e = kk + k + threadIdx.x;
    row[e] = __float2bfloat16_rn((geometry_feature(a, f, col, nb, spread, threadIdx.x) - a.mu[e]) / a.sd[e]);
  }
  for (int e = kk + k + 16 + threadIdx.x; e < k1; e += FT) row[e] = __float2bfloat16_rn(0.0f);
  if (threadIdx.x == 0) a.flag[f] = nb.missing;
  __syncthreads();
  for (int c8 = threadIdx.x; c8 < k1 >> 3; c8 += FT) put(c8, reinterpret_cast<const uint4 *>(row)[c8]);
}

__global__ void __launch_bounds__(FT) k_lrn_apply(LrnApplyArgs a) {
  __shared__ float red[4];
  __shared__ float wb_s[128], ws_s[4][128];
  const int f = blockIdx.x;
  if (f >= a.nfine) return;
  const int col = a.cols[f], k = a.k, kk = k * k;
  const float *y = a.Yn + (size_t)f * a.ldy;
  float q2 = 0.0f;
  if (a.net)
    for (int e = threadIdx.x; e < a.dout; e += FT) q2 += y[e] * y[e];
  const float score = sqrtf(bsum128(q2, red) / (float)a.dout);
  const bool gated = a.flag[f] || (a.net && !(score <= a.tau));
  if (threadIdx.x == 0) {
    if (a.score) a.score[f] = score;
    if (gated) a.gate_cols[atomicAdd(a.gate_n, 1)] = col;
  }
  if (gated) return;   // CTA-uniform
  const Nb nb = neighbours(col, a.nx, a.ny, a.s, a.src_of_col);
  const int unit = a.col2act[col];
  // w-bar first (T's rows need it)
  for (int i = threadIdx.x; i < k; i += FT) {
    const int e = kk + i;
#pragma unroll
    for (int q = 0; q < 4; q++) ws_s[q][i] = nb.src[q] >= 0 ? a.ws[(size_t)nb.src[q] * k + i] : 0.0f;
    wb_s[i] = interp_at(nb, a.Ts, a.ws, k, i, k) + (a.net ? a.mu_out[e] + a.sd_out[e] * y[e] : 0.0f);
  }
  __syncthreads();
  float *T = a.T + (size_t)unit * kk;
  if ((k & 3) == 0) {
    // four elements of a row at a time (289 us for 38,307 columns at k =
    // 32 element by element, now 141)
    for (int e = 4 * threadIdx.x; e < kk; e += 4 * FT) {
      const int i = e / k;
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (nb.w[q] == 0.0f || nb.src[q] < 0) continue;
        const float wb = ws_s[q][i], w = nb.w[q];
        const float4 t = __ldg(reinterpret_cast<const float4 *>(a.Ts + (size_t)nb.src[q] * kk + e));
        v[0] += w * (t.x - wb);
        v[1] += w * (t.y - wb);
        v[2] += w * (t.z - wb);
        v[3] += w * (t.w - wb);
      }
      if (a.net) {
        const float4 m = __ldg(reinterpret_cast<const float4 *>(a.mu_out + e));
        const float4 d = __ldg(reinterpret_cast<const float4 *>(a.sd_out + e));
        const float4 r = *reinterpret_cast<const float4 *>(y + e);
        v[0] += m.x + d.x * r.x;
        v[1] += m.y + d.y * r.y;
        v[2] += m.z + d.z * r.z;
        v[3] += m.w + d.w * r.w;
      }
      const float wb = wb_s[i];
      *reinterpret_cast<float4 *>(T + e) = make_float4(v[0] + wb, v[1] + wb, v[2] + wb, v[3] + wb);
    }
    if (threadIdx.x == 0) a.nkept[unit] = a.nk_fine[f];
    return;
  }
  for (int e = threadIdx.x; e < kk; e += FT) {
    const int i = e / k, j = e % k;
    const float w = interp_at(nb, a.Ts, a.ws, k, i, j) + (a.net ? a.mu_out[e] + a.sd_out[e] * y[e] : 0.0f);
    T[e] = w + wb_s[i];
  }
  if (threadIdx.x == 0) a.nkept[unit] = a.nk_fine[f];
}

// judge: squared error of the inferred T against the exact one, and the
// squared norm of the exact T - I, summed over judged columns (not gated)
__global__ void __launch_bounds__(FT) k_lrn_judge(int nj, const int *jcols, const int *jsub, const float *Tsub,
                                                  const float *T, const int *col2act, const int *gate_mark, int k,
                                                  float *acc) {
  __shared__ float red[4];
  const int f = blockIdx.x;
  if (f >= nj) return;
  const int col = jcols[f];
  if (gate_mark[col]) return;
  const int unit = col2act[col], kk = k * k;
  const float *te = Tsub + (size_t)jsub[f] * kk, *ti = T + (size_t)unit * kk;
  float e2 = 0.0f, r2 = 0.0f;
  for (int e = threadIdx.x; e < kk; e += FT) {
    const float d = ti[e] - te[e];
    const float r = te[e] - ((e / k) == (e % k) ? 1.0f : 0.0f);
    e2 += d * d;
    r2 += r * r;
  }
  e2 = bsum128(e2, red);
  r2 = bsum128(r2, red);
  if (threadIdx.x == 0) {
    atomicAdd(acc + 0, e2);
    atomicAdd(acc + 1, r2);
    atomicAdd(acc + 2, 1.0f);
  }
}

// A unit that keeps no observation has no transform (the update keeps its
// background), and the transform kernels leave its rows as they were.  The
// learned form interpolates between units, judges and trains on them: here
// such a unit's transform becomes `diag` times the identity, its mean weights
// zero.
__global__ void __launch_bounds__(FT) k_lrn_unobserved(int n, int k, const int *nkept, float diag, float *T,
                                                       float *wbar) {
  const int kk = k * k;
  for (int u = blockIdx.x; u < n; u += gridDim.x) {
    if (nkept[u] > 0) continue;
    for (int e = threadIdx.x; e < kk; e += FT) T[(size_t)u * kk + e] = e % (k + 1) == 0 ? diag : 0.0f;
    for (int e = threadIdx.x; e < k; e += FT) wbar[(size_t)u * k + e] = 0.0f;
  }
}

__global__ void k_lrn_mark(int n, const int *cols, int *mark, int v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) mark[cols[i]] = v;
}

// exact transforms of a column list into the per-unit arrays
__global__ void k_lrn_scatter(int n, const int *cols, const int *col2act, const float *Tsub, const int *nk_sub, int k,
                              float *T, int *nkept) {
  const int kk = k * k;
  const long long total = (long long)n * kk;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(t / kk), q = (int)(t % kk);
    const int unit = col2act[cols[e]];
    T[(size_t)unit * kk + q] = Tsub[(size_t)e * kk + q];
    if (q == 0) nkept[unit] = nk_sub[e];
  }
}

// column means and standard deviations of a [rows][n] matrix (n columns,
// leading dimension ld), FP64 sums; sd floored at 1e-6 (and at 1e-3 of the
// largest sd of the matrix, so that constant inputs stay near zero)
__global__ void k_lrn_colstats(const float *M, long long rows, int n, long long ld, float *mu, float *sd) {
  __shared__ double s1[256], s2[256];
  const int c = blockIdx.x;
  double a = 0.0, b = 0.0;
  for (long long r = threadIdx.x; r < rows; r += blockDim.x) {
    const double v = M[r * ld + c];
    a += v;
    b += v * v;
  }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = b;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      s1[threadIdx.x] += s1[threadIdx.x + o];
      s2[threadIdx.x] += s2[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double m = s1[0] / (double)(rows > 0 ? rows : 1);
    const double var = s2[0] / (double)(rows > 0 ? rows : 1) - m * m;
    mu[c] = (float)m;
    sd[c] = (float)sqrt(var > 0.0 ? var : 0.0);
  }
}

__global__ void k_lrn_sdfloor(float *sd, int n) {
  __shared__ float red[256];
  float m = 0.0f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmaxf(m, sd[i]);
  red[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] = fmaxf(red[threadIdx.x], red[threadIdx.x + o]);
    __syncthreads();
  }
  const float fl = fmaxf(1e-6f, 1e-3f * red[0]);
  for (int i = threadIdx.x; i < n; i += blockDim.x) sd[i] = fmaxf(sd[i], fl);
}

// training batch: rows idx[0..b) of the store, standardised; inputs rounded
// to BF16 (the network's input precision)
__global__ void k_lrn_batch(int b, const int *idx, const float *X, long long ldx, int din, const float *Y,
                            long long ldy, int dout, const float *mu, const float *sd, const float *muo,
                            const float *sdo, float *Xb, float *Yb) {
  const long long total = (long long)b * (din + dout);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(t / (din + dout)), c = (int)(t % (din + dout));
    const long long src = idx[r];
    if (c < din) {
      const float v = (X[src * ldx + c] - mu[c]) / sd[c];
      Xb[(size_t)r * din + c] = __bfloat162float(__float2bfloat16_rn(v));
    } else {
      const int o = c - din;
      Yb[(size_t)r * dout + o] = (Y[src * ldy + o] - muo[o]) / sdo[o];
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// launchers

cudaError_t lrn_cellstats(cudaStream_t st, int ncell, const ObsSorted &obs, float4 *c0, float4 *c1, int *launches) {
  if (ncell <= 0) return cudaSuccess;
  k_lrn_cellstats<<<(ncell + 255) / 256, 256, 0, st>>>(ncell, obs, c0, c1);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_obsfeat(cudaStream_t st, int nfine, const int *cols, const ColPar *cp, const DevLoc &loc,
                        const int *cell_start, const float4 *c0, const float4 *c1, const IndexGeom *geom,
                        float *feat, int *nkept, int *launches) {
  if (nfine <= 0) return cudaSuccess;
  const int per = FT / 32;
  k_lrn_obsfeat<<<(nfine + per - 1) / per, FT, 0, st>>>(nfine, cols, cp, loc, cell_start, c0, c1, geom, feat, nkept);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_interp(cudaStream_t st, const LrnInterpArgs &a, int *launches) {
  if (a.nfine <= 0) return cudaSuccess;
  k_lrn_interp<<<a.nfine, FT, 0, st>>>(a);
  (*launches)++;
  return cudaGetLastError();
}

// rows padded to whole blocks of 128
cudaError_t lrn_input(cudaStream_t st, const LrnInterpArgs &a, int k1, unsigned char *Xt, int *launches) {
  if (a.nfine <= 0) return cudaSuccess;
  if (a.k > 128 || !a.mu || a.Yt) return cudaErrorInvalidValue;
  const int rows = (a.nfine + 127) / 128 * 128;
  if (a.k % 4 == 0) k_lrn_input<true><<<rows, FT, 2 * (size_t)k1, st>>>(a, k1, Xt);
  else k_lrn_input<false><<<rows, FT, 2 * (size_t)k1, st>>>(a, k1, Xt);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_unobserved(cudaStream_t st, int n, int k, const int *nkept, float diag, float *T, float *wbar,
                           int *launches) {
  if (n <= 0) return cudaSuccess;
  k_lrn_unobserved<<<std::min(n, 152 * 16), FT, 0, st>>>(n, k, nkept, diag, T, wbar);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_apply(cudaStream_t st, const LrnApplyArgs &a, int *launches) {
  if (a.nfine <= 0) return cudaSuccess;
  if (a.k > 128) return cudaErrorInvalidValue;
  k_lrn_apply<<<a.nfine, FT, 0, st>>>(a);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_judge(cudaStream_t st, int nj, const int *jcols, const int *jsub, const float *Tsub, const float *T,
                      const int *col2act, const int *gate_mark, int k, float *acc, int *launches) {
  if (nj <= 0) return cudaSuccess;
  k_lrn_judge<<<nj, FT, 0, st>>>(nj, jcols, jsub, Tsub, T, col2act, gate_mark, k, acc);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_mark(cudaStream_t st, int n, const int *cols, int *mark, int v) {
  if (n <= 0) return cudaSuccess;
  k_lrn_mark<<<(n + 255) / 256, 256, 0, st>>>(n, cols, mark, v);
  return cudaGetLastError();
}

cudaError_t lrn_scatter(cudaStream_t st, int n, const int *cols, const int *col2act, const float *Tsub,
                        const int *nk_sub, int k, float *T, int *nkept, int *launches) {
  if (n <= 0) return cudaSuccess;
  const long long total = (long long)n * k * k;
  const int grid = (int)std::min<long long>(4096, (total + 255) / 256);
  k_lrn_scatter<<<grid, 256, 0, st>>>(n, cols, col2act, Tsub, nk_sub, k, T, nkept);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t lrn_colstats(cudaStream_t st, const float *M, long long rows, int n, long long ld, float *mu, float *sd) {
  if (n <= 0) return cudaSuccess;
  k_lrn_colstats<<<n, 256, 0, st>>>(M, rows, n, ld, mu, sd);
  k_lrn_sdfloor<<<1, 256, 0, st>>>(sd, n);
  return cudaGetLastError();
}

cudaError_t lrn_batch(cudaStream_t st, int b, const int *idx, const float *X, long long ldx, int din, const float *Y,
                      long long ldy, int dout, const float *mu, const float *sd, const float *muo, const float *sdo,
                      float *Xb, float *Yb) {
  if (b <= 0) return cudaSuccess;
  const long long total = (long long)b * (din + dout);
  const int grid = (int)std::min<long long>(4096, (total + 255) / 256);
  k_lrn_batch<<<grid, 256, 0, st>>>(b, idx, X, ldx, din, Y, ldy, dout, mu, sd, muo, sdo, Xb, Yb);
  return cudaGetLastError();
}

}  // namespace lgpu
