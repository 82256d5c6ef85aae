// lgpu_index.cu -- observation preparation and the spatial index that
// replaces the geoKdTree radius search (src/letkf_obs.F90:492-503 builds
// the tree, :560-573 queries it), plus the per-column localisation
// parameters (localizer%maxhz, search radius, mixed-layer level).
//
// Index: observations bucketed into latitude-band x longitude cells, cells
// band-major; a stable order inside each cell (ascending observation index)
// makes every later reduction deterministic.  The sorted copy holds what the
// Gram kernel streams: unit vector + error (16 B), departure/time/depth/
// surface flag (16 B) and the hx perturbation row padded to KP floats.
//
// The stage is a chain of small kernels, bound by their latencies: the
// observations' and the columns' preparation share one launch (both mostly
// FP64, at 1/64 of the FP32 rate: blocks of two warps spread it over the SMs),
// the scan of the cell counts and the tiles' caps another, an observation's
// slot in its cell comes from the counting atomic itself, and the order inside
// a cell is found by the warp that copies the observation's row.  As eight
// kernels and six memsets, with four barriers per 1,024 cells in the scan, it
// took 86 us at 700 observations and 648 columns, now 39.
#include "lgpu_internal.cuh"

namespace lgpu {

namespace {

constexpr int PT = 64;   // threads of the preparation blocks

__device__ __forceinline__ void obs_prep(const ObsPrepArgs &o, int i) {
  float la = o.lat[i], lo = o.lon[i];
  float3 u = unitvec_exact(la, lo);
  // dep = val - hx_mean (src/letkf_solver.F90:228)
  float dep = __fsub_rn(o.val[i], o.hx_mean[i]);
  // surface classification (src/subclass.letkf_localizer/letkf_loc_ocean.F90:467-479):
  // TRUE unless a non-empty id list misses this observation's id
  float surf = 1.0f;
  if (o.n_sat_obs > 0) {
    bool f = false;
    for (int j = 0; j < o.n_sat_obs; j++) f |= (o.obsid[i] == o.sat_obs[j]);
    if (!f) surf = 0.0f;
  }
  if (o.n_sat_plats > 0) {
    bool f = false;
    for (int j = 0; j < o.n_sat_plats; j++) f |= (o.platid[i] == o.sat_plats[j]);
    if (!f) surf = 0.0f;
  }
  int b = band_of(la);
  int nl = o.geom->nlon[b];
  float ln = norm_lon(lo);
  int c = (int)floorf(ln * (float)nl / 360.0f);
  c = c < 0 ? 0 : (c >= nl ? nl - 1 : c);
  int id = o.geom->off[b] + c;
  o.cell[i] = id;
  o.slot[i] = atomicAdd(&o.count[id], 1);
  o.A[i] = make_float4(u.x, u.y, u.z, o.err[i]);
  o.B[i] = make_float4(dep, o.time[i], o.zdim[i], surf);
}

// Per-column localisation parameters: localizer%maxhz (loc_novrt :155-161,
// loc_ocean :435-443 = MAX(prof, sat)), max_search_dist = maxhz*stdev2max
// (src/letkf_solver.F90:210-212), the index window of the search circle, and
// for loc_ocean with bkg_t vertical localisation calc_mldlvl_bkgt
// (letkf_loc_ocean.F90:408-427) on the background mean.
// The column's diagnostics start at zero.
__device__ __forceinline__ void col_prep(const ColPrepArgs &a, int c) {
  const DevLoc &loc = a.loc;
  float la = a.lat[c], lo = a.lon[c];
  float3 u = unitvec_exact(la, lo);
  ColPar p;
  p.ux = u.x; p.uy = u.y; p.uz = u.z;
  float L1 = interp_get(loc.hz, la), L2 = L1, maxhz = L1;
  if (loc.cls == LOC_OCEAN) {
    L2 = interp_get(loc.hz_sat, la);
    maxhz = L1 > L2 ? L1 : L2;
  }
  p.L1 = L1; p.L2 = L2;
  p.ic1 = inv_c_of(L1); p.ic2 = inv_c_of(L2);
  p.rmax = __fmul_rn(maxhz, kStdev2Max);
  a.diag_maxhz[c] = a.mask[c] ? 0.0f : maxhz;
  a.diag_obscount[c] = 0.0f;
  for (int g = 0; g < loc.groups; g++) {
    a.diag_lg_obscount[(size_t)g * a.ncol + c] = 0.0f;
    a.diag_lg_obsloc[(size_t)g * a.ncol + c] = 0.0f;
  }
  // conservative index window of the search circle
  float alpha = p.rmax / 6371000.0f;
  float adeg = alpha * 57.29577951308232f * 1.0001f + 0.05f;
  bool full = (la + adeg >= 90.0f) || (la - adeg <= -90.0f) || alpha >= 1.5f;
  float dl = 180.0f;
  if (!full) {
    float s = sinf(alpha) / cosf(la * 0.017453292519943295f);
    dl = s >= 1.0f ? 180.0f : asinf(s) * 57.29577951308232f * 1.0001f + 0.05f;
  }
  p.lonn = norm_lon(lo);
  p.dlon = dl;
  p.b0 = band_of(la - adeg);
  p.b1 = band_of(la + adeg);
  int mld = 0;
  if (loc.cls == LOC_OCEAN && loc.vtloc_surf == 1) {
    const float *m = a.mean_b + (size_t)c * a.ns;
    float t0 = m[loc.bkg_t_idx];
    mld = loc.bkg_t_len;
    for (int i = 1; i <= loc.bkg_t_len - 1; i++) {
      float t1 = m[loc.bkg_t_idx + i];
      if (fabsf(__fsub_rn(t0, t1)) > loc.bkg_t_delta) { mld = i; break; }
    }
  }
  p.mld = mld;
  p.pad = 0;
  a.cp[c] = p;
}

// blocks [0, obs_blocks): observations; the others: columns (the first of them
// clears the status words)
__global__ void __launch_bounds__(PT) k_prep(ObsPrepArgs o, int obs_blocks, ColPrepArgs a) {
  if ((int)blockIdx.x < obs_blocks) {
    const int i = blockIdx.x * PT + threadIdx.x;
    if (i < o.nobs) obs_prep(o, i);
    return;
  }
  const int c = (blockIdx.x - obs_blocks) * PT + threadIdx.x;
  if (c < 4) a.status[c] = 0;
  if (c < a.ncol) col_prep(a, c);
}

constexpr int ST = 1024;   // threads of the scan
constexpr int SV = 8;      // 16-byte loads of counts in flight per thread

// exclusive scan of the cell counts, one block: SV x 4 counts a thread and pass
// (41,000 cells: two passes of three barriers)
__device__ void scan_cells(int n, const int *count, int *start) {
  __shared__ int wsum[SV][32];
  __shared__ int csum[SV];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = 0;
  for (int base = 0; base < n; base += SV * ST * 4) {
    int4 v[SV];
    int incl[SV];
#pragma unroll
    for (int q = 0; q < SV; q++) {
      const int i = base + (q * ST + (int)threadIdx.x) * 4;
      if (i + 3 < n) {
        v[q] = *reinterpret_cast<const int4 *>(count + i);
      } else {
        v[q].x = i < n ? count[i] : 0;
        v[q].y = i + 1 < n ? count[i + 1] : 0;
        v[q].z = i + 2 < n ? count[i + 2] : 0;
        v[q].w = 0;
      }
      incl[q] = v[q].x + v[q].y + v[q].z + v[q].w;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < SV; q++) {
        const int y = __shfl_up_sync(0xffffffffu, incl[q], o);
        if (lane >= o) incl[q] += y;
      }
    if (lane == 31)
#pragma unroll
      for (int q = 0; q < SV; q++) wsum[q][w] = incl[q];
    __syncthreads();
    if (w < SV) {
      const int own = wsum[w][lane];
      int x = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      wsum[w][lane] = x - own;
      if (lane == 31) csum[w] = x;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < SV; q++) {
      const int i = base + (q * ST + (int)threadIdx.x) * 4;
      int4 e;
      e.x = carry + wsum[q][w] + incl[q] - (v[q].x + v[q].y + v[q].z + v[q].w);
      e.y = e.x + v[q].x;
      e.z = e.y + v[q].y;
      e.w = e.z + v[q].z;
      if (i + 3 < n) {
        *reinterpret_cast<int4 *>(start + i) = e;
      } else {
        if (i < n) start[i] = e.x;
        if (i + 1 < n) start[i + 1] = e.y;
        if (i + 2 < n) start[i + 2] = e.z;
      }
      carry += csum[q];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) start[n] = carry;
}

// Tile caps: centre = normalised mean of the tile's unit vectors, angular
// radius = max over columns of (angle to centre + search radius / R), then
// the same conservative band / longitude window as a single column.  One
// thread per column of the tile; the FP64 functions of the window run on
// different warps.
constexpr int TPT = 128;
__device__ void tile_cap(const int *cols, const ColPar *cp, TilePar *out) {
  __shared__ double red[TPT / 32][3], rang[TPT / 32], part[4];
  __shared__ float rhm[TPT / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = cols[threadIdx.x];
  float ux = 0.0f, uy = 0.0f, uz = 0.0f, rmax = 0.0f;
  if (col >= 0) {
    ux = cp[col].ux; uy = cp[col].uy; uz = cp[col].uz; rmax = cp[col].rmax;
  }
  double sx = ux, sy = uy, sz = uz;
  for (int o = 16; o > 0; o >>= 1) {
    sx += __shfl_xor_sync(0xffffffffu, sx, o);
    sy += __shfl_xor_sync(0xffffffffu, sy, o);
    sz += __shfl_xor_sync(0xffffffffu, sz, o);
  }
  if (lane == 0) { red[w][0] = sx; red[w][1] = sy; red[w][2] = sz; }
  __syncthreads();
  sx = sy = sz = 0.0;
  for (int q = 0; q < TPT / 32; q++) { sx += red[q][0]; sy += red[q][1]; sz += red[q][2]; }
  const double nrm = sqrt(sx * sx + sy * sy + sz * sz);
  const double cx = nrm > 0 ? sx / nrm : 1.0, cy = nrm > 0 ? sy / nrm : 0.0, cz = nrm > 0 ? sz / nrm : 0.0;
  double ang = 0.0;
  // largest half-chord sqrt(c2max)/2 of a candidate pair (the weight producers' c2max)
  float hm = 0.0f;
  if (col >= 0) {
    const double dot = fmin(1.0, fmax(-1.0, cx * ux + cy * uy + cz * uz));
    ang = acos(dot) + (double)rmax / 6371000.0;
    const float hq = fminf(rmax / 12742000.0f, 1.5707963f);
    const float sh = sinf(hq);
    hm = sqrtf(4.0f * sh * sh * 1.0001f + 1e-12f) * 0.5f;
  }
  for (int o = 16; o > 0; o >>= 1) {
    ang = fmax(ang, __shfl_xor_sync(0xffffffffu, ang, o));
    hm = fmaxf(hm, __shfl_xor_sync(0xffffffffu, hm, o));
  }
  if (lane == 0) { rang[w] = ang; rhm[w] = hm; }
  __syncthreads();
  for (int q = 0; q < TPT / 32; q++) { ang = fmax(ang, rang[q]); hm = fmaxf(hm, rhm[q]); }
  const double alpha = ang * 1.0001 + 1e-6;
  if (lane == 0) {
    if (w == 0) {
      const double lat = asin(fmax(-1.0, fmin(1.0, cz))) * 57.29577951308232;
      part[0] = lat;
      part[3] = cos(lat * 0.017453292519943295);
    } else if (w == 1) {
      double lon = atan2(cy, cx) * 57.29577951308232;
      if (lon < 0) lon += 360.0;
      if (lon >= 360.0) lon -= 360.0;
      part[1] = lon;
    } else if (w == 2) {
      part[2] = sin(alpha);
    } else {
      const double ch = 2.0 * sin(0.5 * fmin(alpha, 3.14159265358979));
      out->c2cap = (float)(ch * ch * 1.00001 + 1e-9);
      out->hmax = hm * 1.0001f;
      out->cx = (float)cx;
      out->cy = (float)cy;
      out->cz = (float)cz;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const double lat = part[0];
    const double adeg = alpha * 57.29577951308232 + 0.05;
    const bool full = (lat + adeg >= 90.0) || (lat - adeg <= -90.0) || alpha >= 1.5;
    double dl = 180.0;
    if (!full) {
      const double sr = part[2] / part[3];
      dl = sr >= 1.0 ? 180.0 : asin(sr) * 57.29577951308232 * 1.0001 + 0.05;
    }
    out->lonn = (float)part[1];
    out->dlon = (float)dl;
    out->b0 = band_of((float)(lat - adeg));
    out->b1 = band_of((float)(lat + adeg));
  }
}

__global__ void __launch_bounds__(TPT) k_tile_prep(const int *tile_cols, const ColPar *cp, TilePar *tp) {
  tile_cap(tile_cols + (size_t)blockIdx.x * TPT, cp, tp + blockIdx.x);
}

// block 0: the scan; block 1 + t: the cap of tile t (on its first TPT threads)
__global__ void __launch_bounds__(ST) k_scan_tiles(int n, const int *count, int *start, const int *tile_cols,
                                                   const ColPar *cp, TilePar *tp) {
  if (blockIdx.x == 0) {
    scan_cells(n, count, start);
  } else if (threadIdx.x < TPT) {
    const int t = blockIdx.x - 1;
    tile_cap(tile_cols + (size_t)t * TPT, cp, tp + t);
  }
}

__global__ void k_scatter(int nobs, const int *cell, const int *start, const int *slot, int *pos_tmp) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nobs) return;
  pos_tmp[start[cell[i]] + slot[i]] = i;
}

// A warp per entry of the cell-grouped list: its place is the cell's start plus
// the count of the cell's smaller observation ids (ids are unique), where the
// warp copies its records and its hx row.
constexpr int GW = 8;   // warps per block
__global__ void __launch_bounds__(32 * GW) k_place(int nobs, int k, int kp, const int *cell, const int *start,
                                                   const int *pos_tmp, const float4 *Atmp, const float4 *Btmp,
                                                   const float *hx, ObsSorted o) {
  const int p = blockIdx.x * GW + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p >= nobs) return;
  const int i = pos_tmp[p], c = cell[i], b = start[c], n = start[c + 1] - b;
  int r = 0;
  for (int j = lane; j < n; j += 32) r += pos_tmp[b + j] < i;
  r = __reduce_add_sync(0xffffffffu, r);
  const size_t q = (size_t)(b + r);
  const float *src = hx + (size_t)i * k;
  unsigned ymax = 0;   // bits of the largest |y| (NaN above all)
  for (int m = lane; m < kp; m += 32) {
    const float y = m < k ? src[m] : 0.0f;
    ymax = max(ymax, __float_as_uint(fabsf(y)));
    o.hx[q * kp + m] = y;
  }
  ymax = __reduce_max_sync(0xffffffffu, ymax);
  const float4 A = Atmp[i], B = Btmp[i];
  if (lane == 0) o.A[q] = A;
  if (lane == 1) o.B[q] = B;
  if (lane == 2) o.idx[q] = i;
  // the observation's largest features over its error: of all, and y_i y_j
  if (lane == 3) {
    const float y = __uint_as_float(ymax), s = y / A.w;
    o.mag[q] = make_float2(s * __uint_as_float(max(ymax, __float_as_uint(fabsf(B.x)))), s * y);
  }
}

}  // namespace

cudaError_t launch_prep(cudaStream_t st, const ObsPrepArgs *o, int ncell, const ColPrepArgs *c, int *launches) {
  cudaError_t e;
  ObsPrepArgs oa{};
  ColPrepArgs ca{};
  int nb = 0, cb = 0;
  if (o) {
    oa = *o;
    if ((e = cudaMemsetAsync(oa.count, 0, sizeof(int) * ncell, st)) != cudaSuccess) return e;
    nb = (oa.nobs + PT - 1) / PT;
  }
  if (c) {
    ca = *c;
    cb = (ca.ncol + PT - 1) / PT;
  }
  if (nb + cb == 0) return cudaSuccess;
  k_prep<<<nb + cb, PT, 0, st>>>(oa, nb, ca);
  (*launches)++;
  return cudaGetLastError();
}

cudaError_t launch_obs_index(cudaStream_t st, const ObsPrepArgs &a, int k, int kp, const float *hx, int ncell,
                             int *pos_tmp, ObsSorted out, int ntiles, const int *tile_cols, const ColPar *cp,
                             TilePar *tp, int *launches) {
  k_scan_tiles<<<1 + ntiles, ST, 0, st>>>(ncell, a.count, out.cell_start, tile_cols, cp, tp);
  (*launches)++;
  const int nobs = a.nobs;
  if (nobs > 0) {
    k_scatter<<<(nobs + 255) / 256, 256, 0, st>>>(nobs, a.cell, out.cell_start, a.slot, pos_tmp);
    k_place<<<(nobs + GW - 1) / GW, 32 * GW, 0, st>>>(nobs, k, kp, a.cell, out.cell_start, pos_tmp, a.A, a.B, hx, out);
    (*launches) += 2;
  }
  return cudaGetLastError();
}

cudaError_t launch_scan(cudaStream_t st, int n, const int *count, int *start) {
  k_scan_tiles<<<1, ST, 0, st>>>(n, count, start, nullptr, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_tile_prep(cudaStream_t st, int ntiles, const int *tile_cols, const ColPar *cp, TilePar *tp,
                             int *launches) {
  if (ntiles <= 0) return cudaSuccess;
  k_tile_prep<<<ntiles, TPT, 0, st>>>(tile_cols, cp, tp);
  (*launches)++;
  return cudaGetLastError();
}

}  // namespace lgpu
