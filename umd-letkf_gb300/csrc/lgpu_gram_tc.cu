// lgpu_gram_tc.cu -- batched Gram on the tensor cores: one CTA per
// (tile of 128 neighbouring columns, localisation group, feature pass).
//
// Same result as k_gram (src/letkf_solver.F90:210-268 and the Gram / RHS half
// of src/letkf_core.F90:92-125), reorganised so that neighbouring columns
// share their observations.  For a tile the Gram entries of every column form
// one GEMM over the tile's candidate observations o:
//
//   G[c, f] = sum_o W[c, o] * P[o, f],   W[c, o] = rloc_c(o) / err_o
//                                        P[o, f] = y_i(o) * y_j(o)   f = (i <= j)
//                                                = y_i(o) * dep(o)   f = (i, rhs)
//
// M = 128 columns, N = the k(k+3)/2 packed features (split into passes of at
// most 480 so the accumulator fits TMEM), K = candidate observations in
// chunks of 16.
//
// Candidate streams.  Before the GEMM, four small kernels turn each tile's
// search window (latitude bands x longitude range of its cap) into a record
// stream: every observation inside the tile's cap, in window order, packed
// per chunk of 16 as ux[16] uy[16] uz[16] 1/err[16] dep[16] time[16] zdim[16]
// surf[16] and member-major y: (k+1 rounded to 4) rows x 16 -- one contiguous
// block per chunk, read once per (group, pass) CTA with one bulk async copy.
//
// GEMM CTA roles (16 + ceil(N / 32) + 1 warps):
//   warps 0-15  weights; thread t owns column t % 128 for observations
//               [4 (t / 128), +4) of each chunk: the distance (fast float path
//               without branches; the exact metric and the per-column
//               localizer where the fast value lies near the search radius or
//               the keep threshold: bit-identical keep decisions to the
//               per-column path), W = rho;
//   then        features, a thread each: P = y_i * y_j / err, y_i * dep / err.
//               Both split their operand into FP16 hi + lo parts (TF32 where
//               the observations' magnitudes need its exponents, then with
//               1 / err on the weights), stored in the no-swizzle K-major
//               core-matrix layout of an operand stage;
//   last warp   one thread keeps the record ring filled (cp.async.bulk, one
//               per round of chunks, mbarrier transaction counts; a slot is
//               refilled once every producer has finished the round in it),
//               issues tcgen05.mma for hi*hi + hi*lo + lo*hi (FP32
//               accumulation in TMEM, relative error ~2^-22 per product) and
//               frees the stages with tcgen05.commit; chunks in which no
//               column keeps an observation issue no MMA.
// What bounds it (720 x 360 columns, k = 40, 2.07 M chunks over both passes,
// 17 ms): with TF32 operands, 16 warps doing weights and features in turn, the
// shared-memory traffic of operand stores and MMA reads (230 KB a chunk), the
// producers' instructions and the MMAs (1,300 cycles) took about the same time
// each, and removing any one alone gained 10 to 20%.  FP16 parts halve the
// traffic and the MMAs, own warps let features and weights overlap: Gram 21.8
// -> 18.7 ms, then two chunks per barrier round 17.9, the segment sum's 1.65
// included; the producers bound it now (without weights 14.9, without features
// 16.5, without MMAs 18.3).  Sharing the weights between the CTAs of two passes
// through distributed shared memory was slower in three forms (23.3 ms and
// more): its cluster-scope fences cost more than the weights.
// The epilogue reads TMEM lane c = column c and writes the packed Gram block
// of each unit.  Every wait is bounded; a wait that runs out sets status bit
// 16, the MMA thread waits (bounded) for its copies in flight and TMEM is
// freed.
//
// Long tile streams are split into accumulation segments, each its
// own CTA, summed in order by k_gram_segsum.  The producers come in two forms
// with bit-identical output (with and without a warp-level cull of records
// out of every column's reach); the first analysis of a configuration times
// both and keeps the faster.
#include "lgpu_internal.cuh"
#include "lgpu_tc.cuh"

namespace lgpu {

namespace {

constexpr int TM = 128;        // columns per tile = MMA M = TMEM lanes
constexpr int KC = 16;         // observations per chunk (one FP16 or two TF32 MMA steps)
// Features per pass: 15 feature warps, 1,024 threads.  At 432 (14 warps) k = 28,
// 29, 52, 60 or 100 took a pass more, with its weights: Gram of 240 x 120
// clustered columns, k = 29 0.244 ms, now 0.189; k = 60 0.756, now 0.684.
constexpr int NPMAX = 480;
constexpr int NW = 16;         // weight warps; then the feature warps (one per 32 features), then the MMA warp
__host__ __device__ constexpr int feature_warps(int np) { return (np + 31) / 32; }
__host__ __device__ constexpr int gram_threads(int np) { return 32 * (NW + feature_warps(np) + 1); }
constexpr int NSMAX = 4, NRMAX = 6;
constexpr uint32_t CMB = 128;                 // bytes per core matrix (8 rows x 16 B)
// bytes of an operand's element, of an 8-row group (all K of the chunk), of a W operand copy
__host__ __device__ constexpr uint32_t el_bytes(bool f16) { return f16 ? 2 : 4; }
__host__ __device__ constexpr uint32_t sbo_of(bool f16) { return KC * el_bytes(f16) / 16 * CMB; }
__host__ __device__ constexpr uint32_t wb_of(bool f16) { return (TM / 8) * sbo_of(f16); }
__host__ __device__ constexpr int stages_of(bool f16) { return f16 ? 4 : 2; }
// chunks per round of the barriers.  A round's waits, fence and arrival cost
// each producer warp a good part of a chunk's time: with FP16 operands two
// chunks share them (Gram of 720 x 360 columns, k = 40: 18.7 ms, now 17.9; the
// TF32 stages have room for two chunks in all).
__host__ __device__ constexpr int round_of(bool f16) { return f16 ? 2 : 1; }
constexpr size_t kSmemBudget = 227 * 1024 - 4096;   // dynamic shared memory (static part below 4 KB)
constexpr int WT = 256;        // threads of the stream kernels
constexpr int YS = 20;         // floats per member row of a chunk record (16 observations + 4: conflict-free rows)
template <bool F16>
__device__ __forceinline__ uint32_t kmaj(int row, int kk) {
  constexpr int PC = F16 ? 8 : 4;   // elements of a core matrix row
  return (uint32_t)(row >> 3) * sbo_of(F16) + (uint32_t)(kk / PC) * CMB + (uint32_t)(row & 7) * 16u +
         (uint32_t)(kk % PC) * el_bytes(F16);
}

// FP16 operands.  W = 2^12 rho lies in (0.4, 4096] for every weight above the
// keep threshold, and the features y_i y_j / err are scaled by a power of two
// per tile that puts the largest of its candidates' into [2^14, 2^15): hi = f16
// (11 bits) and lo = f16 (x - hi) leave at most 2^-22 |x|, or 2^-25 where lo's
// spacing is FP16's smallest (x below 2^-3).  The largest y_i y_j / err of every
// candidate has to be at least 2^-3, 17 powers of two below the tile's top, so
// an observation's operands are off by at most 2^-22 of its own largest y_i y_j
// / err in the features y_i y_j, and of its own largest feature in y_i dep
// (TF32's hi + lo: 2^-21 of each feature).  Where a tile's candidates differ by
// more, in their perturbations or in departures far beyond these, or the
// largest is not finite or beyond 2^+-60 (the factors of a feature stay normal
// FP32 numbers), the run takes the TF32 operands, whose exponents are FP32's.
constexpr float kWScale = 4096.0f;
constexpr int kPTop = 14, kPRange = 17, kPExp = 60;
__host__ __device__ inline int f32_exp(uint32_t bits) { return (int)(bits >> 23) - 127; }
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

__device__ __forceinline__ bool in_cap(const TilePar &t, float4 A) {
  const float dx = __fsub_rn(t.cx, A.x), dy = __fsub_rn(t.cy, A.y), dz = __fsub_rn(t.cz, A.z);
  return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)) <= t.c2cap;
}

// ---------------------------------------------------------------------------
// Search window of a tile as runs of the cell-sorted observation table
// (per latitude band at most two runs, the second for a window across 0/360),
// concatenated: candidate j of the window lives at seg_start[s] + j -
// seg_pref[s] for the last s with seg_pref[s] <= j.  Block of WT threads.
struct Window {
  int seg_start[2 * kNB];
  int seg_pref[2 * kNB + 1];
  int wsc[WT / 32];
  int nseg, total;
};

__device__ void build_window(Window &W, const TilePar &tp, const IndexGeom *geom, const int *cell_start) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nb = tp.b1 - tp.b0 + 1;
  int l0 = 0, l1 = 0;
  if (tid < nb) {
    const int b = tp.b0 + tid;
    const int nl = geom->nlon[b], off = geom->off[b];
    int s0 = 0, s1 = 0;
    bool whole = tp.dlon >= 180.0f;
    int clo = 0, chi = nl - 1;
    if (!whole) {
      clo = (int)floorf((tp.lonn - tp.dlon) * (float)nl / 360.0f);
      chi = (int)floorf((tp.lonn + tp.dlon) * (float)nl / 360.0f);
      if (chi - clo + 1 >= nl) whole = true;
    }
    if (whole) {
      s0 = cell_start[off];
      l0 = cell_start[off + nl] - s0;
    } else if (clo < 0) {
      s0 = cell_start[off + clo + nl];
      l0 = cell_start[off + nl] - s0;
      s1 = cell_start[off];
      l1 = cell_start[off + chi + 1] - s1;
    } else if (chi >= nl) {
      s0 = cell_start[off + clo];
      l0 = cell_start[off + nl] - s0;
      s1 = cell_start[off];
      l1 = cell_start[off + (chi - nl) + 1] - s1;
    } else {
      s0 = cell_start[off + clo];
      l0 = cell_start[off + chi + 1] - s0;
    }
    W.seg_start[2 * tid] = s0;
    W.seg_start[2 * tid + 1] = s1;
  }
  const int x = l0 + l1;
  int incl = x;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) W.wsc[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int sv = lane < WT / 32 ? W.wsc[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sv, o);
      if (lane >= o) sv += y;
    }
    if (lane < WT / 32) W.wsc[lane] = sv;
  }
  __syncthreads();
  const int base = (wid > 0 ? W.wsc[wid - 1] : 0) + incl - x;
  if (tid < nb) {
    W.seg_pref[2 * tid] = base;
    W.seg_pref[2 * tid + 1] = base + l0;
  }
  if (tid == 0) {
    W.nseg = 2 * nb;
    W.total = W.wsc[WT / 32 - 1];
    W.seg_pref[2 * nb] = W.total;
  }
  __syncthreads();
}

__device__ __forceinline__ int window_pos(const Window &W, int j) {
  int lo = 0, hi = W.nseg - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (W.seg_pref[mid] <= j) lo = mid; else hi = mid - 1;
  }
  return W.seg_start[lo] + (j - W.seg_pref[lo]);
}

// the window's candidates of warp w of WT / 32, whole groups of 32
__device__ __forceinline__ void warp_range(const Window &W, int w, int &j0, int &j1) {
  const int per = ((W.total + WT - 1) / WT) * 32;
  j0 = min(W.total, w * per);
  j1 = min(W.total, j0 + per);
}

// candidates per tile: observations of the window inside the tile's cap, per
// warp range (tile_wn) and in all
__global__ void __launch_bounds__(WT) k_tile_count(int ntiles, const TilePar *tps, const IndexGeom *geom,
                                                   const float4 *obsA, const float2 *mag, const int *cell_start,
                                                   int *tile_n, int *tile_wn, uint32_t *tile_mag) {
  __shared__ Window W;
  __shared__ int red[WT / 32];
  __shared__ uint32_t smax[WT / 32], smin[WT / 32];
  const int tile = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const TilePar tp = tps[tile];
  build_window(W, tp, geom, cell_start);
  int cnt = 0, j0, j1;
  warp_range(W, wid, j0, j1);
  uint32_t mx = 0, mn = 0x7f800000u;   // largest feature, smallest positive y_i y_j of an observation's largest (bits)
#pragma unroll 4
  for (int j = j0 + lane; j < j1; j += 32) {
    const int p = window_pos(W, j);
    const bool in = in_cap(tp, __ldg(obsA + p));
    const float2 m = in ? __ldg(mag + p) : make_float2(0.0f, 0.0f);
    cnt += in;
    mx = max(mx, __float_as_uint(m.x));
    mn = m.y != 0.0f ? min(mn, __float_as_uint(m.y)) : mn;
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  mx = __reduce_max_sync(0xffffffffu, mx);
  mn = __reduce_min_sync(0xffffffffu, mn);
  if (lane == 0) {
    red[wid] = cnt;
    smax[wid] = mx;
    smin[wid] = mn;
    tile_wn[(size_t)tile * (WT / 32) + wid] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < WT / 32; w++) {
      t += red[w];
      mx = max(mx, smax[w]);
      mn = min(mn, smin[w]);
    }
    tile_n[tile] = t;
    tile_mag[2 * tile] = mx;
    tile_mag[2 * tile + 1] = mn;
  }
}

// chunk offsets of the tile streams: tile_off[t] = sum over earlier tiles of
// ceil(n / 16); tile_off[ntiles] = total chunks.  One block.
// tile_off[ntiles + 1]: some tile's magnitudes are out of the FP16 operands' range.
__global__ void k_tile_scan(int ntiles, const int *tile_n, const uint32_t *tile_mag, int *tile_off) {
  __shared__ int wsum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int wide = 0;
  for (int base = 0; base < ntiles; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < ntiles ? (tile_n[i] + KC - 1) / KC : 0;
    const uint32_t mx = i < ntiles ? tile_mag[2 * i] : 0u, mn = i < ntiles ? tile_mag[2 * i + 1] : 0u;
    if (mx != 0u) wide |= abs(f32_exp(mx)) > kPExp || f32_exp(mx) - f32_exp(mn) > kPRange;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = lane < nw ? wsum[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      if (lane < nw) wsum[lane] = s;
    }
    __syncthreads();
    const int excl = carry + (w > 0 ? wsum[w - 1] : 0) + x - v;
    if (i < ntiles) tile_off[i] = excl;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
  wide = __syncthreads_or(wide);
  if (threadIdx.x == 0) {
    tile_off[ntiles] = carry;
    tile_off[ntiles + 1] = wide;
  }
}

// The tile streams, in two steps: the positions of the cap's members in window
// order (order preserving; a warp writes its range of the window behind the
// ranges before it), then the records.  In one kernel with a block per tile,
// whose threads each copied an observation's whole row between the block's
// barriers, the step had a few hundred blocks of long serial work (clustered
// 240 x 120, k = 64: counts and streams 281 us, now 108).
__global__ void __launch_bounds__(WT) k_tile_list(const TilePar *tps, const IndexGeom *geom, const float4 *obsA,
                                                  const int *cell_start, const int *tile_n, const int *tile_wn,
                                                  const int *tile_off, int *list, int *status) {
  __shared__ Window W;
  const int tile = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const TilePar tp = tps[tile];
  build_window(W, tp, geom, cell_start);
  const int c0 = tile_off[tile], cap = (tile_off[tile + 1] - c0) * KC, n = tile_n[tile];
  int *out = list + (size_t)c0 * KC;
  int q = 0;
  for (int w = 0; w < wid; w++) q += tile_wn[(size_t)tile * (WT / 32) + w];
  const int qend = q + tile_wn[(size_t)tile * (WT / 32) + wid];
  int j0, j1;
  warp_range(W, wid, j0, j1);
  for (int jb = j0; jb < j1; jb += 128) {
    int p[4];
    bool ok[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = jb + 32 * u + lane;
      p[u] = j < j1 ? window_pos(W, j) : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) ok[u] = p[u] >= 0 && in_cap(tp, __ldg(obsA + p[u]));
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned m = __ballot_sync(0xffffffffu, ok[u]);
      const int at = q + __popc(m & ((1u << lane) - 1u));
      if (ok[u] && at < cap) out[at] = p[u];
      q += __popc(m);
    }
  }
  for (int t = n + (int)threadIdx.x; t < cap; t += WT) out[t] = -1;
  if (lane == 0 && (q != qend || n > cap || cap - n >= KC)) atomicOr(status, 16);   // the two scans disagree
}

// the records, a warp per chunk: lane e (and e + 16) owns entry e, the two
// halves take the member row's 16-byte groups in turn.  A missing entry (the
// last chunk's padding) is a point out of every column's reach with weight 0.
constexpr int RW = 8;   // chunks per block
__global__ void __launch_bounds__(32 * RW) k_tile_rec(int nchunks, ObsSorted obs, int k, int kp, int kr, int cb,
                                                      const int *list, unsigned char *rec) {
  const int c = blockIdx.x * RW + (threadIdx.x >> 5), lane = threadIdx.x & 31, e = lane & 15, h = lane >> 4;
  if (c >= nchunks) return;
  const int p = list[(size_t)c * KC + e];
  const bool in = p >= 0;
  float *r0 = reinterpret_cast<float *>(rec + (size_t)c * cb), *yT = r0 + 128;
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 B = in ? __ldg(obs.B + p) : z;
  if (h == 0) {
    float4 A = make_float4(4.f, 0.f, 0.f, 0.f);
    if (in) {
      A = __ldg(obs.A + p);
      A.w = __frcp_rn(A.w);
    }
    r0[e] = A.x; r0[16 + e] = A.y; r0[32 + e] = A.z; r0[48 + e] = A.w;
  } else {
    r0[64 + e] = B.x; r0[80 + e] = B.y; r0[96 + e] = B.z; r0[112 + e] = B.w;
  }
  const float4 *h4 = reinterpret_cast<const float4 *>(obs.hx + (size_t)(in ? p : 0) * kp);
  const int n4 = in ? kp >> 2 : 0;
  for (int q0 = h; q0 < kr >> 2; q0 += 8) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = q0 + 2 * u < n4 ? __ldg(h4 + q0 + 2 * u) : z;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = 4 * (q0 + 2 * u);
      if (i < kr) {
        yT[(i + 0) * YS + e] = i + 0 < k ? v[u].x : (i + 0 == k ? B.x : 0.0f);
        yT[(i + 1) * YS + e] = i + 1 < k ? v[u].y : (i + 1 == k ? B.x : 0.0f);
        yT[(i + 2) * YS + e] = i + 2 < k ? v[u].z : (i + 2 == k ? B.x : 0.0f);
        yT[(i + 3) * YS + e] = i + 3 < k ? v[u].w : (i + 3 == k ? B.x : 0.0f);
      }
    }
  }
  for (int t = lane; t < kr * (YS - 16); t += 32) yT[(t >> 2) * YS + 16 + (t & 3)] = 0.0f;
}
static_assert(YS - 16 == 4, "pad columns of a member row");

// fp32 pair -> TF32 hi + lo (tc::split_tf32 on both halves)
__device__ __forceinline__ void split2(F2 v, F2 &hi, F2 &lo) {
  uint32_t h0, h1;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h0) : "f"(v.x()));
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h1) : "f"(v.y()));
  hi = F2(__uint_as_float(h0), __uint_as_float(h1));
  lo = f2_fma(hi, F2(kFC.minus_one), v);   // exact
}

// two values -> FP16 hi and lo pairs (the first in the low half)
__device__ __forceinline__ uint32_t pack_f16(float x, float y) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
__device__ __forceinline__ void split_f16(F2 v, uint32_t &hi, uint32_t &lo) {
  hi = pack_f16(v.x(), v.y());
  float a, b;
  asm("{\n\t.reg .f16 l, h;\n\tmov.b32 {l, h}, %2;\n\tcvt.f32.f16 %0, l;\n\tcvt.f32.f16 %1, h;\n\t}"
      : "=f"(a), "=f"(b) : "r"(hi));
  const F2 d = f2_fma(F2(a, b), F2(kFC.minus_one), v);   // exact
  lo = pack_f16(d.x(), d.y());
}

struct TcSmem {
  unsigned long long full[NSMAX], empty[NSMAX], rfull[NRMAX], done;
  unsigned long long accf;   // drain: the accumulation so far is complete in TMEM (commit + MMA thread)
  unsigned long long acce;   // drain: the producer warps have read TMEM (one arrival per warp)
  int anyk[NSMAX];           // chunk index + 1 of the last chunk of the stage with a kept pair
  uint32_t tmem;
  int issued;                // MMAs were issued since the last drain
  int sub_issued;            // the same, for the accumulation a drain hands over
  int fault;
  unsigned char fi[NPMAX];
  unsigned char fj[NPMAX];
};

// per-CTA constants of the localizer's fast path
struct LocK {
  float icv, levg;            // vtgc: vertical 1/c, depth of the group's level
  float tprof, tsat;          // ocean: time scales (0 = off)
  float ictp, icts;           // ocean: their 1/c
};

// a producer thread's column, both halves of the pairs alike
struct ColFast {
  F2 nx, ny, nz;              // negated unit vector
  float ic1, ic2;             // 1/c of the length scales
  float c2in, c2max;          // squared chord of the search radius; with its margin
  float cscale;               // |c2 - c2in| * cscale <= kGuardFast: within the chord band
};

// fast localisation weights of observations e, e + 1 (no branches) at the
// distances d; LOC selects the localizer class.  Beyond the search radius the
// single-factor class may return anything.
template <int LOC>
__device__ __forceinline__ F2 loc_fast(const LocK &lk, const ColFast &cf, int g, F2 d, const float *rec, int e) {
  if (LOC == LOC_VTGC) {
    const float z0 = fabsf(rec[96 + e] - lk.levg), z1 = fabsf(rec[97 + e] - lk.levg);
    return f2_mul(gc_branchless(f2_mul(d, f2_all(cf.ic1)), true), gc_branchless(F2(z0 * lk.icv, z1 * lk.icv), true));
  } else if (LOC == LOC_OCEAN) {
    float w[2];
    const bool s0 = rec[112 + e] != 0.0f, s1 = rec[113 + e] != 0.0f;
    const F2 rh = gc_branchless(f2_mul(d, F2(s0 ? cf.ic2 : cf.ic1, s1 ? cf.ic2 : cf.ic1)), true);
    const F2 rt = gc_branchless(F2(fabsf(rec[80 + e]) * (s0 ? lk.icts : lk.ictp),
                                   fabsf(rec[81 + e]) * (s1 ? lk.icts : lk.ictp)), true);
    w[0] = rh.x() * ((s0 ? lk.tsat : lk.tprof) > 0.0f ? rt.x() : 1.0f);
    w[1] = rh.y() * ((s1 ? lk.tsat : lk.tprof) > 0.0f ? rt.y() : 1.0f);
    return F2(s0 && g == 1 ? 0.0f : w[0], s1 && g == 1 ? 0.0f : w[1]);
  } else {
    return gc_branchless(f2_mul(d, f2_all(cf.ic1)), false);
  }
}

__device__ __forceinline__ void bar_arrive(unsigned long long *b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(b)) : "memory");
}

// CULL: a warp whose 32 columns have none of its four records within their
// search chords skips the distance and localizer evaluation (their weights are
// zero either way; results are bit-identical); pays where search radii are
// small next to the tile caps, costs registers where they are not
template <int LOC, int NR, bool CULL, bool F16>
__global__ void __launch_bounds__(gram_threads(NPMAX), 1) k_gram_tc(TcArgs a) {
  constexpr int NS = stages_of(F16), CPR = round_of(F16), NSR = NS / CPR, NRR = NR / CPR;   // NSR, NRR: in rounds
  constexpr uint32_t SBO = sbo_of(F16), WB = wb_of(F16);
  static_assert(NS <= NSMAX && NR <= NRMAX, "operand stages / record slots beyond the barrier arrays");
  extern __shared__ __align__(1024) unsigned char dsm[];
  __shared__ __align__(16) TcSmem S;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int mma_warp = (int)(blockDim.x >> 5) - 1;   // = the number of producer warps
  // block = (work item, group, pass), pass fastest: the passes of a work item
  // run side by side and share its records in L2
  const int pass = blockIdx.x % a.npass;
  const int g = (blockIdx.x / a.npass) % a.groups;
  const TcWork wk = a.work[blockIdx.x / (a.npass * a.groups)];
  const int tile = wk.tile;
  const int k = a.k, NP = a.np, nf = a.nf, cb = a.cb;
  const int slotb = cb;   // ring slot: one chunk record
  const uint32_t PB = (uint32_t)(NP / 8) * SBO;
  const uint32_t stage_bytes = 2 * WB + 2 * PB;
  auto stage_ptr = [&](int s) { return dsm + (size_t)s * stage_bytes; };
  unsigned char *ring = dsm + (size_t)NS * stage_bytes;
  // this CTA's segment of the tile's chunk stream
  const int t0 = a.tile_off[tile], tn = a.tile_off[tile + 1] - t0;
  const int cs = min(tn, wk.cs), ce = min(tn, wk.ce);
  const int c0 = t0 + cs;
  const int nchunks = ce - cs, nrounds = (nchunks + CPR - 1) / CPR;
  const uint32_t tmem_cols = a.tmem_cols;
  if (nchunks <= 0 && wk.blk0 < 0) {
    // no observation within the tile's cap: nothing is kept, and the G of a
    // unit that keeps nothing is never read
    const int col = tid < TM && pass == 0 ? a.tile_cols[(size_t)tile * TM + tid] : -1;
    if (col >= 0) {
      a.nkept[(size_t)a.col2act[col] * a.groups + g] = 0;
      if (a.diag_lg_obscount) a.diag_lg_obscount[(size_t)g * a.ncol + col] = 0.0f;
      if (a.diag_lg_obsloc) a.diag_lg_obsloc[(size_t)g * a.ncol + col] = 0.0f;
      if (g == 0 && a.diag_obscount) a.diag_obscount[col] = 0.0f;
    }
    return;
  }

  // ---- setup: TMEM, barriers, feature table
  if (wid == 0) tc::tmem_alloc(&S.tmem, tmem_cols);
  if (tid == 0) {
    for (int s = 0; s < NS; s++) S.anyk[s] = 0;
    for (int s = 0; s < NSR; s++) {
      tc::mbar_init(reinterpret_cast<uint64_t *>(&S.full[s]), (uint32_t)mma_warp);
      tc::mbar_init(reinterpret_cast<uint64_t *>(&S.empty[s]), 1);
    }
    for (int r = 0; r < NRR; r++) tc::mbar_init(reinterpret_cast<uint64_t *>(&S.rfull[r]), 1);
    tc::mbar_init(reinterpret_cast<uint64_t *>(&S.done), 1);
    tc::mbar_init(reinterpret_cast<uint64_t *>(&S.accf), 2);
    tc::mbar_init(reinterpret_cast<uint64_t *>(&S.acce), NW);
    S.issued = 0;
    S.sub_issued = 0;
    S.fault = 0;
    tc::mbar_fence_init();
  }
  for (int f = tid; f < NP; f += (int)blockDim.x) {
    const int fg = pass * NP + f;
    int i = 255, j = 255;
    if (fg < nf) packed_ij(fg, k, i, j);
    S.fi[f] = (unsigned char)i;
    S.fj[f] = (unsigned char)j;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = S.tmem;

  // weight thread: column wc, observations [e0, e0 + 4) of each chunk
  const int wc = tid & (TM - 1), wq = (tid >> 7) & 3, e0 = 4 * wq;
  int ncand = 0, nkeep = 0;
  float rsum = 0.0f;

  // the tile's power-of-two scale of the features, and what takes it and the
  // weights' out of the accumulator
  const uint32_t mmax = F16 ? a.tile_mag[2 * tile] : 0u;
  const int pe = F16 && mmax != 0u ? kPTop - f32_exp(mmax) : 0;
  const float pscale = F16 ? pow2(pe) : 1.0f, oscale = F16 ? pow2(-pe) * (1.0f / kWScale) : 1.0f;
  // The CTA's results: TMEM lane = column wc of a weight thread.  A tile whose stream is one
  // drain interval writes the column's G row (thread tid < TM, warps 0-3);
  // otherwise every drain interval goes to its own partial block,
  // feature-major, so that a warp's stores of one feature are 32 consecutive
  // floats (the weight warps drain: warp w its lane quarter w % 4, the
  // features of quarter w / 4).

  const int G = a.groups;
  const int D = a.drain;
  const int nvalid = nf - pass * NP < NP ? nf - pass * NP : NP;
  // the accumulator's lane of this thread (TMEM lane quarter wid % 4; zeros
  // unless from_tmem, which is CTA-uniform), features [16 q, 16 q + 16) for
  // q = q0, q0 + qs, ..., into partial block blk
  auto store_block = [&](int blk, bool from_tmem, int q0, int qs) {
    float *base = a.Gpart + (((size_t)blk * G + g) * nf + (size_t)pass * NP) * TM + wc;
    for (int f0 = 16 * q0; f0 < NP; f0 += 16 * qs) {
      float v[16];
      if (from_tmem) {
        tc::tmem_ld16(tmem + ((uint32_t)((wid & 3) * 32) << 16) + (uint32_t)f0, v);
      } else {
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 16; q++)
        if (f0 + q < nvalid) base[(size_t)(f0 + q) * TM] = F16 ? v[q] * oscale : v[q];
    }
  };
  // drain j (all weight warps):
  // wait until the MMAs before boundary (j + 1) D have completed, move the
  // accumulator to its block, hand TMEM back to the MMA thread
  const int nflush = nchunks > 0 ? (nchunks - 1) / D : 0;
  int nflushed = 0;
  auto flush = [&](int j) {
    if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.accf), j & 1)) S.fault = 1;
    tc::fence_after();
    store_block(wk.blk0 + j, S.sub_issued != 0 && S.fault == 0, wid >> 2, 4);
    tc::fence_before();
    __syncwarp();
    if (lane == 0) bar_arrive(&S.acce);
  };

  if (wid < NW) {
    const int col = a.tile_cols[(size_t)tile * TM + wc];
    const bool colv = col >= 0;
    ColFast cf;
    {
      // no column: a point out of reach of every record
      float ux = -4.0f, uy = 0.0f, uz = 0.0f, rmax = 0.0f;
      cf.ic1 = cf.ic2 = 1.0f;
      if (colv) {
        const ColPar &cp = a.cp[col];
        ux = cp.ux; uy = cp.uy; uz = cp.uz; rmax = cp.rmax;
        cf.ic1 = cp.ic1;
        cf.ic2 = cp.ic2;
      }
      cf.nx = f2_all(-ux);
      cf.ny = f2_all(-uy);
      cf.nz = f2_all(-uz);
      const float sh = sinf(fminf(rmax / 12742000.0f, 1.5707963f));
      cf.c2in = colv ? 4.0f * sh * sh : 0.0f;
      cf.c2max = colv ? cf.c2in * 1.0001f + 1e-12f : -1.0f;
      // (a radius within rounding of zero is all band)
      cf.cscale = colv ? kGuardFast / (kFastChordBand * cf.c2in + 1e-14f) : 1.0f;
    }
    const float hmax = a.tp[tile].hmax;   // CTA-uniform
    const bool short_asin = hmax <= 0.25f, far = hmax > 0.5f;
    LocK lk;
    lk.icv = LOC == LOC_VTGC ? inv_c_of(a.loc.vloc) : 1.0f;
    lk.levg = LOC == LOC_VTGC ? a.loc.lev_depth[g] : 0.0f;
    lk.tprof = a.loc.tloc_prof;
    lk.tsat = a.loc.tloc_sat;
    lk.ictp = (LOC == LOC_OCEAN && lk.tprof > 0.0f) ? inv_c_of(lk.tprof) : 1.0f;
    lk.icts = (LOC == LOC_OCEAN && lk.tsat > 0.0f) ? inv_c_of(lk.tsat) : 1.0f;
    for (int rd = 0; rd < nrounds; rd++) {
      const int sr = rd % NSR, rr = rd % NRR;
      // the producers drain TMEM at boundary b = (j + 1) D (D a multiple of
      // CPR) once the stages of chunks b .. b + NS - 1 are produced: the MMA
      // of chunk b + NS needs the stage chunk b frees, which waits for the drain
      if (nflushed < nflush && rd * CPR == (nflushed + 1) * D + NS) flush(nflushed++);
      if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.rfull[rr]), (rd / NRR) & 1)) { S.fault = 1; break; }
      if (rd >= NSR && !tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.empty[sr]), ((rd / NSR) - 1) & 1)) {
        S.fault = 1;
        break;
      }
#pragma unroll 1
      for (int ch = rd * CPR; ch < min(nchunks, (rd + 1) * CPR); ch++) {
        const int s = ch % NS, r = ch % NR;
        const unsigned char *rec = ring + (size_t)r * slotb;
        const float *R = reinterpret_cast<const float *>(rec);
        unsigned char *Whi = stage_ptr(s), *Wlo = Whi + WB;
        bool anyk = false;
        // ---- weights: four observations, fast path without branches
        float w[4];
        unsigned inr = 0;
        F2 ox[2], oy[2], oz[2], c2[2];
        f2_load2(R + e0, ox[0], ox[1]);
        f2_load2(R + 16 + e0, oy[0], oy[1]);
        f2_load2(R + 32 + e0, oz[0], oz[1]);
        float cmin = 3.0e38f, cmax = 0.0f;
#pragma unroll
        for (int u = 0; u < 4; u++) w[u] = 0.0f;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          c2[h] = chord2_fast(cf.nx, cf.ny, cf.nz, ox[h], oy[h], oz[h]);
          cmin = fminf(cmin, fminf(c2[h].x(), c2[h].y()));
        }
        bool go = true;
        if constexpr (CULL) go = __any_sync(0xffffffffu, cmin <= cf.c2max);
        if (go) {
          float near = 1.0f;   // the smallest distance of a decision from its threshold, in units of kGuardFast's scale
          float c[4], rl[4];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const F2 r2 = loc_fast<LOC>(lk, cf, g, dist_fast(c2[h], short_asin), R, e0 + 2 * h);
            c[2 * h] = c2[h].x();
            c[2 * h + 1] = c2[h].y();
            rl[2 * h] = r2.x();
            rl[2 * h + 1] = r2.y();
          }
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const bool in = c[u] <= cf.c2in;
            near = fminf(near, fminf(fabsf(c[u] - cf.c2in) * cf.cscale, fabsf(rl[u] - kKeep)));
            w[u] = in && rl[u] > kKeep ? rl[u] : 0.0f;
            inr += in;
            cmax = fmaxf(cmax, c[u]);
          }
          // beyond a chord of 1 the fast distance does not hold
          if (far) near = cmax > 1.0f ? 0.0f : near;
          // ---- rare: exact metric and the per-column localizer
          if (__any_sync(0xffffffffu, near <= kGuardFast) && near <= kGuardFast) {
            inr = 0;
#pragma unroll 1
            for (int u = 0; u < 4; u++) {
              float cu = c[0], wu = w[0], ru = rl[0];
#pragma unroll
              for (int v = 1; v < 4; v++) {
                cu = u == v ? c[v] : cu;
                wu = u == v ? w[v] : wu;
                ru = u == v ? rl[v] : ru;
              }
              bool in = cu <= cf.c2in;
              const bool unsure = cu <= cf.c2max && (cu > 1.0f || fabsf(cu - cf.c2in) * cf.cscale <= kGuardFast ||
                                                     (in && fabsf(ru - kKeep) <= kGuardFast));
              if (unsure) {
                const int e = e0 + u;
                // the column's parameters from global memory (keeps them out of
                // the producers' registers)
                const ColPar &cp = a.cp[col];
                const float de = dist_from_chord2(chord2_exact(cp.ux, cp.uy, cp.uz, R[e], R[16 + e], R[32 + e]));
                in = de <= cp.rmax;
                const float re = in ? localize_cls<LOC>(a.loc, cp, g, de, R[80 + e], R[96 + e], R[112 + e]) : 0.0f;
                wu = re > kKeep ? re : 0.0f;
              }
              inr += in;
#pragma unroll
              for (int v = 0; v < 4; v++) w[v] = u == v ? wu : w[v];
            }
          }
        }
        {
          ncand += inr;
          float wmax = 0.0f;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            nkeep += w[u] > 0.0f;
            rsum += w[u];
            wmax = fmaxf(wmax, w[u]);
          }
          anyk = wmax > 0.0f;
          const uint32_t off = kmaj<F16>(wc, e0);
          if constexpr (F16) {
            uint32_t hi[2], lo[2];
#pragma unroll
            for (int h = 0; h < 2; h++)
              split_f16(f2_mul(F2(w[2 * h], w[2 * h + 1]), f2_all(kWScale)), hi[h], lo[h]);
            *reinterpret_cast<uint2 *>(Whi + off) = make_uint2(hi[0], hi[1]);
            *reinterpret_cast<uint2 *>(Wlo + off) = make_uint2(lo[0], lo[1]);
          } else {
            F2 ri[2], hi[2], lo[2];
            f2_load2(R + 48 + e0, ri[0], ri[1]);   // 1/err
#pragma unroll
            for (int h = 0; h < 2; h++) split2(f2_mul(F2(w[2 * h], w[2 * h + 1]), ri[h]), hi[h], lo[h]);
            f2_store2(reinterpret_cast<float *>(Whi + off), hi[0], hi[1]);
            f2_store2(reinterpret_cast<float *>(Wlo + off), lo[0], lo[1]);
          }
        }
        if (__any_sync(0xffffffffu, anyk) && lane == 0) S.anyk[s] = ch + 1;
      }
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bar_arrive(&S.full[sr]);
    }
    while (nflushed < nflush) flush(nflushed++);
  } else if (wid < mma_warp) {
    // ================================================= feature products: feature f over a chunk's 16 observations
    const int f = tid - 32 * NW;
    const bool fin = f < NP;
    const int fi = fin ? S.fi[f] : 255, fj = fin ? S.fj[f] : 255;
    // a feature past the last one multiplies row 0; its accumulator is not read
    const int rowi = (fi != 255 ? fi : 0) * YS, rowj = (fi != 255 ? fj : 0) * YS;
    for (int rd = 0; rd < nrounds; rd++) {
      const int sr = rd % NSR, rr = rd % NRR;
      if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.rfull[rr]), (rd / NRR) & 1)) { S.fault = 1; break; }
      if (rd >= NSR && !tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.empty[sr]), ((rd / NSR) - 1) & 1)) {
        S.fault = 1;
        break;
      }
#pragma unroll 1
      for (int ch = rd * CPR; fin && ch < min(nchunks, (rd + 1) * CPR); ch++) {
        const int s = ch % NS, r = ch % NR;
        unsigned char *Phi = stage_ptr(s) + 2 * WB, *Plo = Phi + PB;
        const float *R = reinterpret_cast<const float *>(ring + (size_t)r * slotb);
        const float *yi = R + 128 + rowi, *yj = R + 128 + rowj;
        if constexpr (F16) {
#pragma unroll
          for (int grp = 0; grp < 2; grp++) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int q = 0; q < 2; q++) {
              const int e = 8 * grp + 4 * q;
              F2 ai[2], bj[2], ri[2];
              f2_load2(yi + e, ai[0], ai[1]);
              f2_load2(yj + e, bj[0], bj[1]);
              f2_load2(R + 48 + e, ri[0], ri[1]);   // 1/err
#pragma unroll
              for (int h = 0; h < 2; h++)
                split_f16(f2_mul(f2_mul(f2_mul(ai[h], ri[h]), f2_all(pscale)), bj[h]), hi[2 * q + h], lo[2 * q + h]);
            }
            const uint32_t off = kmaj<F16>(f, 8 * grp);
            *reinterpret_cast<uint4 *>(Phi + off) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4 *>(Plo + off) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        } else {
#pragma unroll
          for (int grp = 0; grp < 4; grp++) {
            F2 ai[2], bj[2], hi[2], lo[2];
            f2_load2(yi + 4 * grp, ai[0], ai[1]);
            f2_load2(yj + 4 * grp, bj[0], bj[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) split2(f2_mul(ai[h], bj[h]), hi[h], lo[h]);
            const uint32_t off = kmaj<F16>(f, grp * 4);
            f2_store2(reinterpret_cast<float *>(Phi + off), hi[0], hi[1]);
            f2_store2(reinterpret_cast<float *>(Plo + off), lo[0], lo[1]);
          }
        }
      }
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) bar_arrive(&S.full[sr]);
    }
  } else {
    // ================================================= MMA issue + record loads (one thread)
    if (lane == 0) {
      const unsigned char *src = a.rec + (size_t)c0 * cb;
      // the records of a round, one copy
      auto load = [&](int rd) {
        unsigned char *dst = ring + (size_t)(rd % NRR) * CPR * slotb;
        uint64_t *bar = reinterpret_cast<uint64_t *>(&S.rfull[rd % NRR]);
        tc::bulk_load(dst, src + (size_t)rd * CPR * cb, (uint32_t)(min(CPR, nchunks - rd * CPR) * cb), bar);
      };
      int n_loaded = nrounds < NRR ? nrounds : NRR;
      for (int rd = 0; rd < n_loaded; rd++) load(rd);
      const int nb0 = NP < 256 ? NP : 256, nb1 = NP - nb0;
      auto idesc = [](int n) { return F16 ? tc::idesc_f16(TM, n) : tc::idesc_tf32(TM, n); };
      const uint32_t id0 = idesc(nb0), id1 = nb1 > 0 ? idesc(nb1) : 0u;
      auto mma = [](uint32_t d, uint64_t ad, uint64_t bd, uint32_t id, uint32_t acc) {
        if constexpr (F16) tc::mma_f16(d, ad, bd, id, acc);
        else tc::mma_tf32(d, ad, bd, id, acc);
      };
      constexpr int KS = F16 ? 1 : KC / 8;   // MMA steps of a chunk
      bool issued = false;   // since the last drain
      int nmma = 0, fj = 0;
      for (int rd = 0; rd < nrounds; rd++) {
        const int sr = rd % NSR;
        if (rd > 0 && rd * CPR % D == 0) {
          // boundary: hand the accumulation to the producer warps and wait
          // until they have read TMEM; the next MMA starts a fresh accumulation
          S.sub_issued = issued ? 1 : 0;
          tc::commit(reinterpret_cast<uint64_t *>(&S.accf));
          bar_arrive(&S.accf);
          if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.acce), fj & 1)) { S.fault = 1; break; }
          tc::fence_after();
          fj++;
          issued = false;
        }
        if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.full[sr]), (rd / NSR) & 1)) { S.fault = 1; break; }
        // every producer is done with the records of the round: refill the slot
        if (n_loaded < nrounds) load(n_loaded++);
        bool any = false;
        for (int ch = rd * CPR; ch < min(nchunks, (rd + 1) * CPR); ch++) {
          const int s = ch % NS;
          if (S.anyk[s] == ch + 1) {
            tc::fence_after();
            const uint32_t whi = tc::smem_u32(stage_ptr(s)), wlo = whi + WB, phi = whi + 2 * WB, plo = phi + PB;
#pragma unroll
            for (int t = 0; t < 3; t++)
#pragma unroll
              for (int ks = 0; ks < KS; ks++) {
                const uint32_t acc = (issued || t > 0 || ks > 0) ? 1u : 0u;
                const uint32_t aw = t == 2 ? wlo : whi, bp = t == 1 ? plo : phi;
                const uint64_t ad = tc::smem_desc(aw + ks * 2 * CMB, CMB, SBO);
                const uint64_t bd0 = tc::smem_desc(bp + ks * 2 * CMB, CMB, SBO);
                mma(tmem, ad, bd0, id0, acc);
                if (nb1 > 0) {
                  const uint64_t bd1 = tc::smem_desc(bp + (uint32_t)(nb0 / 8) * SBO + ks * 2 * CMB, CMB, SBO);
                  mma(tmem + (uint32_t)nb0, ad, bd1, id1, acc);
                }
              }
            issued = any = true;
            nmma++;
          }
        }
        if (any) tc::commit(reinterpret_cast<uint64_t *>(&S.empty[sr]));
        else bar_arrive(&S.empty[sr]);
      }
      // every MMA issued by this thread has completed once `done` flips
      tc::commit(reinterpret_cast<uint64_t *>(&S.done));
      if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.done), 0)) S.fault = 1;
      S.issued = issued ? 1 : 0;
      if (nmma) atomicAdd(a.status + 2, nmma);   // chunks whose MMAs ran (executed-work counter)
      // no record copy may still be in flight when the CTA exits
      for (int rd = n_loaded > NRR ? n_loaded - NRR : 0; rd < n_loaded; rd++)
        if (!tc::mbar_wait(reinterpret_cast<uint64_t *>(&S.rfull[rd % NRR]), (rd / NRR) & 1)) S.fault = 1;
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const bool fault = S.fault != 0;
  const bool issued = S.issued != 0;
  // per-column partial counts of the observation groups, in the (now idle)
  // operand stage memory
  constexpr int NG = KC / 4;
  int *dcand = reinterpret_cast<int *>(dsm), *dkept = dcand + NG * TM;
  float *drsum = reinterpret_cast<float *>(dkept + NG * TM);
  if (wid < NW) {
    dcand[wq * TM + wc] = ncand;
    dkept[wq * TM + wc] = nkeep;
    drsum[wq * TM + wc] = rsum;
  }
  __syncthreads();

  // ---- per-column diagnostics and kept counts
  int *ckept = reinterpret_cast<int *>(drsum + NG * TM);   // kept by the column
  if (tid < TM) {
    ncand = dcand[tid];
    nkeep = dkept[tid];
    rsum = drsum[tid];
    for (int q = 1; q < NG; q++) {
      ncand += dcand[q * TM + tid];
      nkeep += dkept[q * TM + tid];
      rsum += drsum[q * TM + tid];
    }
    ckept[tid] = nkeep;
    const int col = a.tile_cols[(size_t)tile * TM + tid];
    if (col >= 0 && pass == 0) {
      const size_t unit = (size_t)a.col2act[col] * G + g;
      if (wk.cblk < 0) {
        a.nkept[unit] = nkeep;
        if (a.diag_lg_obscount) a.diag_lg_obscount[(size_t)g * a.ncol + col] = (float)nkeep;
        if (a.diag_lg_obsloc) a.diag_lg_obsloc[(size_t)g * a.ncol + col] = rsum;
        if (g == 0 && a.diag_obscount) a.diag_obscount[col] = (float)ncand;
      } else {
        float *cc = a.cnt + (((size_t)wk.cblk * G + g) * TM + tid) * 3;
        cc[0] = (float)nkeep;
        cc[1] = (float)ncand;
        cc[2] = rsum;
      }
    }
  }
  __syncthreads();
  // ---- epilogue: weight warp w reads TMEM lane quarter w % 4 and stores the
  // features of quarter w / 4.  (On four warps alone it left the CTA's
  // other warps waiting: simple3d, k = 50, with the rows of columns that keep
  // nothing: 121 us for the whole kernel, now 21.)
  if (wid < NW) {
    if (wk.blk0 >= 0) {
      // the last drain interval of the segment
      store_block(wk.blk0 + nflush, issued && !fault, wid >> 2, 4);
    } else {
      // the whole stream in one accumulator: the column's G row (16-byte
      // aligned: nf and NP are multiples of 4) where the column kept any
      const int col = ckept[wc] > 0 ? a.tile_cols[(size_t)tile * TM + wc] : -1;
      float *Gp = col >= 0 ? a.G + ((size_t)a.col2act[col] * G + g) * (size_t)nf + (size_t)pass * NP : nullptr;
      const bool any = __any_sync(0xffffffffu, Gp != nullptr);
      for (int f0 = 16 * (wid >> 2); any && f0 < NP; f0 += 64) {
        float v[16];
        if (issued && !fault) {
          tc::tmem_ld16(tmem + ((uint32_t)((wid & 3) * 32) << 16) + (uint32_t)f0, v);
        } else {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] = 0.0f;
        }
        if constexpr (F16) {
#pragma unroll
          for (int q = 0; q < 16; q++) v[q] *= oscale;
        }
        if (Gp) {
          if (f0 + 16 <= nvalid && (nf & 3) == 0) {
#pragma unroll
            for (int q = 0; q < 16; q += 4)
              *reinterpret_cast<float4 *>(Gp + f0 + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
          } else {
#pragma unroll
            for (int q = 0; q < 16; q++)
              if (f0 + q < nvalid) Gp[f0 + q] = v[q];
          }
        }
      }
    }
  }
  if (fault && tid == 0) atomicOr(a.status, 16);
  tc::fence_before();
  __syncthreads();
  if (wid == 0) tc::tmem_dealloc(tmem, tmem_cols);
}

// Stage / ring depths: four FP16 or two TF32 operand stages (k <= 128: 4 x 38 KB
// or 2 x 76 KB) and six record slots (10.8 KB).  With TF32 operands at k = 40
// six slots made the Gram 1.8 ms faster than three stages with three slots (the
// producers waited on the record copies); twelve slots gained nothing more.
size_t gram_tc_smem(int k, int np, bool f16) {
  const size_t PB = (size_t)(np / 8) * sbo_of(f16);
  return stages_of(f16) * (2 * wb_of(f16) + 2 * PB) + NRMAX * record_bytes(k);
}

}  // namespace

size_t tile_count_ints(int ntiles) { return (size_t)ntiles * (1 + WT / 32 + 2); }

size_t record_bytes(int k) { return 512 + (size_t)(((k + 4) & ~3) * YS) * sizeof(float); }

void gram_tc_passes(int k, int *npass, int *np) {
  const int nf = packed_size(k);
  int p = (nf + NPMAX - 1) / NPMAX;
  int n = (nf + p - 1) / p;
  n = (n + 15) & ~15;
  while (n > NPMAX) { p++; n = ((nf + p - 1) / p + 15) & ~15; }
  *npass = p;
  *np = n;
}

cudaError_t launch_tile_count(cudaStream_t st, int ntiles, const TilePar *tp, const IndexGeom *geom,
                              const ObsSorted &obs, int *tile_n, int *tile_wn, uint32_t *tile_mag, int *tile_off,
                              int *launches) {
  if (ntiles <= 0) return cudaMemsetAsync(tile_off, 0, 2 * sizeof(int), st);
  k_tile_count<<<ntiles, WT, 0, st>>>(ntiles, tp, geom, obs.A, obs.mag, obs.cell_start, tile_n, tile_wn, tile_mag);
  k_tile_scan<<<1, 1024, 0, st>>>(ntiles, tile_n, tile_mag, tile_off);
  (*launches) += 2;
  return cudaGetLastError();
}

cudaError_t launch_tile_fill(cudaStream_t st, int ntiles, int nchunks, const TilePar *tp, const IndexGeom *geom,
                             const ObsSorted &obs, int k, int kp, const int *tile_n, const int *tile_wn,
                             const int *tile_off, int *list, unsigned char *rec, int *status, int *launches) {
  if (ntiles <= 0 || nchunks <= 0) return cudaSuccess;
  const int kr = (k + 4) & ~3;
  k_tile_list<<<ntiles, WT, 0, st>>>(tp, geom, obs.A, obs.cell_start, tile_n, tile_wn, tile_off, list, status);
  k_tile_rec<<<(nchunks + RW - 1) / RW, 32 * RW, 0, st>>>(nchunks, obs, k, kp, kr, (int)record_bytes(k), list, rec);
  (*launches) += 2;
  return cudaGetLastError();
}

template <int LOC, bool CULL, bool F16>
static cudaError_t launch_gram_tc_loc(cudaStream_t st, const TcArgs &a, int *launches) {
  const size_t smem = gram_tc_smem(a.k, a.np, F16);
  if (smem > kSmemBudget) return cudaErrorInvalidValue;   // k <= 128 fits
  const long long grid = (long long)a.nwork * a.groups * a.npass;
  if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
  auto kern = k_gram_tc<LOC, NRMAX, CULL, F16>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kern<<<(int)grid, gram_threads(a.np), smem, st>>>(a);
  (*launches)++;
  return cudaGetLastError();
}

template <int LOC>
static cudaError_t launch_gram_tc_form(cudaStream_t st, const TcArgs &a, int *launches) {
  if (a.f16)
    return a.cull ? launch_gram_tc_loc<LOC, true, true>(st, a, launches)
                  : launch_gram_tc_loc<LOC, false, true>(st, a, launches);
  return a.cull ? launch_gram_tc_loc<LOC, true, false>(st, a, launches)
                : launch_gram_tc_loc<LOC, false, false>(st, a, launches);
}

cudaError_t launch_gram_tc(cudaStream_t st, const TcArgs &a_in, int *launches) {
  if (a_in.ntiles <= 0) return cudaSuccess;
  TcArgs a = a_in;
  a.cb = (int)record_bytes(a.k);
  uint32_t tc = 32;
  while ((int)tc < a.np) tc <<= 1;
  a.tmem_cols = tc;
  switch (a.loc.cls) {
  case LOC_OCEAN: return launch_gram_tc_form<LOC_OCEAN>(st, a, launches);
  case LOC_VTGC: return launch_gram_tc_form<LOC_VTGC>(st, a, launches);
  default: return launch_gram_tc_form<LOC_NOVRT>(st, a, launches);
  }
}

namespace {
// A tile whose stream spans several drain intervals: G = the sum of its
// partial blocks in stream order, compensated in FP32 (Sum2 of Ogita, Rump
// and Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26(6),
// 2005: Knuth's error-free TwoSum carries each addition's rounding error
// into a second accumulator, so the result is as accurate as a sum in twice
// the working precision, rounded once; GB300's FP64 pipe is 1/64 of its FP32
// rate, which an FP64 sum of the partials runs into); kept counts,
// candidate counts and the sums of rho summed over the segments in segment
// order (FP32 for rho, as one CTA accumulates it).  One block per (tile,
// group, 32 features): the sums are formed with threads along the columns
// (coalesced block reads) and written with a warp along a column's row
// (coalesced G writes) through shared memory; the first feature block of a
// (tile, group) also sums the counts.
constexpr int SST = 256;
__global__ void __launch_bounds__(SST) k_gram_segsum(TcArgs a) {
  __shared__ float acc[32][TM + 1];
  const int nfc = (a.nf + 31) / 32;
  const int fc = blockIdx.x % nfc, tg = blockIdx.x / nfc;
  const TcSegTile st = a.segtiles[tg / a.groups];
  const int g = tg % a.groups, G = a.groups, nf = a.nf;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = tid & (TM - 1), fh = tid >> 7;   // column, feature half
  const size_t bstride = (size_t)G * nf * TM;   // between consecutive blocks
  const float *P = a.Gpart + ((size_t)st.blk0 * G + g) * nf * TM;
  {
    const int f0 = 32 * fc;
    // blocks in stream order, the 16 features' loads of a block independent
    float hs[16], ls[16];   // running sum, accumulated rounding errors
#pragma unroll
    for (int i = 0; i < 16; i++) hs[i] = ls[i] = 0.0f;
    const int fb = f0 + fh * 16;
    for (int b = 0; b < st.nblk; b++) {
      const float *Pb = P + b * bstride + (size_t)fb * TM + c;
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; i++) x[i] = fb + i < nf ? Pb[(size_t)i * TM] : 0.0f;
#pragma unroll
      for (int i = 0; i < 16; i++) {
        // TwoSum: s + e == hs + x exactly
        const float s = __fadd_rn(hs[i], x[i]);
        const float z = __fsub_rn(s, hs[i]);
        const float e = __fadd_rn(__fsub_rn(hs[i], __fsub_rn(s, z)), __fsub_rn(x[i], z));
        hs[i] = s;
        ls[i] = __fadd_rn(ls[i], e);
      }
    }
#pragma unroll
    for (int i = 0; i < 16; i++) acc[fh * 16 + i][c] = __fadd_rn(hs[i], ls[i]);
    __syncthreads();
    for (int cc = warp; cc < TM; cc += SST / 32) {
      const int col = a.tile_cols[(size_t)st.tile * TM + cc];
      if (col < 0 || f0 + lane >= nf) continue;
      const size_t unit = (size_t)a.col2act[col] * G + g;
      a.G[unit * nf + f0 + lane] = acc[lane][cc];
    }
  }
  if (fc == 0 && tid < TM) {
    const int col = a.tile_cols[(size_t)st.tile * TM + c];
    if (col >= 0) {
      const size_t unit = (size_t)a.col2act[col] * G + g;
      float kept = 0.0f, cand = 0.0f, rs = 0.0f;
      for (int s = 0; s < st.nseg; s++) {
        const float *cc = a.cnt + (((size_t)(st.cblk0 + s) * G + g) * TM + c) * 3;
        kept += cc[0];
        cand += cc[1];
        rs += cc[2];
      }
      a.nkept[unit] = (int)kept;
      if (a.diag_lg_obscount) a.diag_lg_obscount[(size_t)g * a.ncol + col] = kept;
      if (a.diag_lg_obsloc) a.diag_lg_obsloc[(size_t)g * a.ncol + col] = rs;
      if (g == 0 && a.diag_obscount) a.diag_obscount[col] = cand;
    }
  }
}
}  // namespace

cudaError_t launch_gram_segsum(cudaStream_t st, const TcArgs &a, int *launches) {
  if (a.nsegtiles <= 0) return cudaSuccess;
  const long long grid = (long long)a.nsegtiles * a.groups * ((a.nf + 31) / 32);
  if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_gram_segsum<<<(int)grid, SST, 0, st>>>(a);
  (*launches)++;
  return cudaGetLastError();
}

template <int LOC>
static cudaError_t preload_gram_tc_loc() {
  cudaFuncAttributes fa;
  cudaError_t e = cudaSuccess;
  auto get = [&](const void *f) { if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, f); };
  get((const void *)k_gram_tc<LOC, NRMAX, false, false>);
  get((const void *)k_gram_tc<LOC, NRMAX, true, false>);
  get((const void *)k_gram_tc<LOC, NRMAX, false, true>);
  get((const void *)k_gram_tc<LOC, NRMAX, true, true>);
  get((const void *)k_tile_count);
  get((const void *)k_tile_scan);
  get((const void *)k_tile_list);
  get((const void *)k_tile_rec);
  get((const void *)k_gram_segsum);
  return e;
}

// loads the batched Gram's kernels for a localizer class (CUDA loads a
// kernel at its first use, which must not fall inside a timed trial)
cudaError_t preload_gram_tc(int loc_cls) {
  switch (loc_cls) {
  case LOC_OCEAN: return preload_gram_tc_loc<LOC_OCEAN>();
  case LOC_VTGC: return preload_gram_tc_loc<LOC_VTGC>();
  default: return preload_gram_tc_loc<LOC_NOVRT>();
  }
}

}  // namespace lgpu
