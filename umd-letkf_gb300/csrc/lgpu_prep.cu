// lgpu_prep.cu -- the pre-processing immediately upstream of the analysis,
// on the device:
//   src/letkf_obs.F90:459-488   hx_mean = SUM(hx,1)/k, hx' = hx - hx_mean,
//                               then drop qc > 0 observations keeping order
//   src/letkf_state.F90:326-334 mean = SUM(x,1)/k, x' = x - mean,
//                               sprd = SQRT(DOT(x',x')/(k-1))
// Sums run over members in order with explicitly rounded float operations,
// the reference's REAL arithmetic.
#include "lgpu_internal.cuh"

namespace lgpu {

namespace {

// A block's rows of k members pass through shared memory, RS rows at a time:
// read and written whole, in order, while each thread runs along its own row
// (a pitch of an odd number of words: no bank conflicts).  Straight from
// global memory the rows' strides cost a 32-byte sector per value (members of
// 144 x 72 columns x 21 slabs, k = 40: 59 us, now 22).
constexpr int RS = 128;   // rows (threads) per block
__device__ __forceinline__ void rows_in(float *sm, const float *x, long long r0, int n, int k, int pitch) {
  const float *src = x + r0 * k;
#pragma unroll 4
  for (int t = threadIdx.x; t < n * k; t += RS) sm[(t / k) * pitch + t % k] = src[t];
}
__device__ __forceinline__ void rows_out(const float *sm, float *x, long long r0, int n, int k, int pitch) {
  float *dst = x + r0 * k;
#pragma unroll 4
  for (int t = threadIdx.x; t < n * k; t += RS) dst[t] = sm[(t / k) * pitch + t % k];
}

// per observation: member mean and perturbations in place; keep flag
__global__ void __launch_bounds__(RS) k_hx_stats(int nobs, int k, float *hx, float *hx_mean, const int *qc, int *flag) {
  extern __shared__ float rows[];
  const long long r0 = (long long)blockIdx.x * RS;
  const int n = (int)min((long long)RS, nobs - r0), pitch = k | 1;
  rows_in(rows, hx, r0, n, k, pitch);
  __syncthreads();
  if ((int)threadIdx.x < n) {
    float *h = rows + threadIdx.x * pitch;
    const long long o = r0 + threadIdx.x;
    float sum = 0.0f;
    for (int m = 0; m < k; m++) sum = __fadd_rn(sum, h[m]);
    const float mean = __fdiv_rn(sum, (float)k);
    for (int m = 0; m < k; m++) h[m] = __fsub_rn(h[m], mean);
    hx_mean[o] = mean;
    flag[o] = qc ? (qc[o] > 0 ? 0 : 1) : 1;   // obs_def(i)%qc > 0 is dropped
  }
  __syncthreads();
  rows_out(rows, hx, r0, n, k, pitch);
}

// compaction: i -> pos[i] for kept observations (pos[i] <= i, so the
// destination arrays are separate)
__global__ void k_compact(int nobs, int k, const int *flag, const int *pos, const float *const *src_f, float *const *dst_f,
                          int nf, const int *const *src_i, int *const *dst_i, int ni, const float *hx, float *hx_out,
                          const float *hxm, float *hxm_out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nobs * (k + 1)) return;
  const int o = (int)(t / (k + 1)), m = (int)(t % (k + 1));
  if (!flag[o]) return;
  const int p = pos[o];
  if (m < k) {
    hx_out[(size_t)p * k + m] = hx[(size_t)o * k + m];
  } else {
    hxm_out[p] = hxm[o];
    for (int q = 0; q < nf; q++) dst_f[q][p] = src_f[q][o];
    for (int q = 0; q < ni; q++) dst_i[q][p] = src_i[q][o];
  }
}

// per (column, slab): background mean, perturbations in place, spread
__global__ void __launch_bounds__(RS) k_state_stats(long long ncs, int k, float *x, float *mean, float *sprd) {
  extern __shared__ float rows[];
  const long long r0 = (long long)blockIdx.x * RS;
  const int n = (int)min((long long)RS, ncs - r0), pitch = k | 1;
  rows_in(rows, x, r0, n, k, pitch);
  __syncthreads();
  if ((int)threadIdx.x < n) {
    float *v = rows + threadIdx.x * pitch;
    float sum = 0.0f;
    for (int m = 0; m < k; m++) sum = __fadd_rn(sum, v[m]);
    const float mu = __fdiv_rn(sum, (float)k);
    float dot = 0.0f;
    for (int m = 0; m < k; m++) {
      const float p = __fsub_rn(v[m], mu);
      v[m] = p;
      dot = __fadd_rn(dot, __fmul_rn(p, p));
    }
    mean[r0 + threadIdx.x] = mu;
    sprd[r0 + threadIdx.x] = __fsqrt_rn(__fdiv_rn(dot, (float)(k - 1)));
  }
  __syncthreads();
  rows_out(rows, x, r0, n, k, pitch);
}

constexpr size_t rows_bytes(int k) { return (size_t)RS * (k | 1) * sizeof(float); }   // 66 KB at k = 128

}  // namespace

// the exclusive scan of the keep flags into pos[0 .. nobs]
cudaError_t launch_hx_stats(cudaStream_t st, int nobs, int k, float *hx, float *hx_mean, const int *qc, int *flag,
                            int *pos) {
  if (nobs <= 0) return cudaMemsetAsync(pos, 0, sizeof(int), st);
  const cudaError_t e =
      cudaFuncSetAttribute(k_hx_stats, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_bytes(kMaxK));
  if (e != cudaSuccess) return e;
  k_hx_stats<<<(nobs + RS - 1) / RS, RS, rows_bytes(k), st>>>(nobs, k, hx, hx_mean, qc, flag);
  return launch_scan(st, nobs, flag, pos);
}

cudaError_t launch_compact(cudaStream_t st, int nobs, int k, const int *flag, const int *pos, const float *const *src_f,
                           float *const *dst_f, int nf, const int *const *src_i, int *const *dst_i, int ni,
                           const float *hx, float *hx_out, const float *hxm, float *hxm_out) {
  if (nobs <= 0) return cudaSuccess;
  const long long n = (long long)nobs * (k + 1);
  k_compact<<<(int)((n + 255) / 256), 256, 0, st>>>(nobs, k, flag, pos, src_f, dst_f, nf, src_i, dst_i, ni, hx, hx_out,
                                                      hxm, hxm_out);
  return cudaGetLastError();
}

cudaError_t launch_state_stats(cudaStream_t st, long long ncs, int k, float *x, float *mean, float *sprd) {
  if (ncs <= 0) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(k_state_stats, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_bytes(kMaxK));
  if (e != cudaSuccess) return e;
  k_state_stats<<<(int)((ncs + RS - 1) / RS), RS, rows_bytes(k), st>>>(ncs, k, x, mean, sprd);
  return cudaGetLastError();
}

}  // namespace lgpu
