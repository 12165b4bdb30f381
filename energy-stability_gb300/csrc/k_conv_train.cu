// Element-wise and reduction kernels of the corrector network: packing FP32 fields into haloed BF16 activations, the BF16 weight copies,
// Adam and the training residual.  Activations in the chunk-planar layout of
// sclet_conv.cuh (conv_at).
#include <cuda_bf16.h>
#include <stdint.h>

#include "sclet_conv.cuh"
#include "sclet_internal.cuh"

namespace sclet {
namespace {

__device__ __forceinline__ int wrap_h(int h, int N) { return 1 + (h - 1 + N) % N; }

// every haloed cell from its periodic image in the planar FP32 input
__global__ void pack_kernel(const float *__restrict__ in, int cin, float scale, int N, int batch,
                            __nv_bfloat16 *__restrict__ a) {
  const int Np = N + 2;
  const long long n3 = (long long)N * N * N, cells = (long long)Np * Np * Np;
  const long long total = cells * batch;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(i / cells);
    long long r = i - (long long)b * cells;
    const int z = (int)(r / ((long long)Np * Np));
    r -= (long long)z * Np * Np;
    const int y = (int)(r / Np), x = (int)(r - (long long)y * Np);
    const long long own = ((long long)(wrap_h(z, N) - 1) * N + (wrap_h(y, N) - 1)) * N + (wrap_h(x, N) - 1);
    const float *src = in + (long long)b * cin * n3 + own;
    uint32_t w[CH / 2];
#pragma unroll
    for (int c = 0; c < CH; c += 2) {
      const float v0 = c < cin ? src[c * n3] * scale : 0.0f;
      const float v1 = c + 1 < cin ? src[(c + 1) * n3] * scale : 0.0f;
      const __nv_bfloat162 p = __floats2bfloat162_rn(v0, v1);
      w[c / 2] = *reinterpret_cast<const uint32_t *>(&p);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(a);
    const long long c0 = conv_at(N, b, z, 0, (long long)y * Np + x), cs = conv_chunk_slots(N);
#pragma unroll
    for (int k = 0; k < 4; k++) dst[c0 + k * cs] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
  }
}

__global__ void relu_mask_kernel(uint4 *__restrict__ g, const uint4 *__restrict__ act, long long chunks) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < chunks; i += (long long)gridDim.x * blockDim.x) {
    uint4 gv = g[i];
    const uint4 av = act[i];
    uint32_t *gw = reinterpret_cast<uint32_t *>(&gv);
    const uint32_t aw[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
    for (int h = 0; h < 4; h++) {
      // a BF16 value is > 0 when its sign bit is clear and it is not zero
      const uint32_t lo = aw[h] & 0xffffu, hi = aw[h] >> 16;
      const uint32_t keep_lo = (lo != 0 && !(lo & 0x8000u)) ? 0xffffu : 0u;
      const uint32_t keep_hi = (hi != 0 && !(hi & 0x8000u)) ? 0xffff0000u : 0u;
      gw[h] &= keep_lo | keep_hi;
    }
    g[i] = gv;
  }
}

__global__ void weights_kernel(const float *__restrict__ w, int layers, __nv_bfloat16 *__restrict__ wf,
                               __nv_bfloat16 *__restrict__ wt) {
  const long long per = (long long)TAPS * CH * CH, total = per * layers;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long l = i / per;
    const int r = (int)(i - l * per);
    const int t = r / (CH * CH), co = (r / CH) % CH, ci = r % CH;
    const __nv_bfloat16 v = __float2bfloat16_rn(w[i]);
    wf[i] = v;
    if (wt) wt[l * per + ((long long)(TAPS - 1 - t) * CH + ci) * CH + co] = v;
  }
}

__global__ void adam_kernel(float *p, float *m, float *v, float *g, long long count, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    g[i] = 0.0f;
  }
}

__global__ void residual_kernel(const float *__restrict__ pred, const float *__restrict__ target, float *__restrict__ r,
                                long long count, double *__restrict__ part) {
  __shared__ double red[256];
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
    const float d = pred[i] - target[i];
    r[i] = d;
    s += (double)d * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

int grid_for(long long total, int block) {
  const long long b = (total + block - 1) / block;
  return (int)(b < 152 * 16 ? (b < 1 ? 1 : b) : 152 * 16);
}

}  // namespace

cudaError_t launch_conv_pack(const float *in, int cin, int N, int batch, __nv_bfloat16 *a, cudaStream_t s) {
  if (cin < 1 || cin > CH) return cudaErrorInvalidValue;
  const long long cells = (long long)(N + 2) * (N + 2) * (N + 2) * batch;
  pack_kernel<<<grid_for(cells, 256), 256, 0, s>>>(in, cin, 1.0f, N, batch, a);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_conv_pack_grad(const float *g, int cout, float scale, int N, int batch, __nv_bfloat16 *a,
                                  cudaStream_t s) {
  if (cout < 1 || cout > CH) return cudaErrorInvalidValue;
  const long long cells = (long long)(N + 2) * (N + 2) * (N + 2) * batch;
  pack_kernel<<<grid_for(cells, 256), 256, 0, s>>>(g, cout, scale, N, batch, a);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_conv_relu_mask(__nv_bfloat16 *g, const __nv_bfloat16 *act, int N, int batch, cudaStream_t s) {
  const long long chunks = conv_units(N, batch);
  relu_mask_kernel<<<grid_for(chunks, 256), 256, 0, s>>>(reinterpret_cast<uint4 *>(g),
                                                          reinterpret_cast<const uint4 *>(act), chunks);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_conv_weights(const float *w, int layers, __nv_bfloat16 *wf, __nv_bfloat16 *wt, cudaStream_t s) {
  weights_kernel<<<grid_for((long long)TAPS * CH * CH * layers, 256), 256, 0, s>>>(w, layers, wf, wt);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_adam(float *p, float *m, float *v, float *g, long long count, float lr, float b1, float b2,
                        float eps, float c1, float c2, cudaStream_t s) {
  adam_kernel<<<grid_for(count, 256), 256, 0, s>>>(p, m, v, g, count, lr, b1, b2, eps, c1, c2);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_residual(const float *pred, const float *target, float *r, long long count, double *part,
                            int nparts, cudaStream_t s) {
  residual_kernel<<<nparts, 256, 0, s>>>(pred, target, r, count, part);
  launch_counter()++;
  return cudaGetLastError();
}

}  // namespace sclet
