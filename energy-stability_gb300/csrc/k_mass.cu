// Mass of the conserved (Cahn-Hilliard) field in the mixed-precision form.
//
// The ETD step is linear in the pre-step state u and the right-hand side N:
//   u' = V3 (E . V3^-1 u + phi1 . V3^-1 N)   (ch_updateU_new, calc.c:513-535)
// so the mass the FP64 step would give, M(u') = sum over owned cells of u',
// is a fixed linear functional of (u, N):
//   M(u') = <wE, u> + <wP, N>,  wE = V3^-T (G . E),  wP = V3^-T (G . phi1),
// with G = g x g x g and g[p] = sum over owned rows i of V[i][p]; the ETD2
// corrector (correct_U_new, calc.c:569-583) adds <w2, N2 - N1>, w2 from phi2.
// The weights are computed once in FP64 from the FP64 basis and kept as FP32
// (hi, lo) pairs.  Each mixed step forms the target from the stored state with
// error-free FP32 products and sums of up to 256 cells per thread (about 48
// bits, no FP64 instructions per cell) and compensated FP64 sums of these and
// across threads in a fixed order, then shifts the owned cells of the new state
// uniformly so their sum meets it.  The FP32 state itself rounds that sum at the
// level of its own storage (about 1e-11 relative at 192^3).
#include <algorithm>

#include "sclet_internal.cuh"

namespace sclet {

namespace {

constexpr int MB = 256;

__device__ inline void two_sum(double a, double b, double &s, double &e) {
  s = a + b;
  double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
struct Ks {
  double s, c;
  __device__ void add(double v) {
    double t, e;
    two_sum(s, v, t, e);
    s = t;
    c += e;
  }
};

// per-thread running sum as an FP32 pair (s, e): s + e carries about 48 bits
struct Fs {
  float s, e;
  __device__ void add(float v) {  // TwoSum (Knuth)
    const float t = s + v, bp = t - s;
    e += (s - (t - bp)) + (v - bp);
    s = t;
  }
  // w * x for a weight pair w (hi, lo): the hi product exactly (FMA), the small terms rounded
  __device__ void add_product(float2 w, float x) {
    const float p = w.x * x;
    add(p);
    e += fmaf(w.x, x, -p) + w.y * x;
  }
  // w * (b - c): the difference as an exact pair, then the products
  __device__ void add_product_diff(float2 w, float b, float c) {
    const float d = b - c, bp = d - b;
    const float dl = (b - (d - bp)) + (-c - bp);  // TwoSum(b, -c) error
    add_product(w, d);
    e += w.x * dl;
  }
};

// A thread's sum over many cells: FP32 pairs of up to FLUSH_CELLS cells, whose low
// half is plain FP32, collected in an FP64 pair.
constexpr int FLUSH_CELLS = 256;
struct Sum {
  Fs f = {0.0f, 0.0f};
  Ks d = {0.0, 0.0};
  __device__ void flush() {
    d.add((double)f.s);
    d.c += (double)f.e;
    f = Fs{0.0f, 0.0f};
  }
};

// Block-wide sum of the threads' FP64 pairs (compensated throughout), by one warp
// through shared memory: eight threads a lane, then the lanes.  Lane 0 of that
// warp receives the pair, normalised, and `true`.  Bound by FP64 instructions, 64
// cycles of a scheduler each: 100 of one warp instead of 320 of a butterfly in
// every warp; the warp changes from block to block, so that the four blocks of
// an SM use its four schedulers.  (FP32 pairs merged by butterflies and kept for
// all of a thread's cells: target and correction of a 196^3 block 28 + 40 us for
// now 30 + 44, and at 516^3 an error of 1.2e-16 of the terms' sum for 0.5e-17.)
__device__ bool block_reduce(Sum v, Ks &r) {
  __shared__ double2 sp[MB];
  v.flush();
  sp[threadIdx.x] = make_double2(v.d.s, v.d.c);
  __syncthreads();
  if ((int)(threadIdx.x >> 5) != (int)(blockIdx.x * 4LL / gridDim.x)) return false;
  const int lane = threadIdx.x & 31;
  Ks k = {sp[lane].x, sp[lane].y};
#pragma unroll
  for (int w = 1; w < MB / 32; w++) {
    const double2 o = sp[w * 32 + lane];
    k.add(o.x);
    k.c += o.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double os = __shfl_xor_sync(0xffffffffu, k.s, off), oc = __shfl_xor_sync(0xffffffffu, k.c, off);
    k.add(os);
    k.c += oc;
  }
  two_sum(k.s, k.c, r.s, r.c);
  return lane == 0;
}

// X[k][j][i] = g[i] g[j] g[k] * coefficient of CH eigen-mode (i, j, k):
// which 0: E = 1 - phi1 H, 1: phi1, 2: phi2 (same FP64 arithmetic as the
// coefficient tables of the mixed form).
__global__ void seed_kernel(double *X, const double *g, int n, int which, const double *dx, const double *dy,
                            const double *dz, double epn2, double dt, double L, double K) {
  const long long n3 = (long long)n * n * n;
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n3; o += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(o % n), j = (int)((o / n) % n), k = (int)(o / ((long long)n * n));
    const double tmp = dz[k] + dy[j] + dx[i];
    const double H = L * (tmp * tmp * epn2 - K * tmp);
    double p1, p2;
    if (fabs(H) > 1.0e-8) {
      p1 = -expm1(-dt * H) / H;
      p2 = (1.0 - p1 / dt) / H;
    } else {
      p1 = dt;
      p2 = dt / 2;
    }
    const double Hu = fabs(H) < 1.0e-8 ? 0.0 : H;
    const double c = which == 0 ? 1.0 - p1 * Hu : (which == 1 ? p1 : p2);
    X[o] = g[i] * g[j] * g[k] * c;
  }
}

// Partial target per block: sum of wa*a (or of a over owned cells when wa is
// null) plus sum of wb*(b - bsub).  Each thread takes cells a grid apart, four
// at a time (their loads are in flight together).
__global__ void __launch_bounds__(MB) target_kernel(const float *__restrict__ a, const float2 *__restrict__ wa,
                                                    const float *__restrict__ b, const float *__restrict__ bsub,
                                                    const float2 *__restrict__ wb, int n, double *__restrict__ part) {
  chain_wait();
  constexpr int U = 4;
  const long long n3 = (long long)n * n * n, stride = (long long)gridDim.x * MB;
  Sum sum;
  Fs &acc = sum.f;
  int cells = 0;
  for (long long l0 = blockIdx.x * (long long)MB + threadIdx.x; l0 < n3; l0 += U * stride) {
    float va[U], vb[U], vs[U];
    float2 pa[U], pb[U];
#pragma unroll
    for (int k = 0; k < U; k++) {
      const long long l = l0 + k * stride;
      const bool in = l < n3;
      va[k] = in ? a[l] : 0.0f;
      vb[k] = in ? b[l] : 0.0f;
      pb[k] = in ? wb[l] : make_float2(0.0f, 0.0f);
      vs[k] = in && bsub ? bsub[l] : 0.0f;
      pa[k] = in && wa ? wa[l] : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int k = 0; k < U; k++) {
      if (wa) {
        acc.add_product(pa[k], va[k]);
      } else {
        const long long l = l0 + k * stride;
        const int row = (int)(l / n), x = (int)(l - (long long)row * n), z = row / n, y = row - z * n;
        if (l < n3 && x >= 2 && x < n - 2 && y >= 2 && y < n - 2 && z >= 2 && z < n - 2) acc.add(va[k]);
      }
      if (bsub) acc.add_product_diff(pb[k], vb[k], vs[k]);
      else acc.add_product(pb[k], vb[k]);
    }
    if ((cells += U) % FLUSH_CELLS == 0) sum.flush();
  }
  Ks r;
  if (block_reduce(sum, r)) {
    part[2 * blockIdx.x] = r.s;
    part[2 * blockIdx.x + 1] = r.c;
  }
}

// f(first cell, N, lane) for every owned row (z, y), a warp each
template <typename F>
__device__ __forceinline__ void owned_rows(int n, F &&f) {
  const int N = n - 4, lane = threadIdx.x & 31;
  const int warps = gridDim.x * (MB / 32);
  for (int row = blockIdx.x * (MB / 32) + (threadIdx.x >> 5); row < N * N; row += warps) {
    const int zz = row / N, y = 2 + row - zz * N, z = 2 + zz;
    f(((size_t)z * n + y) * n + 2, N, lane);
  }
}

// Partial owned-cell sum of u per block.
__global__ void __launch_bounds__(MB) owned_sum_kernel(const float *__restrict__ u, int n, double *__restrict__ part) {
  chain_wait();
  Sum sum;
  int rows = 0;
  owned_rows(n, [&](size_t l0, int N, int lane) {
    for (int x0 = lane; x0 < N; x0 += 128) {
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = x0 + 32 * k < N ? u[l0 + x0 + 32 * k] : 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++) sum.f.add(v[k]);
    }
    if (++rows % 16 == 0) sum.flush();  // 256 cells of rows of 512
  });
  Ks r;
  if (block_reduce(sum, r)) {
    part[2 * blockIdx.x] = r.s;
    part[2 * blockIdx.x + 1] = r.c;
  }
}

// Fields that are no increments leave the three inverse products as their parts
// even and odd along each axis: E at positions p < h, O at n - 1 - p, of every
// axis (the products being linear, a part's lines go through the next product
// like any others).  Here the eight parts of a cell and its mirrors are added, as
// pairs (TwoSum), so that the state is rounded once, as after dense sums, and
// each product's sums once.  Added in every product's epilogue instead, E, O and
// their sum rounded each time and with a rounded update of the modes, the
// conserved field's update was 1.18 times as far off as with dense sums; now 0.95.
// In place: a thread has all eight places of its cells.  part (may be null): the
// partial sums of the new owned cells, in the place of owned_sum_kernel.  Bound by
// HBM, 8 B a cell.  A step of 4 + 1 fields of 68^3, 196^3 and 516^3, before and with
// it (elastic stage apart): 184.6 and 184.7 us, 1.538 and 1.547 ms, 32.2 and 32.5 ms.
__global__ void __launch_bounds__(MB) unfold_kernel(float *__restrict__ u, int n, long long stride,
                                                    double *__restrict__ part) {
  chain_wait();
  const int h = fold_half(n);
  u += blockIdx.y * stride;
  Sum sum;
  int cells = 0;
  for (uint32_t i = blockIdx.x * MB + threadIdx.x; i < (uint32_t)h * h * h; i += gridDim.x * MB) {
    const int zy = i / h, x = i - zy * h, z = zy / h, y = zy - z * h;
    const int mx = n - 1 - x, my = n - 1 - y, mz = n - 1 - z;
    // bit 0, 1, 2: the mirror along x, y, z; an odd block's middle has none
    auto at = [&](int b) { return ((long long)(b & 4 ? mz : z) * n + (b & 2 ? my : y)) * n + (b & 1 ? mx : x); };
    const int none = (mx == x ? 1 : 0) | (my == y ? 2 : 0) | (mz == z ? 4 : 0);
    float v[8], e[8];
#pragma unroll
    for (int b = 0; b < 8; b++) {
      v[b] = b & none ? 0.0f : u[at(b)];
      e[b] = 0.0f;
    }
#pragma unroll
    for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
      for (int b = 0; b < 8; b++)
        if (!(b & bit)) {
          const float a = v[b], o = v[b | bit], ea = e[b], eo = e[b | bit];
          const float p = a + o, pb = p - a, q = a - o, qb = q - a;
          v[b] = p;
          e[b] = ((a - (p - pb)) + (o - pb)) + (ea + eo);
          v[b | bit] = q;
          e[b | bit] = ((a - (q - qb)) - (o + qb)) + (ea - eo);
        }
    const bool owned = x >= 2 && y >= 2 && z >= 2;  // the mirrors with it
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (!(b & none)) {
        const float w = v[b] + e[b];
        u[at(b)] = w;
        if (part && owned) sum.f.add(w);
      }
    if ((cells += 8) % FLUSH_CELLS == 0 && part) sum.flush();
  }
  Ks r;
  if (part && block_reduce(sum, r)) {
    part[2 * blockIdx.x] = r.s;
    part[2 * blockIdx.x + 1] = r.c;
  }
}

// One block folds both partial sets in a fixed order, half of its warps each,
// and records (target, before, shift) in res.  Bound by FP64 instructions: few
// warps, a pair's low half (2^-53 of the high one) added plainly.
constexpr int FB = 128;  // threads per set
__global__ void __launch_bounds__(2 * FB) fold_kernel(int n, const double *__restrict__ tpart,
                                                      const double *__restrict__ apart, int np,
                                                      double *__restrict__ res) {
  chain_wait();
  __shared__ double2 sw[2 * FB / 32];
  const int set = threadIdx.x / FB, i = threadIdx.x % FB;
  const double2 *part = reinterpret_cast<const double2 *>(set ? apart : tpart);
  Ks acc = {0.0, 0.0};
  for (int q = i; q < np; q += FB) {
    const double2 v = part[q];
    acc.add(v.x);
    acc.c += v.y;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double os = __shfl_xor_sync(0xffffffffu, acc.s, off), oc = __shfl_xor_sync(0xffffffffu, acc.c, off);
    acc.add(os);
    acc.c += oc;
  }
  if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = make_double2(acc.s, acc.c);
  __syncthreads();
  if (threadIdx.x == 0) {
    double v[2];
    for (int k = 0; k < 2; k++) {
      Ks t = {0.0, 0.0};
      for (int w = 0; w < FB / 32; w++) {
        t.add(sw[k * (FB / 32) + w].x);
        t.c += sw[k * (FB / 32) + w].y;
      }
      v[k] = t.s + t.c;
    }
    const double N = n - 4;
    res[0] = v[0];
    res[1] = v[1];
    res[2] = (v[0] - v[1]) / (N * N * N);
  }
}

// the uniform shift res[2] on the owned cells
__global__ void __launch_bounds__(MB) shift_kernel(float *__restrict__ u, int n, const double *__restrict__ res) {
  chain_wait();
  const float d = (float)res[2];
  owned_rows(n, [&](size_t l0, int N, int lane) {
    for (int x0 = lane; x0 < N; x0 += 128) {
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = x0 + 32 * k < N ? u[l0 + x0 + 32 * k] : 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (x0 + 32 * k < N) u[l0 + x0 + 32 * k] = v[k] + d;
    }
  });
}

// FP64 weights -> FP32 (hi, lo) pairs in place
__global__ void to_pairs_kernel(double *w, long long count) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
    const double v = w[i];
    const float hi = (float)v;
    reinterpret_cast<float2 *>(w)[i] = make_float2(hi, (float)(v - (double)hi));
  }
}

}  // namespace

// Four blocks per SM, each thread with four cells in flight.  (Sixteen blocks per
// SM spent their time in their reductions and left 2432 pairs for the one block
// that folds them: target, and sum, fold and shift, of a 196^3 block 45 and 90 us,
// now 30 and 44.)
int mass_partials() { return 152 * 4; }

cudaError_t mass_weight(double *w, double *tmp, const double *g, const double *viT, int n, int which, const EtdCoef &ec,
                        cudaStream_t s, bool folded) {
  const long long n3 = (long long)n * n * n;
  long long b = (n3 + 255) / 256;
  seed_kernel<<<(int)(b > 152 * 16 ? 152 * 16 : b), 256, 0, s>>>(w, g, n, which, ec.dd[0], ec.dd[1], ec.dd[2], ec.epn2,
                                                                 ec.dt, ec.LCI, ec.KCI);
  launch_counter()++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // three products with V^-T return to the [k][j][i] layout
  auto product = [&](const double *in, double *out) {
    return folded ? launch_fold_inv_f64(viT, in, out, 1, n, 1, 0, s)
                  : launch_modeprod_f64(viT, in, nullptr, out, nullptr, 1, n, 0, ec, n3, n3, s);
  };
  if ((e = product(w, tmp)) != cudaSuccess) return e;
  if ((e = product(tmp, w)) != cudaSuccess) return e;
  if ((e = product(w, tmp)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(w, tmp, sizeof(double) * n3, cudaMemcpyDeviceToDevice, s)) != cudaSuccess) return e;
  to_pairs_kernel<<<(int)(b > 152 * 16 ? 152 * 16 : b), 256, 0, s>>>(w, n3);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t mass_target(const float *a, const double *wa, const float *b, const float *bsub, const double *wb, int n,
                        double *part, cudaStream_t s) {
  chain_launch(false, target_kernel, mass_partials(), MB, 0, s, a, reinterpret_cast<const float2 *>(wa), b, bsub,
                                                reinterpret_cast<const float2 *>(wb), n, part);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t mass_shift(float *u, int n, const double *tpart, const double *apart, double *res, cudaStream_t s) {
  chain_launch(true, fold_kernel, 1, 2 * FB, 0, s, n, tpart, apart, mass_partials(), res);
  chain_launch(false, shift_kernel, mass_partials() * 2, MB, 0, s, u, n, res);
  launch_counter() += 2;
  return cudaGetLastError();
}

cudaError_t mass_fix(float *u, int n, const double *tpart, double *apart, double *res, cudaStream_t s) {
  chain_launch(false, owned_sum_kernel, mass_partials(), MB, 0, s, u, n, apart);
  launch_counter()++;
  return mass_shift(u, n, tpart, apart, res, s);
}

cudaError_t launch_unfold(float *u, int n, int count, long long stride, double *apart, cudaStream_t s) {
  if (apart && count != 1) return cudaErrorInvalidValue;
  const int h = fold_half(n), full = mass_partials();
  const int ctas = apart ? full : (int)std::min<long long>(full, ((long long)h * h * h + MB - 1) / MB);
  for (int b = 0; b < count; b += 65535) {  // the grid's y extent
    chain_launch(false, unfold_kernel, dim3(ctas, std::min(65535, count - b)), MB, 0, s, u + b * stride, n, stride, apart);
    launch_counter()++;
  }
  return cudaGetLastError();
}

}  // namespace sclet
