// FP64 mode-n product with a cyclic layout rotation: the plain-precision form
// of PUX / PUY / PUZ (source_beta_to_omega/src/calc.c:631-684, one cblas_dgemm
// plus xyz_yzx / yzx_zxy / zxy_xyz).
//
// For each tensor t of a batch, in layout (a fastest, then b, then c):
//   out_t[a' * n*n + c*n + b] = sum_a M[a' * n + a] * in_t[(c*n + b) * n + a]
// i.e. a GEMM C[a'][r] = sum_a M[a'][a] In[r][a] over r = c*n + b, stored with r
// contiguous, so that three successive products return to the original axis
// order with every index transformed.  Epilogues fuse the ETD update
// (ac_updateU_new / ch_updateU_new, calc.c:489-535), the ETD2 phi2 scaling
// (prepare_U2_new, calc.c:553-567) and the corrector accumulation
// (correct_U_new, calc.c:569-583); the prologue fuses prepare_U1_new's
// difference (calc.c:537-551).
//
// GB300 executes FP64 at ~1.2 TFLOP/s (measured), so these kernels are bound by
// FP64 issue, not memory.  Two forms:
//   modeprod_f64_kernel: any basis, 64x64 output tiles, 4x4 outputs per thread;
//   fold_*_f64_kernel:   the parity-folded products of the Dirichlet basis
//                        (sclet_basis.cu), half the multiplications.
#include "sclet_internal.cuh"

namespace sclet {

namespace {
constexpr int BM = 64, BN = 64, BK = 16;

struct Tabs {
  const double *phi[2];  // per kind: phi1 (epilogue 1) or phi2 (epilogue 2), layout [k][j][i]
};

template <int EPI, bool SUB>
__global__ void __launch_bounds__(256) modeprod_f64_kernel(const double *__restrict__ M, const double *__restrict__ in,
                                                           const double *__restrict__ sub, double *__restrict__ out,
                                                           const double *__restrict__ aux, int n, long long in_stride,
                                                           long long out_stride, EtdCoef ec, Tabs tabs) {
  __shared__ double As[BK][BM + 1];
  __shared__ double Bs[BK][BN + 1];
  const int t = blockIdx.z;
  const long long nn = (long long)n * n;
  const int a0 = blockIdx.y * BM;
  const long long r0 = (long long)blockIdx.x * BN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const double *inT = in + t * in_stride;
  const double *subT = SUB ? sub + t * in_stride : nullptr;
  double acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.0;

  for (int k0 = 0; k0 < n; k0 += BK) {
    // M tile: rows a0..a0+63, cols k0..k0+15 -> As[k][a]
    for (int e = threadIdx.x; e < BM * BK; e += 256) {
      int row = e / BK, col = e % BK;
      int a = a0 + row, k = k0 + col;
      As[col][row] = (a < n && k < n) ? M[(long long)a * n + k] : 0.0;
    }
    // In tile: rows r0..r0+63, cols k0..k0+15 -> Bs[k][r]
    for (int e = threadIdx.x; e < BN * BK; e += 256) {
      int row = e / BK, col = e % BK;
      long long r = r0 + row;
      int k = k0 + col;
      double v = 0.0;
      if (r < nn && k < n) {
        v = inT[r * n + k];
        if (SUB) v -= subT[r * n + k];
      }
      Bs[col][row] = v;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; k++) {
      double av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; i++) av[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; j++) bv[j] = Bs[k][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }

  double *outT = out + t * out_stride;
  const int kind = (t % ec.F) >= ec.nac ? 1 : 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    int a = a0 + ty * 4 + i;
    if (a >= n) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      long long r = r0 + tx + 16 * j;
      if (r >= nn) continue;
      long long o = (long long)a * nn + r;
      double v = acc[i][j];
      if (EPI == 0) {
        outT[o] = v;
      } else if (EPI == 1) {
        // ETD1 update in eigenspace at mode (i = r % n, j = r / n, k = a)
        int ii = (int)(r % n), jj = (int)(r / n);
        double tmp, H;
        if (kind == 0) {
          tmp = ec.kk[2] * ec.dd[2][a] + ec.kk[1] * ec.dd[1][jj] + ec.kk[0] * ec.dd[0][ii];
          H = -ec.LE * (tmp * ec.epn2 - ec.KE);
        } else {
          tmp = ec.dd[2][a] + ec.dd[1][jj] + ec.dd[0][ii];
          H = ec.LCI * (tmp * tmp * ec.epn2 - ec.KCI * tmp);
        }
        if (fabs(H) < 1.0e-8) H = 0.0;
        double phi = tabs.phi[kind][o];
        double uh = aux[t * out_stride + o];
        outT[o] = (1.0 - phi * H) * uh + phi * v;
      } else if (EPI == 2) {
        outT[o] = tabs.phi[kind][o] * v;
      } else {
        outT[o] += v;
      }
    }
  }
}
// ---- folded products ---------------------------------------------------------
//
// A warp instruction of FP64 occupies its scheduler for 64 cycles, so shared
// memory, loads and index arithmetic hide behind it and the only cost is the
// number of FP64 instructions: no padded outputs.  A thread owns one input row
// (a line along the contracted axis) and MT outputs of it, MT a compile-time
// count (an output that is only predicated off still costs its 64 cycles)
// chosen so that the tiles of a half divide it evenly (fold_tiles); the matrix
// values are read as shared-memory broadcasts.  The products of a step, dense
// 64 x 64 tiles and nine per field before, folded and (order parameters) six
// per field now: 4 fields of 68^3 3.00 -> 0.62 ms, 4 + 1 fields of 132^3
// 35.1 -> 9.6 ms (7.97 ms of multiplications at the measured rate).
constexpr int FR = 128;     // rows per CTA, one per thread
constexpr int FK = 16;      // contraction indices per shared-memory tile
constexpr int FWD_MAX = 36, FWD_STEP = 2;  // outputs per thread: 8, 10, .. 36 forward
constexpr int INV_MAX = 18, INV_STEP = 1;  // and 4, 5, .. 18 of each parity inverse

// Forward: out[2 m + p] = sum_j W[p][j][m] (x[j] +- x[n-1-j]).  blockIdx.y =
// part x tile of m; the sums x[j] +- x[n-1-j] are formed once per CTA as the
// rows enter shared memory.
template <int MT>
__global__ void __launch_bounds__(FR) fold_fwd_f64_kernel(const double *__restrict__ W, TensorList<double> in,
                                                          const double *__restrict__ sub, double *__restrict__ out,
                                                          int n, int tiles, FoldEpi ep, EtdCoef ec) {
  chain_wait();
  __shared__ double xs[FK][FR + 1];
  __shared__ __align__(16) double ws[FK][MT];
  const int t = blockIdx.z, h = fold_half(n);
  const int part = blockIdx.y >= tiles ? 1 : 0, tile = blockIdx.y - part * tiles;
  const int live = part == 0 ? h : n / 2;  // modes, and block positions, of this parity
  const int step = (h + tiles - 1) / tiles, m0 = tile * step, mt = min(step, live - m0);
  if (mt <= 0) return;
  const long long nn = (long long)n * n, n3 = nn * n;
  const long long r0 = (long long)blockIdx.x * FR;
  const int rows = (int)(nn - r0 < FR ? nn - r0 : FR);
  const double *x = in.at(t, n3) + r0 * n;
  const double *xsub = sub ? sub + t * n3 + r0 * n : nullptr;
  const double *w = W + (size_t)part * h * h + m0;
  double acc[MT];
#pragma unroll
  for (int m = 0; m < MT; m++) acc[m] = 0.0;
  for (int k0 = 0; k0 < live; k0 += FK) {
    const int kc = min(FK, live - k0);
    for (int e = threadIdx.x; e < FK * FR; e += FR) {
      const int r = e / FK, k = e % FK;
      double v = 0.0;
      if (r < rows && k < kc) {
        const int j = k0 + k, q = n - 1 - j;
        double a = x[(long long)r * n + j], b = q != j ? x[(long long)r * n + q] : 0.0;
        if (sub) {
          a -= xsub[(long long)r * n + j];
          if (q != j) b -= xsub[(long long)r * n + q];
        }
        v = part == 0 ? a + b : a - b;
      }
      xs[k][r] = v;
    }
    for (int e = threadIdx.x; e < kc * MT; e += FR) {
      const int k = e / MT, m = e - k * MT;
      ws[k][m] = m < mt ? w[(size_t)(k0 + k) * h + m] : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < kc; k++) {
      const double v = xs[k][threadIdx.x];
#pragma unroll
      for (int m = 0; m < MT; m++) acc[m] = fma(ws[k][m], v, acc[m]);
    }
    __syncthreads();
  }
  if ((int)threadIdx.x >= rows) return;
  const long long r = r0 + threadIdx.x;
  const int f = (t + ep.t0) % ec.F, kind = f >= ec.nac ? 1 : 0;
  double *o = out + t * n3 + r;
  const double *phi = ep.phi[kind];
  const int ii = (int)(r % n), jj = (int)(r / n);  // mode (ii, jj, a) of a z-contraction
#pragma unroll
  for (int m = 0; m < MT; m++)
    if (m < mt) {
      const int a = 2 * (m0 + m) + fold_mode0(n, part);
      const long long at = (long long)a * nn;
      double v = acc[m];
      if (ep.etd) {
        double tmp, H;
        if (kind == 0) {
          tmp = ec.kk[2] * ec.dd[2][a] + ec.kk[1] * ec.dd[1][jj] + ec.kk[0] * ec.dd[0][ii];
          H = -ec.LE * (tmp * ec.epn2 - ec.KE);
        } else {
          tmp = ec.dd[2][a] + ec.dd[1][jj] + ec.dd[0][ii];
          H = ec.LCI * (tmp * tmp * ec.epn2 - ec.KCI * tmp);
        }
        if (fabs(H) < 1.0e-8) H = 0.0;
        const double ph = phi[at + r];
        v = (1.0 - ph * H) * o[at] + ph * v;
      } else if (t < ep.scaled) {
        v = phi[at + r] * v;
      }
      o[at] = v;
    }
}

// Inverse: E[i] = sum_m W[0][m][i] x[2 m + p0], O[i] likewise of the odd modes;
// out[i] = E + O, out[n-1-i] = E - O.  Both parities in one thread.
template <int MI>
__global__ void __launch_bounds__(FR) fold_inv_f64_kernel(const double *__restrict__ W, const double *__restrict__ in,
                                                          double *__restrict__ out, int n, int tiles, int F, int accf) {
  chain_wait();
  __shared__ double xs[2][FK][FR + 1];
  __shared__ __align__(16) double ws[2][FK][MI];
  const int t = blockIdx.z, h = fold_half(n), h1 = n / 2;
  const int step = (h + tiles - 1) / tiles, i0 = (int)blockIdx.y * step, mt = min(step, h - i0);
  if (mt <= 0) return;
  const long long nn = (long long)n * n, n3 = nn * n;
  const long long r0 = (long long)blockIdx.x * FR;
  const int rows = (int)(nn - r0 < FR ? nn - r0 : FR);
  const double *x = in + t * n3 + r0 * n;
  const int p0 = fold_mode0(n, 0);
  double E[MI], O[MI];
#pragma unroll
  for (int i = 0; i < MI; i++) E[i] = O[i] = 0.0;
  for (int k0 = 0; k0 < h; k0 += FK) {
    const int kc = min(FK, h - k0);
    // modes 2 k0 .. 2 k0 + 2 FK - 1 of every row, parities apart
    for (int e = threadIdx.x; e < 2 * FK * FR; e += FR) {
      const int r = e / (2 * FK), q = e % (2 * FK), mode = 2 * k0 + q;
      xs[(q & 1) == p0 ? 0 : 1][q >> 1][r] = r < rows && mode < n ? x[(long long)r * n + mode] : 0.0;
    }
    for (int e = threadIdx.x; e < 2 * kc * MI; e += FR) {
      const int part = e / (kc * MI), g = e - part * kc * MI, k = g / MI, i = g - k * MI;
      // zero where the odd part has no entry
      ws[part][k][i] = i < mt ? W[((size_t)part * h + k0 + k) * h + i0 + i] : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < kc; k++) {
      const double ve = xs[0][k][threadIdx.x], vo = xs[1][k][threadIdx.x];
#pragma unroll
      for (int i = 0; i < MI; i++) {
        E[i] = fma(ws[0][k][i], ve, E[i]);
        O[i] = fma(ws[1][k][i], vo, O[i]);
      }
    }
    __syncthreads();
  }
  if ((int)threadIdx.x >= rows) return;
  double *o = out + t * n3 + r0 + threadIdx.x;
  const bool add = t % F < accf;
#pragma unroll
  for (int i = 0; i < MI; i++)
    if (i < mt) {
      const long long a = (long long)(i0 + i) * nn, b = (long long)(n - 1 - i0 - i) * nn;
      const double s = E[i] + O[i], d = E[i] - O[i];
      o[a] = add ? o[a] + s : s;
      if (i0 + i < h1) o[b] = add ? o[b] + d : d;
    }
}

// Tiles of a half of h outputs, lo .. hi in steps per thread: the count whose
// slowest SM finishes first (CTAs per SM times the FP64 instructions of one
// contraction index, the fold's among them).  per: outputs per thread.
int fold_tiles(int h, int lo, int hi, int step, long long ctas_per_tile, int *per) {
  int best = 0;
  long long cost = 0;
  const int q0 = (h + hi - 1) / hi;
  for (int q = q0; q <= q0 + 6; q++) {
    const int live = (h + q - 1) / q, mt = live <= lo ? lo : lo + (live - lo + step - 1) / step * step;
    const long long c = ((ctas_per_tile * q + 151) / 152) * (mt + 1);
    if (!best || c < cost) best = q, cost = c, *per = mt;
  }
  return best;
}

template <int MT>
void run_fwd(int mt, dim3 grid, cudaStream_t s, const double *W, const TensorList<double> &in, const double *sub,
             double *out, int n, int tiles, const FoldEpi &ep, const EtdCoef &ec) {
  if constexpr (MT <= FWD_MAX) {
    if (mt == MT) chain_launch(false, fold_fwd_f64_kernel<MT>, grid, FR, 0, s, W, in, sub, out, n, tiles, ep, ec);
    else run_fwd<MT + FWD_STEP>(mt, grid, s, W, in, sub, out, n, tiles, ep, ec);
  }
}
template <int MI>
void run_inv(int mi, dim3 grid, cudaStream_t s, const double *W, const double *in, double *out, int n, int tiles, int F,
             int acc) {
  if constexpr (MI <= INV_MAX) {
    if (mi == MI) chain_launch(false, fold_inv_f64_kernel<MI>, grid, FR, 0, s, W, in, out, n, tiles, F, acc);
    else run_inv<MI + INV_STEP>(mi, grid, s, W, in, out, n, tiles, F, acc);
  }
}
}  // namespace

cudaError_t launch_fold_fwd_f64(const double *W, const TensorList<double> &in, const double *sub, double *out, int count,
                                int n, const FoldEpi &ep, const EtdCoef &ec, cudaStream_t s) {
  const long long nn = (long long)n * n, rt = (nn + FR - 1) / FR;
  int mt = 0;
  const int tiles = fold_tiles(fold_half(n), 8, FWD_MAX, FWD_STEP, rt * count * 2, &mt);
  run_fwd<8>(mt, dim3((unsigned)rt, 2 * tiles, count), s, W, in, sub, out, n, tiles, ep, ec);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_fold_inv_f64(const double *W, const double *in, double *out, int count, int n, int F, int acc,
                                cudaStream_t s) {
  const long long nn = (long long)n * n, rt = (nn + FR - 1) / FR;
  int mi = 0;
  const int tiles = fold_tiles(fold_half(n), 4, INV_MAX, INV_STEP, rt * count, &mi);
  run_inv<4>(mi, dim3((unsigned)rt, tiles, count), s, W, in, out, n, tiles, F, acc);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t launch_modeprod_f64(const double *M, const double *in, const double *sub, double *out, const double *aux,
                                int count, int n, int epilogue, const EtdCoef &ec, long long in_stride,
                                long long out_stride, cudaStream_t s, const double *const *phi) {
  long long nn = (long long)n * n;
  dim3 grid((unsigned)((nn + BN - 1) / BN), (unsigned)((n + BM - 1) / BM), (unsigned)count);
  const Tabs tb = {{phi ? phi[0] : nullptr, phi ? phi[1] : nullptr}};
  if (sub) {
    modeprod_f64_kernel<0, true><<<grid, 256, 0, s>>>(M, in, sub, out, aux, n, in_stride, out_stride, ec, tb);
  } else if (epilogue == 0) {
    modeprod_f64_kernel<0, false><<<grid, 256, 0, s>>>(M, in, sub, out, aux, n, in_stride, out_stride, ec, tb);
  } else if (epilogue == 1) {
    modeprod_f64_kernel<1, false><<<grid, 256, 0, s>>>(M, in, sub, out, aux, n, in_stride, out_stride, ec, tb);
  } else if (epilogue == 2) {
    modeprod_f64_kernel<2, false><<<grid, 256, 0, s>>>(M, in, sub, out, aux, n, in_stride, out_stride, ec, tb);
  } else {
    modeprod_f64_kernel<3, false><<<grid, 256, 0, s>>>(M, in, sub, out, aux, n, in_stride, out_stride, ec, tb);
  }
  launch_counter()++;
  return cudaGetLastError();
}

}  // namespace sclet
