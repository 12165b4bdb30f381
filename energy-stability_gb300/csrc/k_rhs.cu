// Nonlinear right-hand sides of the ETD step on one periodic block.
//
// Allen-Cahn (ac_calc_FU, source_beta_to_omega/src/calc.c:8-68 ->
// ac_calc_F1 / ac_calc_F2, anisotropic.c:9-628):
//   N_m = LE KE eta_m - LE AC_f(m)                 (SWTICH_AC_FIELD1)
//       + LE epn2 eta_m(outside) / h^2 on each block face (boundary lifting;
//         the outside value is the periodic image of the cell beyond the face)
//       - epn2 LE div(lambda_m grad eta_m)          (ANISOTROPIC; central
//         differences, values outside the block taken as zero)
//       - LE ElasticScale felas_m                  (ELASTIC == 1)
// Cahn-Hilliard, constant mobility (ch_calc_FU_ConstantMobility,
// calc.c:70-473):
//   t   = -LCI KCI c + LCI CH_f - LCI epn2 c(outside) / h^2 on faces
//   N_c = lap(t) (zero outside) - mu(outside) / h^2 on faces, with
//   mu = LCI (epn2 lap(c) - CH_f) at the periodic image of the outside cell
//   (ch_mu, trans.c:1433-1937).
// AC_f and CH_f come from the run's physics plugin (the drop-in form of
// formula.c:9-56, sclet_physics.cuh), a template parameter of every kernel.
#include <algorithm>
#include <type_traits>

#include "sclet_internal.cuh"
#include "sclet_physics.cuh"

namespace sclet {


template <typename T>
struct P {
  int n, nac, nch, F, aniso, elastic;
  T epn2, hx, hy, hz, LE, KE, LCI, KCI, es;
  T ih2x, ih2y, ih2z;   // 1 / h^2 per axis
  T i2hx, i2hy, i2hz;   // 1 / (2 h) per axis
  T K[16];              // plugin constants (reference composition shifted by cshift)
  int zc, runs;         // z-planes per CTA; runs side by side
  const double *krun;   // per-run plugin constant 0, or null
  // anisotropic term folded: kan[m][3 r + c] = epn2 LE (1/2h_r) lam_m[r][c] (1/2h_c),
  // the flux row r differenced along axis r
  T kan[4][9];
  T mob_m0, mob_dg;     // variable mobility M(eta0) = m0 (1 (1 - eta0) + dg eta0)
};

template <typename T>
static P<T> to_p(const Phys &ph) {
  P<T> p;
  p.n = ph.n; p.nac = ph.nac; p.nch = ph.nch; p.F = ph.F; p.aniso = ph.anisotropic; p.elastic = ph.elastic;
  p.epn2 = (T)ph.epn2; p.hx = (T)ph.h[0]; p.hy = (T)ph.h[1]; p.hz = (T)ph.h[2];
  p.ih2x = (T)(1.0 / (ph.h[0] * ph.h[0])); p.ih2y = (T)(1.0 / (ph.h[1] * ph.h[1]));
  p.ih2z = (T)(1.0 / (ph.h[2] * ph.h[2]));
  p.i2hx = (T)(0.5 / ph.h[0]); p.i2hy = (T)(0.5 / ph.h[1]); p.i2hz = (T)(0.5 / ph.h[2]);
  p.LE = (T)ph.LE; p.KE = (T)ph.KE; p.LCI = (T)ph.LCI; p.KCI = (T)ph.KCI; p.es = (T)ph.elastic_scale;
  for (int k = 0; k < 16; k++) p.K[k] = (T)ph.K[k];
  p.zc = ph.rhs_zc;
  p.runs = ph.runs > 0 ? ph.runs : 1;
  p.krun = ph.krun;
  const double i2h[3] = {0.5 / ph.h[0], 0.5 / ph.h[1], 0.5 / ph.h[2]};
  for (int m = 0; m < 4; m++)
    for (int k = 0; k < 9; k++) {
      p.kan[m][k] = (T)(ph.epn2 * ph.LE * i2h[k / 3] * ph.lam[m][k] * i2h[k % 3]);
    }
  p.mob_m0 = (T)ph.mob_m0;
  p.mob_dg = (T)ph.mob_dg;
  return p;
}

// AC_f(m) / CH_f(0) of plugin PL at one cell: NAC order parameters e (known
// at compile time) and the stored concentration c.
template <typename PL, typename T, int NAC>
__device__ __forceinline__ T ac_f_n(const P<T> &p, const T *e, T c, int m) {
  sclet_acv<T> ac[NAC > 0 ? NAC : 1];
  sclet_chv<T> ch[1];
#pragma unroll
  for (int k = 0; k < NAC; k++) ac[k].u = e[k];
  ch[0].c = c;
  return PL::template ac_f<T>(ac, ch, NAC, p.nch, p.K, m);
}

template <typename PL, typename T>
__device__ __forceinline__ T ch_f(const P<T> &p, const T *e, T c) {
  sclet_acv<T> ac[4];
  sclet_chv<T> ch[1];
#pragma unroll
  for (int k = 0; k < 4; k++) ac[k].u = e[k];
  ch[0].c = c;
  return PL::template ch_f<T>(ac, ch, p.nac, 1, p.K, 0);
}

__device__ inline long long L3(int n, int z, int y, int x) { return ((long long)z * n + y) * n + x; }

// img() for v in -1 .. n: one wrap, no division
__device__ __forceinline__ int img1(int n, int v) {
  const int N = n - 4;
  int r = v - 2;
  r += r < 0 ? N : 0;
  r -= r >= N ? N : 0;
  return 2 + r;
}

// The cells on the block's six faces, z faces first: s in 0 .. face_cells(n) - 1.
__host__ __device__ inline int face_cells(int n) { return 2 * n * n + 2 * n * (n - 2) + 2 * (n - 2) * (n - 2); }
__device__ __forceinline__ void face_cell(int n, int s, int &z, int &y, int &x) {
  const int nn = n * n, i = n - 2;
  if (s < 2 * nn) {
    z = s < nn ? 0 : n - 1;
    const int r = s < nn ? s : s - nn;
    y = r / n;
    x = r - y * n;
    return;
  }
  s -= 2 * nn;
  if (s < 2 * n * i) {
    const int q = s / n;  // row: z, then the two y faces
    x = s - q * n;
    z = 1 + (q >> 1);
    y = (q & 1) ? n - 1 : 0;
    return;
  }
  s -= 2 * n * i;
  const int q = s >> 1;
  x = (s & 1) ? n - 1 : 0;
  z = 1 + q / i;
  y = 1 + q % i;
}

// threadIdx.x along x (coalesced), threadIdx.y along y
constexpr int RX = 32, RY = 8;

// ---- Allen-Cahn, no stencil or a diagonal one ------------------------------
// Without the anisotropic term a cell needs its own values only; with a
// diagonal lambda (the usual case: diag(kk) - diag file) it needs the cells two
// away along each axis.  Either way no plane has to be shared: a thread owns an
// (x, y) column, keeps the five z-values of each order parameter in registers
// as it marches, and takes x +- 2 and y +- 2 through L1.  The face cells, whose
// boundary lifting reads far images and would stall whole warps of the march,
// are computed apart by the launch's last CTAs (one cell per thread).
// Bound by the FP32 issue and L1 (FP64: the FP64 pipe).  Before, every case
// took the five-plane shared-memory ring below with the lifting inside; all
// right-hand sides of a step, then and now: 4 fields of 36^3, FP32, no tensor
// 103 -> 8 us; 4 + 1 fields of 196^3, diagonal tensors 525 -> 197 us, of 516^3
// 5.74 -> 2.89 ms; 4 fields of 68^3 in FP64 303 -> 47 us.
template <typename PL, typename T, int NAC, bool DIAG>
__global__ void __launch_bounds__(RX * RY, (sizeof(T) == 4 ? 4 : 2) + (DIAG ? 0 : 1))
    rhs_ac_diag_kernel(P<T> p0, const T *__restrict__ u, const T *__restrict__ felas, T *__restrict__ out, int zblocks) {
  chain_wait();
  const int n = p0.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  P<T> p = p0;
  const bool el = p.elastic == 1, has_c = p.nch > 0;
  if ((int)blockIdx.z < zblocks) {
    const int zchunks = (n + p.zc - 1) / p.zc;
    const int run = blockIdx.z / zchunks, zci = blockIdx.z - run * zchunks;
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    u += (size_t)run * p.F * n3;
    felas += (size_t)run * NAC * n3;
    out += (size_t)run * p.F * n3;
    const int c0 = blockIdx.x * (RX * RY) + threadIdx.x, m2 = n - 2;  // cell of the interior plane
    if (c0 >= m2 * m2) return;
    const int y = c0 / m2 + 1, x = c0 - (y - 1) * m2 + 1;
    const int z0 = max(1, zci * p.zc), z1 = min(n - 1, (zci + 1) * p.zc);
    if (z0 >= z1) return;
    size_t l = (size_t)z0 * nn + (size_t)y * n + x;
    T w[NAC][5];  // planes z - 2 .. z + 2
    if (DIAG) {
#pragma unroll
      for (int m = 0; m < NAC; m++) {
        const T *um = u + m * n3 + l;
        w[m][1] = z0 > 1 ? um[-2 * (long long)nn] : (T)0;
        w[m][2] = um[-(long long)nn];
        w[m][3] = um[0];
        w[m][4] = um[nn];
      }
    }
    for (int z = z0; z < z1; z++, l += nn) {
      T e[NAC], xm[NAC], xp[NAC], ym[NAC], yp[NAC], fe[NAC];
#pragma unroll
      for (int m = 0; m < NAC; m++) {
        const T *um = u + m * n3 + l;
        if (DIAG) {
#pragma unroll
          for (int k = 0; k < 4; k++) w[m][k] = w[m][k + 1];
          w[m][4] = z < n - 2 ? um[2 * nn] : (T)0;
          e[m] = w[m][2];
          xm[m] = x > 1 ? um[-2] : (T)0;
          xp[m] = x < n - 2 ? um[2] : (T)0;
          ym[m] = y > 1 ? um[-2 * n] : (T)0;
          yp[m] = y < n - 2 ? um[2 * n] : (T)0;
        } else {
          e[m] = um[0];
        }
        fe[m] = el ? felas[m * n3 + l] : (T)0;
      }
      const T c = has_c ? u[NAC * n3 + l] : (T)0;
#pragma unroll
      for (int m = 0; m < NAC; m++) {
        T v = p.LE * p.KE * e[m];
        v -= p.LE * ac_f_n<PL, T, NAC>(p, e, c, m);
        if (DIAG) {
          const T *k = p.kan[m];
          const T ar = k[0] * (xp[m] - e[m]), al = k[0] * (e[m] - xm[m]);
          const T at = k[4] * (ym[m] - e[m]), ab = k[4] * (e[m] - yp[m]);
          const T af = k[8] * (w[m][0] - e[m]), ak = k[8] * (e[m] - w[m][4]);
          v -= ((ar - al) + (at - ab)) + (af - ak);
        }
        if (el) v -= p.LE * p.es * fe[m];
        out[m * n3 + l] = v;
      }
    }
    return;
  }
  // face cells of every run
  const int per = face_cells(n), total = per * p.runs;
  const int stride = (int)(gridDim.z - zblocks) * gridDim.x * (RX * RY);
  for (int i = (((int)blockIdx.z - zblocks) * gridDim.x + blockIdx.x) * (RX * RY) + threadIdx.x; i < total; i += stride) {
    const int run = i / per;
    int z, y, x;
    face_cell(n, i - run * per, z, y, x);
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    const T *ur = u + (size_t)run * p.F * n3;
    const size_t l = (size_t)z * nn + (size_t)y * n + x;
    const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
    T e[NAC], lift[NAC];
#pragma unroll
    for (int m = 0; m < NAC; m++) {
      e[m] = ur[m * n3 + l];
      lift[m] = (T)0;
    }
    const T c = has_c ? ur[NAC * n3 + l] : (T)0;
    // per face the cell lies on: the cell beyond it, at its periodic image
    auto add = [&](size_t q, T ih2) {
#pragma unroll
      for (int m = 0; m < NAC; m++) lift[m] += p.LE * p.epn2 * ur[m * n3 + q] * ih2;
    };
    if (x == 0) add(L3(n, iz, iy, lo), p.ih2x);
    if (x == n - 1) add(L3(n, iz, iy, hi), p.ih2x);
    if (y == 0) add(L3(n, iz, lo, ix), p.ih2y);
    if (y == n - 1) add(L3(n, iz, hi, ix), p.ih2y);
    if (z == 0) add(L3(n, lo, iy, ix), p.ih2z);
    if (z == n - 1) add(L3(n, hi, iy, ix), p.ih2z);
#pragma unroll
    for (int m = 0; m < NAC; m++) {
      T v = p.LE * p.KE * e[m];
      v -= p.LE * ac_f_n<PL, T, NAC>(p, e, c, m);
      v += lift[m];
      if (DIAG) {
        const T *um = ur + m * n3 + l, *k = p.kan[m];
        // a flux is zero outside the block, a value outside it too
        const T ar = x < n - 1 ? k[0] * ((x < n - 2 ? um[2] : (T)0) - e[m]) : (T)0;
        const T al = x > 0 ? k[0] * (e[m] - (x > 1 ? um[-2] : (T)0)) : (T)0;
        const T at = y > 0 ? k[4] * ((y > 1 ? um[-2 * n] : (T)0) - e[m]) : (T)0;
        const T ab = y < n - 1 ? k[4] * (e[m] - (y < n - 2 ? um[2 * n] : (T)0)) : (T)0;
        const T af = z > 0 ? k[8] * ((z > 1 ? um[-2 * (long long)nn] : (T)0) - e[m]) : (T)0;
        const T ak = z < n - 1 ? k[8] * (e[m] - (z < n - 2 ? um[2 * nn] : (T)0)) : (T)0;
        v -= ((ar - al) + (at - ab)) + (af - ak);
      }
      if (el) v -= p.LE * p.es * felas[((size_t)run * NAC + m) * n3 + l];
      out[((size_t)run * p.F + m) * n3 + l] = v;
    }
  }
}

// ---- Allen-Cahn, full gradient tensors ---------------------------------------
// 2.5-D: a CTA owns a 32 x 8 (x, y) tile and
// marches over p.zc planes in z, keeping for every order parameter a ring of five
// planes (z-2 .. z+2) with a two-cell halo in x and y in shared memory (zero
// outside the block, as ac_calc_F2 reads it).  Each value comes from global
// memory about once per CTA instead of once per stencil tap.
constexpr int HX = RX + 4, HY = RY + 4;
constexpr int PLANE = HX * HY;     // one haloed plane

template <typename PL, typename T, int NAC>
__global__ void __launch_bounds__(RX * RY, sizeof(T) == 4 ? 3 : 1) rhs_ac_kernel(P<T> p0, const T *__restrict__ u, const T *__restrict__ felas,
                                                         T *__restrict__ out) {
  chain_wait();
  extern __shared__ unsigned char smem_raw[];
  T *ring = reinterpret_cast<T *>(smem_raw);  // [nac][5][HY][HX]
  const int n = p0.n;
  const size_t n3 = (size_t)n * n * n;
  // blockIdx.z = run x z-chunks
  const int zchunks = (n + p0.zc - 1) / p0.zc;
  const int run = blockIdx.z / zchunks, zci = blockIdx.z - run * zchunks;
  P<T> p = p0;
  if (p0.krun) p.K[0] = (T)p0.krun[run];
  u += (size_t)run * p.F * n3;
  felas += (size_t)run * p.nac * n3;
  out += (size_t)run * p.F * n3;
  const int x0 = blockIdx.x * RX, y0 = blockIdx.y * RY;
  const int zb = zci * p.zc, ze = zb + p.zc < n ? zb + p.zc : n;
  const int tid = threadIdx.y * RX + threadIdx.x;
  const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
  // this thread's share of one haloed plane of every order parameter:
  // PLANE / 256 rounded up values per field
  constexpr int PER = (PLANE + RX * RY - 1) / (RX * RY);
  // this thread's cells of a haloed plane: in-plane offset, or -1 outside the block
  int poff[PER];
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int i = tid + q * RX * RY;
    const int ly = i / HX, lx = i - ly * HX;
    const int gx = x0 + lx - 2, gy = y0 + ly - 2;
    poff[q] = i < PLANE && gx >= 0 && gx < n && gy >= 0 && gy < n ? gy * n + gx : -1;
  }
  auto fetch = [&](int z, T *reg) {
    const bool zin = z >= 0 && z < n;
#pragma unroll
    for (int m = 0; m < NAC; m++) {
      const T *um = u + m * n3 + (size_t)z * n * n;
#pragma unroll
      for (int q = 0; q < PER; q++) reg[m * PER + q] = zin && poff[q] >= 0 ? um[poff[q]] : (T)0;
    }
  };
  auto store = [&](int z, const T *reg) {
#pragma unroll
    for (int m = 0; m < NAC; m++) {
      T *dst = ring + (size_t)m * 5 * PLANE + ((z + 5 * 1024) % 5) * PLANE;
#pragma unroll
      for (int q = 0; q < PER; q++) {
        const int i = tid + q * RX * RY;
        if (i < PLANE) dst[i] = reg[m * PER + q];
      }
    }
  };
  T pre[NAC * PER];
  for (int z = zb - 2; z < zb + 2; z++) {
    fetch(z, pre);
    store(z, pre);
  }
  fetch(zb + 2, pre);  // plane z + 2 of the first pass, in flight
  const int lx = threadIdx.x + 2, ly = threadIdx.y + 2;
  for (int z = zb; z < ze; z++) {
    store(z + 2, pre);
    __syncthreads();
    if (z + 3 < ze + 2) fetch(z + 3, pre);  // next plane loads overlap this plane's work
    if (x < n && y < n) {
      const size_t l = ((size_t)z * n + y) * n + x;
      // ring slots of planes z-2 .. z+2, with this thread's (ly, lx) applied
      int so[5];
      const int s0 = (z - 2 + 5 * 1024) % 5;
#pragma unroll
      for (int d = 0; d < 5; d++) so[d] = (s0 + d < 5 ? s0 + d : s0 + d - 5) * PLANE + ly * HX + lx;
      T e[NAC];
#pragma unroll
      for (int m = 0; m < NAC; m++) e[m] = ring[(size_t)m * 5 * PLANE + so[2]];
      const T c = p.nch > 0 ? u[p.nac * n3 + l] : (T)0;
      const bool face = x == 0 || x == n - 1 || y == 0 || y == n - 1 || z == 0 || z == n - 1;
#pragma unroll
      for (int m = 0; m < NAC; m++) {
        const T *um = u + m * n3;
        const T *rg = ring + (size_t)m * 5 * PLANE;
        T v = p.LE * p.KE * e[m];
        v -= p.LE * ac_f_n<PL, T, NAC>(p, e, c, m);
        if (face) {
          const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
          const T w = p.LE * p.epn2;
          if (x == 0) v += w * um[L3(n, iz, iy, lo)] * p.ih2x;
          if (x == n - 1) v += w * um[L3(n, iz, iy, hi)] * p.ih2x;
          if (y == 0) v += w * um[L3(n, iz, lo, ix)] * p.ih2y;
          if (y == n - 1) v += w * um[L3(n, iz, hi, ix)] * p.ih2y;
          if (z == 0) v += w * um[L3(n, lo, iy, ix)] * p.ih2z;
          if (z == n - 1) v += w * um[L3(n, hi, iy, ix)] * p.ih2z;
        }
        {
          // div(lambda grad eta), ac_calc_F2 (anisotropic.c:164-628): the flux
          // component c at a neighbour q is lam[c] . (central differences at q),
          // zero when q is outside the block; y and z differences are
          // (previous - next), as the reference writes them
          auto U = [&](int dz, int dy, int dx) { return rg[so[dz + 2] + dy * HX + dx]; };
          const T c0 = U(0, 0, 0);
          const T xp2 = U(0, 0, 2), xm2 = U(0, 0, -2), yp2 = U(0, 2, 0), ym2 = U(0, -2, 0), zp2 = U(2, 0, 0),
                  zm2 = U(-2, 0, 0);
          const T xpym = U(0, -1, 1), xpyp = U(0, 1, 1), xmym = U(0, -1, -1), xmyp = U(0, 1, -1);
          const T xpzm = U(-1, 0, 1), xpzp = U(1, 0, 1), xmzm = U(-1, 0, -1), xmzp = U(1, 0, -1);
          const T ymzm = U(-1, -1, 0), ymzp = U(1, -1, 0), ypzm = U(-1, 1, 0), ypzp = U(1, 1, 0);
          // folded constants: k[3 r + c] = epn2 LE lam[r][c] / (2 h_r 2 h_c)
          const T *k = p.kan[m];
          const T ar = x < n - 1 ? k[0] * (xp2 - c0) + k[1] * (xpym - xpyp) + k[2] * (xpzm - xpzp) : (T)0;
          const T al = x > 0 ? k[0] * (c0 - xm2) + k[1] * (xmym - xmyp) + k[2] * (xmzm - xmzp) : (T)0;
          const T at = y > 0 ? k[3] * (xpym - xmym) + k[4] * (ym2 - c0) + k[5] * (ymzm - ymzp) : (T)0;
          const T ab = y < n - 1 ? k[3] * (xpyp - xmyp) + k[4] * (c0 - yp2) + k[5] * (ypzm - ypzp) : (T)0;
          const T af = z > 0 ? k[6] * (xpzm - xmzm) + k[7] * (ymzm - ypzm) + k[8] * (zm2 - c0) : (T)0;
          const T ak = z < n - 1 ? k[6] * (xpzp - xmzp) + k[7] * (ymzp - ypzp) + k[8] * (c0 - zp2) : (T)0;
          v -= ((ar - al) + (at - ab)) + (af - ak);
        }
        if (p.elastic == 1) v -= p.LE * p.es * felas[m * n3 + l];
        out[m * n3 + l] = v;
      }
    }
    __syncthreads();
  }
}

// Boundary chemical potential at periodic image cell (z,y,x) (ch_mu).
template <typename PL, typename T>
__device__ inline T ch_mu_at(const P<T> &p, const T *__restrict__ u, int z, int y, int x) {
  int n = p.n;
  long long n3 = (long long)n * n * n;
  const T *cf = u + p.nac * n3;
  T cv = cf[L3(n, z, y, x)];
  T lap = (cf[L3(n, z, y, img1(n, x - 1))] + (T)(-2.0) * cv + cf[L3(n, z, y, img1(n, x + 1))]) * p.ih2x;
  lap += (cf[L3(n, z, img1(n, y - 1), x)] + (T)(-2.0) * cv + cf[L3(n, z, img1(n, y + 1), x)]) * p.ih2y;
  lap += (cf[L3(n, img1(n, z - 1), y, x)] + (T)(-2.0) * cv + cf[L3(n, img1(n, z + 1), y, x)]) * p.ih2z;
  T e[4] = {(T)0, (T)0, (T)0, (T)0};
  for (int m = 0; m < p.nac; m++) e[m] = u[m * n3 + L3(n, z, y, x)];
  T mu = p.LCI * p.epn2 * lap;
  mu -= p.LCI * ch_f<PL>(p, e, cv);
  return mu;
}

// The two constant-mobility kernels: p.zc planes per CTA away from the faces,
// the face cells (whose lifting reads far images) one per thread in the
// launch's last CTAs, so that no warp of the march waits on them.

// t = -LCI KCI c + LCI CH_f, minus the face liftings (first part of
// ch_calc_FU_ConstantMobility).
template <typename PL, typename T>
__global__ void __launch_bounds__(RX * RY) rhs_ch_t_kernel(P<T> p0, const T *__restrict__ u, T *__restrict__ t,
                                                           int zblocks) {
  chain_wait();
  const int n = p0.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  P<T> p = p0;
  auto value = [&](const T *ur, size_t l) {
    T e[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
    for (int m = 0; m < 4; m++)
      if (m < p.nac) e[m] = ur[m * n3 + l];
    const T c = ur[p.nac * n3 + l];
    T v = -p.LCI * p.KCI * c;
    v += p.LCI * ch_f<PL>(p, e, c);
    return v;
  };
  if ((int)blockIdx.z < zblocks) {
    const int zch = (n + p.zc - 1) / p.zc;
    const int run = blockIdx.z / zch, zci = blockIdx.z - run * zch;
    const int c0 = blockIdx.x * (RX * RY) + threadIdx.x, m2 = n - 2;  // cell of the interior plane
    if (c0 >= m2 * m2) return;
    const int y = c0 / m2 + 1, x = c0 - (y - 1) * m2 + 1;
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    u += (size_t)run * p.F * n3;
    t += (size_t)run * n3;
    const int z0 = max(1, zci * p.zc), z1 = min(n - 1, (zci + 1) * p.zc);
#pragma unroll 2
    for (int z = z0; z < z1; z++) {
      const size_t l = (size_t)z * nn + (size_t)y * n + x;
      t[l] = value(u, l);
    }
    return;
  }
  const int per = face_cells(n), total = per * p.runs;
  const int stride = (int)(gridDim.z - zblocks) * gridDim.x * (RX * RY);
  for (int i = (((int)blockIdx.z - zblocks) * gridDim.x + blockIdx.x) * (RX * RY) + threadIdx.x; i < total; i += stride) {
    const int run = i / per;
    int z, y, x;
    face_cell(n, i - run * per, z, y, x);
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    const T *ur = u + (size_t)run * p.F * n3, *cf = ur + p.nac * n3;
    const size_t l = (size_t)z * nn + (size_t)y * n + x;
    T v = value(ur, l);
    const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
    const T w = p.LCI * p.epn2;
    if (x == 0) v -= w * cf[L3(n, iz, iy, lo)] * p.ih2x;
    if (x == n - 1) v -= w * cf[L3(n, iz, iy, hi)] * p.ih2x;
    if (y == 0) v -= w * cf[L3(n, iz, lo, ix)] * p.ih2y;
    if (y == n - 1) v -= w * cf[L3(n, iz, hi, ix)] * p.ih2y;
    if (z == 0) v -= w * cf[L3(n, lo, iy, ix)] * p.ih2z;
    if (z == n - 1) v -= w * cf[L3(n, hi, iy, ix)] * p.ih2z;
    t[(size_t)run * n3 + l] = v;
  }
}

// N_c = lap(t) (zero outside), minus mu(outside)/h^2 on faces.  Six CTAs an SM:
// the face cells' code would take 106 registers and leave the march two (54 us at
// 196^3, now 30).
template <typename PL, typename T>
__global__ void __launch_bounds__(RX * RY, sizeof(T) == 4 ? 6 : 4) rhs_ch_lap_kernel(P<T> p0, const T *__restrict__ u, const T *__restrict__ t,
                                                             T *__restrict__ out, int zblocks) {
  chain_wait();
  const int n = p0.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  P<T> p = p0;
  if ((int)blockIdx.z < zblocks) {
    const int zch = (n + p.zc - 1) / p.zc;
    const int run = blockIdx.z / zch, zci = blockIdx.z - run * zch;
    const int c0 = blockIdx.x * (RX * RY) + threadIdx.x, m2 = n - 2;  // cell of the interior plane
    if (c0 >= m2 * m2) return;
    const int y = c0 / m2 + 1, x = c0 - (y - 1) * m2 + 1;
    t += (size_t)run * n3;
    out += (size_t)run * p.F * n3;
    const int z0 = max(1, zci * p.zc), z1 = min(n - 1, (zci + 1) * p.zc);
    if (z0 >= z1) return;
    size_t l = (size_t)z0 * nn + (size_t)y * n + x;
    T tm = t[l - nn], tc = t[l];  // planes z - 1 and z
#pragma unroll 2
    for (int z = z0; z < z1; z++, l += nn) {
      const T tp = t[l + nn];
      T v = (t[l - 1] + t[l + 1] - (T)2 * tc) * p.ih2x;
      v += (t[l - n] + t[l + n] - (T)2 * tc) * p.ih2y;
      v += (tm + tp - (T)2 * tc) * p.ih2z;
      out[l] = v;
      tm = tc;
      tc = tp;
    }
    return;
  }
  const int per = face_cells(n), total = per * p.runs;
  const int stride = (int)(gridDim.z - zblocks) * gridDim.x * (RX * RY);
  for (int i = (((int)blockIdx.z - zblocks) * gridDim.x + blockIdx.x) * (RX * RY) + threadIdx.x; i < total; i += stride) {
    const int run = i / per;
    int z, y, x;
    face_cell(n, i - run * per, z, y, x);
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    const T *ur = u + (size_t)run * p.F * n3, *tr = t + (size_t)run * n3;
    const size_t l = (size_t)z * nn + (size_t)y * n + x;
    const T tc = tr[l];
    const T fl = x > 0 ? tr[l - 1] : (T)0, fr = x < n - 1 ? tr[l + 1] : (T)0;
    const T ft = y > 0 ? tr[l - n] : (T)0, fb = y < n - 1 ? tr[l + n] : (T)0;
    const T ff = z > 0 ? tr[l - nn] : (T)0, fk = z < n - 1 ? tr[l + nn] : (T)0;
    T v = (fl + fr - (T)2 * tc) * p.ih2x;
    v += (ft + fb - (T)2 * tc) * p.ih2y;
    v += (ff + fk - (T)2 * tc) * p.ih2z;
    const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
    if (x == 0) v -= ch_mu_at<PL>(p, ur, iz, iy, lo) * p.ih2x;
    if (x == n - 1) v -= ch_mu_at<PL>(p, ur, iz, iy, hi) * p.ih2x;
    if (y == 0) v -= ch_mu_at<PL>(p, ur, iz, lo, ix) * p.ih2y;
    if (y == n - 1) v -= ch_mu_at<PL>(p, ur, iz, hi, ix) * p.ih2y;
    if (z == 0) v -= ch_mu_at<PL>(p, ur, lo, iy, ix) * p.ih2z;
    if (z == n - 1) v -= ch_mu_at<PL>(p, ur, hi, iy, ix) * p.ih2z;
    out[(size_t)run * p.F * n3 + l] = v;
  }
}

// ---- variable-mobility Cahn-Hilliard ---------------------------------------
// ch_calc_FU_VariableMobility (source_beta_to_omega/src/mobility.c:838-858),
// update_M_C (:860-922) run first, on the single conserved field:
//   f0 = -LCI KCI c + LCI CH_f                              (ch_calc_F0)
//   t1 = -f0 + KCI c + epn2 c_out / h^2 on faces,  f1 = -C lap0(t1) - C mu_out / h^2
//                                                           (ch_calc_F1)
//   t2 = epn2 lap0(c) - f0 + epn2 c_out / h^2 on faces,
//   f2 = -div0((M - C) grad t2)                             (ch_calc_F2,
//        ch_divergence_M_gradient :435-722: face flux (m_q + m)(a_q - a)/(2 h^2))
//   N  = LCI (f1 + f2)
// with M(eta0) the first concentration's mobility, C its largest value over
// the block, lap0 / div0 zero outside the block (values and mobility), c_out
// the periodic image outside a face and mu_out the boundary chemical potential
// there (ch_mu).  Three launches: the block maxima of M, their maximum C, then
// t1 and t2, then N.

template <typename T>
__device__ __forceinline__ T mobility(const P<T> &p, T e) {
  return p.mob_m0 * ((T)1 * ((T)1 - e) + p.mob_dg * e);
}

// per run (blockIdx.y): the largest M over the block, per CTA
template <typename T>
__global__ void __launch_bounds__(256) mob_max_kernel(P<T> p, const T *__restrict__ u, double *__restrict__ part) {
  chain_wait();
  __shared__ double sm[8];
  const size_t n3 = (size_t)p.n * p.n * p.n;
  const T *e0 = u + (size_t)blockIdx.y * p.F * n3;  // the run's first order parameter
  T top = (T)-1.0e30;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n3; i += (size_t)gridDim.x * blockDim.x)
    top = max(top, mobility(p, e0[i]));
  double mx = (double)top;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) mx = fmax(mx, sm[w]);
    part[(size_t)blockIdx.y * MOB_PARTS + blockIdx.x] = mx;
  }
}

// C of every run: cmax[run] = max of its MOB_PARTS partial maxima
__global__ void __launch_bounds__(256) mob_final_kernel(const double *__restrict__ part, double *__restrict__ cmax) {
  chain_wait();
  __shared__ double sm[8];
  double mx = -1.0e30;
  for (int i = threadIdx.x; i < MOB_PARTS; i += blockDim.x) mx = fmax(mx, part[(size_t)blockIdx.x * MOB_PARTS + i]);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) mx = fmax(mx, sm[w]);
    cmax[blockIdx.x] = mx;
  }
}

// The two kernels over the cells: planes of the march away from the faces, the
// face cells apart in the launch's last CTAs, as the constant-mobility ones, and
// for FP32 four CTAs an SM (with the liftings inside the march and two CTAs an SM
// 27 and 43 us at 104^3, now 13 and 17).
// t1 and t2 of every cell.
template <typename PL, typename T>
__global__ void __launch_bounds__(RX * RY, sizeof(T) == 4 ? 4 : 2) mob_t_kernel(P<T> p0, const T *__restrict__ u0,
                                                                                T *__restrict__ tt, int zblocks) {
  chain_wait();
  const int n = p0.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  P<T> p = p0;
  auto cell = [&](auto face, int run, int z, int y, int x) {
    const T *u = u0 + (size_t)run * p.F * n3;
    T *t1 = tt + (size_t)run * 2 * n3, *t2 = t1 + n3;
    const size_t l = (size_t)z * nn + (size_t)y * n + x;
    const T *cf = u + p.nac * n3;
    T e[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
    for (int m = 0; m < 4; m++)
      if (m < p.nac) e[m] = u[m * n3 + l];
    const T c = cf[l];
    T f0 = -p.LCI * p.KCI * c;
    f0 += p.LCI * ch_f<PL>(p, e, c);
    const T cl = x > 0 ? cf[l - 1] : (T)0, cr = x < n - 1 ? cf[l + 1] : (T)0;
    const T ct = y > 0 ? cf[l - n] : (T)0, cb = y < n - 1 ? cf[l + n] : (T)0;
    const T cz = z > 0 ? cf[l - nn] : (T)0, ck = z < n - 1 ? cf[l + nn] : (T)0;
    T la = (cl + cr - (T)2 * c) * p.ih2x;
    la += (ct + cb - (T)2 * c) * p.ih2y;
    la += (cz + ck - (T)2 * c) * p.ih2z;
    T a = -f0 + p.KCI * c;
    T b = p.epn2 * la - f0;
    if (decltype(face)::value) {
      const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
      T w;
      if (x == 0) { w = p.epn2 * cf[L3(n, iz, iy, lo)] * p.ih2x; a += w; b += w; }
      if (x == n - 1) { w = p.epn2 * cf[L3(n, iz, iy, hi)] * p.ih2x; a += w; b += w; }
      if (y == 0) { w = p.epn2 * cf[L3(n, iz, lo, ix)] * p.ih2y; a += w; b += w; }
      if (y == n - 1) { w = p.epn2 * cf[L3(n, iz, hi, ix)] * p.ih2y; a += w; b += w; }
      if (z == 0) { w = p.epn2 * cf[L3(n, lo, iy, ix)] * p.ih2z; a += w; b += w; }
      if (z == n - 1) { w = p.epn2 * cf[L3(n, hi, iy, ix)] * p.ih2z; a += w; b += w; }
    }
    t1[l] = a;
    t2[l] = b;
  };
  if ((int)blockIdx.z < zblocks) {
    const int zch = (n + p.zc - 1) / p.zc;
    const int run = blockIdx.z / zch, zci = blockIdx.z - run * zch;
    const int c0 = blockIdx.x * (RX * RY) + threadIdx.x, m2 = n - 2;  // cell of the interior plane
    if (c0 >= m2 * m2) return;
    const int y = c0 / m2 + 1, x = c0 - (y - 1) * m2 + 1;
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    const int z0 = max(1, zci * p.zc), z1 = min(n - 1, (zci + 1) * p.zc);
    for (int z = z0; z < z1; z++) cell(std::false_type(), run, z, y, x);
    return;
  }
  const int per = face_cells(n), total = per * p.runs;
  const int stride = (int)(gridDim.z - zblocks) * gridDim.x * (RX * RY);
  for (int i = (((int)blockIdx.z - zblocks) * gridDim.x + blockIdx.x) * (RX * RY) + threadIdx.x; i < total; i += stride) {
    const int run = i / per;
    int z, y, x;
    face_cell(n, i - run * per, z, y, x);
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    cell(std::true_type(), run, z, y, x);
  }
}

// N = LCI (f1 + f2) of every cell.
template <typename PL, typename T>
__global__ void __launch_bounds__(RX * RY, sizeof(T) == 4 ? 4 : 2) mob_n_kernel(P<T> p0, const T *__restrict__ u0,
                                                                                const T *__restrict__ tt,
                                                                                const double *__restrict__ cmax,
                                                                                T *__restrict__ out0, int zblocks) {
  chain_wait();
  const int n = p0.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  P<T> p = p0;
  auto cell = [&](auto face, int run, int z, int y, int x) {
    const T *u = u0 + (size_t)run * p.F * n3;
    T *out = out0 + (size_t)run * p.F * n3;
    const T *t1 = tt + (size_t)run * 2 * n3, *t2 = t1 + n3;
    const T C = (T)cmax[run];
    const size_t l = (size_t)z * nn + (size_t)y * n + x;
    // f1 = -C lap0(t1) - C mu_out / h^2
    const T tc = t1[l];
    const T al = x > 0 ? t1[l - 1] : (T)0, ar = x < n - 1 ? t1[l + 1] : (T)0;
    const T at = y > 0 ? t1[l - n] : (T)0, ab = y < n - 1 ? t1[l + n] : (T)0;
    const T af = z > 0 ? t1[l - nn] : (T)0, ak = z < n - 1 ? t1[l + nn] : (T)0;
    T la = (al + ar - (T)2 * tc) * p.ih2x;
    la += (at + ab - (T)2 * tc) * p.ih2y;
    la += (af + ak - (T)2 * tc) * p.ih2z;
    T f1 = -C * la;
    if (decltype(face)::value) {
      const int iz = img1(n, z), iy = img1(n, y), ix = img1(n, x), lo = img1(n, -1), hi = img1(n, n);
      if (x == 0) f1 -= C * ch_mu_at<PL>(p, u, iz, iy, lo) * p.ih2x;
      if (x == n - 1) f1 -= C * ch_mu_at<PL>(p, u, iz, iy, hi) * p.ih2x;
      if (y == 0) f1 -= C * ch_mu_at<PL>(p, u, iz, lo, ix) * p.ih2y;
      if (y == n - 1) f1 -= C * ch_mu_at<PL>(p, u, iz, hi, ix) * p.ih2y;
      if (z == 0) f1 -= C * ch_mu_at<PL>(p, u, lo, iy, ix) * p.ih2z;
      if (z == n - 1) f1 -= C * ch_mu_at<PL>(p, u, hi, iy, ix) * p.ih2z;
    }
    // f2 = -div0((M - C) grad t2), M - C and t2 zero outside the block
    const T *e0 = u;
    const T bc = t2[l], mc = mobility(p, e0[l]) - C;
    auto nb = [&](bool in, size_t q, T &bq, T &mq) {
      bq = in ? t2[q] : (T)0;
      mq = in ? mobility(p, e0[q]) - C : (T)0;
    };
    T bq, mq, d;
    const T hx = (T)0.5 * p.ih2x, hy = (T)0.5 * p.ih2y, hz = (T)0.5 * p.ih2z;
    nb(x > 0, l - 1, bq, mq);
    d = (mq + mc) * (bq - bc) * hx;
    nb(x < n - 1, l + 1, bq, mq);
    d += (mq + mc) * (bq - bc) * hx;
    nb(y > 0, l - n, bq, mq);
    d += (mq + mc) * (bq - bc) * hy;
    nb(y < n - 1, l + n, bq, mq);
    d += (mq + mc) * (bq - bc) * hy;
    nb(z > 0, l - nn, bq, mq);
    d += (mq + mc) * (bq - bc) * hz;
    nb(z < n - 1, l + nn, bq, mq);
    d += (mq + mc) * (bq - bc) * hz;
    out[(size_t)p.nac * n3 + l] = p.LCI * (f1 - d);
  };
  if ((int)blockIdx.z < zblocks) {
    const int zch = (n + p.zc - 1) / p.zc;
    const int run = blockIdx.z / zch, zci = blockIdx.z - run * zch;
    const int c0 = blockIdx.x * (RX * RY) + threadIdx.x, m2 = n - 2;  // cell of the interior plane
    if (c0 >= m2 * m2) return;
    const int y = c0 / m2 + 1, x = c0 - (y - 1) * m2 + 1;
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    const int z0 = max(1, zci * p.zc), z1 = min(n - 1, (zci + 1) * p.zc);
    for (int z = z0; z < z1; z++) cell(std::false_type(), run, z, y, x);
    return;
  }
  const int per = face_cells(n), total = per * p.runs;
  const int stride = (int)(gridDim.z - zblocks) * gridDim.x * (RX * RY);
  for (int i = (((int)blockIdx.z - zblocks) * gridDim.x + blockIdx.x) * (RX * RY) + threadIdx.x; i < total; i += stride) {
    const int run = i / per;
    int z, y, x;
    face_cell(n, i - run * per, z, y, x);
    if (p0.krun) p.K[0] = (T)p0.krun[run];
    cell(std::true_type(), run, z, y, x);
  }
}

// r = N - H u = N + LE (epn2 sum_a kk_a T_a u - KE u) of the Allen-Cahn fields,
// T_a the second difference along axis a with zero values outside the block
// (the operator the eigenbasis diagonalises).  A thread marches an (x, y)
// column; in FP32 differences are taken first, so a smooth field loses no
// digits; FP64, bound by its pipe, takes 7 operations instead of 14 (r's
// rounding, dt H 2^-53 of u with dt H <= 4, is below the products').
// q0 + blockIdx.z = (run, field) x chunk of planes.  FP32 is bound by HBM (u and
// N read, r written).
template <typename T>
__global__ void __launch_bounds__(RX * RY) increment_rhs_kernel(P<T> p, const T *__restrict__ u,
                                                                const T *__restrict__ rhs, T *__restrict__ r, T cx, T cy,
                                                                T cz, int q0) {
  chain_wait();
  const int n = p.n;
  const size_t nn = (size_t)n * n, n3 = nn * n;
  const int zch = (n + p.zc - 1) / p.zc, q = q0 + blockIdx.z;
  const int t = q / zch, zci = q - t * zch;  // t = run nac + m
  const int c = blockIdx.x * (RX * RY) + threadIdx.x;  // cell of the plane: no idle threads in warps
  if (c >= n * n) return;
  const int y = c / n, x = c - y * n;
  const size_t f = (size_t)(t / p.nac) * p.F + t % p.nac;
  const int z0 = zci * p.zc, z1 = min(n, z0 + p.zc);
  size_t l = (size_t)z0 * nn + c;
  const T *uf = u + f * n3, *nf = rhs + f * n3;
  T *rf = r + (size_t)t * n3;
  const T cc = -(p.LE * p.KE + (T)2 * (cx + cy + cz));
  T um = z0 > 0 ? uf[l - nn] : (T)0, uc = uf[l];
#pragma unroll 2
  for (int z = z0; z < z1; z++, l += nn) {
    const T up = z < n - 1 ? uf[l + nn] : (T)0;
    const T xm = x > 0 ? uf[l - 1] : (T)0, xp = x < n - 1 ? uf[l + 1] : (T)0;
    const T ym = y > 0 ? uf[l - n] : (T)0, yp = y < n - 1 ? uf[l + n] : (T)0;
    if (sizeof(T) == 8) {
      rf[l] = fma(cx, xm + xp, fma(cy, ym + yp, fma(cz, um + up, fma(cc, uc, nf[l]))));
    } else {
      const T lx = (xm - uc) + (xp - uc), ly = (ym - uc) + (yp - uc), lz = (um - uc) + (up - uc);
      rf[l] = (nf[l] - p.LE * p.KE * uc) + (cx * lx + cy * ly + cz * lz);
    }
    um = uc;
    uc = up;
  }
}

// CTAs over a plane's cells in order, a thread each: 32 x 8 tiles of an edge a
// little above a multiple of 32, as every N + 4 is, left up to 44 % of the
// threads idle, which costs FP64 pipe time all the same (4 fields of 68^3 in
// FP64: right-hand side 61 -> 47 us, and the increments 62 -> 30 with their
// fewer operations)
static int plane_tiles(int cells) { return (cells + RX * RY - 1) / (RX * RY); }

// z-planes per CTA: the most of `zmax`, zmax / 2, .. 2 that still gives every SM
// four CTAs (a small block marched 32 planes a CTA left 20 CTAs on 152 SMs:
// 121 us at 36^3).
static int planes_per_cta(int n, int zmax, long long tiles, int runs) {
  int zc = zmax;
  if ((long long)((n + zc - 1) / zc) * runs > 32767) zc = std::max(zc, 32);  // the grid's z extent
  while (zc > 2 && tiles * ((n + zc - 1) / zc) < 4 * 152) zc /= 2;
  return zc;
}

// z-planes per CTA of the Allen-Cahn right-hand side (tiles: CTAs of one plane of
// every run).  A tuned value takes the place of the default bound, so whatever the
// tuner chooses fills the SMs as the default does, and the default is one of its
// candidates.
int rhs_ac_planes(int n, int tuned, bool tensors, long long tiles, int runs) {
  return planes_per_cta(n, tuned > 0 ? tuned : tensors ? 32 : 8, tiles, runs);
}

template <typename T>
cudaError_t launch_increment_rhs(const Phys &ph, const T *u, const T *rhs, T *r, cudaStream_t s) {
  P<T> p = to_p<T>(ph);
  const int count = p.runs * ph.nac, tiles = plane_tiles(ph.n * ph.n);
  p.zc = planes_per_cta(ph.n, 16, (long long)tiles * count, count);
  T c[3];
  for (int a = 0; a < 3; a++) c[a] = (T)(ph.LE * ph.epn2 * ph.kk[a] / (ph.h[a] * ph.h[a]));
  const int total = ((ph.n + p.zc - 1) / p.zc) * count;
  for (int q0 = 0; q0 < total; q0 += 65535) {  // the grid's z extent
    chain_launch(sizeof(T) == 4, increment_rhs_kernel<T>, dim3(tiles, 1, std::min(65535, total - q0)), RX * RY, 0, s, p, u, rhs, r, c[0], c[1],
                                                                                            c[2], q0);
    launch_counter()++;
  }
  return cudaGetLastError();
}
template cudaError_t launch_increment_rhs<double>(const Phys &, const double *, const double *, double *, cudaStream_t);
template cudaError_t launch_increment_rhs<float>(const Phys &, const float *, const float *, float *, cudaStream_t);

template <typename PL, typename T>
static cudaError_t launch_rhs_pl(const Phys &ph, const T *u, const T *felas, T *out, T *scratch, cudaStream_t s) {
  P<T> p = to_p<T>(ph);
  long long n3 = (long long)ph.n * ph.n * ph.n;
  const int gx = (ph.n + RX - 1) / RX, gy = (ph.n + RY - 1) / RY;
  const dim3 blk(RX, RY);
  // interior cells of a plane in order, and CTAs (in z) for the face cells, in the
  // kernels that take them apart
  const int tiles = plane_tiles((ph.n - 2) * (ph.n - 2));
  const int zfaces = (int)(((long long)face_cells(ph.n) * p.runs + RX * RY * tiles - 1) / ((long long)RX * RY * tiles));
  if (ph.nac > 0) {
    bool diag = true;  // every gradient tensor diagonal
    for (int m = 0; m < ph.nac; m++)
      for (int k = 0; k < 9; k++) diag = diag && (k % 4 == 0 || p.kan[m][k] == (T)0);
    const bool ring = ph.anisotropic && !diag;
    p.zc = rhs_ac_planes(ph.n, ph.rhs_zc, ph.anisotropic, (long long)(ring ? gx * gy : tiles) * p.runs, p.runs);
    // more runs than a grid of 32 planes a CTA holds in z are refused
    if ((long long)((ph.n + 31) / 32) * p.runs > 65535) return cudaErrorInvalidConfiguration;
    const int zblocks = ((ph.n + p.zc - 1) / p.zc) * p.runs;
    // the face cells' CTAs come after the march's, in a launch of their own where
    // the grid's z does not hold both (split over y too, the kernel's block index
    // cost the march its registers: 196^3 197 -> 274 us)
    const bool apart = zblocks + zfaces > 65535;
    auto diag_kernels = [&](auto kernel) {
      const dim3 grid(tiles, 1, apart ? zblocks : zblocks + zfaces);
      chain_launch(sizeof(T) == 4, kernel, grid, RX * RY, 0, s, p, u, felas, out, zblocks);
      if (!apart) return;
      chain_launch(sizeof(T) == 4, kernel, dim3(tiles, 1, std::min(zfaces, 65535)), RX * RY, 0, s, p, u, felas, out, 0);
      launch_counter()++;
    };
    const size_t smem = sizeof(T) * ph.nac * 5 * PLANE;
    cudaError_t e = cudaSuccess;
    switch (ph.nac * 3 + (ring ? 2 : ph.anisotropic ? 1 : 0)) {
#define SCLET_RHS_AC(NAC)                                                                                         \
  case NAC * 3: diag_kernels(rhs_ac_diag_kernel<PL, T, NAC, false>); break;                                       \
  case NAC * 3 + 1: diag_kernels(rhs_ac_diag_kernel<PL, T, NAC, true>); break;                                    \
  case NAC * 3 + 2:                                                                                               \
    e = cudaFuncSetAttribute(rhs_ac_kernel<PL, T, NAC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);   \
    if (e == cudaSuccess) chain_launch(sizeof(T) == 4, rhs_ac_kernel<PL, T, NAC>, dim3(gx, gy, zblocks), blk, smem, s, p, u, felas, out);     \
    break;
      SCLET_RHS_AC(1) SCLET_RHS_AC(2) SCLET_RHS_AC(3) SCLET_RHS_AC(4)
#undef SCLET_RHS_AC
      default: e = cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    launch_counter()++;
  }
  if (PL::max_nch > 0 && ph.varmob && ph.nch == 1) {
    if (!ph.mob_t || !ph.mob_part) return cudaErrorInvalidValue;
    T *tt = static_cast<T *>(ph.mob_t);
    double *cmax = ph.mob_part + (size_t)MOB_PARTS * p.runs;
    chain_launch(sizeof(T) == 4, mob_max_kernel<T>, dim3(MOB_PARTS, p.runs), 256, 0, s, p, u, ph.mob_part);
    chain_launch(true, mob_final_kernel, p.runs, 256, 0, s, ph.mob_part, cmax);
    p.zc = planes_per_cta(ph.n, 16, (long long)tiles * p.runs, p.runs);
    const int zblocks = ((ph.n + p.zc - 1) / p.zc) * p.runs;
    const dim3 gmb(tiles, 1, zblocks + zfaces);  // one run: nch > 0
    chain_launch(sizeof(T) == 4, mob_t_kernel<PL, T>, gmb, RX * RY, 0, s, p, u, tt, zblocks);
    chain_launch(sizeof(T) == 4, mob_n_kernel<PL, T>, gmb, RX * RY, 0, s, p, u, tt, cmax, out, zblocks);
    launch_counter() += 4;
  } else if (PL::max_nch > 0) {
    for (int m = 0; m < ph.nch; m++) {
      // one conserved field (the plugins' CH_f is defined for c_0 only)
      p.zc = planes_per_cta(ph.n, 16, (long long)tiles * p.runs, p.runs);
      const int zblocks = ((ph.n + p.zc - 1) / p.zc) * p.runs;
      const dim3 gch(tiles, 1, zblocks + zfaces);
      chain_launch(sizeof(T) == 4, rhs_ch_t_kernel<PL, T>, gch, RX * RY, 0, s, p, u, scratch, zblocks);
      chain_launch(sizeof(T) == 4, rhs_ch_lap_kernel<PL, T>, gch, RX * RY, 0, s, p, u, scratch, out + (long long)ph.nac * n3, zblocks);  // per run: + r F n^3
      launch_counter() += 2;
    }
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_rhs(const Phys &ph, const T *u, const T *felas, T *out, T *scratch, cudaStream_t s) {
  return with_physics(ph.physics, [&](auto *tag) {
    using PL = std::remove_pointer_t<decltype(tag)>;
    return launch_rhs_pl<PL, T>(ph, u, felas, out, scratch, s);
  });
}

template cudaError_t launch_rhs<double>(const Phys &, const double *, const double *, double *, double *, cudaStream_t);
template cudaError_t launch_rhs<float>(const Phys &, const float *, const float *, float *, float *, cudaStream_t);

}  // namespace sclet
