// Diagnostics of the state: check_soln_new (source_beta_to_omega/src/field.c:
// 407-678) as a device reduction.  Per field: max, min and vol = sum(u + 1) h^3
// over the owned cells; energy over the owned cells' corner cubes from the
// 8-corner averages and corner-difference gradients (field.c:487-511):
//   sum_m epn2/2 grad(eta_m).lambda_m.grad(eta_m)  [+ epn2/2 |grad c|^2]
//   + Landau energy of the averages.
// form 0 reproduces the reference's hard-coded 2-3-4 polynomial and its
// separate CH energy ((c^2-1)^2/4); form 1 is the plugin's total free energy
// (its F_bulk, sclet_physics.cuh, plus the gradient terms).
// Sums are compensated (TwoSum pairs) in FP64 and reduced in a fixed order,
// so the result is deterministic.
#include "sclet_internal.cuh"
#include "sclet_physics.cuh"

namespace sclet {

struct KS {
  double s, c;
};
__device__ inline void two_sum(double a, double b, double &s, double &e) {
  s = a + b;
  double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
__device__ inline void ks_add(KS &k, double v) {
  double s, e;
  two_sum(k.s, v, s, e);
  k.s = s;
  k.c += e;
}
__device__ inline KS ks_merge(KS a, KS b) {
  KS r;
  double e;
  two_sum(a.s, b.s, r.s, e);
  r.c = a.c + b.c + e;
  return r;
}

constexpr int EB = 256;  // threads per block

// Per-thread sum of FP32 values with FP64-class accuracy: a float pair (s, e)
// updated by the error-free TwoSum (Knuth), about 48 bits, so a thread's few dozen
// terms cost FP32 instructions, not FP64 ones (the FP64 pipe of this GPU is 1/64 of
// the FP32 rate).
struct Acc {
  float s = 0.0f, e = 0.0f;
  __device__ void add(float v) {
    const float t = s + v;
    const float bp = t - s;
    e += (s - (t - bp)) + (v - bp);
    s = t;
  }
  // pair sum with the partner lane at xor distance off; both lanes end with
  // the same pair (TwoSum is exact and the merge symmetric)
  __device__ void merge_lane(int off) {
    const float os = __shfl_xor_sync(0xffffffffu, s, off), oe = __shfl_xor_sync(0xffffffffu, e, off);
    const float t = s + os, bp = t - s;
    const float err = (s - (t - bp)) + (os - bp);
    e = (e + oe) + err;
    s = t;
  }
};
constexpr int MAXF = 5;

// partial record per block: for f < F: max, min, vol.s, vol.c; then
// eng_ac.s, eng_ac.c, eng_ch.s, eng_ch.c
__host__ __device__ inline int rec_len(int F) { return 4 * F + 4; }

// Reduction of the record (per field max, min, vol; two energies): warp
// butterflies, then the block's warps in lane order; fixed shape, so the
// result is deterministic.  TwoSum is exact and symmetric, so every lane of
// a butterfly holds the same pair.
__device__ __forceinline__ KS shfl_ks(KS v, int off) {
  KS o;
  o.s = __shfl_xor_sync(0xffffffffu, v.s, off);
  o.c = __shfl_xor_sync(0xffffffffu, v.c, off);
  return ks_merge(v, o);
}

// ---- FP32 states: z-marching form of the same reduction --------------------
//
// A CTA of 32 x 8 threads owns 32 x 8 owned (x, y) columns of one unit and
// walks its ZCH planes in z.  Each thread keeps the (x, y), (x, y + 1) values
// of plane z and z + 1 of every field in registers and takes the x + 1
// neighbours from the next lane, so a cell costs two loads per field instead
// of eight.  The conserved field's corner average is an exact FP32 pair sum
// finished in pair arithmetic (no FP64 instructions per cell).  Blocks loop
// over units; one partial record per block (rec_len).  Bound by FP32 issue:
// diagnostics of a 4-field 36^3 block 31 -> 18 us, of a 196^3 block with five
// fields 191 -> 150 us, since a plane's sums are shared by the cubes on both of
// its sides and FP64 adds only the warps' sums.
constexpr int EZ = 8;  // planes per unit

__host__ __device__ inline int energy_units(int N) { return ((N + 31) / 32) * ((N + 7) / 8) * ((N + EZ - 1) / EZ); }

struct Pair {
  float s, e;
};
// exact running sum of floats (TwoSum, Knuth)
__device__ __forceinline__ void pair_add(Pair &p, float v) {
  const float t = p.s + v, bp = t - p.s;
  p.e += (p.s - (t - bp)) + (v - bp);
  p.s = t;
}
// (a.s + a.e) + (b.s + b.e) rounded to float
__device__ __forceinline__ float pair_sum(Pair a, Pair b) {
  const float t = a.s + b.s, bp = t - a.s;
  const float err = (a.s - (t - bp)) + (b.s - bp);
  return t + (err + a.e + b.e);
}

// FP32 constants of energy_partial_f32, rounded once on the host (kernel
// parameters: read from the constant bank, never recomputed in the loop)
struct EConst {
  float i4hx, i4hy, i4hz, half_epn2;
  float K[16];       // plugin constants, the reference composition c0 (if any) as 0
  float p2, p3, p4;  // the 2-3-4 polynomial of energy form 0
  Pair kdp, kcp;     // cshift - c0 and cshift as float pairs
};

// The plugin sees the concentration as c - c0 (exact in pair arithmetic from
// the stored c - cshift) with its c0 constant 0, where it names one.
template <typename PL>
static EConst econst(const Phys &ph) {
  EConst c;
  c.i4hx = (float)(0.25 / ph.h[0]);
  c.i4hy = (float)(0.25 / ph.h[1]);
  c.i4hz = (float)(0.25 / ph.h[2]);
  c.half_epn2 = (float)(0.5 * ph.epn2);
  for (int k = 0; k < 16; k++) c.K[k] = (float)ph.K[k];
  const double kd = PL::c0_index >= 0 ? -ph.K[PL::c0_index] : 0.0;  // ph.K holds c0 - cshift
  if (PL::c0_index >= 0) c.K[PL::c0_index] = 0.0f;
  c.kdp = Pair{(float)kd, (float)(kd - (double)(float)kd)};
  c.p2 = (float)(2376.0 / 2372.0 / 2.0);
  c.p3 = (float)((7128.0 + 12.0 * 2372.0) / 2372.0 / 3.0);
  c.p4 = (float)((4752.0 + 12.0 * 2372.0) / 2372.0 / 4.0);
  c.kcp = Pair{(float)ph.cshift, (float)(ph.cshift - (double)(float)ph.cshift)};
  return c;
}

// (a + b) + c of pairs, rounded to float
__device__ __forceinline__ Pair pair_merge(Pair a, Pair b) {
  const float t = a.s + b.s, bp = t - a.s;
  return Pair{t, (a.e + b.e) + ((a.s - (t - bp)) + (b.s - bp))};
}

// A plane's share of the cubes above and below it, computed once: the corner
// sum, and the sums of the x- and y-differences (differences are formed before
// sums, so a smooth field loses no digits).
template <typename T>
struct Face4 {
  T v0, v1, v2, v3;  // (i, j) (i+1, j) (i, j+1) (i+1, j+1)
  T s, dx, dy;
  __device__ __forceinline__ void set(T a, T b, T c, T d) {
    v0 = a, v1 = b, v2 = c, v3 = d;
    s = (v0 + v1) + (v2 + v3);
    dx = (v1 - v0) + (v3 - v2);
    dy = (v2 - v0) + (v3 - v1);
  }
};

// Half epn2 times the symmetrised gradient tensors, the four-fold spacings
// folded in: xx yy zz xy xz yz (m < 4), then the conserved field's (4).
template <typename T>
__device__ __forceinline__ void energy_tensors(const Phys &ph, const double *elam, T (*q6)[6]) {
  if (threadIdx.x < 5 * 6 && threadIdx.y == 0) {
    const int m = threadIdx.x / 6, c = threadIdx.x % 6;
    const double i4[3] = {0.25 / ph.h[0], 0.25 / ph.h[1], 0.25 / ph.h[2]};
    const int r[6] = {0, 1, 2, 0, 0, 1}, k[6] = {0, 1, 2, 1, 2, 2};
    double v = c < 3 ? 1.0 : 0.0;
    if (m < 4) v = c < 3 ? elam[9 * m + 4 * c] : elam[9 * m + 3 * r[c] + k[c]] + elam[9 * m + 3 * k[c] + r[c]];
    q6[m][c] = (T)(0.5 * ph.epn2 * v * i4[r[c]] * i4[k[c]]);
  }
  __syncthreads();
}
template <typename T>
__device__ __forceinline__ T gradient_energy(const T *q, T ux, T uy, T uz) {
  return ux * (q[0] * ux + q[3] * uy + q[4] * uz) + uy * (q[1] * uy + q[5] * uz) + q[2] * uz * uz;
}

template <typename PL, int NAC, int NCH>
__global__ void __launch_bounds__(256, 2) energy_partial_f32(Phys ph, EConst ec, const float *__restrict__ u,
                                                             const double *__restrict__ elam, int form,
                                                             double *__restrict__ part) {
  chain_wait();
  constexpr int F = NAC + NCH;
  const int n = ph.n, N = n - 4;
  const long long n3 = (long long)n * n * n;
  __shared__ float q6[5][6];
  energy_tensors<float>(ph, elam, q6);
  float Kt[16];
#pragma unroll
  for (int k = 0; k < 16; k++) Kt[k] = ec.K[k];
  // blockIdx.y = run: its fields, its plugin constant 0, its partial records
  if (ph.krun) Kt[0] = (float)ph.krun[blockIdx.y];
  u += (long long)blockIdx.y * F * n3;
  part += (long long)blockIdx.y * gridDim.x * rec_len(F);
  const float p2 = ec.p2, p3 = ec.p3, p4 = ec.p4;
  float mx[F], mn[F];
  Acc vsum[F], eac_p, ech_p;
  int cnt = 0;
#pragma unroll
  for (int f = 0; f < F; f++) {
    mx[f] = -1.0e30f;
    mn[f] = 1.0e30f;
  }
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nti = (N + 31) / 32, ntj = (N + 7) / 8, units = energy_units(N);
  for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const int ti = unit % nti, tj = (unit / nti) % ntj, zc = unit / (nti * ntj);
    const int i = 2 + ti * 32 + tx, j = 2 + tj * 8 + ty;
    const bool own = i <= n - 3 && j <= n - 3, inner = i <= n - 4 && j <= n - 4;
    const int ic = i < n - 2 ? i : n - 2, jc = j < n - 2 ? j : n - 2;  // clamped: loads stay inside the block
    const int k0 = 2 + zc * EZ, k1 = k0 + EZ < n - 2 ? k0 + EZ : n - 2;
    const float *row = u + ((long long)k0 * n + jc) * n + ic;
    Face4<float> a[F];
    Pair ca = {0.0f, 0.0f};  // the conserved field's exact corner sum of plane k
    float nx[F][2], ne[F][2];  // plane in flight: (i, j), (i, j+1); the last lane's (i+1, j), (i+1, j+1)
    auto fetch = [&](const float *q) {
#pragma unroll
      for (int f = 0; f < F; f++) {
        const float *p = q + f * n3;
        nx[f][0] = p[0];
        nx[f][1] = p[n];
        ne[f][0] = tx == 31 ? p[1] : 0.0f;
        ne[f][1] = tx == 31 ? p[n + 1] : 0.0f;
      }
    };
    auto take = [&](int f, Face4<float> &b) {
      float r0 = __shfl_down_sync(0xffffffffu, nx[f][0], 1), r1 = __shfl_down_sync(0xffffffffu, nx[f][1], 1);
      if (tx == 31) r0 = ne[f][0], r1 = ne[f][1];
      b.set(nx[f][0], r0, nx[f][1], r1);
    };
    auto corner_pair = [&](const Face4<float> &b) {
      Pair c = {b.v0, 0.0f};
      pair_add(c, b.v1);
      pair_add(c, b.v2);
      pair_add(c, b.v3);
      return c;
    };
    fetch(row);
#pragma unroll
    for (int f = 0; f < F; f++) take(f, a[f]);
    if (NCH > 0) ca = corner_pair(a[F - 1]);
    row += (long long)n * n;
    fetch(row);
    // unrolled, so that a plane's sums change names instead of registers: 4 + 1
    // fields of 196^3 182 -> 150 us, of 516^3 2.92 -> 2.31 ms
#pragma unroll 4
    for (int k = k0; k < k1; k++) {
      Face4<float> b[F];  // plane k + 1
#pragma unroll
      for (int f = 0; f < F; f++) take(f, b[f]);
      row += (long long)n * n;
      if (k + 1 < k1) fetch(row);  // plane k + 2 while this one is worked on
      Pair cb = {0.0f, 0.0f};
      if (NCH > 0) cb = corner_pair(b[F - 1]);
      if (own) {
        cnt++;
#pragma unroll
        for (int f = 0; f < F; f++) {
          mx[f] = fmaxf(mx[f], a[f].v0);
          mn[f] = fminf(mn[f], a[f].v0);
          vsum[f].add(a[f].v0);
        }
      }
      if (inner && k <= n - 4) {
        float avg[F > 0 ? F : 1];
        float e_ac = 0.0f, e_ch = 0.0f, cd = 0.0f, cval = 0.0f;
#pragma unroll
        for (int f = 0; f < F; f++) {
          avg[f] = (a[f].s + b[f].s) * 0.125f;
          const float ux = a[f].dx + b[f].dx, uy = a[f].dy + b[f].dy;
          const float uz = ((b[f].v0 - a[f].v0) + (b[f].v1 - a[f].v1)) + ((b[f].v2 - a[f].v2) + (b[f].v3 - a[f].v3));
          const float gr = gradient_energy(q6[f < NAC ? f : 4], ux, uy, uz);
          if (f < NAC || form != 0) e_ac += gr;
          else e_ch += gr;
        }
        if (NCH > 0) {
          // exact corner sum, then (sum / 8 + cshift - c0) and (sum / 8 + cshift)
          Pair cs = pair_merge(ca, cb);
          cs.s *= 0.125f;
          cs.e *= 0.125f;
          cd = pair_sum(cs, ec.kdp);
          cval = pair_sum(cs, ec.kcp);
        }
        if (form == 0) {
          if (NAC > 0) {
            float s2 = 0.0f, s3 = 0.0f;
#pragma unroll
            for (int f = 0; f < (NAC < 4 ? NAC : 4); f++) {
              s2 += avg[f] * avg[f];
              s3 += avg[f] * avg[f] * avg[f];
            }
            e_ac += p2 * s2 - p3 * s3 + p4 * s2 * s2;
          }
          if (NCH > 0) e_ch += (cval * cval - 1.0f) * (cval * cval - 1.0f) * 0.25f;
        } else {
          sclet_acv<float> ac[NAC > 0 ? NAC : 1];
          sclet_chv<float> ch[1];
#pragma unroll
          for (int m = 0; m < NAC; m++) ac[m].u = avg[m];
          ch[0].c = cd;
          e_ac += PL::template f_bulk<float>(ac, ch, NAC, NCH, Kt);
        }
        eac_p.add(e_ac);
        if (form == 0) ech_p.add(e_ch);
      }
#pragma unroll
      for (int f = 0; f < F; f++) a[f] = b[f];
      ca = cb;
    }
  }
  // warp butterflies in FP32 (max, min) and exact-pair arithmetic (sums), then the
  // warps' values, sums in FP64 pairs, eight lanes a quantity (an FP64 warp
  // instruction is 64 cycles of its scheduler: the block's merges in FP64, one
  // field after the other, took longer than a small block's cells; in FP32 pairs
  // they would hold 48 bits, for 17.1 us of diagnostics at 36^3 instead of 18.3)
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int f = 0; f < F; f++) {
      mx[f] = fmaxf(mx[f], __shfl_xor_sync(0xffffffffu, mx[f], off));
      mn[f] = fminf(mn[f], __shfl_xor_sync(0xffffffffu, mn[f], off));
      vsum[f].merge_lane(off);
    }
    eac_p.merge_lane(off);
    ech_p.merge_lane(off);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
  }
  constexpr int NW = EB / 32;
  __shared__ float wv[4 * F + 4][NW];
  __shared__ int wc[NW];
  const int lane = tx, wid = ty;
  if (lane == 0) {
#pragma unroll
    for (int f = 0; f < F; f++) {
      wv[4 * f][wid] = mx[f];
      wv[4 * f + 1][wid] = mn[f];
      wv[4 * f + 2][wid] = vsum[f].s;
      wv[4 * f + 3][wid] = vsum[f].e;
    }
    wv[4 * F][wid] = eac_p.s;
    wv[4 * F + 1][wid] = eac_p.e;
    wv[4 * F + 2][wid] = ech_p.s;
    wv[4 * F + 3][wid] = ech_p.e;
    wc[wid] = cnt;
  }
  __syncthreads();
  if (wid < 2) {
    // quantity q (field q's sum, max and min, or an energy) of warp w
    static_assert(NW == 8 && F + 2 <= 8, "eight quantities over two warps");
    const int q = (wid * 32 + lane) >> 3, w = lane & 7;
    const bool on = q < F + 2, field = q < F;
    const int at = field ? 4 * q + 2 : 4 * F + 2 * (q - F);
    KS v = {on ? (double)wv[at][w] : 0.0, on ? (double)wv[at + 1][w] : 0.0};
    float top = field ? wv[4 * q][w] : -1.0e30f, low = field ? wv[4 * q + 1][w] : 1.0e30f;
    int count = wc[w];
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) {
      v = shfl_ks(v, off);
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
      low = fminf(low, __shfl_xor_sync(0xffffffffu, low, off));
      count += __shfl_xor_sync(0xffffffffu, count, off);
    }
    if (on && w == 0) {
      double *dst = part + (long long)blockIdx.x * rec_len(F);
      if (field) {
        const double sh = q >= NAC ? ph.cshift : 0.0;
        ks_add(v, (double)count * (sh + 1.0));  // sum of (value + 1)
        dst[4 * q] = (double)top + sh;
        dst[4 * q + 1] = (double)low + sh;
      }
      dst[at] = v.s;
      dst[at + 1] = v.c;
    }
  }
}

// ---- FP64 states: the same z-marching form in FP64 -------------------------
//
// The column tile and the plane walk of energy_partial_f32, with FP64 values
// and compensated FP64 (TwoSum) running sums.  Bound by FP64 instructions:
// diagnostics of 4 fields of 68^3 205 -> 146 us, of 4 + 1 fields of 132^3 1.54 ->
// 1.12 ms with about 270 of them per cell instead of 370.
// The largest (smallest) of doubles without FP64 instructions: a key that orders
// as the values do; NaN never wins.
__device__ __forceinline__ long long order_key(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double key_value(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
__device__ __forceinline__ bool is_nan_bits(double v) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

template <typename PL, int NAC, int NCH>
__global__ void __launch_bounds__(256, 1) energy_partial_f64z(Phys ph, const double *__restrict__ u,
                                                              const double *__restrict__ elam, int form,
                                                              double *__restrict__ part) {
  chain_wait();
  constexpr int F = NAC + NCH, Q = F + 2;  // sums of a block: one per field, two energies
  const int n = ph.n, N = n - 4;
  const long long n3 = (long long)n * n * n;
  __shared__ double q6[5][6];
  energy_tensors<double>(ph, elam, q6);
  double Kt[16];
#pragma unroll
  for (int k = 0; k < 16; k++) Kt[k] = ph.K[k];
  const double p2 = 2376.0 / 2372.0 / 2.0, p3 = (7128.0 + 12.0 * 2372.0) / 2372.0 / 3.0,
               p4 = (4752.0 + 12.0 * 2372.0) / 2372.0 / 4.0;
  long long mx[F], mn[F];  // order keys
  KS vsum[F], eac = {0.0, 0.0}, ech = {0.0, 0.0};
  int cnt = 0;
#pragma unroll
  for (int f = 0; f < F; f++) {
    mx[f] = order_key(-1.0e30);
    mn[f] = order_key(1.0e30);
    vsum[f] = KS{0.0, 0.0};
  }
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int nti = (N + 31) / 32, ntj = (N + 7) / 8, units = energy_units(N);
  for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
    const int ti = unit % nti, tj = (unit / nti) % ntj, zc = unit / (nti * ntj);
    const int i = 2 + ti * 32 + tx, j = 2 + tj * 8 + ty;
    const bool own = i <= n - 3 && j <= n - 3, inner = i <= n - 4 && j <= n - 4;
    const int ic = i < n - 2 ? i : n - 2, jc = j < n - 2 ? j : n - 2;
    const int k0 = 2 + zc * EZ, k1 = k0 + EZ < n - 2 ? k0 + EZ : n - 2;
    const double *row = u + ((long long)k0 * n + jc) * n + ic;
    Face4<double> a[F];
    auto take = [&](const double *q, Face4<double> &b) {
      const double v0 = q[0], v2 = q[n];
      double v1 = __shfl_down_sync(0xffffffffu, v0, 1), v3 = __shfl_down_sync(0xffffffffu, v2, 1);
      if (tx == 31) v1 = q[1], v3 = q[n + 1];
      b.set(v0, v1, v2, v3);
    };
#pragma unroll
    for (int f = 0; f < F; f++) take(row + f * n3, a[f]);
    for (int k = k0; k < k1; k++) {
      row += (long long)n * n;
      Face4<double> b[F];  // plane k + 1
#pragma unroll
      for (int f = 0; f < F; f++) take(row + f * n3, b[f]);
      if (own) {
        cnt++;
#pragma unroll
        for (int f = 0; f < F; f++) {
          const long long key = order_key(a[f].v0);
          if (!is_nan_bits(a[f].v0)) {
            mx[f] = key > mx[f] ? key : mx[f];
            mn[f] = key < mn[f] ? key : mn[f];
          }
          ks_add(vsum[f], a[f].v0);
        }
      }
      if (inner && k <= n - 4) {
        double avg[F > 0 ? F : 1];
        double e_ac = 0.0, e_ch = 0.0;
#pragma unroll
        for (int f = 0; f < F; f++) {
          avg[f] = (a[f].s + b[f].s) * 0.125;
          const double ux = a[f].dx + b[f].dx, uy = a[f].dy + b[f].dy;
          const double uz = ((b[f].v0 - a[f].v0) + (b[f].v1 - a[f].v1)) + ((b[f].v2 - a[f].v2) + (b[f].v3 - a[f].v3));
          const double gr = gradient_energy(q6[f < NAC ? f : 4], ux, uy, uz);
          if (f < NAC || form != 0) e_ac += gr;
          else e_ch += gr;
        }
        if (form == 0) {
          if (NAC > 0) {
            double s2 = 0.0, s3 = 0.0;
#pragma unroll
            for (int f = 0; f < (NAC < 4 ? NAC : 4); f++) {
              s2 += avg[f] * avg[f];
              s3 += avg[f] * avg[f] * avg[f];
            }
            e_ac += p2 * s2 - p3 * s3 + p4 * s2 * s2;
          }
          if (NCH > 0) e_ch += (avg[F - 1] * avg[F - 1] - 1.0) * (avg[F - 1] * avg[F - 1] - 1.0) * 0.25;
        } else {
          sclet_acv<double> ac[NAC > 0 ? NAC : 1];
          sclet_chv<double> ch[1];
#pragma unroll
          for (int m = 0; m < NAC; m++) ac[m].u = avg[m];
          ch[0].c = NCH > 0 ? avg[F - 1] : 0.0;
          e_ac += PL::template f_bulk<double>(ac, ch, NAC, NCH, Kt);
        }
        ks_add(eac, e_ac);
        if (form == 0) ks_add(ech, e_ch);
      }
#pragma unroll
      for (int f = 0; f < F; f++) a[f] = b[f];
    }
  }
  // The block's sums: every thread's pairs through shared memory, one warp per
  // quantity folding eight threads per lane and then the lanes: 96 FP64 warp
  // instructions per quantity instead of 40 per quantity in each of eight warps
  // (an FP64 warp instruction is 64 cycles of its scheduler).
  extern __shared__ double2 ks_of[];  // [Q][EB]
  __shared__ long long wmx[EB / 32][F], wmn[EB / 32][F];
  __shared__ int wcnt[EB / 32];
  const int tid = ty * 32 + tx;
#pragma unroll
  for (int f = 0; f < F; f++) ks_of[f * EB + tid] = make_double2(vsum[f].s, vsum[f].c);
  ks_of[F * EB + tid] = make_double2(eac.s, eac.c);
  ks_of[(F + 1) * EB + tid] = make_double2(ech.s, ech.c);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int f = 0; f < F; f++) {
      const long long p = __shfl_xor_sync(0xffffffffu, mx[f], off), q = __shfl_xor_sync(0xffffffffu, mn[f], off);
      mx[f] = p > mx[f] ? p : mx[f];
      mn[f] = q < mn[f] ? q : mn[f];
    }
    cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
  }
  if (tx == 0) {
#pragma unroll
    for (int f = 0; f < F; f++) {
      wmx[ty][f] = mx[f];
      wmn[ty][f] = mn[f];
    }
    wcnt[ty] = cnt;
  }
  __syncthreads();
  double *dst = part + (long long)blockIdx.x * rec_len(F);
  for (int q = ty; q < Q; q += EB / 32) {
    KS s = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < EB / 32; w++) {
      const double2 v = ks_of[q * EB + w * 32 + tx];
      s = w == 0 ? KS{v.x, v.y} : ks_merge(s, KS{v.x, v.y});
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s = shfl_ks(s, off);
    if (tx == 0) {
      if (q < F) {
        long long top = wmx[0][q], low = wmn[0][q];
        int count = wcnt[0];
        for (int w = 1; w < EB / 32; w++) {
          top = wmx[w][q] > top ? wmx[w][q] : top;
          low = wmn[w][q] < low ? wmn[w][q] : low;
          count += wcnt[w];
        }
        ks_add(s, (double)count);  // sum of (value + 1)
        dst[4 * q] = key_value(top);
        dst[4 * q + 1] = key_value(low);
      }
      const int at = q < F ? 4 * q + 2 : 4 * F + 2 * (q - F);
      dst[at] = s.s;
      dst[at + 1] = s.c;
    }
  }
}

// Final reduction over the block records: a block per quantity (per field max
// and min together, per field vol, the two energies; blockIdx.y = run), so that
// every quantity's FP64 merges have an SM's FP64 pipe to themselves; each thread
// folds a fixed strided subset of the records, then the lanes, then the warps
// (deterministic).  One block for all quantities took 15 us.
constexpr int FT_THREADS = 128;
__global__ void __launch_bounds__(FT_THREADS) energy_final_kernel(Phys ph, int form, const double *__restrict__ part,
                                                                  int npart, double *__restrict__ out) {
  chain_wait();
  const int F = ph.F, L = rec_len(F), q = blockIdx.x;
  part += (long long)blockIdx.y * npart * L;
  out += (long long)blockIdx.y * 4 * F;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (q < F) {  // max and min
    __shared__ long long sx[FT_THREADS / 32], sn[FT_THREADS / 32];
    long long mx = order_key(-1.0e30), mn = order_key(1.0e30);
    for (int b = tid; b < npart; b += FT_THREADS) {
      const long long x = order_key(part[(long long)b * L + 4 * q]), m = order_key(part[(long long)b * L + 4 * q + 1]);
      mx = x > mx ? x : mx;
      mn = m < mn ? m : mn;
    }
    for (int off = 16; off > 0; off >>= 1) {
      const long long x = __shfl_xor_sync(0xffffffffu, mx, off), m = __shfl_xor_sync(0xffffffffu, mn, off);
      mx = x > mx ? x : mx;
      mn = m < mn ? m : mn;
    }
    if (lane == 0) sx[wid] = mx, sn[wid] = mn;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < FT_THREADS / 32; w++) {
        mx = sx[w] > mx ? sx[w] : mx;
        mn = sn[w] < mn ? sn[w] : mn;
      }
      out[4 * q] = key_value(mx);
      out[4 * q + 1] = key_value(mn);
    }
    return;
  }
  const int s = q - F;  // field s's volume, or (s >= F) an energy
  const int at = s < F ? 4 * s + 2 : 4 * F + 2 * (s - F);
  if (s > F && form != 0) return;  // the separate CH energy belongs to form 0
  __shared__ double2 sk[FT_THREADS / 32];
  KS k = {0.0, 0.0};
  for (int b = tid; b < npart; b += FT_THREADS) {
    const double *r = part + (long long)b * L + at;
    k = ks_merge(k, KS{r[0], r[1]});
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) k = shfl_ks(k, off);
  if (lane == 0) sk[wid] = make_double2(k.s, k.c);
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < FT_THREADS / 32; w++) k = ks_merge(k, KS{sk[w].x, sk[w].y});
    const double v = (k.s + k.c) * (ph.h[0] * ph.h[1] * ph.h[2]);
    if (s < F) {
      out[4 * s + 2] = v;
    } else {
      // energy 0 goes to every field (form 0: the order parameters), 1 to the conserved ones
      for (int f = 0; f < F; f++)
        if ((form == 0 && f >= ph.nac) == (s > F)) out[4 * f + 3] = v;
    }
  }
}

// partial records (blocks) of one reduction: four CTAs per SM at most
int check_soln_partials(int n) {
  const int u = energy_units(n - 4);
  return u > 152 * 4 ? 152 * 4 : (u < 1 ? 1 : u);
}

template <typename PL, int NAC, int NCH>
static void launch_f32(const Phys &ph, const float *u, const double *elam, int form, double *partials, int npart,
                       cudaStream_t s) {
  chain_launch(npart <= 152, energy_partial_f32<PL, NAC, NCH>, dim3(npart, ph.runs > 1 ? ph.runs : 1), dim3(32, 8), 0, s, 
      ph, econst<PL>(ph), u, elam, form, partials);
}

template <typename PL, typename T>
static cudaError_t check_soln_pl(const Phys &ph, const T *u, const double *elam, int form, double *partials,
                                 int npart, cudaStream_t s) {
  if constexpr (sizeof(T) == 4) {
    const float *uf = u;
    switch (ph.nac * 2 + ph.nch) {
      case 1: launch_f32<PL, 0, 1>(ph, uf, elam, form, partials, npart, s); break;
      case 2: launch_f32<PL, 1, 0>(ph, uf, elam, form, partials, npart, s); break;
      case 3: launch_f32<PL, 1, 1>(ph, uf, elam, form, partials, npart, s); break;
      case 4: launch_f32<PL, 2, 0>(ph, uf, elam, form, partials, npart, s); break;
      case 5: launch_f32<PL, 2, 1>(ph, uf, elam, form, partials, npart, s); break;
      case 6: launch_f32<PL, 3, 0>(ph, uf, elam, form, partials, npart, s); break;
      case 7: launch_f32<PL, 3, 1>(ph, uf, elam, form, partials, npart, s); break;
      case 8: launch_f32<PL, 4, 0>(ph, uf, elam, form, partials, npart, s); break;
      default: launch_f32<PL, 4, 1>(ph, uf, elam, form, partials, npart, s); break;
    }
  } else {
    const double *ud = u;
    const dim3 g(npart), b(32, 8);
    switch (ph.nac * 2 + ph.nch) {
#define SCLET_F64Z(NA, NC) \
  case NA * 2 + NC:                                                                                         \
    chain_launch(false, energy_partial_f64z<PL, NA, NC>, g, b, sizeof(double2) * (NA + NC + 2) * EB, s, ph, ud, elam, form, \
                 partials);                                                                                 \
    break;
      SCLET_F64Z(0, 1) SCLET_F64Z(1, 0) SCLET_F64Z(1, 1) SCLET_F64Z(2, 0) SCLET_F64Z(2, 1)
      SCLET_F64Z(3, 0) SCLET_F64Z(3, 1) SCLET_F64Z(4, 0) SCLET_F64Z(4, 1)
#undef SCLET_F64Z
      default: return cudaErrorInvalidValue;
    }
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_check_soln(const Phys &ph, const T *u, const double *elam, int form, double *partials, int npart,
                              double *out, cudaStream_t s) {
  if (ph.F < 1 || ph.F > MAXF || ph.nac > 4 || ph.nch > 1) return cudaErrorInvalidValue;
  if (ph.runs > 1 && sizeof(T) != 4) return cudaErrorInvalidValue;  // several runs: FP32 states
  cudaError_t e = with_physics(ph.physics, [&](auto *tag) {
    using PL = std::remove_pointer_t<decltype(tag)>;
    return check_soln_pl<PL, T>(ph, u, elam, form, partials, npart, s);
  });
  if (e != cudaSuccess) return e;
  chain_launch(true, energy_final_kernel, dim3(2 * ph.F + 2, ph.runs > 1 ? ph.runs : 1), FT_THREADS, 0, s, ph, form, partials, npart, out);
  launch_counter() += 2;
  return cudaGetLastError();
}

template cudaError_t launch_check_soln<double>(const Phys &, const double *, const double *, int, double *, int, double *,
                                               cudaStream_t);
template cudaError_t launch_check_soln<float>(const Phys &, const float *, const double *, int, double *, int, double *,
                                              cudaStream_t);

}  // namespace sclet
