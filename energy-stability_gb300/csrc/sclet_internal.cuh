// Internal declarations shared by the CUDA translation units of sclet_gb300.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "sclet_gb300.h"

namespace sclet {

// Physics-plugin constants and per-run scalars passed by value to kernels.
struct Phys {
  int n, nac, nch, F;
  int anisotropic, elastic;
  double dt, epn2;
  double h[3];
  double kk[3];
  double lam[4][9];      // F2 tensors: diag(kk) - file tensor, row-major
  double elastic_scale;
  // physics plugin (SCLET_PHYSICS_*) and its constants as the kernels see
  // them (the reference composition shifted by cshift, see below); LE, KE,
  // LCI, KCI from the plugin's init_KL
  int physics;
  double K[16];
  double LE, KE, LCI, KCI;
  // Offset of the stored conserved field: the device holds c - cshift.  The
  // mixed form stores c - c0 (cshift = c0), which keeps FP32 storage and the
  // transforms at the scale of the fluctuations; the scheme is linear in c
  // and the constant state c0 is a fixed point, so this changes nothing in
  // exact arithmetic.  It needs a plugin whose c enters only as c - c0
  // (SCLET_C0_INDEX); 0 otherwise and in the FP64 form.
  double cshift;
  // runs of the same block size held side by side (the batched ensemble):
  // run r's fields are the F blocks at r F n^3; krun (device, runs values,
  // or null) replaces plugin constant 0 per run (the Landau a2)
  int runs;
  const double *krun;
  // launch shape chosen by the autotuner (0: the default)
  int rhs_zc;       // most z-planes per CTA of the Allen-Cahn right-hand side (0: default)
  int tc_ctas;      // persistent CTAs of the tensor-core products
  // variable-mobility Cahn-Hilliard (VariableMobility = 1): M(eta0) =
  // mob_m0 (1 - eta0 + mob_dg eta0) (mobility_constants); device scratch of
  // two blocks per run (mob_t, the precision's type) and of the block maxima
  // of M (mob_part: MOB_PARTS per run, then one C per run)
  int varmob;
  double mob_m0, mob_dg;
  void *mob_t;
  double *mob_part;
};

constexpr int MOB_PARTS = 512;  // partial maxima of M per run
void mobility_constants(double *m0, double *dg);

// Geometry helpers (owned cells are 2 .. n-3 per axis, period N = n - 4).
__host__ __device__ inline int img(int n, int v) {
  int N = n - 4;
  int r = (v - 2) % N;
  if (r < 0) r += N;
  return 2 + r;
}
__host__ __device__ inline int wrap1(int n, int v) {
  int N = n - 4;
  return v < 2 ? v + N : (v >= n - 2 ? v - N : v);
}

// ---- kernel launchers (each returns the launch's cudaError_t) -------------
// Ghost fill of `count` blocks (stride n^3) in place.
template <typename T>
cudaError_t launch_ghost_fill(T *u, int count, int n, cudaStream_t s);
// Ghost cells of the elastic force of every field and run (nac blocks per run
// side by side) by the shared-scratch semantics, see k_halo.cu.  first: no
// previous call.
template <typename T>
cudaError_t launch_elastic_ghosts(T *felas, int nac, int n, cudaStream_t s, int runs, bool first);

// Right-hand sides of all fields into out (F blocks).  felas: nac blocks.
template <typename T>
cudaError_t launch_rhs(const Phys &ph, const T *u, const T *felas, T *out, T *scratch, cudaStream_t s);
int rhs_ac_planes(int n, int tuned, bool tensors, long long tiles, int runs);

// Mode-n product with rotation, FP64: for `count` tensors,
// out_t[a'*n*n + r] = sum_a M[a'*n + a] in_t[r*n + a]  (M row-major).
// Epilogues: 0 store; 1 ETD1 update out = (1 - phi H) uhat + phi * acc with
// uhat = aux_t (read) ; 2 out = phi2 * acc ; 3 out += acc.  Prologue `sub`:
// in_t - sub_t.  kinds: per-tensor field kind selector (t % F >= nac -> CH).
// phi: the tables of the two field kinds (phi1 for epilogue 1, phi2 for 2).
struct EtdCoef {
  const double *dd[3];   // eigenvalues / h^2 per axis (device)
  double kk[3];
  double epn2, dt, LE, KE, LCI, KCI;
  int nac, F;
};
// ---- folded transforms (sclet_basis.cu) -----------------------------------
// half edge of a folded product, and the first mode of each parity
// (part 0 even, part 1 odd about the block's centre; mode k is even when
// n - k is odd)
__host__ __device__ inline int fold_half(int n) { return (n + 1) / 2; }
__host__ __device__ inline int fold_mode0(int n, int part) { return part == 0 ? (n + 1) % 2 : n % 2; }
bool basis_is_dirichlet(int n, const double *d, const double *v, const double *vi);
std::vector<double> fold_matrix(int n, const double *m, bool inverse);

// Chained launches: a kernel of a step may be launched before the one ahead of
// it on the stream has ended.  Its CTAs then wait in chain_wait(), the first
// thing every such kernel does (or all but its set-up in shared memory), until
// that one has ended and its writes are visible, so the order of the work stays
// the stream's; what is saved is the launch latency between two kernels: a step
// of 4 fields of 36^3 154 -> 98 us, of 68^3 194 -> 156 us.
// Not for a kernel whose CTAs are dealt to the SMs once, in equal shares: placed
// while the kernel ahead still holds some SMs, they crowd on the others (the FP64
// products of 68^3 0.59 -> 1.04 ms a step).  Those, and what the FP64 pipe
// bounds, are launched with early = false.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
cudaError_t chain_launch(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         A &&...args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Blocks of a batch that do not lie in one run of memory: tensor t is the
// block t - first of the last segment with first <= t (blocks n^3 apart).
template <typename T>
struct TensorList {
  const T *base[3];
  int first[3];
  __host__ __device__ const T *at(int t, long long n3) const {
    const int s = t >= first[2] ? 2 : (t >= first[1] ? 1 : 0);
    return base[s] + (t - first[s]) * n3;
  }
};
template <typename T>
inline TensorList<T> tensor_list(const T *a) {  // one run of blocks
  return TensorList<T>{{a, a, a}, {0, 0x7fffffff, 0x7fffffff}};
}

// Right-hand side of the increment form of the Allen-Cahn fields (m < nac of
// every run): r = N - H u with H the step's linear operator applied as a
// stencil (zero outside the block), so that u' = u + V phi1 V^-1 r.
// u, rhs: F blocks per run; r: nac blocks per run.
template <typename T>
cudaError_t launch_increment_rhs(const Phys &ph, const T *u, const T *rhs, T *r, cudaStream_t s);

// Folded FP64 products of `count` tensors (layout rotation as in
// launch_modeprod_f64).  W: fold_matrix of V^-1 (forward) or V (inverse).
// Forward epilogue: phi[kind] (n^3, may be null: plain store) times the value
// for tensors t < scaled, a plain store for the others; etd: tensor t is N^ of
// field t + t0 and out holds its u^, updated in place (1 - phi1 H) u^ + phi1 N^.
// Inverse: out += for tensors with t % F < acc, a store for the others.
struct FoldEpi {
  const double *phi[2];
  int scaled, etd, t0;
};
cudaError_t launch_fold_fwd_f64(const double *W, const TensorList<double> &in, const double *sub, double *out, int count,
                                int n, const FoldEpi &ep, const EtdCoef &ec, cudaStream_t s);
cudaError_t launch_fold_inv_f64(const double *W, const double *in, double *out, int count, int n, int F, int acc,
                                cudaStream_t s);

cudaError_t launch_modeprod_f64(const double *M, const double *in, const double *sub, double *out,
                                const double *aux, int count, int n, int epilogue, const EtdCoef &ec,
                                long long in_stride, long long out_stride, cudaStream_t s,
                                const double *const *phi = nullptr);

// Elastic force (FFT based) -- see k_fft.cu.
struct ElasticPlan;
cudaError_t elastic_plan_create(ElasticPlan **plan, int big_n, int nac, const double *voigt,
                                const double *eps, int fp32, cudaStream_t s, int runs = 1);
void elastic_plan_destroy(ElasticPlan *plan);
// felas (nac blocks of n^3) from the AC fields u (first nac blocks).
// runs (the plan's): run r's order parameters at u + r ustride, its force at
// felas + r nac n^3
template <typename T>
cudaError_t elastic_compute(ElasticPlan *plan, const T *u, T *felas, int n, cudaStream_t s, long long ustride = 0);

// Diagnostics: out (F*4 doubles, device) per field max, min, vol, energy.
template <typename T>
cudaError_t launch_check_soln(const Phys &ph, const T *u, const double *elam, int form, double *partials,
                              int npart, double *out, cudaStream_t s);
int check_soln_partials(int n);

// Conserved-field mass of the mixed form (see k_mass.cu).  Weight `which`
// (0 E, 1 phi1, 2 phi2) into w (n^3 slots of 8 bytes: computed in FP64, then
// stored as FP32 (hi, lo) pairs) using tmp (n^3 doubles); g (n) and viT
// (n x n row-major, or folded: its fold_matrix) on the device.
cudaError_t mass_weight(double *w, double *tmp, const double *g, const double *viT, int n, int which,
                        const EtdCoef &ec, cudaStream_t s, bool folded);
int mass_partials();
// part (2 * mass_partials()) = partial sums of wa.a (owned sum of a if wa is
// null) + wb.(b - bsub); wa, wb hold the weight pairs of mass_weight
cudaError_t mass_target(const float *a, const double *wa, const float *b, const float *bsub, const double *wb, int n,
                        double *part, cudaStream_t s);
// shifts the owned cells of u so that their sum meets the target partials;
// mass_shift: apart holds that sum's partials already
cudaError_t mass_fix(float *u, int n, const double *tpart, double *apart, double *res, cudaStream_t s);
cudaError_t mass_shift(float *u, int n, const double *tpart, const double *apart, double *res, cudaStream_t s);
// The parts of `count` blocks after three inverse products (TcArgs::acc), block b
// at u + b stride, -> the fields, in place; apart (of one block, may be null): the
// partial sums of its owned cells as mass_fix forms them.
cudaError_t launch_unfold(float *u, int n, int count, long long stride, double *apart, cudaStream_t s);

// 16-bit codes of one field block (see k_codec.cu); kind 0 AC, 1 CH; the
// stored values plus shift are the field's values.
template <typename T>
cudaError_t launch_field_u16(const T *u, int kind, double shift, long long cells, unsigned short *out, cudaStream_t s);

// Counts kernel launches issued by this library (per process).
long long &launch_counter();

}  // namespace sclet
