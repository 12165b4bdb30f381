// Declarations of the tensor-core (tcgen05) mode-n product, see k_modeprod_tc.cu.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "sclet_internal.cuh"

namespace sclet {

constexpr int TC_PLANES = 4;    // fixed-point slices per data operand (tc_slice_bits each)
constexpr int TC_PLANES_M = 5;  // slices per matrix: four of tc_slice_bits and a fifth, stored
                                // pre-scaled by 2^-bits (see k_modeprod_tc.cu)
constexpr int TC_BM = 128;      // lines per tile of input slices
constexpr int TC_BK = 32;       // columns per k-block

struct TcArgs {
  int n, kblocks, count;
  int bits;                 // slice width (set by launch_modeprod_tc)
  int form;                 // 0 any basis, 1 folded forward, 2 folded inverse product
  int epi;                  // 0 none, 1 ETD1 update (aux = uhat), 2 phi scaling
  int outmode;              // 1 FP32 store, 2 FP32 accumulate
  int acc;                  // form 2: fields t % F < acc are increments (outmode 2 accumulates them); of the
                            // others E and O are stored, for launch_unfold
  const float *aux;         // [count][n^3] FP32 uhat, same layout as out
  float *out;               // [count][n^3] FP32, rotated layout
  const float *in_scale;    // [count][n*n] power-of-two scale of each input row's slices ([count][2][n*n] folded)
  const float *row_scale;   // [n] power-of-two scale of each matrix row's slices ([2][h] folded)
  // per field kind (0 AC, 1 CH), per eigen-mode [k][j][i]: ETD1
  // (e = 1 - phi1 H, phi1) and ETD2 (phi2) coefficients computed in FP64
  // (ac_init_phi / ch_init_phi, vars.c:302-359) as hi + lo FP32 pairs
  const float4 *coef[2];
  const float2 *coef2[2];
  int nac, F;
  int *err;                 // set to 1 when a bounded wait gives up
  int max_ctas;             // persistent CTAs (0: as many as can be resident)
  int idle;                 // 1: the producer issues no loads (the bounded-wait self-test)
};

// kp = n rounded up to whole k-blocks of 32.  Slices are stored in the tiles the
// product kernel loads, each one contiguous run (see k_modeprod_tc.cu): input
// slices [part][r / 128][kp / 32][p][128][32], matrix slices
// [part][a' / bn][kp / 32][p][bn][32], columns n .. kp - 1 and rows beyond the
// last one zero.
int tc_kp(int n);
int tc_slice_bits(int n);
// a'-tile width (bn) of a contraction of length h
int tc_bn(bool folded, int h);
// elements of one tensor's slices and of one matrix's, both parts where folded
long long tc_plane_elems(int n, bool folded);
long long tc_matrix_elems(int n, bool folded);
// One part of a matrix: row-major FP64 n x n -> its TC_PLANES_M slices in
// a'-tiles of bn and the power-of-two scale of each row.
cudaError_t tc_slice_matrix(const double *m, __nv_bfloat16 *planes, float *row_scale, int n, int bn, cudaStream_t s);
// FP32 blocks (x - sub; sub may be null), rows of n -> slices with the
// power-of-two scale of each row in scale[count][n*n]; the pad columns and rows
// are never written (zero from allocation).
cudaError_t tc_slice_fields(const float *x, const float *sub, float *scale, __nv_bfloat16 *planes, int n, int count,
                            cudaStream_t s);
// The update of the eigen-modes done where they are sliced for the inverse
// transform: tensors t < nI are multiplied by phi (hi, lo pairs of their
// field kind); the others are u^ and become e u^ + phi1 N^, their N^ the block
// count - nI blocks on (etd: (e, phi1) pairs as TcArgs::coef).
struct SpecUpdate {
  const float2 *phi[2] = {nullptr, nullptr};
  const float4 *etd[2] = {nullptr, nullptr};
  int nI = 0, F = 1, nac = 0;
};
// Lines -> the slices of their two parity parts (see slice_fold_kernel), kp =
// tc_kp(fold_half(n)), scales [count][2][n*n]; forward: x - sub folded (sub may be null), else split by
// mode after the update sp (may be null)
cudaError_t tc_slice_fold(bool forward, const TensorList<float> &x, const float *sub, const SpecUpdate *sp, float *scale,
                          __nv_bfloat16 *planes, int n, int count, cudaStream_t s);
// ETD coefficient tables of one field kind (see TcArgs::coef); null ones are left out
cudaError_t tc_make_coefs(float4 *coef, float2 *phi1, float2 *coef2, int n, int kind, const double *dx, const double *dy,
                          const double *dz, const double *kk, double epn2, double dt, double L, double K,
                          cudaStream_t s);
// out[t] = mat x in[t] (contracting the row axis, rotating), count tensors
cudaError_t launch_modeprod_tc(const __nv_bfloat16 *mat, const __nv_bfloat16 *planes, int count, const TcArgs &args,
                               cudaStream_t s);

}  // namespace sclet
