// Kernels of the learned coarse-step corrector: a periodic 3x3x3 convolution
// network on BF16 activations with FP32 accumulation.
//
// Activation layout (sclet_conv.cuh, conv_at): chunk-planar.  A sample is
// Np = N + 2 haloed planes (the N^3 periodic grid plus one periodic image
// layer per side); a plane holds 4 chunks of 8 channels, each chunk the
// plane's Np^2 cells (slot = yh Np + xh, 16 bytes each) padded to a multiple
// of 8 slots.
//
// conv_tc_kernel is an implicit GEMM on the 5th-generation tensor cores:
//   D[cell][co] = sum_{tap, ci} A[cell + off(tap)][ci] * W[tap][co][ci]
// with M = 128 cells, N = 32 output channels and K = 27 taps x 32 input
// channels.  A tile is 128 consecutive slots of one haloed plane.  For every
// plane and every chunk, the rows all nine in-plane taps read are one
// contiguous run of 128 + 2 Np + 2 slots (whole 128-byte lines, one TMA box), and
// every tap's operand is a descriptor into it (no-swizzle K-major layout: rows
// 16 bytes apart, the chunks of a K step a box apart), offset by dy Np + dx
// rows.
//
// Reading the 128 x 16 input operand from shared memory, not multiplying it by
// 32 columns, is what an MMA of this shape costs (63 cycles against 16).  So a
// CTA marches its column of tiles in z and takes the planes one by one: each
// operand of a plane serves three MMAs, into the tiles before, at and behind the
// plane, read once through the A collector (one MMA of N = 96 into adjoining
// accumulators was slower: 96 us a layer against 87).  A tile still sums its taps in
// the order dz, dy, dx, K step (the order of the FP32 sums decides the BF16
// roundings of all later layers), and each plane is loaded once.
//
// Slots in the x- or y-halo produce outputs that are dropped.  The weights
// (27 x 32 x 32 BF16, 54 KB) stay in shared memory.  Warp 0 issues TMA, warp 1
// the MMAs into eight 32-column TMEM accumulators, warps 2-5 and 6-9 drain
// alternate tiles and run the fused epilogue (bias, ReLU, residual, ReLU-mask,
// FP32 planar output); cells on the grid's faces are also stored at their
// periodic images, so no halo pass follows.  The same kernel computes the data
// gradient of a convolution with the weights flipped and transposed (the
// adjoint of a periodic convolution).  A layer of 4 x 64^3 with its halo: 124 us
// with three planes loaded per tile and a tap per operand read, 104 us with the
// MMAs issued by a uniform warp, 84 us now.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#include "sclet_internal.cuh"
#include "sclet_tc.cuh"
#include "sclet_tc_ptx.cuh"
#include "sclet_conv_tc.cuh"

namespace sclet {
namespace conv {

using tc::fence_after;
using tc::fence_before;
using tc::mbar_arrive;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::elect_one;
using tc::mma_bf16_from;
using tc::mma_commit_from;
using tc::smem_desc;
using tc::smem_u32;
using tc::tmem_ld32;

constexpr int WTILE = CH * CH * 2;         // 2 KB: one tap's 32 x 32 weights
constexpr int NACC = 8;                    // TMEM accumulators of 32 columns
constexpr int TMEM_COLS = NACC * CH;       // 256
constexpr int SETS = 2;                    // groups of four epilogue warps
constexpr int THREADS = 64 + 128 * SETS;
constexpr int MAX_RING = 6;                // planes in flight, at least two

// Per-launch geometry.  ny = 1: per plane and channel chunk one run of
// 128 + 2 Np + 2 slots serves all nine in-plane taps; ny = 3: one run of 130
// slots per stencil row (where two planes of the long runs do not fit).  A run is one box of
// box_rows lines of 128 bytes (8 slots), enough from any slot offset within
// the first line.
struct Geom {
  int ny, box_rows, box_bytes, plane_bytes, ring, smem;
};
static Geom geom_for(int N, int ny) {
  Geom g;
  g.ny = ny;
  const int R = ny == 1 ? ROWS + 2 * (N + 2) + 2 : ROWS + 2;
  g.box_rows = (R + 7 + 7) / 8;
  g.box_bytes = g.box_rows * 128;
  g.plane_bytes = 4 * ny * g.box_bytes;
  g.ring = (SMEM_LIMIT - 1024 - TAPS * WTILE) / g.plane_bytes;
  if (g.ring > MAX_RING) g.ring = MAX_RING;
  g.smem = TAPS * WTILE + g.ring * g.plane_bytes + 1024;
  return g;
}
std::atomic<int> g_runs_per_plane{0};  // 0: by N; 1 or 3: forced (sclet_net_set_conv_runs)
static Geom geom_of(int N) {
  const Geom a = geom_for(N, 1), b = geom_for(N, 3);
  return a.ring >= 2 && a.box_rows <= 256 && g_runs_per_plane.load() != 3 ? a : b;
}

template <bool B>
struct Flag {
  static constexpr bool value = B;
};

// tile t of a launch: z fastest, so that consecutive tiles march a column
struct ZTile {
  int b, zh, s0;  // sample, plane 1..N, first slot of the plane
};
__device__ __forceinline__ ZTile ztile_of(int t, int N, int Np, int per_plane) {
  ZTile x;
  const int col = t / N;
  x.zh = 1 + t - col * N;
  x.b = col / per_plane;
  x.s0 = Np + (col - x.b * per_plane) * ROWS;
  return x;
}

__device__ __forceinline__ float bf(uint32_t w, int hi) {
  return __uint_as_float(hi ? (w & 0xffff0000u) : (w << 16));
}

__global__ void __launch_bounds__(THREADS, 1)
    conv_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, ConvArgs g,
                   Geom gm) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_RING];
  __shared__ __align__(8) uint64_t empty_bar[MAX_RING];
  __shared__ __align__(8) uint64_t tfull_bar[NACC];
  __shared__ __align__(8) uint64_t tempty_bar[NACC];
  __shared__ __align__(8) uint64_t w_bar;
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;
  __shared__ float s_bias[CH];

  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *wsm = base;                    // 27 tap tiles of weights
  uint8_t *ring = base + TAPS * WTILE;    // gm.ring planes of 4 ny runs
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int N = g.N, Np = N + 2, ny = gm.ny;
  const int per_plane = (N * Np + ROWS - 1) / ROWS;
  const int total = g.batch * N * per_plane;
  // a contiguous range of tiles per CTA
  const int t0 = (int)((long long)total * blockIdx.x / gridDim.x);
  const int t1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);

  if (threadIdx.x < CH) s_bias[threadIdx.x] = g.bias ? g.bias[threadIdx.x] : 0.0f;
  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_RING; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < NACC; b++) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 4);
    }
    mbar_init(&w_bar, 1);
    mbar_init(&done_bar, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;

  // The launch is early (chain_launch): the weights, which no kernel since the
  // input's packing wrote, load while the layer ahead ends.  A forward pass of
  // 4 x 64^3 873 -> 850 us.
  if (warp == 0 && lane == 0) {
    mbar_expect_tx(&w_bar, TAPS * WTILE);
    for (int t = 0; t < TAPS; t++) tma_load_2d(wsm + t * WTILE, &tmW, 0, t * CH, &w_bar);
  }
  chain_wait();
  if (warp == 0) {
    if (lane == 0) {
      int q = 0;  // planes loaded
      for (int t = t0; t < t1 && !*(volatile int *)&failed;) {
        // the tiles of one column: planes zh - 1 of the first .. zh + 1 of the last
        const ZTile ti = ztile_of(t, N, Np, per_plane);
        const int len = min(t1 - t, N + 1 - ti.zh);
        for (int z = ti.zh - 1; z <= ti.zh + len; z++, q++) {
          const int s = q % gm.ring;
          if (q >= gm.ring && !mbar_wait(&empty_bar[s], ((q / gm.ring) & 1) ^ 1)) {
            failed = 1;
            break;
          }
          if (*(volatile int *)&failed) break;
          mbar_expect_tx(&full_bar[s], gm.plane_bytes);
          // the run from slot s0 - Np - 1 (ny = 1) or s0 + (r - 1) Np - 1 (ny = 3),
          // >= -1; a line before the buffer or past its end reads as zeros
          for (int r = 0; r < ny; r++)
            for (int k = 0; k < 4; k++) {
              const long long first = (long long)ti.s0 + (r - 1) * Np - 1;
              const long long flat = conv_at(N, ti.b, z, k, first);
              tma_load_2d(ring + s * gm.plane_bytes + (r * 4 + k) * gm.box_bytes, &tmA, 0, (int)(flat >> 3),
                          &full_bar[s]);
            }
        }
        t += len;
      }
      if (*(volatile int *)&failed) {
        for (int i = q - gm.ring < 0 ? 0 : q - gm.ring; i < q; i++) mbar_wait(&full_bar[i % gm.ring], (i / gm.ring) & 1);
      }
      mbar_wait(&w_bar, 0);
    }
  } else if (warp == 1) {
    // the warp runs the loop together, one lane issues (mma_bf16_from)
    const bool issue = elect_one();
    const uint32_t idesc = tc::idesc_bf16(ROWS, CH);
    bool ok = __all_sync(0xffffffffu, mbar_wait(&w_bar, 0));
    fence_after();
    // descriptors: constant high words; a tap adds its run and row offsets
    // (16-byte units) to the low word's address field
    const uint64_t da0 = smem_desc_lin(smem_u32(ring), gm.box_bytes, 128), dw0 = smem_desc(smem_u32(wsm));
    const uint32_t a_hi = (uint32_t)(da0 >> 32), w_hi = (uint32_t)(dw0 >> 32), w_lo = (uint32_t)dw0;
    const uint32_t run16 = (uint32_t)gm.box_bytes >> 4;
    int q = 0;  // planes seen
    for (int t = t0; ok && t < t1;) {
      const ZTile ti = ztile_of(t, N, Np, per_plane);
      const int len = min(t1 - t, N + 1 - ti.zh), it0 = t - t0;
      // per stencil row dy: the run holding it and the row of dx = -1 within it
      uint32_t rofs[3];
#pragma unroll
      for (int dy = 0; dy < 3; dy++) {
        const uint32_t first = (uint32_t)(ti.s0 + (ny == 1 ? -Np : (dy - 1) * Np) - 1);
        rofs[dy] = (uint32_t)da0 + (ny == 1 ? 0u : (uint32_t)(dy * 4) * run16) + (first & 7) +
                   (ny == 1 ? (uint32_t)(dy * Np) : 0u);
      }
      // plane j of the column's len + 2 is stencil plane dz of its tile j - dz
      for (int j = 0; j < len + 2; j++, q++) {
        const int s = q % gm.ring;
        // tile j starts here: its accumulator must be drained
        if (j < len && it0 + j >= NACC) ok = mbar_wait(&tempty_bar[(it0 + j) % NACC], (((it0 + j) / NACC) & 1) ^ 1);
        ok = __all_sync(0xffffffffu, ok && mbar_wait(&full_bar[s], (q / gm.ring) & 1));
        if (!ok) break;
        fence_after();
        const uint32_t pz = (uint32_t)(s * gm.plane_bytes) >> 4;
        const uint32_t acc0 = tmem + (uint32_t)((it0 + j) % NACC * CH);                // dz = 0
        const uint32_t acc1 = tmem + (uint32_t)((it0 + j + NACC - 1) % NACC * CH);     // dz = 1
        const uint32_t acc2 = tmem + (uint32_t)((it0 + j + 2 * NACC - 2) % NACC * CH); // dz = 2
        auto plane = [&](auto inner) {
          constexpr bool INNER = decltype(inner)::value;
          const bool v0 = issue && (INNER || j < len), v1 = issue && (INNER || (j >= 1 && j <= len));
          const bool v2 = issue && (INNER || j >= 2);
#pragma unroll
          for (int dy = 0; dy < 3; dy++) {
#pragma unroll
            for (int dx = 0; dx < 3; dx++) {
#pragma unroll
              for (int ks = 0; ks < 2; ks++) {
                const uint32_t a_lo = rofs[dy] + pz + (uint32_t)(2 * ks) * run16 + (uint32_t)dx;
                const uint32_t w = w_lo + (uint32_t)(((dy * 3 + dx) * WTILE + ks * 32) >> 4);
                constexpr uint32_t DZ = (uint32_t)(9 * WTILE) >> 4;
                mma_bf16_from<INNER ? tc::A_FILL : tc::A_DROP>(v0, acc0, a_lo, a_hi, w, w_hi, idesc,
                                                               (dy == 0 && dx == 0 && ks == 0) ? 0u : 1u);
                mma_bf16_from<INNER ? tc::A_USE : tc::A_DROP>(v1, acc1, a_lo, a_hi, w + DZ, w_hi, idesc, 1u);
                mma_bf16_from<INNER ? tc::A_LAST : tc::A_DROP>(v2, acc2, a_lo, a_hi, w + 2 * DZ, w_hi, idesc, 1u);
              }
            }
          }
        };
        // within the column all three tiles exist; at its ends the operand is
        // read for each MMA (a collector is not used unless it was filled)
        if (j >= 2 && j < len) plane(Flag<true>());
        else plane(Flag<false>());
        mma_commit_from(issue, &empty_bar[s]);
        if (j >= 2) mma_commit_from(issue, &tfull_bar[(it0 + j - 2) % NACC]);
        ok = !__any_sync(0xffffffffu, *(volatile int *)&failed);
        if (!ok) break;
      }
      t += len;
    }
    if (!ok && lane == 0) failed = 1;
    mma_commit_from(issue, &done_bar);
    if (!mbar_wait(&done_bar, 0) && lane == 0) failed = 1;
  } else {
    const int q = warp & 3, set = (warp - 2) >> 2;
    for (int t = t0 + set, j = 0; t < t1; t += SETS, j++) {
      const int it = t - t0, b = it % NACC;
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&tfull_bar[b], (it / NACC) & 1) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) failed = 1;
        break;
      }
      fence_after();
      float acc[CH];
      tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * CH), acc);
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[b]);
      const ZTile ti = ztile_of(t, N, Np, per_plane);
      const int s = ti.s0 + q * 32 + lane;
      const int yh = s / Np, xh = s - yh * Np;
      if (yh >= 1 && yh <= N && xh >= 1 && xh <= N) {
        const long long cell0 = conv_at(N, ti.b, ti.zh, 0, s), cstride = conv_chunk_slots(N);  // chunk k: cell0 + k cstride
        if (g.mode == CONV_OUT_F32) {
          // FP32 planar output of the first `cout` channels (owned cells)
          const long long n3 = (long long)N * N * N;
          const long long own = ((long long)(ti.zh - 1) * N + (yh - 1)) * N + (xh - 1);
          float *o = g.outf + (long long)ti.b * g.cout * n3 + own;
#pragma unroll
          for (int c = 0; c < CH; c++)
            if (c < g.cout) o[c * n3] = (acc[c] + s_bias[c]) * g.scale;
        } else {
          float v[CH];
          if (g.mode == CONV_RELU) {
#pragma unroll
            for (int c = 0; c < CH; c++) v[c] = fmaxf(acc[c] + s_bias[c], 0.0f);
          } else if (g.mode == CONV_LINEAR) {
#pragma unroll
            for (int c = 0; c < CH; c++) v[c] = acc[c] + s_bias[c];
          } else {
            const uint4 *src = reinterpret_cast<const uint4 *>(g.aux);
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const uint4 w = src[cell0 + k * cstride];
              const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
              for (int h = 0; h < 8; h++) {
                const int c = k * 8 + h;
                const float a = bf(ww[h >> 1], h & 1);
                v[c] = g.mode == CONV_RESIDUAL ? a + (acc[c] + s_bias[c]) : (a > 0.0f ? acc[c] : 0.0f);
              }
            }
          }
          uint4 *dst = reinterpret_cast<uint4 *>(g.out);
          uint4 val[4];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; h++) {
              const __nv_bfloat162 p = __floats2bfloat162_rn(v[k * 8 + 2 * h], v[k * 8 + 2 * h + 1]);
              w[h] = *reinterpret_cast<const uint32_t *>(&p);
            }
            val[k] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[cell0 + k * cstride] = val[k];
          }
          // a cell on a face: its periodic images in the halo, one per subset
          // of the axes it is extreme on, at fixed distances from the cell
          const int sz = ti.zh == 1 ? 1 : ti.zh == N ? -1 : 0, sy = yh == 1 ? 1 : yh == N ? -1 : 0;
          const int sx = xh == 1 ? 1 : xh == N ? -1 : 0;
          if (sz | sy | sx) {
            const long long dz = 4LL * N * cstride * sz, dy = (long long)N * Np * sy, dx = (long long)N * sx;
#pragma unroll
            for (int m = 1; m < 8; m++) {
              if (((m & 1) && !sz) || ((m & 2) && !sy) || ((m & 4) && !sx)) continue;
              uint4 *im = dst + cell0 + (m & 1 ? dz : 0) + (m & 2 ? dy : 0) + (m & 4 ? dx : 0);
#pragma unroll
              for (int k = 0; k < 4; k++) im[k * cstride] = val[k];
            }
          }
        }
      }
      if (__any_sync(0xffffffffu, *(volatile int *)&failed != 0)) break;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && failed) atomicExch(g.err, 1);
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}


// 2-D BF16 tensor map with 64-byte swizzle: rows of 32 channels (64 B),
// `rows` rows, boxes of 32 x box_rows.
static cudaError_t make_map_rows(CUtensorMap *map, const void *ptr, long long rows, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)CH, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)CH * 2};
  cuuint32_t box[2] = {(cuuint32_t)CH, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// per device: the shared-memory attribute and the resident CTA count
static cudaError_t conv_setup(int *ctas) {
  constexpr int MAXDEV = 64;
  static std::mutex mu;
  static int resident[MAXDEV] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= MAXDEV) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (!resident[dev]) {
    e = cudaFuncSetAttribute(conv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, conv_tc_kernel, THREADS, SMEM_LIMIT);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    resident[dev] = per_sm * sms;
  }
  *ctas = resident[dev];
  return cudaSuccess;
}

}  // namespace conv

int conv_set_runs(int runs_per_plane) {
  if (runs_per_plane != 0 && runs_per_plane != 1 && runs_per_plane != 3) return -1;
  return conv::g_runs_per_plane.exchange(runs_per_plane);
}

int conv_runs() { return conv::g_runs_per_plane.load(); }

cudaError_t launch_conv(const __nv_bfloat16 *in, const __nv_bfloat16 *w, const ConvArgs &args, cudaStream_t s) {
  int ctas = 0;
  cudaError_t e = conv::conv_setup(&ctas);
  if (e != cudaSuccess) return e;
  const int N = args.N, Np = N + 2;
  if (N < 2 || args.batch < 1) return cudaErrorInvalidValue;
  const conv::Geom gm = conv::geom_of(N);
  if (gm.ring < 2 || gm.box_rows > 256) return cudaErrorInvalidValue;
  const long long lines = conv_units(N, args.batch) / 8;
  if (lines >= 0x7fffffffLL) return cudaErrorInvalidValue;
  CUtensorMap ma, mw;
  if ((e = conv::make_map_lines(&ma, in, lines, gm.box_rows)) != cudaSuccess) return e;
  if ((e = conv::make_map_rows(&mw, w, (long long)TAPS * CH, CH)) != cudaSuccess) return e;
  const long long per_plane = ((long long)N * Np + conv::ROWS - 1) / conv::ROWS;
  const long long tiles = (long long)args.batch * N * per_plane;
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;
  const int grid = (int)(tiles < ctas ? tiles : ctas);
  chain_launch(true, conv::conv_tc_kernel, grid, conv::THREADS, gm.smem, s, ma, mw, args, gm);
  launch_counter()++;
  return cudaGetLastError();
}

}  // namespace sclet
