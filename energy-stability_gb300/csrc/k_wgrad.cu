// Weight gradient of the corrector's 3x3x3 convolutions on the 5th-generation
// tensor cores:
//   dW[tap][co][ci] += sum over owned cells of g[cell][co] x[cell + off(tap)][ci]
//   db[co]          += sum over owned cells of g[cell][co]
// A GEMM whose contraction runs over the cells.  A tile is 128 consecutive
// slots of one haloed plane (as in k_conv.cu).  The activation layout
// (chunk-planar, 8 channels of a cell in 16 bytes, consecutive cells 16 bytes
// apart) is the MN-major operand layout as it lies in memory, so both
// operands go from TMA to the MMA without a transpose, and a tap is an offset
// of the operand's start address.
//   M = 128: the three stencil planes dz x 32 input channels (twelve runs, a
//       run apart), then one run of ones, whose row sums g: the bias gradient
//   N = 32 output channels, from one of three copies of the gradient, shifted by
//       the dx taps; K = the tile's 128 slots in steps of 16
// (dx moved to the gradient: sum_c g[c] x[c + dx] = sum_c' g[c' - dx] x[c'].)
// What such MMAs cost is reading their operands from shared memory: the three dx
// of one input operand read it once, through the A collector.  The nine in-plane
// taps have 32 accumulator columns each in tensor memory, drained into FP32
// registers after every tile with round-to-nearest adds, a stencil row's three
// taps by four warps while the other rows' MMAs run: the accumulator itself
// rounds toward zero, so its eight accumulations are all that may carry that.
// (Drained every eight tiles a layer of 4 x 64^3 took 98 us for 108, but sums of one
// sign were low by 1.2e-6 and those of either sign 1.5 times as far off as with
// FP32 FMAs.  Now, relative to the gradient's norm, FP32 FMAs and this: 4 x 64^3
// 4.8e-7 and 2.7e-7, one sign 2.2e-7 and 1.8e-7; 112^3 5.9e-7 and 2.9e-7, one sign
// 2.5e-7 and 2.1e-7.)  Each CTA adds its sums to the gradient once, at the end.
// Warp 0 issues TMA, warp 1 the MMAs, warps 2-3 write the gradient's shifted
// copies with the slots outside the owned cells cleared (the halo holds periodic
// images, which the data gradient needs), warps 4-15 drain.
//
// A layer on 4 x 64^3: 2.22 ms as an FP32-issue kernel, 0.11 ms now.
#include <mutex>

#include "sclet_conv_tc.cuh"
#include "sclet_internal.cuh"

namespace sclet {
namespace conv {
namespace wg {

using namespace tc;

constexpr int TAPS2 = 9;                    // in-plane taps, 32 accumulator columns each
constexpr int G_ROWS = (ROWS + 2 + 7 + 7) / 8;  // 128-byte lines of one gradient run (130 slots)
constexpr int G_BYTES = G_ROWS * 128;
constexpr int S_BYTES = ROWS * 16;          // one chunk of a shifted copy
constexpr int SHIFTERS = 2;                 // warps writing the shifted copies
constexpr int EPI = 12;                     // draining warps, three per TMEM lane quadrant
constexpr int TAPS_PER_WARP = TAPS2 / 3;
constexpr int WG_THREADS = 32 * (2 + SHIFTERS + EPI);
constexpr int WG_TMEM = 512;                // 288 columns used; allocations are powers of two

// Runs of the input per stage as in k_conv.cu's ny: 1 one run of 128 + 2 Np
// slots per plane and chunk, 3 one run of 128 slots per stencil row.  A stage:
// for each of ny rows the twelve runs (dz, chunk) and the ones run (three run
// lengths more are read as rows 104..127 of M and dropped: they overlay what
// follows), the four gradient runs as they lie, and their twelve shifted
// copies.
struct Geom {
  int ny, box_rows, box_bytes, row_bytes, stage_bytes, stages, smem;
};
static Geom geom_for(int N, int ny) {
  Geom g;
  g.ny = ny;
  const int R = ny == 1 ? ROWS + 2 * (N + 2) : ROWS;
  g.box_rows = (R + 7 + 7) / 8;
  g.box_bytes = g.box_rows * 128;
  g.row_bytes = 13 * g.box_bytes;
  g.stage_bytes = ny * g.row_bytes + 4 * G_BYTES + 12 * S_BYTES;
  const int tail = 3 * g.box_bytes + 128;  // the dropped rows' reads past the last stage
  g.stages = (SMEM_LIMIT - 1024 - tail) / g.stage_bytes;
  if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
  g.smem = (g.stages > 0 ? g.stages : 1) * g.stage_bytes + tail + 1024;
  return g;
}

// SPLIT: drains of an accumulator per tile
template <int SPLIT>
__global__ void __launch_bounds__(WG_THREADS, 1)
    wgrad_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmG, int N, int batch,
                    float *__restrict__ dw, float *__restrict__ db, int *err, Geom gm) {
  constexpr int KSTEPS = ROWS / 16 / SPLIT;  // accumulations between drains
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t ready_bar[MAX_STAGES];  // shifted copies written
  __shared__ __align__(8) uint64_t empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[3], acc_empty[3];  // per stencil row: three taps' accumulators
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int Np = N + 2, ny = gm.ny, stages = gm.stages;
  const int per_plane = (N * Np + ROWS - 1) / ROWS;
  const int total = batch * N * per_plane;
  const int mine = (int)blockIdx.x < total ? (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int g_off = ny * gm.row_bytes, s_off = g_off + 4 * G_BYTES;  // gradient runs and shifted copies of a stage

  // shared memory starts as zeros, the ones runs as ones: what the dropped
  // rows read is initialised too
  {
    const int n16 = (stages * gm.stage_bytes + 3 * gm.box_bytes + 128) / 16;
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < n16; i += WG_THREADS) reinterpret_cast<uint4 *>(base)[i] = z;
    __syncthreads();
    const uint32_t one2 = 0x3f803f80u;  // two BF16 ones
    const int per = gm.box_bytes / 16;
    for (int i = threadIdx.x; i < stages * ny * per; i += WG_THREADS) {
      const int r = i / per, q = i - r * per, s = r / ny, y = r - s * ny;
      reinterpret_cast<uint4 *>(base + s * gm.stage_bytes + y * gm.row_bytes + 12 * gm.box_bytes)[q] =
          make_uint4(one2, one2, one2, one2);
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&ready_bar[s], SHIFTERS);
      mbar_init(&empty_bar[s], 1);
    }
    for (int dy = 0; dy < 3; dy++) {
      mbar_init(&acc_full[dy], 1);
      mbar_init(&acc_empty[dy], EPI / 3);
    }
    mbar_init(&done_bar, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(WG_TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;
  chain_wait();

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (; it < mine && !*(volatile int *)&failed; it++) {
        const Tile ti = tile_of(blockIdx.x + it * gridDim.x, N, Np, per_plane);
        const int s = it % stages;
        if (it >= stages && !mbar_wait(&empty_bar[s], ((it / stages) & 1) ^ 1)) {
          failed = 1;
          break;
        }
        uint8_t *st = base + s * gm.stage_bytes;
        mbar_expect_tx(&full_bar[s], 12 * ny * gm.box_bytes + 4 * G_BYTES);
        for (int r = 0; r < ny; r++)
          for (int dz = 0; dz < 3; dz++)
            for (int k = 0; k < 4; k++) {
              const long long first = (long long)ti.s0 + (ny == 1 ? -Np : (r - 1) * Np);
              const long long flat = conv_at(N, ti.b, ti.zh + dz - 1, k, first);
              tma_load_2d(st + r * gm.row_bytes + (dz * 4 + k) * gm.box_bytes, &tmX, 0, (int)(flat >> 3), &full_bar[s]);
            }
        for (int k = 0; k < 4; k++)
          tma_load_2d(st + g_off + k * G_BYTES, &tmG, 0, (int)(conv_at(N, ti.b, ti.zh, k, ti.s0 - 1) >> 3), &full_bar[s]);
      }
      if (*(volatile int *)&failed)  // drain (bounded) the copies still in flight
        for (int i = it - stages < 0 ? 0 : it - stages; i < it; i++) mbar_wait(&full_bar[i % stages], (i / stages) & 1);
    }
  } else if (warp == 1) {
    // the warp runs the loop together, one lane issues (mma_bf16_from)
    const bool issue = elect_one();
    const uint32_t idesc = idesc_bf16(ROWS, CH) | (1u << 15) | (1u << 16);  // both operands MN-major
    const uint64_t dg0 = smem_desc_lin(smem_u32(base) + s_off, 128, S_BYTES);
    const uint64_t dx0 = smem_desc_lin(smem_u32(base), 128, gm.box_bytes);
    const uint32_t g_hi = (uint32_t)(dg0 >> 32), x_hi = (uint32_t)(dx0 >> 32);
    bool ok = true;
    for (int it = 0; it < mine && ok; it++) {
      const int s = it % stages;
      ok = __all_sync(0xffffffffu, mbar_wait(&ready_bar[s], (it / stages) & 1));
      if (!ok) break;
      fence_after();
      const Tile ti = tile_of(blockIdx.x + it * gridDim.x, N, Np, per_plane);
      const uint32_t st = (uint32_t)(s * gm.stage_bytes >> 4);
      for (int part = 0; part < SPLIT && ok; part++) {
        const int use = it * SPLIT + part;  // of each stencil row's accumulators
#pragma unroll
        for (int dy = 0; dy < 3; dy++) {
          if (use > 0) ok = ok && mbar_wait(&acc_empty[dy], (use - 1) & 1);
          ok = __all_sync(0xffffffffu, ok);
          fence_after();
          // the run holding stencil row dy and its first slot within it
          const uint32_t first = (uint32_t)(ti.s0 + (ny == 1 ? -Np : (dy - 1) * Np));
          const uint32_t x_lo = (uint32_t)dx0 + st + (ny == 1 ? 0u : (uint32_t)(dy * gm.row_bytes) >> 4) + (first & 7) +
                                (ny == 1 ? (uint32_t)(dy * Np) : 0u);
#pragma unroll
          for (int k = 0; k < KSTEPS; k++) {
            // one input operand, the three dx
            const uint32_t acc = tmem + (uint32_t)(dy * 3 * CH), k16 = (uint32_t)((part * KSTEPS + k) * 16), x = x_lo + k16;
            const uint32_t g = (uint32_t)dg0 + st + k16, on = k == 0 ? 0u : 1u;
            constexpr uint32_t DX = (uint32_t)(4 * S_BYTES) >> 4;
            const bool go = issue && ok;
            mma_bf16_from<A_FILL>(go, acc, x, x_hi, g, g_hi, idesc, on);
            mma_bf16_from<A_USE>(go, acc + CH, x, x_hi, g + DX, g_hi, idesc, on);
            mma_bf16_from<A_LAST>(go, acc + 2 * CH, x, x_hi, g + 2 * DX, g_hi, idesc, on);
          }
          if (ok) mma_commit_from(issue, &acc_full[dy]);
        }
      }
      mma_commit_from(issue, &empty_bar[s]);
      ok = ok && !__any_sync(0xffffffffu, *(volatile int *)&failed);
    }
    if (!ok && lane == 0) failed = 1;
    mma_commit_from(issue, &done_bar);
    if (!mbar_wait(&done_bar, 0) && lane == 0) failed = 1;
  } else if (warp < 2 + SHIFTERS) {
    // copy [dx][chunk]: slot i = the gradient at s0 + i - (dx - 1), zero outside
    // the owned cells; the raw runs start at slot s0 - 1
    for (int it = 0; it < mine; it++) {
      const int s = it % stages;
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&full_bar[s], (it / stages) & 1) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) failed = 1;
        break;
      }
      const Tile ti = tile_of(blockIdx.x + it * gridDim.x, N, Np, per_plane);
      const int goff = (int)(conv_at(N, ti.b, ti.zh, 0, ti.s0 - 1) & 7);
      uint8_t *st = base + s * gm.stage_bytes;
      for (int i = (warp - 2) * 32 + lane; i < ROWS + 2; i += 32 * SHIFTERS) {
        const int slot = ti.s0 - 1 + i, yh = slot / Np, xh = slot - yh * Np;
        const bool own = yh >= 1 && yh <= N && xh >= 1 && xh <= N;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (own) v = *reinterpret_cast<const uint4 *>(st + g_off + k * G_BYTES + (goff + i) * 16);
#pragma unroll
          for (int dx = 0; dx < 3; dx++) {
            const int at = i - 1 + dx - 1;  // slot of copy dx that takes it
            if (at >= 0 && at < ROWS) *reinterpret_cast<uint4 *>(st + s_off + (dx * 4 + k) * S_BYTES + at * 16) = v;
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready_bar[s]);
      if (__any_sync(0xffffffffu, *(volatile int *)&failed != 0)) break;
    }
  } else {
    // D row 32 q + lane = (dz = q, ci = lane), row 96 the sums of g; column co
    const int q = warp & 3, row = (warp - 2 - SHIFTERS) >> 2, t0 = row * TAPS_PER_WARP;  // the stencil row dy
    float sum[TAPS_PER_WARP][CH] = {};
    bool good = true;
    for (int use = 0; use < mine * SPLIT; use++) {
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&acc_full[row], use & 1) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) failed = 1;
        good = false;
        break;
      }
      fence_after();
#pragma unroll
      for (int t = 0; t < TAPS_PER_WARP; t++) {
        const uint32_t col = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((t0 + t) * CH);
#pragma unroll
        for (int c0 = 0; c0 < CH; c0 += 16) {  // 16 columns at a time: nothing spills
          uint32_t ra[8], rb[8];
          tmem_ld8_async(col + c0, ra);
          tmem_ld8_async(col + c0 + 8, rb);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 8; c++) {
            sum[t][c0 + c] += __uint_as_float(ra[c]);
            sum[t][c0 + 8 + c] += __uint_as_float(rb[c]);
          }
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[row]);
    }
    if (good) {
#pragma unroll
      for (int t = 0; t < TAPS_PER_WARP; t++) {
        const int tap2 = t0 + t;
        if (q < 3) {
          float *d = dw + ((long long)(q * TAPS2 + tap2) * CH) * CH + lane;
#pragma unroll
          for (int c = 0; c < CH; c++) atomicAdd(d + c * CH, sum[t][c]);
        } else if (tap2 == 4 && lane == 0 && db) {
#pragma unroll
          for (int c = 0; c < CH; c++) atomicAdd(db + c, sum[t][c]);
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && failed) atomicExch(err, 1);
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WG_TMEM) : "memory");
  }
}

}  // namespace wg
}  // namespace conv

cudaError_t launch_conv_wgrad(const __nv_bfloat16 *in, const __nv_bfloat16 *g, int N, int batch, float *dw, float *db,
                              int *err, cudaStream_t s) {
  using namespace conv;
  constexpr int MAXDEV = 64;
  static std::mutex mu;
  static int sms_of[MAXDEV] = {0};
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= MAXDEV) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!sms_of[dev]) {
      e = cudaFuncSetAttribute(wg::wgrad_tc_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wg::wgrad_tc_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
      if (e != cudaSuccess) return e;
      e = cudaDeviceGetAttribute(&sms_of[dev], cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
    }
    sms = sms_of[dev];
  }
  const wg::Geom a = wg::geom_for(N, 1), b = wg::geom_for(N, 3);
  const int forced = conv_runs();
  // one run per plane while it is the smaller load and two stages fit
  const bool planes = forced == 1 ? a.stages >= 1 : forced == 3 ? false : a.stages >= 2;
  const wg::Geom gm = planes ? a : b;
  if (N < 2 || batch < 1 || gm.stages < 1 || gm.box_rows > 256) return cudaErrorInvalidValue;
  const long long lines = conv_units(N, batch) / 8;
  if (lines >= 0x7fffffffLL) return cudaErrorInvalidValue;
  CUtensorMap mx, mg;
  if ((e = make_map_lines(&mx, in, lines, gm.box_rows)) != cudaSuccess) return e;
  if ((e = make_map_lines(&mg, g, lines, wg::G_ROWS)) != cudaSuccess) return e;
  const long long tiles = (long long)batch * N * (((long long)N * (N + 2) + ROWS - 1) / ROWS);
  const int grid = (int)(tiles < sms ? tiles : sms);
  // a tile per CTA at most: nothing averages the accumulators' rounding, so half as
  // many accumulations (16^3: error 1.13e-7 and 0.97e-7, 7.2 and 7.8 us; FP32 FMAs 1.09e-7)
  chain_launch(true, tiles <= sms ? wg::wgrad_tc_kernel<2> : wg::wgrad_tc_kernel<1>, grid, wg::WG_THREADS, gm.smem, s, mx, mg, N, batch, dw, db, err, gm);
  launch_counter()++;
  return cudaGetLastError();
}

}  // namespace sclet
