// Split-precision mode-n product on the 5th-generation tensor cores (tcgen05),
// the mixed-precision form of PUX / PUY / PUZ (source_beta_to_omega/src/
// calc.c:631-684).
//
// Number format: each operand is a power-of-two scale times four fixed-point
// slices of b bits, x = S * sum_p d_p 2^-b(p+1), d_0 in [-2^b, 2^b], d_p in
// [-2^(b-1), 2^(b-1)] (round to nearest at every level; 4b bits below S).
// b = 7 while the contraction length K <= 1024, else 6 (tc_slice_bits).  The
// slices are small integers held exactly in BF16.  The product keeps every
// cross term of weight w = p + q <= 3 (the split-precision scheme of Markidis
// et al. 2018 / Ootomo & Yokota 2022 carried to fixed point, as in the Ozaki
// scheme), one FP32 accumulator in tensor memory per weight class.  In classes
// 0 and 1 every partial sum is an integer below 2^24 (|sum| <= 2^(2b) per k
// times K <= 2^(24-2b)), so their accumulation is exact and unbiased; classes
// 2 and 3 sit 2^-2b and 2^-3b below the result, where accumulator rounding is
// harmless.  The matrix carries a fifth slice (its representation error would
// otherwise act on the leading data slice the same way every step); it is
// stored pre-scaled by 2^-b and its term M4 x0 joins class 3: eleven BF16 MMAs
// per k-step.  The epilogue combines the four classes with round-to-nearest
// adds.
//
// Scales: powers of two per matrix row (static) and per input row (one 1-D
// line along the contracted axis, 2^ceil(log2 max|x|) over the line, found by
// the slicing kernel), so a line holding a spectral peak or a boundary-lifting
// outlier costs precision only within itself.  The scale of an output entry
// is rank one (matrix row a' times input row r), so accumulation stays exact.
//
// Layout: input slices P[t][part][r / 128][kb][p][r % 128][32]: rows r = 0 ..
// n*n-1 are 1-D lines along the contracted axis, k = 32 kb + (k % 32) < kp =
// roundup(n, 32), zero beyond n.  The four slices of one k-block of a tile of
// 128 lines are one contiguous run of 32 KB, already in the 64-byte swizzle that
// the MMAs read, so one bulk copy brings a stage's input operand and one the
// matrix slices (40 KB, likewise [a' / 128][kb][p][a' % 128][32]); nine tensor
// copies of 64-byte rows kept the copy engine busy for 1600 cycles a stage, with
// the MMAs waiting.  Output FP32
// out[t][a' * n*n + r] for input row r = c * n + b, i.e. contracted index
// slowest: three products return to x-fastest order.
//
// Kernel: persistent CTAs (one per SM) looping over output tiles D[128 r x
// 128 a'] (input rows on the MMA's M side, eigen-modes a' on its N side, so
// the last a'-tile runs N = its live rows rounded up to 16 rather than a full
// 128).  Tiles are dealt round robin, a'-tile fastest, then tensor
// (cta_tile): the input slices come from HBM once, the a'-tiles of one input
// tile reading them at about the same time on neighbouring CTAs, and the
// tensors of one input tile share the fused update's coefficient reads through
// L2; the matrix slices stay in L2.  Every CTA loads its own operand tiles (no
// cluster).  The order of tiles and the copies in whole runs: 4 + 1 fields of
// 516^3 24.9 -> 20.8 ms a step, of 196^3 0.98 -> 0.84 ms.
// A = input slices (128 r rows x 32 k, 64-byte swizzle), B = matrix slices
// (128 a' rows x 32 k), both K-major, in a three-stage mbarrier pipeline
// that runs ahead across tiles; a stage is refilled once the MMAs that read
// it have completed.
// The folded forms (the default basis) halve the MMAs of a product and, with
// the increment form, a field needs six products instead of nine.  Kernel time
// of a step, dense and nine products before, now: 4 + 1 fields of 516^3
// 52.8 -> 17.3 ms, of 196^3 1.64 -> 0.65 ms, 4 fields of 68^3 124 -> 72 us; the
// step's error against 64 bits fell from 2.2e-7 to 0.6e-7 (196^3, ten steps).
// Warp 0 issues the copies, warp 1 issues MMAs (one elected thread each) and owns the
// tensor memory (4 classes x 128 columns).  Warps 2-9 run the epilogue (TMEM
// lane quadrant warp % 4): the four classes of the tile are combined into
// registers and the tensor memory is released at once, then the scaling, the
// fused ETD update (ac_updateU_new / ch_updateU_new, calc.c:489-535) or phi2
// scaling (prepare_U2_new, calc.c:553-567) and the FP32 stores overlap the
// next tile's MMAs.  Every mbarrier wait is bounded: on timeout the CTA
// records an error, drains its copies and MMAs (bounded), frees TMEM and
// returns.
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "sclet_internal.cuh"
#include "sclet_tc.cuh"

#include "sclet_tc_ptx.cuh"

namespace sclet {

namespace tc {

// FORM 0: any basis.  FORM 1, 2: the parity-folded forward and inverse products
// of the Dirichlet basis (sclet_basis.cu): the sliced lines and the matrix come
// in two parts (even, odd modes) of h = ceil(n / 2) columns, a tile's parts one
// after the other.  The forward epilogue interleaves
// the parts' modes; the inverse one keeps the even part's tile E in registers
// until the odd part's O is there and stores E + O and E - O, or, for fields that
// are no increments, E at its positions and O at their mirrors (see unfold_kernel, k_mass.cu).
// EPI 0 store, 1 ETD1 update, 2 phi scaling (FORM 0; the folded transforms apply
// them where the lines are sliced for the inverse, slice_fold_kernel).
// OUT 1 store, 2 accumulate (FORM 2: of fields below g.acc, the others store E and
// O; as reductions at the L2, so that no epilogue warp waits for the old values).
// BN: a'-tile width.  128 columns of the four classes fill tensor memory; with
// 64, for halves up to 64, two accumulator sets alternate.
template <int FORM, int EPI, int OUT, int BN>
__global__ void __launch_bounds__(THREADS, 1)
    modeprod_tc_kernel(const char *__restrict__ planes, const char *__restrict__ mat, TcArgs g) {
  using G = TileGeom<BN>;
  constexpr int STAGES = G::STAGES, STAGE_BYTES = G::STAGE_BYTES, PLANE_B = G::PLANE_B, NBUF = G::NBUF;
  constexpr int ACC_COLS = G::ACC_COLS, TMEM_COLS = G::TMEM_COLS, CPW = G::CPW;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tfull_bar[NBUF];   // accumulator set ready (MMA -> epilogue)
  __shared__ __align__(8) uint64_t tempty_bar[NBUF];  // accumulator set drained (epilogue -> MMA)
  __shared__ __align__(8) uint64_t done_bar;       // every MMA of this CTA completed
  __shared__ uint32_t tmem_slot;
  __shared__ int failed;

  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + SMEM_ALIGN - 1) & ~(uintptr_t)(SMEM_ALIGN - 1));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const long long rows = (long long)g.n * g.n;
  constexpr int PARTS = FORM == 0 ? 1 : 2;
  const int h = FORM == 0 ? g.n : fold_half(g.n);  // outputs of one part
  const int a_tiles = (h + BN - 1) / BN;
  const int r_tiles = (int)((rows + BM - 1) / BM);
  const int tiles = r_tiles * g.count * a_tiles;  // dealt round robin (cta_tile)
  const int mine = (int)blockIdx.x < tiles ? PARTS * ((tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) : 0;
  const int nkb = g.kblocks;
  const int last_rows = (h - (a_tiles - 1) * BN + 15) / 16 * 16;  // N of the last a'-tile, at most BN

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < NBUF; b++) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], EPI_WARPS);  // one arrival per epilogue warp
    }
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
  chain_wait();

  if (warp == 0) {
    if (lane == 0) {
      // producer: four input slices and five matrix slices per stage, the
      // k-blocks of all this CTA's tiles in one stream
      int it = 0;
      // the self-test leaves every barrier without arrivals (no copy is issued)
      for (int u = g.idle ? mine : 0; u < mine; u++) {
        const TileIdx ti = cta_tile<PARTS>(u, a_tiles, g.count, blockIdx.x, gridDim.x);
        for (int kb = 0; kb < nkb; kb++, it++) {
          const int s = it % STAGES;
          if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) & 1) ^ 1)) {
            failed = 1;
            break;
          }
          if (*(volatile int *)&failed) break;
          uint8_t *st = base + s * STAGE_BYTES;
          const uint32_t b_rows = ti.a_tile == a_tiles - 1 ? last_rows : BN;
          mbar_expect_tx(&full_bar[s], NP * PLANE_A + NPM * (b_rows * BK * 2));
          // a k-block's input slices are one run, and so are its matrix
          // slices, of which the last a'-tile takes the rows it multiplies
          bulk_load(st, planes + ((((long long)ti.t * PARTS + ti.part) * r_tiles + ti.r_tile) * nkb + kb) * (NP * PLANE_A),
                    NP * PLANE_A, &full_bar[s]);
          const char *mb = mat + (((long long)ti.part * a_tiles + ti.a_tile) * nkb + kb) * (NPM * PLANE_B);
          if (b_rows == BN) {
            bulk_load(st + NP * PLANE_A, mb, NPM * PLANE_B, &full_bar[s]);
          } else {
            for (int p = 0; p < NPM; p++)
              bulk_load(st + NP * PLANE_A + p * PLANE_B, mb + p * PLANE_B, b_rows * BK * 2, &full_bar[s]);
          }
        }
        if (*(volatile int *)&failed) break;
      }
      if (*(volatile int *)&failed) {
        // drain: wait (bounded) for copies still in flight into this CTA
        for (int i = it - STAGES < 0 ? 0 : it - STAGES; i < it; i++) mbar_wait(&full_bar[i % STAGES], (i / STAGES) & 1);
      }
    }
  } else if (warp == 1) {
    // MMA issuer: 2 k-steps of 16 per stage, eleven terms each, grouped by input
    // slice so that each is read from shared memory once (the A collector): the
    // operand reads, not the multiplications, bound MMAs of this shape.  The
    // first term of each class at a tile's first k-step starts its accumulator.  The
    // last a'-tile runs N = its rows rounded up to 16.  The warp runs the loop
    // together, one lane issues (mma_bf16_from).
    const bool issue = elect_one();
    const uint32_t idesc_full = idesc_bf16(BM, BN);
    const uint32_t idesc_last = idesc_bf16(BM, last_rows);
    const bool last_two = h - (nkb - 1) * BK > 16;  // the last k-block needs both k-steps
    // descriptors: the high word is constant, the low word's address field
    // (16-byte units) takes the stage, slice and k-step offsets
    const uint64_t d0 = smem_desc(smem_u32(base));
    const uint32_t hi = (uint32_t)(d0 >> 32), lo0 = (uint32_t)d0;
    int it = 0;
    bool ok = true;
    for (int u = 0; u < mine && ok; u++) {
      const int b = u % NBUF;
      // accumulator set b was last used by tile u - NBUF
      if (u >= NBUF) ok = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[b], ((u / NBUF) & 1) ^ 1));
      if (!ok) break;
      fence_after();
      const uint32_t acc = tmem + (uint32_t)(b * ACC_COLS);
      const uint32_t idesc = cta_tile<PARTS>(u, a_tiles, g.count, blockIdx.x, gridDim.x).a_tile == a_tiles - 1 ? idesc_last
                                                                                                           : idesc_full;
      for (int kb = 0; kb < nkb; kb++, it++) {
        const int s = it % STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[s], (it / STAGES) & 1));
        if (!ok) break;
        fence_after();
        const uint32_t la = lo0 + (uint32_t)(s * STAGE_BYTES >> 4), lb = la + (uint32_t)(NP * PLANE_A >> 4);
#pragma unroll
        for (int ks = 0; ks < BK / 16; ks++) {
          // the last k-block's second k-step holds only zero columns when
          // h mod 32 is in 1..16: skipped (adding zero products changes no
          // accumulator)
          if (ks > 0 && kb == nkb - 1 && !last_two) continue;
          const uint32_t first = (kb == 0 && ks == 0) ? 0u : 1u;
          auto term = [&](auto c, int pa, int pb, int cls, uint32_t keep) {
            mma_bf16_from<decltype(c)::value>(issue, acc + (uint32_t)(cls * BN),
                                              la + (uint32_t)((pa * PLANE_A + ks * 32) >> 4), hi,
                                              lb + (uint32_t)((pb * PLANE_B + ks * 32) >> 4), hi, idesc, keep);
          };
          // (input slice, matrix slice, class)
          term(Keep<A_FILL>(), 0, 4, 3, first);
          term(Keep<A_USE>(), 0, 3, 3, 1u);
          term(Keep<A_USE>(), 0, 2, 2, first);
          term(Keep<A_USE>(), 0, 1, 1, first);
          term(Keep<A_LAST>(), 0, 0, 0, first);
          term(Keep<A_FILL>(), 1, 2, 3, 1u);
          term(Keep<A_USE>(), 1, 1, 2, 1u);
          term(Keep<A_LAST>(), 1, 0, 1, 1u);
          term(Keep<A_FILL>(), 2, 1, 3, 1u);
          term(Keep<A_LAST>(), 2, 0, 2, 1u);
          term(Keep<A_DROP>(), 3, 0, 3, 1u);
        }
        mma_commit_from(issue, &empty_bar[s]);
      }
      if (ok) mma_commit_from(issue, &tfull_bar[b]);
      ok = ok && !__any_sync(0xffffffffu, *(volatile int *)&failed);
    }
    if (!ok && lane == 0) failed = 1;
    // every MMA issued so far must complete before the memory is freed
    mma_commit_from(issue, &done_bar);
    if (!mbar_wait(&done_bar, 0) && lane == 0) failed = 1;
  } else {
    // epilogue warps 2-9: TMEM lane quadrant q = warp % 4 holds input rows
    // q*32 .. q*32+31 of the tile, one per lane; the columns are the tile's
    // a' (eigen-mode) rows, the first half for warps 2-5, the second for
    // warps 6-9.  Each tile: combine the four classes of the warp's live
    // columns into registers, free the accumulators at once (the MMA warp
    // starts the next tile), then scale, apply the fused update and store
    // while those MMAs run.  For one a' the 32 lanes hold 32 consecutive
    // input rows, so every load and store of the warp is one contiguous
    // 128-byte run (512 bytes for the coefficient tables).
    const int q = warp & 3;
    const int c_first = ((warp - 2) >> 2) * CPW;  // the warp's first 32-column chunk
    // class weights 2^-b(w+2); exact integers combined small to large
    const float wt[NACC] = {ldexpf(1.0f, -2 * g.bits), ldexpf(1.0f, -3 * g.bits), ldexpf(1.0f, -4 * g.bits),
                            ldexpf(1.0f, -5 * g.bits)};
    int j = 0;
    // An inverse product's even part E until the odd part's O is there.  With one
    // accumulator set (DEFER) E - O then waits for the next tile: E + O is stored
    // while the next even part's MMAs run, E - O while the odd part's do, instead
    // of both under the even part's and nothing under the odd one's (products of
    // 516^3 21.0 -> 18.9 ms a step, of 196^3 0.85 -> 0.82 ms).  With two sets the
    // MMAs do not wait for the stores, and it would only add a pass over the tile
    // (104^3: 0.26 -> 0.28 ms).
    constexpr bool DEFER = FORM == 2 && NBUF == 1;
    float even[FORM == 2 ? CPW : 1][32];
    // E - O of tile tp, to the mirrored positions
    auto store_mirror = [&](const TileIdx &tp) {
      const long long r = (long long)tp.r_tile * BM + q * 32 + lane;
      const int nch = (min(BN, h - tp.a_tile * BN) + 31) / 32;
      float *outT = g.out + (long long)tp.t * g.n * rows;
      if (tp.t % g.F >= g.acc) return;  // stored as it came
#pragma unroll
      for (int cl = 0; cl < CPW; cl++) {
        const int a0 = tp.a_tile * BN + (c_first + cl) * 32;
        const int lim = min(32, g.n / 2 - a0);  // an odd block's middle cell has no mirror
        const uint32_t q0 = (uint32_t)(g.n - 1 - a0) * (uint32_t)rows + (uint32_t)r;
        if (c_first + cl < nch && r < rows) {
#pragma unroll
          for (int jj = 0; jj < 32; jj++)
            if (jj < lim) {
              float *oz = outT + (q0 - (uint32_t)jj * (uint32_t)rows);
              if (OUT == 2) atomicAdd(oz, even[cl][jj]);
              else *oz = even[cl][jj];
            }
        }
      }
    };
    TileIdx prev;
    bool ok_all = true;
    for (int u = 0; u < mine; u++, j++) {
      const int b = j % NBUF;
      const TileIdx ti = cta_tile<PARTS>(u, a_tiles, g.count, blockIdx.x, gridDim.x);
      const int at0 = ti.a_tile * BN;
      const int nch = (min(BN, h - at0) + 31) / 32;  // 32-column chunks holding live a'
      const long long r = (long long)ti.r_tile * BM + q * 32 + lane;
      const bool live = r < rows;
      // the scales come while the tile's MMAs run: the input row's, and per
      // chunk the 32 matrix rows', one per lane, broadcast below
      const float si = live ? g.in_scale[((long long)ti.t * PARTS + ti.part) * rows + r] : 0.0f;
      float rsv[CPW];
#pragma unroll
      for (int cl = 0; cl < CPW; cl++) {
        const int a = at0 + (c_first + cl) * 32 + lane;
        rsv[cl] = a < h ? g.row_scale[ti.part * h + a] : 0.0f;
      }
      // one lane waits, the warp follows its verdict (tcgen05.ld below needs
      // the whole warp converged)
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&tfull_bar[b], (j / NBUF) & 1) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) {
        if (lane == 0) failed = 1;
        ok_all = false;
        break;
      }
      fence_after();
      const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * ACC_COLS);
      // per live chunk two classes in flight at a time
      float acc[CPW][32];
#pragma unroll
      for (int cl = 0; cl < CPW; cl++) {
        const int c = c_first + cl;
        if (c < nch) {
          if constexpr (DEFER) {
            // Beside E: eight columns of the four classes at a time, so that
            // nothing spills.  Spilled values went to L2, shared memory taking
            // all of L1: products of 516^3 18.9 -> 17.3 ms a step, of 196^3
            // 0.82 -> 0.65 ms.
#pragma unroll
            for (int c8 = 0; c8 < 4; c8++) {
              const uint32_t col = ta + (uint32_t)(c * 32 + c8 * 8);
              uint32_t ra[8], rb[8], rc[8], rd[8];
              tmem_ld8_async(col + 3 * BN, ra);
              tmem_ld8_async(col + 2 * BN, rb);
              tmem_ld8_async(col + BN, rc);
              tmem_ld8_async(col, rd);
              tmem_wait_ld();
              float *o = acc[cl] + c8 * 8;
#pragma unroll
              for (int jj = 0; jj < 8; jj++)
                o[jj] = fmaf(__uint_as_float(rd[jj]), wt[0],
                             fmaf(__uint_as_float(rc[jj]), wt[1],
                                  fmaf(__uint_as_float(rb[jj]), wt[2], __uint_as_float(ra[jj]) * wt[3])));
            }
            continue;
          }
          uint32_t ra[32], rb[32];
          tmem_ld32_async(ta + 3 * BN + c * 32, ra);
          tmem_ld32_async(ta + 2 * BN + c * 32, rb);
          tmem_wait_ld();
#pragma unroll
          for (int jj = 0; jj < 32; jj++)
            acc[cl][jj] = fmaf(__uint_as_float(rb[jj]), wt[2], __uint_as_float(ra[jj]) * wt[3]);
          tmem_ld32_async(ta + 1 * BN + c * 32, ra);
          tmem_ld32_async(ta + c * 32, rb);
          tmem_wait_ld();
#pragma unroll
          for (int jj = 0; jj < 32; jj++)
            acc[cl][jj] = fmaf(__uint_as_float(rb[jj]), wt[0], fmaf(__uint_as_float(ra[jj]), wt[1], acc[cl][jj]));
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[b]);
      if (DEFER && ti.part == 0 && u > 0) store_mirror(prev);
      const bool ch = ti.t % g.F >= g.nac;  // field kind: Cahn-Hilliard
      const float4 *cf = ch ? g.coef[1] : g.coef[0];
      const float2 *cf2 = ch ? g.coef2[1] : g.coef2[0];
      const long long tb = (long long)ti.t * g.n * rows;
      float *outT = g.out + tb;
      // offsets within one tensor stay below n^3 < 2^32 (n <= 1088)
      const uint32_t urows = (uint32_t)rows;
#pragma unroll
      for (int cl = 0; cl < CPW; cl++) {
        const int c = c_first + cl;
        if (c < nch) {
          const int a0 = at0 + c * 32;
          const int lim = min(32, h - a0);  // live a' in the chunk
          const float rs = rsv[cl];
          if (FORM == 2) {
            const uint32_t o0 = (uint32_t)a0 * urows + (uint32_t)(live ? r : 0);
            const uint32_t q0 = (uint32_t)(g.n - 1 - a0) * urows + (uint32_t)(live ? r : 0);  // mirrored position
            if (ti.t % g.F >= g.acc) {
              // E at its positions, O at the mirrored ones (an odd block's middle cell has none)
              const int end = ti.part == 0 ? lim : min(lim, g.n / 2 - a0);
              const uint32_t at = ti.part == 0 ? o0 : q0, step = ti.part == 0 ? urows : 0u - urows;
#pragma unroll
              for (int jj = 0; jj < 32; jj++) {
                const float v = acc[cl][jj] * (si * __shfl_sync(0xffffffffu, rs, jj));
                if (jj < end && live) outT[at + (uint32_t)jj * step] = v;
              }
              continue;
            }
            if (ti.part == 0) {
#pragma unroll
              for (int jj = 0; jj < 32; jj++) even[cl][jj] = acc[cl][jj] * (si * __shfl_sync(0xffffffffu, rs, jj));
              continue;
            }
#pragma unroll
            for (int jj = 0; jj < 32; jj++) {
              const float od = acc[cl][jj] * (si * __shfl_sync(0xffffffffu, rs, jj));
              const float y = even[cl][jj] + od, z = even[cl][jj] - od;
              if (DEFER) even[cl][jj] = z;
              if (jj < lim && live) {
                float *oy = outT + (o0 + (uint32_t)jj * urows), *oz = outT + (q0 - (uint32_t)jj * urows);
                const bool mirror = !DEFER && a0 + jj < g.n / 2;  // an odd block's middle cell has none
                if (OUT == 2) {
                  atomicAdd(oy, y);
                  if (mirror) atomicAdd(oz, z);
                } else {
                  *oy = y;
                  if (mirror) *oz = z;
                }
              }
            }
            continue;
          }
          // output row of column jj: a0 + jj, or mode 2 (a0 + jj) + the part's first
          const int live_o = FORM == 0 ? lim : min(lim, (ti.part == 0 ? h : g.n / 2) - a0);
          const uint32_t ostep = FORM == 0 ? urows : 2 * urows;
          const uint32_t o0 = (FORM == 0 ? (uint32_t)a0 : (uint32_t)(2 * a0 + fold_mode0(g.n, ti.part))) * urows +
                              (uint32_t)(live ? r : 0);  // eigen-mode [k][j][i] of a z-contraction
          // batches of columns: every load of a batch is issued before its
          // first store (aux and the coefficient tables are read-only here:
          // the ETD update never runs in place)
          constexpr int NB = EPI == 1 ? 4 : 8;
#pragma unroll
          for (int j0 = 0; j0 < 32; j0 += NB) {
            float uh[NB], old[NB];
            float4 c1[NB];
            float2 c2[NB];
#pragma unroll
            for (int jj = 0; jj < NB; jj++) {
              const uint32_t o = o0 + (uint32_t)(j0 + jj) * ostep;
              if (j0 + jj < live_o && live) {
                if (EPI == 1) {
                  uh[jj] = __ldg(g.aux + tb + o);
                  c1[jj] = __ldg(cf + o);
                } else if (EPI == 2) {
                  c2[jj] = __ldg(cf2 + o);
                }
                if (OUT == 2) old[jj] = outT[o];
              }
            }
#pragma unroll
            for (int jj = 0; jj < NB; jj++) {
              const uint32_t o = o0 + (uint32_t)(j0 + jj) * ostep;
              const float sc = si * __shfl_sync(0xffffffffu, rs, j0 + jj);
              if (j0 + jj < live_o && live) {
                float y = acc[cl][j0 + jj] * sc;
                if (EPI == 1) {
                  const float4 cc = c1[jj];  // (e_hi, e_lo, phi1_hi, phi1_lo)
                  y = fmaf(cc.x, uh[jj], fmaf(cc.y, uh[jj], fmaf(cc.z, y, cc.w * y)));
                } else if (EPI == 2) {
                  y = fmaf(c2[jj].x, y, c2[jj].y * y);  // (phi2_hi, phi2_lo)
                }
                if (OUT == 2) y += old[jj];
                outT[o] = y;
              }
            }
          }
        }
      }
      prev = ti;
      if (__any_sync(0xffffffffu, *(volatile int *)&failed != 0)) {
        ok_all = false;
        break;
      }
    }
    if (DEFER && mine > 0 && ok_all) store_mirror(prev);
  }
  __syncthreads();
  if (threadIdx.x == 0 && failed) atomicExch(g.err, 1);
  if (warp == 1) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}


// FP32 rows of n (x - sub) -> slices: the row's max gives its power-of-two
// scale S; each slice is exact (the residual is scaled by 2^b and reduced by
// its nearest integer).
constexpr int SLICE_MAXC = 34;  // 32-column chunks per row: rows of up to 32 * 34 = 1088 values

// A warp takes two adjacent rows, one per half-warp (lane l: row l / 16,
// columns 2 (l % 16) + 32 c of chunk c, held in registers, C >= ceil(n / 32)).
// The two rows' columns of k-block c are one contiguous 128-byte run, so every
// store instruction of the warp fills whole lines.  Columns load as float2 when
// n is even.
template <int C>
__global__ void __launch_bounds__(256) slice_fields_kernel(const float *__restrict__ x, const float *__restrict__ sub,
                                                           float *__restrict__ scale, __nv_bfloat16 *__restrict__ out,
                                                           int n, int kp, int count, int bits) {
  chain_wait();
  const float step = ldexpf(1.0f, bits);
  const long long rows = (long long)n * n, total_rows = rows * count;
  const int lane = threadIdx.x & 31, h = lane >> 4, kl = 2 * (lane & 15);
  const int chunks = (n + BK - 1) / BK;
  const bool pairs = (n & 1) == 0;  // every row starts on an 8-byte boundary
  const long long warp0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long w0 = 2 * warp0; w0 < total_rows; w0 += 2 * nwarps) {
    const long long wr = w0 + h;
    const bool live = wr < total_rows;
    const long long in0 = wr * n;  // rows are contiguous lines of n
    float v0[C], v1[C];
    float m = 0.0f;
#pragma unroll
    for (int c = 0; c < C; c++) {
      v0[c] = 0.0f;
      v1[c] = 0.0f;
      const int k = kl + BK * c;
      if (live && c < chunks && k < n) {
        if (pairs) {
          float2 a = *reinterpret_cast<const float2 *>(x + in0 + k);
          if (sub) {
            const float2 b = *reinterpret_cast<const float2 *>(sub + in0 + k);
            a.x -= b.x;
            a.y -= b.y;
          }
          v0[c] = a.x;
          v1[c] = a.y;
        } else {
          v0[c] = sub ? x[in0 + k] - sub[in0 + k] : x[in0 + k];
          if (k + 1 < n) v1[c] = sub ? x[in0 + k + 1] - sub[in0 + k + 1] : x[in0 + k + 1];
        }
      }
      m = fmaxf(m, fmaxf(fabsf(v0[c]), fabsf(v1[c])));
    }
    // the row's max over its half-warp
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (!live) continue;
    const int t = (int)(wr / rows);
    const long long row = wr - (long long)t * rows;
    const float S = pow2_scale(m), inv = 1.0f / S;
    if (kl == 0) scale[wr] = S;
    const long long tile = ((long long)t * ((rows + BM - 1) / BM) + row / BM) * (kp / BK);
    char *const o0 = reinterpret_cast<char *>(out) + tile * (TC_PLANES * PLANE_A) + swizzled((int)(row % BM), kl / 2);
    // stored as bf16 pairs (the pad columns n .. kp - 1 are never written:
    // they stay zero from the allocation)
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int k = kl + BK * c;
      if (c < chunks && k < n) {
        float r0 = v0[c] * inv, r1 = v1[c] * inv;
#pragma unroll
        for (int p = 0; p < TC_PLANES; p++) {
          const float y0 = r0 * step, y1 = r1 * step;
          const float d0 = rintf(y0), d1 = rintf(y1);
          r0 = y0 - d0;
          r1 = y1 - d1;
          *reinterpret_cast<__nv_bfloat162 *>(o0 + (c * TC_PLANES + p) * PLANE_A) = __floats2bfloat162_rn(d0, d1);
        }
      }
    }
  }
}

// Power-of-two scale S > m (as pow2_scale) and 1 / S from m's exponent bits.
__device__ __forceinline__ void scale_of(float m, float &S, float &inv) {
  const uint32_t e = __float_as_uint(m) >> 23;
  if (e >= 1 && e <= 252) {
    S = __uint_as_float((e + 1) << 23);
    inv = __uint_as_float((253 - e) << 23);
  } else {  // zero, subnormal, huge, not finite
    S = pow2_scale(m);
    inv = 1.0f / S;
  }
}

// The four digits of y (|y| < 1) plus a remainder e far below it: y's
// nearest multiples of 1 / step level by level (adding and subtracting
// 1.5 2^23 rounds to the nearest integer; every residual is exact), e joining
// the last one.
__device__ __forceinline__ void digits(float y, float e, float step, float step4, float (&d)[TC_PLANES]) {
  constexpr float M = 12582912.0f;
#pragma unroll
  for (int p = 0; p < TC_PLANES - 1; p++) {
    d[p] = __fadd_rn(__fmaf_rn(y, step, M), -M);
    y = __fmaf_rn(y, step, -d[p]);
  }
  d[TC_PLANES - 1] = __fadd_rn(__fadd_rn(__fmaf_rn(e, step4, y * step), M), -M);
}
// integers of at most 8 bits: their BF16 is the upper half of the FP32
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
}

// Lines -> the slices of their two parity parts, with a
// scale per line and part, one line per half-warp as above.
//   MODE 0 (forward): even x[k] + x[n-1-k], odd x[k] - x[n-1-k], k < h, formed
//        as exact pairs (TwoSum) whose low half joins the last slice, so
//        folding rounds nothing above the slices' own 28 bits; an odd block's
//        middle cell counts once.  x - sub where sub is given.
//   MODE 1 (inverse): the even and the odd modes of the line, interleaved in x
//   MODE 2: the same after the step's update of the eigen-modes: phi x for
//        tensors t < sp.nI, e u^ + phi1 N^ for the others (u^ the block t, N^
//        the block t + count - nI), these as pairs whose low half joins the last
//        slice
// A CTA takes SLICE_ROWS lines of one tensor, the tensors of the same lines in
// neighbouring CTAs (the coefficients of MODE 2 come from HBM about once).  A
// line is held in registers, all its loads in flight at once.  (Reading it twice
// instead, for its maxima and from L1 for its digits, let five CTAs fit an SM
// but waited longer: 0.86 ms a step at 196^3 against 0.72.)  Bound by HBM and
// its write pattern: 4 B read and 8 B written per element.
constexpr int SLICE_ROWS = 64;

template <int C, int MODE>
__global__ void __launch_bounds__(256)
    slice_fold_kernel(TensorList<float> xs, const float *__restrict__ sub, float *__restrict__ scale,
                      __nv_bfloat16 *__restrict__ out, int n, int kp, int count, int bits, SpecUpdate sp) {
  chain_wait();
  const float step = ldexpf(1.0f, bits), step4 = ldexpf(1.0f, 4 * bits);
  const int rows = n * n;
  const long long n3 = (long long)rows * n;
  const int lane = threadIdx.x & 31, hw = lane >> 4, kl = 2 * (lane & 15);
  const int h = fold_half(n), h16 = (h + 15) / 16 * 16, odd0 = fold_mode0(n, 1);
  const int align = n % 4 == 0 ? 4 : n % 2 == 0 ? 2 : 1;  // values per aligned load of a line
  const int t = blockIdx.x % count, rb = blockIdx.x / count;
  const float *xt = xs.at(t, n3);
  const float *st = sub ? sub + t * n3 : nullptr;
  // the parts' tile of these lines: SLICE_ROWS divides its height
  static_assert(BM % SLICE_ROWS == 0, "lines of one tile");
  const long long tile = (long long)(kp / BK) * TC_PLANES * PLANE_A;
  const int tiles = (rows + BM - 1) / BM;
  char *const even = reinterpret_cast<char *>(out) + (2LL * t * tiles + rb * SLICE_ROWS / BM) * tile;
  char *const odd = even + tiles * tile;
  // MODE 2
  const bool etd = MODE == 2 && t >= sp.nI;
  const float4 *ce = MODE == 2 ? sp.etd[t % sp.F >= sp.nac ? 1 : 0] : nullptr;
  const float2 *cp = MODE == 2 ? sp.phi[t % sp.F >= sp.nac ? 1 : 0] : nullptr;
  const long long nhat = (long long)(count - sp.nI) * n3;  // from u^ to N^
  const int mid = MODE == 0 && align == 1 ? h - 1 : -1;    // an odd block's middle cell
  const int row_end = min(rows, (rb + 1) * SLICE_ROWS);
  for (int row0 = rb * SLICE_ROWS + (threadIdx.x >> 5) * 2; row0 < row_end; row0 += 16) {
    const int row = row0 + hw;
    const bool live = row < row_end;
    const long long l0 = (long long)(live ? row : row0) * n;
    const float *x = xt + l0;
    // columns k, k + 1 (k < h): MODE 0: a = x[k], x[k+1], b = their mirrors; else
    // a = the even part's two modes, b = the odd part's
    uint32_t alo[MODE == 2 ? C : 1], blo[MODE == 2 ? C : 1];  // MODE 2: the values' low parts, BF16 pairs
    auto load = [&](int k, int c, float &a0, float &a1, float &b0, float &b1) {
      if (MODE == 0) {
        const int q = n - 1 - k;
        a1 = b1 = 0.0f;
        if (align >= 2) {  // n even: pairs and their mirrors aligned, no middle cell
          float2 a = *reinterpret_cast<const float2 *>(x + k), b = *reinterpret_cast<const float2 *>(x + q - 1);
          if (st) {
            const float2 sa = *reinterpret_cast<const float2 *>(st + l0 + k);
            const float2 s2 = *reinterpret_cast<const float2 *>(st + l0 + q - 1);
            a.x -= sa.x;
            a.y -= sa.y;
            b.x -= s2.x;
            b.y -= s2.y;
          }
          a0 = a.x;
          b0 = b.y;
          if (k + 1 < h) a1 = a.y, b1 = b.x;
        } else {
          auto one = [&](int i) { return st ? x[i] - st[l0 + i] : x[i]; };
          a0 = one(k);
          b0 = q != k ? one(q) : 0.0f;
          if (k + 1 < h) {
            a1 = one(k + 1);
            if (q - 1 != k + 1) b1 = one(q - 1);
          }
        }
      } else {
        const int k2 = 2 * k;
        float v[4];
        auto four = [&](const float *p, float (&w)[4]) {
          if (align == 4) {  // then k2 + 3 < n
            const float4 f = *reinterpret_cast<const float4 *>(p + k2);
            w[0] = f.x, w[1] = f.y, w[2] = f.z, w[3] = f.w;
          } else if (align == 2 && k2 + 3 < n) {
            const float2 f = *reinterpret_cast<const float2 *>(p + k2), g = *reinterpret_cast<const float2 *>(p + k2 + 2);
            w[0] = f.x, w[1] = f.y, w[2] = g.x, w[3] = g.y;
          } else {
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = k2 + i < n ? p[k2 + i] : 0.0f;
          }
        };
        four(x, v);
        if (MODE == 2) {
          float lo[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (etd) {
            float nh[4];
            four(x + nhat, nh);
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (k2 + i < n) {
                // e u^ + phi1 N^ with what its products and sums round off
                const float4 f = __ldg(ce + l0 + k2 + i);  // (e_hi, e_lo, phi1_hi, phi1_lo)
                const float u = v[i], w = fmaf(f.y, u, f.w * nh[i]), p = f.x * u, q = fmaf(f.z, nh[i], w);
                v[i] = __fadd_rn(p, q);
                const float b = __fadd_rn(v[i], -p);
                lo[i] = __fadd_rn(__fadd_rn(p, -__fadd_rn(v[i], -b)), __fadd_rn(q, -b)) +
                        (fmaf(f.x, u, -p) + (fmaf(f.z, nh[i], -q) + w));
              }
          } else {
            float2 f[4];
            if (align >= 2 && k2 + 3 < n) {
              const float4 p = __ldg(reinterpret_cast<const float4 *>(cp + l0 + k2));
              const float4 q = __ldg(reinterpret_cast<const float4 *>(cp + l0 + k2 + 2));
              f[0] = make_float2(p.x, p.y), f[1] = make_float2(p.z, p.w);
              f[2] = make_float2(q.x, q.y), f[3] = make_float2(q.z, q.w);
            } else {
#pragma unroll
              for (int i = 0; i < 4; i++) f[i] = k2 + i < n ? __ldg(cp + l0 + k2 + i) : make_float2(0.0f, 0.0f);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = fmaf(f[i].x, v[i], f[i].y * v[i]);  // (phi_hi, phi_lo)
          }
          if (etd) {
            alo[c] = bf16_pair(odd0 ? lo[0] : lo[1], odd0 ? lo[2] : lo[3]);
            blo[c] = bf16_pair(odd0 ? lo[1] : lo[0], odd0 ? lo[3] : lo[2]);
          }
        }
        a0 = odd0 ? v[0] : v[1];
        a1 = odd0 ? v[2] : v[3];
        b0 = odd0 ? v[1] : v[0];
        b1 = odd0 ? v[3] : v[2];
      }
    };
    float a0[C], a1[C], b0[C], b1[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      a0[c] = a1[c] = b0[c] = b1[c] = 0.0f;
      if (MODE == 2) alo[c] = blo[c] = 0;
      if (kl + BK * c < h) load(kl + BK * c, c, a0[c], a1[c], b0[c], b1[c]);
    }
    float me = 0.0f, mo = 0.0f;
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int k = kl + BK * c;
      if (MODE == 0) {
        me = fmaxf(me, fmaxf(fabsf(a0[c] + b0[c]), fabsf(a1[c] + b1[c])));
        // the middle cell is in the even part only
        mo = fmaxf(mo, fmaxf(k == mid ? 0.0f : fabsf(a0[c] - b0[c]), k + 1 == mid ? 0.0f : fabsf(a1[c] - b1[c])));
      } else {
        me = fmaxf(me, fmaxf(fabsf(a0[c]), fabsf(a1[c])));
        mo = fmaxf(mo, fmaxf(fabsf(b0[c]), fabsf(b1[c])));
      }
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) {
      me = fmaxf(me, __shfl_xor_sync(0xffffffffu, me, off));
      mo = fmaxf(mo, __shfl_xor_sync(0xffffffffu, mo, off));
    }
    if (!live) continue;
    float Se, So, ie, io;
    scale_of(me, Se, ie);
    scale_of(mo, So, io);
    if (kl == 0) {
      scale[2LL * t * rows + row] = Se;
      scale[(2LL * t + 1) * rows + row] = So;
    }
    const uint32_t o = swizzled(row % BM, kl / 2);
    // up to a multiple of 16 columns, the last ones zero: whole 32-byte sectors
    // (a few columns' partial sectors per line and plane, as every edge of N + 4
    // has, cost more than their line)
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int k = kl + BK * c;
      if (k >= h16) break;
      float d0[TC_PLANES], d1[TC_PLANES];
      auto put = [&](char *part) {
#pragma unroll
        for (int p = 0; p < TC_PLANES; p++)
          *reinterpret_cast<uint32_t *>(part + o + (c * TC_PLANES + p) * PLANE_A) = bf16_pair(d0[p], d1[p]);
      };
      if (MODE == 0) {
        // TwoSum (Knuth) of the pair and its difference
        auto fold = [&](float a, float b, float inv, float (&d)[TC_PLANES]) {
          const float s = __fadd_rn(a, b), bp = __fadd_rn(s, -a);
          const float e = __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -bp)), __fadd_rn(b, -bp));
          digits(s * inv, e * inv, step, step4, d);
        };
        fold(a0[c], b0[c], ie, d0);
        fold(a1[c], b1[c], ie, d1);
        put(even);
        fold(k == mid ? 0.0f : a0[c], k == mid ? 0.0f : -b0[c], io, d0);
        fold(k + 1 == mid ? 0.0f : a1[c], k + 1 == mid ? 0.0f : -b1[c], io, d1);
        put(odd);
      } else {
        auto store = [&](auto low) {
          constexpr bool LOW = decltype(low)::value;
          const uint32_t la = LOW ? alo[c] : 0, lb = LOW ? blo[c] : 0;
          digits(a0[c] * ie, LOW ? __uint_as_float(la << 16) * ie : 0.0f, step, step4, d0);
          digits(a1[c] * ie, LOW ? __uint_as_float(la & 0xffff0000u) * ie : 0.0f, step, step4, d1);
          put(even);
          digits(b0[c] * io, LOW ? __uint_as_float(lb << 16) * io : 0.0f, step, step4, d0);
          digits(b1[c] * io, LOW ? __uint_as_float(lb & 0xffff0000u) * io : 0.0f, step, step4, d1);
          put(odd);
        };
        if (MODE == 2 && etd) store(std::integral_constant<bool, MODE == 2>());
        else store(std::false_type());
      }
    }
  }
}

// FP64 matrix rows -> slices with a power-of-two scale per row.
__global__ void slice_matrix_kernel(const double *__restrict__ m, __nv_bfloat16 *__restrict__ out,
                                    float *__restrict__ row_scale, int n, int kp, int bn, int bits) {
  __shared__ double smax[128];
  const double step = ldexp(1.0, bits);
  const int rows = (n + bn - 1) / bn * bn;  // whole a'-tiles, the rows beyond n zero
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    double mx = 0.0;
    for (int c = threadIdx.x; r < n && c < n; c += blockDim.x) mx = fmax(mx, fabs(m[(long long)r * n + c]));
    smax[threadIdx.x] = mx;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
      if (threadIdx.x < w) smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + w]);
      __syncthreads();
    }
    double S = 1.0;
    if (smax[0] > 0.0) {
      int e;
      frexp(smax[0], &e);
      S = ldexp(1.0, e);
    }
    __syncthreads();
    if (threadIdx.x == 0 && r < n) row_scale[r] = (float)S;
    for (int c = threadIdx.x; c < kp; c += blockDim.x) {
      double v = r < n && c < n ? m[(long long)r * n + c] / S : 0.0;
      const long long tile = ((long long)(r / bn) * (kp / BK) + c / BK) * TC_PLANES_M * bn * BK;
      for (int p = 0; p < TC_PLANES_M; p++) {
        double y = v * step;
        double d = rint(y);
        v = y - d;
        // the fifth slice enters class 3, one factor 2^b below its own weight
        float q = p < TC_PLANES ? (float)d : (float)(d / step);
        out[tile + (long long)p * bn * BK + swizzled(r % bn, c % BK / 2) / 2 + c % 2] = __float2bfloat16_rn(q);
      }
    }
  }
}

// ETD coefficients in FP64 (the plain form's ac_init_phi / ch_init_phi and
// ac_updateU_new / ch_updateU_new arithmetic), stored as FP32 hi + lo.
__global__ void coef_kernel(float4 *coef, float2 *phi1, float2 *coef2, int n, int kind, const double *dx, const double *dy,
                            const double *dz, double kkx, double kky, double kkz, double epn2, double dt, double L,
                            double K) {
  const long long n3 = (long long)n * n * n;
  for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < n3; o += (long long)gridDim.x * blockDim.x) {
    int i = (int)(o % n), j = (int)((o / n) % n), k = (int)(o / ((long long)n * n));
    double tmp, H;
    if (kind == 0) {
      tmp = kkz * dz[k] + kky * dy[j] + kkx * dx[i];
      H = -L * (tmp * epn2 - K);
    } else {
      tmp = dz[k] + dy[j] + dx[i];
      H = L * (tmp * tmp * epn2 - K * tmp);
    }
    double p1, p2;
    if (fabs(H) > 1.0e-8) {
      p1 = -expm1(-dt * H) / H;
      p2 = (1.0 - p1 / dt) / H;
    } else {
      p1 = dt;
      p2 = dt / 2;
    }
    double Hu = fabs(H) < 1.0e-8 ? 0.0 : H;
    double e = 1.0 - p1 * Hu;
    float4 c;
    c.x = (float)e;
    c.y = (float)(e - (double)c.x);
    c.z = (float)p1;
    c.w = (float)(p1 - (double)c.z);
    if (coef) coef[o] = c;
    if (phi1) phi1[o] = make_float2(c.z, c.w);
    if (coef2) {
      float2 c2;
      c2.x = (float)p2;
      c2.y = (float)(p2 - (double)c2.x);
      coef2[o] = c2;
    }
  }
}

}  // namespace tc

// ---- host side ------------------------------------------------------------

int tc_kp(int n) { return (n + tc::BK - 1) / tc::BK * tc::BK; }

int tc_bn(bool folded, int h) { return folded && h <= 64 ? 64 : 128; }

long long tc_plane_elems(int n, bool folded) {
  const long long rows = ((long long)n * n + tc::BM - 1) / tc::BM * tc::BM;
  return (folded ? 2LL * tc_kp(fold_half(n)) : tc_kp(n)) * TC_PLANES * rows;
}
long long tc_matrix_elems(int n, bool folded) {
  const int h = folded ? fold_half(n) : n, bn = tc_bn(folded, h);
  return (folded ? 2LL : 1LL) * TC_PLANES_M * ((h + bn - 1) / bn * bn) * tc_kp(h);
}

// Slice width: classes 0 and 1 stay exact while K 2^(2b) <= 2^24, K the
// contraction length rounded up to whole k-blocks.
int tc_slice_bits(int n) {
  const long long K = (long long)tc::BK * ((n + tc::BK - 1) / tc::BK);
  return K <= 1024 ? 7 : 6;
}

cudaError_t tc_slice_matrix(const double *m, __nv_bfloat16 *planes, float *row_scale, int n, int bn,
                            cudaStream_t s) {
  tc::slice_matrix_kernel<<<n < 1024 ? n : 1024, 128, 0, s>>>(m, planes, row_scale, n, tc_kp(n), bn, tc_slice_bits(n));
  launch_counter()++;
  return cudaGetLastError();
}

// Whether a slicing of g CTAs is launched early: with a CTA per SM at most, or in
// four to seven waves.  In fewer waves its CTAs would crowd on the SMs that the
// product ahead leaves first, with the little L1 its shared memory leaves; in more
// the launch latency saved is nothing.  Step times, early over late, of 34 edges
// from 12^3 to 320^3 with 1, 4 and 4 + 1 fields, plain launches and graphs: up to
// 152 CTAs 0.84 to 0.97 and 0.95 to 1.05, 200 to 560 1.01 to 1.16 and 1.02 to
// 1.25, 610 to 1060 0.97 to 1.01 and 0.99 to 1.06, beyond 0.99 to 1.04 and 1.00 to
// 1.05 (1200 to 2400: 1.00 to 1.04 both).
static bool slice_early(int g) { return g <= 152 || (g > 4 * 152 && g <= 7 * 152); }

cudaError_t tc_slice_fields(const float *x, const float *sub, float *scale, __nv_bfloat16 *planes, int n, int count,
                            cudaStream_t s) {
  if (n > tc::BK * tc::SLICE_MAXC) return cudaErrorInvalidValue;
  long long warps = ((long long)n * n * count + 1) / 2;  // two rows per warp
  long long blocks = (warps * 32 + 255) / 256;
  int g = (int)(blocks > 152 * 32 ? 152 * 32 : blocks);
  const int chunks = (n + tc::BK - 1) / tc::BK, kp = tc_kp(n), bits = tc_slice_bits(n);
  const bool early = slice_early(g);
  if (chunks <= 4) chain_launch(early, tc::slice_fields_kernel<4>, g, 256, 0, s, x, sub, scale, planes, n, kp, count, bits);
  else if (chunks <= 8) chain_launch(early, tc::slice_fields_kernel<8>, g, 256, 0, s, x, sub, scale, planes, n, kp, count, bits);
  else if (chunks <= 17) chain_launch(early, tc::slice_fields_kernel<17>, g, 256, 0, s, x, sub, scale, planes, n, kp, count, bits);
  else chain_launch(early, tc::slice_fields_kernel<tc::SLICE_MAXC>, g, 256, 0, s, x, sub, scale, planes, n, kp, count, bits);
  launch_counter()++;
  return cudaGetLastError();
}

template <int MODE>
static void run_slice_fold(int chunks, int g, const TensorList<float> &x, const float *sub, float *scale,
                           __nv_bfloat16 *planes, int n, int kp, int count, int bits, const SpecUpdate &sp,
                           cudaStream_t s) {
  const bool early = slice_early(g);
#define SCLET_SLICE(C) chain_launch(early, tc::slice_fold_kernel<C, MODE>, g, 256, 0, s, x, sub, scale, planes, n, kp, count, bits, sp)
  if (chunks <= 1) SCLET_SLICE(1);
  else if (chunks <= 2) SCLET_SLICE(2);
  else if (chunks <= 3) SCLET_SLICE(3);
  else if (chunks <= 4) SCLET_SLICE(4);
  else if (chunks <= 5) SCLET_SLICE(5);
  else if (chunks <= 7) SCLET_SLICE(7);
  else if (chunks <= 9) SCLET_SLICE(9);
  else if (chunks <= 12) SCLET_SLICE(12);
  else SCLET_SLICE(17);
#undef SCLET_SLICE
}

cudaError_t tc_slice_fold(bool forward, const TensorList<float> &x, const float *sub, const SpecUpdate *sp, float *scale,
                          __nv_bfloat16 *planes, int n, int count, cudaStream_t s) {
  const int h = fold_half(n), kp = tc_kp(h), bits = tc_slice_bits(h);
  const long long g = ((long long)n * n + tc::SLICE_ROWS - 1) / tc::SLICE_ROWS * count;
  // 32-bit row numbers
  if (g > 0x7fffffffLL || kp > 17 * tc::BK) return cudaErrorInvalidValue;
  const int chunks = kp / tc::BK;
  if (forward) run_slice_fold<0>(chunks, (int)g, x, sub, scale, planes, n, kp, count, bits, SpecUpdate(), s);
  else if (!sp) run_slice_fold<1>(chunks, (int)g, x, nullptr, scale, planes, n, kp, count, bits, SpecUpdate(), s);
  else run_slice_fold<2>(chunks, (int)g, x, nullptr, scale, planes, n, kp, count, bits, *sp, s);
  launch_counter()++;
  return cudaGetLastError();
}

cudaError_t tc_make_coefs(float4 *coef, float2 *phi1, float2 *coef2, int n, int kind, const double *dx, const double *dy,
                          const double *dz, const double *kk, double epn2, double dt, double L, double K,
                          cudaStream_t s) {
  long long n3 = (long long)n * n * n;
  long long b = (n3 + 255) / 256;
  tc::coef_kernel<<<(int)(b > 152 * 16 ? 152 * 16 : b), 256, 0, s>>>(coef, phi1, coef2, n, kind, dx, dy, dz, kk[0], kk[1],
                                                                     kk[2], epn2, dt, L, K);
  launch_counter()++;
  return cudaGetLastError();
}

// The kernel's instances, the combinations the step uses: any basis (none,
// store), (none, accumulate), (ETD1, store), (phi2, store); folded forward
// (store) and inverse (store, accumulate), each for halves beyond 64 and up to
// 64.
using TcKernel = void (*)(const char *, const char *, TcArgs);
struct TcInstance {
  int form, epi, out, bn, smem;
  TcKernel kern;
};
constexpr int TC_INSTANCES = 10;
static const TcInstance &tc_instance(int i) {
#define SCLET_TC(F, E, O, B) {F, E, O, B, tc::TileGeom<B>::SMEM_BYTES, tc::modeprod_tc_kernel<F, E, O, B>}
  static const TcInstance k[TC_INSTANCES] = {
      SCLET_TC(0, 0, 1, 128), SCLET_TC(0, 0, 2, 128), SCLET_TC(0, 1, 1, 128), SCLET_TC(0, 2, 1, 128),
      SCLET_TC(1, 0, 1, 128), SCLET_TC(2, 0, 1, 128), SCLET_TC(2, 0, 2, 128),
      SCLET_TC(1, 0, 1, 64),  SCLET_TC(2, 0, 1, 64),  SCLET_TC(2, 0, 2, 64)};
#undef SCLET_TC
  return k[i];
}
static const TcInstance *tc_kernel(int form, int epi, int outmode, int bn) {
  for (int i = 0; i < TC_INSTANCES; i++) {
    const TcInstance &k = tc_instance(i);
    if (k.form == form && k.epi == epi && k.out == outmode && k.bn == bn) return &k;
  }
  return nullptr;
}

// Per-device launch set-up: the dynamic shared-memory attributes (set per
// device, for every instance) and the number of CTAs that can be resident at
// once.
static int tc_setup(int *ctas) {
  constexpr int MAXDEV = 64;
  static std::mutex mu;
  static int resident[MAXDEV] = {0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= MAXDEV) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (!resident[dev]) {
    for (int i = 0; i < TC_INSTANCES; i++) {
      // all of the unified L1/shared capacity as shared memory
      e = cudaFuncSetAttribute(tc_instance(i).kern, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_instance(i).smem);
      if (e != cudaSuccess) return e;
      e = cudaFuncSetAttribute(tc_instance(i).kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      if (e != cudaSuccess) return e;
    }
    int per_sm = 0, sms = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_instance(0).kern, tc::THREADS, tc_instance(0).smem);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    resident[dev] = per_sm * sms;
  }
  *ctas = resident[dev];
  return cudaSuccess;
}

cudaError_t launch_modeprod_tc(const __nv_bfloat16 *mat, const __nv_bfloat16 *planes, int count, const TcArgs &args,
                               cudaStream_t s) {
  int ctas = 0;
  cudaError_t e = (cudaError_t)tc_setup(&ctas);
  if (e != cudaSuccess) return e;
  // contraction length and outputs of one part
  const int n = args.n, parts = args.form == 0 ? 1 : 2, h = parts == 1 ? n : fold_half(n), kp = tc_kp(h);
  const int bn = tc_bn(parts == 2, h);
  const TcInstance *inst = tc_kernel(args.form, args.epi, args.outmode, bn);
  if (!inst) return cudaErrorInvalidValue;
  const int bits = tc_slice_bits(h);
  if ((long long)kp > (1LL << (24 - 2 * bits))) return cudaErrorInvalidValue;
  if ((long long)n * n * n > 0xffffffffLL) return cudaErrorInvalidValue;  // 32-bit offsets within a tensor
  TcArgs g = args;
  g.kblocks = kp / tc::BK;
  g.bits = bits;
  const long long tiles = (((long long)n * n + tc::BM - 1) / tc::BM) * count * ((h + bn - 1) / bn);
  if (tiles * parts > 0x7fffffffLL) return cudaErrorInvalidValue;
  // persistent: as many CTAs as can be resident at once (or the tuned count)
  if (args.max_ctas > 0 && args.max_ctas < ctas) ctas = args.max_ctas;
  const int grid = (int)(tiles < ctas ? tiles : ctas);
  // early but for many tiles a CTA, where it gives nothing (step times, early over
  // late, of 20 edges from 16^3 to 432^3 with 1, 4 and 4 + 1 fields, plain launches
  // and graphs: up to 1 tile a CTA 0.83 to 0.93 and 0.93 to 0.98, 2 to 5 0.94 to 0.98
  // and 0.98 to 1.00, 5 to 16 0.98 to 1.00 both, beyond 1.00 both)
  chain_launch(tiles <= 16LL * ctas, inst->kern, grid, tc::THREADS, inst->smem, s, reinterpret_cast<const char *>(planes),
                                                   reinterpret_cast<const char *>(mat), g);
  launch_counter()++;
  return cudaGetLastError();
}

}  // namespace sclet
