// Device and host helpers of the tensor-core mode-n product kernel
// (k_modeprod_tc.cu): tile constants, mbarrier / TMA / tcgen05 wrappers, the
// tile order and the tensor-map encoder.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include "sclet_tc.cuh"

namespace sclet {
namespace tc {


constexpr int BM = TC_BM, BK = TC_BK, NP = TC_PLANES, NPM = TC_PLANES_M;
constexpr int PLANE_A = BM * BK * 2;  // 8 KB: one input slice (M side, 128 input rows)
constexpr int SMEM_ALIGN = 512;  // period of the 64-byte swizzle pattern
constexpr int NACC = 4;               // weight classes w = 0..3
constexpr int EPI_WARPS = 8;          // two per TMEM lane quadrant, each half of the columns
constexpr int THREADS = 64 + 32 * EPI_WARPS;  // producer, MMA, epilogue warps
constexpr long long WAIT_LIMIT = 1LL << 22;  // polls (with backoff) before giving up

// what follows from the a'-tile width BN (N side)
template <int BN>
struct TileGeom {
  static constexpr int PLANE_B = BN * BK * 2;  // one matrix slice
  static constexpr int STAGE_BYTES = NP * PLANE_A + NPM * PLANE_B;
  static constexpr int STAGES = BN == 128 ? 3 : 4;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + SMEM_ALIGN;
  static constexpr int ACC_COLS = NACC * BN;      // one accumulator set
  static constexpr int NBUF = 512 / ACC_COLS;     // accumulator sets in tensor memory (1 or 2)
  static constexpr int TMEM_COLS = NBUF * ACC_COLS;
  static constexpr int CPW = BN / 32 / 2;         // 32-column chunks per epilogue warp
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory per CTA");
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait; false on timeout (the caller records the error).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (long long i = 0; i < WAIT_LIMIT; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i > 64) __nanosleep(64);
  }
  return false;
}

// bytes (a multiple of 16, both addresses 16-byte aligned) into shared memory
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Byte of (row, column pair at 2 c) in a slice tile of 64-byte rows, the 64-byte
// swizzle the descriptors below name: 16-byte chunk j of row r at j ^ (r / 2) % 4.
__device__ __forceinline__ uint32_t swizzled(int r, int c) {
  return (uint32_t)(r * 64 + ((((c >> 2) ^ (r >> 1)) & 3) << 4) + (c & 3) * 4);
}

// Shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups
// 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;             // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;             // descriptor version
  d |= (uint64_t)4 << 61;             // 64-byte swizzle
  return d;
}

// Instruction descriptor: BF16 x BF16 -> FP32, both K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// MMAs are issued from a loop that the whole warp runs, so that descriptors and
// indices are warp-uniform values the compiler keeps in uniform registers, and
// one elected lane (`issue`) issues; descriptors as a constant high and a low
// word that takes the offsets.  A loop run by a single lane spent most of a
// small MMA's time moving its operands there: convolution layers of 4 x 64^3
// 117 -> 97 us, their weight gradients 136 -> 100 us, the eigenbasis products of
// 516^3 28.0 -> 25.5 ms a step.
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(ok));
  return ok != 0;
}
// What becomes of the A operand: read and dropped, read and kept in the
// collector, taken from the collector, taken from it for the last time.
// Consecutive MMAs of one A operand read it from shared memory once.
enum Collect { A_DROP, A_FILL, A_USE, A_LAST };
template <Collect C>
struct Keep {
  static constexpr Collect value = C;
};
template <Collect C = A_DROP>
__device__ __forceinline__ void mma_bf16_from(bool issue, uint32_t dtmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo,
                                              uint32_t b_hi, uint32_t idesc, uint32_t acc) {
#define SCLET_MMA(MOD)                                                                                     \
  asm volatile(                                                                                            \
      "{\n .reg .pred p, q;\n .reg .b64 a, b;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n"            \
      " setp.ne.b32 p, %6, 0;\n setp.ne.b32 q, %7, 0;\n"                                                   \
      " @q tcgen05.mma.cta_group::1.kind::f16.collector::a::" MOD " [%0], a, b, %5, p;\n}\n" ::"r"(dtmem),  \
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc), "r"((uint32_t)issue)               \
      : "memory")
  if (C == A_DROP) SCLET_MMA("discard");
  else if (C == A_FILL) SCLET_MMA("fill");
  else if (C == A_USE) SCLET_MMA("use");
  else SCLET_MMA("lastuse");
#undef SCLET_MMA
}
__device__ __forceinline__ void mma_commit_from(bool issue, uint64_t *bar) {
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.b32 q, %1, 0;\n"
      " @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar)),
      "r"((uint32_t)issue)
      : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}

// The same load without the wait: the registers are valid after tmem_wait_ld.
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// 8 columns.
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

struct TileIdx {
  int a_tile, r_tile, t, part;
};
// power-of-two scale S >= m (S = 1 for m = 0)
__device__ __forceinline__ float pow2_scale(float m) {
  if (!(m > 0.0f)) return 1.0f;
  int e;
  frexpf(m, &e);  // m = f 2^e, f in [0.5, 1)
  return ldexpf(1.0f, e);
}

// The u-th output tile of CTA `cta`: tiles dealt round robin over the CTAs, the
// a'-tile fastest, then the tensor, then the input tile; the parts of a tile
// one after the other on one CTA.  The a'-tiles of one input tile so run side
// by side on neighbouring CTAs and its slices come from HBM once; a CTA taking
// all of them itself came back to a part after 152 CTAs had read theirs, 90 MB
// at 516^3, and read it from HBM again.  The tensors of one input tile run side
// by side too, so the fused update's coefficient tables (one per field kind)
// come from HBM about once per input tile.
template <int PARTS>
__device__ __forceinline__ TileIdx cta_tile(int u, int a_tiles, int count, int cta, int grid) {
  TileIdx x;
  const int tile = cta + (u / PARTS) * grid, grp = tile / a_tiles;
  x.a_tile = tile - grp * a_tiles;
  x.part = u % PARTS;
  x.t = grp % count;
  x.r_tile = grp / count;
  return x;
}

}  // namespace tc

static inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

}  // namespace sclet
