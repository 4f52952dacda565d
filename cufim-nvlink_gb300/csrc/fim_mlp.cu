// fim_mlp.cu -- the learned warm start: per-vertex features and a small
// MLP (7 -> 128 -> 128 -> 128 -> 1, ReLU) trained and evaluated on the GPU.
//
// One persistent kernel runs the whole network over 128-row tiles,
// mlp_forward_kernel the three hidden layers and the output, mlp_train_kernel
// also the way back: every product a tcgen05 MMA with BF16 operands and an
// FP32 accumulator in tensor memory.  A tile's activations never leave the
// SM: each layer's epilogue (bias + ReLU, or the ReLU mask) writes them as
// BF16 where the next MMA reads them, in tensor memory forward and in shared
// memory in training.  The weight gradients accumulate in tensor memory over
// all tiles of a CTA, and mlp_reduce_kernel adds the CTAs' sums in a fixed
// order and, in a training step, applies Adam.  Master weights, biases,
// output layer, loss and bias gradients are FP32; the MMAs read a BF16 copy
// of the weights refreshed
// after every update.  The input width is padded from 7 features to
// kMlpIn = 64 columns (zeros), one 128-byte K slice.
//
// No counterpart in the reference.
#include "fim_internal.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace fimgb {

namespace {

// ---------------------------------------------------------------------------
// tcgen05 building blocks.  Operands lie in shared memory as blocks of 64
// columns (128 bytes, the span of the 128-byte swizzle) by 128 rows, 16 KB
// each, as a TMA load with that swizzle puts them.  Such a block is a
// K-major operand when its columns are the contraction (activations times
// weights), and an MN-major one when its rows are (weight gradients:
// contraction over the tile's rows; data gradients: over the weights' output
// rows), so no operand is ever transposed in memory.  Every mbarrier wait is
// bounded (%globaltimer): a wait that runs out ends the loops of the CTA's
// warps and sets the error word, and the CTA waits (bounded) for the copies
// and MMAs it issued and frees its tensor memory.
constexpr int kTileM = 128, kBlkCols = 64;
constexpr uint32_t kBlkBytes = kTileM * kBlkCols * 2;  // 16 KB
constexpr uint64_t kMlpWaitNs = 2000000000ull;         // bound of every mbarrier wait

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t gtimer()
{
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// waits until the phase with the given parity has completed; false after limit_ns
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns = kMlpWaitNs)
{
  if (mbar_try(bar, parity)) return true;
  const uint64_t t0 = gtimer();
  for (uint32_t n = 0;; ++n) {
    if (mbar_try(bar, parity)) return true;
    if ((n & 255u) == 255u && gtimer() - t0 > limit_ns) return false;
  }
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
// Shared-memory matrix descriptors (128-byte swizzle: layout type 2,
// descriptor version 1).  K-major: 8-row groups 1024 B apart (stride byte
// offset), leading byte offset unused.  MN-major: 64-column blocks kBlkBytes
// apart (leading byte offset), 8-row groups (of the contraction) 1024 B
// apart (stride byte offset).
// Descriptors are kept as their low words: the high one is kDescHi for both.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_k(uint32_t addr) { return (addr >> 4) | (1u << 16); }
__device__ __forceinline__ uint32_t desc_mn(uint32_t addr) { return (addr >> 4) | ((kBlkBytes >> 4) << 16); }
// Instruction descriptor of tcgen05.mma kind::f16: FP32 accumulator (bits
// 4-5 = 1), BF16 A and B (bits 7-9, 10-12 = 1), A / B MN-major (bits 15,
// 16), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc(int n, bool a_mn, bool b_mn)
{
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}
// One lane of a warp in step issues the MMAs (elect_one, after a branch on a
// warp index that is known to be uniform): operands then stay in uniform
// registers.  Issued by a thread of a divergent branch a step took 80 cycles
// of the issuing thread, more than the 64 of the tensor pipe (predictions of
// 1.03M rows 90 us, 79 this way).
__device__ __forceinline__ bool elect_one()
{
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
  return e != 0;
}
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0); }
// acc (+)= A B; A and B in shared memory
__device__ __forceinline__ void umma_ss(uint32_t acc, uint32_t a, uint32_t b, uint32_t id, bool more)
{
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 x, y;\n setp.ne.b32 p, %5, 0;\n"
      " mov.b64 x, {%1, %3};\n mov.b64 y, {%2, %3};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %4, p;\n}"
      ::"r"(acc), "r"(a), "r"(b), "r"(kDescHi), "r"(id), "r"((uint32_t)more)
      : "memory");
}
// the same with A in tensor memory
__device__ __forceinline__ void umma_ts(uint32_t acc, uint32_t a, uint32_t b, uint32_t id, bool more)
{
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 y;\n setp.ne.b32 p, %5, 0;\n"
      " mov.b64 y, {%2, %3};\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], y, %4, p;\n}"
      ::"r"(acc), "r"(a), "r"(b), "r"(kDescHi), "r"(id), "r"((uint32_t)more)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 32 consecutive FP32 columns of this thread's tensor-memory lane; the load
// and its wait are one statement, so that no use of v can move between them
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t *v)
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
// Accumulator fragments: columns 0..63 of the warp's 32 lanes, thread T with
// columns 8 j + 2 (T % 4) + {0, 1} of lanes T / 4 + 8 k in v[32 (k / 2) + 4 j +
// 2 (k % 2) + {0, 1}], so that a thread needs a quarter of the biases it would
// need with a whole row; the loads and their wait are one statement, so that
// no use of v can move between them
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t *v)
{
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%64];\n"
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, "
      "%44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, "
      "[%65];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]),
        "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]), "=r"(v[37]), "=r"(v[38]), "=r"(v[39]),
        "=r"(v[40]), "=r"(v[41]), "=r"(v[42]), "=r"(v[43]), "=r"(v[44]), "=r"(v[45]), "=r"(v[46]), "=r"(v[47]),
        "=r"(v[48]), "=r"(v[49]), "=r"(v[50]), "=r"(v[51]), "=r"(v[52]), "=r"(v[53]), "=r"(v[54]), "=r"(v[55]),
        "=r"(v[56]), "=r"(v[57]), "=r"(v[58]), "=r"(v[59]), "=r"(v[60]), "=r"(v[61]), "=r"(v[62]), "=r"(v[63])
      : "r"(taddr), "r"(taddr + (16u << 16))
      : "memory");
}
// the packed pairs of such a fragment, v[16 (k / 2) + 2 j + k % 2], as columns
// 0..31
__device__ __forceinline__ void tmem_st_frag(uint32_t taddr, const uint32_t *v)
{
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15};\n"
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%33], {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, "
      "%27, %28, %29, %30, %31};\n"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]),
        "r"(taddr), "r"(taddr + (16u << 16))
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Index of weight i (W1 [kMlpIn x kMlpH], W2, W3 [kMlpH x kMlpH], each
// [in x out] row-major) in the transposed copies [out x in] that the MMAs
// read.
__device__ __forceinline__ int transposed_index(int i)
{
  if (i < kMlpOW2) return kMlpOW1 + (i % kMlpH) * kMlpIn + i / kMlpH;
  const int off = i < kMlpOW3 ? kMlpOW2 : kMlpOW3, k = i - off;
  return off + (k % kMlpH) * kMlpH + k / kMlpH;
}

// acc (tile rows x 128) = A (K-major, kBlocks blocks of 64 columns) times the
// K-major 128 x 64 kBlocks operand B, transposed
template <int kBlocks>
__device__ __forceinline__ void mma_rows(uint32_t acc, uint32_t a, uint32_t b)
{
#pragma unroll
  for (int k = 0; k < kBlocks * kBlkCols / 16; ++k) {
    const uint32_t at = (k / 4) * (kBlkBytes >> 4) + 2 * (k % 4);
    umma_ss(acc, desc_k(a) + at, desc_k(b) + at, idesc(128, false, false), k != 0);
  }
}
// the same for 128 columns with A in tensor memory, two BF16 to a 32-bit column
__device__ __forceinline__ void mma_rows_tmem(uint32_t acc, uint32_t a, uint32_t b)
{
#pragma unroll
  for (int k = 0; k < 128 / 16; ++k)
    umma_ts(acc, a + 8 * k, desc_k(b) + (k / 4) * (kBlkBytes >> 4) + 2 * (k % 4), idesc(128, false, false), k != 0);
}
// acc (tile rows x 128) = A (K-major, 128 columns) times W (128 rows x 128
// columns, contraction over its rows)
__device__ __forceinline__ void mma_data(uint32_t acc, uint32_t a, uint32_t w)
{
#pragma unroll
  for (int k = 0; k < 128 / 16; ++k)
    umma_ss(acc, desc_k(a) + (k / 4) * (kBlkBytes >> 4) + 2 * (k % 4), desc_mn(w) + (2048 >> 4) * k,
            idesc(128, false, true), k != 0);
}
// acc (128 x n) (+)= D^T H over the tile's rows: D 128 columns, H n columns
template <int n>
__device__ __forceinline__ void mma_weight(uint32_t acc, uint32_t d, uint32_t h, bool first)
{
#pragma unroll
  for (int k = 0; k < kTileM / 16; ++k)
    umma_ss(acc, desc_mn(d) + (2048 >> 4) * k, desc_mn(h) + (2048 >> 4) * k, idesc(n, true, true), !(first && k == 0));
}

__device__ __forceinline__ uint64_t f2_pack(float x, float y)
{
  return (uint64_t)__float_as_uint(x) | ((uint64_t)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float f2_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f2_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b)
{
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c)
{
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// two floats as BF16 (round to nearest), first in the low half
__device__ __forceinline__ uint32_t bf2(float lo, float hi)
{
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
// relu of two BF16 values (a NaN becomes 0, as fmaxf(x, 0) makes it)
__device__ __forceinline__ uint32_t bf2_relu(uint32_t x)
{
  uint32_t d;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(x), "r"(0u));
  return d;
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// ---------------------------------------------------------------------------
// Training over 128-row tiles: sixteen warps, warp w with tensor-memory lanes
// 32 (w % 4) .. + 31 (the tile's rows) of a quarter of the columns; warp 0
// issues the TMA loads and the MMAs.  One tile at a time, since a tile's features and
// three activations (112 KB) leave no room for a second one beside the 80 KB
// of weights; the next tile's features are loaded a tile ahead.  Step of
// 4,096 rows (22 launches before, 2 now) 191 -> 42 us; gradients of 131,136
// rows, whose activations and their transposes went through memory, 500 -> 85
// (eight warps with half of the columns each: 96 against 91 us at the time).
constexpr uint32_t kW1Bytes = kBlkBytes, kW2Bytes = 2 * kBlkBytes;
constexpr uint32_t kWBytes = kW1Bytes + 2 * kW2Bytes;  // the weights, [out][in]
constexpr uint32_t kActBytes = 2 * kBlkBytes;          // 128 x 128 activations
constexpr int kTrainThreads = 512, kColParts = kTrainThreads / kTileM, kCols = kMlpH / kColParts;
constexpr int kTrainSmem = (int)(kWBytes + 2 * kBlkBytes + 3 * kActBytes) + 1024;  // + slack to align to 1024 B
constexpr int kTmemCols = 512;
// tensor-memory columns in training: the layer's accumulator, then the
// transposed weight gradients [out][in] of layers 3, 2, 1
constexpr uint32_t kTmW3 = 128, kTmW2 = 256, kTmW1 = 384;
// partial results of a training CTA: gradients in parameter order, then the
// summed squared error
constexpr int kPartStride = (kMlpParams + 1 + 63) & ~63;

__global__ void __launch_bounds__(kTrainThreads, 1) mlp_train_kernel(
    const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw1,
    const __grid_constant__ CUtensorMap tw2, const __grid_constant__ CUtensorMap tw3, int M,
    const float *__restrict__ P, const float *__restrict__ tgt, float *part, unsigned int *bad,
    volatile unsigned int *err)
{
  extern __shared__ unsigned char mlp_smem[];
  __shared__ __align__(8) uint64_t wfull, xfull[2], mdone;
  __shared__ uint32_t tmem_base;
  __shared__ __align__(16) float s_bias[3][kMlpH], s_w4[kMlpH];
  __shared__ float s_part[kColParts - 1][kTileM], s_dy[kTileM];
  __shared__ volatile int s_fail[2];
  const int t = threadIdx.x, lane = t & 31, q = (t >> 5) & 3, h = t >> 7;  // h: column part
  const uint32_t w1 = (smem_u32(mlp_smem) + 1023u) & ~1023u, w2 = w1 + kW1Bytes, w3 = w2 + kW2Bytes;
  unsigned char *const sm = mlp_smem + (w1 - smem_u32(mlp_smem));  // generic address of w1
  const uint32_t xs = w1 + kWBytes, h1 = xs + 2 * kBlkBytes, h2 = h1 + kActBytes, h3 = h2 + kActBytes;
  const int ntiles = (M + kTileM - 1) / kTileM;
  const int tstep = gridDim.x, tile0 = blockIdx.x;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&wfull), 1);
    mbar_init(smem_u32(&xfull[0]), 1);
    mbar_init(smem_u32(&xfull[1]), 1);
    mbar_init(smem_u32(&mdone), 1);
    s_fail[0] = s_fail[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
  const int warp = warp_index();
  const uint32_t bar_m = smem_u32(&mdone);
  int issued = 0, consumed = 0;  // warp 0: feature tiles
  // feature tile i of the CTA: its buffer, barrier and parity
  const auto x_buf = [&](int i) { return xs + (uint32_t)(i & 1) * kBlkBytes; };
  const auto x_bar = [&](int i) { return smem_u32(&xfull[i & 1]); };
  const auto x_par = [&](int i) { return (uint32_t)(i >> 1) & 1u; };
  const auto load_x = [&](int tile) {
    if (lane == 0) {
      mbar_expect_tx(x_bar(issued), kBlkBytes);
      tma_load_2d(x_buf(issued), &tx, 0, tile * kTileM, x_bar(issued));
    }
    ++issued;
  };
  if (warp == 0 && tile0 < ntiles) load_x(tile0);
  if (threadIdx.x == 0) {
    mbar_expect_tx(smem_u32(&wfull), kWBytes);
    tma_load_2d(w1, &tw1, 0, 0, smem_u32(&wfull));
    for (int s = 0; s < 2; ++s) {
      tma_load_2d(w2 + s * kBlkBytes, &tw2, s * kBlkCols, 0, smem_u32(&wfull));
      tma_load_2d(w3 + s * kBlkBytes, &tw3, s * kBlkCols, 0, smem_u32(&wfull));
    }
  }
  for (int i = threadIdx.x; i < 4 * kMlpH; i += kTrainThreads) {
    if (i < 3 * kMlpH) s_bias[i / kMlpH][i % kMlpH] = P[kMlpOB1 + i];
    else s_w4[i - 3 * kMlpH] = P[kMlpOW4 + i - 3 * kMlpH];
  }
  const float b4 = P[kMlpOB4];
  __syncthreads();
  bool wok = true;
  if (warp == 0) wok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&wfull), 0));

  // A phase ends with a barrier; a wait that ran out in phase p
  // is flagged in s_fail[p & 1] before that barrier and read after it, so
  // the whole CTA leaves together (a later phase writes the other word).
  int phase = 0;
  uint32_t mpar = 0;       // parity of the next MMA completion
  int commits = 0;         // warp 0: completions requested
  int waited = 0;
  const auto fail = [&]() { s_fail[phase & 1] = 1; };
  const auto end_phase = [&]() {
    __syncthreads();
    const bool bad = s_fail[phase & 1] != 0;
    ++phase;
    return !bad;
  };
  const auto wait_mma = [&]() {
    if (!mbar_wait(bar_m, mpar)) fail();
    else ++waited;
    mpar ^= 1u;
    __syncwarp();
    tc_fence_after();
  };
  // publishes shared-memory rows written by this thread to the MMAs
  const auto publish = [&]() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    return end_phase();
  };
  const uint32_t tv = tmem + ((uint32_t)(q * 32) << 16);
  const int r = q * 32 + lane;  // this thread's row of the tile
  // kCols columns of the row: from the accumulator, and where they lie in an activation block
  const auto load_acc = [&](uint32_t *v) { tmem_ld32(tv + kCols * h, v); };
  const auto chunk_ptr = [&](uint32_t base, int c) {  // 16-byte chunk c, at chunk c ^ (row % 8)
    return reinterpret_cast<uint4 *>(sm + (base - w1) + (uint32_t)(h >> 1) * kBlkBytes + (uint32_t)r * 128u +
                                     ((uint32_t)((4 * (h & 1) + c) ^ (r & 7)) << 4));
  };

  // training: sums over this thread's rows (columns 2 cp, 2 cp + 1, rows
  // kRgRows rg .. of every tile) of the bias gradients and of gw4; over this
  // thread's own row of dy and of the squared error
  constexpr int kRowGroups = kTrainThreads / 64, kRgRows = kTileM / kRowGroups;
  const int cp = t & 63, rg = t >> 6;
  float gb1[2] = {0.f, 0.f}, gb2[2] = {0.f, 0.f}, gb3[2] = {0.f, 0.f}, gw4[2] = {0.f, 0.f};
  float gb4 = 0.f, sse = 0.f;
  const uint32_t coloff = (uint32_t)(cp >> 5) * kBlkBytes + (uint32_t)(cp & 3) * 4u;
  const auto pair_ptr = [&](uint32_t base, int row) {
    return reinterpret_cast<uint32_t *>(sm + (base - w1) + coloff + (uint32_t)row * 128u +
                                        ((uint32_t)(((cp & 31) >> 2) ^ (row & 7)) << 4));
  };
  const auto colsum = [&](uint32_t base, float *s) {
#pragma unroll 16
    for (int i = 0; i < kRgRows; ++i) {
      const uint32_t w = *pair_ptr(base, kRgRows * rg + i);
      s[0] += bf_lo(w);
      s[1] += bf_hi(w);
    }
  };

  int j = 0;
  bool ok = true;
  for (int tile = tile0; tile < ntiles; tile += tstep, ++j) {
    const bool in = tile * kTileM + r < M;
    // layer 1
    if (warp == 0) {
      if (tile + tstep < ntiles) load_x(tile + tstep);  // its stage was read by MMAs that have completed
      if (!__all_sync(0xffffffffu, wok && mbar_wait(x_bar(j), x_par(j)))) fail();
      else {
        ++consumed;
        tc_fence_after();
        if (elect_one()) {
          mma_rows<1>(tmem, x_buf(j), w1);
          umma_commit(bar_m);
        }
        ++commits;
      }
      __syncwarp();
    }
#pragma unroll 1
    for (int layer = 0; layer < 2; ++layer) {
      wait_mma();
      {
        uint32_t v[kCols];
        load_acc(v);
        const uint32_t dst = layer == 0 ? h1 : h2;
        const ulonglong2 *bias = reinterpret_cast<const ulonglong2 *>(&s_bias[layer][kCols * h]);
#pragma unroll
        for (int c = 0; c < kCols / 8; ++c) {
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const ulonglong2 bb = bias[2 * c + k];
            const uint64_t x0 = f2_add(f2_pack(__uint_as_float(v[8 * c + 4 * k]), __uint_as_float(v[8 * c + 4 * k + 1])), bb.x);
            const uint64_t x1 = f2_add(f2_pack(__uint_as_float(v[8 * c + 4 * k + 2]), __uint_as_float(v[8 * c + 4 * k + 3])), bb.y);
            w[2 * k] = bf2_relu(bf2(f2_lo(x0), f2_hi(x0)));
            w[2 * k + 1] = bf2_relu(bf2(f2_lo(x1), f2_hi(x1)));
            if (!in) w[2 * k] = w[2 * k + 1] = 0u;  // rows past the matrix take no part in the gradients
          }
          *chunk_ptr(dst, c) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      if (!publish()) { ok = false; break; }
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          mma_rows<2>(tmem, layer == 0 ? h1 : h2, layer == 0 ? w2 : w3);
          umma_commit(bar_m);
        }
        ++commits;
        __syncwarp();
      }
    }
    if (!ok) break;
    // layer 3 and the output layer: y = relu(.) . w4 + b4 on the BF16
    // activations, the column parts added in a fixed order
    wait_mma();
    float ysum = 0.f;
    {
      uint32_t v[kCols];
      load_acc(v);
      const ulonglong2 *bias = reinterpret_cast<const ulonglong2 *>(&s_bias[2][kCols * h]);
      const ulonglong2 *wv = reinterpret_cast<const ulonglong2 *>(&s_w4[kCols * h]);
      uint64_t sum0 = 0ull, sum1 = 0ull;
#pragma unroll
      for (int c = 0; c < kCols / 8; ++c) {
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const ulonglong2 bb = bias[2 * c + k], ww = wv[2 * c + k];
          const uint64_t x0 = f2_add(f2_pack(__uint_as_float(v[8 * c + 4 * k]), __uint_as_float(v[8 * c + 4 * k + 1])), bb.x);
          const uint64_t x1 = f2_add(f2_pack(__uint_as_float(v[8 * c + 4 * k + 2]), __uint_as_float(v[8 * c + 4 * k + 3])), bb.y);
          w[2 * k] = bf2_relu(bf2(f2_lo(x0), f2_hi(x0)));
          w[2 * k + 1] = bf2_relu(bf2(f2_lo(x1), f2_hi(x1)));
          if (!in) w[2 * k] = w[2 * k + 1] = 0u;
          sum0 = f2_fma(f2_pack(bf_lo(w[2 * k]), bf_hi(w[2 * k])), ww.x, sum0);
          sum1 = f2_fma(f2_pack(bf_lo(w[2 * k + 1]), bf_hi(w[2 * k + 1])), ww.y, sum1);
        }
        *chunk_ptr(h3, c) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      ysum = (f2_lo(sum0) + f2_hi(sum0)) + (f2_lo(sum1) + f2_hi(sum1));
    }
    if (h > 0) s_part[h - 1][r] = ysum;
    tc_fence_before();  // (the accumulator is read: the next MMA may write it)
    if (!end_phase()) { ok = false; break; }
    if (h == 0) {
      float dy = 0.f;
      if (in) {
        const float e = ((((ysum + s_part[0][r]) + s_part[1][r]) + s_part[2][r]) + b4) - tgt[tile * (int64_t)kTileM + r];
        dy = 2.f * e / (float)M;
        sse += e * e;
        gb4 += dy;
      }
      s_dy[r] = dy;
    }
    if (!end_phase()) { ok = false; break; }
    // dZ3 = bf16(dy w4) where H3 > 0, in place; sums of gw4 and gb3
    {
      const float wa = s_w4[2 * cp], wb = s_w4[2 * cp + 1];
      {
        uint32_t w[kRgRows];
#pragma unroll
        for (int i = 0; i < kRgRows; ++i) w[i] = *pair_ptr(h3, kRgRows * rg + i);
#pragma unroll
        for (int i = 0; i < kRgRows; ++i) {
          const float dy = s_dy[kRgRows * rg + i], x0 = bf_lo(w[i]), x1 = bf_hi(w[i]);
          gw4[0] += x0 * dy;
          gw4[1] += x1 * dy;
          w[i] = bf2(x0 > 0.f ? dy * wa : 0.f, x1 > 0.f ? dy * wb : 0.f);
          gb3[0] += bf_lo(w[i]);
          gb3[1] += bf_hi(w[i]);
        }
#pragma unroll
        for (int i = 0; i < kRgRows; ++i) *pair_ptr(h3, kRgRows * rg + i) = w[i];
      }
    }
    if (!publish()) { ok = false; break; }
    // layers 3 and 2 back: dZ_(l-1) = (dZ_l W_l^T) where H_(l-1) > 0, in
    // place of H_(l-1) once the weight gradient dW_l = H_(l-1)^T dZ_l is done
#pragma unroll 1
    for (int layer = 0; layer < 2; ++layer) {
      const uint32_t dz = layer == 0 ? h3 : h2, hp = layer == 0 ? h2 : h1;
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          mma_data(tmem, dz, layer == 0 ? w3 : w2);
          mma_weight<128>(tmem + (layer == 0 ? kTmW3 : kTmW2), dz, hp, j == 0);
          umma_commit(bar_m);
        }
        ++commits;
        __syncwarp();
      }
      if (layer == 1) colsum(h2, gb2);
      wait_mma();
      {
        uint32_t v[kCols];
        load_acc(v);
#pragma unroll
        for (int c = 0; c < kCols / 8; ++c) {
          uint4 *a = chunk_ptr(hp, c);
          const uint4 mm = *a;
          const uint32_t m[4] = {mm.x, mm.y, mm.z, mm.w};
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
            w[k] = bf2(bf_lo(m[k]) > 0.f ? __uint_as_float(v[8 * c + 2 * k]) : 0.f,
                       bf_hi(m[k]) > 0.f ? __uint_as_float(v[8 * c + 2 * k + 1]) : 0.f);
          *a = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      if (!publish()) { ok = false; break; }
    }
    if (!ok) break;
    // dW1 = X^T dZ1
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
        mma_weight<64>(tmem + kTmW1, h1, x_buf(j), j == 0);
        umma_commit(bar_m);
      }
      ++commits;
      __syncwarp();
    }
    colsum(h1, gb1);
    wait_mma();
    if (!end_phase()) { ok = false; break; }
  }

  if (ok && tile0 < ntiles) {
    // this CTA's sums, in parameter order ([in][out]): lane = output column
    float *o = part + (size_t)blockIdx.x * kPartStride;
#pragma unroll 1
    for (int w = 0; w < 3; ++w) {
      const int in0 = kCols * h;
      if (w == 2 && in0 >= kMlpIn) break;
      float *dst = o + (w == 0 ? kMlpOW3 : (w == 1 ? kMlpOW2 : kMlpOW1)) + r;
      const uint32_t src = tmem + (w == 0 ? kTmW3 : (w == 1 ? kTmW2 : kTmW1)) + ((uint32_t)(q * 32) << 16) + in0;
      uint32_t v[kCols];
      tmem_ld32(src, v);
#pragma unroll
      for (int k = 0; k < kCols; ++k) dst[(in0 + k) * kMlpH] = __uint_as_float(v[k]);
    }
    // the row groups' column sums, in order; the features' stages are free
    float *sum = reinterpret_cast<float *>(mlp_smem + (xs - smem_u32(mlp_smem)));
    float *mine = sum + rg * 4 * kMlpH + 2 * cp;
    const float *src[4] = {gb1, gb2, gb3, gw4};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      mine[k * kMlpH] = src[k][0];
      mine[k * kMlpH + 1] = src[k][1];
    }
    float *red = sum + kRowGroups * 4 * kMlpH;
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
      gb4 += __shfl_xor_sync(0xffffffffu, gb4, k);
      sse += __shfl_xor_sync(0xffffffffu, sse, k);
    }
    if (lane == 0) { red[2 * (t >> 5)] = gb4; red[2 * (t >> 5) + 1] = sse; }
    __syncthreads();
    for (int i = t; i < 4 * kMlpH; i += kTrainThreads) {
      float a = sum[i];
#pragma unroll
      for (int k = 1; k < kRowGroups; ++k) a += sum[4 * kMlpH * k + i];
      o[kMlpOB1 + i] = a;
    }
    if (t < 2) o[kMlpOB4 + t] = ((red[t] + red[2 + t]) + red[4 + t]) + red[6 + t];
  }
  if (t == 0 && (!ok || !wok)) {
    *err = 1u;
    *bad = 1u;  // this CTA's sums are missing: mlp_reduce_kernel leaves everything as it is
    // copies and MMAs still in flight land before the CTA leaves (bounded)
    (void)mbar_wait(smem_u32(&wfull), 0);
    for (int i = consumed; i < issued; ++i) (void)mbar_wait(x_bar(i), x_par(i));
    for (int i = waited; i < commits; ++i) (void)mbar_wait(bar_m, (uint32_t)i & 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// ---------------------------------------------------------------------------
// Forward only: two groups of eight warps, each on a tile of its own (a warp
// holds 32 rows of one column half), and one warp that issues every copy and
// MMA.  A group has 128 columns of tensor memory for the accumulator and 64
// for the BF16 activations, which the epilogue writes there as the A operand
// of the next layer: they never pass through shared memory, where a 128 x 128
// x 16 step then reads 4 KB in its 64 cycles instead of 8.
//
// Predictions of 1.03M rows (features 132 MB): three GEMM kernels with the
// activations in memory 252 us; one kernel, four groups of four warps that
// each issued their own MMAs on operands in shared memory, 106; this one 80
// (73 on the device: the MMAs 38 at 68 cycles a step, the features 19 of
// memory time; no pipe is busy for much more than half of it, and a group
// waits for the other's part of the tensor pipe and of the issue slots).
// Three groups, the third with its activations in shared memory (four warps
// each, or eight on 32 columns at a time): 80 and 79.  An issuing warp per
// group: their MMAs interleave and both groups wait longer, 97 against 92 at
// the time.  Accumulator halves of 64 columns: a step takes as long as one
// of 128.
constexpr int kFwdGroups = 2, kFwdGroupThreads = 256, kFwdThreads = kFwdGroups * kFwdGroupThreads + 32;
constexpr int kFwdSmem = (int)(kWBytes + kFwdGroups * 2 * kBlkBytes) + 1024;  // + slack to align to 1024 B
constexpr uint32_t kTmAct = 128, kTmGroup = 256;  // the activations' columns; from group to group

__global__ void __launch_bounds__(kFwdThreads, 1) mlp_forward_kernel(
    const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw1,
    const __grid_constant__ CUtensorMap tw2, const __grid_constant__ CUtensorMap tw3, int M,
    const float *__restrict__ P, float *y, volatile unsigned int *err)
{
  extern __shared__ unsigned char mlp_smem[];
  // xfull: a group's two feature stages; mdone: its MMA has completed; ready:
  // its epilogue is through (the next MMA may read the activations, or after
  // layer 3 write over them)
  // half: the second column half's part of a result is in s_part
  __shared__ __align__(8) uint64_t wfull, xfull[kFwdGroups][2], mdone[kFwdGroups], ready[kFwdGroups], half[kFwdGroups];
  __shared__ float s_part[kFwdGroups][kTileM];
  __shared__ int xloads[kFwdGroups];  // feature tiles asked for
  __shared__ uint32_t tmem_base;
  __shared__ __align__(16) float s_bias[3][kMlpH], s_w4[kMlpH];
  const int g = warp_index() / (kFwdGroupThreads / 32);
  const int t = threadIdx.x % kFwdGroupThreads, lane = t & 31;
  const uint32_t w1 = (smem_u32(mlp_smem) + 1023u) & ~1023u, w2 = w1 + kW1Bytes, w3 = w2 + kW2Bytes;
  const int ntiles = (M + kTileM - 1) / kTileM, tstep = gridDim.x * kFwdGroups;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&wfull), 1);
    for (int i = 0; i < kFwdGroups; ++i) {
      mbar_init(smem_u32(&xfull[i][0]), 1);
      mbar_init(smem_u32(&xfull[i][1]), 1);
      mbar_init(smem_u32(&mdone[i]), 1);
      mbar_init(smem_u32(&ready[i]), kFwdGroupThreads);
      mbar_init(smem_u32(&half[i]), kTileM);
      xloads[i] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int i = threadIdx.x; i < 4 * kMlpH; i += kFwdThreads) {
    if (i < 3 * kMlpH) s_bias[i / kMlpH][i % kMlpH] = P[kMlpOB1 + i];
    else s_w4[i - 3 * kMlpH] = P[kMlpOW4 + i - 3 * kMlpH];
  }
  const float b4 = P[kMlpOB4];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);

  bool ok = true;
  if (g == kFwdGroups) {  // the issuing warp: in step, lane 0 issues
    {
      const bool lead = elect_one();
      const auto x_buf = [&](int gg, int i) { return w1 + kWBytes + (uint32_t)(2 * gg + (i & 1)) * kBlkBytes; };
      const auto load_x = [&](int gg, int i) {  // tile i of group gg, if there is one
        const int tile = gg * gridDim.x + blockIdx.x + i * tstep;
        if (tile >= ntiles) return;
        if (!lead) return;
        ++xloads[gg];
        mbar_expect_tx(smem_u32(&xfull[gg][i & 1]), kBlkBytes);
        tma_load_2d(x_buf(gg, i), &tx, 0, tile * kTileM, smem_u32(&xfull[gg][i & 1]));
      };
      for (int gg = 0; gg < kFwdGroups; ++gg) load_x(gg, 0);
      if (lead) {
        mbar_expect_tx(smem_u32(&wfull), kWBytes);
        tma_load_2d(w1, &tw1, 0, 0, smem_u32(&wfull));
        for (int s = 0; s < 2; ++s) {
          tma_load_2d(w2 + s * kBlkBytes, &tw2, s * kBlkCols, 0, smem_u32(&wfull));
          tma_load_2d(w3 + s * kBlkBytes, &tw3, s * kBlkCols, 0, smem_u32(&wfull));
        }
      }
      for (int gg = 0; gg < kFwdGroups; ++gg) load_x(gg, 1);
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&wfull), 0));
      int issued[kFwdGroups] = {};
      for (int i = 0; ok && (int)blockIdx.x + i * tstep < ntiles; ++i) {
#pragma unroll
        for (int layer = 0; layer < 3; ++layer) {
#pragma unroll
          for (int gg = 0; gg < kFwdGroups; ++gg) {
            const int n = 3 * i + layer;
            if (!ok || (int)(gg * gridDim.x + blockIdx.x) + i * tstep >= ntiles) continue;
            // the group is through with its last epilogue
            ok = __all_sync(0xffffffffu,
                            (n == 0 || mbar_wait(smem_u32(&ready[gg]), (uint32_t)(n - 1) & 1u)) &&
                                (layer != 0 || mbar_wait(smem_u32(&xfull[gg][i & 1]), (uint32_t)(i >> 1) & 1u)));
            if (!ok) continue;
            tc_fence_after();
            if (lead) {
              const uint32_t acc = tmem + gg * kTmGroup;
              if (layer == 0) mma_rows<1>(acc, x_buf(gg, i), w1);
              else mma_rows_tmem(acc, acc + kTmAct, layer == 1 ? w2 : w3);
              umma_commit(smem_u32(&mdone[gg]));
            }
            issued[gg] = n + 1;
            if (layer == 1) load_x(gg, i + 2);  // layer 1 has read the stage
            __syncwarp();
          }
        }
      }
      if (!ok && lead) {  // what is still in flight lands before the CTA leaves (bounded)
        (void)mbar_wait(smem_u32(&wfull), 0);
        for (int gg = 0; gg < kFwdGroups; ++gg) {
          if (issued[gg]) (void)mbar_wait(smem_u32(&mdone[gg]), (uint32_t)(issued[gg] - 1) & 1u);
          for (int j = max(0, xloads[gg] - 2); j < xloads[gg]; ++j)
            (void)mbar_wait(smem_u32(&xfull[gg][j & 1]), (uint32_t)(j >> 1) & 1u);
        }
      }
    }
    __syncwarp();
  } else {
    const int row = (t & 96) + (lane >> 2) + 8 * (lane & 3);  // the row whose result this thread sums
    const int h = t >> 7;                                     // column half
    const uint32_t acc = tmem + g * kTmGroup + ((uint32_t)(t & 96) << 16) + 64 * h;
    const uint32_t act = tmem + g * kTmGroup + ((uint32_t)(t & 96) << 16) + kTmAct + 32 * h;
    const uint32_t bar_m = smem_u32(&mdone[g]), bar_r = smem_u32(&ready[g]), bar_h = smem_u32(&half[g]);
    // bias and ReLU of a pair of columns
    const auto relu = [&](uint32_t lo, uint32_t hi, uint64_t bias) {
      const uint64_t x = f2_add(f2_pack(__uint_as_float(lo), __uint_as_float(hi)), bias);
      return bf2_relu(bf2(f2_lo(x), f2_hi(x)));
    };
    const auto pair = [&](const float *p, int j) {  // columns 8 j + 2 (lane % 4) + {0, 1} of the half
      return *reinterpret_cast<const uint64_t *>(p + 64 * h + 8 * j + 2 * (lane & 3));
    };
    int n = 0;  // the group's MMAs
    for (int tile = g * gridDim.x + blockIdx.x, i = 0; ok && tile < ntiles; tile += tstep, ++i) {
#pragma unroll 1
      for (int layer = 0; layer < 2; ++layer, ++n) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_m, (uint32_t)n & 1u));
        if (!ok) break;
        tc_fence_after();
        uint32_t v[64], w[32];
        tmem_ld_frag(acc, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint64_t bb = pair(s_bias[layer], j);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int e = 32 * (k >> 1) + 4 * j + 2 * (k & 1);
            w[16 * (k >> 1) + 2 * j + (k & 1)] = relu(v[e], v[e + 1], bb);
          }
        }
        tmem_st_frag(act, w);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(bar_r);
      }
      if (!ok) break;
      // layer 3 and the output layer: y = relu(.) . w4 + b4 on the BF16
      // activations: a thread's 16 columns of four rows, the sums of the four
      // threads that share the rows, then the two column halves
      ok = __all_sync(0xffffffffu, mbar_wait(bar_m, (uint32_t)n & 1u));
      if (!ok) break;
      ++n;
      tc_fence_after();
      uint64_t sum[4] = {0ull, 0ull, 0ull, 0ull};
      {
        uint32_t v[64];
        tmem_ld_frag(acc, v);
        tc_fence_before();
        mbar_arrive(bar_r);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint64_t bb = pair(s_bias[2], j), ww = pair(s_w4, j);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int e = 32 * (k >> 1) + 4 * j + 2 * (k & 1);
            const uint32_t a = relu(v[e], v[e + 1], bb);
            sum[k] = f2_fma(f2_pack(bf_lo(a), bf_hi(a)), ww, sum[k]);
          }
        }
      }
      float ys = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float x = f2_lo(sum[k]) + f2_hi(sum[k]);
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        if ((lane & 3) == k) ys = x;
      }
      // (the next tile's part is written after both halves have been ready for its layers)
      if (h == 1) {
        s_part[g][row] = ys;
        mbar_arrive(bar_h);
      } else {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_h, (uint32_t)i & 1u));
        if (ok && tile * kTileM + row < M) y[tile * (int64_t)kTileM + row] = (ys + s_part[g][row]) + b4;
      }
    }
  }
  if (!ok && lane == 0) *err = 1u;
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
}

// Sums of the CTAs' partial gradients, in a fixed order (four threads per
// parameter take a quarter of the CTAs each), into G; the mean squared error
// into *loss.  With lr > 0 also Adam (bias-corrected) on every parameter and
// the BF16 copies of the weight matrices, transposed to [out][in].  Where a
// CTA's wait ran out (*bad) its sums are missing, and nothing is written.
constexpr int kRedParams = 64;
__global__ void __launch_bounds__(4 * kRedParams) mlp_reduce_kernel(int ctas, const float *__restrict__ part, int rows,
                                                                    float *G, float *loss, float *P, float *m, float *v,
                                                                    float lr, float b1, float b2, float eps, float c1,
                                                                    float c2, __nv_bfloat16 *W16T,
                                                                    const unsigned int *bad)
{
  __shared__ float s[4][kRedParams];
  __shared__ unsigned int s_bad;
  const int k = threadIdx.x / kRedParams, l = threadIdx.x % kRedParams;
  const int i = blockIdx.x * kRedParams + l;  // < kPartStride
  const int lo = ctas * k / 4, hi = ctas * (k + 1) / 4;
  // (launched while the training kernel still runs: it is through, with its
  // writes visible, after this wait)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // (one load per block: every warp's of the same word queued up in one slice
  // of the L2, half a microsecond of a training step)
  if (threadIdx.x == 4 * kRedParams - 1) s_bad = __ldcg(bad);
  float a = 0.f;
  if (i <= kMlpParams) {
#pragma unroll 8
    for (int c = lo; c < hi; ++c) a += part[(size_t)c * kPartStride + i];
  }
  s[k][l] = a;
  __syncthreads();
  if (k != 0 || i > kMlpParams || s_bad != 0u) return;
  const float g = ((s[0][l] + s[1][l]) + s[2][l]) + s[3][l];
  if (i == kMlpParams) {
    *loss = g / (float)rows;
    return;
  }
  G[i] = g;
  if (!(lr > 0.f)) return;
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float p = P[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  P[i] = p;
  if (i < kMlpW16) W16T[transposed_index(i)] = __float2bfloat16(p);
}

__global__ void to_bf16_kernel(const float *__restrict__ src, __nv_bfloat16 *W16T)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpW16; i += gridDim.x * blockDim.x)
    W16T[transposed_index(i)] = __float2bfloat16(src[i]);
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor map of a rows x k BF16 matrix (row-major, k contiguous): boxes of
// 64 columns (128 B, the swizzle span) by 128 rows; rows beyond the matrix
// read as zeros.
bool make_map(CUtensorMap *map, const void *base, uint64_t k, uint64_t rows)
{
  const auto enc = tensor_map_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(base) & 15u) || k % kBlkCols) return false;
  const cuuint64_t dims[2] = {k, rows};
  const cuuint64_t strides[1] = {k * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBlkCols, (cuuint32_t)kTileM};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// ---------------------------------------------------------------------------
// per-vertex features: [x, y, z] scaled to the bounding box, the metric
// distance to the nearest stimulus (its start time plus the straight-line
// distance in the vertex's metric), cf, ct, the fibre angle in the xy-plane

namespace {

__device__ __forceinline__ unsigned int ord_key(float x)
{
  const unsigned int b = __float_as_uint(x);
  return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_val(unsigned int k)
{
  return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// Sums of the fibre, cf, ct and the number of its tets per vertex, eight
// floats each (two unused).  Bound by the atomics: a corner adds with two
// vector reductions (1M slab, 23.7M corners: 0.26 ms), not with six scalar
// ones (0.68 ms).
constexpr int kFeatAcc = 8;

__global__ void feat_accum_kernel(int64_t nT, const int32_t *__restrict__ tslots, const double *__restrict__ fib,
                                  const double *__restrict__ cf, const double *__restrict__ ct, float *acc)
{
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nT; e += (int64_t)gridDim.x * blockDim.x) {
    const float4 s = make_float4((float)fib[3 * e], (float)fib[3 * e + 1], (float)fib[3 * e + 2], (float)cf[e]);
    const float2 t = make_float2((float)ct[e], 1.f);
    const int4 v = reinterpret_cast<const int4 *>(tslots)[e];
    const int32_t vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float *q = acc + kFeatAcc * (int64_t)vs[k];
      atomicAdd(reinterpret_cast<float4 *>(q), s);
      atomicAdd(reinterpret_cast<float2 *>(q + 4), t);
    }
  }
}

// acc -> per-vertex fibre (unit), cf, ct in place and the distance in acc[6];
// reductions, all maxima from zero: red[0..2] complements of the bounding
// box's minimum, red[3..5] its maximum, red[6] the largest distance.  Each
// block reduces its vertices first (1M slab 0.048 ms; with an atomic per
// vertex on each of the seven words 0.16).
constexpr int kFeatThreads = 256;
__global__ void __launch_bounds__(kFeatThreads) feat_dist_kernel(int nV, const double *__restrict__ xyz, float *acc,
                                                                 int nseed, const int32_t *__restrict__ seed_v,
                                                                 const double *__restrict__ seed_t, unsigned int *red)
{
  __shared__ unsigned int s_red[7];
  if (threadIdx.x < 7) s_red[threadIdx.x] = 0u;
  __syncthreads();
  unsigned int m[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nV; v += gridDim.x * blockDim.x) {
    float *q = acc + kFeatAcc * (int64_t)v;
    const float p[3] = {(float)xyz[3 * (int64_t)v], (float)xyz[3 * (int64_t)v + 1], (float)xyz[3 * (int64_t)v + 2]};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      m[k] = max(m[k], ~ord_key(p[k]));
      m[3 + k] = max(m[3 + k], ord_key(p[k]));
    }
    const float4 s = *reinterpret_cast<const float4 *>(q);
    const float2 t = *reinterpret_cast<const float2 *>(q + 4);
    if (!(t.y > 0.f)) continue;  // (acc[6] is zero)
    float f0 = s.x, f1 = s.y, f2 = s.z;
    const float fn = sqrtf(f0 * f0 + f1 * f1 + f2 * f2);
    if (fn > 0.f) { f0 /= fn; f1 /= fn; f2 /= fn; } else { f0 = 1.f; f1 = f2 = 0.f; }
    const float a = s.w / t.y, b = t.x / t.y;
    const float ia = 1.f / (a * a), ib = 1.f / (b * b);
    float best = INFINITY;
    for (int i = 0; i < nseed; ++i) {
      const int64_t c = seed_v[i];
      const float dx = p[0] - (float)xyz[3 * c], dy = p[1] - (float)xyz[3 * c + 1], dz = p[2] - (float)xyz[3 * c + 2];
      const float along = dx * f0 + dy * f1 + dz * f2;
      const float d2 = ia * along * along + ib * (dx * dx + dy * dy + dz * dz - along * along);
      best = fminf(best, (float)seed_t[i] + sqrtf(fmaxf(d2, 0.f)));
    }
    *reinterpret_cast<float4 *>(q) = make_float4(f0, f1, f2, a);
    *reinterpret_cast<float4 *>(q + 4) = make_float4(b, t.y, best, 0.f);
    if (best < INFINITY) m[6] = max(m[6], ord_key(best));
  }
#pragma unroll
  for (int k = 0; k < 7; ++k) {
    const unsigned int w = __reduce_max_sync(0xffffffffu, m[k]);
    if ((threadIdx.x & 31) == 0 && w != 0u) atomicMax(&s_red[k], w);
  }
  __syncthreads();
  if (threadIdx.x < 7 && s_red[threadIdx.x] != 0u) atomicMax(red + threadIdx.x, s_red[threadIdx.x]);
}

// The feature rows: a warp computes 32 of them, a lane each, and writes them
// together, 512 bytes a store (kWide: X on a 16-byte boundary; 1M slab, 132 MB:
// 0.028 ms).  Else each lane writes its row element by element (0.56 ms).
template <bool kWide>
__global__ void __launch_bounds__(kFeatThreads) feat_write_kernel(int nV, const double *__restrict__ xyz,
                                                                  const float *__restrict__ acc,
                                                                  const unsigned int *__restrict__ red, __nv_bfloat16 *X)
{
  float lo[3], hi[3];
  for (int k = 0; k < 3; ++k) { lo[k] = ord_val(~red[k]); hi[k] = ord_val(red[3 + k]); }
  const float T = fmaxf(ord_val(red[6]), 1e-30f);
  const int lane = threadIdx.x & 31;
  const int warps = (int)(gridDim.x * blockDim.x / 32);
  for (int64_t base = 32 * (int64_t)((blockIdx.x * blockDim.x + threadIdx.x) / 32); base < nV; base += 32 * (int64_t)warps) {
    const int64_t v = base + lane;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (v < nV) {
      const float4 s = *reinterpret_cast<const float4 *>(acc + kFeatAcc * v);
      const float4 t = *reinterpret_cast<const float4 *>(acc + kFeatAcc * v + 4);
      float f[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float c = 0.5f * (lo[k] + hi[k]), h = fmaxf(0.5f * (hi[k] - lo[k]), 1e-30f);
        f[k] = ((float)xyz[3 * v + k] - c) / h;
      }
      const bool in = t.y > 0.f;
      const float f3 = in ? t.z / T : 0.f, f4 = in ? s.w : 0.f, f5 = in ? t.x : 0.f;
      const float f6 = in ? atan2f(s.y, s.x) * 0.31830988618379067f : 0.f;
      w = make_uint4(bf2(f[0], f[1]), bf2(f[2], f3), bf2(f4, f5), bf2(f6, 0.f));
    }
    if (kWide) {
      uint4 *out = reinterpret_cast<uint4 *>(X + base * kMlpIn);
#pragma unroll
      for (int i = 0; i < kMlpIn / 8; ++i) {
        const int row = 4 * i + lane / 8;
        uint4 x;
        x.x = __shfl_sync(0xffffffffu, w.x, row);
        x.y = __shfl_sync(0xffffffffu, w.y, row);
        x.z = __shfl_sync(0xffffffffu, w.z, row);
        x.w = __shfl_sync(0xffffffffu, w.w, row);
        if (lane % 8 != 0) x = make_uint4(0u, 0u, 0u, 0u);
        if (base + row < nV) out[32 * i + lane] = x;
      }
    } else if (v < nV) {
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
      unsigned short *row = reinterpret_cast<unsigned short *>(X) + v * kMlpIn;
#pragma unroll
      for (int k = 0; k < kMlpIn; ++k) row[k] = k < 8 ? (unsigned short)(ws[k / 2] >> (16 * (k & 1))) : (unsigned short)0;
    }
  }
}

}  // namespace

size_t features_scratch(int nV) { return kFeatAcc * (size_t)nV + kFeatAcc; }

cudaError_t launch_features(int nV, int64_t nT, const double *xyz, const int32_t *tslots, const double *fib,
                            const double *cf, const double *ct, int nseed, const int32_t *seed_v,
                            const double *seed_t, float *scratch, unsigned int **red_out, void *X, cudaStream_t st)
{
  cudaError_t e;
  if ((e = cudaMemsetAsync(scratch, 0, sizeof(float) * features_scratch(nV), st)) != cudaSuccess) return e;
  unsigned int *red = reinterpret_cast<unsigned int *>(scratch + kFeatAcc * (size_t)nV);
  *red_out = red;
  const int grid = 152 * 8;
  __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(X);
  feat_accum_kernel<<<grid, kFeatThreads, 0, st>>>(nT, tslots, fib, cf, ct, scratch);
  feat_dist_kernel<<<grid, kFeatThreads, 0, st>>>(nV, xyz, scratch, nseed, seed_v, seed_t, red);
  if (reinterpret_cast<uintptr_t>(X) % 16 == 0)
    feat_write_kernel<true><<<grid, kFeatThreads, 0, st>>>(nV, xyz, scratch, red, out);
  else
    feat_write_kernel<false><<<grid, kFeatThreads, 0, st>>>(nV, xyz, scratch, red, out);
  return cudaGetLastError();
}

float features_scale(const unsigned int *host_red)
{
  const unsigned int k = host_red[6];
  const unsigned int b = (k >> 31) ? (k & 0x7fffffffu) : ~k;
  float f;
  memcpy(&f, &b, sizeof(f));
  return f;
}

}  // namespace fimgb

// ---------------------------------------------------------------------------
// C ABI of the network (include/fim.h)

#include "../../include/fim.h"

using namespace fimgb;

static_assert(FIM_MLP_PARAMS == kMlpParams, "parameter count of the C ABI");
static_assert(FIM_MLP_INPUTS == kMlpIn, "feature width of the C ABI");

struct fim_mlp {
  int device = 0, sms = 0;
  cudaStream_t st = nullptr;
  float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;
  __nv_bfloat16 *W16T = nullptr;     // BF16 weights, [out][in]
  CUtensorMap tw1, tw2, tw3;
  float *part = nullptr;             // partial gradients of up to sms CTAs
  unsigned int *bad = nullptr;       // (behind them) set by a training CTA whose bounded wait ran out
  // mapped host memory: the loss of the last reduction, and a word set by a
  // kernel whose bounded wait ran out (read after the stream has drained)
  struct Result { float loss; unsigned int err; };
  volatile Result *h_res = nullptr;
  Result *d_res = nullptr;
  float *y = nullptr;                // predictions on their way to an output that the kernel cannot write directly
  int64_t y_cap = 0;
  int64_t steps = 0;
};

namespace {

int mlp_fail(const char *what, cudaError_t e)
{
  cudaGetLastError();  // reported here, not again by the next launch's check
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  set_last_error(m.c_str());
  return e == cudaErrorMemoryAllocation ? FIM_ERR_OUT_OF_MEMORY : FIM_ERR_CUDA;
}

#define MLP_TRY(what, call)                                   \
  do {                                                        \
    cudaError_t _e = (call);                                  \
    if (_e != cudaSuccess) return mlp_fail((what), _e);       \
  } while (0)

// Reports a bounded wait that ran out (after the stream has drained).
int mlp_status(fim_mlp *m, const char *who)
{
  if (m->h_res->err == 0) return FIM_OK;
  m->h_res->err = 0;
  MLP_TRY(who, cudaMemsetAsync(m->bad, 0, sizeof *m->bad, m->st));
  std::string msg = std::string(who) + ": a tensor-core GEMM wait ran out (results discarded)";
  set_last_error(msg.c_str());
  return FIM_ERR_TIMEOUT;
}

int mlp_check_n(int64_t n, const char *who)
{
  if (n <= 0 || n % 64 != 0 || n > (int64_t)1 << 30) {
    std::string msg = std::string(who) + ": row count must be a positive multiple of 64";
    set_last_error(msg.c_str());
    return FIM_ERR_INVALID_ARGUMENT;
  }
  return FIM_OK;
}

// Launches the network over n rows of X: predictions into y, or with targets
// the partial gradients of *ctas CTAs into m->part.
cudaError_t mlp_launch(fim_mlp *m, int n, const void *X, float *y, const float *tgt, int *ctas)
{
  CUtensorMap tx;
  if (!make_map(&tx, X, kMlpIn, (uint64_t)n)) return cudaErrorInvalidValue;
  const int ntiles = (n + kTileM - 1) / kTileM;
  const int grid = std::min(ntiles, m->sms);
  if (ctas) *ctas = grid;
  if (tgt)
    mlp_train_kernel<<<grid, kTrainThreads, kTrainSmem, m->st>>>(tx, m->tw1, m->tw2, m->tw3, n, m->P, tgt, m->part,
                                                                 m->bad, &m->d_res->err);
  else
    mlp_forward_kernel<<<grid, kFwdThreads, kFwdSmem, m->st>>>(tx, m->tw1, m->tw2, m->tw3, n, m->P, y, &m->d_res->err);
  return cudaGetLastError();
}

// Loss and gradients of n rows; with lr > 0 also an Adam step.  Waits.
int mlp_gradients(fim_mlp *m, int64_t n, const void *X, const float *tgt, float lr, float *grads, float *loss,
                  const char *who)
{
  const float b1 = 0.9f, b2 = 0.999f;
  const int64_t step = m->steps + (lr > 0.f ? 1 : 0);  // counted once its update is made
  const float c1 = 1.f - std::pow(b1, (float)step), c2 = 1.f - std::pow(b2, (float)step);  // (unused without an update)
  int ctas = 0;
  MLP_TRY(who, mlp_launch(m, (int)n, X, nullptr, tgt, &ctas));
  // the launch of the sums is prepared while the training kernel runs (step of
  // 4,096 rows 54 -> 50 us with the parameters read back, gradients of 131,136
  // rows 94 -> 91; let go already at that kernel's start: no better)
  cudaLaunchAttribute early[1] = {};
  early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kPartStride / kRedParams);
  cfg.blockDim = dim3(4 * kRedParams);
  cfg.stream = m->st;
  cfg.attrs = early;
  cfg.numAttrs = 1;
  MLP_TRY(who, cudaLaunchKernelEx(&cfg, mlp_reduce_kernel, ctas, (const float *)m->part, (int)n, m->G, &m->d_res->loss,
                                  m->P, m->M, m->V, lr, b1, b2, 1e-8f, c1, c2, m->W16T,
                                  (const unsigned int *)m->bad));
  if (grads)
    MLP_TRY(who, cudaMemcpyAsync(grads, m->G, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost, m->st));
  MLP_TRY(who, cudaStreamSynchronize(m->st));
  if (loss) *loss = m->h_res->loss;
  const int rc = mlp_status(m, who);
  if (rc == FIM_OK) m->steps = step;
  return rc;
}

}  // namespace

extern "C" int fim_mlp_create(int device, uint64_t seed, fim_mlp **out)
{
  if (!out) { set_last_error("fim_mlp_create: out is NULL"); return FIM_ERR_INVALID_ARGUMENT; }
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    set_last_error("fim_mlp_create: no CUDA device");
    return FIM_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= ndev) { set_last_error("fim_mlp_create: bad device"); return FIM_ERR_INVALID_ARGUMENT; }
  MLP_TRY("fim_mlp_create: set device", cudaSetDevice(device));
  fim_mlp *m = new fim_mlp();
  m->device = device;
  int rc = FIM_OK;
  auto fail = [&](int code) { fim_mlp_destroy(m); return code; };
  cudaError_t e;
  void *h = nullptr;
  if ((e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess ||
      (e = cudaStreamCreateWithFlags(&m->st, cudaStreamDefault)) != cudaSuccess ||
      (e = cudaMalloc(&m->P, sizeof(float) * kMlpParams)) != cudaSuccess ||
      (e = cudaMalloc(&m->G, sizeof(float) * kMlpParams)) != cudaSuccess ||
      (e = cudaMalloc(&m->M, sizeof(float) * kMlpParams)) != cudaSuccess ||
      (e = cudaMalloc(&m->V, sizeof(float) * kMlpParams)) != cudaSuccess ||
      (e = cudaMalloc(&m->W16T, sizeof(__nv_bfloat16) * kMlpW16)) != cudaSuccess ||
      (e = cudaMalloc(&m->part, sizeof(float) * (kPartStride * (size_t)m->sms + 1))) != cudaSuccess ||
      (e = cudaHostAlloc(&h, sizeof(fim_mlp::Result), cudaHostAllocMapped)) != cudaSuccess)
    return fail(mlp_fail("fim_mlp_create", e));
  m->bad = reinterpret_cast<unsigned int *>(m->part + kPartStride * (size_t)m->sms);
  if ((e = cudaMemsetAsync(m->bad, 0, sizeof *m->bad, m->st)) != cudaSuccess) return fail(mlp_fail("fim_mlp_create", e));
  m->h_res = static_cast<volatile fim_mlp::Result *>(h);
  m->h_res->loss = 0.f;
  m->h_res->err = 0;
  void *d = nullptr;
  if ((e = cudaHostGetDevicePointer(&d, h, 0)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem)) !=
          cudaSuccess ||
      (e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem)) !=
          cudaSuccess)
    return fail(mlp_fail("fim_mlp_create", e));
  m->d_res = static_cast<fim_mlp::Result *>(d);
  if (!make_map(&m->tw1, m->W16T + kMlpOW1, kMlpIn, kMlpH) || !make_map(&m->tw2, m->W16T + kMlpOW2, kMlpH, kMlpH) ||
      !make_map(&m->tw3, m->W16T + kMlpOW3, kMlpH, kMlpH))
    return fail(mlp_fail("fim_mlp_create", cudaErrorInvalidValue));
  // He initialisation (fixed seed); padded input rows and biases zero
  std::vector<float> h0(kMlpParams, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  for (int i = 0; i < kMlpFeatures; ++i)
    for (int j = 0; j < kMlpH; ++j) h0[kMlpOW1 + i * kMlpH + j] = nd(rng) * std::sqrt(2.f / kMlpFeatures);
  for (int i = 0; i < kMlpH * kMlpH; ++i) h0[kMlpOW2 + i] = nd(rng) * std::sqrt(2.f / kMlpH);
  for (int i = 0; i < kMlpH * kMlpH; ++i) h0[kMlpOW3 + i] = nd(rng) * std::sqrt(2.f / kMlpH);
  for (int i = 0; i < kMlpH; ++i) h0[kMlpOW4 + i] = nd(rng) * std::sqrt(1.f / kMlpH);
  rc = fim_mlp_set_params(m, h0.data());
  if (rc != FIM_OK) return fail(rc);
  *out = m;
  return FIM_OK;
}

extern "C" int fim_mlp_destroy(fim_mlp *m)
{
  if (!m) return FIM_OK;
  cudaSetDevice(m->device);
  if (m->st) cudaStreamSynchronize(m->st);
  cudaFree(m->P); cudaFree(m->G); cudaFree(m->M); cudaFree(m->V); cudaFree(m->W16T); cudaFree(m->part);
  cudaFree(m->y);
  if (m->h_res) cudaFreeHost(const_cast<fim_mlp::Result *>(m->h_res));
  if (m->st) cudaStreamDestroy(m->st);
  delete m;
  return FIM_OK;
}

extern "C" int fim_mlp_set_params(fim_mlp *m, const float *params)
{
  if (!m || !params) { set_last_error("fim_mlp_set_params: NULL argument"); return FIM_ERR_INVALID_ARGUMENT; }
  MLP_TRY("fim_mlp_set_params: set device", cudaSetDevice(m->device));
  MLP_TRY("fim_mlp_set_params", cudaMemcpyAsync(m->P, params, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice, m->st));
  MLP_TRY("fim_mlp_set_params", cudaMemsetAsync(m->M, 0, sizeof(float) * kMlpParams, m->st));
  MLP_TRY("fim_mlp_set_params", cudaMemsetAsync(m->V, 0, sizeof(float) * kMlpParams, m->st));
  to_bf16_kernel<<<64, 256, 0, m->st>>>(m->P, m->W16T);
  MLP_TRY("fim_mlp_set_params", cudaGetLastError());
  MLP_TRY("fim_mlp_set_params", cudaStreamSynchronize(m->st));
  m->steps = 0;
  return FIM_OK;
}

extern "C" int fim_mlp_get_params(const fim_mlp *m, float *params)
{
  if (!m || !params) { set_last_error("fim_mlp_get_params: NULL argument"); return FIM_ERR_INVALID_ARGUMENT; }
  MLP_TRY("fim_mlp_get_params: set device", cudaSetDevice(m->device));
  MLP_TRY("fim_mlp_get_params", cudaMemcpy(params, m->P, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
  return FIM_OK;
}

extern "C" int fim_mlp_gradients(fim_mlp *m, int64_t n, const void *d_features, const float *d_targets,
                                 float *grads, float *loss)
{
  if (!m || !d_features || !d_targets || !grads) {
    set_last_error("fim_mlp_gradients: NULL argument");
    return FIM_ERR_INVALID_ARGUMENT;
  }
  int rc;
  if ((rc = mlp_check_n(n, "fim_mlp_gradients")) != FIM_OK) return rc;
  MLP_TRY("fim_mlp_gradients: set device", cudaSetDevice(m->device));
  return mlp_gradients(m, n, d_features, d_targets, 0.f, grads, loss, "fim_mlp_gradients");
}

extern "C" int fim_mlp_train_step(fim_mlp *m, int64_t n, const void *d_features, const float *d_targets, float lr,
                                  float *loss)
{
  if (!m || !d_features || !d_targets) {
    set_last_error("fim_mlp_train_step: NULL argument");
    return FIM_ERR_INVALID_ARGUMENT;
  }
  if (!(lr > 0.f) || !std::isfinite(lr)) { set_last_error("fim_mlp_train_step: bad learning rate"); return FIM_ERR_INVALID_ARGUMENT; }
  int rc;
  if ((rc = mlp_check_n(n, "fim_mlp_train_step")) != FIM_OK) return rc;
  MLP_TRY("fim_mlp_train_step: set device", cudaSetDevice(m->device));
  return mlp_gradients(m, n, d_features, d_targets, lr, nullptr, loss, "fim_mlp_train_step");
}

// Test hook (not part of include/fim.h): leaves the error words as a training
// CTA whose wait ran out does, so that the next training call finds them.
extern "C" int fim_mlp_test_timeout(fim_mlp *m)
{
  if (!m) { set_last_error("fim_mlp_test_timeout: NULL argument"); return FIM_ERR_INVALID_ARGUMENT; }
  MLP_TRY("fim_mlp_test_timeout: set device", cudaSetDevice(m->device));
  const unsigned int one = 1u;
  MLP_TRY("fim_mlp_test_timeout", cudaMemcpyAsync(m->bad, &one, sizeof one, cudaMemcpyHostToDevice, m->st));
  MLP_TRY("fim_mlp_test_timeout", cudaStreamSynchronize(m->st));
  m->h_res->err = 1;
  return FIM_OK;
}

extern "C" int fim_mlp_predict(fim_mlp *m, int64_t n, const void *d_features, float *d_out)
{
  if (!m || !d_features || !d_out) { set_last_error("fim_mlp_predict: NULL argument"); return FIM_ERR_INVALID_ARGUMENT; }
  int rc;
  if ((rc = mlp_check_n(n, "fim_mlp_predict")) != FIM_OK) return rc;
  MLP_TRY("fim_mlp_predict: set device", cudaSetDevice(m->device));
  // The kernel writes the predictions in place unless d_out is not aligned
  // to a float, overlaps the features it still reads, or is not on the device.
  const uintptr_t x = reinterpret_cast<uintptr_t>(d_features), o = reinterpret_cast<uintptr_t>(d_out);
  const uintptr_t xn = sizeof(__nv_bfloat16) * kMlpIn * (uintptr_t)n, on = sizeof(float) * (uintptr_t)n;
  const bool direct = o % sizeof(float) == 0 && (o + on <= x || x + xn <= o) && on_device(d_out, m->device);
  if (!direct && n > m->y_cap) {
    cudaFree(m->y);
    m->y = nullptr;
    m->y_cap = 0;
    MLP_TRY("fim_mlp: activations", cudaMalloc(&m->y, sizeof(float) * n));
    m->y_cap = n;
  }
  MLP_TRY("fim_mlp_predict: forward", mlp_launch(m, (int)n, d_features, direct ? d_out : m->y, nullptr, nullptr));
  if (!direct)
    MLP_TRY("fim_mlp_predict", cudaMemcpyAsync(d_out, m->y, sizeof(float) * n, cudaMemcpyDeviceToDevice, m->st));
  MLP_TRY("fim_mlp_predict", cudaStreamSynchronize(m->st));
  return mlp_status(m, "fim_mlp_predict");
}
