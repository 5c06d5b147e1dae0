// General BF16 GEMM on the 5th-generation tensor cores (tcgen05) with FP32
// accumulation, for the contractions of the learned corrector (pointwise
// channel mixing, its weight gradients, the per-mode complex channel mixing and
// the partial DFT stages of its spectral layers).
//
//   D (M x N) = A (M x K) . B (N x K)^T,   A and B rounded to bfloat16.
//
// Operands are read from FP32 arrays of any 2-level strided layout: element
// (r, k) of an operand sits at (r / rc) * s1 + (r % rc) * s2 + (k / kc) * t1 +
// (k % kc) * t2.  The tensor cores read both from shared memory in the K-major,
// 128-byte-swizzled layout (8-row atoms of 128 B, 16-byte chunk c of row r at
// chunk c ^ (r mod 8)).  Output element (r, c) is written at the same kind of
// strided address, so results land directly in pixel-major or transposed
// layouts.  Epilogue: z = acc (+ bias[c]) (+ add[r, c]); out = z or out += z;
// optionally act = gelu(z) (tanh form) into a second array.
//
// Main path (gemm_ws_kernel): a persistent, warp-specialised kernel; A is
// staged in FP32 by bulk or asynchronous copies and rounded to bfloat16 in
// shared memory, B comes from a small packed image (pack_kernel, or
// pack_cplx_kernel for the real embedding of a complex product) or, for the
// long-K weight gradients (N <= 32), is staged and rounded like A while K is
// split over the CTAs.
//
// What bounds it: the products here are narrow (32 to 256 columns), so each is a
// stream over one or two activations and the tensor cores are idle most of the
// time; what is left above the memory time is the instruction chain of a block
// (one warp per scheduler and role).  Hence the roles: four warps that only round,
// one that issues the bulk copies, one that moves the packed B, one that issues
// the MMAs, eight that finish tiles; registers moved from the former to the
// latter (128 at launch -> 120 / 56 / 168), for a spill costs a trip to L2 once
// shared memory has taken the L1; one loop per operand and output form, because
// a quarter of the stalls were instruction fetch when the forms shared one; and
// no division between one block and the next.  At 32 x 256^2 pixels, 32 channels
// (us, before these -> now, memory time at the measured copy rate):
//   pointwise + add + gelu    384 -> 199 (158)   weight gradient   456 -> 160 (79)
//   pointwise, plain          241 ->  95  (79)   x transform       109 ->  69 (49)
//   inverse x                 101 ->  72  (49)   inverse x, added  194 -> 130 (89)
//   y transform                75 ->  28  (12)   inverse y          45 ->  31 (12)
//   mixing                     70 ->  25   (5)
// The per-tile kernel (gemm_kernel, both operands packed)
// remains for split-K products with N > 32.
#include "msx.h"
#include "msx_internal.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cstring>

namespace msx {
namespace tg {

constexpr int BM = 128, BK = 64, STAGES = 3;
constexpr int A_BYTES = BM * BK * 2;  // 16 KB per (tile, K block)

__host__ __device__ __forceinline__ uint32_t sw128(int row, int k) {
  return (uint32_t)row * 128u + ((uint32_t)((k >> 3) ^ (row & 7)) << 4) + (uint32_t)(k & 7) * 2u;
}

__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

template <int BN>
struct Cfg {
  static_assert(BN == 32 || BN == 64 || BN == 128 || BN == 256, "BN must be 32, 64, 128 or 256");
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;
  // kind::f16: D f32 (bit 4), A bf16 (bits 7-9 = 1), B bf16 (bits 10-12 = 1), K-major both, N >> 3, M >> 4
  static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                    ((uint32_t)(BM >> 4) << 24);
};

__device__ __forceinline__ float gelu_t(float z) {
  const float u = 0.7978845608028654f * (z + 0.044715f * z * z * z);
  return 0.5f * z * (1.f + tanhf(u));
}

__host__ __device__ __forceinline__ long long addr_of(const Addr& a, long long r, long long k) {
  return (r / a.rc) * a.s1 + (r % a.rc) * a.s2 + (k / a.kc) * a.t1 + (k % a.kc) * a.t2;
}

// img[(tile * kblocks + kb)][row][k] (swizzled) = bf16(src(r, k)); zero outside rows x K.
// One thread per (padded row, 8 consecutive k): 16 bytes out.  The row part of the
// address and the split of k0 are computed once per thread; the 8 elements step
// through k incrementally, with two 16-byte loads when they are contiguous.
__global__ void pack_kernel(const float* __restrict__ src, Addr a, long long rows, long long K, int tile_rows,
                            long long rows_pad, int kblocks, uint4* __restrict__ img) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long chunks = (long long)kblocks * (BK / 8);
  if (i >= rows_pad * chunks) return;
  const long long r = i / chunks;
  const int ch = (int)(i - r * chunks);
  const long long k0 = (long long)ch * 8;
  __align__(16) __nv_bfloat16 v[8];
  if (r < rows && k0 < K) {
    const float* base = src + (r / a.rc) * a.s1 + (r % a.rc) * a.s2;
    if (a.kc == 1 && a.t1 == 1 && k0 + 8 <= K && ((reinterpret_cast<uintptr_t>(base + k0) & 15u) == 0)) {
      const float4 lo = __ldg(reinterpret_cast<const float4*>(base + k0));
      const float4 hi = __ldg(reinterpret_cast<const float4*>(base + k0) + 1);
      v[0] = __float2bfloat16_rn(lo.x); v[1] = __float2bfloat16_rn(lo.y);
      v[2] = __float2bfloat16_rn(lo.z); v[3] = __float2bfloat16_rn(lo.w);
      v[4] = __float2bfloat16_rn(hi.x); v[5] = __float2bfloat16_rn(hi.y);
      v[6] = __float2bfloat16_rn(hi.z); v[7] = __float2bfloat16_rn(hi.w);
    } else {
      long long q = k0 / a.kc, rem = k0 - q * a.kc;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = (k0 + j < K) ? __ldg(base + q * a.t1 + rem * a.t2) : 0.f;
        v[j] = __float2bfloat16_rn(x);
        if (++rem == a.kc) { rem = 0; ++q; }
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __float2bfloat16_rn(0.f);
  }
  const long long tile = r / tile_rows;
  const int row = (int)(r - tile * tile_rows), kb = (int)(k0 / BK);
  const size_t byte = ((size_t)tile * kblocks + kb) * ((size_t)tile_rows * BK * 2) + sw128(row, (int)(k0 % BK));
  img[byte / 16] = *reinterpret_cast<const uint4*>(v);
}

// Real embedding of a complex product, packed like pack_kernel: B is N x K with
// N = 2 hn, K = 2 hk; row n = (bn, i) = (n / hn, n % hn), column k = (bk, j); the
// element is src[i si + j sj + (bn xor bk) sp] (a complex array, its parts sp apart),
// negated where (bn, bk) = (0, 1) (neg = 1) or (1, 0) (neg = 2).  With the
// right orientation of src, D = A B^T then gives real and imaginary parts of a
// complex product in one GEMM: [Re, Im] of x z^T is [xr, xi] against rows
// [zr, -zi] and [zi, zr].
__global__ void pack_cplx_kernel(const float* __restrict__ src, long long si, long long sj, long long sp,
                                 long long src_bs, int hn, int hk, int neg, int tile_rows, int rows_pad, int kblocks, uint4* __restrict__ img,
                                 int batch) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long chunks = (long long)kblocks * (BK / 8);
  const long long per = (long long)rows_pad * chunks;
  if (i >= per * batch) return;
  const long long bt = i / per;
  i -= bt * per;
  src += bt * src_bs;
  img += bt * (per * 8 * 2 / 16);
  // neighbouring threads along whichever index is nearer in src
  const int r = si < sj ? (int)(i % rows_pad) : (int)(i / chunks);
  const int ch = si < sj ? (int)(i / rows_pad) : (int)(i - (long long)r * chunks);
  const int k0 = ch * 8;
  __align__(16) __nv_bfloat16 v[8];
  const int N = 2 * hn, K = 2 * hk;
  const int bn = r / hn, ii = r - (r / hn) * hn;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int k = k0 + j;
    float x = 0.f;
    if (r < N && k < K) {
      const int bk = k / hk, jj = k - bk * hk;
      x = __ldg(src + ii * si + jj * sj + (bn ^ bk) * sp);
      if ((neg == 1 && bn == 0 && bk == 1) || (neg == 2 && bn == 1 && bk == 0)) x = -x;
    }
    v[j] = __float2bfloat16_rn(x);
  }
  const int tile = r / tile_rows, row = r - tile * tile_rows, kb = k0 / BK;
  const size_t byte = ((size_t)tile * kblocks + kb) * ((size_t)tile_rows * BK * 2) + sw128(row, k0 % BK);
  img[byte / 16] = *reinterpret_cast<const uint4*>(v);
}

// Per-tile kernel: one CTA of 128 threads per 128 x BN tile of D and K split.
// Thread 0 moves each (tile, K block) of the packed images with one bulk copy into
// STAGES stages (full/empty mbarriers), thread 32 issues tcgen05.mma (M = 128,
// N = BN, K = 16) and commits each stage to its empty barrier; all four warps read
// the accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = tile rows).
// Every wait is bounded; on a timeout the kernel sets *err, waits (bounded) for its
// MMAs, frees its tensor memory and returns.
// With part != null the CTA (tile, split) sums K blocks [split * kper, ...) and
// writes its raw 128 x BN partial to part[(split * tiles + tile) * 128 * BN].
template <int BN>
__global__ void __launch_bounds__(128) gemm_kernel(const uint8_t* __restrict__ A, const uint8_t* __restrict__ B,
                                                   int kblocks, int ntiles_n, int ntiles_total, int kper,
                                                   float* __restrict__ part, Epi e, int* __restrict__ err) {
  using C = Cfg<BN>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t full[STAGES], empty[STAGES], done;
  __shared__ uint32_t tmem_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = ntiles_total;
  const int split = (int)blockIdx.x / tiles, tile = (int)blockIdx.x % tiles;
  const int mt = tile / ntiles_n, nt = tile % ntiles_n;
  const int kb0 = split * kper, kb1 = kb0 + kper < kblocks ? kb0 + kper : kblocks;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 32) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    fence_mbar_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;

  if (threadIdx.x == 0) {  // producer
    const uint8_t* a_tile = A + (size_t)mt * kblocks * A_BYTES;
    const uint8_t* b_tile = B + (size_t)nt * kblocks * C::B_BYTES;
    for (int i = 0; i < kb1 - kb0; ++i) {
      const int kb = kb0 + i, s = i % STAGES;
      if (i >= STAGES && !mbar_wait_bounded(&empty[s], ((i / STAGES) - 1) & 1)) {
        atomicOr(err, 2);
        break;
      }
      uint8_t* st = smem + s * C::STAGE_BYTES;
      mbar_expect_tx(&full[s], C::STAGE_BYTES);
      bulk_g2s(st, a_tile + (size_t)kb * A_BYTES, A_BYTES, &full[s]);
      bulk_g2s(st + A_BYTES, b_tile + (size_t)kb * C::B_BYTES, C::B_BYTES, &full[s]);
    }
  } else if (threadIdx.x == 32) {  // MMA issuer
    for (int i = 0; i < kb1 - kb0; ++i) {
      const int s = i % STAGES;
      if (!mbar_wait_bounded(&full[s], (i / STAGES) & 1)) {
        atomicOr(err, 4);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t st = smem_u32(smem + s * C::STAGE_BYTES);
#pragma unroll
      for (int j = 0; j < BK / 16; ++j) {
        const uint32_t off = (uint32_t)j * 32u;
        const uint32_t acc = (i > 0 || j > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t .reg .pred p;\n\t setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
            "l"(sdesc(st + off)), "l"(sdesc(st + A_BYTES + off)), "r"(C::IDESC), "r"(acc)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&empty[s]))
                   : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&done))
                 : "memory");
  }
  __syncwarp();
  const bool ok = mbar_wait_bounded(&done, 0);
  if (!ok && lane == 0) atomicOr(err, 8);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    const long long r = (long long)mt * BM + warp * 32 + lane;
    const bool row_ok = r < e.M;
    const long long rbase = row_ok ? (r / e.out.rc) * e.out.s1 + (r % e.out.rc) * e.out.s2 : 0;
    const bool split_cols = e.out.kc != 1;
    const bool stage_cols = !split_cols && e.out.t1 == 1;
    for (int c0 = 0; c0 < BN; c0 += 32) {
      uint32_t v[32];
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
          "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
            "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
            "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
            "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
          : "r"(taddr)
          : "memory");
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (!part && stage_cols) {
        // columns contiguous in the output: pass the warp's 32 x 32 block through shared
        // memory (the pipeline stages are idle now) and store each row with the lanes
        // along its columns
        float* blk = reinterpret_cast<float*>(smem) + warp * (32 * 33);
#pragma unroll
        for (int i = 0; i < 32; ++i) blk[lane * 33 + i] = __uint_as_float(v[i]);
        __syncwarp();
        const int c = nt * BN + c0 + lane;
        const float bias_c = (e.bias && c < e.N) ? __ldg(e.bias + c) : 0.f;
        for (int rr = 0; rr < 32; ++rr) {
          const long long rw = (long long)mt * BM + warp * 32 + rr;
          if (rw < e.M && c < e.N) {
            const long long o = (rw / e.out.rc) * e.out.s1 + (rw % e.out.rc) * e.out.s2 + c;
            float z = blk[rr * 33 + lane] * e.scale + bias_c;
            if (e.add) z += e.add[o];
            if (e.accumulate) z += e.y[o];
            e.y[o] = z;
            if (e.act) e.act[o] = gelu_t(z);
          }
        }
        __syncwarp();
      } else if (part) {
        float* pp = part + ((size_t)split * tiles + tile) * (size_t)(BM * BN) + (size_t)(warp * 32 + lane) * BN + c0;
#pragma unroll
        for (int i = 0; i < 32; ++i) pp[i] = __uint_as_float(v[i]);
      } else if (row_ok) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int c = nt * BN + c0 + i;
          if (c < e.N) {
            const long long o =
                rbase + (split_cols ? (long long)(c / e.out.kc) * e.out.t1 + (long long)(c % e.out.kc) * e.out.t2
                                    : (long long)c * e.out.t1);
            float z = __uint_as_float(v[i]) * e.scale;
            if (e.bias) z += __ldg(e.bias + c);
            if (e.add) z += e.add[o];
            if (e.accumulate) z += e.y[o];
            e.y[o] = z;
            if (e.act) e.act[o] = gelu_t(z);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

// Sums the split-K partials and applies the epilogue; one warp per (row, column): lane l
// adds splits l, l + 32, ... in order, then the lanes combine by a fixed butterfly, so
// the result does not depend on scheduling.
constexpr int REDUCE_WARPS = 8;  // outputs per block of the reduction
__global__ void splitk_reduce_kernel(const float* __restrict__ part, int splits, int tiles, int ntiles_n, int bn, Epi e) {
  const long long i = (long long)blockIdx.x * REDUCE_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= e.M * (long long)e.N) return;  // warp-uniform
  const long long r = i / e.N;
  const int c = (int)(i % e.N);
  const int mt = (int)(r / BM), nt = c / bn;
  const int tile = mt * ntiles_n + nt;
  const size_t off = (size_t)tile * (BM * bn) + (size_t)(r % BM) * bn + (c % bn);
  float z = 0.f;
  for (int s = lane; s < splits; s += 32) z += part[(size_t)s * tiles * (BM * bn) + off];
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) z += __shfl_xor_sync(0xffffffffu, z, m);
  if (lane != 0) return;
  z *= e.scale;
  const long long o = addr_of(e.out, r, c);
  if (e.bias) z += e.bias[c];
  if (e.add) z += e.add[o];
  if (e.accumulate) z += e.y[o];
  e.y[o] = z;
  if (e.act) e.act[o] = gelu_t(z);
}

// ------------------------------------------------------------ persistent, warp-specialised GEMM
// One CTA of 512 threads per SM loops over the items (batch, split, mt, nt) =
// blockIdx.x, blockIdx.x + gridDim.x, ... (nt fastest):
//   warps 0-3   operand loaders: round the FP32 values of a K block from a staging slot
//               to bfloat16 into the swizzled stage (no packing pass over A; in the FUSE
//               form B too) and, unless every copy is a bulk copy of whole runs, first
//               bring them into the slot (16-byte or 4-byte asynchronous copies, loads);
//   warps 4-11  epilogue, two groups of four taking alternate items; warp w reads
//               TMEM lanes 32 (w mod 4) .. + 31 (tile rows);
//   warp 12     holds two BN-column accumulators in TMEM; lane 0 issues the MMAs;
//   warp 13     the bulk copies of FP32 operands (`bulk` operands only);
//   warp 14     lane 0: the stage's packed B block with one bulk copy (not FUSE).
// The accumulators alternate between items, so an item's epilogue overlaps the next
// one's loads and MMAs.  Barriers: afull[slot] (staging slot filled: warp 13's one
// arrival with the bytes, else 128 loader arrivals), afree[slot] (a loader arrival:
// the slot is rounded, warp 13 may fill it again), full[s] (128 loader arrivals:
// bfloat16 written), bfull[s] (the B bytes, or in the FUSE form a loader arrival),
// empty[s] (MMA commit), accf[b] (MMA commit of accumulator b), acce[b] (one arrival
// per warp of the epilogue group).  Rows of A at or past M
// are not converted (an MMA row depends on its own A row only, and those rows are not
// stored); K steps of 16 past K are not issued, and the rest of the last K step is
// zero.  Every wait is bounded; the loaders take each decision together (a barrier
// reduction), on a timeout a role sets *err and stops, the MMA issuer waits (bounded)
// for its MMAs and the loaders for their copies before the tensor memory is freed.
namespace ws {
constexpr int LOADERS = 128;  // warps 0-3
constexpr int EPI_WARPS = 8;  // warps 4-11
constexpr int MMA_WARP = 12;
constexpr int COPY_WARP = 13;   // bulk copies of FP32 operands
constexpr int IMAGE_WARP = 14;  // bulk copies of the packed B
constexpr int THREADS = 16 * 32;  // warp 15 idle: registers move between groups of four warps
constexpr int SLOT_FLOATS = BM * BK;  // one FP32 staging slot (32 KB)
constexpr int EPI_LD = 36;                // row stride of a warp's 32 x 32 block: 16-byte aligned, conflict-free
constexpr int EPI_BLOCK = 32 * EPI_LD;
template <int BN>
struct Cfg {
  static constexpr int STAGES = BN == 256 ? 2 : 3;  // bfloat16 operand stages
  static constexpr int DEPTH = BN <= 64 ? 3 : 2;    // FP32 staging slots: A stages in flight
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int BROWS = BN;                          // rows of a B tile
  static constexpr int BSLOT_FLOATS = BN == 32 ? 32 * BK : 0;  // FP32 B staging slot (B from FP32: BN = 32)
  static constexpr int EPI_FLOATS = EPI_WARPS * EPI_BLOCK;
  static constexpr int SMEM =
      STAGES * STAGE_BYTES + DEPTH * (SLOT_FLOATS + BSLOT_FLOATS) * 4 + EPI_FLOATS * 4 + 1024;
  static constexpr uint32_t TMEM_COLS = 2 * BN;
};

__device__ __forceinline__ void cp4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// the barrier's phase completes (for this thread's arrival) once this thread's copies have landed
__device__ __forceinline__ void cp_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// barrier 1 over the 128 loader threads: true on all of them iff `ok` on all of them
__device__ __forceinline__ bool loaders_all(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 1, 128, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)ok)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void loaders_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// eight values as bfloat16 to a 16-byte chunk of an operand stage
__device__ __forceinline__ void put_chunk(uint8_t* dst, const float (&x)[8]) {
  __align__(16) __nv_bfloat162 h[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
  *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
}

// mbar_wait_bounded with the clock read only when the phase has not completed yet
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity) {
  return mbar_try_wait(bar, parity) || mbar_wait_bounded(bar, parity);
}

// A cursor over a CTA's items (batch, split, mt, nt), nt fastest: one step is `step`
// items, split once into its four digits, so that moving on takes carries and no division.
struct Walk {
  long long it;
  int bt, split, mt, nt;
  int d_bt, d_split, d_mt, d_nt;
  __device__ __forceinline__ void digits(long long v, int ntiles, int mtiles, int splits, int& bt_, int& split_, int& mt_,
                                         int& nt_) {
    long long q = v / ntiles;
    nt_ = (int)(v - q * ntiles);
    v = q / mtiles;
    mt_ = (int)(q - v * mtiles);
    q = v / splits;
    split_ = (int)(v - q * splits);
    bt_ = (int)q;
  }
  __device__ __forceinline__ void start(long long first, long long step, int ntiles, int mtiles, int splits) {
    it = first;
    digits(first, ntiles, mtiles, splits, bt, split, mt, nt);
    digits(step, ntiles, mtiles, splits, d_bt, d_split, d_mt, d_nt);
  }
  __device__ __forceinline__ void next(long long step, int ntiles, int mtiles, int splits) {
    it += step;
    nt += d_nt;
    const int c0 = nt >= ntiles;
    nt -= c0 ? ntiles : 0;
    mt += d_mt + c0;
    const int c1 = mt >= mtiles;
    mt -= c1 ? mtiles : 0;
    split += d_split + c1;
    const int c2 = split >= splits;
    split -= c2 ? splits : 0;
    bt += d_bt + c2;
  }
};

// How the rows r0 .. r0 + R - 1 of an operand (R = 128 for A, BN for B), K block kb
// (nk = min(64, K - 64 kb) values), reach a staging slot:
//   ROWRUN   k contiguous: row r0 + i to slot[i][0 .. nk) in 16-byte asynchronous copies
//            dealt over all threads where every row is aligned (one bulk copy a row took
//            twice as long to issue), else thread i copies its row, in bulk if it can;
//   GROUPRUN rows contiguous in groups of rc with k stride rc (a group's K block is one
//            run of nk * rc values; rc may be all the operand's rows): thread i < R / rc
//            copies group i to slot[i * 64 rc ..], element (k, r mod rc) at k rc + r mod rc;
//   PIECES   rows contiguous in groups of rc at any k strides, or (pair) with two
//            neighbouring k values to each row: 16-byte asynchronous copies dealt over all
//            threads, group i to slot[i * 64 rc ..], element (k, r mod rc) as in GROUPRUN
//            or (pair) at ((k / 2) rc + r mod rc) 2 + k mod 2;
//   GENERIC  value by value (4-byte asynchronous copies), a row's values dealt over the
//            threads that have no row of their own, element (r, k) at ((k / 8) R + i) 8 + k mod 8;
//   TILERUN  rows of K <= 64 values stored back to back: thread 0 copies the tile's rows
//            as one run (or the loaders load it, when the run is not 16-byte aligned),
//            element (r, k) at r K + k.
// Bulk bytes are announced on the slot's barrier without arriving; each loader thread
// arrives once per slot after its copies of A and B are issued (through the async-copy
// unit when it issued asynchronous copies, so the arrival waits for them).
//
// The loaders are one warp per scheduler, so a block costs them the length of their
// instruction chain and hardly anything else: offsets are hoisted, steps are additions
// and shifts, and four chunks are read before the first is stored.
enum { ANY = -1, ROWRUN = 0, GROUPRUN = 1, GENERIC = 2, TILERUN = 3, PIECES = 4 };
template <int V> using Tag = std::integral_constant<int, V>;

__device__ __forceinline__ void expect_tx_only(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

struct Op {
  const float* p;  // FP32 operand (batch 0)
  Addr a;
  long long bs;    // batch stride (floats)
  long long rows;  // M or N
  int mode, rc;    // rc: rows of a group (GROUPRUN, PIECES)
  int whole;       // TILERUN: every full tile is one 16-byte aligned run; ROWRUN: every row is aligned
  int pair;        // PIECES: two neighbouring k values to a row
  int bulk;        // every block arrives by bulk copies of one warp (issue_bulk)
};

__host__ __device__ inline void op_mode(Op& o, int tile_rows, long long k_total) {
  const Addr& a = o.a;
  o.rc = (int)a.rc;
  o.mode = GENERIC;
  o.whole = 0;
  o.pair = 0;
  o.bulk = 0;
  const bool aligned = o.bs % 4 == 0 && (reinterpret_cast<uintptr_t>(o.p) & 15u) == 0;
  if (a.kc == 1 && a.t1 == 1) {
    o.mode = ROWRUN;
    if (a.rc == 1 && k_total <= BK && a.s1 == k_total) o.mode = TILERUN;
    o.whole = aligned && (o.mode == TILERUN || ((a.rc == 1 || a.s2 % 4 == 0) && a.s1 % 4 == 0));
    o.bulk = o.mode == TILERUN && aligned && o.rows * k_total % 4 == 0;
    return;
  }
  long long g = -1;
  if (a.s2 == 1 && a.rc > 1) g = a.rc;
  else if (a.rc == 1 && a.s1 == 1) g = o.rows;  // all rows contiguous
  // one group may be of any size as long as its K blocks are whole 16-byte pieces
  const bool one = g == o.rows && (k_total % BK) * g % 4 == 0;
  if (g > 0 && g <= tile_rows && a.kc == 1 && a.t1 == g && (one || (g % 4 == 0 && tile_rows % g == 0)) &&
      o.rows % g == 0 && (g == o.rows || a.s1 % 4 == 0) && aligned) {
    o.mode = GROUPRUN;
    o.rc = (int)g;
    o.bulk = tile_rows / o.rc <= 32;
    return;
  }
  // groups of the tile that lie within the operand's
  const bool pair = a.kc == 2 && a.t2 == 1 && a.s2 == 2 && a.rc > 1;
  if (pair) g = a.rc;
  if (g > 0 && aligned && a.t1 % 4 == 0 && (pair ? k_total % 2 == 0 : a.kc == 1 || a.t2 % 4 == 0) &&
      (g == o.rows || a.s1 % 4 == 0)) {
    const long long in = (g & -g) < tile_rows ? g & -g : tile_rows;  // a power of two, as the tile
    if (in * (pair ? 2 : 1) % 4 == 0 && o.rows % in == 0) {
      o.mode = PIECES;
      o.rc = (int)in;
      o.pair = pair;
    }
  }
}

// One warp's bulk copies of a block of a `bulk` operand (TILERUN or GROUPRUN): its bytes,
// or with `go` the copies themselves (lane l the l-th group).
template <int R>
__device__ __forceinline__ uint32_t bulk_block(float* stg, uint64_t* bar, const Op& o, int bt, long long K, long long r0,
                                               int kb, int lane, bool go) {
  const long long kb0 = (long long)kb * BK, left = o.rows - r0;
  const int nk = (int)(K - kb0 < BK ? K - kb0 : BK), nrow = (int)(left < R ? left : R);
  if (nrow <= 0) return 0;
  const uint32_t bytes = (uint32_t)(nrow * nk) * 4u;
  if (!go) return bytes;
  const float* const P = o.p + bt * o.bs;
  if (o.mode == TILERUN) {
    if (lane == 0) bulk_g2s(stg, P + r0 * o.a.s1, bytes, bar);
  } else if (lane * o.rc < nrow) {
    const long long r = r0 + lane * o.rc;
    const long long off = o.a.rc == 1 ? r * o.a.s1 : (r / o.a.rc) * o.a.s1 + (r % o.a.rc) * o.a.s2;
    bulk_g2s(stg + lane * BK * o.rc, P + off + kb0 * o.a.t1, (uint32_t)nk * (uint32_t)o.rc * 4u, bar);
  }
  return bytes;
}

// The loader threads' copies of rows r0 .. r0 + R - 1 of operand o (batch bt) into slot
// stg; true when this thread issued asynchronous (non-bulk) copies.
template <int R, int MODE>
__device__ __forceinline__ bool issue_op(float* stg, uint64_t* bar, const Op& o, int bt, long long K, long long r0,
                                         int kb, int i) {
  const long long kb0 = (long long)kb * BK;
  const int nk = (int)(K - kb0 < BK ? K - kb0 : BK);
  const Addr& a = o.a;
  const int mode = MODE == ANY ? o.mode : MODE;
  if (mode == TILERUN && i != 0 && o.whole && r0 + R <= o.rows) return false;  // thread 0's one copy
  const float* const P = o.p + bt * o.bs;
  // offset of row r; operands with one row stride need no division
  auto row_off = [&](long long r) { return a.rc == 1 ? r * a.s1 : (r / a.rc) * a.s1 + (r % a.rc) * a.s2; };
  if (mode == TILERUN) {
    const long long nrow = o.rows - r0 < R ? o.rows - r0 : R;
    const float* src = P + r0 * a.s1;
    const int n = (int)(nrow * nk);
    if (nrow > 0 && (n & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
      if (i == 0) {
        expect_tx_only(bar, (uint32_t)n * 4u);
        bulk_g2s(stg, src, (uint32_t)n * 4u, bar);
      }
    } else {
      for (int j = i; j < n; j += LOADERS) stg[j] = __ldg(src + j);
    }
    return false;
  }
  if (mode == ROWRUN && o.whole && (nk & 3) == 0) {
    const int nrow = (int)(o.rows - r0 < R ? o.rows - r0 : R), pr = nk >> 2;
    for (int j = i; j < nrow * pr; j += LOADERS) {
      const int row = nk == BK ? j / (BK / 4) : j / pr, q = j - row * pr;
      cp16(stg + row * BK + q * 4, P + row_off(r0 + row) + kb0 + q * 4);
    }
    return true;
  }
  if (mode == ROWRUN) {
    const long long r = r0 + i;
    if (i < R && r < o.rows) {
      const float* src = P + row_off(r) + kb0;
      if ((nk & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
        expect_tx_only(bar, (uint32_t)nk * 4u);
        bulk_g2s(stg + i * BK, src, (uint32_t)nk * 4u, bar);
      } else {
        for (int k = 0; k < nk; ++k) stg[i * BK + k] = __ldg(src + k);
      }
    }
    return false;
  }
  if (mode == GROUPRUN) {
    const int rc = o.rc;
    const long long r = r0 + (long long)i * rc;
    if (i * rc < R && r < o.rows) {
      const uint32_t bytes = (uint32_t)nk * (uint32_t)rc * 4u;
      expect_tx_only(bar, bytes);
      bulk_g2s(stg + i * BK * rc, P + row_off(r) + kb0 * a.t1, bytes, bar);
    }
    return false;
  }
  if (mode == PIECES) {
    const int rc = o.rc, ks = o.pair ? 1 : 0, run = (rc << ks) >> 2;  // 16-byte pieces of a run, a power of two
    const int pieces = (nk >> ks) * run;                              // of a group
    const int sr = 31 - __clz(run);
    const long long step = (long long)(LOADERS >> sr) * a.t1;
    for (int g = 0; g * rc < R && r0 + g * rc < o.rows; ++g) {
      const float* src = P + row_off(r0 + g * rc) + (i & (run - 1)) * 4;
      float* dst = stg + g * rc * BK + i * 4;
      if (o.pair || a.kc == 1) {
        src += ((kb0 >> ks) + (i >> sr)) * a.t1;
        for (int j = i; j < pieces; j += LOADERS, src += step, dst += LOADERS * 4) cp16(dst, src);
      } else {
        for (int j = i; j < pieces; j += LOADERS, dst += LOADERS * 4) {
          const long long k = kb0 + (j >> sr), q = k / a.kc;
          cp16(dst, src + q * a.t1 + (k - q * a.kc) * a.t2);
        }
      }
    }
    return true;
  }
  // GENERIC: `parts` threads per row, part h the values [h * len, (h + 1) * len)
  const long long left = o.rows - r0;
  const int own = left <= 32 ? 32 : left <= 64 ? 64 : LOADERS;  // rows with threads of their own
  const int row_i = i & (own - 1), parts = LOADERS / own, len = (nk + parts - 1) / parts;
  const int k0 = (i / own) * len, k1 = k0 + len < nk ? k0 + len : nk;
  if (row_i >= R || row_i >= left || k0 >= k1) return false;
  const float* base = P + row_off(r0 + row_i);
  int rem = 0;
  if (a.kc == 1) {
    base += (kb0 + k0) * a.t1;
  } else {
    const long long q = (kb0 + k0) / a.kc;
    rem = (int)(kb0 + k0 - q * a.kc);
    base += q * a.t1;
  }
  const float* src = base + rem * a.t2;
  const int kc = (int)(a.kc < BK + 1 ? a.kc : kb0 + BK + 1 < a.kc ? kb0 + BK + 1 : a.kc);
  float* dst = stg + row_i * 8;
#pragma unroll 4
  for (int k = k0; k < k1; ++k) {
    cp4(dst + (k >> 3) * (R * 8) + (k & 7), src);
    src += a.t2;
    if (++rem == kc) {
      rem = 0;
      base += a.t1;
      src = base;
    }
  }
  return true;
}

// Round a landed slot to bfloat16 in the operand stage: 8-value chunk ch of row i
// goes to the 128-byte swizzled tile (sa).  Only the operand's own rows are rounded
// (a row past M or N feeds only output that is not stored).
//
// Convert holds what does not change from one full block to the next: the thread's
// place, the rounds and the steps between them.  Blocks at the ragged end of the rows
// or of K, and forms whose chunks do not deal out evenly, take convert_any.
template <int R, int MODE>
__device__ __forceinline__ void convert_any(uint8_t* sa, const float* stg, const Op& o, long long K, long long r0, int kb,
                                         int i) {
  const long long kb0 = (long long)kb * BK;
  const int nk = (int)(K - kb0 < BK ? K - kb0 : BK);
  const int nch = nk >= BK ? 8 : 2 * ((nk + 15) / 16);  // chunks the MMAs read
  const int nrow = (int)(o.rows - r0 < R ? o.rows - r0 : R);  // rows to convert
  const int mode = MODE == ANY ? o.mode : MODE, rc = o.rc;
  const bool runs = mode == ROWRUN || mode == TILERUN, pair = mode == PIECES && o.pair;
  for (int t = i; t < nrow * nch; t += LOADERS) {  // chunk fastest where k is contiguous, else row
    const int row = runs ? t / nch : t % nrow, ch = runs ? t % nch : t / nrow;
    const float* src = runs              ? stg + row * (mode == ROWRUN ? BK : nk) + ch * 8
                       : mode == GENERIC ? stg + (ch * R + row) * 8
                                         : stg + (row / rc) * (BK * rc) + ch * 8 * rc + (pair ? 2 : 1) * (row % rc);
    const int step = runs || mode == GENERIC ? 1 : rc;
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
      x[e] = ch * 8 + e < nk ? (pair ? src[(e >> 1) * 2 * rc + (e & 1)] : src[e * step]) : 0.f;
    put_chunk(sa + sw128(row, ch * 8), x);
  }
}

template <int R, int MODE>
struct Convert {
  int rounds;            // of LOADERS chunks in a full block; 0: convert_any always
  int m_full, kb_full;   // full row tiles and K blocks
  int src, src_step, nk, ch, ch_step, sg;
  uint32_t dst, dst_step;
  static constexpr bool RUNS = MODE == ROWRUN || MODE == TILERUN;

  __device__ __forceinline__ void init(const Op& o, long long K, int i) {
    const int nrow = (int)(o.rows < R ? o.rows : R);
    nk = (int)(K < BK ? K : BK);
    const int nch = nk >= BK ? 8 : 2 * ((nk + 15) / 16), total = nrow * nch;
    m_full = o.rows < R ? 1 : (int)(o.rows / R);
    kb_full = K < BK ? 1 : (int)(K / BK);
    rounds = 0;
    if (MODE == ANY || total % LOADERS != 0) return;
    if (RUNS) {  // chunk fastest; a round moves on by LOADERS / nch rows, a multiple of 8
      if (nch == 6) return;
      const int row = i / nch, ld = MODE == ROWRUN ? BK : nk;
      ch = i % nch;
      src = row * ld + ch * 8;
      src_step = LOADERS / nch * ld;
      dst = sw128(row, ch * 8);
      dst_step = (uint32_t)(LOADERS / nch) * 128u;
    } else {  // row fastest; a thread keeps its row and moves on by LOADERS / nrow chunks
      if (nk != nch * 8 || (nrow & (nrow - 1)) != 0) return;
      const int row = i % nrow, rc = o.rc;
      ch = i / nrow;
      ch_step = LOADERS / nrow;
      dst = (uint32_t)row * 128u;
      dst_step = (uint32_t)(row & 7);
      if (MODE == GENERIC) {
        src = (ch * R + row) * 8;
        src_step = ch_step * R * 8;
      } else {
        if ((rc & (rc - 1)) != 0) return;
        sg = 31 - __clz(rc);
        const bool pair = MODE == PIECES && o.pair;
        src = (row >> sg) * (BK << sg) + ((ch * 8) << sg) + (pair ? 2 : 1) * (row & (rc - 1));
        src_step = (ch_step * 8) << sg;
        if (pair) sg = -sg;  // sign: pairs of neighbouring k
      }
    }
    rounds = total / LOADERS;
  }

  __device__ __forceinline__ void get(const float* p, int c, float (&x)[8]) const {
    if (RUNS || MODE == GENERIC) {
      if (!RUNS || (nk & 15) == 0) {
        const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
        x[0] = lo.x; x[1] = lo.y; x[2] = lo.z; x[3] = lo.w;
        x[4] = hi.x; x[5] = hi.y; x[6] = hi.z; x[7] = hi.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = c * 8 + e < nk ? p[e] : 0.f;
      }
    } else if (MODE == PIECES && sg <= 0) {  // groups of pairs: rc = 2^-sg rows
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float2 v = *reinterpret_cast<const float2*>(p + (e << -sg));
        x[e] = v.x;
        x[e + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = p[e << sg];
    }
  }
  __device__ __forceinline__ uint8_t* at(uint8_t* sa, int u) const {
    return RUNS ? sa + dst + u * dst_step : sa + dst + ((uint32_t)((ch + u * ch_step) ^ (int)dst_step) << 4);
  }

  __device__ __forceinline__ void run(uint8_t* sa, const float* stg, const Op& o, long long K, int mt, int kb, int i) {
    if (rounds == 0 || mt >= m_full || kb >= kb_full) {
      convert_any<R, MODE>(sa, stg, o, K, (long long)mt * R, kb, i);
      return;
    }
    const float* p = stg + src;
    constexpr int U = 2;  // chunks read before the first is stored
    int u = 0;
#pragma unroll 1
    for (; u + U <= rounds; u += U, p += U * src_step) {
      float x[U][8];
#pragma unroll
      for (int v = 0; v < U; ++v) get(p + v * src_step, ch, x[v]);
#pragma unroll
      for (int v = 0; v < U; ++v) put_chunk(at(sa, u + v), x[v]);
    }
    if (u < rounds) {
      float x[8];
      get(p, ch, x);
      put_chunk(at(sa, u), x);
    }
  }
};
}  // namespace ws

// 16 consecutive accumulator columns of this warp's 32 TMEM lanes (one per lane).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The work of one launch.  Items (batch, split, mt, nt), nt fastest; item `split` sums K
// blocks [split * kper, min(kblocks, (split + 1) * kper)).  B comes either packed
// (b_img, one image per batch) or, for BN = 32, as an FP32 operand (b.p) staged and
// rounded like A.  With part set the epilogue writes raw partial tiles
// part[((batch * splits + split) * tiles + tile) * 128 * BN + row * BN + col] instead.
// Forms of the epilogue's output: raw partial tiles; columns contiguous in whole 16-byte
// pieces; columns along the lanes (contiguous, or nearer than rows); any other layout, rows
// along the lanes; rows contiguous in whole 16-byte pieces; pairs of columns within
// contiguous rows (complex values).
enum { OUT_PART, OUT_VEC, OUT_COLS, OUT_ROWS, OUT_RVEC, OUT_PAIR };

struct WsArgs {
  ws::Op a, b;
  const uint8_t* b_img;
  long long K;
  int kblocks, kper, splits, ntiles;
  long long mtiles, items;
  float* part;
  int form;  // of the output (and of add, act)
};

template <int BN, bool FUSE>
__global__ void __launch_bounds__(ws::THREADS, 1) gemm_ws_kernel(WsArgs w, Epi e, int* __restrict__ err) {
  using C = ws::Cfg<BN>;
  constexpr int ST = C::STAGES, D = C::DEPTH;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  float* const stg0 = reinterpret_cast<float*>(smem + ST * C::STAGE_BYTES);
  float* const stgb = stg0 + D * ws::SLOT_FLOATS;  // B staging (BN = 32 only)
  float* const epi_buf = stgb + D * C::BSLOT_FLOATS;
  __shared__ uint64_t full[ST], bfull[ST], empty[ST], afull[D], afree[D], accf[2], acce[2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ long long off_s[2][ws::EPI_WARPS][32];  // epilogue: per warp, 32 row (or column) offsets
  __shared__ float bias_s[2][ws::EPI_WARPS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == ws::MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const bool bulk = w.a.bulk && (!FUSE || w.b.bulk);  // every copy a bulk copy: COPY_WARP issues them all
  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full[s], ws::LOADERS);
      mbar_init(&bfull[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int d = 0; d < D; ++d) {
      mbar_init(&afull[d], bulk ? 1 : ws::LOADERS);
      mbar_init(&afree[d], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 4);
    }
    mbar_init(&drain, 1);
    fence_mbar_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  const long long tiles = w.mtiles * w.ntiles;
  const int mtiles = (int)w.mtiles;
  auto k_end = [&](int split) { return min((split + 1) * w.kper, w.kblocks); };

  // blocks of this CTA in order: a cursor over (item, K block)
  struct Cur {
    ws::Walk w;
    int kb, kb1;
  };
  auto open = [&](Cur& c) {
    c.kb = c.w.split * w.kper;
    c.kb1 = k_end(c.w.split);
  };
  auto advance = [&](Cur& c) {
    if (++c.kb >= c.kb1) {
      c.w.next(gridDim.x, w.ntiles, mtiles, w.splits);
      open(c);
    }
  };
  if (warp < 4) {  // operand loaders
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;");
    const int i = threadIdx.x;
    // One loop per operand form: what runs is one form's instructions, without the others between
    auto load = [&](auto form_a, auto form_b) {
      constexpr int MA = decltype(form_a)::value;
      [[maybe_unused]] constexpr int MB = decltype(form_b)::value;
      ws::Convert<BM, MA> conv_a;
      conv_a.init(w.a, w.K, i);
      ws::Convert<C::BROWS, FUSE ? MB : ws::ANY> conv_b;
      if constexpr (FUSE) conv_b.init(w.b, w.K, i);
      Cur cur, ahead;
      cur.w.start(blockIdx.x, gridDim.x, w.ntiles, mtiles, w.splits);
      open(cur);
      ahead = cur;
      int flight = 0, di = 0;  // slots issued and not yet converted: d, d + 1, ... up to di (mod D)
      // stage s and slot d of the current block, with the phases their barriers complete next
      int s = 0, d = 0, used = 0;  // used: stages handed to the MMAs, at most ST
      uint32_t sp = 0, dp = 0;
      while (true) {
        for (; !bulk && flight < D && ahead.w.it < w.items; ++flight, advance(ahead)) {
          bool cp = ws::issue_op<BM, MA>(stg0 + di * ws::SLOT_FLOATS, &afull[di], w.a, ahead.w.bt, w.K,
                                         (long long)ahead.w.mt * BM, ahead.kb, i);
          if constexpr (FUSE)
            cp |= ws::issue_op<C::BROWS, MB>(stgb + di * C::BSLOT_FLOATS, &afull[di], w.b, ahead.w.bt, w.K,
                                             (long long)ahead.w.nt * BN, ahead.kb, i ^ 64);  // another warp's bulk copy
          if (cp) ws::cp_arrive(&afull[di]);
          else mbar_arrive(&afull[di]);
          if (++di == D) di = 0;
        }
        if (cur.w.it >= w.items) break;
        bool ok = ws::wait_bar(&afull[d], dp);
        if (ok && used == ST) ok = ws::wait_bar(&empty[s], sp ^ 1u);
        if (ok) {
          uint8_t* st = smem + s * C::STAGE_BYTES;
          if constexpr (FUSE) {
            conv_b.run(st + A_BYTES, stgb + d * C::BSLOT_FLOATS, w.b, w.K, cur.w.nt, cur.kb, i);
          }
          conv_a.run(st, stg0 + d * ws::SLOT_FLOATS, w.a, w.K, cur.w.mt, cur.kb, i);
          fence_proxy_async();  // the tensor cores read the stage through the async proxy
          mbar_arrive(&full[s]);
          if (FUSE && i == 0) mbar_arrive(&bfull[s]);
          if (used < ST) ++used;
          if (++s == ST) { s = 0; sp ^= 1u; }
        }
        // every loader is done with slot d; a wait that ran out on one ends them all
        if (!ws::loaders_all(ok)) {
          if (i == 0) atomicOr(err, 2);
          break;
        }
        if (bulk) {
          if (i == 0) mbar_arrive(&afree[d]);
        } else {
          --flight;
        }
        if (++d == D) { d = 0; dp ^= 1u; }
        advance(cur);
      }
      // copies in flight land before the CTA's shared memory is released
      for (; flight > 0; --flight) {
        mbar_wait_bounded(&afull[d], dp);
        if (++d == D) { d = 0; dp ^= 1u; }
      }
    };
    if constexpr (FUSE) {
      if (w.a.mode == ws::GROUPRUN && w.b.mode == ws::GROUPRUN)
        load(ws::Tag<ws::GROUPRUN>{}, ws::Tag<ws::GROUPRUN>{});
      else
        load(ws::Tag<ws::ANY>{}, ws::Tag<ws::ANY>{});
    } else {
      switch (w.a.mode) {
        case ws::ROWRUN: load(ws::Tag<ws::ROWRUN>{}, ws::Tag<0>{}); break;
        case ws::GROUPRUN: load(ws::Tag<ws::GROUPRUN>{}, ws::Tag<0>{}); break;
        case ws::TILERUN: load(ws::Tag<ws::TILERUN>{}, ws::Tag<0>{}); break;
        case ws::PIECES: load(ws::Tag<ws::PIECES>{}, ws::Tag<0>{}); break;
        default: load(ws::Tag<ws::GENERIC>{}, ws::Tag<0>{}); break;
      }
    }
  } else if (warp >= ws::MMA_WARP) {  // MMA issuer
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == ws::MMA_WARP && lane == 0) {
      long long n = 0;
      int s = 0;
      uint32_t par = 0;
      bool ok = true;
      ws::Walk t;
      t.start(blockIdx.x, gridDim.x, w.ntiles, mtiles, w.splits);
      for (; t.it < w.items && ok; t.next(gridDim.x, w.ntiles, mtiles, w.splits), ++n) {
        const int kb0 = t.split * w.kper, kb1 = k_end(t.split);
        const int buf = (int)(n & 1);
        if (n >= 2 && !ws::wait_bar(&acce[buf], (uint32_t)(((n >> 1) - 1) & 1))) {
          atomicOr(err, 16);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t dacc = tmem + (uint32_t)(buf * BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!ws::wait_bar(&full[s], par) || !ws::wait_bar(&bfull[s], par)) {
            atomicOr(err, 4);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = smem_u32(smem + s * C::STAGE_BYTES);
          const long long krem = w.K - (long long)kb * BK;
          const int nk = krem >= BK ? BK / 16 : (int)((krem + 15) / 16);
          for (int j = 0; j < nk; ++j) {
            const uint32_t off = (uint32_t)j * 32u;
            const uint32_t acc = (kb > kb0 || j > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t .reg .pred p;\n\t setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dacc),
                "l"(sdesc(sa + off)), "l"(sdesc(sa + A_BYTES + off)), "r"(tg::Cfg<BN>::IDESC), "r"(acc)
                : "memory");
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                           smem_u32(&empty[s]))
                       : "memory");
          if (++s == ST) { s = 0; par ^= 1u; }
        }
        if (!ok) break;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&accf[buf]))
                     : "memory");
      }
      // every MMA issued has completed before the tensor memory and the stages are released
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&drain))
                   : "memory");
      if (!mbar_wait_bounded(&drain, 0)) atomicOr(err, 32);
    } else if (warp == ws::COPY_WARP && bulk) {
      // FP32 operands, up to D blocks ahead of the loaders
      Cur c;
      c.w.start(blockIdx.x, gridDim.x, w.ntiles, mtiles, w.splits);
      open(c);
      int d = 0, sent = 0;  // sent: blocks in flight or landed, at most D
      uint32_t dp = 0;
      for (; c.w.it < w.items; advance(c)) {
        if (sent == D && !ws::wait_bar(&afree[d], dp ^ 1u)) {
          if (lane == 0) atomicOr(err, 128);
          break;
        }
        __syncwarp();
        float* const sa = stg0 + d * ws::SLOT_FLOATS;
        float* const sb = stgb + d * C::BSLOT_FLOATS;
        if (lane == 0) {
          uint32_t bytes = ws::bulk_block<BM>(sa, &afull[d], w.a, c.w.bt, w.K, (long long)c.w.mt * BM, c.kb, 0, false);
          if constexpr (FUSE)
            bytes += ws::bulk_block<C::BROWS>(sb, &afull[d], w.b, c.w.bt, w.K, (long long)c.w.nt * BN, c.kb, 0, false);
          mbar_expect_tx(&afull[d], bytes);
        }
        __syncwarp();
        ws::bulk_block<BM>(sa, &afull[d], w.a, c.w.bt, w.K, (long long)c.w.mt * BM, c.kb, lane, true);
        if constexpr (FUSE)
          ws::bulk_block<C::BROWS>(sb, &afull[d], w.b, c.w.bt, w.K, (long long)c.w.nt * BN, c.kb, lane, true);
        if (sent < D) ++sent;
        if (++d == D) { d = 0; dp ^= 1u; }
      }
      // copies in flight land before the CTA's shared memory is released
      if (sent == D) dp ^= 1u;  // the last `sent` blocks: d is the oldest of them
      else d = 0;
      for (int j = 0; j < sent; ++j) {
        mbar_wait_bounded(&afull[d], dp);
        if (++d == D) { d = 0; dp ^= 1u; }
      }
    } else if (!FUSE && warp == ws::IMAGE_WARP && lane == 0) {
      // packed B, into each stage as the MMAs leave it
      Cur c;
      c.w.start(blockIdx.x, gridDim.x, w.ntiles, mtiles, w.splits);
      open(c);
      int s = 0, sent = 0;
      uint32_t sp = 0;
      for (; c.w.it < w.items; advance(c)) {
        if (sent == ST && !ws::wait_bar(&empty[s], sp ^ 1u)) {
          atomicOr(err, 256);
          break;
        }
        mbar_expect_tx(&bfull[s], C::B_BYTES);
        bulk_g2s(smem + s * C::STAGE_BYTES + A_BYTES,
                 w.b_img + (((size_t)c.w.bt * w.ntiles + c.w.nt) * w.kblocks + c.kb) * C::B_BYTES, C::B_BYTES, &bfull[s]);
        if (sent < ST) ++sent;
        if (++s == ST) { s = 0; sp ^= 1u; }
      }
      if (sent == ST) sp ^= 1u;
      else s = 0;
      for (int j = 0; j < sent; ++j) {
        mbar_wait_bounded(&bfull[s], sp);
        if (++s == ST) { s = 0; sp ^= 1u; }
      }
    }
    __syncwarp();
  } else {  // epilogue, warps 4-11: group eg takes this CTA's tiles n = eg, eg + 2, ... (accumulator eg)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int wi = warp - 4, eg = wi >> 2, q = warp & 3;
    float* const blk = epi_buf + wi * ws::EPI_BLOCK;
    const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(eg * BN);
    // the warp's 32 x 32 accumulator block at column c0, to shared memory by rows
    auto block_to_smem = [&](int c0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[16];
        tmem_ld16(acc + (uint32_t)(c0 + h * 16), v);
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4*>(blk + lane * ws::EPI_LD + h * 16 + j) =
              make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]),
                          __uint_as_float(v[j + 3]));
      }
    };
    // One loop per output form.  In each the loads of add / accumulate are unconditional
    // (an invalid element reads word 0 of its array) and a whole block of them is in
    // flight before the accumulator is waited for, for they do not depend on it.
    auto finish = [&](auto form) {
      constexpr int F = decltype(form)::value;
      ws::Walk t;
      t.start(blockIdx.x + (long long)eg * gridDim.x, 2LL * gridDim.x, w.ntiles, mtiles, w.splits);
      for (uint32_t phase = 0; t.it < w.items; t.next(2LL * gridDim.x, w.ntiles, mtiles, w.splits), phase ^= 1u) {
        const int nt = t.nt;
        const long long bt = t.bt, r = (long long)t.mt * BM + q * 32 + lane;
        const bool row_ok = r < e.M;
        auto landed = [&] {
          const bool ok = ws::wait_bar(&accf[eg], phase);
          if (!ok && lane == 0) atomicOr(err, 8);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          return __all_sync(0xffffffffu, ok) != 0;
        };
        bool ok = true;
        if constexpr (F == OUT_PART) {  // raw partial tile: each lane stores its row's BN values
          ok = landed();
          float* pp = w.part + ((bt * w.splits + t.split) * tiles + (long long)t.mt * w.ntiles + nt) * (long long)(BM * BN) +
                      (long long)(q * 32 + lane) * BN;
          for (int c0 = 0; ok && c0 < BN; c0 += 16) {
            uint32_t v[16];
            tmem_ld16(acc + (uint32_t)c0, v);
            if (row_ok) {
#pragma unroll
              for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<float4*>(pp + c0 + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                      __uint_as_float(v[j + 2]),
                                                                      __uint_as_float(v[j + 3]));
            }
          }
        } else {
          float* const ey = e.y + bt * e.ybs;
          const float* const eadd = e.add ? e.add + bt * e.ybs : nullptr;
          float* const eact = e.act ? e.act + bt * e.ybs : nullptr;
          const float* const p1 = eadd ? eadd : ey;  // first addend (add, else the accumulated output)
          const bool have_prev = eadd || e.accumulate, both = eadd && e.accumulate;
          const long long rbase = !row_ok ? -1
                                  : e.out.rc == 1 ? r * e.out.s1
                                                  : (r / e.out.rc) * e.out.s1 + (r % e.out.rc) * e.out.s2;
          if constexpr (F == OUT_VEC || F == OUT_COLS) off_s[0][wi][lane] = rbase;
          __syncwarp();
          for (int c0 = 0; (F == OUT_VEC || F == OUT_COLS) && ok && c0 < BN && nt * BN + c0 < e.N; c0 += 32) {
            const int c = nt * BN + c0 + lane;  // this lane's column
            const bool col_ok = c < e.N;
            if constexpr (F == OUT_VEC) {
              // columns contiguous in the output and in whole 16-byte pieces: the warp's
              // 32 x 32 block goes through shared memory, then a lane takes four columns
              // of a row and neighbouring lanes the rest of the row, so an access covers
              // four whole lines.
              const int cols = e.N - nt * BN - c0;  // 1 << lp lanes cover a row's columns in this block
              const int lp = cols > 16 ? 3 : cols > 8 ? 2 : cols > 4 ? 1 : 0;
              const int q4 = (lane & ((1 << lp) - 1)) * 4, c4 = nt * BN + c0 + q4, row0 = lane >> lp, step = 32 >> lp;
              const bool c_ok = c4 < e.N;
              auto offset = [&](int u) -> long long {  // 1 << lp rounds of `step` rows
                const int row = u * step + row0;
                const long long rb = off_s[0][wi][row & 31];
                return row < 32 && rb >= 0 && c_ok ? rb + c4 : -1;
              };
              float4 prev[4], next[4];
              auto fetch = [&](float4 (&f)[4], int h) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const long long o = offset(h + u);
                  f[u] = *reinterpret_cast<const float4*>(p1 + (o >= 0 ? o : 0));
                }
                if (both) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    const long long o = offset(h + u);
                    const float4 y4 = *reinterpret_cast<const float4*>(ey + (o >= 0 ? o : 0));
                    f[u] = make_float4(f[u].x + y4.x, f[u].y + y4.y, f[u].z + y4.z, f[u].w + y4.w);
                  }
                }
              };
              if (have_prev) {
                fetch(prev, 0);
                if (lp == 3) fetch(next, 4);
              }
              float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
              if (e.bias && c_ok)
                b4 = make_float4(__ldg(e.bias + c4), __ldg(e.bias + c4 + 1), __ldg(e.bias + c4 + 2), __ldg(e.bias + c4 + 3));
              if (c0 == 0) ok = landed();
              if (!ok) break;
              block_to_smem(c0);
              __syncwarp();
#pragma unroll 1
              for (int h = 0; h < (1 << lp); h += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  const long long o = offset(h + u);
                  if (o < 0) continue;
                  const float4 a4 = *reinterpret_cast<const float4*>(blk + ((h + u) * step + row0) * ws::EPI_LD + q4);
                  float4 z = make_float4(fmaf(a4.x, e.scale, b4.x), fmaf(a4.y, e.scale, b4.y),
                                         fmaf(a4.z, e.scale, b4.z), fmaf(a4.w, e.scale, b4.w));
                  if (have_prev) z = make_float4(z.x + prev[u].x, z.y + prev[u].y, z.z + prev[u].z, z.w + prev[u].w);
                  *reinterpret_cast<float4*>(ey + o) = z;
                  if (eact)
                    *reinterpret_cast<float4*>(eact + o) =
                        make_float4(gelu_t(z.x), gelu_t(z.y), gelu_t(z.z), gelu_t(z.w));
                }
                if (have_prev) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) prev[u] = next[u];
                }
              }
              __syncwarp();
            } else if constexpr (F == OUT_COLS) {
              // the block goes through shared memory and each row is stored with the lanes
              // along its columns
              const long long cc = e.out.kc == 1 ? (long long)c * e.out.t1
                                                 : (long long)(c / e.out.kc) * e.out.t1 + (long long)(c % e.out.kc) * e.out.t2;
              if (c0 == 0) ok = landed();
              if (!ok) break;
              block_to_smem(c0);
              __syncwarp();
              const float bias_c = (e.bias && col_ok) ? __ldg(e.bias + c) : 0.f;
#pragma unroll 1
              for (int h = 0; h < 32; h += 16) {
                float prev[16];
                if (have_prev) {
#pragma unroll
                  for (int j = 0; j < 16; ++j) {
                    const long long ro = off_s[0][wi][h + j];
                    prev[j] = p1[(ro >= 0 && col_ok) ? ro + cc : 0];
                  }
                  if (both) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                      const long long ro = off_s[0][wi][h + j];
                      prev[j] += ey[(ro >= 0 && col_ok) ? ro + cc : 0];
                    }
                  }
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const long long ro = off_s[0][wi][h + j];
                  if (ro >= 0 && col_ok) {
                    float z = fmaf(blk[(h + j) * ws::EPI_LD + lane], e.scale, bias_c);
                    if (have_prev) z += prev[j];
                    ey[ro + cc] = z;
                    if (eact) eact[ro + cc] = gelu_t(z);
                  }
                }
              }
              __syncwarp();
            }
          }
          if constexpr (F == OUT_ROWS || F == OUT_RVEC || F == OUT_PAIR) {
            // Lanes along rows; the columns' offsets (this lane's for column c0 + lane) and
            // biases in shared memory, two blocks deep: block c0 + 32's added values are
            // requested before block c0 is finished.
            auto columns = [&](int c0) {
              const int c = nt * BN + c0 + lane, par = (c0 >> 5) & 1;
              const bool col_ok = c0 < BN && c < e.N;
              off_s[par][wi][lane] = !col_ok ? -1
                                     : e.out.kc == 1
                                         ? (long long)c * e.out.t1
                                         : (long long)(c / e.out.kc) * e.out.t1 + (long long)(c % e.out.kc) * e.out.t2;
              bias_s[par][wi][lane] = (e.bias && col_ok) ? __ldg(e.bias + c) : 0.f;
              __syncwarp();
            };
            auto fetch = [&](float (&f)[32], int c0) {
              const long long* const co = off_s[(c0 >> 5) & 1][wi];
#pragma unroll
              for (int j = 0; j < 32; ++j) f[j] = p1[(row_ok && co[j] >= 0) ? rbase + co[j] : 0];
              if (both) {
#pragma unroll
                for (int j = 0; j < 32; ++j) f[j] += ey[(row_ok && co[j] >= 0) ? rbase + co[j] : 0];
              }
            };
            if constexpr (F == OUT_RVEC || F == OUT_PAIR) {
              // Four rows of a column (two rows of a pair of columns) are 16 bytes: the block
              // goes through shared memory transposed, lane l takes rows 4 (l % 8) of columns
              // 4 u + l / 8 (rows 2 (l % 16) of the pairs of columns 2 u + l / 16).
              constexpr bool PAIR = F == OUT_PAIR;
              const int rl = PAIR ? (lane & 15) * 2 : (lane & 7) * 4, cl = PAIR ? (lane >> 4) * 2 : lane >> 3;
              const long long rb = __shfl_sync(0xffffffffu, rbase, rl);
              auto fetch4 = [&](float4 (&f)[8], int c0) {
                const long long* const co = off_s[(c0 >> 5) & 1][wi];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                  const long long c = co[u * 4 + cl];
                  f[u] = *reinterpret_cast<const float4*>(p1 + (rb >= 0 && c >= 0 ? rb + c : 0));
                }
                if (both) {
#pragma unroll
                  for (int u = 0; u < 8; ++u) {
                    const long long c = co[u * 4 + cl];
                    const float4 y4 = *reinterpret_cast<const float4*>(ey + (rb >= 0 && c >= 0 ? rb + c : 0));
                    f[u] = make_float4(f[u].x + y4.x, f[u].y + y4.y, f[u].z + y4.z, f[u].w + y4.w);
                  }
                }
              };
              float4 prev[8], next[8];
              columns(0);
              if (have_prev) fetch4(prev, 0);
              ok = landed();
#pragma unroll 1
              for (int c0 = 0; ok && c0 < BN && nt * BN + c0 < e.N; c0 += 32) {
                columns(c0 + 32);
                if (have_prev && c0 + 32 < BN && nt * BN + c0 + 32 < e.N) fetch4(next, c0 + 32);
                const long long* const co = off_s[(c0 >> 5) & 1][wi];
                const float* const bi = bias_s[(c0 >> 5) & 1][wi];
#pragma unroll
                for (int h = 0; h < 32; h += 16) {
                  uint32_t v[16];
                  tmem_ld16(acc + (uint32_t)(c0 + h), v);
#pragma unroll
                  for (int j = 0; j < 16; ++j) blk[(h + j) * ws::EPI_LD + lane] = __uint_as_float(v[j]);
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                  const long long c = co[u * 4 + cl];
                  if (rb < 0 || c < 0) continue;
                  const float* const q = blk + (u * 4 + cl) * ws::EPI_LD + rl;
                  const float b = bi[u * 4 + cl];
                  float4 z;
                  if (PAIR) {
                    const float2 x = *reinterpret_cast<const float2*>(q);
                    const float2 y = *reinterpret_cast<const float2*>(q + ws::EPI_LD);
                    const float b1 = bi[u * 4 + cl + 1];
                    z = make_float4(fmaf(x.x, e.scale, b), fmaf(y.x, e.scale, b1), fmaf(x.y, e.scale, b),
                                    fmaf(y.y, e.scale, b1));
                  } else {
                    const float4 x = *reinterpret_cast<const float4*>(q);
                    z = make_float4(fmaf(x.x, e.scale, b), fmaf(x.y, e.scale, b), fmaf(x.z, e.scale, b),
                                    fmaf(x.w, e.scale, b));
                  }
                  if (have_prev) z = make_float4(z.x + prev[u].x, z.y + prev[u].y, z.z + prev[u].z, z.w + prev[u].w);
                  *reinterpret_cast<float4*>(ey + rb + c) = z;
                  if (eact)
                    *reinterpret_cast<float4*>(eact + rb + c) =
                        make_float4(gelu_t(z.x), gelu_t(z.y), gelu_t(z.z), gelu_t(z.w));
                }
                __syncwarp();
                if (have_prev) {
#pragma unroll
                  for (int u = 0; u < 8; ++u) prev[u] = next[u];
                }
              }
            } else {
            float prev[32], next[32];
            columns(0);
            if (have_prev) fetch(prev, 0);
            ok = landed();
#pragma unroll 1
            for (int c0 = 0; ok && c0 < BN && nt * BN + c0 < e.N; c0 += 32) {
              columns(c0 + 32);
              if (have_prev && c0 + 32 < BN && nt * BN + c0 + 32 < e.N) fetch(next, c0 + 32);
              const long long* const co = off_s[(c0 >> 5) & 1][wi];
              const float* const bi = bias_s[(c0 >> 5) & 1][wi];
#pragma unroll
              for (int h = 0; h < 32; h += 16) {
                uint32_t v[16];
                tmem_ld16(acc + (uint32_t)(c0 + h), v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const long long cj = co[h + j];
                  if (row_ok && cj >= 0) {
                    float z = fmaf(__uint_as_float(v[j]), e.scale, bi[h + j]);
                    if (have_prev) z += prev[h + j];
                    ey[rbase + cj] = z;
                    if (eact) eact[rbase + cj] = gelu_t(z);
                  }
                }
              }
              __syncwarp();
              if (have_prev) {
#pragma unroll
                for (int j = 0; j < 32; ++j) prev[j] = next[j];
              }
            }
            }
            __syncwarp();
          }
        }
        if (!ok) break;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[eg]);
      }
    };
    switch (w.form) {
      case OUT_PART: finish(ws::Tag<OUT_PART>{}); break;
      case OUT_VEC: finish(ws::Tag<OUT_VEC>{}); break;
      case OUT_COLS: finish(ws::Tag<OUT_COLS>{}); break;
      case OUT_RVEC: finish(ws::Tag<OUT_RVEC>{}); break;
      case OUT_PAIR: finish(ws::Tag<OUT_PAIR>{}); break;
      default: finish(ws::Tag<OUT_ROWS>{}); break;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == ws::MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TMEM_COLS) : "memory");
}

// Resident CTAs per SM of gemm_ws_kernel<BN, FUSE> (shared memory, registers and the two
// accumulators' tensor-memory columns), per device.
template <int BN, bool FUSE>
cudaError_t ws_slots(int& slots) {
  static std::atomic<int> cache[64];
  int dev = 0;
  cudaError_t c = cudaGetDevice(&dev);
  if (c != cudaSuccess) return c;
  const int d = dev & 63;
  int v = cache[d].load(std::memory_order_acquire);
  if (v <= 0) {
    // the registers the roles take must be there at launch, or setmaxnreg waits for good
    cudaFuncAttributes fa{};
    c = cudaFuncGetAttributes(&fa, gemm_ws_kernel<BN, FUSE>);
    if (c != cudaSuccess) return c;
    if (fa.numRegs * ws::THREADS < 128 * (120 + 56 + 2 * 168)) return cudaErrorInvalidConfiguration;
    c = cudaFuncSetAttribute(gemm_ws_kernel<BN, FUSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, ws::Cfg<BN>::SMEM);
    if (c != cudaSuccess) return c;
    // all of the unified L1 as shared memory
    c = cudaFuncSetAttribute(gemm_ws_kernel<BN, FUSE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (c != cudaSuccess) return c;
    int occ = 0, sms = 0;
    c = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, gemm_ws_kernel<BN, FUSE>, ws::THREADS, ws::Cfg<BN>::SMEM);
    if (c != cudaSuccess) return c;
    c = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (c != cudaSuccess) return c;
    occ = std::min(occ, (int)(512 / ws::Cfg<BN>::TMEM_COLS));
    if (occ < 1) return cudaErrorInvalidConfiguration;
    v = occ * sms;
    cache[d].store(v, std::memory_order_release);
  }
  slots = v;
  return cudaSuccess;
}

template <int BN, bool FUSE = false>
cudaError_t launch_ws_bn(WsArgs w, const Epi& e, int* err, cudaStream_t st, long long batch) {
  int slots = 0;
  cudaError_t c = ws_slots<BN, FUSE>(slots);
  if (c != cudaSuccess) return c;
  ws::op_mode(w.a, BM, w.K);
  if (FUSE) ws::op_mode(w.b, BN, w.K);
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };  // null included
  const Addr& o = e.out;
  const bool cols = o.kc == 1 && o.t1 == 1, whole = e.ybs % 4 == 0 && al(e.y) && al(e.add) && al(e.act);
  const bool rows = o.rc == 1 ? o.s1 == 1 : o.s2 == 1 && o.rc % 4 == 0 && o.s1 % 4 == 0;
  const bool pair = o.kc == 2 && o.t2 == 1 && o.s2 == 2 && o.rc > 1 && o.rc % 2 == 0;
  w.form = w.part ? OUT_PART
           : cols ? (whole && e.N % 4 == 0 && o.s1 % 4 == 0 && (o.rc == 1 || o.s2 % 4 == 0) ? OUT_VEC : OUT_COLS)
           : o.kc >= 32 && o.t2 < (o.rc == 1 ? o.s1 : o.s2) ? OUT_COLS
           : pair && whole && e.M % 2 == 0 && e.N % 2 == 0 && o.t1 % 4 == 0 && o.s1 % 4 == 0 ? OUT_PAIR
           : rows && whole && e.M % 4 == 0 && o.t1 % 4 == 0 && (o.kc == 1 || o.t2 % 4 == 0) ? OUT_RVEC
                                                                                         : OUT_ROWS;
  w.items = batch * w.splits * w.mtiles * w.ntiles;
  const unsigned grid = (unsigned)std::min<long long>(w.items, slots);
  gemm_ws_kernel<BN, FUSE><<<grid, ws::THREADS, ws::Cfg<BN>::SMEM, st>>>(w, e, err);
  return cudaGetLastError();
}

cudaError_t launch_ws(int bn, const WsArgs& w, const Epi& e, int* err, cudaStream_t st, long long batch) {
  switch (bn) {
    case 32:
      return w.b_img ? launch_ws_bn<32>(w, e, err, st, batch) : launch_ws_bn<32, true>(w, e, err, st, batch);
    case 64: return launch_ws_bn<64>(w, e, err, st, batch);
    case 128: return launch_ws_bn<128>(w, e, err, st, batch);
    default: return launch_ws_bn<256>(w, e, err, st, batch);
  }
}

// Split-K with B from FP32 (BN = 32): one split per resident CTA.
int ws_split_count(int kblocks, int ksplit) {
  int slots = 0;
  if (ws_slots<32, true>(slots) != cudaSuccess) slots = 1;
  return std::max(1, std::min(kblocks, std::max(ksplit, slots)));
}

template <int BN>
cudaError_t launch_gemm_bn(const uint8_t* a, const uint8_t* b, long long mtiles, int ntiles, int kblocks, int kper,
                           float* part, const Epi& e, int* err, cudaStream_t st) {
  // the shared-memory attribute is set once per device (it belongs to the device's context)
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t c0 = cudaGetDevice(&dev);
  if (c0 != cudaSuccess) return c0;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(configured.load(std::memory_order_acquire) & bit)) {
    cudaError_t c = cudaFuncSetAttribute(gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM);
    if (c != cudaSuccess) return c;
    configured.fetch_or(bit, std::memory_order_release);
  }
  const int splits = (kblocks + kper - 1) / kper;
  gemm_kernel<BN><<<(unsigned)(mtiles * ntiles * splits), 128, Cfg<BN>::SMEM, st>>>(
      a, b, kblocks, ntiles, (int)(mtiles * ntiles), kper, part, e, err);
  if (part) {
    const long long n = e.M * (long long)e.N;
    splitk_reduce_kernel<<<(unsigned)((n + REDUCE_WARPS - 1) / REDUCE_WARPS), 32 * REDUCE_WARPS, 0, st>>>(
        part, splits, (int)(mtiles * ntiles), ntiles, BN, e);
  }
  return cudaGetLastError();
}

}  // namespace tg

// ------------------------------------------------------------------ host side
namespace {
int bn_for(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256; }
}  // namespace

int TcGemm::reserve(size_t a_bytes, size_t b_bytes) {
  if (!err) {
    if (cudaMalloc(&err, sizeof(int)) != cudaSuccess || cudaMemset(err, 0, sizeof(int)) != cudaSuccess)
      return MSX_ERR_ALLOC;
  }
  if (a_bytes > a_cap) {
    if (a_img) cudaFree(a_img);
    a_img = nullptr;
    a_cap = 0;
    if (cudaMalloc(&a_img, a_bytes) != cudaSuccess) return MSX_ERR_ALLOC;
    a_cap = a_bytes;
  }
  if (b_bytes > b_cap) {
    if (b_img) cudaFree(b_img);
    b_img = nullptr;
    b_cap = 0;
    if (cudaMalloc(&b_img, b_bytes) != cudaSuccess) return MSX_ERR_ALLOC;
    b_cap = b_bytes;
  }
  return MSX_OK;
}

void TcGemm::release() {
  for (void* p : {(void*)a_img, (void*)b_img, (void*)err, (void*)part})
    if (p) cudaFree(p);
  a_img = b_img = nullptr;
  err = nullptr;
  part = nullptr;
  a_cap = b_cap = part_cap = 0;
}

int TcGemm::run(const float* a, Addr aa, const float* b, Addr ba, long long M, int N, long long K, const Epi& epi,
                cudaStream_t st, int ksplit) {
  if (M <= 0 || N <= 0 || K <= 0 || N > 4096 || ksplit < 1) return MSX_ERR_INVALID;
  const int bn = bn_for(N);
  const long long mtiles = (M + tg::BM - 1) / tg::BM;
  const int ntiles = (N + bn - 1) / bn;
  const long long kbl = (K + tg::BK - 1) / tg::BK;
  if (kbl > (1LL << 30) || mtiles * ntiles > (1LL << 30)) return MSX_ERR_INVALID;
  const int kblocks = (int)kbl;
  Epi e = epi;
  e.M = M;
  e.N = N;
  e.ybs = 0;
  tg::WsArgs w{};
  w.a = tg::ws::Op{a, aa, 0, M, 0, 0, 0, 0, 0};
  w.b = tg::ws::Op{b, ba, 0, N, 0, 0, 0, 0, 0};
  w.K = K;
  w.kblocks = kblocks;
  w.ntiles = ntiles;
  w.mtiles = mtiles;
  auto ensure_part = [&](size_t need) -> int {
    if (need > part_cap) {
      if (part) cudaFree(part);
      part = nullptr;
      part_cap = 0;
      if (cudaMalloc(&part, need * sizeof(float)) != cudaSuccess) return MSX_ERR_ALLOC;
      part_cap = need;
    }
    return MSX_OK;
  };
  if (ksplit > 1 && bn == 32) {
    // long K, narrow output (weight gradients): split K over the persistent CTAs, both
    // operands rounded to bfloat16 as they are loaded, partial tiles summed in split order
    const int splits = tg::ws_split_count(kblocks, ksplit);
    w.kper = (kblocks + splits - 1) / splits;
    w.splits = (kblocks + w.kper - 1) / w.kper;
    int rc = reserve(0, 0);
    if (rc != MSX_OK) return rc;
    rc = ensure_part((size_t)w.splits * mtiles * ntiles * tg::BM * bn);
    if (rc != MSX_OK) return rc;
    w.part = part;
    w.b_img = nullptr;
    cudaError_t c = tg::launch_ws(bn, w, e, err, st, 1);
    if (c != cudaSuccess) return MSX_ERR_CUDA;
    const long long n = M * (long long)N;
    tg::splitk_reduce_kernel<<<(unsigned)((n + tg::REDUCE_WARPS - 1) / tg::REDUCE_WARPS), 32 * tg::REDUCE_WARPS, 0,
                               st>>>(part, w.splits, (int)(mtiles * ntiles), ntiles, bn, e);
    return cudaGetLastError() == cudaSuccess ? MSX_OK : MSX_ERR_CUDA;
  }
  int kper = kblocks;
  if (ksplit > 1) kper = (kblocks + ksplit - 1) / ksplit;
  const int splits = (kblocks + kper - 1) / kper;
  const size_t a_bytes = splits > 1 ? (size_t)mtiles * kblocks * tg::A_BYTES : 0;
  const size_t b_bytes = (size_t)ntiles * kblocks * bn * tg::BK * 2;
  int rc = reserve(a_bytes, b_bytes);
  if (rc != MSX_OK) return rc;
  const long long a_rows = mtiles * tg::BM, b_rows = (long long)ntiles * bn;
  const long long a_thr = a_rows * kblocks * (tg::BK / 8), b_thr = b_rows * kblocks * (tg::BK / 8);
  tg::pack_kernel<<<(unsigned)((b_thr + 255) / 256), 256, 0, st>>>(b, ba, N, K, bn, b_rows, kblocks,
                                                                   reinterpret_cast<uint4*>(b_img));
  const uint8_t* bi = reinterpret_cast<const uint8_t*>(b_img);
  cudaError_t c;
  if (splits == 1) {  // persistent kernel, A rounded to bfloat16 as it is loaded
    w.kper = kblocks;
    w.splits = 1;
    w.b_img = bi;
    c = tg::launch_ws(bn, w, e, err, st, 1);
    return c == cudaSuccess ? MSX_OK : MSX_ERR_CUDA;
  }
  // split K with a wide output: both operands packed, one CTA per (tile, split)
  rc = ensure_part((size_t)splits * mtiles * ntiles * tg::BM * bn);
  if (rc != MSX_OK) return rc;
  tg::pack_kernel<<<(unsigned)((a_thr + 255) / 256), 256, 0, st>>>(a, aa, M, K, tg::BM, a_rows, kblocks,
                                                                   reinterpret_cast<uint4*>(a_img));
  const uint8_t* ai = reinterpret_cast<const uint8_t*>(a_img);
  switch (bn) {
    case 64: c = tg::launch_gemm_bn<64>(ai, bi, mtiles, ntiles, kblocks, kper, part, e, err, st); break;
    case 128: c = tg::launch_gemm_bn<128>(ai, bi, mtiles, ntiles, kblocks, kper, part, e, err, st); break;
    default: c = tg::launch_gemm_bn<256>(ai, bi, mtiles, ntiles, kblocks, kper, part, e, err, st); break;
  }
  return c == cudaSuccess ? MSX_OK : MSX_ERR_CUDA;
}

int TcGemm::run_cplx(const float* a, Addr aa, long long a_bs, const float* src, long long si, long long sj, long long sp,
                     long long src_bs, int hn, int hk, int neg, long long M, const Epi& epi, long long y_bs, int batch,
                     cudaStream_t st) {
  if (batch < 1 || M <= 0 || hn <= 0 || hk <= 0 || 2 * hn > 4096 || neg < 0 || neg > 2) return MSX_ERR_INVALID;
  const int N = 2 * hn;
  const long long K = 2LL * hk;
  const int bn = bn_for(N);
  const long long mtiles = (M + tg::BM - 1) / tg::BM;
  const int ntiles = (N + bn - 1) / bn;
  const int kblocks = (int)((K + tg::BK - 1) / tg::BK);
  if (mtiles * ntiles * batch > (1LL << 30)) return MSX_ERR_INVALID;
  const size_t b_bytes = (size_t)batch * ntiles * kblocks * bn * tg::BK * 2;
  int rc = reserve(0, b_bytes);
  if (rc != MSX_OK) return rc;
  const int b_rows = ntiles * bn;
  const long long b_thr = (long long)b_rows * kblocks * (tg::BK / 8) * batch;
  tg::pack_cplx_kernel<<<(unsigned)((b_thr + 255) / 256), 256, 0, st>>>(src, si, sj, sp, src_bs, hn, hk, neg, bn, b_rows,
                                                                        kblocks, reinterpret_cast<uint4*>(b_img),
                                                                        batch);
  Epi e = epi;
  e.M = M;
  e.N = N;
  e.ybs = y_bs;
  const uint8_t* bi = reinterpret_cast<const uint8_t*>(b_img);
  cudaError_t c;
  tg::WsArgs w{};
  w.a = tg::ws::Op{a, aa, a_bs, M, 0, 0, 0, 0, 0};
  w.b_img = bi;
  w.K = K;
  w.kblocks = kblocks;
  w.kper = kblocks;
  w.splits = 1;
  w.ntiles = ntiles;
  w.mtiles = mtiles;
  c = tg::launch_ws(bn, w, e, err, st, batch);
  return c == cudaSuccess ? MSX_OK : MSX_ERR_CUDA;
}

int TcGemm::check() {
  if (!err) return MSX_OK;
  int h = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return MSX_ERR_CUDA;  // a copy alone does not wait for non-blocking streams
  if (cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return MSX_ERR_CUDA;
  if (h) {
    cudaMemset(err, 0, sizeof(int));
    return MSX_ERR_TIMEOUT;
  }
  return MSX_OK;
}

}  // namespace msx

namespace {
// scratch of msx_gemm_bf16, per host thread and device
struct GemmScratch {
  msx::TcGemm gemm;
  msx::ScratchOrder order;
};
thread_local msx::PerDevice<GemmScratch> g_gemm;
}  // namespace

extern "C" int msx_gemm_bf16(const float* a_dev, int lda, const float* b_dev, int ldb, int m, int n, int k,
                             float* c_dev, int ldc, const float* bias_dev, int accumulate, void* stream) {
  if (!a_dev || !b_dev || !c_dev || m <= 0 || n <= 0 || k <= 0 || lda < k || ldb < k || ldc < n || n > 4096) {
    msx::set_last_error("gemm_bf16: bad arguments (need m, n, k > 0, n <= 4096, leading dimensions >= row lengths)");
    return MSX_ERR_INVALID;
  }
  msx::Epi e{};
  e.y = c_dev;
  e.out = msx::rowmajor(ldc);
  e.bias = bias_dev;
  e.accumulate = accumulate ? 1 : 0;
  e.scale = 1.f;
  // long K with few output tiles: split K over CTAs
  const long long tiles = ((m + 127) / 128) * (long long)((n + 255) / 256);
  const int ksplit = (k >= 4096 && tiles < 64) ? (int)((k / 2048) < 64 ? (k / 2048) : 64) : 1;
  const cudaStream_t st = (cudaStream_t)stream;
  GemmScratch* g = g_gemm.here();
  if (!g || g->order.enter(st) != cudaSuccess) {
    msx::set_last_error("gemm_bf16: no device, or its stream is unusable");
    return MSX_ERR_CUDA;
  }
  int rc = g->gemm.run(a_dev, msx::rowmajor(lda), b_dev, msx::rowmajor(ldb), m, n, k, e, st, ksplit);
  if (g->order.leave(st) != cudaSuccess && rc == MSX_OK) rc = MSX_ERR_CUDA;
  if (rc == MSX_ERR_ALLOC) msx::set_last_error("gemm_bf16: operand image allocation failed");
  else if (rc == MSX_ERR_CUDA) msx::set_last_error("gemm_bf16: launch failed");
  else if (rc != MSX_OK) msx::set_last_error("gemm_bf16: bad sizes");
  return rc;
}

extern "C" int msx_gemm_check(void) {
  GemmScratch* g = g_gemm.here();
  const int rc = g ? g->gemm.check() : MSX_ERR_CUDA;
  if (rc == MSX_ERR_TIMEOUT) msx::set_last_error("a tensor-core GEMM wait gave up");
  return rc;
}
