// Split-KV attention forward for short query blocks (decode shapes), fp16 / bf16, sm_100a.
//
// The reference has no such path: with seqQ = 1 its grid is one CTA per (batch, Q head) walking every KV tile and
// every Q head of a GQA group re-reads the same K/V (reference csrc/flash_attn/launcher.cuh:32,
// params.cuh:25-27).  This path is bound by HBM bandwidth - K and V are read exactly once - so it is organised
// around memory parallelism, not around the tcgen05 pipe:
//   * the (seqQ x group) query rows that share one KV head (at most 16) form one 16-row MMA tile, so a KV head is
//     streamed once for all of its Q heads;
//   * the key blocks of all batch entries are cut into equal runs, so that every CTA that fits the GPU streams the same
//     amount whatever the batch and the lengths are (packed input: key-range splits of every sequence);
//   * each CTA streams 64-key K and V blocks through a 3-stage cp.async ring (16-byte chunks, XOR-swizzled so that
//     ldmatrix is conflict-free); each of its 4 warps owns 16 keys of a block with its own online softmax
//     (mma.sync m16n8k16, fp32 accumulate: the tensor work is negligible next to the memory stream);
//   * warps are merged through shared memory, partial results through a small fp32 scratch buffer and a combine kernel
//     that is launched while the split kernel runs (programmatic dependent launch) and reads a row's partials side by side.
// Measured against a fixed number of splits per pair and a combine kernel that walked them (8 KV heads, D = 128, three sets of
// inputs in turn, both builds in one job; floor in brackets at 6.54 TB/s): batch 1 x 32768 keys 37.3 -> 28.3 us (20.5), 8 x 20011
// 112.5 -> 101.3 (100), 40 x 5000 168.9 -> 128.3 (125), 13 x 8000 75.9 -> 70.8 (65), 6 x 12000 61.6 -> 52.0 (45).  What is left at
// small batch is launch, the first loads and the combine.
// Numerical contract as in the main kernel (reference csrc/flash_attn/mma/softmax.cuh:67-138): scale 1/sqrt(D)
// folded into exp2, top-left causal mask, "col >= seqLenKV" mask, P rounded to the 16-bit type before P.V, row sum
// from unrounded P, empty rows give 0.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <mutex>

#include "../../include/tinyfa_b200.h"
#include "build_config.cuh"
#include "ptx_sm100.cuh"
#include "tfa_common.cuh"

namespace tfa_b200 {

int device_num_sms(int device);  // c_abi.cu

namespace decode {

constexpr int kThreads = 128;
constexpr int kBlockKeys = 64;
constexpr int kStages = 3;
constexpr int kRows = 16;  // query rows per CTA (MMA M)

struct Params {
  const void* Q;
  const void* K;
  const void* V;
  void* O;          // final output (16-bit)
  float* partO;     // [splits][totalQRows][Hq][D] normalised partial outputs (splits > 1)
  float* partLse;   // [splits][totalQRows][Hq]   log2-domain log-sum-exp of each partial
  const int* cuQ;
  const int* cuKV;
  int seqLenQ;
  int seqLenKV;
  int headsQ;
  int headsKV;
  int group;
  int causal;
  // Even partition (fixed-length input): the key blocks of all batch entries, in order, are cut into `runs` equal runs; a
  // CTA is one KV head of a run.  runs == 0: one CTA per (split, KV head, batch entry) of a three-dimensional grid.
  int runs;
  int blocksPerEntry;
  long long totalBlocks;
  int splits;        // three-dimensional grid: key-range splits
  int keysPerSplit;  // three-dimensional grid: multiple of kBlockKeys
  long long totalQ;  // rows of Q (for the partial buffers' stride)
  float scaleLog2;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
template <bool kBf16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fmax_nan(float a, float b) {  // NaN is kept
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

// Byte offset of 16-byte chunk `c` of row `r` in a tile whose rows hold D 16-bit elements.
// Rows are D * 2 bytes and contiguous, so which banks a row starts on depends on D: for D = 64, 128, 192, 256 every
// row starts on bank 0 and chunk c is exchanged with c ^ (r & 7) (stays inside its group of eight chunks); for D = 32
// and 96 (64- and 192-byte rows) rows alternate between the two halves of the 128-byte bank line and the chunk is
// exchanged inside its group of four, c ^ ((r >> 1) & 3).  Either way the eight rows of an ldmatrix hit eight
// different 16-byte bank groups.
template <int D>
__device__ __forceinline__ uint32_t swz(int r, int c) {
  if constexpr (D == 32 || D == 96) {
    return (uint32_t)(r * (D * 2) + ((c ^ ((r >> 1) & 3)) << 4));
  } else {
    return (uint32_t)(r * (D * 2) + ((c ^ (r & 7)) << 4));
  }
}

// Row pitch (floats) of the merge buffer: eight floats past a multiple of the 32 banks, so that the eight rows of a warp's
// accumulator fragment do not share a bank.
template <int D>
constexpr int merge_ld() {
  return D + 8;
}

// 64 keys x D of one KV head -> one stage; keys >= keyEnd are zero-filled.
template <int D>
__device__ __forceinline__ void load_block(uint32_t smemDst, const uint16_t* base, long long rowStride, long long key0,
                                           long long keyEnd) {
  constexpr int kChunksPerRow = D / 8;
  constexpr int kChunks = kBlockKeys * kChunksPerRow;
#pragma unroll
  for (int i = 0; i < kChunks / kThreads; i++) {
    const int idx = threadIdx.x + i * kThreads;
    const int r = idx / kChunksPerRow, c = idx % kChunksPerRow;
    const bool valid = (key0 + r) < keyEnd;
    const uint16_t* src = base + (valid ? (key0 + r) * rowStride + c * 8 : 0);
    cp_async16(smemDst + swz<D>(r, c), src, valid);
  }
}

// Run of the even partition that holds block `u`, i.e. the c with total * c / runs <= u < total * (c + 1) / runs.
__host__ __device__ __forceinline__ int run_of_block(long long u, long long total, int runs) {
  return (int)(((u + 1) * runs - 1) / total);
}

// kEven: the even partition; else one CTA per (split, KV head, batch entry).  Instantiations of their own, and a load address worked out
// anew for every block: the code that carries a run on into the next entry cost calls of whole pairs up to 3 % (16 x 16384 keys, 32 heads over 32
// of 128 667 -> 641 us).  The number of CTAs per SM is stated because without it the compiler keeps to 168 registers at head dim 128, where two
// CTAs have 255 each: runs 665 -> 617 us there.  Head dim 32 is better off with 8 CTAs than with 7 of 65 registers.
template <int D, bool kBf16, bool kEven>
__global__ void __launch_bounds__(kThreads, (D == 32 && !kEven) ? 8 : 1) fwd_splitkv_kernel(const Params p) {
  constexpr int kTileBytes = kBlockKeys * D * 2;
  constexpr int kNT = D / 8;  // 8-wide output column tiles
  constexpr int kLdO = merge_ld<D>();
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sBase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  // merge buffer: behind the ring where the next entry's blocks are on their way into it meanwhile, one warp after the other; else
  // in the ring, all warps at once (320 CTAs of six blocks at head dim 256: 43.2 -> 39.4 us)
  constexpr int kParts = kEven ? 1 : 4;
  float* sO = reinterpret_cast<float*>(smem + (kEven ? kStages * 2 * kTileBytes : 0));  // [kParts][16][kLdO]
  float* sM = sO + kParts * kRows * kLdO;                                 // [4][16]
  float* sL = sM + 4 * kRows;                                             // [4][16]

  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  int b, part;         // batch entry and partial-result slot of the current segment
  int hkv;
  int sq, skv;
  long long qRow0, kvRow0;
  int key0, keyEnd;    // keys of the entry that this CTA starts at / may see
  int count;           // blocks of this CTA
  if constexpr (kEven) {
    // neighbouring CTAs are the KV heads of one run: they read neighbouring parts of the same rows at the same time
    const int run = (int)blockIdx.x / p.headsKV;
    hkv = (int)blockIdx.x - run * p.headsKV;
    const long long u0 = p.totalBlocks * run / p.runs, u1 = p.totalBlocks * (run + 1) / p.runs;
    b = (int)(u0 / p.blocksPerEntry);
    const long long first = (long long)b * p.blocksPerEntry;
    key0 = (int)(u0 - first) * kBlockKeys;
    count = (int)(u1 - u0);
    part = run - run_of_block(first, p.totalBlocks, p.runs);
    sq = p.seqLenQ;
    skv = p.seqLenKV;
    qRow0 = (long long)b * sq;
    kvRow0 = (long long)b * skv;
    keyEnd = p.causal ? min(skv, sq) : skv;  // top-left causal: key j needs j <= i <= sq-1
  } else {
    part = blockIdx.x;
    hkv = blockIdx.y;
    b = blockIdx.z;
    if (p.cuQ != nullptr) {
      qRow0 = p.cuQ[b];
      sq = p.cuQ[b + 1] - p.cuQ[b];
      kvRow0 = p.cuKV[b];
      skv = p.cuKV[b + 1] - p.cuKV[b];
    } else {
      sq = p.seqLenQ;
      skv = p.seqLenKV;
      qRow0 = (long long)b * sq;
      kvRow0 = (long long)b * skv;
    }
    if (sq <= 0) return;
    if (skv <= 0) return;  // nothing to write
    keyEnd = p.causal ? min(skv, sq) : skv;
    // keysPerSplit comes from the caller's maximum key length, which only sizes the launch: the last split runs to
    // the real end of the sequence, so an understated maximum loses no keys (the reference derives its key loop from
    // the actual length as well, reference csrc/flash_attn/params.cuh:156-163).
    key0 = part * p.keysPerSplit;
    if (part != p.splits - 1) keyEnd = min(key0 + p.keysPerSplit, keyEnd);
    count = (keyEnd > key0) ? (keyEnd - key0 + kBlockKeys - 1) / kBlockKeys : 0;
  }
  // <= 16 by dispatch; packed input may hold a sequence longer than the caller's maximum: its further rows are not computed
  const int nRows = min(sq * p.group, kRows);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;

  const long long qStride = (long long)p.headsQ * D;
  const long long kvStride = (long long)p.headsKV * D;

  // rows of this thread's fragments: r0 = g, r1 = g + 8; row r <-> (query position r / group, head hkv*group + r % group)
  const int rowA = g, rowB = g + 8;
  const int qposA = rowA / p.group, qposB = rowB / p.group;
  const bool validA = rowA < nRows, validB = rowB < nRows;
  const float c = p.scaleLog2;

  float o[kNT][4];
  float mA, mB, lA, lB;
  uint32_t qf[D / 16][4];
  auto startSegment = [&]() {
#pragma unroll
    for (int i = 0; i < kNT; i++) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    mA = mB = -INFINITY;
    lA = lB = 0.f;
    // Q fragments (A operand), straight from global memory.
    const uint16_t* gQ = reinterpret_cast<const uint16_t*>(p.Q);
    const uint16_t* qa = gQ + (qRow0 + qposA) * qStride + (long long)(hkv * p.group + rowA % p.group) * D;
    const uint16_t* qb = gQ + (qRow0 + qposB) * qStride + (long long)(hkv * p.group + rowB % p.group) * D;
#pragma unroll
    for (int ks = 0; ks < D / 16; ks++) {
      const int c0 = ks * 16 + 2 * tig;
      qf[ks][0] = validA ? *reinterpret_cast<const uint32_t*>(qa + c0) : 0u;
      qf[ks][1] = validB ? *reinterpret_cast<const uint32_t*>(qb + c0) : 0u;
      qf[ks][2] = validA ? *reinterpret_cast<const uint32_t*>(qa + c0 + 8) : 0u;
      qf[ks][3] = validB ? *reinterpret_cast<const uint32_t*>(qb + c0 + 8) : 0u;
    }
  };

  // Merges the four warps (each saw a disjoint quarter of the keys of every block) and stores the segment's result:
  // the final output when `whole`, else partial `part`.
  auto storeSegment = [&](bool whole) {
    lA += __shfl_xor_sync(0xffffffffu, lA, 1);
    lA += __shfl_xor_sync(0xffffffffu, lA, 2);
    lB += __shfl_xor_sync(0xffffffffu, lB, 1);
    lB += __shfl_xor_sync(0xffffffffu, lB, 2);
    if (tig == 0) {
      sM[warp * kRows + rowA] = mA;
      sM[warp * kRows + rowB] = mB;
      sL[warp * kRows + rowA] = lA;
      sL[warp * kRows + rowB] = lB;
    }
    __syncthreads();
    float MA = -INFINITY, MB = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; w++) {
      MA = fmaxf(MA, sM[w * kRows + rowA]);
      MB = fmaxf(MB, sM[w * kRows + rowB]);
    }
    const float fA = (mA == -INFINITY) ? 0.f : ex2((mA - MA) * c), fB = (mB == -INFINITY) ? 0.f : ex2((mB - MB) * c);
    if constexpr (kEven) {
#pragma unroll 1
      for (int w = 0; w < 4; w++) {  // one warp after the other adds its share
        if (w == warp) {
#pragma unroll
          for (int nt = 0; nt < kNT; nt++) {
            float2* a = reinterpret_cast<float2*>(sO + rowA * kLdO + nt * 8 + 2 * tig);
            float2* bq = reinterpret_cast<float2*>(sO + rowB * kLdO + nt * 8 + 2 * tig);
            const float2 za = (w == 0) ? make_float2(0.f, 0.f) : *a, zb = (w == 0) ? make_float2(0.f, 0.f) : *bq;
            *a = make_float2(fmaf(o[nt][0], fA, za.x), fmaf(o[nt][1], fA, za.y));
            *bq = make_float2(fmaf(o[nt][2], fB, zb.x), fmaf(o[nt][3], fB, zb.y));
          }
        }
        __syncthreads();
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < kNT; nt++) {
        *reinterpret_cast<float2*>(sO + (warp * kRows + rowA) * kLdO + nt * 8 + 2 * tig) = make_float2(o[nt][0] * fA, o[nt][1] * fA);
        *reinterpret_cast<float2*>(sO + (warp * kRows + rowB) * kLdO + nt * 8 + 2 * tig) = make_float2(o[nt][2] * fB, o[nt][3] * fB);
      }
      __syncthreads();
    }
    for (int idx = threadIdx.x; idx < nRows * (D / 4); idx += kThreads) {
      const int r = idx / (D / 4), c4 = idx % (D / 4);
      float m = -INFINITY;
#pragma unroll
      for (int w = 0; w < 4; w++) m = fmaxf(m, sM[w * kRows + r]);
      float l = 0.f;
#pragma unroll
      for (int w = 0; w < 4; w++) {
        const float mw = sM[w * kRows + r];
        l += sL[w * kRows + r] * ((mw == -INFINITY) ? 0.f : ex2((mw - m) * c));
      }
      const float inv = (l > 0.f) ? (1.f / l) : 0.f;
      float4 acc = *reinterpret_cast<const float4*>(sO + r * kLdO + c4 * 4);
#pragma unroll
      for (int w = 1; w < kParts; w++) {
        const float4 v = *reinterpret_cast<const float4*>(sO + (w * kRows + r) * kLdO + c4 * 4);
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
      }
      acc.x *= inv;
      acc.y *= inv;
      acc.z *= inv;
      acc.w *= inv;
      const long long orow = (qRow0 + r / p.group) * p.headsQ + hkv * p.group + r % p.group;
      if (whole) {
        uint2 out;
        out.x = pack2<kBf16>(acc.x, acc.y);
        out.y = pack2<kBf16>(acc.z, acc.w);
        *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.O) + orow * D + c4 * 4) = out;
      } else {
        const long long prow = (long long)part * p.totalQ * p.headsQ + orow;
        *reinterpret_cast<float4*>(p.partO + prow * D + c4 * 4) = acc;
        if (c4 == 0) p.partLse[prow] = (l == 0.f) ? -INFINITY : (m * c + log2f(l));  // NaN stays NaN
      }
    }
  };

  startSegment();
  // load cursor: runs kStages - 1 blocks ahead, across segment ends
  [[maybe_unused]] int ldKey = key0;
  const uint16_t* gK = reinterpret_cast<const uint16_t*>(p.K) + kvRow0 * kvStride + (long long)hkv * D;
  const uint16_t* gV = reinterpret_cast<const uint16_t*>(p.V) + kvRow0 * kvStride + (long long)hkv * D;
  auto loadBlock = [&](int blk) {
    const uint32_t stage = sBase + (blk % kStages) * 2 * kTileBytes;
    if constexpr (kEven) {
      load_block<D>(stage, gK, kvStride, ldKey, keyEnd);
      load_block<D>(stage + kTileBytes, gV, kvStride, ldKey, keyEnd);
      ldKey += kBlockKeys;
      if (ldKey >= keyEnd) {  // the next batch entry
        ldKey = 0;
        const long long step = (long long)skv * kvStride;
        gK += step;
        gV += step;
      }
    } else {
      load_block<D>(stage, gK, kvStride, key0 + blk * kBlockKeys, keyEnd);
      load_block<D>(stage + kTileBytes, gV, kvStride, key0 + blk * kBlockKeys, keyEnd);
    }
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; s++) {
    if (s < count) loadBlock(s);
    cp_async_commit();
  }
  [[maybe_unused]] int segStart = key0, kbase = key0;  // first key of the segment / of the block
  for (int blk = 0; blk < count; blk++) {
    if (blk + kStages - 1 < count) loadBlock(blk + kStages - 1);
    cp_async_commit();
    cp_async_wait<kStages - 1>();
    __syncthreads();
    const uint32_t sK = sBase + (blk % kStages) * 2 * kTileBytes;
    const uint32_t sV = sK + kTileBytes;
    const int kb = (kEven ? kbase : key0 + blk * kBlockKeys) + warp * 16;  // first key of this warp's 16-key slice
    if (kb < keyEnd) {
      // ---- S = Q K^T for 16 rows x 16 keys
      float sc[2][4];
#pragma unroll
      for (int n = 0; n < 2; n++) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < D / 16; ks++) {
        // matrices: (keys 0-7, dims lo), (keys 0-7, dims hi), (keys 8-15, dims lo), (keys 8-15, dims hi)
        const int r = warp * 16 + (lane & 7) + ((lane >> 4) << 3);
        const int ch = ks * 2 + ((lane >> 3) & 1);
        uint32_t kf[4];
        ldmatrix_x4(sK + swz<D>(r, ch), kf);
        mma16816<kBf16>(sc[0], qf[ks], kf[0], kf[1]);
        mma16816<kBf16>(sc[1], qf[ks], kf[2], kf[3]);
      }
      // ---- mask (tail of the key range, top-left causal)
      const bool needMask = (kb + 16 > keyEnd) || p.causal;
      if (needMask) {
#pragma unroll
        for (int n = 0; n < 2; n++) {
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int key = kb + n * 8 + 2 * tig + (e & 1);
            const int qpos = (e < 2) ? qposA : qposB;
            if (key >= keyEnd || (p.causal && key > qpos)) sc[n][e] = -INFINITY;
          }
        }
      }
      // ---- online softmax for rows g (A) and g+8 (B)
      float mxA = fmaxf(fmaxf(sc[0][0], sc[0][1]), fmaxf(sc[1][0], sc[1][1]));
      float mxB = fmaxf(fmaxf(sc[0][2], sc[0][3]), fmaxf(sc[1][2], sc[1][3]));
      mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 1));
      mxA = fmaxf(mxA, __shfl_xor_sync(0xffffffffu, mxA, 2));
      mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 1));
      mxB = fmaxf(mxB, __shfl_xor_sync(0xffffffffu, mxB, 2));
      const float mnA = fmaxf(mA, mxA), mnB = fmaxf(mB, mxB);
      const float muA = (mnA == -INFINITY) ? 0.f : mnA, muB = (mnB == -INFINITY) ? 0.f : mnB;
      const float scA = (mA == -INFINITY) ? 0.f : ex2((mA - muA) * c);
      const float scB = (mB == -INFINITY) ? 0.f : ex2((mB - muB) * c);
      mA = mnA;
      mB = mnB;
      float pA[4], pB[4];
#pragma unroll
      for (int n = 0; n < 2; n++) {
        pA[n * 2 + 0] = ex2(fmaf(sc[n][0], c, -muA * c));
        pA[n * 2 + 1] = ex2(fmaf(sc[n][1], c, -muA * c));
        pB[n * 2 + 0] = ex2(fmaf(sc[n][2], c, -muB * c));
        pB[n * 2 + 1] = ex2(fmaf(sc[n][3], c, -muB * c));
      }
      lA = lA * scA + (pA[0] + pA[1] + pA[2] + pA[3]);  // per-thread partial, reduced over the quad at the end
      lB = lB * scB + (pB[0] + pB[1] + pB[2] + pB[3]);
      uint32_t pf[4];
      pf[0] = pack2<kBf16>(pA[0], pA[1]);
      pf[1] = pack2<kBf16>(pB[0], pB[1]);
      pf[2] = pack2<kBf16>(pA[2], pA[3]);
      pf[3] = pack2<kBf16>(pB[2], pB[3]);
      // ---- O = O * scale + P V
#pragma unroll
      for (int nt = 0; nt < kNT; nt += 2) {
        // matrices (transposed on load): (keys 0-7, dims nt), (keys 8-15, dims nt), (keys 0-7, dims nt+1), (keys 8-15, dims nt+1)
        const int r = warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3);
        const int ch = nt + (lane >> 4);
        uint32_t vf[4];
        ldmatrix_x4_trans(sV + swz<D>(r, ch), vf);
        o[nt][0] *= scA;
        o[nt][1] *= scA;
        o[nt][2] *= scB;
        o[nt][3] *= scB;
        o[nt + 1][0] *= scA;
        o[nt + 1][1] *= scA;
        o[nt + 1][2] *= scB;
        o[nt + 1][3] *= scB;
        mma16816<kBf16>(o[nt], pf, vf[0], vf[1]);
        mma16816<kBf16>(o[nt + 1], pf, vf[2], vf[3]);
      }
    }
    __syncthreads();
    if constexpr (kEven) {
      kbase += kBlockKeys;
      const bool entryDone = kbase >= keyEnd;
      if (entryDone || blk + 1 == count) {
        storeSegment(entryDone && segStart == 0);
        if (blk + 1 < count) {  // on to the next batch entry, whose blocks are already on their way
          qRow0 += sq;
          segStart = kbase = 0;
          part = 0;
          startSegment();
        }
      }
    }
  }
  cp_async_wait<0>();
  if constexpr (!kEven) storeSegment(p.splits == 1);  // a split without keys: zeros, lse = -inf
}

// O[row] = sum_s 2^(lse_s - M) O_s / sum_s 2^(lse_s - M), one CTA per output row.  Bound by the latency of two dependent
// reads (the partials' log-sum-exps, the partials), so both are spread over the CTA: every warp reads all lse of the row,
// D / 4 threads read one split's partial row and 128 / (D / 4) such groups take turns over the splits, four in flight each.
// The kernel is launched while the split kernel still runs (launch_kernel in tfa_common.cuh): the partials change during
// its lifetime, so they are read with coherent loads and their pointers promise the compiler nothing.
// Packed input: the grid is that of the split kernel with the rows of a tile in place of the splits, so that exactly the rows
// that have partials are stored - none before cu_seqlens_q[0], past the last sequence or past a tile's sixteen.
constexpr int kCombineThreads = 128;
template <int D, bool kBf16>
__global__ void __launch_bounds__(kCombineThreads)
combine_kernel(const float* partO, const float* partLse, void* O, long long rows /* totalQ * Hq */, int splits, const int* cuQ,
               const int* cuKV, int headsQ, int group, int runs, int blocksPerEntry, long long totalBlocks, int seqLenQ) {
  constexpr int kVec = D / 4, kGroups = kCombineThreads / kVec;
  __shared__ float4 sAcc[kGroups][kVec];
  __shared__ float sSum[kGroups];
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  int r = 0, nRows = 1;  // rows of this CTA: r, r + gridDim.x, ... (packed input), one (fixed length)
  long long row = blockIdx.x, qRow0 = 0;
  if (cuQ != nullptr) {
    const int b = blockIdx.z;
    if (cuKV[b + 1] <= cuKV[b]) return;  // no keys: leave O untouched
    qRow0 = cuQ[b];
    r = blockIdx.x;
    nRows = min((cuQ[b + 1] - cuQ[b]) * group, kRows);  // as in the split kernel
  } else if (runs > 0) {  // even partition: how many runs touch this row's batch entry
    const long long first = row / headsQ / seqLenQ * blocksPerEntry;
    splits = run_of_block(first + blocksPerEntry - 1, totalBlocks, runs) - run_of_block(first, totalBlocks, runs) + 1;
    if (splits == 1) return;  // the split kernel has written the output
  }
  for (; r < nRows; r += gridDim.x) {
    if (cuQ != nullptr) row = (qRow0 + r / group) * headsQ + blockIdx.y * group + r % group;
    float M = -INFINITY;
    for (int s = threadIdx.x & 31; s < splits; s += 32) M = fmax_nan(M, __ldcg(partLse + (long long)s * rows + row));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmax_nan(M, __shfl_xor_sync(0xffffffffu, M, off));
    if (M == -INFINITY) M = 0.f;  // no key with a score above -inf: all weights and the row are 0, as in the unsplit kernels
    const int g = threadIdx.x / kVec, c4 = threadIdx.x % kVec;
    if (g < kGroups) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float wsum = 0.f;
#pragma unroll 4
      for (int s = g; s < splits; s += kGroups) {
        const float lse = __ldcg(partLse + (long long)s * rows + row);
        const float4 v = __ldcg(reinterpret_cast<const float4*>(partO + ((long long)s * rows + row) * D + c4 * 4));
        const float w = exp2f(lse - M);  // 0 for a split without a score above -inf, whose partial is zero
        acc.x += w * v.x;
        acc.y += w * v.y;
        acc.z += w * v.z;
        acc.w += w * v.w;
        wsum += w;
      }
      sAcc[g][c4] = acc;
      if (c4 == 0) sSum[g] = wsum;
    }
    __syncthreads();
    if (threadIdx.x < kVec) {
      float4 acc = sAcc[0][threadIdx.x];
      float wsum = sSum[0];
#pragma unroll
      for (int i = 1; i < kGroups; i++) {
        const float4 v = sAcc[i][threadIdx.x];
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
        wsum += sSum[i];
      }
      const float inv = (wsum == 0.f) ? 0.f : (1.f / wsum);  // NaN stays NaN
      uint2 out;
      out.x = pack2<kBf16>(acc.x * inv, acc.y * inv);
      out.y = pack2<kBf16>(acc.z * inv, acc.w * inv);
      *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(O) + row * D + threadIdx.x * 4) = out;
    }
    if (r + (int)gridDim.x < nRows) __syncthreads();  // sAcc is written again
  }
}

// Partial results of the tensor-core kernel's key ranges (kModeFixedSplit), many rows and few ranges: D / 4 threads per
// row, several rows per CTA.
template <int D, bool kBf16>
__global__ void __launch_bounds__(kCombineThreads)
combine_parts_kernel(const float* partO, const float* partLse, void* O, long long rows, int partBlocks,
                     int seqLenQ, int seqLenKV, int headsQ, int causal, int rowsPerTile) {
  constexpr int kVec = D / 4, kGroups = kCombineThreads / kVec;
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  const int g = threadIdx.x / kVec, c4 = threadIdx.x % kVec;
  const long long row = (long long)blockIdx.x * kGroups + g;
  if (g >= kGroups || row >= rows) return;
  int blocks = (seqLenKV + 127) / 128;
  if (causal) {  // key blocks of this row's query tile, as in make_work
    const int tile = (int)(row / headsQ % seqLenQ) / rowsPerTile;
    blocks = min(blocks, (min((tile + 1) * rowsPerTile, seqLenQ) + 127) / 128);
  }
  const int parts = (blocks + partBlocks - 1) / partBlocks;
  if (parts == 1) return;  // the attention kernel has written the output
  float M = -INFINITY;
#pragma unroll 8
  for (int s = 0; s < parts; s++) M = fmax_nan(M, __ldcg(partLse + s * rows + row));
  if (M == -INFINITY) M = 0.f;  // no score above -inf: all weights and the row are 0, as in the unsplit kernel
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float wsum = 0.f;
#pragma unroll 4
  for (int s = 0; s < parts; s++) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(partO + (s * rows + row) * D + c4 * 4));
    const float w = exp2f(__ldcg(partLse + s * rows + row) - M);
    acc.x += w * v.x;
    acc.y += w * v.y;
    acc.z += w * v.z;
    acc.w += w * v.w;
    wsum += w;
  }
  const float inv = (wsum == 0.f) ? 0.f : (1.f / wsum);  // NaN stays NaN
  uint2 out;
  out.x = pack2<kBf16>(acc.x * inv, acc.y * inv);
  out.y = pack2<kBf16>(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(O) + row * D + c4 * 4) = out;
}

template <int D, bool kBf16>
int launch_combine(const FwdProblem& p, int packShift, const TcSplit& split) {
  constexpr int kGroups = kCombineThreads / (D / 4);
  const long long rows = p.totalQ * p.headsQ;
  cudaError_t e;
  if (!p.causal && (rows <= 1024 || (rows <= 3072 && split.parts >= 12))) {
    // Few rows: one CTA per row, whose threads read the ranges side by side (without the mask every tile has all ranges).  us a call
    // at head dim 128, the kernel below -> this one, with 3, 6, 12 ranges: 512 rows 15.4 -> 14.7, 16.8 -> 15.1, 17.7 -> 15.8; 1024 16.7 -> 16.2,
    // 17.9 -> 16.5, 19.2 -> 17.4; 3072 17.4 -> 18.8, 24.8 -> 23.7, 38.7 -> 37.6; 4096 and 4, 6, 8 ranges 22.7 -> 20.6, 24.3 -> 26.0, 24.1 ->
    // 26.6; 8192 25.9 -> 29.4, 44.0 -> 45.9, 46.6 -> 50.6.
    e = launch_kernel(combine_kernel<D, kBf16>, dim3((unsigned)rows), kCombineThreads, 0, p.stream, p.overlap, split.partO,
                      split.partLse, p.O, rows, split.parts, nullptr, nullptr, p.headsQ, 1, 0, 0, 0ll, p.seqLenQ);
  } else {
    e = launch_kernel(combine_parts_kernel<D, kBf16>, dim3((unsigned)((rows + kGroups - 1) / kGroups)), kCombineThreads, 0, p.stream,
                      p.overlap, split.partO, split.partLse, p.O, rows, split.partBlocks, p.seqLenQ, p.seqLenKV, p.headsQ, p.causal,
                      128 >> packShift);
  }
  if (e != cudaSuccess) {
    set_error_string("combine kernel launch failed: %s", cudaGetErrorString(e));
    return kCudaError;
  }
  return kOk;
}

constexpr int kMaxSmem = 227 * 1024, kSmemReserved = 1024, kSmemPerSm = 228 * 1024;  // of a CTA, taken by the system per CTA, of an SM
constexpr int ring_bytes(int D) { return kStages * 2 * kBlockKeys * D * 2; }
constexpr int merge_bytes(int D, int parts) { return (parts * kRows * (D + 8) + 8 * kRows) * (int)sizeof(float); }
// CTAs of the even partition, in quarters of an SM's share.  Not all that shared memory holds where it holds more than
// one: measured us at 8 KV heads, batch 4 / 8 / 28 of D = 128: 296 CTAs 93.2 / 110.6 / 114.4, 280 89.3 / 106.0 / 112.1, 256
// 86.8 / 102.6 / 108.3, 224 88.5 / 105.1 / 106.6, 148 107 / 125 / 137; D = 64, batch 4 / 24: 592 49.9 / 72.8, 444 46.8 / 66.8,
// 296 46.8 / 68.0; D = 32: 592 47.3, 444 50.4, 296 58.6; D = 96: 296 44.2, 256 44.5; D = 192 / 256 hold one per SM.
constexpr int quarter_ctas_per_sm(int D) { return D == 32 ? 16 : D == 64 ? 12 : D <= 128 ? 7 : 4; }

// CTAs of an SM without the even partition: the stated 8, registers up to head dim 96, shared memory above.
constexpr int whole_ctas_per_sm(int D) { return D == 32 ? 8 : D == 64 ? 4 : D == 96 ? 3 : D == 128 ? 2 : 1; }

template <int D, bool kBf16>
int launch(const FwdProblem& pr, const SplitPlan& plan, float* partO, float* partLse) {
  constexpr int kSmem = ring_bytes(D) + merge_bytes(D, 1);
  static_assert(kSmem <= kMaxSmem && merge_bytes(D, 4) <= ring_bytes(D) && merge_ld<D>() == D + 8, "shared memory");
  auto kernel = plan.runs > 0 ? fwd_splitkv_kernel<D, kBf16, true> : fwd_splitkv_kernel<D, kBf16, false>;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return kCudaError;
  static std::once_flag once[64];
  static cudaError_t attrErr[64];
  std::call_once(once[device], [&] {
    attrErr[device] = cudaFuncSetAttribute(fwd_splitkv_kernel<D, kBf16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (attrErr[device] == cudaSuccess) {
      attrErr[device] = cudaFuncSetAttribute(fwd_splitkv_kernel<D, kBf16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    }
    // all of it as shared memory: the spread below counts on it
    if (attrErr[device] == cudaSuccess) {
      attrErr[device] = cudaFuncSetAttribute(fwd_splitkv_kernel<D, kBf16, true>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    if (attrErr[device] == cudaSuccess) {
      attrErr[device] = cudaFuncSetAttribute(fwd_splitkv_kernel<D, kBf16, false>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
  });
  if (attrErr[device] != cudaSuccess) {
    set_error_string("cudaFuncSetAttribute(%d bytes): %s", kMaxSmem, cudaGetErrorString(attrErr[device]));
    return kCudaError;
  }
  const int numSMs = device_num_sms(device);
  Params p;
  p.Q = pr.Q;
  p.K = pr.K;
  p.V = pr.V;
  p.O = pr.O;
  p.partO = partO;
  p.partLse = partLse;
  p.cuQ = pr.cuQ;
  p.cuKV = pr.cuKV;
  p.seqLenQ = pr.seqLenQ;
  p.seqLenKV = pr.seqLenKV;
  p.headsQ = pr.headsQ;
  p.headsKV = pr.headsKV;
  p.group = pr.headsQ / pr.headsKV;
  p.causal = pr.causal;
  p.splits = plan.splits;
  p.runs = plan.runs;
  p.blocksPerEntry = plan.blocksPerEntry;
  p.totalBlocks = (long long)plan.blocksPerEntry * pr.batch;
  const int blocks = (pr.seqLenKV + kBlockKeys - 1) / kBlockKeys;
  p.keysPerSplit = ((blocks + plan.splits - 1) / plan.splits) * kBlockKeys;
  p.totalQ = pr.totalQ;
  p.scaleLog2 = (float)(1.4426950408889634 / sqrt((double)D));
  const dim3 grid = plan.runs > 0 ? dim3((unsigned)(plan.runs * pr.headsKV)) : dim3((unsigned)plan.splits, (unsigned)pr.headsKV, (unsigned)pr.batch);
  // head dim 96 fits three CTAs per SM without the merge buffer, two with it: packed, 223 x up to 5432 keys, 2 heads 138 -> 118 us
  size_t smem = plan.runs > 0 ? kSmem : ring_bytes(D);
  // A grid that fits the GPU at once must not crowd on part of the SMs: its CTAs come in while those of the kernel before leave, and would
  // fill up the SMs that are done first.  So shared memory holds no more CTAs of an SM than an even spread needs.  17 x 2 x 2513 keys, 64
  // heads over 32 of 32, whole pairs: 42.6 -> 31.3 us.  A grid of several waves does not start early at all (200 x 5360 keys, 16 heads of 32,
  // whole pairs: 417 -> 368 us).
  const long long perSm = ((long long)grid.x * grid.y * grid.z + numSMs - 1) / numSMs;
  const size_t share = (kSmemPerSm / (size_t)(perSm + 1) - kSmemReserved + 255) / 128 * 128;  // perSm + 1 CTAs of it do not fit
  if (smem < share) smem = share;
  const bool early = pr.overlap && perSm <= whole_ctas_per_sm(D);
  cudaError_t e = launch_kernel(kernel, grid, kThreads, smem, pr.stream, early, p);
  if (e == cudaSuccess && plan.splits > 1) {
    const long long rows = pr.totalQ * pr.headsQ;
    const int tileRows = pr.seqLenQ * p.group;  // a longer sequence than the caller's maximum: the CTAs take turns
    const dim3 combineGrid = pr.cuQ != nullptr ? dim3((unsigned)tileRows, (unsigned)pr.headsKV, (unsigned)pr.batch) : dim3((unsigned)rows);
    e = launch_kernel(combine_kernel<D, kBf16>, combineGrid, kCombineThreads, 0, pr.stream, pr.overlap, partO, partLse, pr.O, rows,
                      plan.splits, pr.cuQ, pr.cuKV, pr.headsQ, p.group, p.runs, p.blocksPerEntry, p.totalBlocks, pr.seqLenQ);
  }
  if (e != cudaSuccess) {
    set_error_string("split-KV kernel launch failed: %s", cudaGetErrorString(e));
    return kCudaError;
  }
  return kOk;
}

}  // namespace decode

bool splitkv_applicable(const FwdProblem& p) {
  if (p.dtype != kFp16 && p.dtype != kBf16) return false;
  if (!dtype_compiled(p.dtype) || !head_dim_compiled(p.headDim)) return false;  // left out at build time
  const int group = p.headsQ / p.headsKV;
  return (long long)p.seqLenQ * group <= decode::kRows && p.seqLenKV >= 256;
}

// Key-range splits of every (batch, KV head) pair: none from one wave of pairs on, otherwise as many as fit two waves of
// two CTAs per SM, at most 32, at least 256 keys each.
static int splits_of_pairs(const FwdProblem& p, int numSMs) {
  const long long pairs = (long long)p.batch * p.headsKV;
  if (pairs >= 2ll * numSMs) return 1;
  long long splits = 4ll * numSMs / pairs;
  if (splits > 32) splits = 32;
  if (splits > (p.seqLenKV + 255) / 256) splits = (p.seqLenKV + 255) / 256;
  return splits < 1 ? 1 : (int)splits;
}

// How a call is cut.  forced > 0: that many key-range splits of every pair, on a three-dimensional grid (-2: the even partition
// below wherever it is possible, whatever it costs); the same with a number of its own for packed input, whose lengths the host does not know.  Fixed-length input is cut evenly: the key
// blocks of all batch entries in a row, as many equal runs as the GPU holds at once, so that no SM waits for another at the
// end whatever the batch is.  All KV heads of a run are cut at the same keys: cut one by one, their CTAs drift apart and
// read the pieces of a row of K at different times, which cost up to half of the bandwidth (D = 32, 64-byte pieces).
SplitPlan splitkv_plan(const FwdProblem& p, int numSMs, int forced) {
  SplitPlan plan = {1, 0, 0};
  const long long pairs = (long long)p.batch * p.headsKV;
  const int maxSplits = (p.seqLenKV + decode::kBlockKeys - 1) / decode::kBlockKeys;
  if (forced > 0) {
    plan.splits = forced < maxSplits ? forced : maxSplits;
    return plan;
  }
  const int seen = p.causal ? (p.seqLenQ < p.seqLenKV ? p.seqLenQ : p.seqLenKV) : p.seqLenKV;
  const long long blocks = (seen + decode::kBlockKeys - 1) / decode::kBlockKeys;
  const long long slots = (long long)numSMs * decode::quarter_ctas_per_sm(p.headDim) / 4;
  if (p.cuQ == nullptr && blocks >= 4 && pairs < 8 * slots && p.headsKV <= slots) {
    const long long total = p.batch * blocks;
    long long runs = total / 4 > p.batch ? total / 4 : p.batch;  // a run has at least four blocks, an entry at least one run
    if (runs > slots / p.headsKV) runs = slots / p.headsKV;
    plan.runs = (int)runs;
    plan.blocksPerEntry = (int)blocks;
    const long long run = total / runs;  // the shortest run; partial results per pair:
    plan.splits = (int)(p.batch % runs == 0 ? 1 : runs % p.batch == 0 ? runs / p.batch : (blocks - 2) / run + 2);
    // Against whole pairs, one CTA each.  In us, a block of one CTA: 3.81e-5 D at the memory rate, 0.2 + 0.00415 D at least, and 0.0042 D
    // for each of the CTAs that share its SM; the combine kernel: 5, and 1e-4 + 1.13e-5 D a row.  Fitted to 791 drawn calls of 40 pairs and
    // more, all head dims: the pick is
    // within 0.8 % of the faster cut on average, on 250 others within 1.4 %.  us per call, runs against whole pairs: 59 x 2 x 442 keys, 128 heads over 16 of 32 30.7, 11.4;
    // 172 x 1 x 839, 64 over 4 of 32 31.1, 14.5; 398 x 16 x 519, 4 heads of 128 109, 83; on the other side 40 x 5000, 32 over 8 of 128
    // 128, 172; 5 x 13900, 32 heads of 128 169, 216.
    const double D = p.headDim, block = 3.81e-5 * D;
    auto step = [&](long long ctas) { return fmax(0.2 + 0.00415 * D, (double)((ctas + numSMs - 1) / numSMs) * 0.0042 * D); };
    const long long held = (long long)numSMs * decode::whole_ctas_per_sm(p.headDim), rest = pairs % held;
    const double whole = (double)(pairs / held) * blocks * held * block + (rest > 0 ? blocks * fmax(rest * block, step(rest)) : 0.0);
    const double cut = fmax((double)pairs * blocks * block, (double)((total + runs - 1) / runs) * step(runs * p.headsKV)) +
                       (plan.splits > 1 ? 5.0 + (double)p.totalQ * p.headsQ * (1e-4 + 1.13e-5 * D) : 0.0);
    // (the factor: without a combine pass both estimates are the bytes, and runs end more evenly than pairs)
    if (whole <= (plan.splits > 1 ? cut : 0.99 * cut) && forced != -2) return SplitPlan{1, 0, 0};
    return plan;
  }
  plan.splits = splits_of_pairs(p, numSMs);  // packed input, and more pairs than the even partition is for
  // causal calls see few keys: 5 x 3 x 556, 64 heads over 32 of 256 24.7 us in three splits, 12.4 whole
  if (p.cuQ == nullptr && plan.splits > (seen + 255) / 256) plan.splits = (seen + 255) / 256;
  return plan;
}

size_t splitkv_scratch_floats(const FwdProblem& p, const SplitPlan& plan) {
  if (plan.splits <= 1) return 0;
  const size_t rows = (size_t)p.totalQ * p.headsQ;
  return (size_t)plan.splits * rows * (p.headDim + 1);
}

int launch_combine_parts(const FwdProblem& p, int packShift, const TcSplit& split) {
  const bool bf = (p.dtype == kBf16);
#define TFA_COMBINE_CASE(D)                                                                    \
  case D:                                                                                      \
    if (bf) {                                                                                  \
      if constexpr (TFA_HAVE_BF16) return decode::launch_combine<D, true>(p, packShift, split);  \
    } else {                                                                                   \
      if constexpr (TFA_HAVE_FP16) return decode::launch_combine<D, false>(p, packShift, split); \
    }                                                                                          \
    return kBadDtype;
  (void)bf;
  (void)packShift;
  (void)split;
  switch (p.headDim) {
#if TFA_HAVE_HD32
    TFA_COMBINE_CASE(32)
#endif
#if TFA_HAVE_HD64
    TFA_COMBINE_CASE(64)
#endif
#if TFA_HAVE_HD96
    TFA_COMBINE_CASE(96)
#endif
#if TFA_HAVE_HD128
    TFA_COMBINE_CASE(128)
#endif
#if TFA_HAVE_HD192
    TFA_COMBINE_CASE(192)
#endif
#if TFA_HAVE_HD256
    TFA_COMBINE_CASE(256)
#endif
    default:
      return kBadHeadDim;
  }
#undef TFA_COMBINE_CASE
}

// partO = scratch, partLse = scratch + splits*rows*D
int launch_fwd_splitkv(const FwdProblem& p, const SplitPlan& plan, float* scratch) {
  const size_t rows = (size_t)p.totalQ * p.headsQ;
  float* partO = scratch;
  float* partLse = scratch ? scratch + (size_t)plan.splits * rows * p.headDim : nullptr;
  const bool bf = (p.dtype == kBf16);
#define TFA_DECODE_CASE(D)                                                                   \
  case D:                                                                                    \
    if (bf) {                                                                                \
      if constexpr (TFA_HAVE_BF16) return decode::launch<D, true>(p, plan, partO, partLse);  \
    } else {                                                                                 \
      if constexpr (TFA_HAVE_FP16) return decode::launch<D, false>(p, plan, partO, partLse); \
    }                                                                                        \
    return kBadDtype;
  (void)bf; (void)partO; (void)partLse;
  switch (p.headDim) {
#if TFA_HAVE_HD32
    TFA_DECODE_CASE(32)
#endif
#if TFA_HAVE_HD64
    TFA_DECODE_CASE(64)
#endif
#if TFA_HAVE_HD96
    TFA_DECODE_CASE(96)
#endif
#if TFA_HAVE_HD128
    TFA_DECODE_CASE(128)
#endif
#if TFA_HAVE_HD192
    TFA_DECODE_CASE(192)
#endif
#if TFA_HAVE_HD256
    TFA_DECODE_CASE(256)
#endif
    default:
      return kBadHeadDim;
  }
#undef TFA_DECODE_CASE
}

}  // namespace tfa_b200

// ---------------------------------------------------------------------------------------------------------------
// Allocation-free variant of the split-KV path.
//
// Who needs it: serving processes that give all device memory to their own planner at start-up (a fixed KV-cache
// budget, nothing left for the driver to hand out later) and latency-critical decode loops in which a driver
// allocation may stall or fail.  For them the fp32 partial results of the key-range splits live in the fixed array
// below instead of a stream-ordered allocation.  The price: every GPU that loads this library carries the array
// (TFA_B200_NOALLOC_SCRATCH_FLOATS floats) until the process exits, and all calls share it.
namespace tfa_b200 {
namespace decode {

static __device__ __align__(256) float g_static_scratch[TFA_B200_NOALLOC_SCRATCH_FLOATS];

// Device address of g_static_scratch on the current device.  In host code the symbol's name is only a handle, not
// a device pointer, so the address is fetched once per device with cudaGetSymbolAddress (that device current).
static int static_scratch_ptr(float** out) {
  static std::mutex mutex;
  static float* cached[64] = {nullptr};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess || device < 0 || device >= 64) {
    set_error_string("cudaGetDevice: %s", cudaGetErrorString(e));
    return kCudaError;
  }
  std::lock_guard<std::mutex> lock(mutex);
  if (cached[device] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error_string("cudaGetSymbolAddress(static split-KV scratch) on device %d: %s", device, cudaGetErrorString(e));
      return kCudaError;
    }
    cached[device] = static_cast<float*>(p);
  }
  *out = cached[device];
  return kOk;
}

}  // namespace decode
}  // namespace tfa_b200

extern "C" int tfa_b200_fwd_decode_noalloc(const void* Q, const void* K, const void* V, void* O, int dtype,
                                           int batchSize, int seqLenQ, int seqLenKV, int numHeadsQ, int numHeadsKV,
                                           int headDim, int isCausal, int numSplits, void* stream) {
  using namespace tfa_b200;
  int rc = validate_common(Q, K, V, O, dtype, batchSize, seqLenQ, seqLenKV, numHeadsQ, numHeadsKV, headDim);
  if (rc != kOk) return rc;
  if (batchSize == 0 || seqLenQ == 0 || seqLenKV == 0) return kOk;
  if ((rc = check_device()) != kOk) return rc;
  FwdProblem p;
  p.Q = Q;
  p.K = K;
  p.V = V;
  p.O = O;
  p.cuQ = nullptr;
  p.cuKV = nullptr;
  p.dtype = dtype;
  p.batch = batchSize;
  p.seqLenQ = seqLenQ;
  p.seqLenKV = seqLenKV;
  p.totalQ = (long long)batchSize * seqLenQ;
  p.totalKV = (long long)batchSize * seqLenKV;
  p.headsQ = numHeadsQ;
  p.headsKV = numHeadsKV;
  p.headDim = headDim;
  p.causal = isCausal ? 1 : 0;
  p.stream = static_cast<cudaStream_t>(stream);
  p.overlap = may_overlap(p.stream);
  if (!splitkv_applicable(p)) {
    set_error_string("tfa_b200_fwd_decode_noalloc handles fp16/bf16, seqLenQ * (Hq/Hkv) <= 16 and "
                     "seqLenKV >= 256 only (got dtype %d, headDim %d, seqLenQ %d, group %d, seqLenKV %d)",
                     dtype, headDim, seqLenQ, numHeadsQ / numHeadsKV, seqLenKV);
    return kBadArgument;
  }
  int device = 0, sms = 148;
  if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  SplitPlan plan = splitkv_plan(p, sms, numSplits > 0 ? numSplits : 0);
  // What the entry point accepts is stated in splits of pairs; an even partition whose partials do not fit the array gives
  // way to whole pairs, as many at a time as the GPU holds.
  const SplitPlan stated = {numSplits > 0 ? plan.splits : splits_of_pairs(p, sms), 0, 0};
  const size_t limit = (size_t)TFA_B200_NOALLOC_SCRATCH_FLOATS, statedNeed = splitkv_scratch_floats(p, stated);
  if (statedNeed > limit) {
    set_error_string("split-KV partials need %zu floats (%d splits x %lld rows x (%d + 1)) but the built-in scratch holds "
                     "%zu; use fewer splits or tfa_b200_fwd",
                     statedNeed, stated.splits, (long long)p.totalQ * numHeadsQ, headDim, limit);
    return kTooLarge;
  }
  if (splitkv_scratch_floats(p, plan) > limit) plan = SplitPlan{1, 0, 0};
  const size_t need = splitkv_scratch_floats(p, plan);
  float* scratch = nullptr;
  if ((rc = decode::static_scratch_ptr(&scratch)) != kOk) return rc;
  // Every (split, row) partial that the combine kernel reads is written by the split kernel of the same call, so
  // nothing in the array has to start at zero and contents left by an earlier call are never consumed.
  return launch_fwd_splitkv(p, plan, need > 0 ? scratch : nullptr);
}
