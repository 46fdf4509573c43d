// FP32 attention forward on the tensor cores of sm_100a, at the precision of 32-bit arithmetic.
//
// A float's 24-bit significand is cut into three bf16 numbers of 8 bits each, x = x0 + x1 + x2, which is exact for
// 2^-100 <= |x| < 2^60.  A product of two floats is then nine bf16 products, all exact in the tensor core's fp32
// accumulator; the three below 2^-24 of the leading one (x1 y2, x2 y1, x2 y2) are left out and six are issued, the
// small ones first, so that only the last of the six passes adds to an accumulator of full magnitude.  Everything
// around the two products stays what it is in the CUDA-core kernels of fwd_fp32.cu: fp32 scores, exact running
// maximum, ex2.approx, fp32 row sums, P as all 24 bits (three bf16 parts), and O summed in fp32 registers with round to
// nearest - the tensor core only ever sums the 128 keys of one block.
//
// Measured against the CUDA-core kernels (2-norm error against 64 bits in brackets): non-causal B2 S2048 H16 D128 1596 ->
// 394 us (9.1e-7 -> 3.1e-7), causal B2 S1999 16 over 4 heads D64 563 -> 127 us (3.9e-7 -> 1.8e-7).  Over ten distributions
// (zero-mean, one-sign and offset Q, K and V, large and nearly equal scores) x twelve shapes the error is 0.12 to 1.01 of that of the
// CUDA-core kernels, whose sums run over all keys one at a time; the largest is the accumulator's bias where all values of V are
// positive and the keys are one block (1.78e-7 against 1.77e-7).
// One pass over a block takes 7.7 k clocks at D = 128, of which the tensor pipe needs 96 x 64 = 6.1 k; with both products
// issued by one thread it was 9.4 k.  Left: the dependency S -> softmax -> P.V -> S two blocks on (the two S buffers), the
// last wave of tiles, and 40 us for the split at that shape (6.2 TB/s).
//
// Two kernels.  split_kernel writes the three parts of Q, K and V to a workspace (6 bytes per element) and notes
// whether any value is outside the exact range (NaN, infinity, huge or denormal-like values; zero is fine).  If one is,
// fwd_kernel returns at once and the CUDA-core kernel, which is launched behind it with the same condition the other way
// round, computes the call: results for such inputs are those of the CUDA-core kernel to the last bit.
//
// fwd_kernel, one CTA of 12 warps per 128-row query tile, one CTA per SM:
//   warps 0, 2   issue the TMA loads: Q (three tiles) and the parts of K; the parts of V.  Each has a ring of its own,
//                filled in order of use
//   warps 1, 3   issue the tcgen05.mma of Q.K^T and of P.V (one thread each)
//   warps 4-7    softmax, one thread per query row: S from tensor memory, P as three parts back into it
//   warps 8-11   output: adds every block's P.V to its row in registers, divides and stores
// Tensor memory: S of block j at columns (j & 1) * 128; the first two parts of P overwrite it, the third sits at
// 256 + (j & 1) * 64; P.V of the block at 384.  Q.K^T of block j + 1 and P.V of block j run at the same time: the tensor pipe
// alternates between the two issuing threads, so what one of them loses to a wait, a commit or a loop is filled by the
// other's MMAs.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <mutex>

#include "build_config.cuh"
#include "fwd_tc.cuh"
#include "tfa_common.cuh"

namespace tfa_b200 {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();     // c_abi.cu
int* device_status_word(int device);  // c_abi.cu
int device_num_sms(int device);       // c_abi.cu

namespace fp32tc {

using tc::kBlockM;
using tc::kBlockN;
using tc::kSubTileBytes;

constexpr int kThreads = 384;
constexpr int kSplitThreads = 256;
constexpr int kRegsIssue = 56, kRegsSoftmax = 208, kRegsOut = 240;
// the sum over the three warpgroups must fit the launch allocation (65536 / 384 = 168 registers a thread)
static_assert(kRegsIssue + kRegsSoftmax + kRegsOut <= 3 * ((65536 / kThreads) / 8 * 8), "register budget");

// ---------------------------------------------------------------------------------------------------- split
struct SplitParams {
  const float* src[3];  // Q, K, V
  uint16_t* dst[3];     // three parts each, count[i] elements apart
  long long count[3];   // elements, multiples of 8
  int width[3];         // elements of a row that are taken ...
  int pitch[3];         // ... and of a row in memory
  const int* cu[3];     // packed input: row ranges of the sequences, else null
  int batches;
  int* flag;            // set to epoch when a value is outside the exact range
  int epoch;
};

// x = p0 + p1 + p2 for two values at once, each part packed as bf16x2 (first value in the low half)
__device__ __forceinline__ void split3(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = tc::pack2<true>(a, b);
  const float a1 = a - __uint_as_float(p0 << 16), b1 = b - __uint_as_float(p0 & 0xffff0000u);
  p1 = tc::pack2<true>(a1, b1);
  p2 = tc::pack2<true>(a1 - __uint_as_float(p1 << 16), b1 - __uint_as_float(p1 & 0xffff0000u));
}

__device__ __forceinline__ bool outside(float x) {
  const float a = fabsf(x);
  return !(a < 0x1p60f) || (a < 0x1p-100f && a != 0.f);
}

// Bound by memory: 4 bytes read and 6 written per element.  Eight elements per thread and step.
__global__ void __launch_bounds__(kSplitThreads) split_kernel(const SplitParams p) {
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  bool bad = false;
#pragma unroll
  for (int t = 0; t < 3; t++) {
    const long long n8 = p.count[t] >> 3;
    const int w8 = p.width[t] >> 3, gap8 = (p.pitch[t] - p.width[t]) >> 3;
    const float4* src = reinterpret_cast<const float4*>(p.src[t]);
    uint4* d0 = reinterpret_cast<uint4*>(p.dst[t]);
    uint4* d1 = reinterpret_cast<uint4*>(p.dst[t] + p.count[t]);
    uint4* d2 = reinterpret_cast<uint4*>(p.dst[t] + 2 * p.count[t]);
    long long first = 0, end = n8;
    if (p.cu[t] != nullptr) {  // rows of no sequence: zeros in their place, whatever they hold
      first = (long long)p.cu[t][0] * w8;
      end = (long long)p.cu[t][p.batches] * w8;
    }
    for (long long i = (long long)blockIdx.x * kSplitThreads + threadIdx.x; i < n8; i += (long long)gridDim.x * kSplitThreads) {
      const long long at = gap8 == 0 ? i : i + i / w8 * gap8;
      float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
      if (i >= first && i < end) {
        u = src[2 * at];
        v = src[2 * at + 1];
      }
      uint4 a, b, c;
      split3(u.x, u.y, a.x, b.x, c.x);
      split3(u.z, u.w, a.y, b.y, c.y);
      split3(v.x, v.y, a.z, b.z, c.z);
      split3(v.z, v.w, a.w, b.w, c.w);
      d0[i] = a;
      d1[i] = b;
      d2[i] = c;
      bad |= outside(u.x) | outside(u.y) | outside(u.z) | outside(u.w) | outside(v.x) | outside(v.y) | outside(v.z) | outside(v.w);
    }
  }
  if (bad) *reinterpret_cast<volatile int*>(p.flag) = p.epoch;
}

// ---------------------------------------------------------------------------------------------------- attention
template <int HDP>
struct Cfg {
  static constexpr int kSub = HDP / 64;
  static constexpr int kTileBytes = kSub * kSubTileBytes;  // one part of a 128-row tile
  static constexpr int kStages = (HDP == 128) ? 2 : 4;  // of each ring
  static constexpr int kSmemBytes = 3 * kTileBytes + 2 * kStages * kTileBytes + 3072 /*barriers, scales*/;
};

enum Bar : int {
  kBarQFull = 0,
  kBarSFull = 1,      // [2] S of block j finished
  kBarPReady = 3,     // [2] P of block j written (4 warps)
  kBarScaleFull = 5,  // [4] rescale factors of block j published (4 warps)
  kBarOFull = 9,      // [2] P.V of block j finished: O may be read, P's columns may be overwritten
  kBarOFree = 11,     // O of a block read by the output warps (4 warps)
  kBarSumFull = 12,   // final row sums published (4 warps)
  kBarKvFull = 13,    // [2 rings][kStages <= 4]
  kBarKvEmpty = 21,   // [2 rings][kStages <= 4]
  kNumBars = 29,
};

struct Ctl {
  uint64_t bars[kNumBars];
  float scale[4][kBlockM];  // four slots: the softmax is at most two blocks ahead of the output warps
  float sum[kBlockM];
  uint32_t tmemBase;
  int failed;
};
static_assert(sizeof(Ctl) <= 3072, "control block");

struct Params {
  TcParams w;        // work description (make_work), output, mask, scale, status word
  int batches;       // batch entries of the tensor maps (1 for packed input): part i of entry b is entry i * batches + b
  const int* flag;   // inputs outside the exact range: leave the call to the CUDA-core kernel
  // Key ranges (fixed-length input with few tiles): blockIdx.y is the range, partBlocks key blocks of the tile.  Partial
  // results of a tile with more than one: O, row maximum, row sum relative to it.
  int partBlocks;
  long long rows;  // batch * seqLenQ * headsQ
  float* partO;    // [ranges][rows][headDim]
  float* partM;    // [ranges][rows]
  float* partL;    // [ranges][rows]
};

template <int HDP, int kHD, bool kVarlen>
__global__ void __launch_bounds__(kThreads, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
           const __grid_constant__ CUtensorMap tmV, const Params p) {
  using C = Cfg<HDP>;
  constexpr int NS = C::kStages;
  if constexpr (kVarlen) ptx::grid_wait_previous();  // the lengths are in global memory
  tc::Work w;
  if (!tc::make_work<1, kVarlen>(p.w, (int)blockIdx.x, w)) return;
  int n = w.nblk[0], j0 = 0;  // key blocks of this CTA and the first of them
  bool whole = true;
  if constexpr (!kVarlen) {
    whole = n <= p.partBlocks;
    j0 = (int)blockIdx.y * p.partBlocks;
    n = min(n - j0, p.partBlocks);
    // causal: a range past the end of an early tile.  Waiting first keeps this grid's end behind the end of the one before.
    if (n <= 0) {
      ptx::grid_wait_previous();
      return;
    }
  }

  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sQ = ptx::smem_u32(smem);
  const uint32_t sKV = sQ + 3 * C::kTileBytes;
  if ((sQ & 1023u) != 0) {  // swizzled tiles need 1024-byte alignment; the launcher leaves no room to make up for it
    if (threadIdx.x == 0) atomicExch(p.w.status, (p.w.epoch << 8) | 50);
    return;
  }
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + (3 + 2 * NS) * C::kTileBytes);
  const uint32_t barBase = ptx::smem_u32(&ctl->bars[0]);
  auto bar = [&](int slot) { return barBase + 8u * (uint32_t)slot; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    ptx::mbar_init(bar(kBarQFull), 1);
    for (int i = 0; i < 2; i++) {
      ptx::mbar_init(bar(kBarSFull + i), 1);
      ptx::mbar_init(bar(kBarPReady + i), 4);
      ptx::mbar_init(bar(kBarOFull + i), 1);
    }
    for (int i = 0; i < 4; i++) ptx::mbar_init(bar(kBarScaleFull + i), 4);
    ptx::mbar_init(bar(kBarOFree), 4);
    ptx::mbar_init(bar(kBarSumFull), 4);
    for (int s = 0; s < 8; s++) {
      ptx::mbar_init(bar(kBarKvFull + s), 1);
      ptx::mbar_init(bar(kBarKvEmpty + s), 1);
    }
    ctl->failed = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmemBase), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmemBase;
  const tc::WaitCtx wc{&ctl->failed, p.w.status, p.w.epoch};
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  const bool skip = (*p.flag == p.w.epoch);  // left to the CUDA-core kernel
  constexpr uint32_t kPLoCol = 256, kOCol = 384;

  if (skip) {
    // straight to the end
  } else if (warp < 4) {
    ptx::setmaxnreg_dec<kRegsIssue>();
    const bool isV = warp >= 2;  // which of the two streams
    const uint32_t ring = sKV + (isV ? NS * C::kTileBytes : 0u);
    const int full = kBarKvFull + (isV ? 4 : 0), empty = kBarKvEmpty + (isV ? 4 : 0);
    if ((warp & 1) == 0 && lane == 0) {
      // ============================================================== TMA loads
      if (!isV) {
        const int gp = 1 << p.w.packShift;
        ptx::mbar_arrive_expect_tx(bar(kBarQFull), 3 * C::kTileBytes);
#pragma unroll
        for (int part = 0; part < 3; part++) {
#pragma unroll
          for (int a = 0; a < C::kSub; a++) {
            ptx::tma_load_4d(sQ + part * C::kTileBytes + a * kSubTileBytes, &tmQ, bar(kBarQFull), a * 64, w.unit * gp,
                             w.qRowTma + w.qlo[0], part * p.batches + w.batchTma);
          }
        }
      }
      const CUtensorMap* tm = isV ? &tmV : &tmK;
      int ld = 0;
      for (int j = 0; j < n; j++) {
        for (int part = 2; part >= 0; part--, ld++) {  // smallest part first
          const int s = ld % NS;
          if (ld >= NS) tc::wait_bar(bar(empty + s), ((ld / NS) - 1) & 1, wc, 41);
          ptx::mbar_arrive_expect_tx(bar(full + s), C::kTileBytes);
#pragma unroll
          for (int a = 0; a < C::kSub; a++) {
            ptx::tma_load_4d(ring + s * C::kTileBytes + a * kSubTileBytes, tm, bar(full + s), a * 64, w.hkv,
                             w.kvRowTma + (j0 + j) * kBlockN, part * p.batches + w.batchTma);
          }
        }
      }
    } else if (lane == 0) {
      // ============================================================== MMA issue
      // Six passes per product and block: part i of K (V), smallest first, against the parts 0 .. 2 - i of Q (P), smallest
      // first.  Loops stay loops down to one pass of 8 MMAs: with all 48 in a line, executed by one thread once per block,
      // an MMA took ~100 clocks instead of 64 (instruction fetch).
      const uint64_t descK = ptx::smem_desc_sw128(16, 1024);
      const uint64_t descV = ptx::smem_desc_sw128(kSubTileBytes, 1024);
      const uint32_t kHi = (uint32_t)(descK >> 32), vHi = (uint32_t)(descV >> 32);
      const uint32_t kLoT = (uint32_t)descK, vLoT = (uint32_t)descV;
      int ld = 0;
      auto stageReady = [&]() -> int {
        const int s = ld % NS;
        tc::wait_bar(bar(full + s), (ld / NS) & 1, wc, 42);
        ptx::tc_fence_after();
        ld++;
        return s;
      };
      if (!isV) {
        const uint32_t idQK = ptx::instr_desc_f16(1, kBlockM, kBlockN, 0, 0);
        tc::wait_bar(bar(kBarQFull), 0, wc, 43);
        for (int j = 0; j < n; j++) {
          // the columns of this S hold P of block j - 2 (its S has been read: P.V of that block waited for its P).  One
          // barrier per parity: P.V of block j - 1 may be done as well by now, P.V of block j cannot
          if (j >= 2) tc::wait_bar(bar(kBarOFull + (j & 1)), ((j >> 1) - 1) & 1, wc, 44);
          const uint32_t dS = tmem + (uint32_t)((j & 1) * 128);
          uint32_t acc = 0;
#pragma unroll 1
          for (int part = 2; part >= 0; part--) {
            const int s = stageReady();
            const uint32_t kLo = kLoT | ((ring + (uint32_t)(s * C::kTileBytes)) >> 4);
#pragma unroll 1
            for (int qPart = 2 - part; qPart >= 0; qPart--) {
              const uint32_t qLo = kLoT | ((sQ + (uint32_t)(qPart * C::kTileBytes)) >> 4);
#pragma unroll
              for (int kk = 0; kk < kHD / 16; kk++) {
                const uint32_t off = (uint32_t)((kk >> 2) * kSubTileBytes + (kk & 3) * 32) >> 4;
                ptx::mma_ss_lohi(dS, qLo + off, kHi, kLo + off, kHi, idQK, kk > 0 ? 1u : acc);
              }
              acc = 1;
            }
            ptx::tc_commit(bar(empty + s));
          }
          ptx::tc_commit(bar(kBarSFull + (j & 1)));
        }
      } else {
        const uint32_t idPV = ptx::instr_desc_f16(1, kBlockM, kHD, 0, 1);
        const uint32_t dO = tmem + kOCol;
        for (int j = 0; j < n; j++) {
          const uint32_t aP = tmem + (uint32_t)((j & 1) * 128), aP2 = tmem + kPLoCol + (uint32_t)((j & 1) * 64);
          if (j > 0) tc::wait_bar(bar(kBarOFree), (j - 1) & 1, wc, 51);
          tc::wait_bar(bar(kBarPReady + (j & 1)), (j >> 1) & 1, wc, 45);
          uint32_t acc = 0;
#pragma unroll 1
          for (int part = 2; part >= 0; part--) {
            const int s = stageReady();
            const uint32_t vLo = vLoT | ((ring + (uint32_t)(s * C::kTileBytes)) >> 4);
#pragma unroll 1
            for (int pPart = 2 - part; pPart >= 0; pPart--) {
              const uint32_t a = pPart == 2 ? aP2 : aP + (uint32_t)(pPart * 64);
#pragma unroll
              for (int kk = 0; kk < kBlockN / 16; kk++) {
                ptx::mma_ts_lohi(dO, a + kk * 8, vLo + ((kk * 2048) >> 4), vHi, idPV, kk > 0 ? 1u : acc);
              }
              acc = 1;
            }
            ptx::tc_commit(bar(empty + s));
          }
          ptx::tc_commit(bar(kBarOFull + (j & 1)));
        }
      }
    }
  } else if (warp < 8) {
    // ================================================================ softmax
    ptx::setmaxnreg_inc<kRegsSoftmax>();
    const int r = threadIdx.x & 127;
    const uint32_t laneOff = (uint32_t)((warp & 3) * 32) << 16;
    const int qpos = w.qlo[0] + (r >> p.w.packShift);
    const float c = p.w.scaleLog2;
    float m = -INFINITY, l = 0.f;
    for (int j = 0; j < n; j++) {
      tc::wait_bar(bar(kBarSFull + (j & 1)), (j >> 1) & 1, wc, 46);
      ptx::tc_fence_after();
      const uint32_t tS = tmem + laneOff + (uint32_t)((j & 1) * 128);
      uint32_t v[4][32];
#pragma unroll
      for (int q = 0; q < 4; q++) ptx::tmem_ld_32x32b_x32(tS + q * 32, v[q]);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 4; q++) ptx::tmem_ld_fence(v[q]);
      const int kbase = (j0 + j) * kBlockN;
      if ((kbase + kBlockN > w.skv) || (p.w.causal && (kbase + kBlockN - 1 > w.qlo[0]))) {
        int lim = w.skv - kbase;
        if (p.w.causal) lim = min(lim, qpos - kbase + 1);
#pragma unroll
        for (int q = 0; q < 4; q++) {
#pragma unroll
          for (int i = 0; i < 32; i++) {
            if (q * 32 + i >= lim) v[q][i] = 0xff800000u;  // -inf
          }
        }
      }
      float mx4[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        mx4[q] = tc::fmax2(__uint_as_float(v[q][0]), __uint_as_float(v[q][1]));
#pragma unroll
        for (int i = 2; i < 32; i += 2) mx4[q] = tc::fmax3(mx4[q], __uint_as_float(v[q][i]), __uint_as_float(v[q][i + 1]));
      }
      const float mNew = fmaxf(m, tc::fmax2(tc::fmax2(mx4[0], mx4[1]), tc::fmax2(mx4[2], mx4[3])));
      const float mUse = (mNew == -INFINITY) ? 0.f : mNew;
      const float scale = (m == -INFINITY) ? 0.f : tc::ex2((m - mUse) * c);
      m = mNew;
      ctl->scale[j & 3][r] = scale;
      const float negMc = -mUse * c;
      const float2 c2 = make_float2(c, c), negMc2 = make_float2(negMc, negMc);
      const uint32_t tLo = tmem + laneOff + kPLoCol + (uint32_t)((j & 1) * 64);
      float2 sum2[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        uint32_t p0[16], p1[16], p2[16];
        sum2[q] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float2 x = tc::ffma2(make_float2(__uint_as_float(v[q][i]), __uint_as_float(v[q][i + 1])), c2, negMc2);
          x.x = tc::ex2(x.x);
          x.y = tc::ex2(x.y);
          sum2[q] = tc::fadd2(sum2[q], x);
          split3(x.x, x.y, p0[i >> 1], p1[i >> 1], p2[i >> 1]);
        }
        ptx::tmem_st_32x32b_x16(tS + q * 16, p0);
        ptx::tmem_st_32x32b_x16(tS + 64 + q * 16, p1);
        ptx::tmem_st_32x32b_x16(tLo + q * 16, p2);
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(bar(kBarPReady + (j & 1)));
        ptx::mbar_arrive(bar(kBarScaleFull + (j & 3)));
      }
      const float2 s2 = tc::fadd2(tc::fadd2(sum2[0], sum2[1]), tc::fadd2(sum2[2], sum2[3]));
      l = l * scale + (s2.x + s2.y);
    }
    ctl->sum[r] = l;
    if (!whole && qpos < w.sq) {
      const long long row = blockIdx.y * p.rows + (w.qRow0 + qpos) * p.w.headsQ + (w.unit << p.w.packShift) + (r & ((1 << p.w.packShift) - 1));
      p.partM[row] = m;
      p.partL[row] = l;
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(bar(kBarSumFull));
  } else {
    // ================================================================ output
    ptx::setmaxnreg_inc<kRegsOut>();
    const int r = threadIdx.x & 127;
    const uint32_t tO = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kOCol;
    float2 o[kHD / 2];
#pragma unroll
    for (int i = 0; i < kHD / 2; i++) o[i] = make_float2(0.f, 0.f);
    for (int j = 0; j < n; j++) {
      // Slot j & 3 is published again for block j + 4, whose scores need P.V of block j + 2 and with it this warp's arrival
      // on kBarOFree for block j + 1: it is never two phases behind.
      tc::wait_bar(bar(kBarScaleFull + (j & 3)), (j >> 2) & 1, wc, 47);
      const float scale = ctl->scale[j & 3][r];
      const float2 scale2 = make_float2(scale, scale);
      tc::wait_bar(bar(kBarOFull + (j & 1)), (j >> 1) & 1, wc, 48);
      ptx::tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < kHD / 32; ch++) {
        uint32_t t[32];
        ptx::tmem_ld_32x32b_x32(tO + ch * 32, t);
        ptx::tmem_wait_ld();
        ptx::tmem_ld_fence(t);
        if (ch == kHD / 32 - 1) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar(kBarOFree));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          o[ch * 16 + (i >> 1)] = tc::ffma2(o[ch * 16 + (i >> 1)], scale2, make_float2(__uint_as_float(t[i]), __uint_as_float(t[i + 1])));
        }
      }
    }
    tc::wait_bar(bar(kBarSumFull), 0, wc, 49);
    const float l = ctl->sum[r];
    const float inv = !whole ? 1.f : (l > 0.f) ? (1.f / l) : 0.f;
    const int qpos = w.qlo[0] + (r >> p.w.packShift);
    const int head = (w.unit << p.w.packShift) + (r & ((1 << p.w.packShift) - 1));
    if (qpos < w.sq) {
      const long long row = (w.qRow0 + qpos) * p.w.headsQ + head;
      float4* dst = reinterpret_cast<float4*>(whole ? reinterpret_cast<float*>(p.w.O) + row * kHD : p.partO + (blockIdx.y * p.rows + row) * kHD);
#pragma unroll
      for (int i = 0; i < kHD / 4; i++) {
        dst[i] = make_float4(o[2 * i].x * inv, o[2 * i].y * inv, o[2 * i + 1].x * inv, o[2 * i + 1].y * inv);
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*wc.failed) __nanosleep(200000);  // a wait gave up: let whatever is still in flight drain before freeing
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// ---------------------------------------------------------------------------------------------------- head dims 192, 256
// The same computation where three parts of a Q tile (192 KB at 256) leave no room for K and V: parts 0 and 1 of Q stay in
// shared memory, part 2 passes through the ring once per key block, and the ring holds units of 128 rows x 128 head-dim
// elements (the second unit of head dim 192 is half as wide).  Each unit's share of S has an accumulator of its own, [0, 128)
// and [128, 256) of tensor memory: the tensor core cuts off what it adds below the accumulator's last bit, and one
// accumulator for all of the head dim was further off 64 bits than the CUDA cores (8.5e-7 against 5.1e-7 at S128 D256).
// The softmax first writes the sum (rounded to nearest, masked) over the first share, then reads it again for the
// exponentials - 128 scores do not fit beside two output warpgroups' registers - and leaves part 0 of P over the scores
// already read and parts 1 and 2 over the second share; P.V is at 256.  With one S position the two products and the
// softmax of a block follow one another, so one thread issues all MMAs.  16 warps: 0 loads, 1 issues, 4-7 softmax, 8-11
// and 12-15 output columns [0, 128) and [128, head dim).  A block moves 14 units of 32 KB from L2 for 12.3 k clocks of MMAs.
// Measured against the CUDA-core kernels at B2 S2048 H16 (2-norm error against 64 bits): D256 3670 -> 925 us (9.9e-7 -> 3.2e-7),
// causal D192 1599 -> 475 us (4.0e-7 -> 1.8e-7).
template <int kHD>
struct CfgWide {
  static constexpr int kSub = kHD / 64;
  static constexpr int kUnitBytes = 2 * kSubTileBytes;
  static constexpr int kQBytes = 2 * kSub * kSubTileBytes;  // parts 0 and 1
  static constexpr int kStages = kHD == 256 ? 3 : 4;
  static constexpr int kSmemBytes = kQBytes + kStages * kUnitBytes + 3072;
};
constexpr int kThreadsWide = 512;
constexpr int kRegsIssueW = 64, kRegsSoftmaxW = 96, kRegsOutW = 176;
static_assert(kRegsIssueW + kRegsSoftmaxW + 2 * kRegsOutW <= 4 * ((65536 / kThreadsWide) / 8 * 8), "register budget");

template <int kHD, bool kVarlen>
__global__ void __launch_bounds__(kThreadsWide, 1)
fwd_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const Params p) {
  using C = CfgWide<kHD>;
  constexpr int NS = C::kStages;
  if constexpr (kVarlen) ptx::grid_wait_previous();  // the lengths are in global memory
  tc::Work w;
  if (!tc::make_work<1, kVarlen>(p.w, (int)blockIdx.x, w)) return;
  int n = w.nblk[0], j0 = 0;  // key blocks of this CTA and the first of them
  bool whole = true;
  if constexpr (!kVarlen) {
    whole = n <= p.partBlocks;
    j0 = (int)blockIdx.y * p.partBlocks;
    n = min(n - j0, p.partBlocks);
    if (n <= 0) {  // causal: a range past the end of an early tile
      ptx::grid_wait_previous();
      return;
    }
  }

  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sQ = ptx::smem_u32(smem);
  const uint32_t ring = sQ + C::kQBytes;
  if ((sQ & 1023u) != 0) {
    if (threadIdx.x == 0) atomicExch(p.w.status, (p.w.epoch << 8) | 50);
    return;
  }
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + C::kQBytes + NS * C::kUnitBytes);
  const uint32_t barBase = ptx::smem_u32(&ctl->bars[0]);
  auto bar = [&](int slot) { return barBase + 8u * (uint32_t)slot; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    ptx::mbar_init(bar(kBarQFull), 1);
    ptx::mbar_init(bar(kBarSFull), 1);
    ptx::mbar_init(bar(kBarPReady), 4);
    for (int i = 0; i < 4; i++) ptx::mbar_init(bar(kBarScaleFull + i), 4);
    ptx::mbar_init(bar(kBarOFull), 1);
    ptx::mbar_init(bar(kBarOFree), 8);
    ptx::mbar_init(bar(kBarSumFull), 4);
    for (int s = 0; s < NS; s++) {
      ptx::mbar_init(bar(kBarKvFull + s), 1);
      ptx::mbar_init(bar(kBarKvEmpty + s), 1);
    }
    ctl->failed = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&ctl->tmemBase), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = ctl->tmemBase;
  const tc::WaitCtx wc{&ctl->failed, p.w.status, p.w.epoch};
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  const bool skip = (*p.flag == p.w.epoch);  // left to the CUDA-core kernel
  constexpr uint32_t kPCol1 = 128, kPCol2 = 192, kOCol = 256;

  if (skip) {
    // straight to the end
  } else if (warp < 4) {
    ptx::setmaxnreg_dec<kRegsIssueW>();
    if (warp == 0 && lane == 0) {
      // ============================================================== TMA loads
      const int gp = 1 << p.w.packShift;
      ptx::mbar_arrive_expect_tx(bar(kBarQFull), C::kQBytes);
#pragma unroll
      for (int part = 0; part < 2; part++) {
#pragma unroll
        for (int a = 0; a < C::kSub; a++) {
          ptx::tma_load_4d(sQ + (part * C::kSub + a) * kSubTileBytes, &tmQ, bar(kBarQFull), a * 64, w.unit * gp,
                           w.qRowTma + w.qlo[0], part * p.batches + w.batchTma);
        }
      }
      int ld = 0;
      auto load = [&](const CUtensorMap* tm, int part, int h, int y, int z) {  // one unit: head-dim elements from 128 h on
        const int s = ld % NS, slabs = min(2, C::kSub - 2 * h);
        if (ld >= NS) tc::wait_bar(bar(kBarKvEmpty + s), ((ld / NS) - 1) & 1, wc, 41);
        ptx::mbar_arrive_expect_tx(bar(kBarKvFull + s), slabs * kSubTileBytes);
        for (int a = 0; a < slabs; a++) {
          ptx::tma_load_4d(ring + s * C::kUnitBytes + a * kSubTileBytes, tm, bar(kBarKvFull + s), h * 128 + a * 64, y, z,
                           part * p.batches + w.batchTma);
        }
        ld++;
      };
      for (int j = 0; j < n; j++) {
        const int row = w.kvRowTma + (j0 + j) * kBlockN;
        for (int part = 2; part >= 0; part--) {
          for (int h = 0; h < 2; h++) {
            if (part == 0) load(&tmQ, 2, h, w.unit * gp, w.qRowTma + w.qlo[0]);
            load(&tmK, part, h, w.hkv, row);
          }
        }
        for (int part = 2; part >= 0; part--) {
          for (int h = 0; h < 2; h++) load(&tmV, part, h, w.hkv, row);
        }
      }
    } else if (warp == 1 && lane == 0) {
      // ============================================================== MMA issue
      const uint32_t idQK = ptx::instr_desc_f16(1, kBlockM, kBlockN, 0, 0);
      const uint64_t descK = ptx::smem_desc_sw128(16, 1024);
      const uint64_t descV = ptx::smem_desc_sw128(kSubTileBytes, 1024);
      const uint32_t kHi = (uint32_t)(descK >> 32), vHi = (uint32_t)(descV >> 32);
      const uint32_t kLoT = (uint32_t)descK, vLoT = (uint32_t)descV;
      int ld = 0;
      auto unitReady = [&]() -> int {
        const int s = ld % NS;
        tc::wait_bar(bar(kBarKvFull + s), (ld / NS) & 1, wc, 42);
        ptx::tc_fence_after();
        ld++;
        return s;
      };
      tc::wait_bar(bar(kBarQFull), 0, wc, 43);
      for (int j = 0; j < n; j++) {
        // S, whose columns hold P of block j - 1: its P.V was issued earlier by this thread, MMAs run in order
        uint32_t accS = 0;  // bit h: the accumulator of head-dim unit h holds something
#pragma unroll 1
        for (int part = 2; part >= 0; part--) {
#pragma unroll 1
          for (int h = 0; h < 2; h++) {
            const int q2 = part == 0 ? unitReady() : 0;
            const int s = unitReady();
            const uint32_t kLo = kLoT | ((ring + (uint32_t)(s * C::kUnitBytes)) >> 4);
            const int steps = (kHD == 192 && h == 1) ? 4 : 8;
#pragma unroll 1
            for (int qPart = 2 - part; qPart >= 0; qPart--) {
              const uint32_t qAddr = qPart == 2 ? ring + (uint32_t)(q2 * C::kUnitBytes)
                                                : sQ + (uint32_t)((qPart * C::kSub + 2 * h) * kSubTileBytes);
              const uint32_t qLo = kLoT | (qAddr >> 4);
#pragma unroll
              for (int kk = 0; kk < 8; kk++) {
                const uint32_t off = (uint32_t)((kk >> 2) * kSubTileBytes + (kk & 3) * 32) >> 4;
                if (kHD == 256 || kk < 4 || steps == 8) {
                  ptx::mma_ss_lohi(tmem + h * 128, qLo + off, kHi, kLo + off, kHi, idQK, kk > 0 ? 1u : (accS >> h) & 1u);
                }
              }
              accS |= 1u << h;
            }
            if (part == 0) ptx::tc_commit(bar(kBarKvEmpty + q2));
            ptx::tc_commit(bar(kBarKvEmpty + s));
          }
        }
        ptx::tc_commit(bar(kBarSFull));
        if (j > 0) tc::wait_bar(bar(kBarOFree), (j - 1) & 1, wc, 44);
        tc::wait_bar(bar(kBarPReady), j & 1, wc, 45);
        uint32_t accH[2] = {0, 0};
#pragma unroll 1
        for (int part = 2; part >= 0; part--) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const uint32_t idPV = ptx::instr_desc_f16(1, kBlockM, (kHD == 192 && h == 1) ? 64 : 128, 0, 1);
            const int s = unitReady();
            const uint32_t vLo = vLoT | ((ring + (uint32_t)(s * C::kUnitBytes)) >> 4);
#pragma unroll 1
            for (int pPart = 2 - part; pPart >= 0; pPart--) {
              const uint32_t a = tmem + (pPart == 0 ? 0u : pPart == 1 ? kPCol1 : kPCol2);
#pragma unroll
              for (int kk = 0; kk < kBlockN / 16; kk++) {
                ptx::mma_ts_lohi(tmem + kOCol + h * 128, a + kk * 8, vLo + ((kk * 2048) >> 4), vHi, idPV, kk > 0 ? 1u : accH[h]);
              }
              accH[h] = 1;
            }
            ptx::tc_commit(bar(kBarKvEmpty + s));
          }
        }
        ptx::tc_commit(bar(kBarOFull));
      }
    }
  } else if (warp < 8) {
    // ================================================================ softmax
    ptx::setmaxnreg_dec<kRegsSoftmaxW>();
    const int r = threadIdx.x & 127;
    const uint32_t tS = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int qpos = w.qlo[0] + (r >> p.w.packShift);
    const float c = p.w.scaleLog2;
    float m = -INFINITY, l = 0.f;
    for (int j = 0; j < n; j++) {
      tc::wait_bar(bar(kBarSFull), j & 1, wc, 46);
      ptx::tc_fence_after();
      const int kbase = (j0 + j) * kBlockN;
      int lim = kBlockN;  // columns [0, lim) are real keys that are not in the future
      if ((kbase + kBlockN > w.skv) || (p.w.causal && (kbase + kBlockN - 1 > w.qlo[0]))) {
        lim = w.skv - kbase;
        if (p.w.causal) lim = min(lim, qpos - kbase + 1);
      }
      float mNew = m;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t v[16], v2[16];
        ptx::tmem_ld_32x32b_x16(tS + q * 16, v);
        ptx::tmem_ld_32x32b_x16(tS + 128 + q * 16, v2);
        ptx::tmem_wait_ld();
        ptx::tmem_ld_fence(v);
        ptx::tmem_ld_fence(v2);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(v2[i]));
        if (lim < q * 16 + 16) {
#pragma unroll
          for (int i = 0; i < 16; i++) {
            if (q * 16 + i >= lim) v[i] = 0xff800000u;  // -inf
          }
        }
        float mx = tc::fmax2(__uint_as_float(v[0]), __uint_as_float(v[1]));
#pragma unroll
        for (int i = 2; i < 16; i += 2) mx = tc::fmax3(mx, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
        mNew = fmaxf(mNew, mx);
        ptx::tmem_st_32x32b_x16(tS + q * 16, v);
      }
      ptx::tmem_wait_st();
      const float mUse = (mNew == -INFINITY) ? 0.f : mNew;
      const float scale = (m == -INFINITY) ? 0.f : tc::ex2((m - mUse) * c);
      m = mNew;
      ctl->scale[j % 3][r] = scale;
      const float negMc = -mUse * c;
      const float2 c2 = make_float2(c, c), negMc2 = make_float2(negMc, negMc);
      float2 sum2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t v[16];
        ptx::tmem_ld_32x32b_x16(tS + q * 16, v);
        ptx::tmem_wait_ld();
        ptx::tmem_ld_fence(v);
        uint32_t p0[8], p1[8], p2[8];
        float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float2 x = tc::ffma2(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), c2, negMc2);
          x.x = tc::ex2(x.x);
          x.y = tc::ex2(x.y);
          s2 = tc::fadd2(s2, x);
          split3(x.x, x.y, p0[i >> 1], p1[i >> 1], p2[i >> 1]);
        }
        sum2 = tc::fadd2(sum2, s2);
        ptx::tmem_st_32x32b_x8(tS + q * 8, p0);  // inside the columns read so far
        ptx::tmem_st_32x32b_x8(tS + kPCol1 + q * 8, p1);
        ptx::tmem_st_32x32b_x8(tS + kPCol2 + q * 8, p2);
      }
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        ptx::mbar_arrive(bar(kBarPReady));
        ptx::mbar_arrive(bar(kBarScaleFull + j % 3));
      }
      l = l * scale + (sum2.x + sum2.y);
    }
    ctl->sum[r] = l;
    if (!whole && qpos < w.sq) {
      const long long row = blockIdx.y * p.rows + (w.qRow0 + qpos) * p.w.headsQ + (w.unit << p.w.packShift) + (r & ((1 << p.w.packShift) - 1));
      p.partM[row] = m;
      p.partL[row] = l;
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(bar(kBarSumFull));
  } else {
    // ================================================================ output, 128 (or the last 64) columns per warpgroup
    ptx::setmaxnreg_inc<kRegsOutW>();
    const int r = threadIdx.x & 127;
    const int half = (warp >= 12) ? 1 : 0;
    const int chunks = (kHD == 192 && half == 1) ? 2 : 4;
    const uint32_t tO = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kOCol + half * 128;
    float2 o[64];
#pragma unroll
    for (int i = 0; i < 64; i++) o[i] = make_float2(0.f, 0.f);
    for (int j = 0; j < n; j++) {
      // Slot j % 3 is published again for block j + 3, whose scores are issued behind P.V of block j + 2 and with it behind
      // this warp's arrival on kBarOFree for block j + 1: it is never two phases behind.
      tc::wait_bar(bar(kBarScaleFull + j % 3), (j / 3) & 1, wc, 47);
      const float scale = ctl->scale[j % 3][r];
      const float2 scale2 = make_float2(scale, scale);
      tc::wait_bar(bar(kBarOFull), j & 1, wc, 48);
      ptx::tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        if (kHD == 192 && ch >= chunks) break;
        uint32_t t[32];
        ptx::tmem_ld_32x32b_x32(tO + ch * 32, t);
        ptx::tmem_wait_ld();
        ptx::tmem_ld_fence(t);
        if (ch == chunks - 1) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(bar(kBarOFree));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          o[ch * 16 + (i >> 1)] = tc::ffma2(o[ch * 16 + (i >> 1)], scale2, make_float2(__uint_as_float(t[i]), __uint_as_float(t[i + 1])));
        }
      }
    }
    tc::wait_bar(bar(kBarSumFull), 0, wc, 49);
    const float l = ctl->sum[r];
    const float inv = !whole ? 1.f : (l > 0.f) ? (1.f / l) : 0.f;
    const int qpos = w.qlo[0] + (r >> p.w.packShift);
    const int head = (w.unit << p.w.packShift) + (r & ((1 << p.w.packShift) - 1));
    if (qpos < w.sq) {
      const long long row = (w.qRow0 + qpos) * p.w.headsQ + head;
      float4* dst = reinterpret_cast<float4*>((whole ? reinterpret_cast<float*>(p.w.O) + row * kHD : p.partO + (blockIdx.y * p.rows + row) * kHD) + half * 128);
#pragma unroll
      for (int i = 0; i < 32; i++) {
        if (kHD == 192 && i >= chunks * 8) break;
        dst[i] = make_float4(o[2 * i].x * inv, o[2 * i].y * inv, o[2 * i + 1].x * inv, o[2 * i + 1].y * inv);
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*wc.failed) __nanosleep(200000);  // a wait gave up: let whatever is still in flight drain before freeing
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, 512);
  }
}

// Adds up the key ranges of the tiles that have several: D / 4 threads per row.
constexpr int kMergeThreads = 128;
template <int kHD>
__global__ void __launch_bounds__(kMergeThreads) merge_kernel(const Params p) {
  constexpr int kVec = kHD / 4, kGroups = kMergeThreads / kVec;
  ptx::grid_wait_previous();
  ptx::grid_allow_next();
  const int g = threadIdx.x / kVec, c4 = threadIdx.x % kVec;
  const long long row = (long long)blockIdx.x * kGroups + g;
  if (*p.flag == p.w.epoch || g >= kGroups || row >= p.rows) return;
  int blocks = (p.w.seqLenKV + kBlockN - 1) / kBlockN;
  if (p.w.causal) {  // key blocks of this row's query tile, as in make_work
    const int rowsPerTile = kBlockM >> p.w.packShift;
    const int tile = (int)(row / p.w.headsQ % p.w.seqLenQ) / rowsPerTile;
    blocks = min(blocks, (min((tile + 1) * rowsPerTile, p.w.seqLenQ) + kBlockN - 1) / kBlockN);
  }
  const int parts = (blocks + p.partBlocks - 1) / p.partBlocks;
  if (parts == 1) return;  // the attention kernel has written the output
  float M = -INFINITY;
#pragma unroll 4
  for (int s = 0; s < parts; s++) M = fmaxf(M, __ldcg(p.partM + s * p.rows + row));
  if (M == -INFINITY) M = 0.f;  // no score above -inf: all weights and the row are 0
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
#pragma unroll 4
  for (int s = 0; s < parts; s++) {
    const long long i = s * p.rows + row;
    const float4 v = __ldcg(reinterpret_cast<const float4*>(p.partO + i * kHD + c4 * 4));
    const float f = tc::ex2((__ldcg(p.partM + i) - M) * p.w.scaleLog2);
    l = fmaf(__ldcg(p.partL + i), f, l);
    acc.x = fmaf(v.x, f, acc.x);
    acc.y = fmaf(v.y, f, acc.y);
    acc.z = fmaf(v.z, f, acc.z);
    acc.w = fmaf(v.w, f, acc.w);
  }
  const float inv = (l > 0.f) ? (1.f / l) : 0.f;
  *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.w.O) + row * kHD + c4 * 4) =
      make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
}

// ---------------------------------------------------------------------------------------------------- host
// [3 parts x batches, rows, heads, headDim] bf16 workspace tensor; box = 64 elements x boxHeads x boxRows x 1
static int make_map(CUtensorMap* m, const void* base, long long batches, long long rows, int heads, int headDim,
                    int boxHeads, int boxRows) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return kCudaError;
  cuuint64_t dims[4] = {(cuuint64_t)headDim, (cuuint64_t)heads, (cuuint64_t)rows, (cuuint64_t)(3 * batches)};
  cuuint64_t strides[3] = {(cuuint64_t)headDim * 2, (cuuint64_t)heads * headDim * 2, (cuuint64_t)rows * heads * headDim * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)boxHeads, (cuuint32_t)boxRows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error_string("cuTensorMapEncodeTiled failed with CUresult %d (fp32 parts: batches=%lld rows=%lld heads=%d headDim=%d)",
                     (int)r, batches, rows, heads, headDim);
    return kCudaError;
  }
  return kOk;
}

// Key ranges for fixed-length input with fewer query tiles than half of the SMs: as many as fill the GPU, at least two
// blocks each, where that saves more than the two microseconds a block takes less than the merge kernel costs.
struct Ranges {
  int parts = 1, blocks = 0x7FFFFFFF;  // ranges, key blocks of each
};
static Ranges plan_ranges(const FwdProblem& pr, const Fp32Piece& piece, int packShift, int numSMs) {
  Ranges r;
  if (pr.cuQ != nullptr || piece.heads != pr.headsKV) return r;
  const int rows = kBlockM >> packShift;
  const long long tiles = (long long)((pr.seqLenQ + rows - 1) / rows) * (pr.headsQ >> packShift) * piece.batches;
  const int seen = pr.causal && pr.seqLenQ < pr.seqLenKV ? pr.seqLenQ : pr.seqLenKV;
  const int n = (seen + kBlockN - 1) / kBlockN;
  long long parts = numSMs / tiles;
  if (parts > n / 2) parts = n / 2;
  if (parts < 2) return r;
  const int blocks = (int)((n + parts - 1) / parts);
  if (n - blocks < 3) return r;
  r.blocks = blocks;
  r.parts = (n + blocks - 1) / blocks;
  return r;
}

struct Layout {
  size_t q, k, v, part, partRows, bytes;  // byte offsets of the parts behind the flag, and of the partial results
};
// Rows of Q and of K / V that a piece covers (packed input: all of them).
static long long rows_q(const FwdProblem& pr, const Fp32Piece& piece) { return pr.cuQ != nullptr ? pr.totalQ : (long long)piece.batches * pr.seqLenQ; }
static long long rows_kv(const FwdProblem& pr, const Fp32Piece& piece) { return pr.cuQ != nullptr ? pr.totalKV : (long long)piece.batches * pr.seqLenKV; }

static Layout layout(const FwdProblem& pr, const Fp32Piece& piece, const Ranges& ranges) {
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  const size_t rowsQ = (size_t)rows_q(pr, piece), headsQ = (size_t)piece.heads * (pr.headsQ / pr.headsKV);
  const size_t q = rowsQ * headsQ * pr.headDim * 6, kv = (size_t)rows_kv(pr, piece) * piece.heads * pr.headDim * 6;
  Layout l;
  l.q = 1024;
  l.k = l.q + up(q);
  l.v = l.k + up(kv);
  l.part = l.v + up(kv);
  l.partRows = ranges.parts > 1 ? ranges.parts * rowsQ * headsQ : 0;
  l.bytes = l.part + l.partRows * (pr.headDim + 2) * sizeof(float);
  return l;
}

// The kernel of a head dim: two 128-row K / V rings up to 128, the wide form above.
template <int kHD, bool kVarlen>
constexpr auto kernel_of() {
  if constexpr (kHD > 128) {
    return fwd_wide_kernel<kHD, kVarlen>;
  } else {
    return fwd_kernel<(kHD <= 64 ? 64 : 128), kHD, kVarlen>;
  }
}

template <int kHD>
int launch(const FwdProblem& pr, const Fp32Piece& piece, int packShift, uint8_t* ws, int epoch) {
  constexpr int kSmem = kHD > 128 ? CfgWide<(kHD > 128 ? kHD : 256)>::kSmemBytes : Cfg<(kHD <= 64 ? 64 : 128)>::kSmemBytes;
  constexpr int threads = kHD > 128 ? kThreadsWide : kThreads;
  const bool varlen = (pr.cuQ != nullptr);
  auto kernel = varlen ? kernel_of<kHD, true>() : kernel_of<kHD, false>();
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return kCudaError;
  static std::once_flag once[64];
  static cudaError_t attrErr[64];
  std::call_once(once[device], [&] {
    attrErr[device] = cudaFuncSetAttribute(kernel_of<kHD, true>(), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (attrErr[device] == cudaSuccess) {
      attrErr[device] = cudaFuncSetAttribute(kernel_of<kHD, false>(), cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    }
  });
  if (attrErr[device] != cudaSuccess) {
    set_error_string("cudaFuncSetAttribute(%d bytes): %s", kSmem, cudaGetErrorString(attrErr[device]));
    return kCudaError;
  }
  const Ranges ranges = plan_ranges(pr, piece, packShift, device_num_sms(device));
  const Layout lay = layout(pr, piece, ranges);
  const int gp = 1 << packShift, rowsPerTile = kBlockM >> packShift, group = pr.headsQ / pr.headsKV, headsQ = piece.heads * group;
  const long long nb = varlen ? 1 : piece.batches;
  const long long rowsQ = varlen ? pr.totalQ : pr.seqLenQ, rowsKV = varlen ? pr.totalKV : pr.seqLenKV;
  // elements of Q (and O) and of K / V ahead of the piece
  const long long skipQ = ((long long)piece.batch0 * pr.seqLenQ * pr.headsQ + piece.head0 * group) * pr.headDim;
  const long long skipKV = ((long long)piece.batch0 * pr.seqLenKV * pr.headsKV + piece.head0) * pr.headDim;
  CUtensorMap tmQ, tmK, tmV;
  int rc;
  if ((rc = make_map(&tmQ, ws + lay.q, nb, rowsQ, headsQ, pr.headDim, gp, rowsPerTile)) != kOk) return rc;
  if ((rc = make_map(&tmK, ws + lay.k, nb, rowsKV, piece.heads, pr.headDim, 1, kBlockN)) != kOk) return rc;
  if ((rc = make_map(&tmV, ws + lay.v, nb, rowsKV, piece.heads, pr.headDim, 1, kBlockN)) != kOk) return rc;

  Params p = {};
  p.w.O = static_cast<float*>(pr.O) + skipQ;
  p.w.cuQ = pr.cuQ;
  p.w.cuKV = pr.cuKV;
  p.w.seqLenQ = pr.seqLenQ;
  p.w.seqLenKV = pr.seqLenKV;
  p.w.headsQ = pr.headsQ;
  p.w.headsKV = pr.headsKV;
  p.w.headDim = pr.headDim;
  p.w.group = group;
  p.w.packShift = packShift;
  p.w.numPairs = (pr.seqLenQ + rowsPerTile - 1) / rowsPerTile;
  p.w.numUnits = headsQ / gp;
  p.w.causal = pr.causal;
  p.w.scaleLog2 = (float)(1.4426950408889634 / sqrt((double)pr.headDim));
  p.w.epoch = epoch;
  p.w.status = device_status_word(device);
  if (p.w.status == nullptr) return kCudaError;
  const long long per = (long long)p.w.numUnits * piece.batches, numWork = per * p.w.numPairs;
  if (numWork > 0x7FFFFFFFll) {
    set_error_string("too many work items (%lld)", numWork);
    return kTooLarge;
  }
  p.w.numWork = (int)numWork;
  if (pr.causal) {
    // heaviest tiles first, over as many heads as have their K and V parts (12 bytes per element) in half of L2, but at
    // least two items per SM
    long long width = (64ll << 20) / (12ll * pr.seqLenKV * pr.headDim) * ((p.w.group >> packShift) > 0 ? (p.w.group >> packShift) : 1);
    const long long minWidth = (2ll * device_num_sms(device) + p.w.numPairs - 1) / p.w.numPairs;
    if (width < minWidth) width = minWidth;
    p.w.chunk = (int)(width < per ? width : per);
  }
  p.partBlocks = ranges.blocks;
  p.rows = rows_q(pr, piece) * headsQ;
  p.partO = reinterpret_cast<float*>(ws + lay.part);
  p.partM = p.partO + lay.partRows * kHD;
  p.partL = p.partM + lay.partRows;
  p.batches = (int)nb;
  p.flag = reinterpret_cast<const int*>(ws);

  SplitParams sp;
  sp.src[0] = static_cast<const float*>(pr.Q) + skipQ;
  sp.src[1] = static_cast<const float*>(pr.K) + skipKV;
  sp.src[2] = static_cast<const float*>(pr.V) + skipKV;
  sp.dst[0] = reinterpret_cast<uint16_t*>(ws + lay.q);
  sp.dst[1] = reinterpret_cast<uint16_t*>(ws + lay.k);
  sp.dst[2] = reinterpret_cast<uint16_t*>(ws + lay.v);
  sp.width[0] = headsQ * pr.headDim;
  sp.pitch[0] = pr.headsQ * pr.headDim;
  sp.width[1] = sp.width[2] = piece.heads * pr.headDim;
  sp.pitch[1] = sp.pitch[2] = pr.headsKV * pr.headDim;
  sp.cu[0] = pr.cuQ;
  sp.cu[1] = sp.cu[2] = pr.cuKV;
  sp.batches = pr.batch;
  sp.count[0] = rows_q(pr, piece) * sp.width[0];
  sp.count[1] = sp.count[2] = rows_kv(pr, piece) * sp.width[1];
  sp.flag = reinterpret_cast<int*>(ws);
  sp.epoch = epoch;
  cudaError_t e = launch_kernel(split_kernel, dim3(8u * (unsigned)device_num_sms(device)), kSplitThreads, 0, pr.stream, pr.overlap, sp);
  if (e == cudaSuccess) e = launch_kernel(kernel, dim3((unsigned)numWork, (unsigned)ranges.parts), threads, kSmem, pr.stream, pr.overlap, tmQ, tmK, tmV, p);
  if (e == cudaSuccess && ranges.parts > 1) {
    constexpr int kGroups = kMergeThreads / (kHD / 4);
    e = launch_kernel(merge_kernel<kHD>, dim3((unsigned)((p.rows + kGroups - 1) / kGroups)), kMergeThreads, 0, pr.stream, pr.overlap, p);
  }
  if (e != cudaSuccess) {
    set_error_string("fp32 tensor-core kernel launch failed: %s", cudaGetErrorString(e));
    return kCudaError;
  }
  return kOk;
}

}  // namespace fp32tc

// Mean number of `block`-key blocks that a query row reads.
static double mean_blocks(double sq, double skv, bool causal, int block) {
  const double n = ceil((causal ? fmin(sq, skv) : skv) / block);
  if (!causal) return n;
  return sq <= skv ? (n + 1.0) * 0.5 : n - (n - 1.0) * 0.5 * skv / sq;
}

// A known number of rows, and by size: where a model of both paths' times says so.  In us, at 148 SMs: the CUDA cores take 0.13 +
// 0.062 D per 64 x 64 block and SM (head dim 128 from three CTAs per SM on: 128 x 128 tiles); here a float costs 2e-6 for the
// split pass, a tile 4.2 + 0.0137 D and a 128 x 128 block 1.34 + 0.027 D, on one CTA per SM.  So short sequences, few
// keys and masked keys behind few queries stay on the CUDA cores whatever the batch is.  Fitted to 420 drawn calls of all head dims, 1 to 400
// sequences of 1 to 1500 rows, a quarter of them packed: the pick is within 0.3 % of the faster path on average, 25 % at worst.  us per
// call (CUDA cores, tensor cores): B512 S64 8 heads of 64 125, 348; B512 S49 12 heads of 32 111, 405; 2 x 100 x 3000 causal 8 heads of
// 128 18.6, 32.8; B4 4096 x 16 8 heads of 64 61, 88; on the other side B64 S256 8 heads of 64 213, 137; B4 4096 x 77 113, 89.
// Below the first line the launches decide: S128 4 heads of 64 11.7, 13.6; S128 4 heads of 128 18.6, 15.4; S256 4 heads of 64 21.2, 15.7.
bool fp32tc_applicable(const FwdProblem& p, int packShift, int numSMs, int option) {
  if (!TFA_HAVE_FP32 || p.dtype != kFp32 || p.totalQ < 0 || p.totalKV < 0) return false;
  const bool packed = p.cuQ != nullptr;
  const int rows = fp32tc::kBlockM >> packShift;
  if ((long long)((p.seqLenQ + rows - 1) / rows) * (p.headsQ >> packShift) * p.batch > 0x7FFFFFFFll) return false;  // grid
  if (option > 0) return true;
  const int seenMax = p.causal ? (p.seqLenQ < p.seqLenKV ? p.seqLenQ : p.seqLenKV) : p.seqLenKV;
  const long long ctasMax = (long long)((p.seqLenQ + 63) / 64) * p.headsQ * p.batch;
  if ((ctasMax + numSMs - 1) / numSMs * ((seenMax + 63) / 64) * p.headDim < 256) return false;
  // packed input: as if all sequences had the mean length
  const double sq = packed ? ceil((double)p.totalQ / p.batch) : p.seqLenQ, skv = packed ? ceil((double)p.totalKV / p.batch) : p.seqLenKV;
  const double seen = p.causal ? fmin(sq, skv) : skv, D = p.headDim, heads = (double)p.headsQ * p.batch;
  const bool wide = p.headDim == 128 && (double)((p.seqLenQ + 127) / 128) * heads >= 3.0 * numSMs;
  const double coreWaves = wide ? ceil(2.0 * ceil(sq / 128) * heads / numSMs) : ceil(ceil(sq / 64) * heads / numSMs);
  const double coreMean = wide ? 2.0 * mean_blocks(sq, skv, p.causal, 128) : mean_blocks(sq, skv, p.causal, 64);
  const double coreLongest = wide ? 2.0 * ceil(seen / 128) : ceil(seen / 64);
  const double cores = (0.13 + 0.062 * D) * fmax(coreWaves * coreMean, coreLongest);
  const fp32tc::Ranges ranges = fp32tc::plan_ranges(p, Fp32Piece{0, p.batch, 0, p.headsKV}, packShift, numSMs);
  const double tiles = ceil(sq / rows) * (p.headsQ >> packShift) * p.batch, waves = ceil(tiles * ranges.parts / numSMs);
  const double longest = ranges.parts > 1 ? ranges.blocks : ceil(seen / fp32tc::kBlockN);
  const double mean = ranges.parts > 1 ? longest : mean_blocks(sq, skv, p.causal, fp32tc::kBlockN);
  const double floats = (sq * heads + 2.0 * skv * p.headsKV * p.batch) * D;
  const double here = (ranges.parts > 1 ? 3.0 : 0.0) + 2e-6 * floats + (4.2 + 0.0137 * D) * waves +
                      (1.34 + 0.027 * D) * fmax(waves * mean, longest);
  return here < cores;
}

size_t fp32tc_workspace_bytes(const FwdProblem& p, const Fp32Piece& piece, int packShift, int numSMs) {
  return fp32tc::layout(p, piece, fp32tc::plan_ranges(p, piece, packShift, numSMs)).bytes;
}

// Enqueues the split and the attention kernel of a piece.  *ws begins with the word that reads `epoch` when the call is left to the
// CUDA-core kernel.
int launch_fwd_fp32tc(const FwdProblem& p, const Fp32Piece& piece, int packShift, void* ws, int epoch) {
#if TFA_HAVE_FP32
  uint8_t* w = static_cast<uint8_t*>(ws);
  switch (p.headDim) {
#if TFA_HAVE_HD32
    case 32:
      return fp32tc::launch<32>(p, piece, packShift, w, epoch);
#endif
#if TFA_HAVE_HD64
    case 64:
      return fp32tc::launch<64>(p, piece, packShift, w, epoch);
#endif
#if TFA_HAVE_HD96
    case 96:
      return fp32tc::launch<96>(p, piece, packShift, w, epoch);
#endif
#if TFA_HAVE_HD128
    case 128:
      return fp32tc::launch<128>(p, piece, packShift, w, epoch);
#endif
#if TFA_HAVE_HD192
    case 192:
      return fp32tc::launch<192>(p, piece, packShift, w, epoch);
#endif
#if TFA_HAVE_HD256
    case 256:
      return fp32tc::launch<256>(p, piece, packShift, w, epoch);
#endif
    default:
      break;
  }
#endif
  (void)piece;
  (void)packShift;
  (void)ws;
  (void)epoch;
  return kBadHeadDim;
}

}  // namespace tfa_b200
