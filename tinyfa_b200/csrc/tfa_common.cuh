// Types shared by the host launchers and the C-ABI of the B200 attention-forward library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tfa_b200 {

// Status codes returned by every C-ABI entry point (0 = success).
enum Status : int {
  kOk = 0,
  kBadDtype = 1,       // dtype code is not 1 (fp16), 2 (bf16) or 3 (fp32)
  kBadHeadDim = 2,     // head dim not in {32, 64, 96, 128, 192, 256}
  kBadArgument = 3,    // null pointer, negative size, Hq % Hkv != 0, misaligned pointer ...
  kCudaError = 4,      // a CUDA runtime / driver call failed (see tfa_b200_last_error_string)
  kWrongDevice = 5,    // current device is not compute capability 10.x
  kTooLarge = 6,       // a size exceeds what an entry point supports
  kDeviceTimeout = 7,  // a bounded wait inside a kernel gave up (reported by tfa_b200_device_status)
};

// dtype codes follow the reference binding (reference csrc/binding/flash_attn_binding.cu:22).
enum DType : int { kFp16 = 1, kBf16 = 2, kFp32 = 3 };

// One attention-forward problem, fixed-length or packed variable-length.
// Layouts (reference csrc/flash_attn/params.cuh:49-68, 97-116):
//   fixed : Q,O [B,Sq,Hq,D]   K,V [B,Skv,Hkv,D]        cuQ == cuKV == nullptr
//   varlen: Q,O [totalQ,Hq,D] K,V [totalKV,Hkv,D]      cuQ/cuKV = int32 [B+1] prefix sums on the device;
//           seqLenQ / seqLenKV then hold the maximum lengths and only size the grid
//           (reference csrc/flash_attn/launcher.cuh:94-98).
struct FwdProblem {
  const void* Q;
  const void* K;
  const void* V;
  void* O;
  const int* cuQ;
  const int* cuKV;
  int dtype;
  int batch;
  int seqLenQ;
  int seqLenKV;
  long long totalQ;   // rows of Q/O  (fixed: B*Sq; varlen: upper bound known on the host, or -1)
  long long totalKV;  // rows of K/V
  int headsQ;
  int headsKV;
  int headDim;
  int causal;
  cudaStream_t stream;
  // fp32 CUDA-core kernels: when not null, they return at once unless this device word reads gateEpoch (see fwd_fp32_tc.cu)
  const int* gate = nullptr;
  int gateEpoch = 0;
  bool overlap = false;  // launch with programmatic stream serialization (launch_kernel below); not under stream capture
};

// How the split-KV path cuts a call (fwd_decode.cu): `runs` equal runs over the key blocks of all batch entries, or, with
// runs == 0, `splits` key ranges of every (batch, KV head) pair.  splits is the largest number of partial results of a pair.
struct SplitPlan {
  int splits;
  int runs;
  int blocksPerEntry;
};

// How the tensor-core path cuts a call with few query tiles into key ranges: `parts` ranges of partBlocks 128-key blocks
// (parts == 1: not at all), and where their partial results go ([parts][rows][headDim] and [parts][rows] floats).
struct TcSplit {
  int parts = 1;
  int partBlocks = 0;
  float* partO = nullptr;
  float* partLse = nullptr;
};

// A piece of an fp32 call on the tensor cores, which works with one workspace at a time (dispatch_fp32 in c_abi.cu): batch
// entries [batch0, batch0 + batches) and KV heads [head0, head0 + heads) with their Q heads.  Packed input: all entries.
struct Fp32Piece {
  int batch0, batches;
  int head0, heads;
};

// The device status word holds 0, or (launch epoch << 8) | site code once a bounded wait inside a kernel gave up.

// Kernels of this library let the next kernel of the stream start early (griddepcontrol.launch_dependents) and, launched
// through here with overlap, start early themselves: every thread waits with griddepcontrol.wait for the end of the kernel
// before, ahead of its first access to global memory, so that only launch and set-up overlap.  The next kernel is let in
// after that wait, not before: let in at the top, kernels pile up ahead of time and their CTAs share SMs that they would
// have had alone (fp32 S176 16 over 4 heads of 96 22.7 -> 28.1 us).  Back to back calls gain about 2 us each; behind a kernel
// that does not let others start early nothing changes.
template <class... Params, class... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, int threads, size_t smemBytes, cudaStream_t stream, bool overlap,
                          const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smemBytes;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

int launch_fwd_fp32(const FwdProblem& p);    // fp32: CUDA-core FMA kernel
void set_error_string(const char* fmt, ...);
// argument checks shared by every entry point (c_abi.cu); both return a Status
int validate_common(const void* Q, const void* K, const void* V, void* O, int dtype, int batch, int sq, int skv, int hq,
                    int hkv, int d);
bool may_overlap(cudaStream_t stream);  // c_abi.cu: false under stream capture
int check_device();  // current device must be compute capability 10.x

}  // namespace tfa_b200
