// probes.cu — microbenchmarks that measure the roofline denominators of the TE
// kernels' reported fractions (no vendor figure exists for them):
//   mode 0: conflict-free shared-memory atomicAdd (int32): lane l of every warp
//           updates a word in bank l; all SMs, 1024 threads per CTA.
//   mode 1: the same with 16-bit halves (increment 1 or 1<<16), the TE kernel's
//           packed-counter form.
//   mode 2: uniformly random words in a 4096-word region (bank conflicts and
//           same-address collisions as random data produces them).
//   mode 3: lane-striped but every warp of the CTA updates the same 32 words
//           each time (no bank conflict inside an instruction, same addresses
//           across consecutive instructions).
// The entry point times the kernel with CUDA events on `stream` and returns the
// number of increments and the milliseconds (synchronises the stream).
//
// tc_seq_probe: the GEMM-B2 kernel's MMA sequence back to back (below).
//
// tc_int8_probe: dense INT8 tensor-pipe throughput, the roofline of the GEMM-B2
// path. One CTA per SM (its shared-memory request admits one), one thread issues
// back-to-back tcgen05.mma.cta_group::1.kind::i8 of M = 128, N = 256, K = 32 from
// fixed shared-memory operands into two alternating int32 TMEM accumulators
// (512 columns), commits to an mbarrier and waits for it (bounded); nothing is
// loaded from global memory, so this is the issue-limited MMA rate. The FP4
// variant issues kind::mxf4 (packed E2M1, K = 64, unit block scales): the rate of
// the 4-bit GEMM-B2 form.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace tenex {

__global__ void __launch_bounds__(1024, 1) smem_atomic_probe(int mode, int iters,
                                                             unsigned* sink) {
  __shared__ unsigned s[4096];
  const int tid = threadIdx.x;
  for (int i = tid; i < 4096; i += blockDim.x) s[i] = 0u;
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5;
  uint32_t x = 0x9e3779b9u * (uint32_t)(blockIdx.x * blockDim.x + tid + 1);
  if (mode == 0) {
#pragma unroll 8
    for (int i = 0; i < iters; ++i) atomicAdd(&s[lane + 32 * ((i + warp) & 127)], 1u);
  } else if (mode == 1) {
#pragma unroll 8
    for (int i = 0; i < iters; ++i)
      atomicAdd(&s[lane + 32 * ((i + warp) & 127)], 1u << ((i & 1) << 4));
  } else if (mode == 3) {
#pragma unroll 8
    for (int i = 0; i < iters; ++i) atomicAdd(&s[lane], 1u);
  } else {
#pragma unroll 8
    for (int i = 0; i < iters; ++i) {
      x ^= x << 13;
      x ^= x >> 17;
      x ^= x << 5;
      atomicAdd(&s[x & 4095u], 1u);
    }
  }
  __syncthreads();
  unsigned acc = 0;
  for (int i = tid; i < 4096; i += blockDim.x) acc += s[i];
  if (acc == 0xffffffffu) sink[0] = acc;  // keeps the work observable
}

constexpr int kProbeM = 128, kProbeN = 256, kProbeK = 32;
constexpr int kProbeSmem = 120 * 1024;  // > half of an SM's shared memory: one CTA per SM

// FP4 = true: the same with tcgen05.mma.kind::mxf4 (packed E2M1, M = 128, N = 256,
// K = 64 from the same 32-byte operand rows) and unit UE8M0 block scales in TMEM,
// one float32 accumulator (256 columns) plus the scale columns.
template <bool FP4>
__global__ void __launch_bounds__(128, 1) tc_probe(int iters, int* err) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)sm_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* a = sm;                                  // 128 rows x 32 B: 2 planes of 2 KB
  unsigned char* b = sm + kProbeM * kProbeK;              // 256 rows x 32 B: 2 planes of 4 KB
  uint64_t* bar = reinterpret_cast<uint64_t*>(b + kProbeN * kProbeK);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x;
  for (int i = tid; i < (kProbeM + kProbeN) * kProbeK / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(a)[i] = 0x01010101u * (uint32_t)(i & 3);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // operands visible to the MMA
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  constexpr uint32_t kSf = 256;  // FP4: scale-factor columns (8 each for A and B)
  if (FP4) {
    tmem_st8(tmem + ((uint32_t)(tid & ~31) << 16) + kSf, 0x7f7f7f7fu);       // 4 warps
    tmem_st8(tmem + ((uint32_t)(tid & ~31) << 16) + kSf + 8, 0x7f7f7f7fu);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (tid == 0) {
    const uint64_t ad = smem_desc(smem_u32(a), kProbeM * 16, 128);
    const uint64_t bd = smem_desc(smem_u32(b), kProbeN * 16, 128);
    if (FP4) {
      const uint32_t idesc = idesc_mxf4(kProbeM, kProbeN);
      for (int it = 0; it < iters; ++it)
        mma_mxf4(tmem, ad, bd, idesc, it >= 1 ? 1u : 0u, tmem + kSf, tmem + kSf + 8);
    } else {
      const uint32_t idesc = idesc_i8(kProbeM, kProbeN);
      for (int it = 0; it < iters; ++it)
        mma_i8(tmem + (uint32_t)((it & 1) * kProbeN), ad, bd, idesc, it >= 2 ? 1u : 0u);
    }
    mma_commit(bar);
    if (!mbar_wait(bar, 0)) atomicExch(err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
}

// The GEMM-B2 kernel's own MMA sequence issued back to back: per 128-byte K
// stage, four K steps of two MMAs (the source tile as A against the targets
// [FP; P] at N = 2 TN into TMEM columns 0.., and F at N = TN into columns 256..),
// 128-byte swizzled K-major descriptors walking three stage buffers, as the
// GEMM's main loop issues them, but with no copies and no waits: the rate that
// bounds the GEMM's main loop for this instruction mix.
constexpr int kSeqStageMax = (3 * 128 + 128) * 128;  // the widest stage (TN = 128)

template <bool FP4>
__global__ void __launch_bounds__(128, 1) tc_seq_probe(int tn, int stages, int* err) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)sm_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 3 * kSeqStageMax);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x;
  for (int i = tid; i < 3 * kSeqStageMax / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(sm)[i] = 0x22222222u * (uint32_t)(i & 1);  // E2M1 1.0 / int8 34
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  constexpr uint32_t kSfa = 384, kSfb = 392;  // the GEMM's scale-factor columns
  if (FP4) {
    tmem_st8(tmem + ((uint32_t)(tid & ~31) << 16) + kSfa, 0x7f7f7f7fu);
    tmem_st8(tmem + ((uint32_t)(tid & ~31) << 16) + kSfb, 0x7f7f7f7fu);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (tid == 0) {
    const uint32_t i2 = FP4 ? idesc_mxf4(128, 2 * tn) : idesc_i8(128, 2 * tn);
    const uint32_t i1 = FP4 ? idesc_mxf4(128, tn) : idesc_i8(128, tn);
    const int stage = (3 * tn + 128) * 128, tgt = tn * 128;
    for (int k = 0; k < stages; ++k) {
      unsigned char* buf = sm + (k % 3) * stage;
      const uint32_t bFPP = smem_u32(buf), bF = smem_u32(buf + 2 * tgt);
      const uint32_t aP = smem_u32(buf + 3 * tgt);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        const uint32_t off = kk * 32;
        const uint32_t acc = (k > 0 || kk > 0) ? 1u : 0u;
        const uint64_t ad = smem_desc_sw128(aP + off);
        if (FP4) {
          mma_mxf4(tmem, ad, smem_desc_sw128(bFPP + off), i2, acc, tmem + kSfa, tmem + kSfb);
          mma_mxf4(tmem + 256, ad, smem_desc_sw128(bF + off), i1, acc, tmem + kSfa, tmem + kSfb);
        } else {
          mma_i8(tmem, ad, smem_desc_sw128(bFPP + off), i2, acc);
          mma_i8(tmem + 256, ad, smem_desc_sw128(bF + off), i1, acc);
        }
      }
    }
    mma_commit(bar);
    if (!mbar_wait(bar, 0)) atomicExch(err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
}

}  // namespace tenex

using namespace tenex;

extern "C" int tenex_probe_tc_gemm_b2(int kind, int tile_n, int stages, double* ops, float* ms,
                                      void* stream_) {
  if ((kind != 1 && kind != 2) || stages < 1 || !ops || !ms ||
      !(tile_n == 128 || tile_n == 112 || tile_n == 96 || tile_n == 80 || tile_n == 64))
    return fail(TENEX_ERR_BADARG,
                "kind 1 (int8) or 2 (4-bit), tile_n in {128,112,96,80,64}, stages >= 1, outputs "
                "non-NULL");
  DevAttr A;
  int st = current_device_attr(&A);
  if (st) return st;
  cudaStream_t s = as_stream(stream_);
  int* err = nullptr;
  cudaError_t e = cudaMallocAsync(&err, sizeof(int), s);
  if (e != cudaSuccess) return check_cuda(e, "cudaMallocAsync");
  cudaMemsetAsync(err, 0, sizeof(int), s);
  const int smem = 3 * kSeqStageMax + 2048;
  const bool fp4 = kind == 2;
  e = fp4 ? cudaFuncSetAttribute(tc_seq_probe<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem)
          : cudaFuncSetAttribute(tc_seq_probe<false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) {
    cudaFreeAsync(err, s);
    return check_cuda(e, "cudaFuncSetAttribute");
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  for (int rep = 0; rep < 2; ++rep) {  // warm-up launch, then the timed one
    if (rep == 1) cudaEventRecord(e0, s);
    const int n = rep == 0 ? (stages < 16 ? stages : 16) : stages;
    if (fp4)
      tc_seq_probe<true><<<A.sm_count, 128, smem, s>>>(tile_n, n, err);
    else
      tc_seq_probe<false><<<A.sm_count, 128, smem, s>>>(tile_n, n, err);
  }
  cudaEventRecord(e1, s);
  st = check_launch("tc_seq_probe");
  e = cudaEventSynchronize(e1);
  if (!st && e != cudaSuccess) st = check_cuda(e, "cudaEventSynchronize");
  float t = 0.f;
  cudaEventElapsedTime(&t, e0, e1);
  int h = 0;
  cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s);
  cudaStreamSynchronize(s);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(err, s);
  if (st) return st;
  if (h) return fail(TENEX_ERR_TIMEOUT, "tensor-pipe sequence probe: commit wait expired");
  *ms = t;
  *ops = 2.0 * 128 * 3 * tile_n * (fp4 ? 64 : 32) * 4.0 * stages * A.sm_count;
  return TENEX_OK;
}

template <bool FP4>
static int probe_tc(int iters, double* ops, float* ms, void* stream_) {
  if (iters < 1 || !ops || !ms) return fail(TENEX_ERR_BADARG, "iters >= 1, outputs non-NULL");
  DevAttr A;
  int st = current_device_attr(&A);
  if (st) return st;
  cudaStream_t s = as_stream(stream_);
  int* err = nullptr;
  cudaError_t e = cudaMallocAsync(&err, sizeof(int), s);
  if (e != cudaSuccess) return check_cuda(e, "cudaMallocAsync");
  cudaMemsetAsync(err, 0, sizeof(int), s);
  e = cudaFuncSetAttribute(tc_probe<FP4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kProbeSmem + 1024);
  if (e != cudaSuccess) {
    cudaFreeAsync(err, s);
    return check_cuda(e, "cudaFuncSetAttribute");
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  tc_probe<FP4><<<A.sm_count, 128, kProbeSmem + 1024, s>>>(iters < 64 ? iters : 64, err);
  cudaEventRecord(e0, s);
  tc_probe<FP4><<<A.sm_count, 128, kProbeSmem + 1024, s>>>(iters, err);
  cudaEventRecord(e1, s);
  st = check_launch("tc_probe");
  e = cudaEventSynchronize(e1);
  if (!st && e != cudaSuccess) st = check_cuda(e, "cudaEventSynchronize");
  float t = 0.f;
  cudaEventElapsedTime(&t, e0, e1);
  int h = 0;
  cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, s);
  cudaStreamSynchronize(s);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(err, s);
  if (st) return st;
  if (h) return fail(TENEX_ERR_TIMEOUT, "tensor-pipe probe: commit wait expired");
  *ms = t;
  *ops = 2.0 * kProbeM * kProbeN * (FP4 ? 2 * kProbeK : kProbeK) * (double)iters * A.sm_count;
  return TENEX_OK;
}

extern "C" int tenex_probe_tc_int8(int iters, double* ops, float* ms, void* stream) {
  return probe_tc<false>(iters, ops, ms, stream);
}

extern "C" int tenex_probe_tc_fp4(int iters, double* ops, float* ms, void* stream) {
  return probe_tc<true>(iters, ops, ms, stream);
}

extern "C" int tenex_probe_smem_atomics(int mode, int iters, int64_t* increments, float* ms,
                                        void* stream_) {
  if (mode < 0 || mode > 3 || iters < 1 || !increments || !ms)
    return fail(TENEX_ERR_BADARG, "mode in 0..3, iters >= 1, outputs non-NULL");
  DevAttr A;
  int st = current_device_attr(&A);
  if (st) return st;
  cudaStream_t s = as_stream(stream_);
  unsigned* sink = nullptr;
  cudaError_t e = cudaMallocAsync(&sink, sizeof(unsigned), s);
  if (e != cudaSuccess) return check_cuda(e, "cudaMallocAsync");
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int grid = A.sm_count, block = 1024;
  smem_atomic_probe<<<grid, block, 0, s>>>(mode, iters, sink);  // warm-up
  cudaEventRecord(e0, s);
  smem_atomic_probe<<<grid, block, 0, s>>>(mode, iters, sink);
  cudaEventRecord(e1, s);
  st = check_launch("smem_atomic_probe");
  e = cudaEventSynchronize(e1);
  if (!st && e != cudaSuccess) st = check_cuda(e, "cudaEventSynchronize");
  float t = 0.f;
  cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(sink, s);
  *ms = t;
  *increments = (int64_t)grid * block * iters;
  return st;
}

// ---- FP32 min/max issue rate (denominator of the DPI trimming kernel) -------
// Eight independent chains per thread, each step one three-input max.f32 and two
// min.f32 (the DPI kernel's instruction mix); volatile asm keeps every
// instruction. 2 CTAs of 1024 threads per SM.
namespace {
__global__ void __launch_bounds__(1024, 2) minmax_probe(int iters, float seed, float* sink) {
  float a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = seed + (float)(threadIdx.x + k);
  const float x = seed * 0.5f, y = seed * 0.25f;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float m1, m2;
      asm volatile("min.f32 %0, %1, %2;" : "=f"(m1) : "f"(a[k]), "f"(x));
      asm volatile("min.f32 %0, %1, %2;" : "=f"(m2) : "f"(a[(k + 1) & 7]), "f"(y));
      asm volatile("max.f32 %0, %1, %2, %3;" : "=f"(a[k]) : "f"(a[k]), "f"(m1), "f"(m2));
    }
  }
  float t = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) t += a[k];
  if (t == 12345.678f) sink[0] = t;  // never true for the probe's inputs; keeps the chains live
}
}  // namespace

extern "C" int tenex_probe_minmax(int iters, double* instructions, float* ms, void* stream_) {
  if (iters < 1 || !instructions || !ms)
    return fail(TENEX_ERR_BADARG, "iters >= 1, outputs non-NULL");
  DevAttr A;
  int st = current_device_attr(&A);
  if (st) return st;
  cudaStream_t s = as_stream(stream_);
  float* sink = nullptr;
  cudaError_t e = cudaMallocAsync(&sink, sizeof(float), s);
  if (e != cudaSuccess) return check_cuda(e, "cudaMallocAsync");
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int grid = 2 * A.sm_count, block = 1024;
  minmax_probe<<<grid, block, 0, s>>>(iters, 1.5f, sink);  // warm-up
  cudaEventRecord(e0, s);
  minmax_probe<<<grid, block, 0, s>>>(iters, 1.5f, sink);
  cudaEventRecord(e1, s);
  st = check_launch("minmax_probe");
  e = cudaEventSynchronize(e1);
  if (!st && e != cudaSuccess) st = check_cuda(e, "cudaEventSynchronize");
  float t = 0.f;
  cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFreeAsync(sink, s);
  *ms = t;
  *instructions = (double)grid * block * iters * 8.0 * 3.0;
  return st;
}

namespace tenex {
// dev::rcp_count against the correctly rounded reciprocal, one count per thread and step.
__global__ void rcp_count_check(uint32_t last, unsigned* differ) {
  unsigned n = 0;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x + 1; c <= last;
       c += gridDim.x * blockDim.x)
    n += __float_as_uint(dev::rcp_count((float)c)) != __float_as_uint(__frcp_rn((float)c));
  if (n) atomicAdd(differ, n);
}
}  // namespace tenex

extern "C" int tenex_check_rcp_count(int64_t last, int64_t* differ, void* stream_) {
  if (last < 1 || last > ((int64_t)1 << 24) || !differ)
    return fail(TENEX_ERR_BADARG, "need 1 <= last <= 2^24 and an output");
  cudaStream_t s = as_stream(stream_);
  unsigned* d = nullptr;
  unsigned h = 0;
  cudaError_t e = cudaMallocAsync(&d, sizeof(unsigned), s);
  if (e != cudaSuccess) return check_cuda(e, "cudaMallocAsync");
  e = cudaMemsetAsync(d, 0, sizeof(unsigned), s);
  int st = e == cudaSuccess ? TENEX_OK : check_cuda(e, "cudaMemsetAsync");
  if (!st) {
    rcp_count_check<<<592, 256, 0, s>>>((uint32_t)last, d);
    st = check_launch("rcp_count_check");
  }
  if (!st) {
    e = cudaMemcpyAsync(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) st = check_cuda(e, "tenex_check_rcp_count");
  }
  cudaFreeAsync(d, s);
  *differ = h;
  return st;
}
