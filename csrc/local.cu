// Memory-bound ops that need no other rank: RMSNorm, and what all-reduce (+ bias) and all-reduce + bias
// + RMSNorm come down to at world size 1 (no staging copy, no barrier, no tags). bf16 data, fp32 math.
// Reference counterparts: kraken/fused/rms_norm.py:9-72, kraken/fused/one_shot_all_reduce_bias.py:20-173,
// kraken/fused/one_shot_all_reduce_bias_rms_norm.py:23-169.
//
// All of them are bound by HBM, or by the launch for a few rows. Blocks are small, take one row (or 16 KB)
// each and are started in address order: on a B200 that reads and writes faster than a persistent grid
// whose blocks stride through memory. Measured: RMSNorm of 16384 x 8192 83 us (6.47 TB/s; persistent
// 256-thread blocks with a prefetched next row 92 us, rows through a ring of bulk copies 99 us); 256 MB
// copied by 512-thread blocks of two vectors per thread 82 us, by a persistent grid 93 us, with bulk copies 90 us.
#include "kraken/host.h"
#include "kraken/norm_core.cuh"
#include "kraken/tcgen05.cuh"

namespace kraken {

enum LocalNormMode : int {
  NORM_PLAIN = 0,         // y = norm(x)
  NORM_BIAS = 1,          // y = norm(x + bias), the sum kept in fp32
  NORM_ROUND_BIAS = 2,    // y = norm(bf16(x + bias)): the sum as a bf16 tensor would hold it
  NORM_ROUND_BIAS_F32 = 3 // the same with x in fp32, rounded to bf16 before the bias is added
};

struct LocalNormParams {
  const void* x;
  const void* bias;
  const void* w;
  void* y;
  unsigned long long bias_rows;   // rows of the bias: row r takes bias row r % bias_rows
  int D;
  float eps;
};

// One block per row; a thread keeps VPT vectors of eight elements (vectors threadIdx.x + i * blockDim.x).
template <int VPT, int MODE>
__global__ void __launch_bounds__(VPT <= 2 ? 1024 : 512) norm_row_kernel(const LocalNormParams p) {
  __shared__ float partial[32];
  pdl_launch();
  const int nvec = p.D / 8;
  const size_t row = blockIdx.x;
  const char* x = (const char*)p.x + row * (size_t)p.D * (MODE == NORM_ROUND_BIAS_F32 ? 4 : 2);
  const char* bias = MODE == NORM_PLAIN ? nullptr : (const char*)p.bias + (size_t)(p.bias_rows == 1 ? 0 : row % p.bias_rows) * p.D * 2;
  pdl_wait();
  U4 q[VPT], q2[MODE == NORM_ROUND_BIAS_F32 ? VPT : 1], wq[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      if (MODE == NORM_ROUND_BIAS_F32) {
        q[i] = ld16(x + (size_t)v * 32);
        q2[MODE == NORM_ROUND_BIAS_F32 ? i : 0] = ld16(x + (size_t)v * 32 + 16);
      } else {
        q[i] = ld16(x + (size_t)v * 16);
      }
    }
  }
  U4 bq[MODE == NORM_PLAIN ? 1 : VPT];
  if (MODE != NORM_PLAIN) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) bq[MODE == NORM_PLAIN ? 0 : i] = ld16_nc(bias + (size_t)v * 16);
    }
  }
  // the sums; kept packed when they are bf16 values, in fp32 otherwise (the weights are then fetched only
  // after the reduction: they would not fit the registers)
  constexpr bool kFp32 = MODE == NORM_BIAS;
  if (!kFp32) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) wq[i] = ld16_nc((const char*)p.w + (size_t)v * 16);
    }
  }
  float f[kFp32 ? VPT : 1][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float (&g)[8] = f[kFp32 ? i : 0];
      if (MODE == NORM_ROUND_BIAS_F32) {
        const U4 hi = q2[MODE == NORM_ROUND_BIAS_F32 ? i : 0];
        const float t[8] = {__uint_as_float(q[i].x), __uint_as_float(q[i].y), __uint_as_float(q[i].z), __uint_as_float(q[i].w),
                            __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z), __uint_as_float(hi.w)};
        q[i] = pack8(t);
      }
      unpack8(q[i], g);
      if (MODE != NORM_PLAIN) acc8(bq[MODE == NORM_PLAIN ? 0 : i], g);
      if (MODE == NORM_ROUND_BIAS || MODE == NORM_ROUND_BIAS_F32) {
        q[i] = pack8(g);
        unpack8(q[i], g);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += g[j] * g[j];
    }
  }
  ss = warp_sum(ss);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = (int)(blockDim.x >> 5);
  if (lane == 0) partial[warp] = ss;
  __syncthreads();
  ss = warp_sum(lane < nwarps ? partial[lane] : 0.f);
  const float inv = rsqrtf(ss / (float)p.D + p.eps);
  char* y = (char*)p.y + row * (size_t)p.D * 2;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float (&g)[8] = f[kFp32 ? i : 0];
      if (kFp32) wq[i] = ld16_nc((const char*)p.w + (size_t)v * 16);
      else unpack8(q[i], g);
      float h[8];
      unpack8(wq[i], h);
#pragma unroll
      for (int j = 0; j < 8; ++j) h[j] = g[j] * inv * h[j];
      st16(y + (size_t)v * 16, pack8(h));
    }
  }
}

// Thousands of rows: the row is fetched into shared memory with one bulk copy and read from there twice,
// so a block holds no row in registers and as many rows are in flight as shared memory takes (13 of 16 KB
// per SM). Rows kept in registers measured 2-50 % slower here, following each kernel's register count
// (16384 rows: D 8192 87.5 to 83.0 us, D 6144 95 to 62.7, D 5120 58 to 53.4; floor 81.9 / 61.4 / 51.2).
template <int T>
__global__ void __launch_bounds__(T) norm_stream_kernel(const LocalNormParams p, const SyncCtx sync) {
  extern __shared__ __align__(128) unsigned char row_smem[];
  __shared__ __align__(8) unsigned long long bar;
  __shared__ float partial[T / 32];
  pdl_launch();
  const int nvec = p.D / 8;
  const uint32_t row_bytes = (uint32_t)p.D * 2u;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    mbar_fence_init();
    pdl_wait();
    mbar_expect_tx(smem_u32(&bar), row_bytes);
    bulk_load_1d(smem_u32(row_smem), (const char*)p.x + (size_t)blockIdx.x * row_bytes, row_bytes, smem_u32(&bar));
  }
  __syncthreads();
  pdl_wait();
  if (!mbar_wait(smem_u32(&bar), 0, sync, 90)) return;
  float ss = 0.f;
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += T) {
    float g[8];
    unpack8(*(const U4*)(row_smem + (size_t)v * 16), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += g[j] * g[j];
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int k = 0; k < T / 32; ++k) ss += partial[k];
  const float inv = rsqrtf(ss / (float)p.D + p.eps);
  char* y = (char*)p.y + (size_t)blockIdx.x * row_bytes;
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += T) {
    float g[8], h[8];
    unpack8(*(const U4*)(row_smem + (size_t)v * 16), g);
    unpack8(ld16_nc((const char*)p.w + (size_t)v * 16), h);
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = g[j] * inv * h[j];
    st16(y + (size_t)v * 16, pack8(h));
  }
}

// Rows longer than the register budget: two passes over global memory.
__global__ void __launch_bounds__(kNormMaxThreads) rms_norm_long_kernel(const LocalNormParams p) {
  __shared__ float smem[32];
  pdl_launch();
  pdl_wait();
  const int nvec = p.D / 8;
  const char* xrow = (const char*)p.x + (size_t)blockIdx.x * p.D * 2;
  char* yrow = (char*)p.y + (size_t)blockIdx.x * p.D * 2;
  float ss = 0.f;
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8];
    unpack8(ld16(xrow + (size_t)v * 16), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum(ss, smem);
  const float inv = rsqrtf(ss / (float)p.D + p.eps);
  for (int v = threadIdx.x; v < nvec; v += blockDim.x) {
    float f[8], g[8];
    unpack8(ld16(xrow + (size_t)v * 16), f);
    unpack8(ld16_nc((const char*)p.w + (size_t)v * 16), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = f[j] * inv * g[j];
    st16(yrow + (size_t)v * 16, pack8(g));
  }
}

// ---- out = in (+ bias) ------------------------------------------------------------------------
constexpr int kLocalThreads = 512;
constexpr int kLocalVpt = 2;
struct LocalSumParams {
  const void* in;
  const void* bias;
  void* out;
  unsigned long long nvec, bias_vecs;   // 16-byte vectors of the tensor and of the bias
};
template <bool BIAS>
__global__ void __launch_bounds__(kLocalThreads) local_sum_kernel(const LocalSumParams p) {
  pdl_launch();
  pdl_wait();
  const size_t v0 = (size_t)blockIdx.x * (kLocalThreads * kLocalVpt) + threadIdx.x;
  U4 x[kLocalVpt], b[kLocalVpt];
#pragma unroll
  for (int i = 0; i < kLocalVpt; ++i) {
    const size_t v = v0 + (size_t)i * kLocalThreads;
    if (v < p.nvec) {
      x[i] = ld16((const char*)p.in + v * 16);
      if (BIAS) b[i] = ld16_nc((const char*)p.bias + (v % p.bias_vecs) * 16);
    }
  }
#pragma unroll
  for (int i = 0; i < kLocalVpt; ++i) {
    const size_t v = v0 + (size_t)i * kLocalThreads;
    if (v < p.nvec) {
      if (BIAS) {
        float f[8];
        unpack8(b[i], f);
        acc8(x[i], f);
        x[i] = pack8(f);
      }
      st16((char*)p.out + v * 16, x[i]);
    }
  }
}

typedef void (*NormKernel)(const LocalNormParams);
template <int MODE>
static NormKernel norm_row(int vpt) {
  switch (vpt) {
    case 1: return norm_row_kernel<1, MODE>;
    case 2: return norm_row_kernel<2, MODE>;
    case 3: return norm_row_kernel<3, MODE>;
    case 4: return norm_row_kernel<4, MODE>;
    case 5: return norm_row_kernel<5, MODE>;
    case 6: return norm_row_kernel<6, MODE>;
    case 7: return norm_row_kernel<7, MODE>;
    default: return norm_row_kernel<8, MODE>;
  }
}

static int launch_norm(const DeviceState* d, int mode, LocalNormParams p, int rows, cudaStream_t stream) {
  const int nvec = p.D / 8;
  if (mode == NORM_PLAIN && rows >= 24 * d->num_sms && p.D <= 32768) {
    // from here on the rows stream through shared memory (4096 x 4096: 12.2 us against 14.3; 2048 x 8192, which
    // L2 mostly holds: 15 against 12.6)
    SyncCtx sync = sync_ctx(d);
    void* args[] = {(void*)&p, (void*)&sync};
    const bool small = p.D < 2560;
    return launch_overlapped(small ? (const void*)norm_stream_kernel<64> : (const void*)norm_stream_kernel<128>, (unsigned)rows, small ? 64 : 128,
                             args, (size_t)p.D * 2, stream);
  }
  // Two rows per SM or fewer: the row's latency counts, so as many threads as it has vectors. Beyond, half as
  // many: fewer barriers' worth of warps (512 x 8192 3.9 us against 4.8, with 128 threads 5.7). Kernels of
  // three vectors and more per thread are built for 512 threads.
  int threads = ((rows <= 2 * d->num_sms ? nvec : (nvec + 1) / 2) + 31) / 32 * 32;
  if (threads > 1024) threads = nvec <= 2048 ? 1024 : 512;
  if (rows > 2 * d->num_sms && threads > 512) threads = 512;
  const int vpt = (nvec + threads - 1) / threads;
  void* args[] = {(void*)&p};
  if (vpt > 8) return launch_overlapped((const void*)rms_norm_long_kernel, (unsigned)rows, kNormMaxThreads, args, 0, stream);
  NormKernel fn = mode == NORM_PLAIN ? norm_row<NORM_PLAIN>(vpt) : mode == NORM_BIAS ? norm_row<NORM_BIAS>(vpt)
                  : mode == NORM_ROUND_BIAS ? norm_row<NORM_ROUND_BIAS>(vpt) : norm_row<NORM_ROUND_BIAS_F32>(vpt);
  return launch_overlapped((const void*)fn, (unsigned)rows, (unsigned)threads, args, 0, stream);
}

}  // namespace kraken

using namespace kraken;

// y = x * rsqrt(mean(x^2) + eps) * w over rows of D elements
KR_API int kr_rms_norm(const void* x, const void* w, void* y, int rows, int D, float eps, cudaStream_t stream) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(rows >= 0 && D > 0 && D % 8 == 0, "rms_norm needs D % 8 == 0");
  KR_REQUIRE((((uintptr_t)x | (uintptr_t)y | (uintptr_t)w) & 15) == 0, "tensors must be 16-byte aligned");
  if (rows == 0) return KR_SUCCESS;
  LocalNormParams p{x, nullptr, w, y, 1, D, eps};
  return launch_norm(d, NORM_PLAIN, p, rows, stream);
}

// y = rms_norm(x + bias) * w on this GPU alone. bias: nullptr, one row or `rows` rows (bias_numel
// elements). round_sum != 0: the sum is rounded to bf16 before the norm, and x, which then may be
// fp32 (x_fp32), before the sum.
KR_API int kr_local_bias_rms_norm(const void* x, int x_fp32, const void* bias, unsigned long long bias_numel, const void* w, void* y,
                                  int rows, int D, float eps, int round_sum, cudaStream_t stream) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(rows >= 0 && D > 0 && D % 8 == 0, "needs D % 8 == 0");
  KR_REQUIRE(D / 8 <= 8 * 512, "row too long for the bias + RMSNorm kernel");
  KR_REQUIRE((((uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (uintptr_t)bias) & 15) == 0, "tensors must be 16-byte aligned");
  KR_REQUIRE(!x_fp32 || round_sum, "fp32 input is rounded to bf16");
  if (bias) KR_REQUIRE(bias_numel > 0 && bias_numel % D == 0, "the bias must be whole rows");
  KR_REQUIRE(bias || !round_sum, "rounding is for the sum with a bias");
  if (rows == 0) return KR_SUCCESS;
  LocalNormParams p{x, bias, w, y, bias ? bias_numel / D : 1, D, eps};
  const int mode = !bias ? NORM_PLAIN : !round_sum ? NORM_BIAS : x_fp32 ? NORM_ROUND_BIAS_F32 : NORM_ROUND_BIAS;
  return launch_norm(d, mode, p, rows, stream);
}

// output = input (+ bias): the all-reduce of one rank. numel and bias_numel are multiples of 8.
KR_API int kr_local_all_reduce(const void* input, void* output, const void* bias, unsigned long long bias_numel,
                               unsigned long long numel, cudaStream_t stream) {
  KR_REQUIRE(numel % 8 == 0 && (!bias || (bias_numel > 0 && bias_numel % 8 == 0)), "sizes must be multiples of 8");
  KR_REQUIRE((((uintptr_t)input | (uintptr_t)output | (uintptr_t)bias) & 15) == 0, "tensors must be 16-byte aligned");
  if (numel == 0 || (!bias && input == output)) return KR_SUCCESS;
  LocalSumParams p{input, bias, output, numel / 8, bias ? bias_numel / 8 : 1};
  void* args[] = {(void*)&p};
  const void* fn = bias ? (const void*)local_sum_kernel<true> : (const void*)local_sum_kernel<false>;
  return launch_overlapped(fn, cdiv(p.nvec, kLocalThreads * kLocalVpt), kLocalThreads, args, 0, stream);
}
