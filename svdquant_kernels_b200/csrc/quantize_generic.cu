// Shape-agnostic quantizer kernels: the NVFP4 row packer (used for weights at
// load time and as the path for activation shapes the fused kernel does not
// take) and a plain LoRA-down projection.  CUDA-core only; the fused
// tensor-core kernel lives in quantize_fused.cu.
//
// Reference behaviour restated: baseline/kernels/_nvfp4.py:60-95 (row packer)
// and baseline/kernels/quantize_w4a4_act_fuse_lora/ref.py:36-48 (raw-x LoRA-down,
// smooth divide only on the quantised branch, zero rows up to the padded height).
#include "nvfp4_math.cuh"
#include "quantize_math.cuh"
#include "sm100.cuh"
#include "svdq_internal.h"

#include <type_traits>

namespace svdq {

// A block packs a tile of 128 rows x 4 groups, one 512-byte atom of the tensor core's scale layout.  It is bound by
// memory (15360 x 3840 fp32: 236 MB in, 33 MB out), so every access is laid out for it: consecutive lanes load
// consecutive 16 bytes of a row (four lanes per group for fp32, two for 16-bit types; the group's amax meets through
// shuffles) with several loads of a thread in flight, codes leave as whole sectors, and the scale bytes, which belong
// to one column of the tile each, are turned in shared memory so that both layouts are written in runs of 128 bytes
// and more.  That matrix takes 48 us, 5.6 TB/s (a thread per group, whose loads lie 64 bytes apart and whose scale
// bytes each touch a sector of their own: 75 us).  Small blocks, ten per SM (48 registers), because a block loads
// nothing while it turns its scales: 3072 x 3840 fp32 takes 12.5 us (8 groups, 256 threads, six blocks per SM: 14.4;
// nine of the small blocks: 15.6, a second wave; twelve: 14.7).
// A 16-byte piece of a 16-bit type holds eight elements, and their arithmetic is the bound: 16-bit values take the
// near quotients of quantize_math.cuh, one multiplication an element instead of a multiplication, a truncation and
// another, and their maximum two elements at a time.  15360 x 3840 bf16 37.8 -> 33.5 us, 4526 x 10304 30.0 -> 27.3.
constexpr int kPackRows = 128, kPackGroups = 4, kPackThreads = 128;

template <typename T>
__global__ void __launch_bounds__(kPackThreads, 10)
quantize_rows_kernel(const T* __restrict__ x, const T* __restrict__ smooth, uint8_t* __restrict__ codes,
                     uint8_t* __restrict__ scales, uint8_t* __restrict__ scales_swz, int rows, int rows_pad, int K) {
  constexpr int EPL = 16 / sizeof(T);                     // elements per lane
  constexpr int LPG = 16 / EPL;                           // lanes per group
  constexpr int ITEMS = kPackRows * kPackGroups * LPG;    // 16-byte pieces of a tile
  constexpr int BATCH = 4;
  using Code = typename std::conditional<EPL == 4, uint16_t, uint32_t>::type;
  __shared__ __align__(16) uint8_t sc[kPackGroups][kPackRows];
  constexpr bool k16 = sizeof(T) == 2;
  using Pair = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  __shared__ float near_lut[qmath::kScaleLutEntries];
  qmath::fill_near_lut(near_lut, threadIdx.x, kPackThreads);
  __syncthreads();
  // launched with programmatic serialization: nothing below may run before the kernel ahead has finished
  pdl_trigger();
  pdl_wait();
  const int groups = K >> 4;
  const int gtiles = (groups + kPackGroups - 1) / kPackGroups;      // neighbouring blocks: the same rows, the next columns
  const int m0 = static_cast<int>(blockIdx.x / gtiles) * kPackRows, g0 = static_cast<int>(blockIdx.x % gtiles) * kPackGroups;
  // piece of the tile handled by this thread: part fastest, then group, then row
  const int part = threadIdx.x % LPG, gl = threadIdx.x / LPG % kPackGroups;
  const int g = g0 + gl, k = g * 16 + part * EPL;
  float sm[EPL];
  if (smooth != nullptr && g < groups) {
    const uint4 v = *reinterpret_cast<const uint4*>(smooth + k);
#pragma unroll
    for (int i = 0; i < EPL; ++i) sm[i] = to_f32(reinterpret_cast<const T*>(&v)[i]);
  }
  constexpr int ROWS_PER_STEP = kPackThreads / (kPackGroups * LPG);
  const int r0 = threadIdx.x / (kPackGroups * LPG);
#pragma unroll 1
  for (int step = 0; step < ITEMS / kPackThreads; step += BATCH) {
    uint4 raw[BATCH];
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int m = m0 + r0 + (step + b) * ROWS_PER_STEP;
      raw[b] = make_uint4(0u, 0u, 0u, 0u);
      if (m < rows && g < groups) raw[b] = __ldcs(reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * K + k));
    }
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      const int r = r0 + (step + b) * ROWS_PER_STEP, m = m0 + r;
      // amax as the reference has it (a NaN does not count), and whether there is a NaN
      float f[EPL], amax = 0.0f;
      bool odd = false, packed = false;
#pragma unroll
      for (int i = 0; i < EPL; ++i) {
        f[i] = to_f32(reinterpret_cast<const T*>(&raw[b])[i]);
        if (smooth != nullptr) f[i] = __fdiv_rn(f[i], sm[i]);
        if constexpr (!k16) {
          amax = fmaxf(amax, fabsf(f[i]));
          odd |= f[i] != f[i];
        }
      }
      if constexpr (k16) {
        if (smooth == nullptr) {                          // two elements an instruction; a NaN comes through
          const Pair* h = reinterpret_cast<const Pair*>(&raw[b]);
          const Pair top = __hmax2_nan(__hmax2_nan(__habs2(h[0]), __habs2(h[1])), __hmax2_nan(__habs2(h[2]), __habs2(h[3])));
          amax = to_f32(__hmax_nan(top.x, top.y));
          packed = amax == amax;
        }
        if (!packed) {
          amax = 0.0f;
#pragma unroll
          for (int i = 0; i < EPL; ++i) {
            amax = fmaxf(amax, fabsf(f[i]));
            odd |= f[i] != f[i];
          }
        }
      }
#pragma unroll
      for (int d = 1; d < LPG; d *= 2) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
      uint32_t code = 0, sbyte = 0;
      if (m < rows && g < groups) {                       // rows of the padding get zero codes and scales
        const float2 zero = make_float2(0.0f, 0.0f);      // the + 0 below makes a -0 a +0
        if constexpr (k16) sbyte = qmath::scale_byte_near(amax);
        else sbyte = qmath::scale_byte(fminf(amax, 1e30f));   // the three-step divide wants a finite value; 448 is reached long before
        const float c = near_lut[sbyte];
        if (c != 0.0f && !odd) {
          // the conversion instruction's paths of quantize_math.cuh: near quotients for 16-bit values, cut values for fp32
          const float2 mult = make_float2(c, c);
          float w[EPL];
#pragma unroll
          for (int i = 0; i < EPL; i += 2) {
            float2 q;
            if constexpr (k16) {
              q = __ffma2_rn(make_float2(f[i], f[i + 1]), mult, zero);
            } else {
              // + 0 before the cut, which leaves a value below all bounds its sign
              q = __fadd2_rn(make_float2(f[i], f[i + 1]), zero);
              q = __fmul2_rn(make_float2(qmath::cut12(q.x), qmath::cut12(q.y)), mult);
            }
            w[i] = q.x; w[i + 1] = q.y;
          }
          code = qmath::cvt_e2m1<EPL>(w);
        } else if (!k16 || amax != 0.0f) {                // a group of zeros (and NaN) has zero codes
          const GroupBounds gb = bounds_for_scale(e4m3_to_f32(static_cast<uint8_t>(sbyte)));
#pragma unroll
          for (int i = 0; i < EPL; ++i) code |= e2m1_code(f[i], gb) << (4 * i);
        }
      }
      if (m < rows_pad && g < groups) *reinterpret_cast<Code*>(codes + static_cast<size_t>(m) * (K >> 1) + (k >> 1)) = static_cast<Code>(code);
      if (part == 0) sc[gl][r] = static_cast<uint8_t>(sbyte);
    }
  }
  __syncthreads();
  const bool words = (rows_pad & 3) == 0 && (reinterpret_cast<uintptr_t>(scales) & 3u) == 0;
  if (words) {
    const int gw = threadIdx.x >> 5, r = (threadIdx.x & 31) * 4;
    if (g0 + gw < groups && m0 + r < rows_pad)
      *reinterpret_cast<uint32_t*>(scales + static_cast<size_t>(g0 + gw) * rows_pad + m0 + r) = *reinterpret_cast<const uint32_t*>(&sc[gw][r]);
  } else {
    for (int i = threadIdx.x; i < kPackGroups * kPackRows; i += kPackThreads) {
      const int gw = i / kPackRows, r = i % kPackRows;
      if (g0 + gw < groups && m0 + r < rows_pad) scales[static_cast<size_t>(g0 + gw) * rows_pad + m0 + r] = sc[gw][r];
    }
  }
  // the tensor-core order exists only for whole tiles of 128 rows and 4 groups: word w of an atom is row
  // 32 (w % 4) + w / 4, its bytes the row's four groups
  if (scales_swz != nullptr) {
    const int w = threadIdx.x, r = 32 * (w & 3) + (w >> 2);
    *reinterpret_cast<uint32_t*>(scales_swz + sf_swizzled_offset(m0 + r, g0, groups)) =
        sc[0][r] | (sc[1][r] << 8) | (sc[2][r] << 16) | (static_cast<uint32_t>(sc[3][r]) << 24);
  }
}

// out[m, r] = sum_k x[m, k] * w[k, r] in fp32; rows >= M are written as zeros.
// 8 rows per block; threads stride over r so the w reads are coalesced.
template <typename T>
__global__ void __launch_bounds__(128)
lora_down_kernel(const T* __restrict__ x, const T* __restrict__ w, float* __restrict__ out, void* __restrict__ out16,
                 int M, int M_pad, int K, int R) {
  constexpr int ROWS = 8, KC = 128;
  __shared__ float xs[ROWS][KC];
  const int m0 = blockIdx.x * ROWS;
  for (int r0 = 0; r0 < R; r0 += blockDim.x) {
    const int r = r0 + threadIdx.x;
    float acc[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) acc[i] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += KC) {
      __syncthreads();
      for (int i = threadIdx.x; i < ROWS * KC; i += blockDim.x) {
        const int rr = i / KC, kk = i % KC;
        const int m = m0 + rr, k = k0 + kk;
        xs[rr][kk] = (m < M && k < K) ? to_f32(x[static_cast<size_t>(m) * K + k]) : 0.0f;
      }
      __syncthreads();
      if (r < R) {
        const int kmax = min(KC, K - k0);
        for (int kk = 0; kk < kmax; ++kk) {
          const float wv = to_f32(w[static_cast<size_t>(k0 + kk) * R + r]);
#pragma unroll
          for (int i = 0; i < ROWS; ++i) acc[i] = fmaf(xs[i][kk], wv, acc[i]);
        }
      }
    }
    if (r < R) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int m = m0 + i;
        if (m < M_pad) {
          out[static_cast<size_t>(m) * R + r] = acc[i];
          if (out16 != nullptr) store_lora16<T>(out16, static_cast<size_t>(m) * R + r, static_cast<size_t>(M_pad) * R, acc[i]);
        }
      }
    }
  }
}

// canonical [groups, rows] scale bytes -> 128x4 atom order
__global__ void swizzle_scales_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int groups, int rows) {
  const long long total = static_cast<long long>(groups) * rows;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int g = static_cast<int>(i / rows), m = static_cast<int>(i % rows);
    dst[sf_swizzled_offset(m, g, groups)] = src[i];
  }
}

// fp32 lora_act -> the 16-bit form of type T (see store_lora16)
template <typename T>
__global__ void cast_lora16_kernel(const float* __restrict__ src, void* __restrict__ dst, long long n) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    store_lora16<T>(dst, static_cast<size_t>(i), static_cast<size_t>(n), src[i]);
}

// bf16 -> fp16, eight values a thread where both sides are 16-byte aligned; unfit[block]: some value of the block's is NaN or
// beyond fp16's range.  Launched with SVDQ_LORA_UP_WORDS blocks.
__global__ void __launch_bounds__(256)
lora_up_f16_kernel(const __nv_bfloat16* __restrict__ src, __half* __restrict__ dst, uint32_t* __restrict__ unfit, long long n, int vec) {
  bool bad = false;
  auto one = [&](__nv_bfloat16 b) -> __half {
    const float v = __bfloat162float(b);
    bad |= !(fabsf(v) <= 65504.0f);
    return __float2half_rn(v);
  };
  const long long at = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x, step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long whole = vec ? n / 8 : 0;
  for (long long i = at; i < whole; i += step) {
    const uint4 in = reinterpret_cast<const uint4*>(src)[i];
    uint4 out;
#pragma unroll
    for (int j = 0; j < 8; ++j) reinterpret_cast<__half*>(&out)[j] = one(reinterpret_cast<const __nv_bfloat16*>(&in)[j]);
    reinterpret_cast<uint4*>(dst)[i] = out;
  }
  for (long long i = whole * 8 + at; i < n; i += step) dst[i] = one(src[i]);
  const int any = __syncthreads_or(bad ? 1 : 0);
  if (threadIdx.x == 0) unfit[blockIdx.x] = any != 0 ? 1u : 0u;
}

static int grid_for(long long items, int block) {
  long long g = (items + block - 1) / block;
  const long long cap = 148ll * 16;
  return static_cast<int>(g < 1 ? 1 : (g > cap ? cap : g));
}

int launch_quantize_rows(const void* x, const void* smooth, void* codes, void* scales, void* scales_swz, int rows,
                         int rows_pad, int K, int dtype, cudaStream_t stream) {
  if (rows_pad == 0 || K == 0) return SVDQ_OK;
  const long long tiles = static_cast<long long>((rows_pad + kPackRows - 1) / kPackRows) * ((K / 16 + kPackGroups - 1) / kPackGroups);
  if (tiles > 0x7fffffffll) return SVDQ_ERR_SHAPE;
  const unsigned int grid = static_cast<unsigned int>(tiles);
  uint8_t* c = static_cast<uint8_t*>(codes);
  uint8_t* s = static_cast<uint8_t*>(scales);
  uint8_t* sw = static_cast<uint8_t*>(scales_swz);
  auto launch = [&](auto kern, auto* xp, auto* sp) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kPackThreads, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, xp, sp, c, s, sw, rows, rows_pad, K) == cudaSuccess ? SVDQ_OK : SVDQ_ERR_LAUNCH;
  };
  switch (dtype) {
    case SVDQ_DTYPE_F16: return launch(quantize_rows_kernel<__half>, static_cast<const __half*>(x), static_cast<const __half*>(smooth));
    case SVDQ_DTYPE_BF16: return launch(quantize_rows_kernel<__nv_bfloat16>, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(smooth));
    case SVDQ_DTYPE_F32: return launch(quantize_rows_kernel<float>, static_cast<const float*>(x), static_cast<const float*>(smooth));
    default: return SVDQ_ERR_DTYPE;
  }
}

// The CUDA-core paths do not look at magnitudes: they mark every row block of a bf16 form as
// "does not fit fp16", which sends the GEMM down its two-pass bf16 route.
static int mark_lora16_unfit(void* out16, int rows, int R, int dtype, cudaStream_t stream) {
  if (out16 == nullptr || dtype != SVDQ_DTYPE_BF16 || rows == 0) return SVDQ_OK;
  uint32_t* flags = lora16_flags(out16, static_cast<size_t>(rows) * R);
  return cudaMemsetAsync(flags, 0xFF, sizeof(uint32_t) * ((rows + 31) / 32), stream) == cudaSuccess ? SVDQ_OK : SVDQ_ERR_CUDA;
}

int launch_lora_down(const void* x, const void* w, float* out, void* out16, int M, int M_pad, int K, int R, int dtype,
                     cudaStream_t stream) {
  if (M_pad == 0 || R == 0) return SVDQ_OK;
  const int grid = (M_pad + 7) / 8;
  if (dtype == SVDQ_DTYPE_F16)
    lora_down_kernel<__half><<<grid, 128, 0, stream>>>(static_cast<const __half*>(x), static_cast<const __half*>(w), out, out16, M, M_pad, K, R);
  else if (dtype == SVDQ_DTYPE_BF16)
    lora_down_kernel<__nv_bfloat16><<<grid, 128, 0, stream>>>(static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), out, out16, M, M_pad, K, R);
  else
    return SVDQ_ERR_DTYPE;
  if (cudaGetLastError() != cudaSuccess) return SVDQ_ERR_LAUNCH;
  return mark_lora16_unfit(out16, M_pad, R, dtype, stream);
}

int launch_swizzle_scales(const void* src, void* dst, int groups, int rows, cudaStream_t stream) {
  const long long n = static_cast<long long>(groups) * rows;
  if (n == 0) return SVDQ_OK;
  swizzle_scales_kernel<<<grid_for(n, 256), 256, 0, stream>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), groups, rows);
  return cudaGetLastError() == cudaSuccess ? SVDQ_OK : SVDQ_ERR_LAUNCH;
}

int launch_lora_up_f16(const void* src, void* dst, uint32_t* unfit, long long n, cudaStream_t stream) {
  const int vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0 ? 1 : 0;
  lora_up_f16_kernel<<<SVDQ_LORA_UP_WORDS, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(src), static_cast<__half*>(dst), unfit, n, vec);
  return cudaGetLastError() == cudaSuccess ? SVDQ_OK : SVDQ_ERR_LAUNCH;
}

int launch_cast_f32(const float* src, void* dst, int rows, int R, int dtype, cudaStream_t stream) {
  const long long n = static_cast<long long>(rows) * R;
  if (n == 0) return SVDQ_OK;
  if (dtype == SVDQ_DTYPE_F16)
    cast_lora16_kernel<__half><<<grid_for(n, 256), 256, 0, stream>>>(src, dst, n);
  else if (dtype == SVDQ_DTYPE_BF16)
    cast_lora16_kernel<__nv_bfloat16><<<grid_for(n, 256), 256, 0, stream>>>(src, dst, n);
  else
    return SVDQ_ERR_DTYPE;
  if (cudaGetLastError() != cudaSuccess) return SVDQ_ERR_LAUNCH;
  return mark_lora16_unfit(dst, rows, R, dtype, stream);
}

}  // namespace svdq
