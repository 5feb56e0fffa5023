// Block-scaled fp8 on the way in: the quantisation of an activation (one UE8M0 scale per 32 K-elements) and the
// repacking of the scales into the 512-byte blocks tcgen05 reads. Both are bound by HBM / L2 bytes: the activation is
// read once and its fp8 values written once (3 bytes per 16-bit element), where a chain of element-wise passes moves
// about 40. Measured, 4096 x 7168 bf16: 23.6 us (88 MB, 3.7 TB/s) with the launch; the element-wise passes and the
// packing by permutation took 470 us of the linear's 828.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "catcoc/capi.h"
#include "catcoc/host_util.h"
#include "catcoc/params.h"
#include "catcoc/ptx.cuh"

using namespace catcoc;

namespace {

constexpr int kMxBlock = 32;       // elements per scale
constexpr int kQuantChunks = 4;    // 8-element chunks per thread: their loads are independent

// Eight consecutive elements as floats.
template <int FMT>
CATCOC_DEVICE void load8(const void* x, int64_t chunk, float (&f)[8]) {
  if constexpr (FMT == FMT_F32) {
    const uint4* p = static_cast<const uint4*>(x) + 2 * chunk;
    const uint4 a = p[0], b = p[1];
    const uint32_t u[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(u[i]);
  } else {
    const uint4 a = static_cast<const uint4*>(x)[chunk];
    const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (FMT == FMT_BF16) {
        f[2 * i] = __uint_as_float(u[i] << 16);
        f[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u);
      } else {
        const __half2 h = *reinterpret_cast<const __half2*>(&u[i]);
        f[2 * i] = __low2float(h);
        f[2 * i + 1] = __high2float(h);
      }
    }
  }
}

template <bool E5M2>
CATCOC_DEVICE uint32_t cvt_fp8x2(float lo, float hi) {
  uint16_t r;
  if constexpr (E5M2) asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  else asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}

// What the saturating conversion above does not give: a block that holds an infinity or a NaN keeps values above the
// fp8 range, which become NaN (e4m3) or infinity (e5m2) as in a conversion without saturation.
template <bool E5M2>
CATCOC_DEVICE uint32_t cvt_fp8_special(float v) {
  const uint32_t sign = (__float_as_uint(v) >> 24) & 0x80u;
  const float a = fabsf(v);
  if (E5M2) {
    if (a != a) return sign | 0x7fu;
    if (a >= 61440.0f) return sign | 0x7cu;
  } else if (!(a <= 464.0f)) {
    return sign | 0x7fu;
  }
  return cvt_fp8x2<E5M2>(v, 0.0f) & 0xffu;
}

// q = fp8(x / 2^e), scale = e + 127 with e = ceil(log2(amax / fp8_max)) per 32 elements. A thread converts 8
// consecutive elements, four neighbouring lanes share a block.
template <int FMT, bool E5M2>
__global__ void __launch_bounds__(256) mx_quantize_kernel(const void* x, uint8_t* q, uint8_t* scales, int64_t chunks) {
  const int64_t base = static_cast<int64_t>(blockIdx.x) * (blockDim.x * kQuantChunks) + threadIdx.x;
  ptx::grid_dependency_wait();
  float f[kQuantChunks][8];
#pragma unroll
  for (int j = 0; j < kQuantChunks; ++j) {
    const int64_t c = base + static_cast<int64_t>(j) * blockDim.x;
    if (c < chunks) load8<FMT>(x, c, f[j]);
    else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[j][i] = 0.0f;
    }
  }
#pragma unroll
  for (int j = 0; j < kQuantChunks; ++j) {
    const int64_t c = base + static_cast<int64_t>(j) * blockDim.x;
    float amax = 0.0f;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) { amax = fmaxf(amax, fabsf(f[j][i])); nan = nan || (f[j][i] != f[j][i]); }
    amax = nan ? __uint_as_float(0x7fffffffu) : amax;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      const float other = __shfl_xor_sync(0xffffffffu, amax, o);
      amax = (amax != amax || other != other) ? __uint_as_float(0x7fffffffu) : fmaxf(amax, other);
    }
    int e = 0;
    if (amax > 0.0f) {   // false for a NaN
      constexpr float kInvMax = 1.0f / (E5M2 ? 57344.0f : 448.0f);
      const float l = ceilf(log2f(fmaxf(amax, 1.17549435e-38f) * kInvMax));
      e = static_cast<int>(fminf(fmaxf(l, -127.0f), 127.0f));
    }
    if (c >= chunks) continue;
    const float inv = __uint_as_float(e < 127 ? static_cast<uint32_t>(127 - e) << 23 : 0x00400000u);   // 2^-e
    uint32_t w[2];
    if (amax < INFINITY) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        w[h] = cvt_fp8x2<E5M2>(f[j][4 * h] * inv, f[j][4 * h + 1] * inv) |
               (cvt_fp8x2<E5M2>(f[j][4 * h + 2] * inv, f[j][4 * h + 3] * inv) << 16);
    } else {
      w[0] = w[1] = 0u;
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i >> 2] |= cvt_fp8_special<E5M2>(f[j][i] * inv) << (8 * (i & 3));
    }
    *reinterpret_cast<uint2*>(q + c * 8) = make_uint2(w[0], w[1]);
    if ((c & 3) == 0) scales[c >> 2] = static_cast<uint8_t>(e + 127);
  }
}

// out[rt][kt][l * 16 + j * 4 + s] = scales[rt * 128 + j * 32 + l][kt * 4 + s]; rows and K-blocks past the end read as
// 127 (= 1.0). One thread per 4-byte word; eight neighbouring threads walk along K so that their reads share a sector.
__global__ void __launch_bounds__(256) mx_pack_kernel(const uint8_t* scales, int rows, int kb, uint32_t* out, int row_tiles, int k_tiles) {
  const int kt_groups = (k_tiles + 7) / 8;
  ptx::grid_dependency_wait();
  const int64_t total = static_cast<int64_t>(row_tiles) * kt_groups * 1024;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t blk = i >> 10;
    const int t = static_cast<int>(i & 1023);
    const int rt = static_cast<int>(blk / kt_groups);
    const int kt = static_cast<int>(blk - static_cast<int64_t>(rt) * kt_groups) * 8 + (t & 7);
    if (kt >= k_tiles) continue;
    const int word = t >> 3;                                  // 0..127: l = word / 4, j = word % 4
    const int row = rt * 128 + (word & 3) * 32 + (word >> 2);
    uint32_t v = 0x7f7f7f7fu;
    if (row < rows) {
      const uint8_t* s = scales + static_cast<int64_t>(row) * kb + kt * 4;
      const int left = min(4, kb - kt * 4);
      if (left == 4 && (kb & 3) == 0) v = *reinterpret_cast<const uint32_t*>(s);   // base and row pitch are whole words
      else
        for (int b = 0; b < left; ++b) v = (v & ~(0xffu << (8 * b))) | (static_cast<uint32_t>(s[b]) << (8 * b));
    }
    out[(static_cast<int64_t>(rt) * k_tiles + kt) * 128 + word] = v;
  }
}

}  // namespace

extern "C" int catcoc_mx_quantize(const void* x, int fmt, int64_t elems, int e5m2, void* q, void* scales, void* stream) {
  if (x == nullptr || q == nullptr || scales == nullptr || elems <= 0 || elems % kMxBlock != 0 ||
      (fmt != CATCOC_FMT_F16 && fmt != CATCOC_FMT_BF16 && fmt != CATCOC_FMT_F32)) {
    host::set_error("mx_quantize: bad argument");
    return CATCOC_E_BAD_ARG;
  }
  if ((reinterpret_cast<uintptr_t>(x) & 15) != 0 || (reinterpret_cast<uintptr_t>(q) & 7) != 0) {
    host::set_error("mx_quantize: the input must be 16-byte aligned, the output 8-byte aligned");
    return CATCOC_E_ALIGNMENT;
  }
  const int64_t chunks = elems / 8;
  const int64_t per_block = 256 * kQuantChunks;
  const int64_t blocks = (chunks + per_block - 1) / per_block;
  if (blocks > 0x7fffffff) { host::set_error("mx_quantize: too many elements"); return CATCOC_E_TOO_LARGE; }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaSuccess;
  auto launch = [&](auto kernel) {
    e = host::launch_overlapped(kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, st, x, static_cast<uint8_t*>(q),
                                static_cast<uint8_t*>(scales), chunks);
  };
  if (fmt == CATCOC_FMT_BF16) e5m2 ? launch(mx_quantize_kernel<FMT_BF16, true>) : launch(mx_quantize_kernel<FMT_BF16, false>);
  else if (fmt == CATCOC_FMT_F16) e5m2 ? launch(mx_quantize_kernel<FMT_F16, true>) : launch(mx_quantize_kernel<FMT_F16, false>);
  else e5m2 ? launch(mx_quantize_kernel<FMT_F32, true>) : launch(mx_quantize_kernel<FMT_F32, false>);
  CATCOC_CUDA_OK(e);
  return CATCOC_OK;
}

extern "C" int catcoc_mx_pack_scales(const void* scales, int rows, int kb, void* out, void* stream) {
  if (scales == nullptr || out == nullptr || rows <= 0 || kb <= 0 || (reinterpret_cast<uintptr_t>(out) & 3) != 0 ||
      (reinterpret_cast<uintptr_t>(scales) & 3) != 0) {
    host::set_error("mx_pack_scales: bad argument");
    return CATCOC_E_BAD_ARG;
  }
  const int rt = (rows + 127) / 128, kt = (kb + 3) / 4;
  int64_t blocks = static_cast<int64_t>(rt) * ((kt + 7) / 8) * 4;
  if (blocks > 148 * 16) blocks = 148 * 16;
  CATCOC_CUDA_OK(host::launch_overlapped(mx_pack_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                         static_cast<const uint8_t*>(scales), rows, kb, static_cast<uint32_t*>(out), rt, kt));
  return CATCOC_OK;
}
