// absmax-u8 quantiser and dequantiser, replacing
// adrastea_kernels/cpp/quantize.cu:3-56 (quantize_absmax_uint8,
// dequantize_absmax_uint8) for contiguous [rows, k] operands.
#include "u8_common.cuh"

namespace adr {

namespace {

// One thread per 16 weights; the same dequant4 the matmul kernels use, so a
// bit-exact check of this kernel's output checks their weight path too.
template <bool HAS_ZERO>
__global__ void __launch_bounds__(256) dequantize_u8_kernel(__half* out, const __half* scales,
                                                            const __half* zeros, const uint8_t* q,
                                                            int rows, int k, int block_size) {
  const int per_row = k / 16;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)rows * per_row) return;
  const int r = (int)(idx / per_row);
  const int kk = (int)(idx % per_row) * 16;
  const int groups = k / block_size;
  const int g = kk / block_size;
  ScalePair sp = make_scale(scales[(size_t)r * groups + g], HAS_ZERO,
                            HAS_ZERO ? zeros[(size_t)r * groups + g] : __half());
  uint4 w = ldg_nc_16(q + (size_t)r * k + kk);
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __half2 lo, hi;
    dequant4(ww[j], sp, lo, hi);
    o[2 * j] = half2_as_u32(lo);
    o[2 * j + 1] = half2_as_u32(hi);
  }
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)r * k + kk);
  dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
  dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// embed_uint8 (adrastea_kernels/cpp/embed_uint8.cu:3-19): out[t, :] = the dequantised row
// in_ids[t] of the table (implicit zero point 127.5).  One thread per 16 values, as above.
__global__ void __launch_bounds__(256) embed_u8_kernel(int n_dim, int n_ids, const short* in_ids,
                                                       __half* out, const uint8_t* table,
                                                       const __half* scales, int block_size) {
  const int per_row = n_dim / 16;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n_ids * per_row) return;
  const int t = (int)(idx / per_row);
  const int kk = (int)(idx % per_row) * 16;
  const int groups = n_dim / block_size;
  const int64_t id = in_ids[t];
  ScalePair sp = make_scale(scales[id * groups + kk / block_size], false, __half());
  uint4 w = ldg_nc_16(table + id * n_dim + kk);
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __half2 lo, hi;
    dequant4(ww[j], sp, lo, hi);
    o[2 * j] = half2_as_u32(lo);
    o[2 * j + 1] = half2_as_u32(hi);
  }
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)t * n_dim + kk);
  dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
  dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// One warp per (row, group): absmax by shuffles, then the scale in fp16 and
// the codes  u8(round(127.5 + x / float(scale)))  (quantize.cu:33, 42).
__device__ __forceinline__ uint8_t quantize_one(float x, float sf) {
  return static_cast<uint8_t>(roundf(127.5f + x / sf));
}
__global__ void __launch_bounds__(256) quantize_u8_kernel(uint8_t* q, __half* scales,
                                                          const __half* in, int rows, int k,
                                                          int block_size) {
  const int groups = k / block_size;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= (int64_t)rows * groups) return;
  const int r = (int)(wid / groups), g = (int)(wid % groups);
  const __half* src = in + (size_t)r * k + (size_t)g * block_size;
  float absmax = 0.0f;
  for (int i = lane; i < block_size; i += 32) absmax = fmaxf(absmax, fabsf(__half2float(src[i])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
  const __half s = __float2half_rn(absmax / 127.5f);
  if (lane == 0) scales[(size_t)r * groups + g] = s;
  const float sf = __half2float(s);
  uint8_t* dst = q + (size_t)r * k + (size_t)g * block_size;
  for (int i = lane; i < block_size; i += 32) dst[i] = quantize_one(__half2float(src[i]), sf);
}

// The same codes for blocks of 16 * LPG weights (LPG a power of two up to 32): lane l of a group takes
// its weights 8 l .. and 8 (l + LPG) .. as two 16-byte loads, so that the loads and the 8-byte stores
// of a warp are consecutive, the weights stay in registers between the maximum and the codes, and the
// two divisions a lane makes for its group are shared by 16 weights; two groups per lane are in
// flight.  HBM bound (2 bytes in, 1 out per weight); the kernel above spends its time in 2-byte loads,
// 1-byte stores and one IEEE division per weight: 11008 x 4096 in blocks of 128 took it 99 us, this
// one 37 us (135 MB: 21 us at the measured copy rate).
// The division is replaced by a multiplication with 1 / scale wherever that cannot change the code.
// With a normal fp16 scale |x / scale| < 128: the reciprocal, the quotient and either sum with 127.5
// are each off by at most 2^-17, so the two sums differ by at most 2^-15 and round to the same
// integer unless one lies within 2^-14 of a half-integer.  There (one weight in 8000, and every
// exact zero: 127.5), and for groups with a subnormal, zero or infinite scale, the lane divides.
// Rounding: t + 2^23 leaves the integer next to t in the low bits of the float.
template <int LPG>
__global__ void __launch_bounds__(256) quantize_u8_vec_kernel(uint8_t* q, __half* scales,
                                                              const __half* in, int64_t groups) {
  constexpr int U = 2;          // groups in flight per lane
  constexpr int GPW = 32 / LPG;  // groups per warp and step
  const int lane = threadIdx.x & 31;
  const int64_t g0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (GPW * U) + lane / LPG;
  const int64_t off0 = g0 * (16 * LPG) + (lane % LPG) * 8;
  uint4 raw[U][2];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h)  // (a group's lanes are live together; all lanes shuffle)
      raw[u][h] = g0 + u * GPW < groups ? ldg_nc_16(in + off0 + u * (GPW * 16 * LPG) + h * (8 * LPG))
                                        : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 f = __half22float2(u32_as_half2((&raw[u][i >> 2].x)[i & 3]));
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
    float absmax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) absmax = fmaxf(absmax, fabsf(x[i]));
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
    const __half s = __float2half_rn(absmax / 127.5f);
    const float sf = __half2float(s);
    const float inv = 1.0f / sf;
    constexpr float MAGIC = 8388608.0f;
    uint32_t c[16];
    bool safe = sf >= 6.103515625e-05f && sf <= 65504.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float t = fmaf(x[j], inv, 127.5f);
      const float m = t + MAGIC;
      c[j] = __float_as_uint(m);
      safe = safe && fabsf(t - (m - MAGIC)) < 0.5f - 6.103515625e-05f;  // (false for NaN)
    }
    if (!safe) {
#pragma unroll
      for (int j = 0; j < 16; ++j) c[j] = quantize_one(x[j], sf);
    }
    if (g0 + u * GPW < groups) {
      if (lane % LPG == 0) scales[g0 + u * GPW] = s;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t* d = c + h * 8;
        uint2 codes;
        codes.x = prmt(prmt(d[0], d[1], 0x0040u), prmt(d[2], d[3], 0x0040u), 0x5410u);
        codes.y = prmt(prmt(d[4], d[5], 0x0040u), prmt(d[6], d[7], 0x0040u), 0x5410u);
        *reinterpret_cast<uint2*>(q + off0 + u * (GPW * 16 * LPG) + h * (8 * LPG)) = codes;
      }
    }
  }
}

}  // namespace

int launch_dequantize_u8(adr_ctx* ctx, cudaStream_t stream, __half* out, const __half* scales,
                         const __half* zeros, const uint8_t* q, int rows, int k, int block_size) {
  int64_t threads = (int64_t)rows * (k / 16);
  int64_t grid = (threads + 255) / 256;
  if (grid > 0x7fffffffLL) return ADR_ERR_SHAPE;
  if (zeros)
    dequantize_u8_kernel<true><<<(unsigned)grid, 256, 0, stream>>>(out, scales, zeros, q, rows, k, block_size);
  else
    dequantize_u8_kernel<false><<<(unsigned)grid, 256, 0, stream>>>(out, scales, zeros, q, rows, k, block_size);
  return after_launch(ctx);
}

int launch_quantize_u8(adr_ctx* ctx, cudaStream_t stream, uint8_t* q, __half* scales,
                       const __half* in, int rows, int k, int block_size) {
  // 16 weights per lane where a block is a power of two of them within a warp and the buffers allow
  // 16-byte loads; any other block size or alignment takes the warp-per-group kernel
  const bool aligned = (reinterpret_cast<uintptr_t>(in) & 15u) == 0 && (reinterpret_cast<uintptr_t>(q) & 7u) == 0;
  const int lpg = block_size / 16;
  if (aligned && block_size % 16 == 0 && lpg <= 32 && (lpg & (lpg - 1)) == 0) {
    const int64_t groups = (int64_t)rows * (k / block_size);
    const int per_block = 8 * 2 * (32 / lpg);
    const int64_t grid = (groups + per_block - 1) / per_block;
    if (grid > 0x7fffffffLL) return ADR_ERR_SHAPE;
    auto kfn = lpg == 1   ? quantize_u8_vec_kernel<1>
               : lpg == 2 ? quantize_u8_vec_kernel<2>
               : lpg == 4 ? quantize_u8_vec_kernel<4>
               : lpg == 8 ? quantize_u8_vec_kernel<8>
               : lpg == 16 ? quantize_u8_vec_kernel<16>
                           : quantize_u8_vec_kernel<32>;
    kfn<<<(unsigned)grid, 256, 0, stream>>>(q, scales, in, groups);
    return after_launch(ctx);
  }
  int64_t warps = (int64_t)rows * (k / block_size);
  int64_t grid = (warps * 32 + 255) / 256;
  if (grid > 0x7fffffffLL) return ADR_ERR_SHAPE;
  quantize_u8_kernel<<<(unsigned)grid, 256, 0, stream>>>(q, scales, in, rows, k, block_size);
  return after_launch(ctx);
}

int launch_embed_u8(adr_ctx* ctx, cudaStream_t stream, int n_dim, int n_ids, const short* in_ids,
                    __half* out, const uint8_t* table, const __half* scales, int block_size) {
  int64_t threads = (int64_t)n_ids * (n_dim / 16);
  int64_t grid = (threads + 255) / 256;
  if (grid > 0x7fffffffLL) return ADR_ERR_SHAPE;
  embed_u8_kernel<<<(unsigned)grid, 256, 0, stream>>>(n_dim, n_ids, in_ids, out, table, scales, block_size);
  return after_launch(ctx);
}

}  // namespace adr
