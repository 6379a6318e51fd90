// absmax-u8 quantiser and dequantiser, replacing
// adrastea_kernels/cpp/quantize.cu:3-56 (quantize_absmax_uint8,
// dequantize_absmax_uint8) for contiguous [rows, k] operands.
#include "u8_common.cuh"

namespace adr {

namespace {

// The same dequant4 the matmul kernels use, so a bit-exact check of this kernel's output checks their
// weight path too.  HBM bound (1 byte in, 2 out per weight).  A lane takes 8 weights, so that the
// 16-byte stores of a warp are consecutive, and four such pieces, a block's width apart, in flight;
// rows are contiguous, so a piece's scale is found from its number alone, by a shift where the block
// size is a power of two.  With 16 weights per lane each store instruction wrote half of every 32-byte
// sector it touched, behind a 64-bit division: 11008 x 4096 25.1 -> 23.3 us.
constexpr int DEQ_U = 4;
template <bool HAS_ZERO, typename I>
__global__ void __launch_bounds__(256) dequantize_u8_kernel(__half* out, const __half* scales,
                                                            const __half* zeros, const uint8_t* q,
                                                            I pieces, unsigned per_block, int shift) {
  const I first = (I)blockIdx.x * (256 * DEQ_U) + threadIdx.x;
  uint2 w[DEQ_U];
  __half sc[DEQ_U], zp[DEQ_U];
#pragma unroll
  for (int u = 0; u < DEQ_U; ++u) {
    const I i = first + u * 256;
    w[u] = make_uint2(0, 0);
    sc[u] = zp[u] = __half();
    if (i < pieces) {
      w[u] = *reinterpret_cast<const uint2*>(q + (size_t)i * 8);
      const I g = shift >= 0 ? i >> shift : i / per_block;
      sc[u] = scales[g];
      if (HAS_ZERO) zp[u] = zeros[g];
    }
  }
#pragma unroll
  for (int u = 0; u < DEQ_U; ++u) {
    const I i = first + u * 256;
    if (i >= pieces) break;
    const ScalePair sp = make_scale(sc[u], HAS_ZERO, zp[u]);
    __half2 h[4];
    dequant4(w[u].x, sp, h[0], h[1]);
    dequant4(w[u].y, sp, h[2], h[3]);
    reinterpret_cast<uint4*>(out)[i] =
        make_uint4(half2_as_u32(h[0]), half2_as_u32(h[1]), half2_as_u32(h[2]), half2_as_u32(h[3]));
  }
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
// flight.  Bound by instruction issue: 11008 x 4096 in blocks of 128 takes 32.5 us where its 135 MB (2 bytes
// in, 1 out per weight) take 21 at the measured copy rate.  The kernel above spends its time in 2-byte loads,
// 1-byte stores and one IEEE division per weight: 99 us.
// The division is replaced by a multiplication with 1 / scale wherever that cannot change the code.
// With a normal fp16 scale |x / scale| < 128: the reciprocal, the quotient and either sum with 127.5
// are each off by at most 2^-17, so the two sums differ by at most 2^-15 and round to the same
// integer unless one lies within 2^-14 of a half-integer.  There (one weight in 8000, and every
// exact zero: 127.5), and for groups with a subnormal, zero or infinite scale, the lane divides.
// Rounding: t + 2^23 leaves the integer next to t in the low bits of the float.
// The maximum is taken on packed halves, codes are packed four at a time, and where the lane has a weight
// to divide for, only that one is divided (all sixteen, and as many codes in registers: 38.7 us).  Two
// groups per lane and four CTAs per SM: one group and six 34.5 us, four and three 37.8.
constexpr int QUANT_U = 2;  // groups in flight per lane
template <int LPG>
__global__ void __launch_bounds__(256, 4) quantize_u8_vec_kernel(uint8_t* q, __half* scales,
                                                                 const __half* in, int64_t groups) {
  constexpr int U = QUANT_U;
  constexpr int GPW = 32 / LPG;  // groups per warp and step
  constexpr float MAGIC = 8388608.0f, NEAR = 0.5f - 6.103515625e-05f;
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
    const uint32_t w[8] = {raw[u][0].x, raw[u][0].y, raw[u][0].z, raw[u][0].w,
                           raw[u][1].x, raw[u][1].y, raw[u][1].z, raw[u][1].w};
    __half2 top = __habs2(u32_as_half2(w[0]));
#pragma unroll
    for (int i = 1; i < 8; ++i) top = __hmax2(top, __habs2(u32_as_half2(w[i])));
    // (fmaxf from zero, like __hmax2, passes over NaN)
    float absmax = fmaxf(fmaxf(0.0f, __low2float(top)), __high2float(top));
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1) absmax = fmaxf(absmax, __shfl_xor_sync(0xffffffffu, absmax, o));
    const __half s = __float2half_rn(absmax / 127.5f);
    const float sf = __half2float(s);
    const float inv = 1.0f / sf;
    const bool normal = sf >= 6.103515625e-05f && sf <= 65504.0f;
    bool safe = normal;
    uint32_t codes[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2 h = u32_as_half2(w[2 * i + j / 2]);
        const float t = fmaf((j & 1) ? __high2float(h) : __low2float(h), inv, 127.5f);
        const float m = t + MAGIC;
        c[j] = __float_as_uint(m);
        safe = safe && fabsf(t - (m - MAGIC)) < NEAR;  // (false for NaN)
      }
      codes[i] = prmt(prmt(c[0], c[1], 0x0040u), prmt(c[2], c[3], 0x0040u), 0x5410u);
    }
    if (!safe && g0 + u * GPW < groups) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const __half2 h = u32_as_half2(w[i / 2]);
        const float x = (i & 1) ? __high2float(h) : __low2float(h);
        const float t = fmaf(x, inv, 127.5f);
        if (!(normal && fabsf(t - ((t + MAGIC) - MAGIC)) < NEAR)) {
          const uint32_t sel = 0x3210u & ~(0xFu << (4 * (i % 4)));
          codes[i / 4] = prmt(codes[i / 4], quantize_one(x, sf), sel | (4u << (4 * (i % 4))));
        }
      }
    }
    if (g0 + u * GPW < groups) {
      if (lane % LPG == 0) scales[g0 + u * GPW] = s;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<uint2*>(q + off0 + u * (GPW * 16 * LPG) + h * (8 * LPG)) =
            make_uint2(codes[2 * h], codes[2 * h + 1]);
    }
  }
}

}  // namespace

int launch_dequantize_u8(adr_ctx* ctx, cudaStream_t stream, __half* out, const __half* scales,
                         const __half* zeros, const uint8_t* q, int rows, int k, int block_size) {
  const int64_t pieces = (int64_t)rows * (k / 8), per_cta = 256 * DEQ_U;
  const int64_t grid = (pieces + per_cta - 1) / per_cta;
  if (grid > 0x7fffffffLL) return ADR_ERR_SHAPE;
  const unsigned per_block = (unsigned)block_size / 8;
  int shift = -1;
  if ((per_block & (per_block - 1)) == 0)
    for (shift = 0; (1u << shift) < per_block;) ++shift;
  const bool narrow = pieces + per_cta < 0xffffffffLL;  // piece numbers in 32 bits
  auto go = [&](auto kfn, auto n) {
    kfn<<<(unsigned)grid, 256, 0, stream>>>(out, scales, zeros, q, n, per_block, shift);
  };
  if (zeros) {
    if (narrow) go(dequantize_u8_kernel<true, uint32_t>, (uint32_t)pieces);
    else go(dequantize_u8_kernel<true, uint64_t>, (uint64_t)pieces);
  } else {
    if (narrow) go(dequantize_u8_kernel<false, uint32_t>, (uint32_t)pieces);
    else go(dequantize_u8_kernel<false, uint64_t>, (uint64_t)pieces);
  }
  return after_launch(ctx);
}

int launch_quantize_u8(adr_ctx* ctx, cudaStream_t stream, uint8_t* q, __half* scales,
                       const __half* in, int rows, int k, int block_size) {
  // 16 weights per lane where a block is a power of two of them within a warp and the buffers allow
  // 16-byte loads; any other block size or alignment takes the warp-per-group kernel
  const bool aligned = (reinterpret_cast<uintptr_t>(in) & 15u) == 0 && (reinterpret_cast<uintptr_t>(q) & 7u) == 0;
  const int lpg = block_size / 16;
  const int64_t groups = (int64_t)rows * (k / block_size);
  // (and so does a small tensor, whose groups make no more than a warp each for the GPU: a lane's sixteen weights are
  // a longer chain than a warp's four.  16 x 4096 in blocks of 128 2.2 / 3.1 us, 1024 x 512 2.9 / 3.3, 1024 x 1024, past
  // the line, 4.0 / 3.3)
  const bool small = groups <= 4096 && groups * block_size <= 1 << 20;
  if (aligned && !small && block_size % 16 == 0 && lpg <= 32 && (lpg & (lpg - 1)) == 0) {
    const int per_block = 8 * QUANT_U * (32 / lpg);
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
  const int64_t grid = (groups * 32 + 255) / 256;
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
