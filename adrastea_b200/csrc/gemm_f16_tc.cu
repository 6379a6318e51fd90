// fp16 strided/batched GEMM on the 5th-generation tensor cores:
//   out[b,y,x] = store(sum_k lhs[b,y,k] * rhs[b,k,x])
// replacing matmul_f16_fast / matmul_f16 (adrastea_kernels/cpp/matmul.cu:236-416,
// 493-513) and the WMMA kernels (matmul_nt_wmma_128x64x64.cu:8-78,
// matmul_nt_wmma_16x128x256.cu:8-68) for views TMA can describe.
//
// Tiles of 128 x BN outputs.  Warps are specialised:
//   warp 0    producer: one thread issues TMA loads of the A (128 x 64) and B (BN x 64)
//             k-blocks into a ring of 128-byte-swizzled shared-memory stages
//   warp 1    owns tensor memory (alloc/dealloc); one thread issues tcgen05.mma
//             (M = 128, N = BN, K = 16 per instruction, fp32 accumulators in TMEM) and
//             frees each stage with tcgen05.commit
//   warps 2.. epilogue: tcgen05.ld the accumulator (warp w reads TMEM lanes
//             32*(w%4)..+31 = tile rows), apply the reference's fused store op, mask
//             and scale, write fp16 to the (arbitrarily strided) output; eight warps in
//             the persistent kernel (two per lane quarter, alternating 32-column chunks),
//             four in the split-k kernel
// Three kernels share these roles (a fourth, for views TMA cannot describe, its MMA and epilogue):
//   gemm_f16_tc_kernel         persistent: one CTA per SM walks a list of tiles; two
//                              accumulator buffers in TMEM let the epilogue of one tile
//                              overlap the MMAs of the next
//   gemm_f16_pair_kernel       the same with a pair of CTAs per 256 x 256 tile, for large products
//   gemm_f16_tc_splitk_kernel  for grids that would leave most SMs idle (skinny m, prefill
//                              of a few hundred rows): a cluster of S CTAs splits k for one
//                              tile, the fp32 partial tiles are exchanged through distributed
//                              shared memory and added in rank order (deterministic, no
//                              scratch memory in HBM)
// Rows and k beyond the operands' extents are zero-filled by TMA, so m, n and k need no
// divisibility; only the 16-byte alignment rules of TMA apply (gemm_f16_tc_supports).
// Every mbarrier wait is bounded: a wait that runs out sets the context's status word,
// the kernel still frees its tensor memory and returns.
#include <algorithm>
#include <cmath>
#include <map>

#include "tcgen05.cuh"

namespace adr {

namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // fp16 elements: one 128-byte swizzle row
constexpr int TC_THREADS = 320;   // split-k kernel: producer, MMA, eight epilogue warps
constexpr int TCP_THREADS = 320;  // persistent kernel: producer, MMA, eight epilogue warps
constexpr size_t SMEM_BUDGET = 200 * 1024;
constexpr int EPI_LD = 34;                    // fp16 between rows of an epilogue warp's staging tile (17 words:
                                              // a row per lane and a column per lane are both conflict-free)
constexpr int EPI_TILE_BYTES = 32 * EPI_LD * 2;

template <int BN>
struct TcCfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (int)((SMEM_BUDGET - 2048) / STAGE_BYTES) > 8
                                    ? 8
                                    : (int)((SMEM_BUDGET - 2048) / STAGE_BYTES);
  static constexpr size_t SMEM = 1024 /*alignment slack*/ + (size_t)STAGES * STAGE_BYTES + 1024;
  static constexpr size_t EPI_OFF = (size_t)STAGES * STAGE_BYTES + 1024;  // persistent kernel, ragged rows: staging tiles
  static constexpr size_t SMEM_TILES = 1024 + EPI_OFF + 8 * EPI_TILE_BYTES;
  static constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;  // two accumulator buffers
  // split-k: the fp32 partial tile, row-major with rows padded by 4 floats (row pitch = 16
  // bytes mod 128) so that the 16-byte row-wise writes of 8 lanes hit distinct bank groups
  // and the remote reads of a warp are 512 contiguous bytes
  static constexpr int PART_LD = BN + 4;
  static constexpr size_t PART_BYTES = (size_t)BM * PART_LD * 4;
  static_assert(PART_BYTES <= (size_t)STAGES * STAGE_BYTES, "partial tile must fit in the ring");
};

struct TcParams {
  __half* out;
  const __half* bias;
  int batches, m, k, n;
  int s_ox, s_oy, s_oz;
  int a_bcast, b_bcast;  // operand is shared by all batches (z-stride 0)
  float beta, scale;
  uint32_t store, load, mask;
  unsigned int* status;
};

__device__ __forceinline__ __half half_lo(uint32_t w) { return __ushort_as_half((unsigned short)(w & 0xFFFFu)); }
__device__ __forceinline__ __half half_hi(uint32_t w) { return __ushort_as_half((unsigned short)(w >> 16)); }

// The epilogue of one accumulator tile for one warp: the warp's 32 TMEM lanes are 32 tile
// rows (one per thread), and it walks the 32-column chunks chunk0, chunk0 + 2, ...  The
// loads of the old output and of the bias are in flight while tcgen05.ld completes.
// QuickGelu uses the fast exponential and reciprocal (the tensor-core path is held to a
// tolerance, not to the bits of the sequential reference sum).
template <int STORE>
__device__ __forceinline__ __half epilogue_op(const TcParams& p, float a, __half old, float bias,
                                              __half hscale) {
  if constexpr (STORE == ADR_STORE_QUICK_GELU_BIAS) {
    const float t = __half2float(__float2half_rn(a)) + bias;
    return __float2half_rn(__fdividef(t, 1.0f + __expf(-1.702f * t)));
  } else {
    return store_apply<STORE>(a, old, bias, p.beta, hscale);
  }
}

// `bar` (optional): the barrier that says the accumulator is complete.  It is awaited here,
// after the old outputs of the warp's first chunk have been requested (later chunks request
// theirs under their tensor-memory load; requesting them a chunk ahead into a second register
// set spilled and measured slower).  BIAS_AHEAD: the bias of a chunk, 64 bytes, is requested a chunk ahead into a
// second register set; only in a kernel compiled for one store operation, where the registers are there.  Returns
// false if the wait ran out.
template <int STORE, int BN, bool BIAS_AHEAD = false>
__device__ __forceinline__ bool epilogue_tile(const TcParams& p, uint32_t tmem_acc, __half* orow,
                                              int y, int n0, int chunk0, float pre, __half hscale,
                                              uint64_t* bar = nullptr, unsigned parity = 0) {
  const bool causal = p.mask == ADR_MASK_CAUSAL;
  const bool row_ok = y < p.m;
  // tcgen05.ld and its wait are warp-collective: every branch that contains one must be
  // uniform across the warp, so the vector path is taken only when all live rows allow it
  const bool lane_vec = p.s_ox == 1 && (reinterpret_cast<uintptr_t>(orow) & 15u) == 0 &&
                        (!store_uses_bias(STORE) || (reinterpret_cast<uintptr_t>(p.bias) & 15u) == 0);
  const bool row_vec = __all_sync(0xffffffffu, lane_vec || !row_ok);
  const __half ninf = __ushort_as_half((unsigned short)0xFC00);
  constexpr int NCH = (BN / 32 + 1) / 2;  // chunks per warp (chunk0, chunk0 + 2, ...)
  uint4 oldw[4], biasw[BIAS_AHEAD ? 2 : 1][4];
  auto prefetch_bias = [&](int c, uint4 (&bsv)[4]) {
    const int x0 = n0 + c * 32;
    if (c < BN / 32 && row_vec && x0 + 32 <= p.n && row_ok) {
#pragma unroll
      for (int q = 0; q < 4; ++q) bsv[q] = reinterpret_cast<const uint4*>(p.bias + x0)[q];
    }
  };
  if (store_uses_bias(STORE)) prefetch_bias(chunk0, biasw[0]);
  auto prefetch = [&](int c, uint4 (&o)[4]) {
    const int x0 = n0 + c * 32;
    if (c < BN / 32 && row_vec && x0 + 32 <= p.n && row_ok) {
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = reinterpret_cast<const uint4*>(orow + x0)[q];
    }
  };
  if (store_reads_out(STORE)) prefetch(chunk0, oldw);
  if (bar) {
    if (!mbar_wait(bar, parity)) return false;
    tc_fence_after_sync();
  }
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    const int c = chunk0 + 2 * i;
    if (c >= BN / 32) break;
    const int x0 = n0 + c * 32;
    if (x0 >= p.n) break;  // uniform across the warp
    uint32_t acc[32];
    __syncwarp();
    tmem_ld_32x32(tmem_acc + (uint32_t)(c * 32), acc);
    if (i > 0 && store_reads_out(STORE)) prefetch(c, oldw);
    if (BIAS_AHEAD) {
      if (i + 1 < NCH) prefetch_bias(c + 2, biasw[(i + 1) & 1]);
    } else if (i > 0 && store_uses_bias(STORE)) {
      prefetch_bias(c, biasw[0]);
    }
    if (row_vec && x0 + 32 <= p.n) {
      __syncwarp();
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (!row_ok) break;
        const uint4 oq = oldw[q], bq = biasw[BIAS_AHEAD ? (i & 1) : 0][q];
        const uint32_t ow[4] = {oq.x, oq.y, oq.z, oq.w};
        const uint32_t bw[4] = {bq.x, bq.y, bq.z, bq.w};
        uint32_t rw[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = q * 8 + e * 2;
          const float a0 = __uint_as_float(acc[j]) * pre, a1 = __uint_as_float(acc[j + 1]) * pre;
          const float b0 = store_uses_bias(STORE) ? __half2float(half_lo(bw[e])) : 0.0f;
          const float b1 = store_uses_bias(STORE) ? __half2float(half_hi(bw[e])) : 0.0f;
          const __half o0 = store_reads_out(STORE) ? half_lo(ow[e]) : __float2half_rn(0.0f);
          const __half o1 = store_reads_out(STORE) ? half_hi(ow[e]) : __float2half_rn(0.0f);
          __half r0 = epilogue_op<STORE>(p, a0, o0, b0, hscale);
          __half r1 = epilogue_op<STORE>(p, a1, o1, b1, hscale);
          if (causal && x0 + j > y) r0 = ninf;
          if (causal && x0 + j + 1 > y) r1 = ninf;
          rw[e] = (uint32_t)__half_as_ushort(r0) | ((uint32_t)__half_as_ushort(r1) << 16);
        }
        reinterpret_cast<uint4*>(orow + x0)[q] = make_uint4(rw[0], rw[1], rw[2], rw[3]);
      }
    } else {
      // strided, unaligned or ragged rows: one element at a time
      __syncwarp();
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int x = x0 + j;
        if (row_ok && x < p.n) {
          __half* dst = orow + (int64_t)x * p.s_ox;
          const float bias = store_uses_bias(STORE) ? __half2float(p.bias[x]) : 0.0f;
          const __half old = store_reads_out(STORE) ? *dst : __float2half_rn(0.0f);
          __half r = epilogue_op<STORE>(p, __uint_as_float(acc[j]) * pre, old, bias, hscale);
          if (causal && x > y) r = ninf;
          *dst = r;
        }
      }
    }
  }
  return true;
}

// Whether the rows of the output are neither 16-byte aligned nor strided: they go through
// epilogue_ragged.  (STORE_NT_BETA rounds once, from fp32, and has dense outputs: it stays above.)
__host__ __device__ __forceinline__ bool rows_ragged(const TcParams& p) {
  return p.s_ox == 1 && p.store != STORE_NT_BETA &&
         ((reinterpret_cast<uintptr_t>(p.out) & 15u) != 0 || p.s_oy % 8 != 0 || p.s_oz % 8 != 0);
}

// The epilogue of one tile for unaligned rows (a 514-byte pitch): the fp16 accumulators of 32 rows x 32
// columns go through the warp's staging tile, so that an instruction reads or writes 32 columns of ONE row.
// With a row per lane, 32 distinct lines per 2-byte instruction, the SM's load-store unit was busy for
// longer than everything else: q.k^T of 16 heads, 257 x 257 x 64: 21.2 -> 6.5 us.
template <int BN>
__device__ __forceinline__ bool epilogue_ragged(const TcParams& p, uint32_t tmem_acc, __half* orow, int y,
                                                int n0, int chunk0, float pre, __half hscale, uint8_t* tile,
                                                uint64_t* bar, unsigned parity) {
  const int lane = threadIdx.x & 31, store = (int)p.store;
  const bool reads = store_reads_out(store), biased = store_uses_bias(store);
  const bool causal = p.mask == ADR_MASK_CAUSAL;
  const int rows = min(32, p.m - (y - lane));  // of this warp; not positive: none
  // identity and scale are applied before the tile (identity: times one, exactly), the rest behind it
  const bool simple = store == ADR_STORE_IDENTITY || store == ADR_STORE_SCALE;
  const __half2 factor = __half2half2(store == ADR_STORE_SCALE ? hscale : __float2half_rn(1.0f));
  const __half ninf = __ushort_as_half((unsigned short)0xFC00);
  uint32_t* words = reinterpret_cast<uint32_t*>(tile) + lane * (EPI_LD / 2);
  const __half* column = reinterpret_cast<const __half*>(tile) + lane;
  if (bar) {
    if (!mbar_wait(bar, parity)) return false;
    tc_fence_after_sync();
  }
#pragma unroll 1
  for (int c = chunk0; c < BN / 32; c += 2) {
    const int x = n0 + c * 32 + lane;
    if (x - lane >= p.n) break;  // uniform across the warp
    uint32_t acc[32];
    __syncwarp();
    tmem_ld_32x32(tmem_acc + (uint32_t)(c * 32), acc);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      __half2 h = __floats2half2_rn(__uint_as_float(acc[2 * j]) * pre, __uint_as_float(acc[2 * j + 1]) * pre);
      if (simple) {
        const int xj = x - lane + 2 * j;
        h = __hmul2(h, factor);
        if (causal && xj > y) h.x = ninf;
        if (causal && xj + 1 > y) h.y = ninf;
      }
      words[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    __syncwarp();
    if (x < p.n && simple) {
      __half* dst = orow - (int64_t)lane * p.s_oy + x;
#pragma unroll
      for (int r = 0; r < 32; ++r)
        if (r < rows) dst[(int64_t)r * p.s_oy] = column[r * EPI_LD];
    } else if (x < p.n) {
      const float bias = biased ? __half2float(p.bias[x]) : 0.0f;
      __half* dst = orow - (int64_t)lane * p.s_oy + x;
      for (int r0 = 0; r0 < rows; r0 += 8) {
        __half old[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          old[i] = reads && r0 + i < rows ? dst[(int64_t)(r0 + i) * p.s_oy] : __float2half_rn(0.0f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = r0 + i;
          __half v = store_apply_rt(store, __half2float(column[r * EPI_LD]), old[i], bias, p.beta, hscale);
          if (causal && x > y - lane + r) v = ninf;
          if (r < rows) dst[(int64_t)r * p.s_oy] = v;
        }
      }
    }
    __syncwarp();
  }
  return true;
}

template <int BN>
__device__ __forceinline__ bool epilogue_tile_rt(const TcParams& p, uint32_t tmem_acc, __half* orow,
                                                 int y, int n0, int chunk0, float pre,
                                                 __half hscale, uint64_t* bar = nullptr,
                                                 unsigned parity = 0) {
  switch (p.store) {
    case ADR_STORE_SCALE: return epilogue_tile<ADR_STORE_SCALE, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    case ADR_STORE_ADD: return epilogue_tile<ADR_STORE_ADD, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    case ADR_STORE_BETA_BIAS: return epilogue_tile<ADR_STORE_BETA_BIAS, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    case ADR_STORE_BETA_GELU_BIAS: return epilogue_tile<ADR_STORE_BETA_GELU_BIAS, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    case ADR_STORE_QUICK_GELU_BIAS: return epilogue_tile<ADR_STORE_QUICK_GELU_BIAS, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    case STORE_NT_BETA: return epilogue_tile<STORE_NT_BETA, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
    default: return epilogue_tile<ADR_STORE_IDENTITY, BN>(p, tmem_acc, orow, y, n0, chunk0, pre, hscale, bar, parity);
  }
}

// Issues the four K=16 MMAs of one 64-wide k-block held in stage memory at `sa`.
// B_MN: the B stage holds an N-contiguous operand as BN/64 chunks of [64 k][64 n] (8 KB each).
template <int BN, bool B_MN>
__device__ __forceinline__ void mma_k_block(uint32_t tmem_d, uint32_t sa, bool first) {
  constexpr uint32_t idesc = umma_idesc_f16(BN, B_MN);
  const uint64_t adesc = umma_desc_k_sw128(sa);
  const uint64_t bdesc = B_MN ? umma_desc_mn_sw128(sa + TcCfg<BN>::A_BYTES, 8192)
                              : umma_desc_k_sw128(sa + TcCfg<BN>::A_BYTES);
  // per K=16 step: a k-major tile moves 32 bytes along its swizzled rows (+2 in the address
  // field), an n-major tile moves 16 k-rows of 128 bytes (+128)
  constexpr uint64_t b_step = B_MN ? 128 : 2;
#pragma unroll
  for (int kk = 0; kk < BK / 16; ++kk) {
    umma_f16(tmem_d, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)kk * b_step, idesc,
             (!first || kk > 0) ? 1u : 0u);
  }
}

// One k-block of B into stage memory at `sb`.
template <int BN, bool B_MN>
__device__ __forceinline__ void load_b_block(uint8_t* sb, const CUtensorMap* map_b, int kb, int n0,
                                             int bz, uint64_t* bar) {
  if (B_MN) {
#pragma unroll
    for (int c = 0; c < BN / 64; ++c) tma_load_3d(sb + c * 8192, map_b, n0 + c * 64, kb * BK, bz, bar);
  } else {
    tma_load_3d(sb, map_b, kb * BK, n0, bz, bar);
  }
}

// Persistent tile scheduler: CTA c works on tiles c, c + gridDim.x, ...  Tiles are numbered
// batch-major, then in groups of GROUP_M row tiles swept along n, so that the tiles in
// flight at one time share A and B panels in L2.
struct TileCoord {
  int m0, n0, b;
};
constexpr int GROUP_M = 8;
__device__ __forceinline__ TileCoord tile_coord(int t, int mt, int nt, int bn) {
  const int per_batch = mt * nt;
  const int b = t / per_batch;
  const int r = t - b * per_batch;
  const int group = r / (GROUP_M * nt);
  const int first_m = group * GROUP_M;
  const int gsz = min(GROUP_M, mt - first_m);
  const int local = r - group * GROUP_M * nt;
  return {(first_m + local % gsz) * BM, (local / gsz) * bn, b};
}

// EPILOGUE: the one store operation that the kernel is compiled for; EPI_ANY, chosen at run time; EPI_RAGGED, rows
// that go through epilogue_ragged.  (Chosen at run time, that one made the kernel spill registers and cost aligned
// outputs 5 to 8 %: 3000 x 512 x 4096 23.8 us, compiled apart 22.3.)
constexpr int EPI_ANY = -1, EPI_RAGGED = -2;
template <int BN, bool B_MN, int EPILOGUE>
__global__ void __launch_bounds__(TCP_THREADS, 1)
    gemm_f16_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                       const __grid_constant__ CUtensorMap map_b, TcParams p) {
  using Cfg = TcCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stages = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + (size_t)Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_full = empty_bar + Cfg::STAGES;  // [2]: accumulator buffer complete
  uint64_t* acc_empty = acc_full + 2;            // [2]: accumulator buffer drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.k + BK - 1) / BK;
  const int mt = (p.m + BM - 1) / BM, nt = (p.n + BN - 1) / BN;
  const int total_tiles = mt * nt * p.batches;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);  // one arrival per epilogue warp
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait_trigger();
  bool ok = true;

  if (warp == 0) {
    // ---------------- producer: TMA loads, one ring across all of this CTA's tiles ----------
    if (lane == 0) {
      int it = 0;  // k-blocks issued so far
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const TileCoord tc = tile_coord(t, mt, nt, BN);
        const int az = p.a_bcast ? 0 : tc.b, bz = p.b_bcast ? 0 : tc.b;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % Cfg::STAGES;
          const unsigned phase = (unsigned)(it / Cfg::STAGES) & 1u;
          if (!mbar_wait(&empty_bar[s], phase ^ 1u)) { ok = false; break; }
          uint8_t* sa = stages + (size_t)s * Cfg::STAGE_BYTES;
          mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
          tma_load_3d(sa, &map_a, kb * BK, tc.m0, az, &full_bar[s]);
          load_b_block<BN, B_MN>(sa + Cfg::A_BYTES, &map_b, kb, tc.n0, bz, &full_bar[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issue: alternate between two accumulator buffers in TMEM ----------
    if (lane == 0) {
      int it = 0, local = 0;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
        const int buf = local & 1;
        const unsigned use = (unsigned)(local >> 1) & 1u;
        if (!mbar_wait(&acc_empty[buf], use ^ 1u)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % Cfg::STAGES;
          const unsigned phase = (unsigned)(it / Cfg::STAGES) & 1u;
          if (!mbar_wait(&full_bar[s], phase)) { ok = false; break; }
          tc_fence_after_sync();
          mma_k_block<BN, B_MN>(tmem_d, smem_u32(stages + (size_t)s * Cfg::STAGE_BYTES), kb == 0);
          umma_commit(&empty_bar[s]);  // the stage is free once these MMAs have read it
        }
        umma_commit(&acc_full[buf]);  // the accumulator is complete once every MMA is done
      }
    }
  } else {
    // ---------------- epilogue: drains one buffer while the other is being filled ----------
    // Warps 2-5 take the even 32-column chunks of the tile, warps 6-9 the odd ones.
    const int quarter = warp & 3;  // TMEM lanes a warp may read: 32 * (warp id % 4) ..
    const int chunk0 = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const __half hscale = __float2half_rn(p.scale);
    // a load-side scale multiplies both operands (matmul.cu:62): s^2 on the product
    const float hs = __half2float(hscale);
    const float pre = p.load == ADR_LOAD_SCALE ? hs * hs : 1.0f;
    int local = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++local) {
      const TileCoord tc = tile_coord(t, mt, nt, BN);
      const int buf = local & 1;
      const unsigned use = (unsigned)(local >> 1) & 1u;
      const int y = tc.m0 + row;
      __half* orow = p.out + (int64_t)tc.b * p.s_oz + (int64_t)y * p.s_oy;
      // (the accumulator's barrier is awaited inside, behind the first loads of old outputs)
      const uint32_t tacc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN);
      bool done;
      if constexpr (EPILOGUE == EPI_RAGGED)
        done = epilogue_ragged<BN>(p, tacc, orow, y, tc.n0, chunk0, pre, hscale,
                                   smem + Cfg::EPI_OFF + (warp - 2) * EPI_TILE_BYTES, &acc_full[buf], use);
      else if constexpr (EPILOGUE == EPI_ANY)
        done = epilogue_tile_rt<BN>(p, tacc, orow, y, tc.n0, chunk0, pre, hscale, &acc_full[buf], use);
      else
        done = epilogue_tile<EPILOGUE, BN, true>(p, tacc, orow, y, tc.n0, chunk0, pre, hscale, &acc_full[buf], use);
      if (!done) {
        ok = false;
        break;
      }
      // this warp's reads of the buffer are complete: hand it back to the MMA warp
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }
  if (!ok) atomicOr(p.status, 2u);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------
// Large products: a PAIR of CTAs (two SMs) per 256 x 256 tile, tcgen05.mma.cta_group::2.  With one CTA
// per 128 x 256 tile the shared memory is the bound: per 128 x 256 x 16 MMA the tensor core reads 4 KB
// of A and 8 KB of B and TMA writes as much, 24 KB against the 16 KB that 128 bytes per clock give in
// the 128 clocks of the MMA.  In a pair each SM holds its 128 rows of A and HALF of B (the tensor
// cores exchange the halves), 8 KB read and 8 KB written per 128 clocks.
// Roles as above, in both CTAs, except that one thread of CTA 0 issues the MMAs of both:
//   * each CTA's producer loads its own halves; the copies of both complete on CTA 0's barrier;
//   * a commit arrives in both CTAs (the stage is free / the accumulator is complete);
//   * the sixteen epilogue warps of the pair hand the accumulator back to CTA 0's barrier.
// The epilogue goes through shared memory: a warp turns 32 rows x 32 columns at a time into fp16,
// writes them to a swizzled 2 KB tile and stores it by TMA; store operations that read the old output
// get it the same way, loaded into that tile by TMA a chunk ahead.  Row-wise 16-byte accesses, one
// row per lane, cost a 32-byte sector each way for half its bytes.
// Measured against one CTA per 128 x 256 tile (cold L2, identity / bias with the old output read):
// 2048 x 4096 x 4096 60.5 / 64.7 -> 50.2 / 54.2 us, 8192 x 22016 x 4096 1186 / 1248 -> 1012 / 1057 us
// (1.46 PFLOP/s), 16448 x 3072 x 1024 101 / 129 -> 86 / 95 us.  What bounds it now: the tensor cores
// and, over many launches, the power limit.
// ---------------------------------------------------------------------------------------
constexpr int PR_BN = 256;
constexpr int PR_A_BYTES = BM * BK * 2;
constexpr int PR_STAGE_BYTES = 2 * PR_A_BYTES;  // A half and B half
constexpr int PR_STAGES = 6;
constexpr int PR_TILE_BYTES = 32 * 32 * 2;      // staging tile of an epilogue warp
constexpr size_t PR_SMEM = 1024 + (size_t)PR_STAGES * PR_STAGE_BYTES + 8 * 2 * PR_TILE_BYTES + 512;

// What one epilogue warp carries from tile to tile.
struct PairEpilogue {
  uint8_t* buf;    // two staging tiles
  uint64_t* bar;   // two barriers: the old outputs have landed in the tile
  unsigned count;  // chunks done: tile count & 1, parity (count >> 1) & 1
};

// The chunks chunk0, chunk0 + 2, ... (32 columns) of one accumulator tile for one warp (TMEM lanes =
// rows y0 .. y0 + 31).  Returns false if a wait ran out.  (Compiled for each store operation: choosing it
// per element at run time made the epilogue of a scaled product four times as long, q.k^T of 32 heads,
// 1000 x 1000 x 128: 121 us against 27.4.)
template <int STORE>
__device__ __forceinline__ bool pair_epilogue_tile(const TcParams& p, const CUtensorMap* map_o,
                                                   PairEpilogue& st, uint32_t tmem_acc, int y0, int n0,
                                                   int bz, int chunk0, float pre, __half hscale,
                                                   uint64_t* acc_full, unsigned parity,
                                                   uint32_t acc_empty) {
  constexpr int NCH = PR_BN / 64;
  const int lane = threadIdx.x & 31;
  constexpr bool reads = store_reads_out(STORE), biased = store_uses_bias(STORE);
  const bool causal = p.mask == ADR_MASK_CAUSAL;
  const int y = y0 + lane;
  const __half ninf = __ushort_as_half((unsigned short)0xFC00);
  const bool bias_vec = (reinterpret_cast<uintptr_t>(p.bias) & 15u) == 0;
  const int swz = (lane >> 1) & 3;
  auto x_of = [&](int i) { return n0 + (chunk0 + 2 * i) * 32; };
  auto load_old = [&](int i, unsigned count) {  // lane 0
    uint64_t* bar = st.bar + (count & 1);
    mbar_expect_tx(bar, PR_TILE_BYTES);
    tma_load_3d(st.buf + (count & 1) * PR_TILE_BYTES, map_o, x_of(i), y0, bz, bar);
  };
  // (rows wholly outside the output: nothing to read or write, the accumulator is still handed back)
  const bool rows_live = y0 < p.m;
  if (reads && rows_live && x_of(0) < p.n && lane == 0) {
    bulk_wait_read<1>();  // the store before the last one used this tile
    load_old(0, st.count);
  }
  if (!mbar_wait(acc_full, parity)) {
    // (old outputs on their way to the tile are awaited all the same, here as below)
    if (reads && rows_live && x_of(0) < p.n) mbar_wait(st.bar + (st.count & 1), (st.count >> 1) & 1u);
    return false;
  }
  tc_fence_after_sync();
  bool ok = true;
  bool released = false;
#pragma unroll 1
  for (int i = 0; i < NCH; ++i) {
    const int x0 = x_of(i);
    if (x0 >= p.n || !rows_live) break;  // uniform across the warp
    uint32_t acc[32];
    __syncwarp();
    tmem_ld_32x32(tmem_acc + (uint32_t)((chunk0 + 2 * i) * 32), acc);
    if (lane == 0) {
      if (!reads) {
        bulk_wait_read<1>();
      } else if (i + 1 < NCH && x_of(i + 1) < p.n) {
        bulk_wait_read<0>();
        load_old(i + 1, st.count + 1);
      }
    }
    uint4 bv[4];
    if (biased) {
      if (bias_vec && x0 + 32 <= p.n) {
#pragma unroll
        for (int q = 0; q < 4; ++q) bv[q] = reinterpret_cast<const uint4*>(p.bias + x0)[q];
      } else {
        unsigned short* bh = reinterpret_cast<unsigned short*>(bv);
#pragma unroll
        for (int j = 0; j < 32; ++j)
          bh[j] = x0 + j < p.n ? reinterpret_cast<const unsigned short*>(p.bias)[x0 + j] : (unsigned short)0;
      }
    }
    tmem_ld_wait();
    if (i + 1 == NCH || x_of(i + 1) >= p.n) {
      // this warp's reads of the accumulator are complete
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty);
      released = true;
    }
    uint8_t* row = st.buf + (st.count & 1) * PR_TILE_BYTES + lane * 64;
    if (reads) ok = mbar_wait(st.bar + (st.count & 1), (st.count >> 1) & 1u) && ok;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint4* cell = reinterpret_cast<uint4*>(row + ((q ^ swz) << 4));
      uint4 oq = make_uint4(0, 0, 0, 0);
      if (reads) oq = *cell;
      const uint32_t ow[4] = {oq.x, oq.y, oq.z, oq.w};
      const uint32_t bw[4] = {bv[q].x, bv[q].y, bv[q].z, bv[q].w};
      uint32_t rw[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = q * 8 + e * 2;
        const float a0 = __uint_as_float(acc[j]) * pre, a1 = __uint_as_float(acc[j + 1]) * pre;
        const float b0 = biased ? __half2float(half_lo(bw[e])) : 0.0f;
        const float b1 = biased ? __half2float(half_hi(bw[e])) : 0.0f;
        __half r0 = epilogue_op<STORE>(p, a0, half_lo(ow[e]), b0, hscale);
        __half r1 = epilogue_op<STORE>(p, a1, half_hi(ow[e]), b1, hscale);
        if (causal && x0 + j > y) r0 = ninf;
        if (causal && x0 + j + 1 > y) r1 = ninf;
        rw[e] = (uint32_t)__half_as_ushort(r0) | ((uint32_t)__half_as_ushort(r1) << 16);
      }
      *cell = make_uint4(rw[0], rw[1], rw[2], rw[3]);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      tma_store_3d(map_o, st.buf + (st.count & 1) * PR_TILE_BYTES, x0, y0, bz);
      bulk_commit();
    }
    ++st.count;
  }
  if (!released) {
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(acc_empty);
  }
  return ok;
}

template <bool B_MN, int STORE>
__global__ void __launch_bounds__(TCP_THREADS, 1)
    gemm_f16_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         const __grid_constant__ CUtensorMap map_o, TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stages = smem;
  uint8_t* staging = smem + (size_t)PR_STAGES * PR_STAGE_BYTES;  // [8 warps][2 tiles]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + 8 * 2 * PR_TILE_BYTES);  // (CTA 0's are used)
  uint64_t* empty_bar = full_bar + PR_STAGES;
  uint64_t* acc_full = empty_bar + PR_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;          // [2] (CTA 0's are used)
  uint64_t* old_full = acc_empty + 2;          // [8 warps][2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(old_full + 16);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_kb = (p.k + BK - 1) / BK;
  const int mt = (p.m + 2 * BM - 1) / (2 * BM), nt = (p.n + PR_BN - 1) / PR_BN;
  const int total_tiles = mt * nt * p.batches;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    tma_prefetch_desc(&map_o);
    for (int s = 0; s < PR_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 16);  // one arrival per epilogue warp of the pair
    }
    for (int i = 0; i < 16; ++i) mbar_init(&old_full[i], 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before_sync();
  cluster_arrive_wait();  // both CTAs' barriers exist
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait_trigger();
  bool ok = true;

  // tile t of the list: (row tile, column tile, batch), grouped as in tile_coord
  auto coord = [&](int t) {
    const int per_batch = mt * nt;
    const int b = t / per_batch;
    const int r = t - b * per_batch;
    const int group = r / (GROUP_M * nt);
    const int first_m = group * GROUP_M;
    const int gsz = min(GROUP_M, mt - first_m);
    const int local = r - group * GROUP_M * nt;
    return TileCoord{(first_m + local % gsz) * (2 * BM), (local / gsz) * PR_BN, b};
  };

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      for (int t = pair; t < total_tiles && ok; t += pairs) {
        const TileCoord tc = coord(t);
        const int az = p.a_bcast ? 0 : tc.b, bz = p.b_bcast ? 0 : tc.b;
        const int m0 = tc.m0 + rank * BM, n0 = tc.n0 + rank * (PR_BN / 2);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % PR_STAGES;
          if (!mbar_wait(&empty_bar[s], ((unsigned)(it / PR_STAGES) & 1u) ^ 1u)) { ok = false; break; }
          uint8_t* sa = stages + (size_t)s * PR_STAGE_BYTES;
          const uint32_t bar = cluster_addr(&full_bar[s], 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * PR_STAGE_BYTES);
          tma_load_3d_pair(sa, &map_a, kb * BK, m0, az, bar);
          if (B_MN) {
            tma_load_3d_pair(sa + PR_A_BYTES, &map_b, n0, kb * BK, bz, bar);
            tma_load_3d_pair(sa + PR_A_BYTES + 8192, &map_b, n0 + 64, kb * BK, bz, bar);
          } else {
            tma_load_3d_pair(sa + PR_A_BYTES, &map_b, kb * BK, n0, bz, bar);
          }
        }
      }
      // Nothing may be on its way to this pair's shared memory when it ends: no copy, and no arrival of
      // CTA 0's commits in CTA 1 (that of acc_full, which the epilogue awaits, does not say that the earlier
      // ones have arrived).  So the last fill of every stage is awaited until its MMAs have handed it back.
      // If that runs out, its copies at least are awaited: those of both CTAs complete on CTA 0's barrier.
      // (After one wait has run out the others are only looked at.)
      bool copies_ok = true;
      for (int f = max(0, it - PR_STAGES); f < it; ++f) {
        uint64_t *handed_back = &empty_bar[f % PR_STAGES], *landed = &full_bar[f % PR_STAGES];
        const unsigned use = (unsigned)(f / PR_STAGES) & 1u;
        if (ok ? mbar_wait(handed_back, use) : mbar_try_wait(handed_back, use)) continue;
        ok = false;
        if (rank == 0) copies_ok = copies_ok ? mbar_wait(landed, use) : mbar_try_wait(landed, use);
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = umma_idesc_f16_pair(PR_BN, B_MN);
      constexpr uint64_t b_step = B_MN ? 128 : 2;
      int it = 0, local = 0;
      for (int t = pair; t < total_tiles && ok; t += pairs, ++local) {
        const int buf = local & 1;
        if (!mbar_wait(&acc_empty[buf], ((unsigned)(local >> 1) & 1u) ^ 1u)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * PR_BN);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % PR_STAGES;
          if (!mbar_wait(&full_bar[s], (unsigned)(it / PR_STAGES) & 1u)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(stages + (size_t)s * PR_STAGE_BYTES);
          const uint64_t adesc = umma_desc_k_sw128(sa);
          const uint64_t bdesc = B_MN ? umma_desc_mn_sw128(sa + PR_A_BYTES, 8192) : umma_desc_k_sw128(sa + PR_A_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_f16_pair(tmem_d, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)kk * b_step, idesc,
                          (kb > 0 || kk > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s]);
        }
        umma_commit_pair(&acc_full[buf]);
      }
    }
  } else {
    const int quarter = warp & 3, chunk0 = (warp - 2) >> 2;
    PairEpilogue st{staging + (warp - 2) * 2 * PR_TILE_BYTES, old_full + (warp - 2) * 2, 0u};
    const __half hscale = __float2half_rn(p.scale);
    const float hs = __half2float(hscale);
    const float pre = p.load == ADR_LOAD_SCALE ? hs * hs : 1.0f;
    int local = 0;
    for (int t = pair; t < total_tiles; t += pairs, ++local) {
      const TileCoord tc = coord(t);
      const int buf = local & 1;
      ok = pair_epilogue_tile<STORE>(p, &map_o, st,
                                     tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * PR_BN),
                                     tc.m0 + rank * BM + quarter * 32, tc.n0, tc.b, chunk0, pre, hscale,
                                     &acc_full[buf], (unsigned)(local >> 1) & 1u,
                                     cluster_addr(&acc_empty[buf], 0));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
    }
    if (lane == 0) bulk_wait_all();
  }
  if (!ok) atomicOr(p.status, 2u);
  __syncwarp();
  tc_fence_before_sync();
  cluster_arrive_wait();  // the peer's tiles, barriers and tensor memory are in use until here
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Split-k: grid (S, n tiles, m tiles * batches), cluster (S, 1, 1).  CTA `rank` of a cluster
// accumulates k-blocks [rank*num_kb/S, (rank+1)*num_kb/S) of its tile.
template <int BN, bool B_MN>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_f16_tc_splitk_kernel(const __grid_constant__ CUtensorMap map_a,
                              const __grid_constant__ CUtensorMap map_b, TcParams p, int S) {
  using Cfg = TcCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stages = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + (size_t)Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_full = empty_bar + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x;
  const int mt = (p.m + BM - 1) / BM;
  const int n0 = blockIdx.y * BN, m0 = (blockIdx.z % mt) * BM, b = blockIdx.z / mt;
  const int num_kb = (p.k + BK - 1) / BK;
  const int kb0 = (int)((long long)rank * num_kb / S);
  const int kb1 = (int)((long long)(rank + 1) * num_kb / S);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait_trigger();
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      const int az = p.a_bcast ? 0 : b, bz = p.b_bcast ? 0 : b;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0;
        const int s = it % Cfg::STAGES;
        const unsigned phase = (unsigned)(it / Cfg::STAGES) & 1u;
        if (!mbar_wait(&empty_bar[s], phase ^ 1u)) { ok = false; break; }
        uint8_t* sa = stages + (size_t)s * Cfg::STAGE_BYTES;
        mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
        tma_load_3d(sa, &map_a, kb * BK, m0, az, &full_bar[s]);
        load_b_block<BN, B_MN>(sa + Cfg::A_BYTES, &map_b, kb, n0, bz, &full_bar[s]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0;
        const int s = it % Cfg::STAGES;
        const unsigned phase = (unsigned)(it / Cfg::STAGES) & 1u;
        if (!mbar_wait(&full_bar[s], phase)) { ok = false; break; }
        tc_fence_after_sync();
        mma_k_block<BN, B_MN>(tmem_base, smem_u32(stages + (size_t)s * Cfg::STAGE_BYTES), kb == kb0);
        umma_commit(&empty_bar[s]);
      }
      umma_commit(acc_full);
    }
  }
  // ---- every warp: wait until the accumulator is complete (so the ring is idle too) ----
  ok = mbar_wait(acc_full, 0) && ok;
  tc_fence_after_sync();
  __syncthreads();  // producer and MMA threads are past their loops: the ring can be reused
  float* part = reinterpret_cast<float*>(stages);  // [BM][PART_LD], row-major, padded
  const int live = min(BM, p.m - m0);              // rows of the tile that the output has
  if (warp >= 2 && (warp & 3) * 32 < live) {
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
#pragma unroll 1
    for (int c = (warp - 2) >> 2; c < BN / 32; c += 2) {
      uint32_t acc[32];
      tmem_ld_32x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 32), acc);
      tmem_ld_wait();
      float4* dst = reinterpret_cast<float4*>(part + (size_t)row * Cfg::PART_LD + c * 32);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        dst[q] = make_float4(__uint_as_float(acc[4 * q]), __uint_as_float(acc[4 * q + 1]),
                             __uint_as_float(acc[4 * q + 2]), __uint_as_float(acc[4 * q + 3]));
    }
  }
  if (!ok) atomicOr(p.status, 4u);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");

  // ---- the live rows are shared out among the ranks, who sum the S partial tiles in rank order.  A
  // thread takes four consecutive columns, two such pieces at a time; a warp reads 512 contiguous bytes
  // per peer.  (This part is most of the kernel's time at a few hundred KB of weights per CTA.  With four
  // warps, one piece at a time, 2-byte stores and the rows shared out dead or alive, 64 x 4096 x 4096 took
  // 15.5 us, now 13.4.)
  {
    constexpr int U = 2, CPR = BN / 4;
    const int rpr = (live + S - 1) / S, row_end = min(live, (rank + 1) * rpr);
    const int items = max(0, row_end - rank * rpr) * CPR;
    const uint32_t pbase = smem_u32(part);
    const __half hscale = __float2half_rn(p.scale);
    const float hs = __half2float(hscale);
    const float pre = p.load == ADR_LOAD_SCALE ? hs * hs : 1.0f;
    const bool causal = p.mask == ADR_MASK_CAUSAL;
    const int store = (int)p.store;
    const bool rd_out = store_reads_out(store), use_bias = store_uses_bias(store);
    __half* obase = p.out + (int64_t)b * p.s_oz;
    for (int e0 = threadIdx.x; e0 < items; e0 += TC_THREADS * U) {
      // all remote reads are issued before the first is used, then added in rank order
      float4 pv[U][8];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * TC_THREADS, col = (e % CPR) * 4, row = rank * rpr + e / CPR;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          pv[u][r] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < S && e < items) {
            uint32_t remote;
            asm("mapa.shared::cluster.u32 %0, %1, %2;"
                : "=r"(remote)
                : "r"(pbase + (uint32_t)(row * Cfg::PART_LD + col) * 4u), "r"(r));
            asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                         : "=f"(pv[u][r].x), "=f"(pv[u][r].y), "=f"(pv[u][r].z), "=f"(pv[u][r].w)
                         : "r"(remote));
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * TC_THREADS;
        const int x0 = n0 + (e % CPR) * 4, y = m0 + rank * rpr + e / CPR;
        if (e >= items || x0 >= p.n) continue;
        float v[4] = {pv[u][0].x, pv[u][0].y, pv[u][0].z, pv[u][0].w};
#pragma unroll
        for (int r = 1; r < 8; ++r)
          if (r < S) {
            v[0] += pv[u][r].x;
            v[1] += pv[u][r].y;
            v[2] += pv[u][r].z;
            v[3] += pv[u][r].w;
          }
        __half* dst = obase + (int64_t)y * p.s_oy + (int64_t)x0 * p.s_ox;
        const bool vec = p.s_ox == 1 && x0 + 4 <= p.n && (reinterpret_cast<uintptr_t>(dst) & 7u) == 0;
        __align__(8) __half old[4], res[4];
        if (rd_out && vec) *reinterpret_cast<uint2*>(old) = *reinterpret_cast<const uint2*>(dst);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int x = x0 + j;
          if (!rd_out || x >= p.n) old[j] = __float2half_rn(0.0f);
          else if (!vec) old[j] = dst[(int64_t)j * p.s_ox];
          const float bias = use_bias && x < p.n ? __half2float(p.bias[x]) : 0.0f;
          res[j] = causal && x > y ? __ushort_as_half((unsigned short)0xFC00)
                                   : store_apply_rt(store, v[j] * pre, old[j], bias, p.beta, hscale);
        }
        if (vec) {
          *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(res);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (x0 + j < p.n) dst[(int64_t)j * p.s_ox] = res[j];
        }
      }
    }
    __syncwarp();
  }
  // every CTA stays resident until its peers have read its partial tile
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------
// The same tensor-core tile for views the copy engine cannot describe (a row pitch that is
// not a multiple of 16 bytes, an unaligned base, neither operand dimension contiguous): the
// [heads, 257, 257] score and probability tensors of a 257-token encoder have a 514-byte
// pitch (adrastea_models/src/clip.rs:374-388).  Eight loader warps read the operands and write
// them into the 128-byte-swizzled stage layout themselves (zeros outside the extents),
// fence.proxy.async, arrive; the MMA warp and the eight epilogue warps are those of the
// persistent kernel.  One CTA per 128 x BN tile.
// B_MN: rhs rows are n-contiguous ([K,N] storage): the stage holds chunks of [64 k][64 n],
// described to the tensor core as an N-major operand.
// An operand with unit stride along its stage rows is read in aligned 16-byte chunks, two per
// 16-byte piece of the stage where the row is not 16-byte aligned, shifted together in registers;
// all of a k-block's loads are in flight before the first is used.  With 2-byte loads, four in
// flight, the kernel was bound by their latency: 16 heads, 257 x 64 x 257: 41.4 -> 13.5 us.
// Other strides keep the 2-byte loads.
// ---------------------------------------------------------------------------------------
constexpr int GATHER_LOAD_WARPS = 8;
constexpr int GATHER_THREADS = (2 + 8 + GATHER_LOAD_WARPS) * 32;
constexpr int GATHER_STAGES = 3;

struct GatherParams {
  const __half* lhs;
  const __half* rhs;
  int s_lx, s_ly, s_lz, s_rx, s_ry, s_rz;
  // chunks: the operand is read in aligned 16-byte chunks, as far as they lie inside [lhs, lhs_end) or
  // [rhs, rhs_end) (the whole operand, all batches)
  const __half* lhs_end;
  const __half* rhs_end;
  int a_chunks, b_chunks;
};

// A 16-byte piece of a stage row: elements src[0 .. nv - 1] (nv <= 8; none if not positive) and zeros
// behind them, from the one or two aligned chunks that hold it.
struct GatherPiece {
  uint4 c0, c1;
  static __device__ __forceinline__ int offset(const __half* src) {
    return (int)((reinterpret_cast<uintptr_t>(src) & 15u) >> 1);
  }
  // (at either end of the operand a chunk may reach past it: such a piece is read by elements)
  static __device__ __forceinline__ bool inside(const __half* src, int nv, const __half* lo, const __half* hi) {
    const int off = offset(src);
    return src - off >= lo && src - off + (off + nv > 8 ? 16 : 8) <= hi;
  }
  __device__ __forceinline__ void request(const __half* src, int nv, const __half* lo, const __half* hi) {
    c0 = c1 = make_uint4(0, 0, 0, 0);
    nv = min(nv, 8);
    if (nv > 0 && inside(src, nv, lo, hi)) {
      const int off = offset(src);
      c0 = *reinterpret_cast<const uint4*>(src - off);
      if (off + nv > 8) c1 = *reinterpret_cast<const uint4*>(src - off + 8);
    }
  }
  __device__ __forceinline__ uint4 value(const __half* src, int nv, const __half* lo, const __half* hi) const {
    uint32_t w[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    nv = min(nv, 8);
    const int off = offset(src);
    if (off & 4) {
#pragma unroll
      for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
    }
    if (off & 2) {
#pragma unroll
      for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
    }
    const unsigned sh = (off & 1) * 16u;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], sh);
    if (nv > 0 && !inside(src, nv, lo, hi)) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t a = 2 * i < nv ? __half_as_ushort(src[2 * i]) : 0u;
        const uint32_t b = 2 * i + 1 < nv ? __half_as_ushort(src[2 * i + 1]) : 0u;
        w[i] = a | (b << 16);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = 2 * i + 1 < nv ? w[i] : 2 * i < nv ? (w[i] & 0xFFFFu) : 0u;
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};

template <int BN, bool B_MN>
__global__ void __launch_bounds__(GATHER_THREADS, 1)
    gemm_f16_tc_gather_kernel(GatherParams g, TcParams p) {
  using Cfg = TcCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stages = smem;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + (size_t)GATHER_STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + GATHER_STAGES;
  uint64_t* acc_full = empty_bar + GATHER_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  uint8_t* tiles = smem + (size_t)GATHER_STAGES * Cfg::STAGE_BYTES + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (p.k + BK - 1) / BK;
  const int n0 = blockIdx.x * BN;
  const int mt = (p.m + BM - 1) / BM;
  const int m0 = (blockIdx.y % mt) * BM, b = blockIdx.y / mt;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GATHER_STAGES; ++s) {
      mbar_init(&full_bar[s], GATHER_LOAD_WARPS);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, BN < 32 ? 32 : BN);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait_trigger();
  bool ok = true;

  if (warp == 1) {
    if (lane == 0) {
      for (int kb = 0; kb < num_kb; ++kb) {
        const int s = kb % GATHER_STAGES;
        if (!mbar_wait(&full_bar[s], (unsigned)(kb / GATHER_STAGES) & 1u)) { ok = false; break; }
        tc_fence_after_sync();
        mma_k_block<BN, B_MN>(tmem_base, smem_u32(stages + (size_t)s * Cfg::STAGE_BYTES), kb == 0);
        umma_commit(&empty_bar[s]);
      }
      umma_commit(acc_full);
    }
  } else if (warp >= 2 && warp < 10) {
    const int quarter = warp & 3;
    const int chunk0 = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const __half hscale = __float2half_rn(p.scale);
    const float hs = __half2float(hscale);
    const float pre = p.load == ADR_LOAD_SCALE ? hs * hs : 1.0f;
    if (!mbar_wait(acc_full, 0)) ok = false;
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after_sync();
    if (ok) {
      const int y = m0 + row;
      __half* orow = p.out + (int64_t)b * p.s_oz + (int64_t)y * p.s_oy;
      const uint32_t tacc = tmem_base + ((uint32_t)(quarter * 32) << 16);
      if (rows_ragged(p))
        epilogue_ragged<BN>(p, tacc, orow, y, n0, chunk0, pre, hscale, tiles + (warp - 2) * EPI_TILE_BYTES, nullptr, 0);
      else
        epilogue_tile_rt<BN>(p, tacc, orow, y, n0, chunk0, pre, hscale);
    }
  } else if (warp >= 10) {
    // ---------------- loaders ----------------
    const int lt = threadIdx.x - 10 * 32;  // 0 .. 255
    constexpr int LT = GATHER_LOAD_WARPS * 32;
    const __half* abase = g.lhs + (p.a_bcast ? 0 : (int64_t)b * g.s_lz);
    const __half* bbase = g.rhs + (p.b_bcast ? 0 : (int64_t)b * g.s_rz);
    const unsigned short zero = 0;
    constexpr int PA = BM * BK / 8 / LT, PB = BN * BK / 8 / LT;  // pieces per thread
    for (int kb = 0; kb < num_kb && ok; ++kb) {
      const int s = kb % GATHER_STAGES;
      uint8_t* sa = stages + (size_t)s * Cfg::STAGE_BYTES;
      uint8_t* sb = sa + Cfg::A_BYTES;
      const int k0 = kb * BK;
      // piece u of this thread: its first element and how many of them the operand has
      auto a_src = [&](int u) { return abase + (int64_t)(m0 + ((lt + u * LT) >> 3)) * g.s_ly + k0 + (lt & 7) * 8; };
      auto a_nv = [&](int u) { return m0 + ((lt + u * LT) >> 3) < p.m ? p.k - (k0 + (lt & 7) * 8) : 0; };
      auto b_row = [&](int u) { return B_MN ? (lt + u * LT) / (BN / 8) : (lt + u * LT) >> 3; };
      auto b_col = [&](int u) { return B_MN ? (lt + u * LT) % (BN / 8) : lt & 7; };
      auto b_src = [&](int u) {
        return B_MN ? bbase + (int64_t)(k0 + b_row(u)) * g.s_ry + n0 + b_col(u) * 8
                    : bbase + (int64_t)(n0 + b_row(u)) * g.s_rx + k0 + b_col(u) * 8;
      };
      auto b_nv = [&](int u) {
        return B_MN ? (k0 + b_row(u) < p.k ? p.n - (n0 + b_col(u) * 8) : 0)
                    : (n0 + b_row(u) < p.n ? p.k - (k0 + b_col(u) * 8) : 0);
      };
      // (the loads do not wait for the stage)
      GatherPiece pa[PA], pb[PB];
      if (g.a_chunks) {
#pragma unroll
        for (int u = 0; u < PA; ++u) pa[u].request(a_src(u), a_nv(u), g.lhs, g.lhs_end);
      }
      if (g.b_chunks) {
#pragma unroll
        for (int u = 0; u < PB; ++u) pb[u].request(b_src(u), b_nv(u), g.rhs, g.rhs_end);
      }
      if (!mbar_wait(&empty_bar[s], ((unsigned)(kb / GATHER_STAGES) & 1u) ^ 1u)) { ok = false; break; }
      if (g.a_chunks) {
#pragma unroll
        for (int u = 0; u < PA; ++u) {
          const int r = (lt + u * LT) >> 3, c = lt & 7;
          *reinterpret_cast<uint4*>(sa + r * 128 + ((c ^ (r & 7)) << 4)) =
              pa[u].value(a_src(u), a_nv(u), g.lhs, g.lhs_end);
        }
      } else {
        // A: [128 rows][64 k], lanes along k
#pragma unroll 8
        for (int idx = lt; idx < BM * BK; idx += LT) {
          const int r = idx >> 6, kk = idx & 63;
          const int y = m0 + r, k = k0 + kk;
          unsigned short v = zero;
          if (y < p.m && k < p.k)
            v = __half_as_ushort(abase[(int64_t)y * g.s_ly + (int64_t)k * g.s_lx]);
          *reinterpret_cast<unsigned short*>(sa + r * 128 + ((((kk >> 3) ^ (r & 7))) << 4) + (kk & 7) * 2) = v;
        }
      }
      if (g.b_chunks) {
#pragma unroll
        for (int u = 0; u < PB; ++u) {
          const int r = b_row(u), c = b_col(u);
          uint8_t* dst = B_MN ? sb + (c >> 3) * 8192 + r * 128 + (((c & 7) ^ (r & 7)) << 4)
                              : sb + r * 128 + ((c ^ (r & 7)) << 4);
          *reinterpret_cast<uint4*>(dst) = pb[u].value(b_src(u), b_nv(u), g.rhs, g.rhs_end);
        }
      } else if (B_MN) {
        // B: chunks of [64 k][64 n], lanes along n
#pragma unroll 8
        for (int idx = lt; idx < BN * BK; idx += LT) {
          const int kk = idx / BN, nn = idx % BN;
          const int x = n0 + nn, k = k0 + kk;
          unsigned short v = zero;
          if (x < p.n && k < p.k)
            v = __half_as_ushort(bbase[(int64_t)k * g.s_ry + (int64_t)x * g.s_rx]);
          const int c = nn >> 6, ni = nn & 63;
          *reinterpret_cast<unsigned short*>(sb + c * 8192 + kk * 128 + ((((ni >> 3) ^ (kk & 7))) << 4) +
                                             (ni & 7) * 2) = v;
        }
      } else {
        // B: [BN rows of n][64 k], lanes along k
#pragma unroll 8
        for (int idx = lt; idx < BN * BK; idx += LT) {
          const int r = idx >> 6, kk = idx & 63;
          const int x = n0 + r, k = k0 + kk;
          unsigned short v = zero;
          if (x < p.n && k < p.k)
            v = __half_as_ushort(bbase[(int64_t)k * g.s_ry + (int64_t)x * g.s_rx]);
          *reinterpret_cast<unsigned short*>(sb + r * 128 + ((((kk >> 3) ^ (r & 7))) << 4) + (kk & 7) * 2) = v;
        }
      }
      // make the generic-proxy writes visible to the tensor core's async-proxy reads
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
    }
  }
  if (!ok) atomicOr(p.status, 2u);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN < 32 ? 32 : BN);
  }
}

template <int BN, bool B_MN>
int launch_gather(adr_ctx* ctx, cudaStream_t stream, const MatmulArgs& a) {
  using Cfg = TcCfg<BN>;
  auto kfn = gemm_f16_tc_gather_kernel<BN, B_MN>;
  constexpr size_t smem = 1024 + (size_t)GATHER_STAGES * Cfg::STAGE_BYTES + 256 + 8 * EPI_TILE_BYTES;
  int rc = opt_in_smem(ctx, kfn, smem);
  if (rc != ADR_OK) return rc;
  const bool a_bcast = a.batches > 1 && a.s_lz == 0;
  const bool b_bcast = a.batches > 1 && a.s_rz == 0;
  TcParams p{a.out, a.bias, a.batches, a.m, a.k, a.n, a.s_ox, a.s_oy, a.s_oz,
             a_bcast ? 1 : 0, b_bcast ? 1 : 0, a.beta, a.scale, a.store, a.load, a.mask,
             ctx->d_status};
  // the last element of an operand plus one, and whether its stage rows are contiguous in memory (and
  // its elements lie behind its base)
  const long long lz = a.batches - 1;
  const __half* lhs_end = a.lhs + lz * a.s_lz + (a.m - 1LL) * a.s_ly + (a.k - 1LL) * a.s_lx + 1;
  const __half* rhs_end = a.rhs + lz * a.s_rz + (a.k - 1LL) * a.s_ry + (a.n - 1LL) * a.s_rx + 1;
  const bool a_chunks = a.s_lx == 1 && a.s_ly >= 0 && a.s_lz >= 0;
  const bool b_chunks = (B_MN ? a.s_rx : a.s_ry) == 1 && a.s_rx >= 0 && a.s_ry >= 0 && a.s_rz >= 0;
  GatherParams g{a.lhs, a.rhs, a.s_lx, a.s_ly, a.s_lz, a.s_rx, a.s_ry, a.s_rz,
                 lhs_end, rhs_end, a_chunks ? 1 : 0, b_chunks ? 1 : 0};
  const long long nt = (a.n + BN - 1) / BN, mt = (a.m + BM - 1) / BM;
  if (mt * a.batches > 65535) return ADR_ERR_SHAPE;
  return launch_whole_sm(ctx, stream, kfn, dim3((unsigned)nt, (unsigned)(mt * a.batches)), GATHER_THREADS, smem, 1,
                         true, g, p);
}

template <int BN, bool B_MN>
int make_maps(adr_ctx* ctx, const MatmulArgs& a, CUtensorMap* map_a, CUtensorMap* map_b,
              TcParams* p) {
  const bool a_bcast = a.batches > 1 && a.s_lz == 0;
  const bool b_bcast = a.batches > 1 && a.s_rz == 0;
  {
    const uint64_t za = a_bcast || a.batches == 1 ? 1 : (uint64_t)a.batches;
    const uint64_t dims[3] = {(uint64_t)a.k, (uint64_t)a.m, za};
    const uint64_t zs = za == 1 ? (uint64_t)a.s_ly * 2 * (uint64_t)a.m : (uint64_t)a.s_lz * 2;
    const uint64_t strides[2] = {(uint64_t)a.s_ly * 2, zs};
    const uint32_t box[3] = {BK, BM, 1};
    int rc = tma_get(ctx, map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, a.lhs, dims, strides, box,
                     CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != ADR_OK) return rc;
  }
  {
    const uint64_t zb = b_bcast || a.batches == 1 ? 1 : (uint64_t)a.batches;
    // k-major B: (k, n, batch) with rows of n; n-major B: (n, k, batch) with rows of k
    const uint64_t inner = B_MN ? (uint64_t)a.n : (uint64_t)a.k;
    const uint64_t outer = B_MN ? (uint64_t)a.k : (uint64_t)a.n;
    const uint64_t pitch = (uint64_t)(B_MN ? a.s_ry : a.s_rx) * 2;
    const uint64_t dims[3] = {inner, outer, zb};
    const uint64_t zs = zb == 1 ? pitch * outer : (uint64_t)a.s_rz * 2;
    const uint64_t strides[2] = {pitch, zs};
    const uint32_t box[3] = {BK, B_MN ? 64u : (uint32_t)BN, 1};
    int rc = tma_get(ctx, map_b, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, a.rhs, dims, strides, box,
                     CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc != ADR_OK) return rc;
  }
  *p = TcParams{a.out, a.bias, a.batches, a.m, a.k, a.n, a.s_ox, a.s_oy, a.s_oz,
                a_bcast ? 1 : 0, b_bcast ? 1 : 0, a.beta, a.scale, a.store, a.load, a.mask,
                ctx->d_status};
  return ADR_OK;
}

template <int BN, bool B_MN>
int launch_tc(adr_ctx* ctx, cudaStream_t stream, const MatmulArgs& a, int S) {
  using Cfg = TcCfg<BN>;
  CUtensorMap map_a, map_b;
  TcParams p;
  int rc = make_maps<BN, B_MN>(ctx, a, &map_a, &map_b, &p);
  if (rc != ADR_OK) return rc;
  const int nt = (a.n + BN - 1) / BN, mt = (a.m + BM - 1) / BM;
  if (S <= 1) {
    const long long tiles = (long long)nt * mt * a.batches;
    const long long sms = ctx->sm_count > 0 ? ctx->sm_count : 148;
    const unsigned grid = (unsigned)std::min<long long>(tiles, sms);
    const bool ragged = rows_ragged(p);
    auto kfn = ragged ? gemm_f16_tc_kernel<BN, B_MN, EPI_RAGGED> : gemm_f16_tc_kernel<BN, B_MN, EPI_ANY>;
    // Bias, and bias + QuickGelu, on 256-wide tiles: the epilogue behind the last tile shows, and a kernel compiled
    // for the one store operation is faster.  Chosen at run time / compiled, bias and QuickGelu: 300 x 12288 x 1024 with
    // weights in L2 15.9 / 15.3 and 17.8 / 14.8 us, 300 x 12288 x 4096 from HBM 40.9 / 39.9 and 42.6 / 38.8.
    if constexpr (BN == 256 && !B_MN) {
      if (!ragged && p.store == ADR_STORE_QUICK_GELU_BIAS) kfn = gemm_f16_tc_kernel<BN, B_MN, (int)ADR_STORE_QUICK_GELU_BIAS>;
      if (!ragged && p.store == ADR_STORE_BETA_BIAS) kfn = gemm_f16_tc_kernel<BN, B_MN, (int)ADR_STORE_BETA_BIAS>;
    }
    const size_t smem = ragged ? Cfg::SMEM_TILES : Cfg::SMEM;
    rc = opt_in_smem(ctx, kfn, smem);
    if (rc != ADR_OK) return rc;
    return launch_whole_sm(ctx, stream, kfn, dim3(grid), TCP_THREADS, smem, 1, true, map_a, map_b, p);
  }
  auto kfn = gemm_f16_tc_splitk_kernel<BN, B_MN>;
  rc = opt_in_smem(ctx, kfn, Cfg::SMEM);
  if (rc != ADR_OK) return rc;
  return launch_whole_sm(ctx, stream, kfn, dim3(S, nt, mt * a.batches), TC_THREADS, Cfg::SMEM, (unsigned)S, true,
                         map_a, map_b, p, S);
}

// Pairs of CTAs of gemm_f16_pair_kernel that the GPU holds at once (both CTAs of a cluster have to find
// room on one GPC), asked once per device; 0: none, or the runtime does not say.
int pairs_resident(adr_ctx* ctx) {
  static std::mutex mu;
  static std::map<int, int> known;
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(ctx->device);
  if (it == known.end()) {
    auto kfn = gemm_f16_pair_kernel<false, (int)ADR_STORE_IDENTITY>;
    int nc = 0;
    if (opt_in_smem(ctx, kfn, PR_SMEM) == ADR_OK) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * 64, 1, 1);
      cfg.blockDim = dim3(TCP_THREADS, 1, 1);
      cfg.dynamicSmemBytes = PR_SMEM;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&nc, kfn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        nc = 0;
      }
    }
    it = known.emplace(ctx->device, nc < 0 ? 0 : nc).first;
  }
  return it->second;
}

// Whether the output is something TMA can store: unit column stride, 16-byte rows.
bool pair_supports(const MatmulArgs& a) {
  if (a.s_ox != 1 || a.s_oy % 8 != 0 || a.s_oy < a.n || (reinterpret_cast<uintptr_t>(a.out) & 15u)) return false;
  if (a.batches > 1 && (a.s_oz % 8 != 0 || a.s_oz == 0)) return false;
  return true;
}

template <bool B_MN>
int launch_pair(adr_ctx* ctx, cudaStream_t stream, const MatmulArgs& a) {
  CUtensorMap map_a, map_b, map_o;
  TcParams p;
  // (the box of B is the half tile of one CTA)
  int rc = make_maps<PR_BN / 2, B_MN>(ctx, a, &map_a, &map_b, &p);
  if (rc != ADR_OK) return rc;
  {
    const uint64_t dims[3] = {(uint64_t)a.n, (uint64_t)a.m, (uint64_t)a.batches};
    const uint64_t zs = a.batches == 1 ? (uint64_t)a.s_oy * 2 * (uint64_t)a.m : (uint64_t)a.s_oz * 2;
    const uint64_t strides[2] = {(uint64_t)a.s_oy * 2, zs};
    const uint32_t box[3] = {32, 32, 1};
    rc = tma_get(ctx, &map_o, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, a.out, dims, strides, box,
                 CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc != ADR_OK) return rc;
  }
  const long long tiles = (long long)((a.m + 2 * BM - 1) / (2 * BM)) * ((a.n + PR_BN - 1) / PR_BN) * a.batches;
  const long long pairs = std::min<long long>(tiles, pairs_resident(ctx));
  auto kfn = p.store == ADR_STORE_IDENTITY          ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_IDENTITY>
             : p.store == ADR_STORE_ADD             ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_ADD>
             : p.store == ADR_STORE_BETA_BIAS       ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_BETA_BIAS>
             : p.store == ADR_STORE_QUICK_GELU_BIAS ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_QUICK_GELU_BIAS>
             : p.store == ADR_STORE_SCALE           ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_SCALE>
             : p.store == ADR_STORE_BETA_GELU_BIAS  ? gemm_f16_pair_kernel<B_MN, (int)ADR_STORE_BETA_GELU_BIAS>
                                                    : gemm_f16_pair_kernel<B_MN, (int)STORE_NT_BETA>;
  rc = opt_in_smem(ctx, kfn, PR_SMEM);
  if (rc != ADR_OK) return rc;
  return launch_whole_sm(ctx, stream, kfn, dim3((unsigned)(2 * pairs)), TCP_THREADS, PR_SMEM, 2, true, map_a,
                         map_b, map_o, p);
}

struct TcPlan {
  int bn, S;
  bool pair = false;
};

// Picks the N-tile, the k-split or CTA pairs by the time each schedule should take, in us, fitted to what 8000 of
// them took (417 products: m 1 to 16448, n 200 to 12288, k 64 to 11008, up to 32 batches, weights from HBM and from L2;
// every tile width and split, and pairs; median error 12 %):
//   a k-block of a tile       0.295 us for 32 and 64 columns, 0.314 for 128, 0.306 for 256 while few SMs are at work
//                             (the ring's latency), up to 0.042 / 0.06 / 0 / 0.213 more with all of them
//   operands and output       at 6.0 and 4.4 TB/s, whatever the schedule
//   an epilogue               0.46 us + 2.9 for 128 x 256 outputs, under the next tile's MMAs if there is one
//   a split's reduction       2.2 us + (3.4 + 12.5 / S) for 128 x 256 outputs
//   launch and set-up         1.85 us, of a split's second wave 1.5
//   a pair                    0.326 to 0.406 us per k-block, at least 2.15 us per tile, 4.8 for everything else
// A wave of split tiles is as many clusters as ran at once on this GPU's 148 SMs: 72 of two CTAs, 35 of four, 14 of
// eight (16 already took two waves).
// Over those products the choice is 1 % slower than the best schedule of each.  Constants fitted without pairs, without
// batches and up to m = 400 were 4.2 % slower; they took pairs for products of a few tiles (2048 x 1024 x 1024: 11.3 us,
// now 9.3; 400 x 4096 x 1024 11.4, now 9.3) and small tiles where outputs are most of the bytes (12 x 1024 x 1024 x 128:
// 17.1, now 13.1).  A score of tile efficiency times SM utilisation was 57 % slower.  Pairs against 128 x 256 tiles of
// one CTA in a single wave are the closest call: 768 x 4096 x 4096 29.1 / 30.4 us with weights from HBM, 27.8 / 26.2 from
// L2.
TcPlan pick_plan(adr_ctx* ctx, const MatmulArgs& a) {
  const double sms = ctx->sm_count > 0 ? ctx->sm_count : 148;
  const double mt = (a.m + BM - 1) / BM;
  const int num_kb = (a.k + BK - 1) / BK;
  TcPlan best{64, 1};
  double best_us = 1e30;
  const bool b_mn = a.s_ry != 1;  // n-contiguous B needs 64-column chunks
  const int want = ctx->tune_tc_pair;
  const int pairs = want != 1 && pair_supports(a) ? pairs_resident(ctx) : 0;
  if (want == 2 && pairs > 0) return {PR_BN, 1, true};
  const double za = a.s_lz == 0 ? 1.0 : a.batches, zb = a.s_rz == 0 ? 1.0 : a.batches;
  const double memory_us = 2.0 * a.k * (za * a.m + zb * a.n) / 6.0e6 + 2.0 * a.batches * a.m * a.n / 4.4e6;
  for (int bn : {256, 128, 64, 32}) {
    if (b_mn && bn < 64) continue;
    if (ctx->tune_tc_bn && bn != ctx->tune_tc_bn) continue;
    if (!ctx->tune_tc_bn && bn > 32 && a.n <= bn / 2) continue;  // do not pad n beyond the next tile size
    const double tiles = mt * ((a.n + bn - 1) / bn) * a.batches;
    const double kb_us = bn == 256 ? 0.306 : bn == 128 ? 0.314 : 0.295;
    const double kb_full = bn == 256 ? 0.213 : bn == 128 ? 0.0 : bn == 64 ? 0.06 : 0.042;
    const double area = bn * std::min(a.m, BM) / 32768.0;
    for (int S : {1, 2, 4, 8}) {
      if (ctx->tune_tc_split && S != ctx->tune_tc_split) continue;
      if (S > 1 && (num_kb < 2 * S || mt * a.batches > 65535)) continue;
      const double at_once = sms / 148.0 * (S == 1 ? 148 : S == 2 ? 72 : S == 4 ? 35 : 14);
      const double waves = std::ceil(tiles / at_once);
      const double kb = ((num_kb + S - 1) / S) * (kb_us + kb_full * std::min(1.0, tiles * S / sms));
      double us;
      if (S == 1) {
        const double epilogue = 0.46 + 2.9 * area;
        us = 1.85 + std::max(waves * std::max(kb, epilogue), memory_us) + epilogue;
      } else {
        us = 1.85 + std::max(waves * kb, memory_us) + waves * (2.2 + area * (3.4 + 12.5 / S)) + (waves - 1) * 1.5;
      }
      if (us < best_us) {
        best_us = us;
        best = {bn, S};
      }
    }
  }
  if (pairs > 0 && a.m > BM && a.n > PR_BN / 2 && !ctx->tune_tc_bn && !ctx->tune_tc_split) {
    const double tiles = (double)((a.m + 2 * BM - 1) / (2 * BM)) * ((a.n + PR_BN - 1) / PR_BN) * a.batches;
    const double mma_us = std::ceil(tiles / pairs) * std::max(num_kb * (0.326 + 0.08 * std::min(1.0, tiles / pairs)), 2.15);
    if (4.8 + std::max(mma_us, memory_us) < best_us) best.pair = true;
  }
  return best;
}

}  // namespace

bool gemm_f16_tc_supports(const adr_ctx* ctx, const MatmulArgs& a) {
  if (!ctx->encode_tiled_fn) return false;
  if (a.s_lx != 1 || a.s_ly % 8 != 0) return false;  // lhs k-contiguous, 16-byte row pitch
  // rhs either k-contiguous ([N,K] storage passed permuted) or n-contiguous ([K,N] storage)
  const bool b_k = a.s_ry == 1 && a.s_rx % 8 == 0;
  const bool b_n = a.s_rx == 1 && a.s_ry % 8 == 0 && a.s_ry != 1;
  if (!b_k && !b_n) return false;
  if (a.batches > 1 && (a.s_lz % 8 != 0 || a.s_rz % 8 != 0)) return false;
  if ((reinterpret_cast<uintptr_t>(a.lhs) & 15u) || (reinterpret_cast<uintptr_t>(a.rhs) & 15u))
    return false;
  if (a.batches > 65535 || (a.m + BM - 1) / BM > 65535) return false;
  return true;
}

int launch_gemm_f16_tc(adr_ctx* ctx, cudaStream_t stream, const MatmulArgs& a) {
  const TcPlan pl = pick_plan(ctx, a);
  ctx->last_f16_schedule = pl.bn | pl.S << 16 | (pl.pair ? 1 << 24 : 0);
  if (pl.pair) return a.s_ry != 1 ? launch_pair<true>(ctx, stream, a) : launch_pair<false>(ctx, stream, a);
  if (a.s_ry != 1) {
    switch (pl.bn) {
      case 256: return launch_tc<256, true>(ctx, stream, a, pl.S);
      case 128: return launch_tc<128, true>(ctx, stream, a, pl.S);
      default: return launch_tc<64, true>(ctx, stream, a, pl.S);
    }
  }
  switch (pl.bn) {
    case 256: return launch_tc<256, false>(ctx, stream, a, pl.S);
    case 128: return launch_tc<128, false>(ctx, stream, a, pl.S);
    case 64: return launch_tc<64, false>(ctx, stream, a, pl.S);
    default: return launch_tc<32, false>(ctx, stream, a, pl.S);
  }
}

// Tensor-core tiles behind a gathering loader: any strides, any alignment.
int launch_gemm_f16_gather(adr_ctx* ctx, cudaStream_t stream, const MatmulArgs& a) {
  // lanes of a loader warp run along the contiguous dimension of rhs
  const bool b_mn = a.s_rx == 1 && a.s_ry != 1;
  if (a.n > 64) return b_mn ? launch_gather<128, true>(ctx, stream, a) : launch_gather<128, false>(ctx, stream, a);
  return b_mn ? launch_gather<64, true>(ctx, stream, a) : launch_gather<64, false>(ctx, stream, a);
}

int init_gemm_f16_tc(adr_ctx*) { return ADR_OK; }
void destroy_gemm_f16_tc(adr_ctx*) {}

}  // namespace adr
