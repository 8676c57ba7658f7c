// Block-scaled FP8 GEMM on tcgen05:  C[M,N] = (A . sfa)[M,K] (B . sfb)[N,K]^T with e4m3 operands and one E8M0 scale per
// 32 elements along K for every row of A and of B (MXFP8), accumulated in fp32 in TMEM.  The scales are applied by the
// tensor core itself (`tcgen05.mma.kind::mxf8f6f4.block_scale`): no dequantised copy of the weights ever exists.
//
// Same skeleton as the bf16 GEMM (persistent CTAs, warp 0 = TMA producer, warp 1 = MMA issuer, both as whole warps of which one
// elected lane issues, warps 2..5 = epilogue, 128-byte-swizzled K-major tiles, two TMEM accumulator stages), plus the
// scale-factor path:
//   * scales live in global memory in the layout the tensor core wants, one 512-byte block per (128 rows, 128 k):
//     byte (row % 32) * 16 + (row / 32) * 4 + (k / 32) % 4  (act_quant / weight preparation write this directly);
//   * the producer fetches the block of A and of B with a bulk copy onto the stage's full barrier;
//   * the MMA warp copies both blocks to tensor memory (`tcgen05.cp.32x128b.warpx4`: 32 rows x 16 bytes, replicated
//     to the four lane quadrants) and issues four K=32 MMAs per stage whose descriptors select scale byte 0..3.
// Tile 128 x 128 x 128 bytes of K; TMEM: 2 x 128 accumulator columns + 8 scale columns per stage.
// Every wait is bounded (status word + normal teardown).  Reference paths replaced: engine-rs/shim/ds41_mx.cu
// fp8_gemm_mx* (warp-level block-scaled mma.sync), fp8.cu / fp8pf.cu (wmma + scale promotion).
#include "../common/decode.cuh"
#include <cstdlib>
#include <mutex>

namespace spark {

constexpr int MX_BM = 128, MX_BN = 128, MX_BK = 128;       // BK in elements = bytes (fp8)
constexpr int MX_STAGES = 5;
constexpr int MX_ACC_STAGES = 2;
constexpr int MX_THREADS = 192;
constexpr int MX4_THREADS = 224;       // grouped MXFP4 kernel: + one warp that fetches the scale blocks
constexpr int MX_A_BYTES = MX_BM * MX_BK, MX_B_BYTES = MX_BN * MX_BK, MX_SF_BYTES = 512;
constexpr int MX_STAGE_BYTES = MX_A_BYTES + MX_B_BYTES + 2 * MX_SF_BYTES;
constexpr int MX_SMEM = MX_STAGES * MX_STAGE_BYTES + 256 + 1024;
constexpr int MX_TMEM_COLS = 512;                           // 256 accumulator + 40 scale columns, power of two
constexpr int MX_SF_COL0 = MX_ACC_STAGES * MX_BN;

struct MxGemmArgs {
  int M, N, K;
  const uint8_t* sfa; const uint8_t* sfb;     // [ceil(M/128)][K/128][512], [ceil(N/128)][K/128][512]
  void* C; int ldc; int out_f32;
  int* status;
};

// 32 rows x 16 bytes of shared memory -> 4 consecutive 32-bit TMEM columns, replicated over the 4 lane quadrants
__device__ __forceinline__ void tmem_cp_32x128b_x4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// un-swizzled K-major descriptor of a 32 x 16-byte block: 8-row groups 128 bytes apart
__device__ __forceinline__ uint64_t make_sf_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(16 >> 4) << 16;        // leading byte offset (one 16-byte column only)
  d |= static_cast<uint64_t>(128 >> 4) << 32;       // stride byte offset between 8-row groups
  d |= 1ull << 46;                                  // descriptor version of this architecture
  return d;
}
__device__ __forceinline__ void umma_mxf8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t tsfa,
                                          uint32_t tsfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n"
      "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(tsfa), "r"(tsfb) : "memory");
}
// block-scaled instruction descriptor: [4,6) B scale byte, [7,10) A format, [10,13) B format (0 = e4m3), [17,23) N>>3,
// bit 23 scale format (1 = E8M0), [24,29) M>>4, [29,31) A scale byte, bit 31 K size (0 = 32 for 8-bit operands)
__host__ __device__ constexpr uint32_t make_idesc_mx(uint32_t M, uint32_t N) {
  return ((N >> 3) << 17) | (1u << 23) | ((M >> 4) << 24);
}

__global__ void __launch_bounds__(MX_THREADS, 1)
gemm_mxfp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, MxGemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + MX_STAGES * MX_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + MX_STAGES;
  uint64_t* tmem_full = empty_bar + MX_STAGES;
  uint64_t* tmem_empty = tmem_full + MX_ACC_STAGES;
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(tmem_empty + MX_ACC_STAGES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_k = g.K / MX_BK;
  const int mt_n = (g.M + MX_BM - 1) / MX_BM, nt_n = (g.N + MX_BN - 1) / MX_BN;
  const int num_tiles = mt_n * nt_n;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < MX_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < MX_ACC_STAGES; ++s) { mbar_init(&tmem_full[s], 1); mbar_init(&tmem_empty[s], 4); }
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc<MX_TMEM_COLS>(tmem_base_ptr); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_ptr;

  // (the whole warp walks the loops of the issuing roles, one elected lane issues: see moe_mxfp4_kernel.  2048 rows, two products of the shared expert: 85 -> 72 us)
  if (warp == 0) {
    int stage = 0; uint32_t phase = 0; bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int mt = t / nt_n, nt = t % nt_n;
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, kb); break; }
        if (elect_one()) {
          uint8_t* a_dst = smem + stage * MX_STAGE_BYTES;
          uint8_t* b_dst = a_dst + MX_A_BYTES;
          uint8_t* sfa_dst = b_dst + MX_B_BYTES;
          mbar_arrive_expect_tx(&full_bar[stage], MX_STAGE_BYTES);
          tma_load_2d(a_dst, &tmA, &full_bar[stage], kb * MX_BK, mt * MX_BM);
          tma_load_2d(b_dst, &tmB, &full_bar[stage], kb * MX_BK, nt * MX_BN);
          bulk_load(sfa_dst, g.sfa + (static_cast<size_t>(mt) * num_k + kb) * MX_SF_BYTES, MX_SF_BYTES, &full_bar[stage]);
          bulk_load(sfa_dst + MX_SF_BYTES, g.sfb + (static_cast<size_t>(nt) * num_k + kb) * MX_SF_BYTES, MX_SF_BYTES,
                    &full_bar[stage]);
        }
        __syncwarp();
        if (++stage == MX_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc0 = make_idesc_mx(MX_BM, MX_BN);
    const uint32_t s0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_empty[acc], acc_phase ^ 1))) {
        set_status(g.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, t, acc); break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tm + acc * MX_BN;
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, kb); break; }
        tc_fence_after();
        const uint32_t a_addr = s0 + stage * MX_STAGE_BYTES;
        const uint64_t a_desc = make_smem_desc_sw128(a_addr);
        const uint64_t b_desc = make_smem_desc_sw128(a_addr + MX_A_BYTES);
        const uint64_t sfa_desc = make_sf_desc(a_addr + MX_A_BYTES + MX_B_BYTES), sfb_desc = make_sf_desc(a_addr + MX_A_BYTES + MX_B_BYTES + MX_SF_BYTES);
        const uint32_t tsfa = tm + MX_SF_COL0 + stage * 8, tsfb = tsfa + 4;
        if (elect_one()) {
          tmem_cp_32x128b_x4(tsfa, sfa_desc);
          tmem_cp_32x128b_x4(tsfb, sfb_desc);
#pragma unroll
          for (int k = 0; k < MX_BK / 32; ++k) {
            // 32 fp8 = 32 bytes along K inside the swizzled row: +2 in the encoded address; scale byte k of the block
            const uint32_t idesc = idesc0 | (static_cast<uint32_t>(k) << 4) | (static_cast<uint32_t>(k) << 29);
            umma_mxf8(d_tmem, a_desc + 2 * k, b_desc + 2 * k, idesc, tsfa, tsfb, (kb | k) != 0);
          }
          umma_commit(&empty_bar[stage]);
          if (kb == num_k - 1) umma_commit(&tmem_full[acc]);
        }
        __syncwarp();
        if (++stage == MX_STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (++acc == MX_ACC_STAGES) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    const int quarter = warp & 3;
    int acc = 0; uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const int mt = t / nt_n, nt = t % nt_n;
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[acc], acc_phase))) {
        set_status(g.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, acc); break;
      }
      tc_fence_after();
      const int row = mt * MX_BM + quarter * 32 + lane;
      const uint32_t t_addr = tmem_base + acc * MX_BN + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < MX_BN; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(t_addr + c, r);
        tmem_ld_wait();
        const int col = nt * MX_BN + c;
        if (row < g.M) {
          if (g.out_f32) {
            float* dst = reinterpret_cast<float*>(g.C) + static_cast<size_t>(row) * g.ldc + col;
            for (int i = 0; i < 32 && col + i < g.N; ++i) dst[i] = __uint_as_float(r[i]);
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(g.C) + static_cast<size_t>(row) * g.ldc + col;
            if (col + 32 <= g.N && (g.ldc & 7) == 0) {
#pragma unroll
              for (int i = 0; i < 32; i += 8) {
                uint4 o;
                __nv_bfloat162 p0 = __floats2bfloat162_rn(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                __nv_bfloat162 p1 = __floats2bfloat162_rn(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
                __nv_bfloat162 p2 = __floats2bfloat162_rn(__uint_as_float(r[i + 4]), __uint_as_float(r[i + 5]));
                __nv_bfloat162 p3 = __floats2bfloat162_rn(__uint_as_float(r[i + 6]), __uint_as_float(r[i + 7]));
                o.x = *reinterpret_cast<uint32_t*>(&p0); o.y = *reinterpret_cast<uint32_t*>(&p1);
                o.z = *reinterpret_cast<uint32_t*>(&p2); o.w = *reinterpret_cast<uint32_t*>(&p3);
                *reinterpret_cast<uint4*>(dst + i) = o;
              }
            } else {
              for (int i = 0; i < 32 && col + i < g.N; ++i) dst[i] = __float2bfloat16(__uint_as_float(r[i]));
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      if (++acc == MX_ACC_STAGES) { acc = 0; acc_phase ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc<MX_TMEM_COLS>(tmem_base); }
}

// ------------------------------------------------------------------------------------------------------------------
// Grouped MoE GEMM with MXFP4 expert weights: for every work item (a run of <= 128 activation rows routed to one
// expert) and every 128-column tile of that expert, C[rows, cols] = (A . sfa)(W_e . sfw)^T with A in MXFP8 (e4m3 + one
// E8M0 per 32 k) and W_e in MXFP4 (e2m1 + one E8M0 per 32 k).  The packed nibbles go from global memory to the tensor
// core untouched: the tensor map type 16U4_ALIGN16B makes TMA expand 16 nibbles (8 bytes) into the 16-byte padded
// slots that `tcgen05.mma.kind::mxf8f6f4` reads for a 4-bit operand, so a 128-k slice of a weight row is 128 bytes of
// shared memory exactly like an fp8 row, and the descriptors of the fp8 kernel apply unchanged (B format = e2m1).
// An item fetches only the 16-row pieces of the activation tile that it has.  The A scale blocks are tile-local (row r of the item, not of the matrix): mx_sf_tile_blocks_kernel.
// Reference paths replaced: engine-rs/shim/ds41_mx.cu (mxfp4 expert GEMMs through dequantised tiles).
struct Mx4Args {
  const int4* items;          // (first A row, rows, expert, first C row)
  const int* n_items;         // device count (<= max_items)
  int max_items;
  int N, K;                   // per expert
  const uint8_t* sfa;         // [max_items][K/128][512]
  const uint8_t* sfw;         // [E * N/128][K/128][512]
  void* C; int ldc; int out_f32;
  int* status;
  uint32_t w_tx_bytes;        // bytes one weight tile adds to the stage barrier's transaction count (packed size)
};

// ROWS: the most rows of an item.  16: decode pairs, a stage is 19 KB (2 KB activations, 16 KB weights, two scale blocks) and ten stages fit.
// 64: prompts of a few dozen rows per expert, 25 KB, nine stages; 128: 33 KB, six.  The packed bytes in flight per SM are what the weight
// stream runs on: 40 KB of them (five stages of 128 rows) reach 4.9 TB/s, 72 KB (nine of 64) 5.6: 1065 -> 933 us for both products of 2048
// rows, six experts each of 384 of [4096 -> 2 x 2048 -> 4096].
template <int ROWS>
struct Mx4Cfg {
  static constexpr int STAGES = ROWS == 16 ? 10 : ROWS == 64 ? 9 : 6;
  static constexpr int A_REGION = ROWS * MX_BK;
  static constexpr int B_OFF = STAGES * A_REGION;
  static constexpr int SF_OFF = B_OFF + STAGES * MX_B_BYTES;
  static constexpr int BAR_OFF = SF_OFF + STAGES * 2 * MX_SF_BYTES;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;
  static_assert(SMEM <= 232448 && MX_SF_COL0 + STAGES * 8 <= MX_TMEM_COLS, "shared memory, scale columns");
};

template <int ROWS>
__global__ void __launch_bounds__(MX4_THREADS, 1)
moe_mxfp4_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA16,
                 const __grid_constant__ CUtensorMap tmW, Mx4Args g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  using Cfg = Mx4Cfg<ROWS>;
  constexpr int STAGES = Cfg::STAGES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::BAR_OFF);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;
  uint64_t* tmem_empty = tmem_full + MX_ACC_STAGES;
  uint32_t* tmem_base_ptr = reinterpret_cast<uint32_t*>(tmem_empty + MX_ACC_STAGES);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int num_k = g.K / MX_BK;
  const int nt_n = g.N / MX_BN;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmA16);
    tma_prefetch_desc(&tmW);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 2); mbar_init(&empty_bar[s], 1); }    // two producers
    for (int s = 0; s < MX_ACC_STAGES; ++s) { mbar_init(&tmem_full[s], 1); mbar_init(&tmem_empty[s], 4); }
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc<MX_TMEM_COLS>(tmem_base_ptr); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_ptr;
  pdl_wait();                                                    // (barriers and tensor memory are set up beside the kernel before)
  pdl_trigger();
  const int n_items = min(*g.n_items, g.max_items);
  const int num_tiles = n_items * nt_n;

  if (warp == 0) {
    int stage = 0; uint32_t phase = 0; bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int it = t / nt_n, nt = t - it * nt_n;
      const int4 item = g.items[it];
      const int row0 = __shfl_sync(0xffffffffu, item.x, 0), rows = __shfl_sync(0xffffffffu, item.y, 0), expert = __shfl_sync(0xffffffffu, item.z, 0);
      if (expert < 0 || rows <= 0) continue;                     // expert of another rank / empty item
      if (rows > ROWS) { set_status(g.status, ST_BOUNDS, blockIdx.x, t, rows); break; }
      const int pieces = ROWS == 16 ? 1 : (rows + 15) >> 4;   // 16-row pieces of the activation tile that the item has
      const uint32_t bytes = pieces * 16 * MX_BK + g.w_tx_bytes;
      const int wrow = expert * g.N + nt * MX_BN;
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, kb); break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&full_bar[stage], bytes);
          uint8_t* a_dst = smem + stage * Cfg::A_REGION;
          if (pieces * 16 == 128) tma_load_2d(a_dst, &tmA, &full_bar[stage], kb * MX_BK, row0);
          else for (int p = 0; p < pieces; ++p) tma_load_2d(a_dst + p * 16 * MX_BK, &tmA16, &full_bar[stage], kb * MX_BK, row0 + p * 16);
          tma_load_2d(smem + Cfg::B_OFF + stage * MX_B_BYTES, &tmW, &full_bar[stage], kb * MX_BK, wrow);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 6) {
    // second producer: the two scale blocks of every stage, so that the tile loads and the scale copies are issued
    // by different threads
    int stage = 0; uint32_t phase = 0; bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int it = t / nt_n, nt = t - it * nt_n;
      const int4 item = g.items[it];
      const int rows = __shfl_sync(0xffffffffu, item.y, 0), expert = __shfl_sync(0xffffffffu, item.z, 0);
      if (expert < 0 || rows <= 0) continue;
      if (rows > ROWS) break;
      const uint8_t* sa = g.sfa + static_cast<size_t>(it) * num_k * MX_SF_BYTES;
      const uint8_t* sw = g.sfw + static_cast<size_t>(expert * nt_n + nt) * num_k * MX_SF_BYTES;
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, -kb - 1); break; }
        if (elect_one()) {
          uint8_t* sf_dst = smem + Cfg::SF_OFF + stage * 2 * MX_SF_BYTES;
          mbar_arrive_expect_tx(&full_bar[stage], 2 * MX_SF_BYTES);
          bulk_load(sf_dst, sa + static_cast<size_t>(kb) * MX_SF_BYTES, MX_SF_BYTES, &full_bar[stage]);
          bulk_load(sf_dst + MX_SF_BYTES, sw + static_cast<size_t>(kb) * MX_SF_BYTES, MX_SF_BYTES, &full_bar[stage]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // The weights are the 128-row operand (format e2m1 in bits [7,10)), the rows of the item the other, rounded up to 16: decode pairs
    // run at memory speed, and the 30 or 40 rows of an expert in a prompt do not pay for 128 (2048 rows: 639 -> 535 us per product).
    // The whole warp walks the loop and one elected lane issues: addresses and descriptors are warp-uniform then and stay in
    // uniform registers, where the instructions want them (in a branch of one lane every
    // operand was moved over for every instruction: 720 cycles per block of 128 k, whatever the memory did).  The producers do the same.
    // 24 pairs of an MXFP4 layer 57 -> 36 us per product, 2048 rows 757 -> 639.
    const uint32_t s0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const int4 item = g.items[t / nt_n];
      const int expert = __shfl_sync(0xffffffffu, item.z, 0), rows = __shfl_sync(0xffffffffu, item.y, 0);
      if (expert < 0 || rows <= 0) continue;
      if (rows > ROWS) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_empty[acc], acc_phase ^ 1))) {
        set_status(g.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, t, acc); break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tm + acc * MX_BN;
      const uint32_t idesc0 = make_idesc_mx(MX_BN, ROWS == 16 ? 16 : (rows + 15) & ~15) | (5u << 7);
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, kb); break; }
        tc_fence_after();
        const uint64_t x_desc = make_smem_desc_sw128(s0 + stage * Cfg::A_REGION);            // activations
        const uint64_t w_desc = make_smem_desc_sw128(s0 + Cfg::B_OFF + stage * MX_B_BYTES);  // weights
        const uint32_t sf_addr = s0 + Cfg::SF_OFF + stage * 2 * MX_SF_BYTES;                 // [activations | weights]
        const uint32_t tsfa = tm + MX_SF_COL0 + stage * 8, tsfb = tsfa + 4;
        const uint64_t sfa_desc = make_sf_desc(sf_addr + MX_SF_BYTES), sfb_desc = make_sf_desc(sf_addr);
        if (elect_one()) {
          tmem_cp_32x128b_x4(tsfa, sfa_desc);
          tmem_cp_32x128b_x4(tsfb, sfb_desc);
#pragma unroll
          for (int k = 0; k < MX_BK / 32; ++k) {
            const uint32_t idesc = idesc0 | (static_cast<uint32_t>(k) << 4) | (static_cast<uint32_t>(k) << 29);
            umma_mxf8(d_tmem, w_desc + 2 * k, x_desc + 2 * k, idesc, tsfa, tsfb, (kb | k) != 0);
          }
          umma_commit(&empty_bar[stage]);
          if (kb == num_k - 1) umma_commit(&tmem_full[acc]);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (++acc == MX_ACC_STAGES) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    const int quarter = warp & 3;
    int acc = 0; uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const int it = t / nt_n, nt = t - it * nt_n;
      const int4 item = g.items[it];
      if (item.z < 0 || item.y <= 0) continue;
      if (item.y > ROWS) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full[acc], acc_phase))) {
        set_status(g.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, acc); break;
      }
      tc_fence_after();
      const int r = quarter * 32 + lane;
      const uint32_t t_addr = tmem_base + acc * MX_BN + (static_cast<uint32_t>(quarter * 32) << 16);
      // lane = weight row (output column), TMEM column j = activation row j of the item
      const int col = nt * MX_BN + r;
#pragma unroll 1
      for (int c = 0; c < (ROWS == 16 ? 16 : item.y); c += 32) {
        uint32_t v[32];
        tmem_ld_32x32(t_addr + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < (ROWS == 16 ? 16 : 32); ++j) {
          if (c + j < item.y) {
            const size_t o = (static_cast<size_t>(item.w) + c + j) * g.ldc + col;
            if (g.out_f32) reinterpret_cast<float*>(g.C)[o] = __uint_as_float(v[j]);
            else reinterpret_cast<__nv_bfloat16*>(g.C)[o] = __float2bfloat16(__uint_as_float(v[j]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      if (++acc == MX_ACC_STAGES) { acc = 0; acc_phase ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc<MX_TMEM_COLS>(tmem_base); }
}

// Work items of the grouped kernel.  mode 0: from the expert-sorted tile list (first row, end row, expert, rows or 0: up to 128): one item
// per tile, C rows = A rows.  mode 1: one item per (token, expert) pair: A row = pair_row[p] (or p), C row = p.
__global__ void mx4_items_kernel(int mode, const int4* __restrict__ tiles, const int* __restrict__ ntile,
                                 const int* __restrict__ pair_expert, const int* __restrict__ pair_row, int pairs,
                                 int max_items, int4* __restrict__ items, int* __restrict__ n_items) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = mode == 0 ? min(*ntile, max_items) : min(pairs, max_items);
  if (i == 0) *n_items = n;
  if (i >= max_items) return;
  int4 it = make_int4(0, 0, -1, 0);
  if (i < n) {
    if (mode == 0) {
      const int4 td = tiles[i];
      it = make_int4(td.x, td.w ? td.w : min(128, td.y - td.x), td.z, td.x);
    } else {
      it = make_int4(pair_row ? pair_row[i] : i, 1, pair_expert[i], i);
    }
  }
  items[i] = it;
}

// Activation scale bytes [R, K/32] (row-major) -> item-local blocks [max_items][K/128][512]: byte
// (r % 32) * 16 + (r / 32) * 4 + k32 % 4 of block (item, k128) is the scale of row item.x + r; rows past the item's
// end read exponent 0.
__global__ void mx_sf_tile_blocks_kernel(const uint8_t* __restrict__ sf, const int4* __restrict__ items,
                                         const int* __restrict__ n_items, int max_items, int kblocks32,
                                         uint8_t* __restrict__ out) {
  const int kb128 = kblocks32 >> 2;
  const int it = blockIdx.x;
  if (it >= min(*n_items, max_items)) return;
  const int4 item = items[it];
  for (int i = threadIdx.x; i < kb128 * 512; i += blockDim.x) {
    const int kt = i >> 9, within = i & 511;
    const int r32 = within >> 4, q = (within >> 2) & 3, kk = within & 3;
    const int r = q * 32 + r32;
    uint8_t v = 0;
    if (item.z >= 0 && r < item.y) v = sf[static_cast<size_t>(item.x + r) * kblocks32 + kt * 4 + kk];
    out[(static_cast<size_t>(it) * kb128 + kt) * 512 + within] = v;
  }
}

// Work items and their activation scale blocks in one launch (one block per item): the decode path runs this twice
// per MoE layer, and a launch saved there is worth more than the few redundant loads.
__global__ void mx4_prep_kernel(int mode, const int4* __restrict__ tiles, const int* __restrict__ ntile,
                                const int* __restrict__ pair_expert, const int* __restrict__ pair_row, int pairs,
                                int max_items, const uint8_t* __restrict__ sf, int kblocks32, int4* __restrict__ items,
                                int* __restrict__ n_items, uint8_t* __restrict__ out, int words) {
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.x;
  const int n = mode == 0 ? min(*ntile, max_items) : min(pairs, max_items);
  int4 item = make_int4(0, 0, -1, 0);
  if (i < n) {
    if (mode == 0) {
      const int4 td = tiles[i];
      item = make_int4(td.x, td.w ? td.w : min(128, td.y - td.x), td.z, td.x);
    } else {
      item = make_int4(pair_row ? pair_row[i] : i, 1, pair_expert[i], i);
    }
  }
  if (threadIdx.x == 0) {
    items[i] = item;
    if (i == 0) *n_items = n;
  }
  if (i >= n) return;
  const int kb128 = kblocks32 >> 2;
  if (words) {                                                   // the four scales of a row and block are one word on both sides
    for (int j = threadIdx.x; j < kb128 * 128; j += blockDim.x) {
      const int kt = j >> 7, r = (j & 3) * 32 + ((j >> 2) & 31);
      uint32_t v = 0u;
      if (item.z >= 0 && r < item.y) v = reinterpret_cast<const uint32_t*>(sf)[static_cast<size_t>(item.x + r) * kb128 + kt];
      reinterpret_cast<uint32_t*>(out)[static_cast<size_t>(i) * kb128 * 128 + j] = v;
    }
    return;
  }
  for (int j = threadIdx.x; j < kb128 * 512; j += blockDim.x) {
    const int kt = j >> 9, within = j & 511;
    const int r32 = within >> 4, q = (within >> 2) & 3, kk = within & 3;
    const int r = q * 32 + r32;
    uint8_t v = 0;
    if (item.z >= 0 && r < item.y) v = sf[static_cast<size_t>(item.x + r) * kblocks32 + kt * 4 + kk];
    out[(static_cast<size_t>(i) * kb128 + kt) * 512 + within] = v;
  }
}

// Scale bytes [rows, K/32] (row-major) -> the tensor core's block layout [ceil(rows/128)][K/128][512]; rows past the
// end get exponent 0 (scale 2^-127: their products vanish and are never stored anyway).
__global__ void mx_sf_to_blocks_kernel(const uint8_t* __restrict__ sf, uint8_t* __restrict__ out, int rows, int kblocks32) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int kb128 = kblocks32 >> 2;
  const long long total = static_cast<long long>((rows + 127) / 128) * kb128 * 512;
  if (i >= total) return;
  const int within = static_cast<int>(i & 511);
  const long long blk = i >> 9;
  const int kt = static_cast<int>(blk % kb128);
  const int rt = static_cast<int>(blk / kb128);
  const int r32 = within >> 4, q = (within >> 2) & 3, kk = within & 3;
  const int row = rt * 128 + q * 32 + r32;
  out[i] = row < rows ? sf[static_cast<size_t>(row) * kblocks32 + kt * 4 + kk] : 0;
}

typedef CUresult (*EncodeTiledFnMx)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFnMx encode_fn_mx() {
  static EncodeTiledFnMx fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFnMx>(p);
  });
  return fn;
}
static int make_tmap_u8(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K, uint64_t ld, uint32_t box_rows = 128) {
  EncodeTiledFnMx fn = encode_fn_mx();
  if (!fn) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld & 15)) return -2;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {ld};
  cuuint32_t box[2] = {MX_BK, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// packed e2m1 [rows, K/2 bytes]: 128 nibbles of a row (64 bytes of global memory) land as 128 bytes of shared memory
static int make_tmap_u4(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K) {
  EncodeTiledFnMx fn = encode_fn_mx();
  if (!fn) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 31) || ((K / 2) & 31) || (K & 127)) return -2;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K / 2};
  cuuint32_t box[2] = {MX_BK, 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace spark

using namespace spark;

extern "C" int spark_mx4_items(int mode, const void* tiles, const int* ntile, const int* pair_expert, const int* pair_row,
                               int pairs, int max_items, void* items, int* n_items, cudaStream_t stream) {
  if (max_items <= 0) return 0;
  mx4_items_kernel<<<(max_items + 127) / 128, 128, 0, stream>>>(mode, (const int4*)tiles, ntile, pair_expert, pair_row, pairs,
                                                                max_items, (int4*)items, n_items);
  return spark_launch_rc(__func__);
}

extern "C" int spark_mx_sf_tile_blocks(const void* sf, const void* items, const int* n_items, int max_items, int kblocks32,
                                       void* out, cudaStream_t stream) {
  if (max_items <= 0 || kblocks32 <= 0) return 0;
  if (kblocks32 % 4) return -5;
  mx_sf_tile_blocks_kernel<<<max_items, 256, 0, stream>>>((const uint8_t*)sf, (const int4*)items, n_items, max_items, kblocks32,
                                                         (uint8_t*)out);
  return spark_launch_rc(__func__);
}

extern "C" int spark_mx4_prep(int mode, const void* tiles, const int* ntile, const int* pair_expert, const int* pair_row,
                              int pairs, int max_items, const void* sf, int kblocks32, void* items, int* n_items, void* out,
                              cudaStream_t stream) {
  if (max_items <= 0 || kblocks32 <= 0) return 0;
  if (kblocks32 % 4) return -5;
  const cudaError_t err = spark_launch_pdl(mx4_prep_kernel, dim3(max_items), dim3(256), 0, stream, dim3(1, 1, 1), mode, (const int4*)tiles, ntile,
                                           pair_expert, pair_row, pairs, max_items, (const uint8_t*)sf, kblocks32, (int4*)items, n_items,
                                           (uint8_t*)out, ((reinterpret_cast<uintptr_t>(sf) | reinterpret_cast<uintptr_t>(out)) & 3) == 0 ? 1 : 0);
  return err == cudaSuccess ? 0 : -4;
}

// A e4m3 [rows_a, K] (row stride lda bytes); W packed e2m1 [E * N, K / 2]; sfa item-local blocks
// (spark_mx_sf_tile_blocks), sfw blocks of the flattened [E * N, K / 32] scales (spark_mx_sf_to_blocks);
// C [*, ldc] bf16 or fp32.  N % 128 == 0, K % 128 == 0.  item_rows: the most rows of an item, 16, 64 or 128
// (longer ones: an error in the status word).
extern "C" int spark_moe_mxfp4(const void* A, int lda, int rows_a, const void* W, const void* sfa, const void* sfw,
                               const void* items, const int* n_items, int max_items, int E, int N, int K, void* C, int ldc,
                               int out_f32, int item_rows, int* status, cudaStream_t stream) {
  if (max_items <= 0 || rows_a <= 0) return 0;
  if (item_rows != 16 && item_rows != 64 && item_rows != 128) return -5;
  if (K % MX_BK || N % MX_BN || (ldc & 7) || (reinterpret_cast<uintptr_t>(C) & 15)) return -5;
  CUtensorMap tA, tA16, tW;
  int r = make_tmap_u8(&tA, A, rows_a, K, lda);
  if (r) return r;
  r = make_tmap_u8(&tA16, A, rows_a, K, lda, 16);
  if (r) return r;
  r = make_tmap_u4(&tW, W, static_cast<uint64_t>(E) * N, K);
  if (r) return r - 10;
  // a 16U4_ALIGN16B copy completes the barrier with the packed bytes it read (64 per row), not the 128 it writes
  const uint32_t w_tx = MX_B_BYTES / 2;
  Mx4Args g{(const int4*)items, n_items, max_items, N, K, (const uint8_t*)sfa, (const uint8_t*)sfw, C, ldc, out_f32, status, w_tx};
  void (*kern)(CUtensorMap, CUtensorMap, CUtensorMap, Mx4Args) = item_rows == 16 ? moe_mxfp4_kernel<16> : item_rows == 64 ? moe_mxfp4_kernel<64> : moe_mxfp4_kernel<128>;
  const int smem = item_rows == 16 ? Mx4Cfg<16>::SMEM : item_rows == 64 ? Mx4Cfg<64>::SMEM : Mx4Cfg<128>::SMEM;
  static bool attr_done = false;
  if (!attr_done) {
    cudaFuncSetAttribute(moe_mxfp4_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, Mx4Cfg<16>::SMEM);
    cudaFuncSetAttribute(moe_mxfp4_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, Mx4Cfg<64>::SMEM);
    cudaFuncSetAttribute(moe_mxfp4_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, Mx4Cfg<128>::SMEM);
    attr_done = true;
  }
  static int sms = 0;
  if (!sms) { int dev; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  const long long tiles = static_cast<long long>(max_items) * (N / MX_BN);
  const int grid = tiles < sms ? static_cast<int>(tiles) : sms;
  return spark_launch_pdl(kern, dim3(grid), dim3(MX4_THREADS), smem, stream, dim3(1, 1, 1), tA, tA16, tW, g) == cudaSuccess ? 0 : -4;
}

// A e4m3 [M,K] (row stride lda bytes), B e4m3 [N,K]; sfa / sfb in block layout (spark_mx_sf_to_blocks); K % 128 == 0.
extern "C" int spark_gemm_mxfp8(const void* A, const void* B, const void* sfa, const void* sfb, void* C, int M, int N, int K,
                                int lda, int ldb, int ldc, int out_f32, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (K % MX_BK) return -5;
  CUtensorMap tA, tB;
  int r = make_tmap_u8(&tA, A, M, K, lda);
  if (r) return r;
  r = make_tmap_u8(&tB, B, N, K, ldb);
  if (r) return r;
  MxGemmArgs g{M, N, K, (const uint8_t*)sfa, (const uint8_t*)sfb, C, ldc, out_f32, status};
  static bool attr_done = false;
  if (!attr_done) { cudaFuncSetAttribute(gemm_mxfp8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MX_SMEM); attr_done = true; }
  static int sms = 0;
  if (!sms) { int dev; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  const int tiles = ((M + MX_BM - 1) / MX_BM) * ((N + MX_BN - 1) / MX_BN);
  gemm_mxfp8_kernel<<<tiles < sms ? tiles : sms, MX_THREADS, MX_SMEM, stream>>>(tA, tB, g);
  return spark_launch_rc(__func__);
}

extern "C" int spark_mx_sf_to_blocks(const void* sf, void* out, int rows, int kblocks32, cudaStream_t stream) {
  if (rows <= 0 || kblocks32 <= 0) return 0;
  if (kblocks32 % 4) return -5;
  const long long total = static_cast<long long>((rows + 127) / 128) * (kblocks32 / 4) * 512;
  mx_sf_to_blocks_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>((const uint8_t*)sf, (uint8_t*)out, rows,
                                                                                         kblocks32);
  return spark_launch_rc(__func__);
}
