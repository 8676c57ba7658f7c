// EXL3 grouped GEMM of prompt-size MoE batches on tcgen05: packed trellises -> fp16 operands in tensor memory.
//   plain: y[rows, N]   = had128(xh @ inner_e) * svh_e                                   (fp32 or bf16)
//   glu:   y[rows, F]   = had128(bf16(act(gate) * up) * suh2_e) as fp16, the input rows of the down product
// with xh = had128(x * suh_e) in fp16, rows in expert order, work items of one expert and <= 192 rows.
//
// The product runs transposed: the weights are the 128-row M operand, the rows of the item the N operand (a multiple of 16, so
// that 20 rows of an expert cost 32 columns and not 128).  A lane that takes four consecutive words of a packed tile owns all 16 k
// of two output columns (c and c + 8), which is one K = 16 row of an A operand in tensor memory each: the decoded values go from
// the registers straight to TMEM (tcgen05.st), never through shared memory, and the two column halves are two accumulators.
//
// Roles (one CTA per SM, 23 warps): warp 0 streams packed tiles (bulk copies) into a ring of ten stages of 64 k, warp 22 activation boxes
// (TMA, 128-byte swizzle) into one of three (the tiles come from DRAM and are what has to be in flight); 16 warps decode, two groups of
// eight in turn, two 16-k tile rows of a stage each; warp 1 issues the MMAs; 4 warps run the epilogue (TMEM -> shared memory -> output
// Hadamard, eight lanes per 128-block).  Items of <= 96 rows use half of the accumulator columns each, so that one item's epilogue
// overlaps the next one's products; a larger one (<= 192 rows, so that an expert of 160 rows is decoded once) takes both, and the
// decoders, who have nothing to do meanwhile, read it out.
//
// What bounds it: the decode, about 35 integer instructions per 256 weights and sub-partition (194 us of 512 experts of [2048 x 1024] and
// [512 x 2048], whatever the rows), and beyond some 100 rows of an expert the transforms of the read-out, 96 to 144 shuffles of 16 rows and
// warp.  us of gate / up + down, one item per 128 rows and one ring of eight stages before: 1021 rows of ten experts 270 + 147 -> 262 + 144,
// 8192 rows 865 + 551 -> 513 + 400 (items of 160 rows on average are decoded once instead of twice).  Where a CTA has one item at most, the two
// groups' alternation lengthens its chain: 33 rows for each of 8 experts of [2048 x 1024] and [512 x 2048] 27.4 + 10.7 -> 29.2 + 11.6.
//
// Reference: engine-rs/shim/moe_exl3.cuh:521-1233 (gemm_grouped / gux / gu2 kernels, mma.sync m16n8k16).
#include "exl3_common.cuh"

namespace spark {

int make_tmap_bf16(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K, uint64_t ld, int box_rows, int fmt);

struct Exl3TcArgs {
  const uint32_t* trellis; long long t_stride;        // [E][K/16][N/16][32] words
  const __half* svh; long long svh_stride;            // [E][N]
  const __half* suh2; long long suh2_stride;          // glu: [E][F] input scales of the next product
  const int4* tiles; const int* ntile;                // {row0, row_end, expert, rows}, and their count; rows <= 192, 0: up to 128 of them
  void* y; int ldy; int out_f32;
  int K, N; float limit;
  int wide;                                           // rows of a 16-bit y start on 16 bytes (else 8)
  int* status;
};

constexpr int TC_THREADS = 23 * 32, TC_DECODERS = 8, TC_ROWS = 192;      // (decoders of a stage)
constexpr int TC_BSTAGES = 3, TC_B_BYTES = TC_ROWS * 128, TC_TSTAGES = 10, TC_T_BYTES = 4 * 16 * 128;
constexpr int TC_T_OFF = TC_BSTAGES * TC_B_BYTES, TC_XP_OFF = TC_T_OFF + TC_TSTAGES * TC_T_BYTES;
constexpr int TC_XP = 16 * 256 * 4, TC_GROUPS = 4;     // epilogue exchange of a group of four warps: 16 rows x 256 columns; groups of decoders
constexpr int TC_BAR_OFF = TC_XP_OFF + TC_GROUPS * TC_XP, TC_SMEM = TC_BAR_OFF + 512 + 1024;
constexpr int TC_A_COLS = 64, TC_A_BUFS = 2, TC_D_COLS = 2 * TC_ROWS;
static_assert(TC_D_COLS + TC_A_BUFS * TC_A_COLS <= 512 && TC_SMEM <= 232448, "tensor memory, shared memory");
static_assert(TC_TSTAGES % 2 == 0 && TC_A_BUFS == 2, "a stage's barriers belong to one of the two groups of decoders, which waits for each of their phases");

// Accumulator halves an item takes, the same sequence in every role: an item of <= 96 rows takes the next half, a larger one both.  Each
// role waits for every phase of the barriers it waits on (one that skips a phase cannot tell the next from the one before): d_full[h] are the
// small items' (epilogue warps), d_big the large ones' (decoders).
struct AccRing {
  int half = 0;
  __device__ __forceinline__ int take(int n) { const int m = n <= TC_ROWS / 2 ? 1 << half : 3; half = n <= TC_ROWS / 2 ? half ^ 1 : 0; return m; }
};

struct TcItem { int row0, rows, n, expert, strip; };

__device__ __forceinline__ TcItem tc_item(const Exl3TcArgs& a, int t, int strips) {
  const int4 td = a.tiles[t / strips];
  TcItem it;
  it.row0 = td.x; it.rows = td.w ? td.w : min(td.y - td.x, 128); it.n = (it.rows + 15) & ~15; it.expert = td.z; it.strip = t % strips;
  return it;
}

// 16 columns of a row from the exchange: 8 and 8 of a tile, 32 floats apart; sw: 4 where the two halves of 8 are swapped
__device__ __forceinline__ void tc_ld_block(const float* p, int sw, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 t = *reinterpret_cast<const float4*>(p + (i >> 1) * 32 + (((i & 1) << 2) ^ sw));
    v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
  }
}
// by 16 of a scale vector (rows of it start on 8 bytes), with or without the transform's normalisation
template <bool NORM>
__device__ __forceinline__ void tc_by(const __half* p, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint2 w = __ldg(reinterpret_cast<const uint2*>(p) + i);
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
    v[4 * i] *= NORM ? a.x * INV_SQRT_128 : a.x; v[4 * i + 1] *= NORM ? a.y * INV_SQRT_128 : a.y;
    v[4 * i + 2] *= NORM ? b.x * INV_SQRT_128 : b.x; v[4 * i + 3] *= NORM ? b.y * INV_SQRT_128 : b.y;
  }
}
__device__ __forceinline__ void tc_scale(const __half* p, float (&v)[16]) { tc_by<true>(p, v); }
__device__ __forceinline__ void tc_mul(const __half* p, float (&v)[16]) { tc_by<false>(p, v); }
__device__ __forceinline__ void tc_store16(void* p, int wide, const uint32_t (&w)[8]) {
  if (wide) {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint2*>(p)[i] = make_uint2(w[2 * i], w[2 * i + 1]);
  }
}

// Waits for an item's accumulator; the four warps of a group take the same way (the exchange below has barriers of the group): one
// that has failed before comes here all the same
__device__ __forceinline__ bool tc_wait_acc(uint64_t* full, uint32_t parity, int bar, bool ok = true) {
  ok = ok && mbar_wait(full, parity);
  int bad = !ok;
  asm volatile("{\n.reg .pred p, r;\nsetp.ne.b32 p, %0, 0;\nbarrier.cta.red.or.pred r, %1, 128, p;\nselp.b32 %0, 1, 0, r;\n}\n" : "+r"(bad) : "r"(bar) : "memory");
  tc_fence_after();
  return !bad;
}

// Rows of an item from its accumulators: `groups` groups of four warps take 16 rows in turn, this one (barrier `bar`) the group-th.  The
// epilogue warps, a single group with two buffers in turn, share them with the decoders: an item's products wait until the item before is read out.
template <bool GLU>
__device__ __forceinline__ void tc_epilogue(const Exl3TcArgs& a, const TcItem& it, int mask, uint32_t tmem, float* xp, int group, int groups,
                                            int bar, int& buf, uint64_t* d_empty) {
  const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) & 3;   // TMEM lanes [32 q, 32 q + 32): columns 64 q .. 64 q + 63 of the strip
  const int NT = a.N >> 4, F = a.N >> 1;
  const uint32_t d0 = tmem + (mask == 2 ? TC_ROWS : 0) + (static_cast<uint32_t>(q * 32) << 16), d1 = d0 + (mask == 3 ? TC_ROWS : TC_ROWS / 2);
  const int c0 = it.strip * (GLU ? 128 : 256);
  const bool one = !GLU && it.strip * 16 + 8 >= NT;
  const int oct = lane & 7;                               // this lane's 16 columns of a 128-block, of row lane >> 3 of the warp's four
  const __half* sv0 = a.svh + it.expert * a.svh_stride + c0 + oct * 16;
  const __half* sv1 = sv0 + (GLU ? F : 128);
  const __half* sv2 = GLU ? a.suh2 + it.expert * a.suh2_stride + c0 + oct * 16 : nullptr;
  float* x = xp + group * (TC_XP / 4);
  const int at = q * 64 + (lane ^ ((q & 1) << 2));        // (odd quarters swap halves of 8 columns: the loads below miss each other's banks)
  for (int c = group * 16; c < it.n; c += groups * 16) {
    uint32_t v0[16], v1[16];
    tmem_ld_32x16(d0 + c, v0);
    tmem_ld_32x16(d1 + c, v1);
    tmem_ld_wait();
    if (groups > 1) asm volatile("barrier.cta.sync %0, 128;" ::"r"(bar) : "memory");       // the 16 rows before are read
    else { x = xp + buf * (TC_XP / 4); buf ^= 1; }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      x[i * 256 + at] = __uint_as_float(v0[i]);
      x[i * 256 + at + 32] = __uint_as_float(v1[i]);
    }
    asm volatile("barrier.cta.sync %0, 128;" ::"r"(bar) : "memory");
    const int r = q * 4 + (lane >> 3);
    const bool live = c + r < it.rows;
    const float* xr = x + r * 256 + (oct >> 2) * 64 + (oct & 3) * 8;
    const int sw = (oct >> 2) << 2;
    const size_t row = static_cast<size_t>(it.row0 + c + r) * a.ldy;
    if (GLU) {
      float g[16], u[16];
      tc_ld_block(xr, sw, g);
      fwht128_oct(g, lane);
      tc_scale(sv0, g);
      tc_ld_block(xr + 128, sw, u);
      fwht128_oct(u, lane);
      tc_scale(sv1, u);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float gg = __bfloat162float(__float2bfloat16(g[i])), uu = __bfloat162float(__float2bfloat16(u[i]));
        if (a.limit > 0.f) { gg = fminf(gg, a.limit); uu = fminf(fmaxf(uu, -a.limit), a.limit); }
        u[i] = __bfloat162float(__float2bfloat16(gg / (1.f + __expf(-gg)) * uu));
      }
      tc_mul(sv2, u);
      fwht128_oct(u, lane);
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const __half2 h = __floats2half2_rn(u[2 * i] * INV_SQRT_128, u[2 * i + 1] * INV_SQRT_128);
        o[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
      if (live) tc_store16(static_cast<__half*>(a.y) + row + c0 + oct * 16, a.wide, o);
    } else {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (b && one) break;
        float v[16];
        tc_ld_block(xr + b * 128, sw, v);
        fwht128_oct(v, lane);
        tc_scale(b ? sv1 : sv0, v);
        const size_t o = row + c0 + b * 128 + oct * 16;
        if (a.out_f32) {
          float4* p = reinterpret_cast<float4*>(static_cast<float*>(a.y) + o);
#pragma unroll
          for (int i = 0; i < 4; ++i) if (live) p[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
          if (live) tc_store16(static_cast<__nv_bfloat16*>(a.y) + o, a.wide, w);
        }
      }
    }
  }
  // this warp's share is read: 4 TC_GROUPS arrivals free the accumulator, of which a warp of a single group makes TC_GROUPS
  tc_fence_before();
  __syncwarp();
  if (lane == 0) for (int h = 0; h < 2; ++h) if (mask >> h & 1) mbar_arrive_n(&d_empty[h], TC_GROUPS / groups);
}

// BIG: the decoders read out large items.  Without it they are one loop over the stages of all items (262 + 144 us for 1021 rows, 272 + 159
// with the items and their epilogue in it) and the epilogue warps do it.
template <int CB, bool GLU, bool BIG>
__global__ void __launch_bounds__(TC_THREADS, 1)
exl3_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ Exl3TcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* xp = reinterpret_cast<float*>(smem + TC_XP_OFF);
  uint64_t* b_full = reinterpret_cast<uint64_t*>(smem + TC_BAR_OFF);
  uint64_t* b_empty = b_full + TC_BSTAGES;
  uint64_t* t_full = b_empty + TC_BSTAGES;
  uint64_t* t_empty = t_full + TC_TSTAGES;
  uint64_t* a_full = t_empty + TC_TSTAGES;
  uint64_t* a_empty = a_full + TC_A_BUFS;
  uint64_t* d_full = a_empty + TC_A_BUFS;
  uint64_t* d_big = d_full + 2;
  uint64_t* d_empty = d_big + 1;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(d_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int NT = a.N >> 4, stages = a.K >> 6;
  const int F = a.N >> 1;
  const int strips = GLU ? F >> 7 : (a.N + 255) >> 8;
  const int total = *a.ntile * strips;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < TC_BSTAGES; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
    for (int s = 0; s < TC_TSTAGES; ++s) { mbar_init(&t_full[s], 1); mbar_init(&t_empty[s], TC_DECODERS); }
    for (int s = 0; s < TC_A_BUFS; ++s) { mbar_init(&a_full[s], TC_DECODERS); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&d_full[s], 1); mbar_init(&d_empty[s], 4 * TC_GROUPS); }
    mbar_init(d_big, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc<512>(tmem_ptr); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr, tmem_a = tmem + TC_D_COLS;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    // (the whole warp walks the loops of both issuing roles and one elected lane issues: what the instructions want in uniform
    // registers stays there.  1021 rows of 512 experts 390 + 210 -> 271 + 147 us, 8192 rows 1180 + 720 -> 863 + 552)
    int st = 0; uint32_t ph = 0; bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int expert = __shfl_sync(0xffffffffu, it.expert, 0);
      const bool one = !GLU && it.strip * 16 + 8 >= NT;                    // only 128 columns left
      const uint32_t* tw = a.trellis + expert * a.t_stride + static_cast<size_t>(it.strip) * (GLU ? 8 : 16) * 32;
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&t_empty[st], ph ^ 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, s); break; }
        if (elect_one()) {
          uint8_t* p = smem + TC_T_OFF + st * TC_T_BYTES;
          mbar_arrive_expect_tx(&t_full[st], one ? TC_T_BYTES / 2 : TC_T_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t* src = tw + static_cast<size_t>(s * 4 + k) * NT * 32;
            if (GLU) {
              bulk_load(p + k * 2048, src, 1024, &t_full[st]);
              bulk_load(p + k * 2048 + 1024, src + (F >> 4) * 32, 1024, &t_full[st]);
            } else {
              bulk_load(p + k * 2048, src, one ? 1024 : 2048, &t_full[st]);
            }
          }
        }
        __syncwarp();
        if (++st == TC_TSTAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 22) {
    // ------------------------------------------------------------ second producer: the rows, boxes of 32
    int st = 0; uint32_t ph = 0; bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int boxes = __shfl_sync(0xffffffffu, (it.n + 31) >> 5, 0), row0 = __shfl_sync(0xffffffffu, it.row0, 0);
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&b_empty[st], ph ^ 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, -s - 1); break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&b_full[st], boxes * 4096);
          for (int i = 0; i < boxes; ++i) tma_load_2d(smem + st * TC_B_BYTES + i * 4096, &tmX, &b_full[st], s * 64, row0 + i * 32);
        }
        __syncwarp();
        if (++st == TC_BSTAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t s_base = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
    int st = 0, ab = 0; uint32_t ph = 0, aph = 0, uses[2] = {0u, 0u}; bool ok = true;
    AccRing ring;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int n = __shfl_sync(0xffffffffu, it.n, 0);
      const int mask = ring.take(n);
      for (int h = 0; h < 2; ++h)
        if (mask >> h & 1) {
          if (!__all_sync(0xffffffffu, mbar_wait(&d_empty[h], (uses[h] & 1) ^ 1))) { set_status(a.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, t, h); ok = false; }
          ++uses[h];
        }
      if (!ok) break;
      tc_fence_after();
      const uint32_t idesc = make_idesc(0, 0, 128, n);
      const uint32_t d0 = tm + (mask == 2 ? TC_ROWS : 0), d1 = d0 + (mask == 3 ? TC_ROWS : TC_ROWS / 2);
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&b_full[st], ph) && mbar_wait(&a_full[ab], aph));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, s); break; }
        tc_fence_after();
        const uint64_t bd = make_smem_desc_sw128(s_base + st * TC_B_BYTES);
        const uint32_t ta = tm + TC_D_COLS + ab * TC_A_COLS;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_f16_ts(d0, ta + k * 16, bd + 2 * k, idesc, (s | k) != 0);
            umma_f16_ts(d1, ta + k * 16 + 8, bd + 2 * k, idesc, (s | k) != 0);
          }
          umma_commit(&b_empty[st]);
          umma_commit(&a_empty[ab]);
          if (s == stages - 1) umma_commit(mask == 3 ? d_big : &d_full[mask >> 1]);
        }
        __syncwarp();
        if (++st == TC_BSTAGES) { st = 0; ph ^= 1; }
        if (++ab == TC_A_BUFS) { ab = 0; aph ^= 1; }
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------ epilogue (BIG: of items that take one half)
    AccRing ring;
    uint32_t u0 = 0u, u1 = 0u, u2 = 0u;
    int buf = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int mask = ring.take(it.n);
      if (BIG && mask == 3) continue;
      const uint32_t use = mask == 1 ? u0++ : mask == 2 ? u1++ : u2++;
      if (!tc_wait_acc(mask == 3 ? d_big : &d_full[mask >> 1], use & 1, 1)) { set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, 0); break; }
      tc_epilogue<GLU>(a, it, mask, tmem, xp, 0, 1, 1, buf, d_empty);
    }
  } else {
    // ------------------------------------------------------------ decoders: two groups of eight warps take the stages in turn (so that
    // one group's waits lie under the other's decode), a warp k-tiles 2 p and 2 p + 1 of a stage, tiles 4 q .. 4 q + 3 of the strip
    const int q = warp & 3, p = ((warp - 6) >> 2) & 1, set = (warp - 6) >> 3;
    const uint32_t ta = tmem_a + set * TC_A_COLS + p * 32 + (static_cast<uint32_t>(q * 32) << 16);
    const uint8_t* src = smem + TC_T_OFF + p * 4096 + q * 512 + lane * 16;
    const int from = (lane & 24) | ((lane + 7) & 7);          // lane with the word before this lane's first (a tile is a ring)
    int st = set; uint32_t ph = 0, aph = 0; bool ok = true;
    auto decode = [&](int s) {                                // this group's next stage
      ok = __all_sync(0xffffffffu, mbar_wait(&t_full[st], ph));
      if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, -1, s); return; }
      uint4 w[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) w[k] = *reinterpret_cast<const uint4*>(src + st * TC_T_BYTES + k * 2048);
      __syncwarp();
      if (lane == 0) mbar_arrive(&t_empty[st]);
      uint32_t r[32];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t prev = __shfl_sync(0xffffffffu, w[k].w, from);
        uint32_t* d = r + 16 * k;
        uint32_t f[4];
        exl3_decode8_b4<CB>(w[k].x, prev, f);   d[0] = f[0]; d[4] = f[1]; d[8] = f[2]; d[12] = f[3];
        exl3_decode8_b4<CB>(w[k].y, w[k].x, f); d[1] = f[0]; d[5] = f[1]; d[9] = f[2]; d[13] = f[3];
        exl3_decode8_b4<CB>(w[k].z, w[k].y, f); d[2] = f[0]; d[6] = f[1]; d[10] = f[2]; d[14] = f[3];
        exl3_decode8_b4<CB>(w[k].w, w[k].z, f); d[3] = f[0]; d[7] = f[1]; d[11] = f[2]; d[15] = f[3];
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&a_empty[set], aph ^ 1));
      if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, -1, s); return; }
      tc_fence_after();
      tmem_st_32x32(ta, r);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&a_full[set]);
      aph ^= 1;
      st += 2;
      if (st >= TC_TSTAGES) { st -= TC_TSTAGES; ph ^= 1; }
    };
    if (!BIG) {
      const int mine = total > static_cast<int>(blockIdx.x) ? (total - 1 - blockIdx.x) / gridDim.x + 1 : 0;
      for (int s = set; s < mine * stages && ok; s += 2) decode(s);
    } else {
      const int group = (warp - 6) / 4;
      AccRing ring;
      int none = 0, next = set; uint32_t big = 0;                       // next: this group's next stage, from the item's first
      // (a warp whose wait ran out decodes no more, but still meets its group at every large item)
      for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const TcItem it = tc_item(a, t, strips);
        for (; next < stages && ok; next += 2) decode(next);
        next -= stages;
        if (ring.take(it.n) == 3) {
          // nothing is decoded while a large item is read out: the sixteen decoders do that
          ok = tc_wait_acc(d_big, big++ & 1, 2 + group, ok);
          if (ok) tc_epilogue<GLU>(a, it, 3, tmem, xp, group, TC_GROUPS, 2 + group, none, d_empty);
          else set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, group);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc<512>(tmem); }
}

template <int CB, bool GLU, bool BIG>
static int launch_tc(const CUtensorMap& tm, const Exl3TcArgs& a, int max_items, cudaStream_t s) {
  auto kern = exl3_tc_kernel<CB, GLU, BIG>;
  static int sms = 0;
  if (!sms) {
    int dev;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
  }
  kern<<<max_items < sms ? max_items : sms, TC_THREADS, TC_SMEM, s>>>(tm, a);
  return spark_launch_rc("spark_exl3_tc");
}

}  // namespace spark

using namespace spark;

// xh fp16 [P, K] (row stride ldx), rows in expert order; tiles = the tile list of the MoE sort (128 rows, or even ones of
// up to 192; max_tiles allocated, *ntile valid); big: many of them have more than 96 rows.  K, N multiples of 128.  glu: N = 2F with F % 128 == 0, `suh2` [E][F], y fp16 [P, F]; else y [P, N] fp32 / bf16.
extern "C" int spark_exl3_tc(const void* xh, int ldx, int P, const void* trellis, const void* svh, long long t_stride_words,
                             long long svh_stride, const void* suh2, long long suh2_stride, const void* tiles, const int* ntile,
                             int max_tiles, void* y, int ldy, int out_f32, int K, int N, int glu, float limit, int codebook,
                             int* status, cudaStream_t s, int big) {
  if (max_tiles <= 0 || P <= 0) return 0;
  if ((K & 127) || (N & 127) || K <= 0 || N <= 0 || (ldx & 7) || (ldy & 3) || (glu && (N & 255))) return -5;
  if (reinterpret_cast<uintptr_t>(trellis) & 15) return -5;
  CUtensorMap tm;
  if (int r = make_tmap_bf16(&tm, xh, P, K, ldx, 32, 0)) return r;
  Exl3TcArgs a;
  a.trellis = (const uint32_t*)trellis; a.t_stride = t_stride_words; a.svh = (const __half*)svh; a.svh_stride = svh_stride;
  a.suh2 = (const __half*)suh2; a.suh2_stride = suh2_stride; a.tiles = (const int4*)tiles; a.ntile = ntile;
  a.y = y; a.ldy = ldy; a.out_f32 = out_f32; a.K = K; a.N = N; a.limit = limit; a.status = status;
  a.wide = (ldy & 7) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  const int items = max_tiles * (glu ? N / 256 : (N + 255) / 256);
#define SPARK_TC(CB) (big ? (glu ? launch_tc<CB, true, true>(tm, a, items, s) : launch_tc<CB, false, true>(tm, a, items, s)) \
                          : (glu ? launch_tc<CB, true, false>(tm, a, items, s) : launch_tc<CB, false, false>(tm, a, items, s)))
  return codebook == 0 ? SPARK_TC(0) : SPARK_TC(1);
#undef SPARK_TC
}
