// EXL3 grouped GEMM of prompt-size MoE batches on tcgen05: packed trellises -> fp16 operands in tensor memory.
//   plain: y[rows, N]   = had128(xh @ inner_e) * svh_e                                   (fp32 or bf16)
//   glu:   y[rows, F]   = had128(bf16(act(gate) * up) * suh2_e) as fp16, the input rows of the down product
// with xh = had128(x * suh_e) in fp16, rows in expert order, work items of one expert and <= 128 rows.
//
// The product runs transposed: the weights are the 128-row M operand, the rows of the item the N operand (a multiple of 16, so
// that 20 rows of an expert cost 32 columns and not 128).  A lane that takes four consecutive words of a packed tile owns all 16 k
// of two output columns (c and c + 8), which is one K = 16 row of an A operand in tensor memory each: the decoded values go from
// the registers straight to TMEM (tcgen05.st), never through shared memory, and the two column halves are two accumulators.
//
// Roles (one CTA per SM, 22 warps): warp 0 streams packed tiles (bulk copies) and activation boxes (TMA, 128-byte swizzle) into
// an 8-stage ring of 64 k; 16 warps decode, one 16-k tile row of a stage per group of four; warp 1 issues the MMAs; 4 warps
// run the epilogue (TMEM -> shared memory -> output Hadamard per row, one warp per 128-block).  Items of <= 64 rows use half of
// the accumulator columns each, so that one item's epilogue overlaps the next one's products.
//
// What bounds it: the decode takes half of the time or less.  A word of 8 weights costs about 35 instructions, of which 8 multiplies
// and 8 byte sums go through the half-rate FMA-heavy pipe and 15 through the half-rate ALU pipe: 194 us of issue for 512 experts of
// 2048 x 512, once, of the 271 + 147 measured at 1021 rows.  The rest is each decoder's chain per 64 k (wait, load, decode, wait, store,
// wait, arrive; four warps a scheduler in step).  8192 rows decode twice, 390 us of 861 + 550: items of more than 64 rows take both
// accumulator halves, so that nothing runs beside their epilogue, in which four warps transform a row at a time.
// Reference: engine-rs/shim/moe_exl3.cuh:521-1233 (gemm_grouped / gux / gu2 kernels, mma.sync m16n8k16).
#include "exl3_common.cuh"

namespace spark {

int make_tmap_bf16(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K, uint64_t ld, int box_rows, int fmt);

struct Exl3TcArgs {
  const uint32_t* trellis; long long t_stride;        // [E][K/16][N/16][32] words
  const __half* svh; long long svh_stride;            // [E][N]
  const __half* suh2; long long suh2_stride;          // glu: [E][F] input scales of the next product
  const int4* tiles; const int* ntile;                // {row0, row_end, expert, 0}: <= 128 rows each, and their count
  void* y; int ldy; int out_f32;
  int K, N; float limit;
  int* status;
};

constexpr int TC_STAGES = 8, TC_THREADS = 22 * 32, TC_DECODERS = 16;
constexpr int TC_B_BYTES = 128 * 128, TC_T_BYTES = 4 * 16 * 128, TC_STAGE = TC_B_BYTES + TC_T_BYTES;
constexpr int TC_XP = 2 * 16 * 256 * 4;               // epilogue exchange: two buffers of 16 rows x 256 columns
constexpr int TC_SMEM = TC_STAGES * TC_STAGE + TC_XP + 256 + 1024;
constexpr int TC_A_COLS = 64, TC_A_BUFS = 4, TC_D_COLS = 256;

// Accumulator halves an item takes, the same sequence in the MMA and the epilogue role: an item of <= 64 rows takes the next
// half, a larger one both.
struct AccRing {
  int half = 0;
  uint32_t uses[2] = {0u, 0u};
  __device__ __forceinline__ int take(int n) { const int m = n <= 64 ? 1 << half : 3; half = n <= 64 ? half ^ 1 : 0; return m; }
};

struct TcItem { int row0, rows, n, expert, strip; };

__device__ __forceinline__ TcItem tc_item(const Exl3TcArgs& a, int t, int strips) {
  const int4 td = a.tiles[t / strips];
  TcItem it;
  it.row0 = td.x; it.rows = min(td.y - td.x, 128); it.n = (it.rows + 15) & ~15; it.expert = td.z; it.strip = t % strips;
  return it;
}

template <int CB, bool GLU>
__global__ void __launch_bounds__(TC_THREADS, 1)
exl3_tc_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ Exl3TcArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* xp = reinterpret_cast<float*>(smem + TC_STAGES * TC_STAGE);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + TC_STAGES * TC_STAGE + TC_XP);
  uint64_t* empty = full + TC_STAGES;
  uint64_t* a_full = empty + TC_STAGES;
  uint64_t* a_empty = a_full + TC_A_BUFS;
  uint64_t* d_full = a_empty + TC_A_BUFS;
  uint64_t* d_empty = d_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(d_empty + 2);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int NT = a.N >> 4, stages = a.K >> 6;
  const int F = a.N >> 1;
  const int strips = GLU ? F >> 7 : (a.N + 255) >> 8;
  const int total = *a.ntile * strips;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < TC_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < TC_A_BUFS; ++s) { mbar_init(&a_full[s], TC_DECODERS); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&d_full[s], 1); mbar_init(&d_empty[s], 4); }
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
      const int boxes = __shfl_sync(0xffffffffu, (it.n + 31) >> 5, 0), row0 = __shfl_sync(0xffffffffu, it.row0, 0);
      const int expert = __shfl_sync(0xffffffffu, it.expert, 0);
      const bool one = !GLU && it.strip * 16 + 8 >= NT;                    // only 128 columns left
      const uint32_t* tw = a.trellis + expert * a.t_stride + static_cast<size_t>(it.strip) * (GLU ? 8 : 16) * 32;
      const uint32_t bytes = boxes * 4096 + (one ? TC_T_BYTES / 2 : TC_T_BYTES);
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[st], ph ^ 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, s); break; }
        if (elect_one()) {
          uint8_t* b = smem + st * TC_STAGE;
          uint8_t* p = b + TC_B_BYTES;
          mbar_arrive_expect_tx(&full[st], bytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t* src = tw + static_cast<size_t>(s * 4 + k) * NT * 32;
            if (GLU) {
              bulk_load(p + k * 2048, src, 1024, &full[st]);
              bulk_load(p + k * 2048 + 1024, src + (F >> 4) * 32, 1024, &full[st]);
            } else {
              bulk_load(p + k * 2048, src, one ? 1024 : 2048, &full[st]);
            }
          }
          for (int i = 0; i < boxes; ++i) tma_load_2d(b + i * 4096, &tmX, &full[st], s * 64, row0 + i * 32);
        }
        __syncwarp();
        if (++st == TC_STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t s_base = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
    int st = 0, ab = 0; uint32_t ph = 0, aph = 0; bool ok = true;
    AccRing ring;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int n = __shfl_sync(0xffffffffu, it.n, 0);
      const int mask = ring.take(n);
      for (int h = 0; h < 2; ++h)
        if (mask >> h & 1) {
          if (!__all_sync(0xffffffffu, mbar_wait(&d_empty[h], (ring.uses[h] & 1) ^ 1))) { set_status(a.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, t, h); ok = false; }
          ++ring.uses[h];
        }
      if (!ok) break;
      tc_fence_after();
      const uint32_t idesc = make_idesc(0, 0, 128, n);
      const uint32_t d0 = tm + (mask == 2 ? 128 : 0), d1 = d0 + (mask == 3 ? 128 : 64);
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[st], ph) && mbar_wait(&a_full[ab], aph));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, s); break; }
        tc_fence_after();
        const uint64_t bd = make_smem_desc_sw128(s_base + st * TC_STAGE);
        const uint32_t ta = tm + TC_D_COLS + ab * TC_A_COLS;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_f16_ts(d0, ta + k * 16, bd + 2 * k, idesc, (s | k) != 0);
            umma_f16_ts(d1, ta + k * 16 + 8, bd + 2 * k, idesc, (s | k) != 0);
          }
          umma_commit(&empty[st]);
          umma_commit(&a_empty[ab]);
          if (s == stages - 1)
            for (int h = 0; h < 2; ++h)
              if (mask >> h & 1) umma_commit(&d_full[h]);
        }
        __syncwarp();
        if (++st == TC_STAGES) { st = 0; ph ^= 1; }
        if (++ab == TC_A_BUFS) { ab = 0; aph ^= 1; }
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;                                   // TMEM lanes [32 q, 32 q + 32): columns 64 q .. 64 q + 63 of the strip
    AccRing ring;
    int buf = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      const TcItem it = tc_item(a, t, strips);
      const int mask = ring.take(it.n);
      bool ok = true;
      for (int h = 0; h < 2; ++h)
        if (mask >> h & 1) { ok = ok && mbar_wait(&d_full[h], ring.uses[h] & 1); ++ring.uses[h]; }
      // all four warps take the same way: the exchange below has barriers of the group
      int bad = !ok;
      asm volatile("{\n.reg .pred p, r;\nsetp.ne.b32 p, %0, 0;\nbarrier.cta.red.or.pred r, 1, 128, p;\nselp.b32 %0, 1, 0, r;\n}\n" : "+r"(bad)::"memory");
      if (bad) { set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, 0); break; }
      tc_fence_after();
      const uint32_t d0 = tmem + (mask == 2 ? 128 : 0) + (static_cast<uint32_t>(q * 32) << 16), d1 = d0 + (mask == 3 ? 128 : 64);
      const __half* svh = a.svh + it.expert * a.svh_stride;
      // the lane's four columns of a 128-block n = 64 q' + 16 tile + 8 half + c, as the exchange holds them
      const int pos = (lane >> 4) * 64 + ((lane >> 1) & 1) * 32 + ((lane >> 2) & 3) * 8 + (lane & 1) * 4;
      const int c0 = GLU ? it.strip * 128 : it.strip * 256;
      const bool one = !GLU && it.strip * 16 + 8 >= NT;
      float sc[2][4], s2[4];
      {
        const int cb1 = GLU ? F + c0 : (one ? c0 : c0 + 128);
        const uint2 r0 = *reinterpret_cast<const uint2*>(svh + c0 + lane * 4), r1 = *reinterpret_cast<const uint2*>(svh + cb1 + lane * 4);
        const __half2 *h0 = reinterpret_cast<const __half2*>(&r0), *h1 = reinterpret_cast<const __half2*>(&r1);
        float2 f = __half22float2(h0[0]); sc[0][0] = f.x * INV_SQRT_128; sc[0][1] = f.y * INV_SQRT_128;
        f = __half22float2(h0[1]); sc[0][2] = f.x * INV_SQRT_128; sc[0][3] = f.y * INV_SQRT_128;
        f = __half22float2(h1[0]); sc[1][0] = f.x * INV_SQRT_128; sc[1][1] = f.y * INV_SQRT_128;
        f = __half22float2(h1[1]); sc[1][2] = f.x * INV_SQRT_128; sc[1][3] = f.y * INV_SQRT_128;
        if (GLU) {
          const uint2 r2 = *reinterpret_cast<const uint2*>(a.suh2 + it.expert * a.suh2_stride + c0 + lane * 4);
          const __half2* h2 = reinterpret_cast<const __half2*>(&r2);
          f = __half22float2(h2[0]); s2[0] = f.x; s2[1] = f.y;
          f = __half22float2(h2[1]); s2[2] = f.x; s2[3] = f.y;
        }
      }
      for (int c = 0; c < it.n; c += 16) {
        uint32_t v0[16], v1[16];
        tmem_ld_32x16(d0 + c, v0);
        tmem_ld_32x16(d1 + c, v1);
        tmem_ld_wait();
        if (c + 16 >= it.n) {                                 // last columns read: the accumulator may be overwritten
          tc_fence_before();
          __syncwarp();
          if (lane == 0) for (int h = 0; h < 2; ++h) if (mask >> h & 1) mbar_arrive(&d_empty[h]);
        }
        float* x = xp + buf * (16 * 256);
        buf ^= 1;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          x[i * 256 + q * 64 + lane] = __uint_as_float(v0[i]);
          x[i * 256 + q * 64 + 32 + lane] = __uint_as_float(v1[i]);
        }
        asm volatile("barrier.cta.sync 1, 128;" ::: "memory");
        const int live = min(16, it.rows - c);
        for (int r = q; r < live; r += 4) {
          float v[2][4];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const float4 p = *reinterpret_cast<const float4*>(x + r * 256 + b * 128 + pos);
            v[b][0] = p.x; v[b][1] = p.y; v[b][2] = p.z; v[b][3] = p.w;
            fwht128_warp(v[b], lane);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[b][i] *= sc[b][i];
          }
          const size_t row = static_cast<size_t>(it.row0 + c + r) * a.ldy;
          if (GLU) {
            float u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float gg = __bfloat162float(__float2bfloat16(v[0][i])), uu = __bfloat162float(__float2bfloat16(v[1][i]));
              if (a.limit > 0.f) { gg = fminf(gg, a.limit); uu = fminf(fmaxf(uu, -a.limit), a.limit); }
              u[i] = __bfloat162float(__float2bfloat16(gg / (1.f + __expf(-gg)) * uu)) * s2[i];
            }
            fwht128_warp(u, lane);
            const __half2 h0 = __floats2half2_rn(u[0] * INV_SQRT_128, u[1] * INV_SQRT_128);
            const __half2 h1 = __floats2half2_rn(u[2] * INV_SQRT_128, u[3] * INV_SQRT_128);
            uint2 o; o.x = *reinterpret_cast<const uint32_t*>(&h0); o.y = *reinterpret_cast<const uint32_t*>(&h1);
            *reinterpret_cast<uint2*>(static_cast<__half*>(a.y) + row + c0 + lane * 4) = o;
          } else {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              if (b && one) break;
              const size_t o = row + c0 + b * 128 + lane * 4;
              if (a.out_f32) {
                *reinterpret_cast<float4*>(static_cast<float*>(a.y) + o) = make_float4(v[b][0], v[b][1], v[b][2], v[b][3]);
              } else {
                const __nv_bfloat162 b0 = __floats2bfloat162_rn(v[b][0], v[b][1]), b1 = __floats2bfloat162_rn(v[b][2], v[b][3]);
                uint2 ov; ov.x = *reinterpret_cast<const uint32_t*>(&b0); ov.y = *reinterpret_cast<const uint32_t*>(&b1);
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(a.y) + o) = ov;
              }
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ decoders: k-tile g of every stage, tiles 4 q .. 4 q + 3 of the strip
    const int q = warp & 3, g = (warp - 6) >> 2;
    const uint32_t ta = tmem_a + g * 16 + (static_cast<uint32_t>(q * 32) << 16);
    const uint8_t* src = smem + TC_B_BYTES + g * 2048 + q * 512 + lane * 16;
    const int from = (lane & 24) | ((lane + 7) & 7);          // lane with the word before this lane's first (a tile is a ring)
    int st = 0, ab = 0; uint32_t ph = 0, aph = 0; bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      for (int s = 0; s < stages; ++s) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[st], ph));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, s); break; }
        const uint4 w = *reinterpret_cast<const uint4*>(src + st * TC_STAGE);
        const uint32_t prev = __shfl_sync(0xffffffffu, w.w, from);
        uint32_t r[16], f[4];
        exl3_decode8_b4<CB>(w.x, prev, f); r[0] = f[0]; r[4] = f[1]; r[8] = f[2]; r[12] = f[3];
        exl3_decode8_b4<CB>(w.y, w.x, f);  r[1] = f[0]; r[5] = f[1]; r[9] = f[2]; r[13] = f[3];
        exl3_decode8_b4<CB>(w.z, w.y, f);  r[2] = f[0]; r[6] = f[1]; r[10] = f[2]; r[14] = f[3];
        exl3_decode8_b4<CB>(w.w, w.z, f);  r[3] = f[0]; r[7] = f[1]; r[11] = f[2]; r[15] = f[3];
        ok = __all_sync(0xffffffffu, mbar_wait(&a_empty[ab], aph ^ 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, s); break; }
        tc_fence_after();
        tmem_st_32x16(ta + ab * TC_A_COLS, r);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&a_full[ab]);
        if (++st == TC_STAGES) { st = 0; ph ^= 1; }
        if (++ab == TC_A_BUFS) { ab = 0; aph ^= 1; }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc<512>(tmem); }
}

template <int CB, bool GLU>
static int launch_tc(const CUtensorMap& tm, const Exl3TcArgs& a, int max_items, cudaStream_t s) {
  auto kern = exl3_tc_kernel<CB, GLU>;
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

// xh fp16 [P, K] (row stride ldx), rows in expert order; tiles = the <= 128-row tile list of the MoE sort (max_tiles allocated,
// *ntile valid).  K, N multiples of 128.  glu: N = 2F with F % 128 == 0, `suh2` [E][F], y fp16 [P, F]; else y [P, N] fp32 / bf16.
extern "C" int spark_exl3_tc(const void* xh, int ldx, int P, const void* trellis, const void* svh, long long t_stride_words,
                             long long svh_stride, const void* suh2, long long suh2_stride, const void* tiles, const int* ntile,
                             int max_tiles, void* y, int ldy, int out_f32, int K, int N, int glu, float limit, int codebook,
                             int* status, cudaStream_t s) {
  if (max_tiles <= 0 || P <= 0) return 0;
  if ((K & 127) || (N & 127) || K <= 0 || N <= 0 || (ldx & 7) || (ldy & 3) || (glu && (N & 255))) return -5;
  if (reinterpret_cast<uintptr_t>(trellis) & 15) return -5;
  CUtensorMap tm;
  if (int r = make_tmap_bf16(&tm, xh, P, K, ldx, 32, 0)) return r;
  Exl3TcArgs a;
  a.trellis = (const uint32_t*)trellis; a.t_stride = t_stride_words; a.svh = (const __half*)svh; a.svh_stride = svh_stride;
  a.suh2 = (const __half*)suh2; a.suh2_stride = suh2_stride; a.tiles = (const int4*)tiles; a.ntile = ntile;
  a.y = y; a.ldy = ldy; a.out_f32 = out_f32; a.K = K; a.N = N; a.limit = limit; a.status = status;
  const int items = max_tiles * (glu ? N / 256 : (N + 255) / 256);
  if (codebook == 0) return glu ? launch_tc<0, true>(tm, a, items, s) : launch_tc<0, false>(tm, a, items, s);
  return glu ? launch_tc<1, true>(tm, a, items, s) : launch_tc<1, false>(tm, a, items, s);
}
