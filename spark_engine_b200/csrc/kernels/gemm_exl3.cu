// Prompt-size EXL3 projections:  y[M, N] = had128(xh[M, K] W[N, K]^T) * svh  (fp16 in, bf16 out), W the reconstructed inner weights.
// The output transform is the epilogue: a thread owns a row and has the 128 columns of a block in registers.
//
// CTA pairs (cta_group::2): a pair computes 256 x BN, every CTA brings its 128 rows of A and half of the rows of W into its own shared
// memory, and the leader issues for both.  What bounds it: a CTA by itself (128 x 256) asks L2 for 48 KB per 512 cycles of products, more than
// the 64 bytes a cycle an SM gets; a pair asks for 32 KB per CTA.  The transform as a pass of its own wrote and read the products in fp32
// (12 bytes per output where 2 are left).  4096 rows of 2048 x 12288 and 4096 x 2048, product and transform: 342 -> 215 us.  Few rows of
// wide matrices are left to the two launches (`exl3_linear`).
//   warp 0      TMA: both CTAs' tiles are counted by the leader's barrier
//   warp 1      the leader's issues the MMAs; commits reach both CTAs
//   warps 2..5  epilogue of the CTA's 128 rows, two accumulator stages
#include "exl3_common.cuh"

namespace spark {

int make_tmap_bf16(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K, uint64_t ld, int box_rows, int fmt);

struct GemmExl3Args {
  int M, N, K, nt_n, tiles;
  const __half* svh;
  __nv_bfloat16* C; int ldc, wide;                    // wide: rows of C start on 16 bytes (else 8)
  int* status;
};

constexpr int GX_BM = 128, GX_BK = 64, GX_THREADS = 192;       // rows of a CTA
template <int BN> struct Gx {
  static constexpr int A_BYTES = GX_BM * GX_BK * 2, B_BYTES = BN / 2 * GX_BK * 2, STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 256 ? 6 : 8, SMEM = STAGES * STAGE + 256 + 1024;
  static constexpr int COLS = 2 * BN;                 // two accumulator stages
};

__device__ __forceinline__ uint32_t gx_leader(const void* p) {           // the leader's copy of a shared variable
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ void gx_load(void* dst, const CUtensorMap* m, uint32_t leader_bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void gx_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void gx_commit_both(uint64_t* bar) {           // arrives on the barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void gx_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool gx_wait_cluster(uint64_t* bar, uint32_t parity) {      // bounded, arrivals of both CTAs
  const uint64_t t0 = global_timer_ns();
  for (uint32_t i = 0; i < SPARK_WAIT_POLLS; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred P;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n"
        "selp.u32 %0, 1, 0, P;\n"
        "}\n" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 15u) == 15u && global_timer_ns() - t0 > SPARK_WAIT_NS) return false;
  }
  return false;
}
__device__ __forceinline__ void gx_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 128-point transform of a thread's 128 values: the pairs of fwht128_oct in the same order
__device__ __forceinline__ void fwht128_thread(uint64_t (&p)[64]) {
  const uint64_t minus = f2_pack(-1.f, -1.f);
#pragma unroll
  for (int i = 0; i < 64; ++i) { float a, b; f2_unpack(p[i], a, b); p[i] = f2_pack(a + b, a - b); }
#pragma unroll
  for (int st = 1; st < 64; st <<= 1)
#pragma unroll
    for (int i = 0; i < 64; ++i)
      if (!(i & st)) { const uint64_t a = p[i], b = p[i | st]; p[i] = f2_add(a, b); p[i | st] = f2_fma(b, minus, a); }
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GX_THREADS, 1)
gemm_exl3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ GemmExl3Args g) {
  using S = Gx<BN>;
  constexpr int STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * S::STAGE);      // the leader's is in use
  uint64_t* empty = full + STAGES;
  uint64_t* t_full = empty + STAGES;                                           // [2]
  uint64_t* t_empty = t_full + 2;                                              // [2], the leader's is in use
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(t_empty + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int num_k = (g.K + GX_BK - 1) / GX_BK;
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&t_full[s], 1); mbar_init(&t_empty[s], 8); }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "n"(S::COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  gx_cluster_sync();                                                           // barriers of both CTAs are there
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    int st = 0; uint32_t ph = 0; bool ok = true;
    for (int t = pair; t < g.tiles && ok; t += pairs) {
      const int a_row = (t / g.nt_n) * 2 * GX_BM + rank * GX_BM, b_row = (t % g.nt_n) * BN + rank * (BN / 2);
      for (int kb = 0; kb < num_k; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[st], ph ^ 1));
        if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, t, kb); break; }
        if (elect_one()) {
          uint8_t* a_dst = smem + st * S::STAGE;
          const uint32_t bar = gx_leader(&full[st]);
          if (rank == 0) mbar_arrive_expect_tx(&full[st], 2 * S::STAGE);
          gx_load(a_dst, &tmA, bar, kb * GX_BK, a_row);
          gx_load(a_dst + S::A_BYTES, &tmB, bar, kb * GX_BK, b_row);
        }
        __syncwarp();
        if (++st == STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (the leader's)
    if (rank == 0) {
      const uint32_t idesc = make_idesc(0, 0, 2 * GX_BM, BN);
      const uint32_t s0 = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
      int st = 0, acc = 0; uint32_t ph = 0, aph = 0; bool ok = true;
      for (int t = pair; t < g.tiles && ok; t += pairs) {
        ok = __all_sync(0xffffffffu, gx_wait_cluster(&t_empty[acc], aph ^ 1));
        if (!ok) { set_status(g.status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, t, acc); break; }
        tc_fence_after();
        const uint32_t d = tm + acc * BN;
        for (int kb = 0; kb < num_k; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full[st], ph));
          if (!ok) { set_status(g.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, t, kb); break; }
          tc_fence_after();
          const uint64_t ad = make_smem_desc_sw128(s0 + st * S::STAGE), bd = make_smem_desc_sw128(s0 + st * S::STAGE + S::A_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < GX_BK / 16; ++k) gx_mma(d, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0);
            gx_commit_both(&empty[st]);
            if (kb == num_k - 1) gx_commit_both(&t_full[acc]);
          }
          __syncwarp();
          if (++st == STAGES) { st = 0; ph ^= 1; }
        }
        if (++acc == 2) { acc = 0; aph ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: a row of this CTA per thread
    const int q = warp & 3;
    int acc = 0; uint32_t aph = 0;
    for (int t = pair; t < g.tiles; t += pairs) {
      if (!__all_sync(0xffffffffu, mbar_wait(&t_full[acc], aph))) { set_status(g.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, t, acc); break; }
      tc_fence_after();
      const int row = (t / g.nt_n) * 2 * GX_BM + rank * GX_BM + q * 32 + lane, n0 = (t % g.nt_n) * BN;
      const uint32_t ta = tmem + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll 1
      for (int b = 0; b < BN; b += 128) {
        uint64_t p[64];
        {
          uint32_t r[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32(ta + b + c * 32, r[c]);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 64; ++i) p[i] = f2_pack(__uint_as_float(r[i >> 4][(2 * i) & 31]), __uint_as_float(r[i >> 4][(2 * i + 1) & 31]));
        }
        if (b + 128 >= BN) {                                                   // the accumulator is read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) gx_arrive_remote(gx_leader(&t_empty[acc]));
        }
        if (n0 + b >= g.N) continue;
        fwht128_thread(p);
        const uint2* sv = reinterpret_cast<const uint2*>(g.svh + n0 + b);
        const uint64_t inv = f2_pack(INV_SQRT_128, INV_SQRT_128);
        __nv_bfloat16* dst = g.C + static_cast<size_t>(row) * g.ldc + n0 + b;
#pragma unroll
        for (int i = 0; i < 16; ++i) {                                         // eight columns
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const uint2 w = __ldg(sv + 2 * i + j / 2);
            const float2 s0 = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), s1 = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
            float a, c;
            f2_unpack(f2_mul(f2_mul(p[4 * i + j], inv), f2_pack(s0.x, s0.y)), a, c);
            const __nv_bfloat162 h0 = __floats2bfloat162_rn(a, c);
            f2_unpack(f2_mul(f2_mul(p[4 * i + j + 1], inv), f2_pack(s1.x, s1.y)), a, c);
            const __nv_bfloat162 h1 = __floats2bfloat162_rn(a, c);
            o[j] = *reinterpret_cast<const uint32_t*>(&h0); o[j + 1] = *reinterpret_cast<const uint32_t*>(&h1);
          }
          if (row < g.M) {
            if (g.wide) {
              reinterpret_cast<uint4*>(dst)[i] = make_uint4(o[0], o[1], o[2], o[3]);
            } else {
              reinterpret_cast<uint2*>(dst)[2 * i] = make_uint2(o[0], o[1]);
              reinterpret_cast<uint2*>(dst)[2 * i + 1] = make_uint2(o[2], o[3]);
            }
          }
        }
      }
      if (++acc == 2) { acc = 0; aph ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  gx_cluster_sync();                                                           // nobody reads the other's memory or signals it any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(S::COLS) : "memory");
  }
}

template <int BN>
static int launch_gemm_exl3(const CUtensorMap& tA, const CUtensorMap& tB, const GemmExl3Args& g, int sms, cudaStream_t s) {
  static bool done = false;
  if (!done) { cudaFuncSetAttribute(gemm_exl3_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Gx<BN>::SMEM); done = true; }
  const int pairs = g.tiles < sms / 2 ? g.tiles : sms / 2;
  gemm_exl3_kernel<BN><<<2 * pairs, GX_THREADS, Gx<BN>::SMEM, s>>>(tA, tB, g);
  return spark_launch_rc("spark_gemm_exl3");
}

}  // namespace spark

using namespace spark;

// xh fp16 [M, K] (row stride lda), W fp16 [N, K], svh fp16 [N], C bf16 [M, N] (row stride ldc, a multiple of 4).  N and K multiples of 128; svh
// and C start on 8 bytes.
extern "C" int spark_gemm_exl3(const void* xh, int lda, const void* W, const void* svh, void* C, int ldc, int M, int N, int K, int* status,
                               cudaStream_t s) {
  if (M <= 0) return 0;
  if (N <= 0 || K <= 0 || (N & 127) || (K & 127) || (ldc & 3)) return -5;
  if ((reinterpret_cast<uintptr_t>(svh) | reinterpret_cast<uintptr_t>(C)) & 7) return -5;
  static int sms = 0;
  if (!sms) { int dev; cudaGetDevice(&dev); cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev); }
  const int mt = (M + 2 * GX_BM - 1) / (2 * GX_BM);
  // 256 columns once every pair has a tile of them; below, 128 put twice as many to work
  const int bn = mt * ((N + 255) / 256) >= sms / 2 ? 256 : 128;
  CUtensorMap tA, tB;
  if (int r = make_tmap_bf16(&tA, xh, M, K, lda, GX_BM, 0)) return r;
  if (int r = make_tmap_bf16(&tB, W, N, K, K, bn / 2, 0)) return r;
  GemmExl3Args g;
  g.M = M; g.N = N; g.K = K; g.nt_n = (N + bn - 1) / bn; g.tiles = mt * g.nt_n;
  g.svh = (const __half*)svh; g.C = (__nv_bfloat16*)C; g.ldc = ldc; g.status = status;
  g.wide = (ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  return bn == 256 ? launch_gemm_exl3<256>(tA, tB, g, sms, s) : launch_gemm_exl3<128>(tA, tB, g, sms, s);
}
