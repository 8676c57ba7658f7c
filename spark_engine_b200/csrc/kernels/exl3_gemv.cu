// EXL3 GEMV for <= 16 rows (decode / verify rows, MoE (row, expert) pairs):
//   y = had128( had128(x * suh) @ inner ) * svh
// One launch: input Hadamard, trellis decode, product, output Hadamard.  Grid (N/128, S, items) with a
// thread-block cluster of S CTAs along the K-slices of one 128-column strip.  Two warps share a k-tile of the strip (512 bytes each),
// four such pairs take every fourth k-tile of the slice with the loads of two in flight; a lane decodes 8 weights of a tile straight
// into the 16-row operand of one m16n8k16 product, whose 8 columns are the activation rows.  The warps' partial strips meet in
// shared memory, the slices' in that of cluster rank 0 (distributed shared memory), which adds them in order (no global
// scratch, no atomics), applies the output Hadamard transform and scales.  Fixed reduction order => bitwise reproducible and independent of the rows in flight.
// What bounds it: issue.  A tile of 256 weights takes about 35 instructions to decode and 46 in all; short slices add the transform of
// the activations and the ends of the pipeline, so that pairs get as few slices as still fill the SMs (`_pick_slices`).  us, before (weights as the
// 8-column operand of two products, a warp per 16 columns of every k-tile, slices of 256) and after: 40 pairs of 1024 x 2048 33.6 -> 27.6, of 2048 x 512,
// gated, 18.5 -> 15.2; 160 pairs 120 -> 81 and 60 -> 46; 16 pairs of 3072 x 4096 74 -> 55, of 4096 x 1536, gated, 41 -> 33; one row of
// 12288 x 2048 12.2 -> 10.2, of 2048 x 4096 8.9 -> 7.8.  40 pairs of 1024 x 2048: 51 instructions a tile in all, 65 % of the issue slots of the
// busy SMs, 49 % over the launch.
// M <= 16 is bandwidth / decode-ALU bound, so the warp-level MMA feeds it; GEMM-shaped EXL3 work goes
// through exl3_reconstruct to the tcgen05 GEMM.
// Replaces engine-rs/shim/qwen_exl3.cuh:427-626 (gemv_kernel / gemv_fused_kernel / finish_kernel) and
// the decode half of moe_exl3.cuh:273-399.
#include "exl3_common.cuh"
#include "../common/comm.cuh"
#include "../common/decode.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace spark {

struct Exl3GemvArgs {
  const __nv_bfloat16* x; int ldx;             // activations [rows, K] (or [rows, 2K] = [gate | up] when act == 1)
  const uint32_t* trellis;                      // [E][K/16][N/16][32] words (4 bpw)
  const __half* suh; const __half* svh;         // [E][K], [E][N]
  long long t_stride, suh_stride, svh_stride;   // per expert, in elements
  void* y; int ldy; int out_f32;                // [items*R, N]
  const int* pair_expert; const int* pair_row;
  int R, K, N, S, act; float limit;
  int fuse_ar;                                  // 1: row-parallel layer under TP: the epilogue pushes the strip to every
  ArRows ar;                                    //    rank's slots and raises the flag; a tail launch reduces the rows
  int pairs_early;                              // pair tables were written at least two launches back: they may be read
                                                // (and the weight loads issued) before the dependency wait
  int x_align;                                  // bytes that activation rows are aligned to: 16, 8 or 2
  int chunk;                                    // k-tiles that are summed before they join the others (see below)
};

constexpr int EXL3_MAX_KS = 2048;              // K-slice per CTA (activation slice lives in shared memory)
// n-tiles of a warp, k-tiles whose loads are in flight, warps of a CTA, warps that fit an SM (48 registers; 80 with 9 to 16 rows)
constexpr int EXL3_TN = 4, EXL3_DEPTH = 2, EXL3_WARPS = 8, EXL3_OCC = 40, EXL3_OCC2 = 24;

// Fused all-reduce, push side (kept out of line so that it costs the GEMV no registers): the last strip of this rank
// to finish raises this rank's flag on every peer.  The reduction itself (wait for every rank's flag, rank-ordered
// sum + residual + RMSNorm) runs as a second launch with one CTA per row (ar_tail_kernel): a single finisher CTA
// serialised all rows (measured 29 us for 4 rows against 6 + 11 us for the GEMV and a stand-alone all-reduce).
__device__ __noinline__ void exl3_fused_ar_arrive(const Exl3GemvArgs& a) {
  const uint32_t seq = comm_seq(a.ar.seq_ptr, a.ar.seq);
  __syncthreads();
  if (threadIdx.x == 0) {
    ArRows ar = a.ar;
    ar.seq_ptr = nullptr;                                  // the tail kernel closes the sequence
    ar_arrive_and_is_last(ar, seq, gridDim.x);
  }
}

// 16 consecutive activations of a row as floats; `al`: bytes the rows are aligned to (16, 8 or 2)
__device__ __forceinline__ void exl3_ld16(const __nv_bfloat16* p, int al, float (&v)[16]) {
  uint32_t w[8];
  if (al == 16) {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else if (al == 8) {
#pragma unroll
    for (int i = 0; i < 4; ++i) { const uint2 a = reinterpret_cast<const uint2*>(p)[i]; w[2 * i] = a.x; w[2 * i + 1] = a.y; }
  } else {
    const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = h[2 * i] | static_cast<uint32_t>(h[2 * i + 1]) << 16;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}

__device__ __forceinline__ void exl3_ld4(const __nv_bfloat16* p, int al, float (&v)[4]) {
  uint32_t w[2];
  if (al >= 8) {
    const uint2 a = *reinterpret_cast<const uint2*>(p);
    w[0] = a.x; w[1] = a.y;
  } else {
    const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
    w[0] = h[0] | static_cast<uint32_t>(h[1]) << 16; w[1] = h[2] | static_cast<uint32_t>(h[3]) << 16;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
__device__ __forceinline__ float exl3_gate(float g, float u, float limit) {
  if (limit > 0.f) { g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit); }
  return g / (1.f + __expf(-g)) * u;
}
// fwht128_warp of v * (s0, s1); the first stage's products are fused with its sums, as the compiler does it ahead of fwht128_oct (a test
// holds the two together: a row's bits must not depend on how many there are)
__device__ __forceinline__ void exl3_fwht128_scaled(float (&v)[4], float2 s0, float2 s1, int lane) {
  const float p1 = __fmul_rn(v[1], s0.y), p3 = __fmul_rn(v[3], s1.y);
  const float a = __fmaf_rn(v[0], s0.x, p1), b = __fmaf_rn(v[0], s0.x, -p1), c = __fmaf_rn(v[2], s1.x, p3), d = __fmaf_rn(v[2], s1.x, -p3);
  v[0] = a + c; v[2] = a - c; v[1] = b + d; v[3] = b - d;
#pragma unroll
  for (int m = 1; m < 32; m <<= 1)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float o = __shfl_xor_sync(0xffffffffu, v[i], m);
      v[i] = (lane & m) ? o - v[i] : v[i] + o;
    }
}

template <int CB, int NB>                  // NB: blocks of 8 activation rows
__global__ void __launch_bounds__(EXL3_WARPS * 32, (NB == 1 ? EXL3_OCC : EXL3_OCC2) / EXL3_WARPS)
exl3_gemv_kernel(const __grid_constant__ Exl3GemvArgs a) {
  constexpr int WARPS = EXL3_WARPS, WN = 8 / EXL3_TN, WK = WARPS / WN;              // WN warps share a k-tile's eight n-tiles
  // (the argument block stays in constant memory: a local copy would put every field access on the stack)
  // Weight loads depend on no earlier launch; everything else is read after the dependency wait.
  const bool early = a.pair_expert == nullptr || a.pairs_early;
  if (!early) pdl_wait();
  if (a.pair_expert && a.pair_expert[blockIdx.z] < 0) {         // expert on another rank (whole cluster leaves)
    if (early) pdl_wait();
    return;
  }
  extern __shared__ __align__(16) uint8_t smem_dyn[];
  __half* xh = reinterpret_cast<__half*>(smem_dyn);          // [R][Ks + 16]
  cg::cluster_group cluster = cg::this_cluster();
  const int strip = blockIdx.x, slice = blockIdx.y, item = blockIdx.z;
  const int R = a.R;
  const int NT = a.N >> 4;
  const int Ks = a.K / a.S, kts = Ks >> 4;
  const int ldh = Ks + 16;                                    // rows 32 bytes apart modulo 128: four rows' 32-byte pieces miss each other
  float* red = reinterpret_cast<float*>(smem_dyn + R * ldh * 2);    // [S * chunks][R][128]: partials, used on rank 0
  const int nch = kts / a.chunk;                                    // chunks of this slice
  float* part = red + a.S * nch * R * 128;                          // [chunks][WK][R][128]: the warps' partials
  const int k_begin = slice * Ks;
  const int e = a.pair_expert ? a.pair_expert[item] : 0;
  const int xr0 = a.pair_row ? a.pair_row[item] : item * R;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wn = warp % WN, wk = warp / WN;

  // every CTA of the cluster must be running before its shared memory is written remotely: arrive now, wait
  // right before the first remote store
  if (a.S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // ---- issue this warp's first trellis loads (they do not depend on the prologue)
  const int nk = kts / WK, per = a.chunk / WK;                // k-tiles wk, wk + WK, ..., `per` of them in a chunk
  const uint32_t* tw = a.trellis + e * a.t_stride + (static_cast<size_t>(slice * kts + wk) * NT + strip * 8 + wn * EXL3_TN) * 32 + lane;
  const size_t tstep = static_cast<size_t>(NT) * 32 * WK;
  uint32_t buf[EXL3_DEPTH][EXL3_TN];
#pragma unroll
  for (int d = 0; d < EXL3_DEPTH; ++d) {
    if (d < nk) {
#pragma unroll
      for (int j = 0; j < EXL3_TN; ++j) buf[d][j] = __ldg(tw + j * 32);
    }
    tw += tstep;
  }

  if (early) pdl_wait();
  // ---- prologue: xh = had128(x * suh) / sqrt(128) for this K-slice; eight lanes per 128-block, a lane holds one k-tile of its row and
  // stores it in the order in which the products' lanes take it: k = 2t, 2t + 1, 2t + 8, 2t + 9 for t = 0 .. 3
  const __half* suh = a.suh + e * a.suh_stride + k_begin;
  const int nblk = Ks >> 7, jobs = R * nblk;
  if (a.act == 1 && jobs <= 2 * WARPS) {
    // few gated blocks (a pair's, as a rule): a warp each, so that a lane has four gates instead of sixteen one after the other, with the
    // same bits.  1 / 40 pairs of 512 x 2048 6.6 -> 5.0 / 16.3 -> 15.1 us, of 256 x 1024 5.8 -> 4.3 / 8.0 -> 6.5
    for (int job = warp; job < jobs; job += WARPS) {
      const int r = job / nblk, c0 = (job - r * nblk) * 128 + lane * 4;
      const __nv_bfloat16* xr = a.x + static_cast<size_t>(xr0 + r) * a.ldx + k_begin + c0;
      float v[4], u[4];
      exl3_ld4(xr, a.x_align, v);
      exl3_ld4(xr + a.K, a.x_align, u);
      const uint2 sraw = *reinterpret_cast<const uint2*>(suh + c0);
      const __half2* sp = reinterpret_cast<const __half2*>(&sraw);
      const float2 s0 = __half22float2(sp[0]), s1 = __half22float2(sp[1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = exl3_gate(v[i], u[i], a.limit);
      exl3_fwht128_scaled(v, s0, s1, lane);
      // columns 4 q .. 4 q + 3 of a k-tile: t = 2 q and 2 q + 1 modulo 4, of its first or second half
      __half2* dst = reinterpret_cast<__half2*>(xh + r * ldh + (c0 & ~15) + ((lane & 1) << 3) + (lane & 2));
      dst[0] = __floats2half2_rn(v[0] * INV_SQRT_128, v[1] * INV_SQRT_128);
      dst[2] = __floats2half2_rn(v[2] * INV_SQRT_128, v[3] * INV_SQRT_128);
    }
  } else {
    for (int j0 = warp * 4; j0 < jobs; j0 += WARPS * 4) {
      const int job = min(j0 + (lane >> 3), jobs - 1);
      const int r = job / nblk, c0 = (job - r * nblk) * 128 + (lane & 7) * 16;
      const __nv_bfloat16* xr = a.x + static_cast<size_t>(xr0 + r) * a.ldx + k_begin + c0;
      float v[16];
      exl3_ld16(xr, a.x_align, v);
      if (a.act == 1) {
        float u[16];
        exl3_ld16(xr + a.K, a.x_align, u);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = exl3_gate(v[i], u[i], a.limit);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint2 sraw = reinterpret_cast<const uint2*>(suh + c0)[i];
        const __half2* sp = reinterpret_cast<const __half2*>(&sraw);
        const float2 s0 = __half22float2(sp[0]), s1 = __half22float2(sp[1]);
        v[4 * i] *= s0.x; v[4 * i + 1] *= s0.y; v[4 * i + 2] *= s1.x; v[4 * i + 3] *= s1.y;
      }
      fwht128_oct(v, lane);
      uint32_t o[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const __half2 lo = __floats2half2_rn(v[2 * i] * INV_SQRT_128, v[2 * i + 1] * INV_SQRT_128);
        const __half2 hi = __floats2half2_rn(v[2 * i + 8] * INV_SQRT_128, v[2 * i + 9] * INV_SQRT_128);
        o[2 * i] = *reinterpret_cast<const uint32_t*>(&lo); o[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&hi);
      }
      uint4* dst = reinterpret_cast<uint4*>(xh + r * ldh + c0);
      dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
      dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  }
  __syncthreads();

  // ---- main loop: the weights are the 16-row operand, the activation rows the 8 columns of the other one.  Lanes past the last
  // row read it again: their columns are never looked at.
  const __half* xrow[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) xrow[b] = xh + min(b * 8 + g, R - 1) * ldh + wk * 16 + 4 * t;
  const int ring = (lane + 31) & 31;                          // a tile is a ring of words
  float* pw = part + wk * R * 128 + wn * (16 * EXL3_TN) + g;
  float acc[NB][EXL3_TN][4];
  int ahead = nk - EXL3_DEPTH;                                // k-tiles whose loads are still to be issued
  // one k-tile from `b`, whose place the k-tile EXL3_DEPTH further takes
  auto step = [&](uint32_t (&bt)[EXL3_TN], bool first) {
    uint2 xb[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) { xb[b] = *reinterpret_cast<const uint2*>(xrow[b]); xrow[b] += WK * 16; }
#pragma unroll
    for (int j = 0; j < EXL3_TN; ++j) {
      const uint32_t prev = __shfl_sync(0xffffffffu, bt[j], ring);
      uint32_t w[4];
      exl3_decode8_b4<CB>(bt[j], prev, w);
      const uint32_t af[4] = {w[0], w[2], w[1], w[3]};       // columns c: k 2t, c + 8: k 2t, c: k 2t + 8, c + 8: k 2t + 8
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (first) mma_f16_16816_zero(acc[b][j], af, xb[b].x, xb[b].y);
        else mma_f16_16816(acc[b][j], af, xb[b].x, xb[b].y);
      }
    }
    if (ahead > 0) {
#pragma unroll
      for (int j = 0; j < EXL3_TN; ++j) bt[j] = __ldg(tw + j * 32);
    }
    --ahead;
    tw += tstep;
  };
#pragma unroll 1
  for (int c = 0; c < nch; ++c) {
    step(buf[0], true);
    step(buf[1], false);
#pragma unroll 1
    for (int i = 2; i < per; i += 2) { step(buf[0], false); step(buf[1], false); }
    // this warp's partials of the chunk
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = b * 8 + 2 * t + i;
        if (r < R) {
#pragma unroll
          for (int j = 0; j < EXL3_TN; ++j) { pw[r * 128 + j * 16] = acc[b][j][i]; pw[r * 128 + j * 16 + 8] = acc[b][j][2 + i]; }
        }
      }
    pw += WK * R * 128;
  }
  // This CTA's weight stream is done: let the next kernel's CTAs start (they issue their own weight loads while this
  // grid reduces and stores).  Triggering earlier only makes the two kernels' loads compete (measured: slower).
  pdl_trigger();
  // ---- a chunk's partials meet in the order of wk, their sums go to cluster rank 0 as plain remote stores; the other ranks arrive and
  // leave, rank 0 adds the chunks in their order: y = had128(sum) * svh.
  if (a.S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  __syncthreads();
  {
    float* dst = (a.S > 1 ? cluster.map_shared_rank(red, 0) : red) + static_cast<size_t>(slice) * nch * R * 128;
    const int n = R * 128;
    for (int i = threadIdx.x; i < nch * n; i += WARPS * 32) {
      const int c = nch == 1 ? 0 : i / n;
      const float* p = part + i + c * (WK - 1) * n;
      float s = p[0];
#pragma unroll
      for (int w = 1; w < WK; ++w) s += p[w * n];
      dst[i] = s;
    }
  }
  if (a.S > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (slice != 0) return;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  const __half* svh = a.svh + e * a.svh_stride + strip * 128;
  for (int r = warp; r < R; r += WARPS) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < a.S * nch; ++s) {
      const float4 p = *reinterpret_cast<const float4*>(red + (static_cast<size_t>(s) * R + r) * 128 + lane * 4);
      v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    fwht128_warp(v, lane);
    const uint2 sraw = *reinterpret_cast<const uint2*>(svh + lane * 4);
    const __half2* sp = reinterpret_cast<const __half2*>(&sraw);
    const float2 s0 = __half22float2(sp[0]), s1 = __half22float2(sp[1]);
    v[0] *= INV_SQRT_128 * s0.x; v[1] *= INV_SQRT_128 * s0.y; v[2] *= INV_SQRT_128 * s1.x; v[3] *= INV_SQRT_128 * s1.y;
    if (a.fuse_ar) {
      // fused all-reduce: this rank's partial strip goes straight into slot[rank] of every peer's arena
      const uint32_t ar_seq = comm_seq(a.ar.seq_ptr, a.ar.seq);
      if (a.ar.ll_off >= 0) {                     // decode rows: {value, sequence} words, the tail polls the data itself
        for (int p = 0; p < a.ar.c.world; ++p) {
          uint4* dst = ll_slot(a.ar.c.peers[p], a.ar.ll_off, ar_seq, a.ar.c.world, a.ar.c.rank, r, a.ar.N, strip * 128 + lane * 4);
          st_ll(dst, v[0], v[1], ar_seq);
          st_ll(dst + 1, v[2], v[3], ar_seq);
        }
        continue;
      }
      const size_t so = static_cast<size_t>(ar_seq & 1) * a.ar.c.world * a.ar.rows_cap * a.ar.N +
                        (static_cast<size_t>(a.ar.c.rank) * a.ar.rows_cap + r) * a.ar.N + strip * 128 + lane * 4;
      for (int p = 0; p < a.ar.c.world; ++p)
        st_f4(reinterpret_cast<float*>(a.ar.c.peers[p] + a.ar.slot_off) + so, make_float4(v[0], v[1], v[2], v[3]));
      continue;
    }
    const size_t o = static_cast<size_t>(item * R + r) * a.ldy + strip * 128 + lane * 4;
    if (a.out_f32) {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.y) + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      __nv_bfloat162 b0 = __floats2bfloat162_rn(v[0], v[1]), b1 = __floats2bfloat162_rn(v[2], v[3]);
      uint2 ov; ov.x = *reinterpret_cast<uint32_t*>(&b0); ov.y = *reinterpret_cast<uint32_t*>(&b1);
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.y) + o) = ov;
    }
  }
  if (a.fuse_ar && a.ar.ll_off < 0) exl3_fused_ar_arrive(a);
}

}  // namespace spark

using namespace spark;

// rows_per_item <= 16; K, N multiples of 128; S in 1..8 with (K/128) % S == 0 and K/S <= 2048.  Pairs (one row of an expert each) are
// summed in chunks of 256 (128 where K or the slices ask for it) whatever S is, so that S may follow their number; several rows of one matrix in S chunks.
// codebook: 0 mul1, 1 mcg.  ldx, ldy multiples of 4 elements.
extern "C" int spark_exl3_gemv(const void* x, int ldx, const void* trellis, const void* suh, const void* svh,
                               long long t_stride_words, long long suh_stride, long long svh_stride, void* y, int ldy,
                               int out_f32, const int* pair_expert, const int* pair_row, int items, int rows_per_item,
                               int K, int N, int S, int act, float limit, int codebook, cudaStream_t s, const void* ar_args,
                               int pairs_early) {
  if (items <= 0 || rows_per_item <= 0) return 0;
  if (rows_per_item > 16 || (K & 127) || (N & 127) || S < 1 || S > 8 || ((K >> 7) % S) || K / S > EXL3_MAX_KS) return -5;
  if ((ldx & 3) || (ldy & 3)) return -5;
  Exl3GemvArgs a;
  a.x = (const __nv_bfloat16*)x; a.ldx = ldx; a.trellis = (const uint32_t*)trellis;
  a.suh = (const __half*)suh; a.svh = (const __half*)svh;
  a.t_stride = t_stride_words; a.suh_stride = suh_stride; a.svh_stride = svh_stride;
  a.y = y; a.ldy = ldy; a.out_f32 = out_f32;
  a.pair_expert = pair_expert; a.pair_row = pair_row;
  a.R = rows_per_item; a.K = K; a.N = N; a.S = S; a.act = act; a.limit = limit;
  a.fuse_ar = 0;
  a.pairs_early = pairs_early;
  if (ar_args) {
    if (items != 1) return -5;
    a.fuse_ar = 1;
    a.ar = *static_cast<const ArRows*>(ar_args);
  }
  const uintptr_t xa = reinterpret_cast<uintptr_t>(x) | static_cast<uintptr_t>(ldx) * 2;
  a.x_align = (xa & 15) == 0 ? 16 : (xa & 7) == 0 ? 8 : 2;
  const bool two = rows_per_item > 8;
  const bool pairs = pair_expert && rows_per_item == 1;
  a.chunk = pairs ? (K / S % 256 == 0 ? 16 : 8) : K / S / 16;
  const int nch = K / 16 / S / a.chunk;
  const size_t smem_bytes = static_cast<size_t>(rows_per_item) * ((K / S + 16) * 2 + nch * (S + EXL3_WARPS * EXL3_TN / 8) * 128 * 4);
  void (*kern)(Exl3GemvArgs) = codebook == 0 ? (two ? exl3_gemv_kernel<0, 2> : exl3_gemv_kernel<0, 1>)
                                             : (two ? exl3_gemv_kernel<1, 2> : exl3_gemv_kernel<1, 1>);
  {
    static bool done[4] = {false, false, false, false};
    const int id = (codebook ? 2 : 0) + (two ? 1 : 0);
    if (!done[id]) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 * ((EXL3_MAX_KS + 16) * 2 + (8 + 8) * 128 * 4));
      done[id] = true;
    }
  }
  cudaError_t err = spark_launch_pdl(kern, dim3(N / 128, S, items), dim3(EXL3_WARPS * 32), smem_bytes, s, dim3(1, S, 1), a);
  return err == cudaSuccess ? 0 : -4;
}
