// EXL3 helpers for the GEMM (prefill) path:
//   exl3_reconstruct: trellis -> inner codebook weights as fp16 [N,K] (K-major B operand of the tcgen05 GEMM),
//                     all experts of a stacked tensor in one launch;
//   exl3_had_rows   : y = had128(x * scale) (input side, fp16 out) or had128(x) * scale (output side, bf16 out),
//                     with an optional per-row expert index selecting the scale vector.
// Format contract: engine-rs/shim/qwen_exl3.cuh:17-117,634-661; reference/qwen38/exl3.py:66-110.
#include "exl3_common.cuh"

namespace spark {

// inner -> fp16 Wt[N, K] (K contiguous).  One warp per tile.
template <int CB>
__global__ void exl3_reconstruct_kernel(const uint32_t* __restrict__ trellis, __half* __restrict__ Wt, int K, int N,
                                        int E) {
  const int KT = K >> 4, NT = N >> 4;
  const long long per = static_cast<long long>(KT) * NT;
  long long tile = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (tile >= per * E) return;
  const int lane = threadIdx.x & 31;
  const uint32_t cur = __ldg(trellis + tile * 32 + lane);
  const long long e = tile / per;
  tile -= e * per;
  Wt += e * static_cast<long long>(N) * K;
  const int kt = static_cast<int>(tile / NT), nt = static_cast<int>(tile % NT);
  const uint32_t prev = __shfl_sync(0xffffffffu, cur, (lane + 31) & 31);
  uint32_t w[4];
  exl3_decode8_b4<CB>(cur, prev, w);
  const int r0 = (lane & 3) * 2, c0 = lane >> 2;
  uint32_t* dst0 = reinterpret_cast<uint32_t*>(Wt + static_cast<size_t>(nt * 16 + c0) * K + kt * 16);
  uint32_t* dst1 = reinterpret_cast<uint32_t*>(Wt + static_cast<size_t>(nt * 16 + c0 + 8) * K + kt * 16);
  dst0[r0 >> 1] = w[0]; dst0[(r0 + 8) >> 1] = w[1];
  dst1[r0 >> 1] = w[2]; dst1[(r0 + 8) >> 1] = w[3];
}

// Any bit width (2..8 bits/weight: checkpoints mix 3 to 6 bits per tensor, heads often 6): a tile is 8 * bits words;
// the state of stream position t is the 16 bits that start at bit ((t + 1) * bits - 16) of the tail-biting ring, read
// MSB-first over little-endian 32-bit words.  Lane l still decodes positions 8l .. 8l+7, so the fragment assembly
// and the store pattern are those of the 4-bit kernel; only the window extraction reads its two words per state
// from memory (L1) instead of from the lane's own register.
template <int CB>
__global__ void exl3_reconstruct_bits_kernel(const uint32_t* __restrict__ trellis, __half* __restrict__ Wt, int K, int N,
                                             int E, int bits) {
  const int KT = K >> 4, NT = N >> 4;
  const long long per = static_cast<long long>(KT) * NT;
  long long tile = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (tile >= per * E) return;
  const int lane = threadIdx.x & 31;
  const int n_words = 8 * bits, n_bits = 256 * bits;
  const uint32_t* tw = trellis + tile * n_words;
  uint32_t st[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    int first = (8 * lane + j + 1) * bits - 16;
    if (first < 0) first += n_bits;
    const int wi = first >> 5, off = first & 31;
    const uint32_t hi = __ldg(tw + wi), lo = __ldg(tw + (wi + 1 == n_words ? 0 : wi + 1));
    st[j] = __funnelshift_l(lo, hi, off) >> 16;
  }
  const long long e = tile / per;
  tile -= e * per;
  Wt += e * static_cast<long long>(N) * K;
  const int kt = static_cast<int>(tile / NT), nt = static_cast<int>(tile % NT);
  uint32_t w[4];
  w[0] = exl3_pair<CB>(st[0], st[1]); w[1] = exl3_pair<CB>(st[2], st[3]);
  w[2] = exl3_pair<CB>(st[4], st[5]); w[3] = exl3_pair<CB>(st[6], st[7]);
  const int r0 = (lane & 3) * 2, c0 = lane >> 2;
  uint32_t* dst0 = reinterpret_cast<uint32_t*>(Wt + static_cast<size_t>(nt * 16 + c0) * K + kt * 16);
  uint32_t* dst1 = reinterpret_cast<uint32_t*>(Wt + static_cast<size_t>(nt * 16 + c0 + 8) * K + kt * 16);
  dst0[r0 >> 1] = w[0]; dst0[(r0 + 8) >> 1] = w[1];
  dst1[r0 >> 1] = w[2]; dst1[(r0 + 8) >> 1] = w[3];
}

// y[r, :] = had128(x[r, :] * scale[:]) (pre) or had128(x[r, :]) * scale[:] (post); 128-blocks along the row.
// Eight lanes per 128-block, four blocks per warp: a lane moves 16 consecutive elements as 16-byte vectors.  With one block per
// warp (four elements a lane, five shuffle stages, an index division per 128 elements) the pass was bound by issue and shuffles:
// 4096 rows of 12288 and of 2048 columns out (fp32 -> bf16) 96 -> 75 us, 4096 rows in (bf16 -> fp16) 21 -> 13 us.
__device__ __forceinline__ void ld16(const float* p, float (&v)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 t = reinterpret_cast<const float4*>(p)[i];
    v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
  }
}
template <typename T2, typename T> __device__ __forceinline__ float2 up2(uint32_t w);
template <> __device__ __forceinline__ float2 up2<__nv_bfloat162, __nv_bfloat16>(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
template <> __device__ __forceinline__ float2 up2<__half2, __half>(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
// 16 elements of 16 bits; rows are aligned to 8 bytes (`wide`: to 16)
template <typename T2, typename T>
__device__ __forceinline__ void ld16h(const T* p, bool wide, float (&v)[16]) {
  uint32_t w[8];
  if (wide) {
    const uint4 a = reinterpret_cast<const uint4*>(p)[0], b = reinterpret_cast<const uint4*>(p)[1];
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) { const uint2 a = reinterpret_cast<const uint2*>(p)[i]; w[2 * i] = a.x; w[2 * i + 1] = a.y; }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) { const float2 f = up2<T2, T>(w[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void ld16(const __nv_bfloat16* p, bool wide, float (&v)[16]) { ld16h<__nv_bfloat162>(p, wide, v); }
__device__ __forceinline__ void ld16(const __half* p, bool wide, float (&v)[16]) { ld16h<__half2>(p, wide, v); }
__device__ __forceinline__ void ld16(const float* p, bool, float (&v)[16]) { ld16(p, v); }
__device__ __forceinline__ uint32_t pk(const __half*, float a, float b) { const __half2 h = __floats2half2_rn(a, b); return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ uint32_t pk(const __nv_bfloat16*, float a, float b) { const __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const uint32_t*>(&h); }
template <typename T> __device__ __forceinline__ void st16(T* p, bool wide, const float (&v)[16]) {
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = pk(p, v[2 * i], v[2 * i + 1]);
  if (wide) {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) reinterpret_cast<uint2*>(p)[i] = make_uint2(w[2 * i], w[2 * i + 1]);
  }
}

// thread id -> (row, 128-block); lanes past the end take part in the shuffles with the last block's values
struct HadAt { int r, c0; bool live; };
__device__ __forceinline__ HadAt had_at(int R, int nblk) {
  const long long b = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) >> 3, total = static_cast<long long>(R) * nblk;
  HadAt h;
  h.live = b < total;
  const long long bb = h.live ? b : total - 1;
  // R * nblk < 2^31 in all that fits a device: 32-bit division
  h.r = static_cast<int>(static_cast<uint32_t>(bb) / static_cast<uint32_t>(nblk));
  h.c0 = static_cast<int>(bb - static_cast<long long>(h.r) * nblk) * 128 + (threadIdx.x & 7) * 16;
  return h;
}

template <typename TI, typename TOUT>
__global__ void __launch_bounds__(256)
exl3_had_rows_kernel(const TI* __restrict__ x, int ldx, const __half* __restrict__ scale, TOUT* __restrict__ y, int ldy,
                     int post, const int* __restrict__ row_expert, long long expert_stride, int R, int nblk, int wide) {
  const HadAt at = had_at(R, nblk);
  float v[16], sc[16];
  ld16(x + static_cast<size_t>(at.r) * ldx + at.c0, wide & 1, v);
  ld16(scale + (row_expert ? row_expert[at.r] * expert_stride : 0) + at.c0, wide & 4, sc);
  if (!post) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= sc[i];
  }
  fwht128_oct(v, threadIdx.x & 31);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] *= INV_SQRT_128;
    if (post) v[i] *= sc[i];
  }
  if (at.live) st16(y + static_cast<size_t>(at.r) * ldy + at.c0, wide & 2, v);
}

// Rows of a prompt batch in expert order: y[i] = had128(x[perm[i] / top_k] * suh[expert of pair perm[i]]), fp16.  The gather, the
// row-to-expert lookup and the transform are one pass (before: a bf16 gather, four index kernels and exl3_had_rows).
// Bound by writing y: 81920 rows of 2048 took 278 us with one block per warp and take 139 (2.4 TB/s written).
__global__ void __launch_bounds__(256)
exl3_had_gather_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const int* __restrict__ perm, const int* __restrict__ ids, int top_k,
                       const __half* __restrict__ suh, long long suh_stride, __half* __restrict__ y, int ldy, int R, int nblk, int wide) {
  const HadAt at = had_at(R, nblk);
  const int pair = perm[at.r], e = max(ids[pair], 0);        // filler rows past this rank's pairs may name an expert elsewhere
  float v[16], sc[16];
  ld16(x + static_cast<size_t>(pair / top_k) * ldx + at.c0, wide & 1, v);
  ld16(suh + e * suh_stride + at.c0, wide & 4, sc);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] *= sc[i];
  fwht128_oct(v, threadIdx.x & 31);
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] *= INV_SQRT_128;
  if (at.live) st16(y + static_cast<size_t>(at.r) * ldy + at.c0, wide & 2, v);
}

// bit 0: rows of x start on 16 bytes, bit 1: rows of y, bit 2: scale vectors
static int had_wide(const void* x, size_t x_row_bytes, const void* y, size_t y_row_bytes, const void* sc, long long sc_row_bytes) {
  auto ok = [](const void* p, size_t row) { return ((reinterpret_cast<uintptr_t>(p) | row) & 15) == 0; };
  return (ok(x, x_row_bytes) ? 1 : 0) | (ok(y, y_row_bytes) ? 2 : 0) | (ok(sc, static_cast<size_t>(sc_row_bytes)) ? 4 : 0);
}

}  // namespace spark

using namespace spark;

// E stacked tensors (experts) in one launch: trellis [E][K/16][N/16][32 words] -> Wt [E][N][K].
extern "C" int spark_exl3_reconstruct(const void* trellis, void* Wt, int K, int N, int codebook, cudaStream_t s, int E) {
  const long long tiles = (long long)(K >> 4) * (N >> 4) * E;
  const unsigned blocks = (unsigned)((tiles * 32 + 255) / 256);
  if (codebook == 0) exl3_reconstruct_kernel<0><<<blocks, 256, 0, s>>>((const uint32_t*)trellis, (__half*)Wt, K, N, E);
  else exl3_reconstruct_kernel<1><<<blocks, 256, 0, s>>>((const uint32_t*)trellis, (__half*)Wt, K, N, E);
  return spark_launch_rc(__func__);
}

// The same for any bit width 2..8 (trellis [E][K/16][N/16][8 * bits words]).
extern "C" int spark_exl3_reconstruct_bits(const void* trellis, void* Wt, int K, int N, int codebook, cudaStream_t s, int E,
                                           int bits) {
  if (bits < 2 || bits > 8 || (K & 15) || (N & 15) || E < 1) return -5;
  const long long tiles = (long long)(K >> 4) * (N >> 4) * E;
  const unsigned blocks = (unsigned)((tiles * 32 + 255) / 256);
  if (codebook == 0) exl3_reconstruct_bits_kernel<0><<<blocks, 256, 0, s>>>((const uint32_t*)trellis, (__half*)Wt, K, N, E, bits);
  else exl3_reconstruct_bits_kernel<1><<<blocks, 256, 0, s>>>((const uint32_t*)trellis, (__half*)Wt, K, N, E, bits);
  return spark_launch_rc(__func__);
}

// pre (post = 0): x bf16 -> y fp16 = had128(x * scale);  post = 1: x fp32 -> y bf16 = had128(x) * scale.
// row_expert (optional): per-row expert id selecting scale + row_expert[r] * expert_stride.
extern "C" int spark_exl3_had_rows(const void* x, int ldx, const void* scale, void* y, int ldy, int R, int C, int post,
                                   const int* row_expert, cudaStream_t s, long long expert_stride) {
  if (R <= 0) return 0;
  if (C & 127) return -5;
  if ((ldx & 3) || (ldy & 3)) return -5;               // 8- / 16-byte vector accesses along the rows
  const int nblk = C / 128;
  const long long total = static_cast<long long>(R) * nblk;
  if (total > 0x7fffffffLL) return -5;
  const unsigned grid = static_cast<unsigned>((total * 8 + 255) / 256);
  const int wide = had_wide(x, static_cast<size_t>(ldx) * (post ? 4 : 2), y, static_cast<size_t>(ldy) * 2, scale, row_expert ? expert_stride * 2 : 0);
  if (!post) exl3_had_rows_kernel<__nv_bfloat16, __half><<<grid, 256, 0, s>>>((const __nv_bfloat16*)x, ldx, (const __half*)scale, (__half*)y, ldy, 0, row_expert, expert_stride, R, nblk, wide);
  else exl3_had_rows_kernel<float, __nv_bfloat16><<<grid, 256, 0, s>>>((const float*)x, ldx, (const __half*)scale, (__nv_bfloat16*)y, ldy, 1, row_expert, expert_stride, R, nblk, wide);
  return spark_launch_rc(__func__);
}

// x bf16 [rows, C] -> y fp16 [P, C]: row i is pair perm[i] of the routing table `ids` [rows, top_k], scaled by its expert's vector.
extern "C" int spark_exl3_had_gather(const void* x, int ldx, const int* perm, const int* ids, int top_k, const void* suh,
                                     long long suh_stride, void* y, int ldy, int P, int C, cudaStream_t s) {
  if (P <= 0) return 0;
  if ((C & 127) || (ldx & 3) || (ldy & 3) || top_k < 1) return -5;
  const int nblk = C / 128;
  const long long total = static_cast<long long>(P) * nblk;
  if (total > 0x7fffffffLL) return -5;
  exl3_had_gather_kernel<<<static_cast<unsigned>((total * 8 + 255) / 256), 256, 0, s>>>(
      (const __nv_bfloat16*)x, ldx, perm, ids, top_k, (const __half*)suh, suh_stride, (__half*)y, ldy, P, nblk,
      had_wide(x, static_cast<size_t>(ldx) * 2, y, static_cast<size_t>(ldy) * 2, suh, suh_stride * 2));
  return spark_launch_rc(__func__);
}
