// Gated-DeltaNet prefill in chunked (WY) form: 64-token chunks, all matrix work on tensor cores (tf32 MMA, fp32
// accumulate), the state carried through a short sequential pass.
//
// Per value head, with d_t = exp(g_t), D_t = prod_{j<=t} d_j inside a chunk, S0 the state entering the chunk
// (S is [Dv, Dk]; row i is what one thread of the sequential kernel owns):
//     u_t = beta_t (v_t - d_t S_{t-1} k_t),   S_t = d_t S_{t-1} + u_t k_t^T,   o_t = S_t q_t
// unrolls to
//     (I + A) U = diag(beta) V - diag(beta D) K S0^T,     A_tj = beta_t (D_t/D_j) (k_t.k_j)  (j < t)
//     O = diag(D) Q S0^T + P U,                           P_tj = (D_t/D_j) (q_t.k_j)         (j <= t)
//     S_C = D_C S0 + U^T diag(D_C / D) K
// so with T = (I + A)^-1 everything that does not involve S0 is computed for all chunks in parallel:
//   kernel 1 (chunk, head):  conv(k=4)+SiLU, L2 norms, gates;  K K^T, Q K^T -> A, P;  T by blocks;
//                            W = T diag(beta D) K,  Ut = T diag(beta) V,  Qt = diag(D) Q,  Kt = diag(D_C/D) K
//   kernel 2 (v-slice, head, segment), sequential over the chunks of one sequence, S kept in registers:
//                            U = Ut - W S0^T;  O = Qt S0^T + P U;  S <- D_C S + U^T Kt
//                            (the Dv rows of S are independent, so a head is split over 2 CTAs of 64 rows)
//   kernel 3 (chunk, head):  RMSNorm(o) * w * sigmoid(z) -> bf16
// All decay ratios are exp() of non-positive numbers: nothing can overflow.  Operands are rounded to tf32
// (10-bit mantissa) once, when they are written; sums are fp32.  Decode and verify rows keep using the
// sequential kernel (bitwise chained == one-pass there); this path serves committed segments of >= 64 rows.
// Reference: engine-rs/shim/qwen_gdn.cu rows_kernel / rows4_kernel (sequential over rows, 4 rows per step).
#include "../common/ptx.cuh"

namespace spark {

constexpr int GC = 64;            // chunk length
constexpr int GD = 128;           // head dim (k and v)
constexpr int LD128 = 136;        // smem row stride of 128-wide arrays (8 mod 32: conflict-free fragment loads)
constexpr int LD64 = 72;
constexpr int GVS = 64;           // value rows of S per CTA in the state pass
// Workspace per (chunk, head), floats: the shared-memory images of the state pass's operands, so that plain bulk copies bring them in.
// K-major rows of 32 floats (128 bytes, 128-byte swizzle): [Qt; W] as four tiles of 128 rows, Kt^T as two of 128, P as two of 64;
// Ut per slice of GVS value columns as [column / 4][row][4].
constexpr int WS_QW = 0, WS_UT = 2 * GC * GD, WS_KT = 3 * GC * GD, WS_P = 4 * GC * GD,
              WS_DC = 4 * GC * GD + GC * GC, WS_STRIDE = 4 * GC * GD + GC * GC + 64;
// float of row r, column k in tiles of `rows` rows
__device__ __forceinline__ int ws_at(int rows, int r, int k) { return (k >> 5) * rows * 32 + r * 32 + ((((k >> 2) ^ r) & 7) << 2) + (k & 3); }
__device__ __forceinline__ int ws_ut(int r, int v) { return (v >> 2) * GC * 4 + r * 4 + (v & 3); }

__device__ __forceinline__ float tf32r(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], float a0, float a1, float a2, float a3, float b0, float b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}
__device__ __forceinline__ float silu(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------- kernel 1
// grid (chunks, Hv); 256 threads.  Two CTAs share an SM (107 KB each): A and T take the place of Q once its products are through.
// What bounds it: the chain of its phases, of which the convolution with its SiLU is the longest, hidden only by the second CTA;
// 302 MB are written at 1.2 TB/s.  64 chunks of 32 heads: 544 -> 245 us (one CTA per SM, one channel per lane with its rows loaded
// one after the other: 20 us for the convolution of a CTA).  47 us of it are the IEEE divisions of the SiLU: an approximate one
// gives 0 below -87.3, and values that small are numbers of the state.
constexpr int SM_AT = GC * LD128, SM_AT_EXTRA = 2 * GC * LD64 - SM_AT;      // floats of A and T past the end of Q
constexpr int PREP_SMEM = (3 * GC * LD128 + SM_AT_EXTRA + 3 * GC) * 4;

// Rows 8 warp - 3 .. 8 warp + 7 of four consecutive channels as they are in memory (zero outside the segment)
__device__ __forceinline__ void gdn_load_rows(const __nv_bfloat16* __restrict__ proj, int ldp, int r0, int first, int n, int ch, uint2 (&x)[11]) {
#pragma unroll
  for (int j = 0; j < 11; ++j) {
    const int p = first + j;
    x[j] = p >= 0 && p < n ? __ldg(reinterpret_cast<const uint2*>(proj + static_cast<size_t>(r0 + p) * ldp + ch)) : make_uint2(0u, 0u);
  }
}
// The same in fp32, rows before the segment's start from the slot's history
__device__ __forceinline__ void gdn_widen_rows(const uint2 (&u)[11], const float* __restrict__ hist, size_t hist_ld, int first, float4 (&x)[11]) {
#pragma unroll
  for (int j = 0; j < 11; ++j) {
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j].x)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j].y));
    x[j] = make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  if (first < 0) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (first + j < 0) {                                   // (three rows of a segment: no vectors, the caller's tail may start anywhere)
        const float* p = hist + static_cast<size_t>(first + j + 3) * hist_ld;
        x[j] = make_float4(p[0], p[1], p[2], p[3]);
      }
  }
}
// conv(k = 4) of row i (x[i .. i + 3]); w[c]: taps of channel c
__device__ __forceinline__ float4 gdn_conv(const float4 (&x)[11], int i, const float4 (&w)[4]) {
  return make_float4(x[i].x * w[0].x + x[i + 1].x * w[0].y + x[i + 2].x * w[0].z + x[i + 3].x * w[0].w,
                     x[i].y * w[1].x + x[i + 1].y * w[1].y + x[i + 2].y * w[1].z + x[i + 3].y * w[1].w,
                     x[i].z * w[2].x + x[i + 1].z * w[2].y + x[i + 2].z * w[2].z + x[i + 3].z * w[2].w,
                     x[i].w * w[3].x + x[i + 1].w * w[3].y + x[i + 2].w * w[3].z + x[i + 3].w * w[3].w);
}
__device__ __forceinline__ float4 scale_tf32(float4 v, float f) { return make_float4(tf32r(v.x * f), tf32r(v.y * f), tf32r(v.z * f), tf32r(v.w * f)); }

// w_wide: the convolution's taps start on 16 bytes
__global__ void __launch_bounds__(256, 2)
gdn_chunk_prep_kernel(const __nv_bfloat16* __restrict__ proj, int ldp, const __nv_bfloat16* __restrict__ ab, int ldab,
                      const float* __restrict__ conv_w, const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                      const float* __restrict__ tail, const int* __restrict__ seg, const int* __restrict__ chunks,
                      float* __restrict__ ws, int Hk, int Hv, float eps, int w_wide) {
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                          // [64][136]
  float* As = sm;                          // [64][72]   A, over Q
  float* Ts = As + GC * LD64;              // [64][72]   T
  float* Ks = sm + SM_AT + SM_AT_EXTRA;
  float* Vs = Ks + GC * LD128;
  float* beta_s = Vs + GC * LD128;         // [64]
  float* G_s = beta_s + GC;                // [64] cumulative log decay
  float* D_s = G_s + GC;                   // [64] exp of it
  const int ci = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sg = chunks[2 * ci], c = chunks[2 * ci + 1];
  const int slot = seg[sg * 4], r0 = seg[sg * 4 + 1], n = seg[sg * 4 + 2];
  const int t0 = c * GC, nv = min(GC, n - t0);
  const int hk = h / (Hv / Hk);
  float* wsb = ws + (static_cast<size_t>(ci) * Hv + h) * WS_STRIDE;

  // ---- inputs of this warp's eight rows are asked for first: a lane owns four channels of q, of k and of v
  const float* hist = tail + (static_cast<size_t>(slot) * 3 * Hv + h) * 3 * GD + lane * 4;
  const size_t hist_ld = static_cast<size_t>(Hv) * 3 * GD;
  const int first = t0 + warp * 8 - 3;
  const int chq = hk * GD + lane * 4, chk = Hk * GD + chq, chv = 2 * Hk * GD + h * GD + lane * 4;
  uint2 raw[3][11];
  gdn_load_rows(proj, ldp, r0, first, n, chq, raw[0]);
  gdn_load_rows(proj, ldp, r0, first, n, chk, raw[1]);
  gdn_load_rows(proj, ldp, r0, first, n, chv, raw[2]);
  // ---- gates and the prefix sum of the log decays: warp 0, two rows per lane
  if (warp == 0) {
    float beta[2], lg[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = lane * 2 + i;
      beta[i] = 0.f; lg[i] = 0.f;
      if (r < nv) {
        const float bl = __bfloat162float(ab[static_cast<size_t>(r0 + t0 + r) * ldab + h]);
        const float al = __bfloat162float(ab[static_cast<size_t>(r0 + t0 + r) * ldab + Hv + h]);
        beta[i] = 1.f / (1.f + __expf(-bl));
        const float xa = al + dt_bias[h];
        const float sp = xa > 20.f ? xa : log1pf(__expf(xa));
        lg[i] = -__expf(A_log[h]) * sp;
      }
    }
    float inc = lg[0] + lg[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, inc, o); if (lane >= o) inc += u; }
    float before = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) before = 0.f;
    const float G0 = before + lg[0], G1 = G0 + lg[1];
    *reinterpret_cast<float2*>(beta_s + lane * 2) = make_float2(beta[0], beta[1]);
    *reinterpret_cast<float2*>(G_s + lane * 2) = make_float2(G0, G1);
    *reinterpret_cast<float2*>(D_s + lane * 2) = make_float2(__expf(G0), __expf(G1));
  }
  __syncthreads();
  // ---- conv -> shared memory, then SiLU + L2 norms (TF32) in place, Qt = diag(D) Q and Kt = diag(D_C / D) K -> workspace.  Every lane
  // goes over what it wrote itself, as a short loop: 96 IEEE divisions unrolled behind the convolution spilled (64 chunks of 32 heads: 257 us)
  {
    const float Gl = G_s[GC - 1];
    float4 w[4];
#pragma unroll
    for (int part = 0; part < 3; ++part) {                  // q, k, v
      const int ch = part == 0 ? chq : part == 1 ? chk : chv;
      float4 x[11];
      gdn_widen_rows(raw[part], hist + part * GD, hist_ld, first, x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float* p = conv_w + static_cast<size_t>(ch + i) * 4;
        w[i] = w_wide ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(p[0], p[1], p[2], p[3]);
      }
      float* dst = (part == 0 ? Qs : part == 1 ? Ks : Vs) + warp * 8 * LD128 + lane * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(dst + i * LD128) = gdn_conv(x, i, w);
    }
#pragma unroll 4
    for (int i = 0; i < 24; ++i) {
      const int part = i >> 3, r = warp * 8 + (i & 7);
      float4* at = reinterpret_cast<float4*>((part == 0 ? Qs : part == 1 ? Ks : Vs) + r * LD128 + lane * 4);
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);           // rows past the end stay zero, whatever eps is
      if (r < nv) {
        y = *at;
        y = make_float4(silu(y.x), silu(y.y), silu(y.z), silu(y.w));
        float f = 1.f;
        if (part < 2) {
          const float ss = warp_sum(fmaf(y.w, y.w, fmaf(y.z, y.z, fmaf(y.y, y.y, y.x * y.x))));
          f = rsqrtf(ss + eps) * (part == 0 ? rsqrtf(static_cast<float>(GD)) : 1.f);
        }
        y = scale_tf32(y, f);
      }
      *at = y;
      if (part == 0) *reinterpret_cast<float4*>(wsb + WS_QW + ws_at(2 * GC, r, lane * 4)) = scale_tf32(y, D_s[r]);
    }
    if (tid == 0) wsb[WS_DC] = __expf(Gl);
  }
  __syncthreads();
  {
    // Kt^T: a thread moves four rows of a channel; two lanes fill a 32-byte sector
    const float Gl = G_s[GC - 1];
#pragma unroll 2
    for (int i = tid; i < GD * (GC / 4); i += 256) {
      const int k = (i >> 1) & (GD - 1), r = ((i >> 8) * 2 + (i & 1)) * 4;
      const float* kp = Ks + r * LD128 + k;
      *reinterpret_cast<float4*>(wsb + WS_KT + ws_at(GD, k, r)) =
          make_float4(tf32r(kp[0] * __expf(Gl - G_s[r])), tf32r(kp[LD128] * __expf(Gl - G_s[r + 1])),
                      tf32r(kp[2 * LD128] * __expf(Gl - G_s[r + 2])), tf32r(kp[3 * LD128] * __expf(Gl - G_s[r + 3])));
    }
  }

  const int g = lane >> 2, t = lane & 3;
  // ---- K K^T and Q K^T (lower triangle only): warp -> m-tile (warp&3), n-tiles 4*(warp>>2) .. +4
  {
    const int mt = warp & 3, nt0 = (warp >> 2) * 4;
    float ckk[4][4], cqk[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) { ckk[a][b] = 0.f; cqk[a][b] = 0.f; }
    if (nt0 * 8 <= mt * 16 + 15) {
      const float* ka = Ks + (mt * 16 + g) * LD128 + t;
      const float* qa = Qs + (mt * 16 + g) * LD128 + t;
#pragma unroll 4
      for (int ks = 0; ks < GD / 8; ++ks) {
        const float k0 = ka[ks * 8], k1 = ka[8 * LD128 + ks * 8], k2 = ka[ks * 8 + 4], k3 = ka[8 * LD128 + ks * 8 + 4];
        const float q0 = qa[ks * 8], q1 = qa[8 * LD128 + ks * 8], q2 = qa[ks * 8 + 4], q3 = qa[8 * LD128 + ks * 8 + 4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const int nt = nt0 + a;
          if (nt * 8 > mt * 16 + 15) continue;                      // strictly above the diagonal
          const float* kb = Ks + (nt * 8 + g) * LD128 + ks * 8 + t;
          const float b0 = kb[0], b1 = kb[4];
          mma_tf32(ckk[a], k0, k1, k2, k3, b0, b1);
          mma_tf32(cqk[a], q0, q1, q2, q3, b0, b1);
        }
      }
    }
    __syncthreads();                                                // Q is read: A takes its place
    float* Pg = wsb + WS_P;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int col = (nt0 + a) * 8 + 2 * t;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = mt * 16 + g + e * 8;
        float av[2], pv[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          av[u] = 0.f; pv[u] = 0.f;
          if (col + u <= row) {
            const float dec = __expf(G_s[row] - G_s[col + u]);
            pv[u] = tf32r(dec * cqk[a][e * 2 + u]);
            if (col + u < row) av[u] = beta_s[row] * dec * ckk[a][e * 2 + u];
          }
        }
        *reinterpret_cast<float2*>(As + row * LD64 + col) = make_float2(av[0], av[1]);
        *reinterpret_cast<float2*>(Pg + ws_at(GC, row, col)) = make_float2(pv[0], pv[1]);
      }
    }
  }
  __syncthreads();
  // ---- T = (I + A)^-1 by blocks, all in fp32: the four 16 x 16 blocks on the diagonal by forward substitution (a thread per
  // column), then twice T21 = -T22 (A21 T11).  A's unused upper blocks hold A21 T11.  (One thread per column of the whole matrix
  // was a chain of 2016 steps on two warps.)
  if (tid < GC) {
    const int b0 = tid & ~15, cc = tid & 15;
    float tc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float4* row = reinterpret_cast<const float4*>(As + (b0 + i) * LD64 + b0);
      float s0 = i == cc ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
      for (int j = 0; j < i; j += 4) {
        const float4 av = row[j >> 2];
        s0 = fmaf(-av.x, tc[j], s0);
        if (j + 1 < i) s1 = fmaf(-av.y, tc[j + 1 < 16 ? j + 1 : 15], s1);
        if (j + 2 < i) s0 = fmaf(-av.z, tc[j + 2 < 16 ? j + 2 : 15], s0);
        if (j + 3 < i) s1 = fmaf(-av.w, tc[j + 3 < 16 ? j + 3 : 15], s1);
      }
      tc[i] = s0 + s1;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) Ts[(b0 + i) * LD64 + tid] = tc[i];
  }
  __syncthreads();
  {
    const int o = (tid >> 7) * 32, i = (tid >> 3) & 15, j = (tid & 7) * 2;      // 32-blocks at (o, o): rows 16 + i, columns j, j + 1
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float av = As[(o + 16 + i) * LD64 + o + k];
      const float2 tv = *reinterpret_cast<const float2*>(Ts + (o + k) * LD64 + o + j);
      s0 = fmaf(av, tv.x, s0); s1 = fmaf(av, tv.y, s1);
    }
    *reinterpret_cast<float2*>(As + (o + i) * LD64 + o + 16 + j) = make_float2(s0, s1);
    __syncthreads();
    s0 = 0.f; s1 = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const float tv = Ts[(o + 16 + i) * LD64 + o + 16 + k];
      const float2 xv = *reinterpret_cast<const float2*>(As + (o + k) * LD64 + o + 16 + j);
      s0 = fmaf(-tv, xv.x, s0); s1 = fmaf(-tv, xv.y, s1);
    }
    *reinterpret_cast<float2*>(Ts + (o + 16 + i) * LD64 + o + j) = make_float2(s0, s1);
    *reinterpret_cast<float2*>(Ts + (o + i) * LD64 + o + 16 + j) = make_float2(0.f, 0.f);
  }
  __syncthreads();
  {
    const int i = tid >> 3, j = (tid & 7) * 4;                                  // rows 32 + i, columns j .. j + 3
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float av = As[(32 + i) * LD64 + k];
      const float4 tv = *reinterpret_cast<const float4*>(Ts + k * LD64 + j);
      s.x = fmaf(av, tv.x, s.x); s.y = fmaf(av, tv.y, s.y); s.z = fmaf(av, tv.z, s.z); s.w = fmaf(av, tv.w, s.w);
    }
    *reinterpret_cast<float4*>(As + i * LD64 + 32 + j) = s;
    __syncthreads();
    s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float tv = Ts[(32 + i) * LD64 + 32 + k];
      const float4 xv = *reinterpret_cast<const float4*>(As + k * LD64 + 32 + j);
      s.x = fmaf(-tv, xv.x, s.x); s.y = fmaf(-tv, xv.y, s.y); s.z = fmaf(-tv, xv.z, s.z); s.w = fmaf(-tv, xv.w, s.w);
    }
    *reinterpret_cast<float4*>(Ts + (32 + i) * LD64 + j) = s;
  }
  __syncthreads();
  // ---- W = T diag(beta D) K, Ut = T diag(beta) V: warp -> m-tile (warp&3), n-tiles 8*(warp>>2) .. +8; k-steps up to the diagonal
  // (the diagonals are multiplied into the fragments of T)
  {
    const int mt = warp & 3, nt0 = (warp >> 2) * 8;
    const float* aa = Ts + (mt * 16 + g) * LD64 + t;
#pragma unroll 1
    for (int which = 0; which < 2; ++which) {
      const float* Bm = which == 0 ? Ks : Vs;
      float acc[8][4];
#pragma unroll
      for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
      for (int ks = 0; ks < 2 * (mt + 1); ++ks) {
        const float e0 = which == 0 ? D_s[ks * 8 + t] : 1.f, e1 = which == 0 ? D_s[ks * 8 + t + 4] : 1.f;
        const float f0 = beta_s[ks * 8 + t], f1 = beta_s[ks * 8 + t + 4];
        const float a0 = tf32r(aa[ks * 8] * f0 * e0), a1 = tf32r(aa[8 * LD64 + ks * 8] * f0 * e0);
        const float a2 = tf32r(aa[ks * 8 + 4] * f1 * e1), a3 = tf32r(aa[8 * LD64 + ks * 8 + 4] * f1 * e1);
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const float* bb = Bm + (ks * 8 + t) * LD128 + (nt0 + a) * 8 + g;
          mma_tf32(acc[a], a0, a1, a2, a3, bb[0], bb[4 * LD128]);
        }
      }
      float* Og = wsb + (which == 0 ? WS_QW : WS_UT);
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const int col = (nt0 + a) * 8 + 2 * t, row = mt * 16 + g;
        float2 lo = make_float2(acc[a][0], acc[a][1]), hi = make_float2(acc[a][2], acc[a][3]);
        if (which == 0) { lo.x = tf32r(lo.x); lo.y = tf32r(lo.y); hi.x = tf32r(hi.x); hi.y = tf32r(hi.y); }
        *reinterpret_cast<float2*>(Og + (which == 0 ? ws_at(2 * GC, GC + row, col) : ws_ut(row, col))) = lo;
        *reinterpret_cast<float2*>(Og + (which == 0 ? ws_at(2 * GC, GC + row + 8, col) : ws_ut(row + 8, col))) = hi;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------- kernel 2
// grid (2, Hv, nseg); sequential over the chunks of one segment, 64 value rows of S per CTA.  Products on tcgen05 (kind::tf32), the state
// in registers:
//   [O; X] = [Qt; W] S^T          M = 128 rows, N = 64 values, K = 128          D1 (two buffers)
//   U      = Ut - X                by the warps that own the lanes of X
//   D3     = Kt^T U                M = 128 keys, N = 64, K = 64                  then S^T <- D_C S^T + D3 in registers
//   O     += P U                   the M = 128 operand's rows past P's 64 are whatever follows it: their lanes are off, as are those of
//                                  the blocks of 16 rows in front of a step's rows of U (P is 0 there, and 0 times a NaN is none)
// Warp 0 brings the operands in, tiles of 16 KB through a ring of 11 (eight per chunk); warp 1 issues; eight warps (two per lane quarter,
// 32 value columns each) keep S, write it and U as K-major operands and store O.
// What bounds it: the chain state -> product -> U -> product of a chunk, and the 128 KB per chunk that a CTA pulls from L2.
// 64 chunks of 32 heads: 188 us (of 5473 cycles a chunk 3220 are the products, 860 writing S as an operand, 910 U); 293 with warp-level
// TF32 products and the operands copied between them (four CTAs of 32 values a head).  Several segments, whole layer before and now: 4 x 1024
// rows 1027 -> 689, 16 x 256 1011 -> 704, 64 x 64 1082 -> 787.
constexpr int ST_SLOTS = 11, ST_SLOT = 16384, ST_THREADS = 10 * 32;
constexpr int ST_B1 = GVS * GD * 4, ST_B2 = GVS * GC * 4;
constexpr int ST_SMEM = ST_SLOTS * ST_SLOT + ST_B1 + ST_B2 + 256 + 1024;
static_assert(ST_SMEM <= 232448, "shared memory of the state pass");

__global__ void __launch_bounds__(ST_THREADS, 1)
gdn_chunk_state_kernel(const float* __restrict__ ws, const int* __restrict__ seg, const int* __restrict__ seg_chunk0,
                       const __nv_bfloat16* __restrict__ proj, int ldp, float* __restrict__ S, float* __restrict__ tail,
                       float* __restrict__ o_raw, int ldo, int Hk, int Hv, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  const int vs = blockIdx.x, h = blockIdx.y, sg = blockIdx.z;
  const int ci0 = seg_chunk0[sg];
  if (ci0 < 0) return;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* B1 = smem + ST_SLOTS * ST_SLOT;                   // S^T as [64 values][128 keys]: four tiles of 64 rows
  uint8_t* B2 = B1 + ST_B1;                                  // U^T as [64 values][64 rows]: two tiles of 64 rows
  uint64_t* full = reinterpret_cast<uint64_t*>(B2 + ST_B2);
  uint64_t* empty = full + ST_SLOTS;
  uint64_t* s_ready = empty + ST_SLOTS;
  uint64_t* x_full = s_ready + 1;
  uint64_t* u_ready = x_full + 1;
  uint64_t* s_full = u_ready + 1;
  uint64_t* o_full = s_full + 1;                             // [2]: its waiters may be a chunk behind
  uint64_t* o_read = o_full + 2;                             // [2]
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(o_read + 2);
  const int slot_id = seg[sg * 4], r0 = seg[sg * 4 + 1], n = seg[sg * 4 + 2];
  const int nch = (n + GC - 1) / GC;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST_SLOTS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(s_ready, 8); mbar_init(x_full, 1); mbar_init(u_ready, 4); mbar_init(s_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&o_full[i], 1); mbar_init(&o_read[i], 4); }
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc<256>(tmem_ptr); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  constexpr uint32_t D3 = 128;                               // D1 buffers at columns 0 and 64
  const float* wsh = ws + (static_cast<size_t>(ci0) * Hv + h) * WS_STRIDE;
  const size_t ws_step = static_cast<size_t>(Hv) * WS_STRIDE;

  if (warp == 0) {
    // ------------------------------------------------------------ producer: a chunk is [Qt; W] x 4, Ut, Kt^T x 2, P
    int sl = 0; uint32_t ph = 0; bool ok = true;
    for (int c = 0; c < nch && ok; ++c) {
      const float* w = wsh + c * ws_step;
      for (int i = 0; i < 8; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[sl], ph ^ 1));
        if (!ok) { set_status(status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, blockIdx.y, c); break; }
        if (elect_one()) {
          const float* src = i < 4 ? w + WS_QW + i * 4096 : i == 4 ? w + WS_UT + vs * GVS * GC : i < 7 ? w + WS_KT + (i - 5) * 4096 : w + WS_P;
          mbar_arrive_expect_tx(&full[sl], ST_SLOT);
          bulk_load(smem + sl * ST_SLOT, src, ST_SLOT, &full[sl]);
        }
        __syncwarp();
        if (++sl == ST_SLOTS) { sl = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = make_idesc(2, 2, 128, GVS);
    const uint32_t sb = __shfl_sync(0xffffffffu, smem_u32(smem), 0), tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint32_t b1 = sb + ST_SLOTS * ST_SLOT, b2 = b1 + ST_B1;
    int sl = 0; uint32_t ph = 0; bool ok = true;
    auto next = [&]() { if (++sl == ST_SLOTS) { sl = 0; ph ^= 1; } };
    for (int c = 0; c < nch && ok; ++c) {
      const uint32_t d1 = tm + (c & 1) * GVS;
      ok = __all_sync(0xffffffffu, mbar_wait(s_ready, c & 1) && (c < 2 || mbar_wait(&o_read[c & 1], ((c >> 1) & 1) ^ 1)));
      if (!ok) { set_status(status, ST_TIMEOUT_TMEM_EMPTY, blockIdx.x, blockIdx.y, c); break; }
      for (int i = 0; i < 4 && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[sl], ph));
        tc_fence_after();
        if (ok && elect_one()) {
          const uint64_t ad = make_smem_desc_sw128(sb + sl * ST_SLOT), bd = make_smem_desc_sw128(b1 + i * (GVS * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32(d1, ad + 2 * k, bd + 2 * k, idesc, (i | k) != 0);
          umma_commit(&empty[sl]);
          if (i == 3) umma_commit(x_full);
        }
        __syncwarp();
        next();
      }
      if (!ok) { set_status(status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, c); break; }
      const int ut = sl;                                     // freed with P's tile: U is written, so Ut is read
      next();
      ok = __all_sync(0xffffffffu, mbar_wait(u_ready, c & 1));
      if (!ok) { set_status(status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, c); break; }
      for (int i = 0; i < 2 && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full[sl], ph));
        tc_fence_after();
        if (ok && elect_one()) {
          const uint64_t ad = make_smem_desc_sw128(sb + sl * ST_SLOT), bd = make_smem_desc_sw128(b2 + i * (GVS * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32(tm + D3, ad + 2 * k, bd + 2 * k, idesc, (i | k) != 0);
          umma_commit(&empty[sl]);
          if (i == 1) umma_commit(s_full);
        }
        __syncwarp();
        next();
      }
      ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[sl], ph));
      if (!ok) { set_status(status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, c); break; }
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint64_t ad = make_smem_desc_sw128(sb + sl * ST_SLOT + i * (GC * 128)), bd = make_smem_desc_sw128(b2 + i * (GVS * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int b = 2 * i + (k >> 1);                    // rows 16 b .. of U: lanes from 16 b on, and none past P's 64
            umma_tf32_add_lanes(d1, ad + 2 * k, bd + 2 * k, idesc, b == 0 ? 0u : b == 1 ? 0xffffu : ~0u, b == 3 ? 0xffffu : 0u, ~0u);
          }
        }
        umma_commit(&empty[sl]);
        umma_commit(&empty[ut]);
        umma_commit(&o_full[c & 1]);
      }
      __syncwarp();
      next();
    }
  } else {
    // ------------------------------------------------------------ state, U and O: lanes 32 q .. of tensor memory, value columns 32 hc ..
    const int q = warp & 3, hc = (warp - 2) >> 2;
    const int row = q * 32 + lane, v0 = vs * GVS + hc * 32;
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(q * 32) << 16) + hc * 32;
    float* Sg = S + ((static_cast<size_t>(slot_id) * Hv + h) * GD + v0) * GD + row;       // value v0 + i: Sg[i * GD]
    // this thread's float of value row i of an operand tile of 64 rows: key `row` of S^T, row `row - 64` of U^T
    uint8_t* s_tile = B1 + q * (GVS * 128) + hc * 32 * 128 + (lane & 3) * 4;
    uint8_t* u_tile = B2 + (q & 1) * (GVS * 128) + hc * 32 * 128 + (lane & 3) * 4;
    float s[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) s[i] = Sg[i * GD];
    bool ok = true;
    auto store_o = [&](int c) {                              // lanes of O: rows of chunk c
      if (!mbar_wait(&o_full[c & 1], (c >> 1) & 1)) return false;
      tc_fence_after();
      uint32_t o[32];
      tmem_ld_32x32(t_lane + (c & 1) * GVS, o);
      tmem_ld_wait();
      tc_fence_before();
      if (c * GC + row < n) {
        float4* dst = reinterpret_cast<float4*>(o_raw + static_cast<size_t>(r0 + c * GC + row) * ldo + h * GD + v0);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          dst[i] = make_float4(__uint_as_float(o[4 * i]), __uint_as_float(o[4 * i + 1]), __uint_as_float(o[4 * i + 2]), __uint_as_float(o[4 * i + 3]));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_read[c & 1]);
      return true;
    };
    float dc = 1.f;
    for (int c = 0; c <= nch; ++c) {
      const float dc_next = c < nch ? __ldg(wsh + c * ws_step + WS_DC) : 1.f;
      if (c > 0) {
        ok = __all_sync(0xffffffffu, mbar_wait(s_full, (c - 1) & 1));
        if (!ok) { set_status(status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, c); break; }
        tc_fence_after();
        uint32_t d[32];
        tmem_ld_32x32(t_lane + D3, d);
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int i = 0; i < 32; ++i) s[i] = fmaf(dc, s[i], __uint_as_float(d[i]));
      }
      dc = dc_next;
      if (c < nch) {
#pragma unroll
        for (int i = 0; i < 32; ++i) *reinterpret_cast<float*>(s_tile + i * 128 + ((((lane >> 2) ^ i) & 7) << 4)) = tf32r(s[i]);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_ready);
      }
      if (q < 2) {
        if (c > 0) {
          ok = __all_sync(0xffffffffu, store_o(c - 1));
          if (!ok) { set_status(status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, c); break; }
        }
      } else if (c < nch) {
        const int use = 8 * c + 4, sl = use % ST_SLOTS;
        ok = __all_sync(0xffffffffu, mbar_wait(&full[sl], (use / ST_SLOTS) & 1) && mbar_wait(x_full, c & 1));
        if (!ok) { set_status(status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, c); break; }
        tc_fence_after();
        uint32_t x[32];
        tmem_ld_32x32(t_lane + (c & 1) * GVS, x);
        const float4* ut = reinterpret_cast<const float4*>(smem + sl * ST_SLOT) + hc * 8 * GC + row - GC;
        float4 u[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) u[i] = ut[i * GC];
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float uv = i % 4 == 0 ? u[i / 4].x : i % 4 == 1 ? u[i / 4].y : i % 4 == 2 ? u[i / 4].z : u[i / 4].w;
          *reinterpret_cast<float*>(u_tile + i * 128 + ((((lane >> 2) ^ i) & 7) << 4)) = tf32r(uv - __uint_as_float(x[i]));
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(u_ready);
      }
    }
    if (ok) {
#pragma unroll
      for (int i = 0; i < 32; ++i) Sg[i * GD] = s[i];
    }
    if (vs == 0 && hc == 0) {          // conv history for the next call: raw inputs of the last three positions
      const int hk = h / (Hv / Hk), i = row;
      float* tl = tail + (static_cast<size_t>(slot_id) * 3 * Hv + h) * 3 * GD;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const __nv_bfloat16* pr = proj + static_cast<size_t>(r0 + n - 3 + j) * ldp;
        float* tj = tl + static_cast<size_t>(j) * Hv * 3 * GD;
        tj[i] = __bfloat162float(pr[hk * GD + i]);
        tj[GD + i] = __bfloat162float(pr[Hk * GD + hk * GD + i]);
        tj[2 * GD + i] = __bfloat162float(pr[2 * Hk * GD + h * GD + i]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc<256>(tmem); }
}

// ---------------------------------------------------------------------------------------------- kernel 3
// grid (chunks, Hv); 256 threads: warp w -> rows 8w..8w+7 of the chunk
__global__ void __launch_bounds__(256)
gdn_chunk_out_kernel(const float* __restrict__ o_raw, int ldo, const __nv_bfloat16* __restrict__ proj, int ldp,
                     const float* __restrict__ norm_w, const int* __restrict__ seg, const int* __restrict__ chunks,
                     __nv_bfloat16* __restrict__ out, int ldout, int Hk, int Hv, float eps) {
  const int ci = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sg = chunks[2 * ci], c = chunks[2 * ci + 1];
  const int r0 = seg[sg * 4 + 1], n = seg[sg * 4 + 2];
  const int zc = 2 * Hk * GD + Hv * GD + h * GD + lane * 4;
  const float4 nw = *reinterpret_cast<const float4*>(norm_w + lane * 4);
  for (int rr = 0; rr < 8; ++rr) {
    const int tt = c * GC + warp * 8 + rr;
    if (tt >= n) break;
    const size_t row = static_cast<size_t>(r0 + tt);
    const float4 o = *reinterpret_cast<const float4*>(o_raw + row * ldo + h * GD + lane * 4);
    const float o2 = warp_sum(o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w);
    const float rs = rsqrtf(o2 / GD + eps);
    const uint2 zr = *reinterpret_cast<const uint2*>(proj + row * ldp + zc);
    const float2 z0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zr.x));
    const float2 z1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zr.y));
    const __nv_bfloat162 b0 = __floats2bfloat162_rn(o.x * rs * nw.x / (1.f + __expf(-z0.x)), o.y * rs * nw.y / (1.f + __expf(-z0.y)));
    const __nv_bfloat162 b1 = __floats2bfloat162_rn(o.z * rs * nw.z / (1.f + __expf(-z1.x)), o.w * rs * nw.w / (1.f + __expf(-z1.y)));
    uint2 ov; ov.x = *reinterpret_cast<const uint32_t*>(&b0); ov.y = *reinterpret_cast<const uint32_t*>(&b1);
    *reinterpret_cast<uint2*>(out + row * ldout + h * GD + lane * 4) = ov;
  }
}

}  // namespace spark

using namespace spark;

extern "C" long long spark_gdn_chunk_ws_floats(int n_chunks, int Hv) {
  return static_cast<long long>(n_chunks) * Hv * WS_STRIDE;
}

// chunks: int [n_chunks][2] = (segment, chunk in segment); seg_chunk0: int [nseg] first chunk of a segment or -1
// (segment not served here).  head_dim must be 128; o_raw fp32 [R, Hv*128]; ws from spark_gdn_chunk_ws_floats.
extern "C" int spark_gdn_chunk_prefill(const void* proj, int ldp, const void* ab, int ldab, const float* conv_w,
                                       const float* A_log, const float* dt_bias, const float* norm_w, float* S, float* tail,
                                       const int* seg, int nseg, const int* chunks, int n_chunks, const int* seg_chunk0,
                                       float* ws, float* o_raw, void* out, int ldo, int Hk, int Hv, int D, float eps,
                                       int* status, cudaStream_t s) {
  if (n_chunks <= 0) return 0;
  if (D != GD || Hv % Hk || ((reinterpret_cast<uintptr_t>(ws) | reinterpret_cast<uintptr_t>(o_raw)) & 15)) return -5;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(gdn_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PREP_SMEM);
    cudaFuncSetAttribute(gdn_chunk_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM);
    attr = true;
  }
  gdn_chunk_prep_kernel<<<dim3(n_chunks, Hv), 256, PREP_SMEM, s>>>((const __nv_bfloat16*)proj, ldp, (const __nv_bfloat16*)ab, ldab,
                                                              conv_w, A_log, dt_bias, tail, seg, chunks, ws, Hk, Hv, eps,
                                                                  (reinterpret_cast<uintptr_t>(conv_w) & 15) == 0);
  gdn_chunk_state_kernel<<<dim3(GD / GVS, Hv, nseg), ST_THREADS, ST_SMEM, s>>>(ws, seg, seg_chunk0, (const __nv_bfloat16*)proj, ldp, S,
                                                                              tail, o_raw, Hv * GD, Hk, Hv, status);
  gdn_chunk_out_kernel<<<dim3(n_chunks, Hv), 256, 0, s>>>(o_raw, Hv * GD, (const __nv_bfloat16*)proj, ldp, norm_w, seg, chunks,
                                                          (__nv_bfloat16*)out, ldo, Hk, Hv, eps);
  return spark_launch_rc(__func__);
}
