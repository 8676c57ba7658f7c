// MoE routing and combine kernels.
//   moe_route    : router scores -> top-k (ties -> lowest expert id) -> renormalised weights; three
//                  router kinds (softmax-renorm, sigmoid+bias x scale, sqrt-softplus+bias x scale);
//                  also emits the (row, expert) pair table the grouped GEMV/GEMM kernels consume.
//   moe_sort     : stable counting sort of the (row, slot) pairs by expert -> permuted row list, expert
//                  offsets and the tile list (16 to 192 rows) of the grouped tcgen05 GEMMs (int atomics only,
//                  order inside an expert = ascending pair index, so the result is deterministic).
//   moe_combine  : residual += sum over slots (slot order) of weight * expert output (+ gated shared).
// Reference: engine-rs/shim/qwen_moe.cu:10-92, dataflow.cu:370-572, ds41_ops.cu:375-421 (routers);
// moe_exl3.cuh:141-231 (count/scan/fill), :1085 (slot-order combine).
#include "../common/decode.cuh"
#include <type_traits>

namespace spark {

constexpr int ROUTE_MAXE = 1024;
constexpr int ROUTE_ROWS = 8;                // rows (warps) per CTA

// Best of a lane's EPL selection scores and the lowest position that holds it: a max tree and a bit mask, not a serial compare chain.
// A score that is no number is never the best.
template <int EPL>
__device__ __forceinline__ void lane_best(const float (&s)[EPL], float& best, int& bj) {
  float m[EPL];
#pragma unroll
  for (int j = 0; j < EPL; ++j) m[j] = s[j];
#pragma unroll
  for (int w = EPL / 2; w >= 1; w >>= 1)
#pragma unroll
    for (int j = 0; j < w; ++j) m[j] = fmaxf(m[j], m[j + w]);
  best = m[0] == m[0] ? m[0] : -INFINITY;
  unsigned mask = 0u;
#pragma unroll
  for (int j = 0; j < EPL; ++j) mask |= (s[j] == best ? 1u : 0u) << j;
  bj = __ffs(mask) - 1;
  if (bj < 0) bj = 0;
}

// kind: 0 softmax, 1 sigmoid+bias, 2 sqrt(softplus)+bias, 3 softmax+bias (the bias enters the choice only), 4 sigmoid, not
// renormalised (ranked by the logits, which a saturated sigmoid would tie), 5 softmax over the chosen logits alone (bias, if any,
// added to the logits; ranked by them, and only the chosen ones are exponentiated, against the largest).
// The last n_self of the E router outputs are identity experts: they leave -1 in `ids` and their weight in self_w[row].
// One warp per row, EPL experts per lane; a choice is two warp reductions (the largest score's order-preserving key, the lowest expert
// among the lanes that hold it).  A CTA per row with three block barriers per choice took 107 us for 8192 rows of 512 experts, top
// 10; this takes 31.
template <int EPL>
__global__ void __launch_bounds__(ROUTE_ROWS * 32)
moe_route_kernel(const float* __restrict__ logits, int ld, int R, int E, int top_k, int kind, const float* __restrict__ bias,
                 float scale, int shared_gate, float* __restrict__ wts, int* __restrict__ ids,
                 int* __restrict__ pair_row, float* __restrict__ sg, int e_lo, int e_hi, int n_self, float* __restrict__ self_w) {
  const int r = blockIdx.x * ROUTE_ROWS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= R) return;
  const float* x = logits + static_cast<size_t>(r) * ld;
  float p[EPL], s[EPL];                                     // p: what the weights are made of; s: selection score
  float mx = -INFINITY;
#pragma unroll
  for (int j = 0; j < EPL; ++j) {
    const int e = lane + 32 * j;
    p[j] = e < E ? x[e] : -INFINITY;
    if (kind == 5 && bias && e < E) p[j] += bias[e];
    mx = fmaxf(mx, p[j]);
  }
  if (kind == 0 || kind == 3) {
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      p[j] = lane + 32 * j < E ? expf(p[j] - mx) : 0.f;
      sum += p[j];
    }
    sum = warp_sum(sum);
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      p[j] = p[j] / sum;
      s[j] = p[j];
      if (kind == 3 && lane + 32 * j < E) s[j] += bias[lane + 32 * j];
    }
  } else if (kind == 4) {
#pragma unroll
    for (int j = 0; j < EPL; ++j) { s[j] = p[j]; p[j] = 1.f / (1.f + expf(-p[j])); }
  } else if (kind == 5) {
#pragma unroll
    for (int j = 0; j < EPL; ++j) s[j] = p[j];
  } else {
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = lane + 32 * j;
      if (e < E) {
        const float v = p[j];
        if (kind == 1) p[j] = 1.f / (1.f + expf(-v));
        else p[j] = sqrtf(v > 20.f ? v : log1pf(expf(v)));
        s[j] = p[j] + (bias ? bias[e] : 0.f);
      } else { p[j] = 0.f; s[j] = -INFINITY; }
    }
  }
#pragma unroll
  for (int j = 0; j < EPL; ++j) if (lane + 32 * j >= E) s[j] = -INFINITY;
  float selp = 0.f, best; int seli = 0x7fffffff, bj;          // lane k keeps slot k's weight numerator and expert
  lane_best(s, best, bj);
  for (int k = 0; k < top_k; ++k) {
    const uint32_t bits = __float_as_uint(best + 0.f);        // -0 ranks as 0
    const uint32_t key = best == -INFINITY ? 0u : (bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u));
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, key);
    const int cand = (key == wmax && key != 0u) ? lane + 32 * bj : 0x7fffffff;
    const int wi = __reduce_min_sync(0xffffffffu, cand);
    float bp = 0.f;
    if (wi == cand && wi != 0x7fffffff) {                     // this lane owns the winner
#pragma unroll
      for (int j = 0; j < EPL; ++j) if (j == bj) { bp = p[j]; s[j] = -INFINITY; }
      lane_best(s, best, bj);
    }
    const float wp = __shfl_sync(0xffffffffu, bp, wi & 31);
    if (lane == k) { selp = wp; seli = wi; }
  }
  if (kind == 5) {                                            // the first one chosen is the largest
    const float top = __shfl_sync(0xffffffffu, selp, 0);
    selp = lane < top_k ? expf(selp - top) : 0.f;
  }
  float sum = 0.f, own = 0.f;
  for (int k = 0; k < top_k; ++k) sum += __shfl_sync(0xffffffffu, selp, k);      // slot order
  sum = kind == 4 ? 1.f : fmaxf(sum, 1e-20f);
  const float w = selp / sum * scale;
  if (self_w) {
    for (int k = 0; k < top_k; ++k) {
      const float wk = __shfl_sync(0xffffffffu, w, k);
      if (__shfl_sync(0xffffffffu, seli, k) >= E - n_self) own += wk;
    }
    if (lane == 0) self_w[r] = own;
  }
  if (lane < top_k) {
    const size_t o = static_cast<size_t>(r) * top_k + lane;
    wts[o] = w;
    // expert-parallel ranks keep only their own experts [e_lo, e_hi): others become -1 (skipped downstream)
    ids[o] = (seli >= e_lo && seli < e_hi) ? seli - e_lo : -1;
    if (pair_row) pair_row[o] = r;
  }
  if (lane == 0 && shared_gate) sg[r] = 1.f / (1.f + expf(-x[E]));
}


// ---------------------------------------------------------------------------------- decode router (fused)
// One launch for <= 16 rows: router GEMV over the E (+1 shared-gate) columns, then the CTA that finishes last
// (integer arrival counter, nobody waits) scores, picks the top-k experts of every row with one warp per row and
// writes the pair tables the expert GEMVs read: ids / weights / source row for top_k routed slots plus an optional
// shared-expert slot (the shared expert is stored as one more matrix of the expert stack, so it is just another
// pair; under tensor parallelism row r's shared pair belongs to rank r % world).
// Replaces three launches (norm, GEMV, route); reference: engine-rs/shim/qwen_moe.cu:10-92, dataflow.cu:370-572.
struct RouterArgs {
  const __nv_bfloat16* x; int ldx;           // [R, K]
  const __nv_bfloat16* Wg; int ldw;          // [E (+1), K]
  float* logits; int ld;                     // scratch [R, ld]
  int R, K, E, top_k, kind;                  // kind: 0 softmax, 1 sigmoid+bias, 2 sqrt(softplus)+bias, 3 softmax+bias, 4 sigmoid, 5 softmax of the chosen
  const float* bias; float scale; int shared_gate;
  int slots;                                 // top_k, or top_k + 1 when the shared expert is a pair
  int shared_expert;                         // index of the shared expert in the local stack (slot top_k)
  int e_lo, e_hi, rank, world;
  float* wts; int* ids; int* pair_row;       // [R, slots]
  float* sg;                                 // optional [R]: shared gate (when the shared expert is NOT a pair)
  int* counter;
  int n_self; float* self_w;                 // identity experts: the last n_self outputs, their weight per row [R]
};

constexpr int ROUTER_RB = 16, ROUTER_WARPS = 16, ROUTER_COLS = 4;

// A CTA owns four gate columns, a warp one of them for every fourth row (NR of them).  A lane adds the products of every 32nd 16-byte
// vector in one 32-bit chain per row, the lanes' sums meet by shuffles: the order of a row's sum depends on neither R nor NR.  The
// loads are 16 bytes, straight from memory, a batch of a row's and a column's vectors in flight (the rows of a CTA stay in L1).
// What bounds it: a memory round trip per batch and the chain of the choices, one warp per row.  4 rows of 2048 and 513 columns 13.7 ->
// 7.5 us, 16 rows 32 -> 15.2, 4 rows of the MXFP4 preset 37 -> 13.6 (before: a warp per column for all rows, the rows staged in shared
// memory, two rows' choices after one another, one kernel for all kinds).  Tensor cores in place of the FP32 units (9.3, 13, 16 us) add
// 16 products at a time with fewer bits: the logits' error grew 1.2 to 15 times over K = 256 .. 7168.
// KIND: a kernel per kind (it is fetched anew in every layer: what a kind does not run costs instruction misses; kinds 3, 4 and 5 in one took
// 11.9, 10.4 and 10.0 us for 4 rows of 2048 and 512 columns, alone 10.0, 7.1 and 7.0; all six in one 10.7, 7.9 and 8.1)
template <int EPL, int NR, int KIND>                        // NR: rows of a warp (R <= 4 NR)
__global__ void __launch_bounds__(ROUTER_WARPS * 32)
moe_router_topk_kernel(const __grid_constant__ RouterArgs a) {
  __shared__ int last_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kind = KIND;
  const int R = a.R;
  const int NE = a.E + (a.shared_gate ? 1 : 0);
  const int n = blockIdx.x * ROUTER_COLS + (warp & 3), r0 = warp >> 2;
  const int KV = a.K >> 3;                                  // 16-byte vectors of a row
  constexpr int BATCH = NR == 1 ? 8 : NR == 4 && EPL == 32 ? 2 : 4;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* w = reinterpret_cast<const uint4*>(a.Wg + static_cast<size_t>(min(n, NE - 1)) * a.ldw);
  // the gate matrix depends on no earlier launch: its first batch of loads is in flight before the dependency wait
  uint4 wv[BATCH];
#pragma unroll
  for (int u = 0; u < BATCH; ++u) {
    const int kv = lane + 32 * u;
    wv[u] = kv < KV ? __ldg(w + kv) : zero;
  }
  pdl_wait();
  pdl_trigger();
  if (n < NE && r0 < R) {
    float acc[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) acc[i] = 0.f;
    for (int k0 = lane; k0 < KV; k0 += 32 * BATCH) {
      uint4 xv[NR][BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int kv = k0 + 32 * u;
        if (k0 != lane) wv[u] = kv < KV ? __ldg(w + kv) : zero;
#pragma unroll
        for (int i = 0; i < NR; ++i)
          xv[i][u] = kv < KV ? reinterpret_cast<const uint4*>(a.x + static_cast<size_t>(min(r0 + 4 * i, R - 1)) * a.ldx)[kv] : zero;
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        if (k0 + 32 * u >= KV) break;
        const __nv_bfloat162* pw = reinterpret_cast<const __nv_bfloat162*>(&wv[u]);
        float2 f[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) f[j] = __bfloat1622float2(pw[j]);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const __nv_bfloat162* px = reinterpret_cast<const __nv_bfloat162*>(&xv[i][u]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 t = __bfloat1622float2(px[j]);
            acc[i] = fmaf(f[j].x, t.x, acc[i]); acc[i] = fmaf(f[j].y, t.y, acc[i]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      float v = warp_sum(acc[i]);
      // kinds whose score is a function of the logit alone are scored here, on every SM, and not by the last CTA
      if (n < a.E && kind == 1) v = 1.f / (1.f + expf(-v));
      if (n < a.E && kind == 2) v = sqrtf(v > 20.f ? v : log1pf(expf(v)));
      if (lane == 0 && r0 + 4 * i < R) a.logits[static_cast<size_t>(r0 + 4 * i) * a.ld + n] = v;
    }
  }
  // ---- arrival: the last CTA to get here routes every row
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const int old = atomicAdd(a.counter, 1);
    last_s = old == static_cast<int>(gridDim.x) - 1;
    if (last_s) *a.counter = 0;
  }
  __syncthreads();
  if (!last_s) return;
  // (the writers fenced before they arrived; the logits are read with L2 loads, so no reader-side fence)
  // EPL experts per lane (E <= 32 * EPL).  The k selection rounds are a serial chain, so each round is kept short (lane_best: a
  // serial compare chain in its place spent 5.8 us per group of rows).
  const int nj = (a.E + 31) >> 5;
  for (int r = warp; r < R; r += ROUTER_WARPS) {
    const float* lg = a.logits + static_cast<size_t>(r) * a.ld;
    float p[EPL], s[EPL];                                   // p: what the weights are made of; s: selection score
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
      const int e = lane + 32 * j;
      p[j] = (j < nj && e < a.E) ? __ldcg(lg + e) : -INFINITY;
      if (kind == 5 && a.bias && j < nj && e < a.E) p[j] += a.bias[e];
      s[j] = p[j];
      mx = fmaxf(mx, p[j]);
    }
    if (kind == 4) {
      // ranked by the logits, only the k winners' sigmoids are formed
    } else if (kind == 5) {
      mx = warp_max(mx);
    } else if (kind == 0) {
      // softmax -> top-k -> renormalise: the softmax denominator cancels, so experts are ranked by their logits and
      // only the k winners are exponentiated
      mx = warp_max(mx);
    } else if (kind == 3) {
      // the bias is added to the probabilities, so the ranking needs the denominator
      mx = warp_max(mx);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        p[j] = p[j] == -INFINITY ? 0.f : expf(p[j] - mx);
        sum += p[j];
      }
      sum = warp_sum(sum);
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        const bool in = j < nj && e < a.E;
        p[j] = p[j] / sum;
        s[j] = in ? p[j] + a.bias[e] : -INFINITY;
      }
    } else {
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        if (j < nj && e < a.E) s[j] = p[j] + (a.bias ? a.bias[e] : 0.f);
        else { p[j] = 0.f; s[j] = -INFINITY; }
      }
    }
    float selp = 0.f; int seli = -1;                        // lane k keeps slot k's weight numerator and expert
    float tot = 0.f;
    // A round: warp maximum of the candidates' order-preserving integer keys (one redux), lowest expert id among the
    // lanes that hold it (one redux), the winning lane takes its expert out and finds its next best.
    float best; int bj;
    lane_best(s, best, bj);
    for (int k = 0; k < a.top_k; ++k) {
      const uint32_t bits = __float_as_uint(best);
      const uint32_t key = best == -INFINITY ? 0u : (bits ^ ((bits >> 31) ? 0xffffffffu : 0x80000000u));
      const uint32_t wmax = __reduce_max_sync(0xffffffffu, key);
      const int cand = (key == wmax && key != 0u) ? lane + 32 * bj : 0x7fffffff;
      const int wi = __reduce_min_sync(0xffffffffu, cand);
      float bp = 0.f;
      if (wi == cand && wi != 0x7fffffff) {                 // this lane owns the winner
#pragma unroll
        for (int j = 0; j < EPL; ++j) if (j == bj) { bp = p[j]; s[j] = -INFINITY; }
        if (kind == 0) bp = __expf(bp - mx);
        if (kind == 5) bp = expf(bp - mx);
        if (kind == 4) bp = 1.f / (1.f + expf(-bp));
        lane_best(s, best, bj);
      }
      const float wp = __shfl_sync(0xffffffffu, bp, wi & 31);
      if (lane == k) { selp = wp; seli = wi; }
      tot += wp;                                            // slot order, identical on every lane
    }
    tot = kind == 4 ? 1.f : fmaxf(tot, 1e-20f);
    if (a.self_w) {
      float own = 0.f;
      for (int k = 0; k < a.top_k; ++k) {                   // slot order, as the combine adds the others
        const float w = __shfl_sync(0xffffffffu, selp, k) / tot * a.scale;
        if (__shfl_sync(0xffffffffu, seli, k) >= a.E - a.n_self) own += w;
      }
      if (lane == 0) a.self_w[r] = own;
    }
    const size_t o = static_cast<size_t>(r) * a.slots;
    if (lane < a.top_k) {
      a.wts[o + lane] = selp / tot * a.scale;
      a.ids[o + lane] = (seli >= a.e_lo && seli < a.e_hi) ? seli - a.e_lo : -1;
      if (a.pair_row) a.pair_row[o + lane] = r;
    }
    if (lane == 0) {
      const float g = a.shared_gate ? 1.f / (1.f + __expf(-__ldcg(lg + a.E))) : 1.f;
      if (a.slots > a.top_k) {
        a.wts[o + a.top_k] = g;
        a.ids[o + a.top_k] = (r % a.world) == a.rank ? a.shared_expert : -1;
        if (a.pair_row) a.pair_row[o + a.top_k] = r;
      }
      if (a.sg) a.sg[r] = g;
    }
  }
}

// Decode combine fused with the residual update and the next RMSNorm: one CTA per row.
//   res[r] += sum over slots (slot order) of weight * y[pair] (+ gated shared);  h[r] = rmsnorm(res[r]) * w  (bf16)
// Replaces combine + add_rmsnorm (two launches); reference: engine-rs/shim/moe_exl3.cuh:1381 finish_combine_kernel.
__global__ void __launch_bounds__(1024)
moe_combine_norm_kernel(const float* __restrict__ y, const float* __restrict__ wts, const int* __restrict__ ids, int slots,
                        int H, float* __restrict__ res, const float* __restrict__ norm_w, float eps, int one_plus,
                        __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ shared,
                        const float* __restrict__ sg) {
  __shared__ float red[32];
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x;
  float4 keep[2];                                          // H <= 2 * 4 * blockDim.x
  float ss = 0.f;
  int ki = 0;
  for (int col = threadIdx.x * 4; col < H; col += blockDim.x * 4, ++ki) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k0 = 0; k0 < slots; k0 += 4) {                // four slots' loads in flight; summed in slot order
      float4 v[4]; float w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int pi = r * slots + k0 + u;
        const bool live = (k0 + u) < slots && ids[pi] >= 0;
        w[u] = live ? wts[pi] : 0.f;
        v[u] = live ? __ldcg(reinterpret_cast<const float4*>(y + static_cast<size_t>(pi) * H + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        acc.x = fmaf(w[u], v[u].x, acc.x); acc.y = fmaf(w[u], v[u].y, acc.y);
        acc.z = fmaf(w[u], v[u].z, acc.z); acc.w = fmaf(w[u], v[u].w, acc.w);
      }
    }
    if (shared) {
      const uint2 raw = *reinterpret_cast<const uint2*>(shared + static_cast<size_t>(r) * H + col);
      const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
      const float2 f0 = __bfloat1622float2(p2[0]), f1 = __bfloat1622float2(p2[1]);
      const float g = sg ? sg[r] : 1.f;
      acc.x += g * f0.x; acc.y += g * f0.y; acc.z += g * f1.x; acc.w += g * f1.y;
    }
    float* rp = res + static_cast<size_t>(r) * H + col;
    float4 o4 = *reinterpret_cast<const float4*>(rp);
    o4.x += acc.x; o4.y += acc.y; o4.z += acc.z; o4.w += acc.w;
    *reinterpret_cast<float4*>(rp) = o4;
    ss += o4.x * o4.x + o4.y * o4.y + o4.z * o4.z + o4.w * o4.w;
    if (ki < 2) keep[ki] = o4;
  }
  ss = warp_sum(ss);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  float tot = 0.f;
  for (int w = 0; w < nw; ++w) tot += red[w];              // fixed order
  const float rs = rsqrtf(tot / H + eps);
  ki = 0;
  for (int col = threadIdx.x * 4; col < H; col += blockDim.x * 4, ++ki) {
    const float4 v = keep[ki < 2 ? ki : 1];
    const float4 g = *reinterpret_cast<const float4*>(norm_w + col);
    const float o = one_plus ? 1.f : 0.f;
    __nv_bfloat162 b0 = __floats2bfloat162_rn(v.x * rs * (g.x + o), v.y * rs * (g.y + o));
    __nv_bfloat162 b1 = __floats2bfloat162_rn(v.z * rs * (g.z + o), v.w * rs * (g.w + o));
    uint2 ov; ov.x = *reinterpret_cast<uint32_t*>(&b0); ov.y = *reinterpret_cast<uint32_t*>(&b1);
    *reinterpret_cast<uint2*>(h + static_cast<size_t>(r) * H + col) = ov;
  }
}

// ---------------------------------------------------------------------------------- counting sort
// ids [P] expert per pair (P = R * top_k) -> perm [P] (pair index in expert order), offsets [E + 1], list of row tiles, its length.
// Stable: rank of pair i inside its expert = exclusive count over earlier pairs.  Two passes over blocks of pairs with per-block histograms (deterministic, int atomics only in smem).
__global__ void moe_hist_kernel(const int* __restrict__ ids, int P, int E, int* __restrict__ block_hist) {
  extern __shared__ int sh[];
  for (int e = threadIdx.x; e < E; e += blockDim.x) sh[e] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P && ids[i] >= 0) atomicAdd(&sh[ids[i]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) block_hist[static_cast<size_t>(blockIdx.x) * E + e] = sh[e];
}
// Offsets and row tiles of experts with `mine` rows each, a thread per expert (two scans over the CTA: rows -> offsets, tiles -> first tile);
// each writes its own tiles (one thread walking 512 experts took 72 us).  Returns the expert's first row.  sa, sb: [blockDim.x].
template <int NT>                                      // threads of the CTA, 0: blockDim.x
__device__ __forceinline__ int moe_tiles(int mine, int E, int tile_rows, int* sa, int* sb, int* __restrict__ offsets, int4* __restrict__ tile_list,
                                         int* __restrict__ tile_count) {
  const int e = threadIdx.x;
  const int my_tiles = (mine + tile_rows - 1) / tile_rows;
  sa[e] = mine; sb[e] = my_tiles;
  __syncthreads();
  for (int st = 1; st < (NT ? NT : blockDim.x); st <<= 1) {         // inclusive scans of rows and of tiles
    const int a = e >= st ? sa[e - st] : 0, b = e >= st ? sb[e - st] : 0;
    __syncthreads();
    sa[e] += a; sb[e] += b;
    __syncthreads();
  }
  const int off = sa[e] - mine, t0 = sb[e] - my_tiles;
  if (e < E) {
    offsets[e] = off;
    if (tile_rows == 128) {                              // the consumer cuts a tile at the expert's end
      for (int i = 0; i < my_tiles; ++i) tile_list[t0 + i] = make_int4(off + i * 128, off + mine, e, 0);
    } else if (my_tiles) {                               // even split
      const int q = mine / my_tiles, more = mine % my_tiles;
      for (int i = 0; i < my_tiles; ++i) tile_list[t0 + i] = make_int4(off + i * q + min(i, more), off + mine, e, q + (i < more));
    }
    if (e == E - 1) { offsets[E] = sa[e]; *tile_count = sb[e]; }
  }
  return off;
}

// Few pairs and experts in one launch, a thread per pair and per expert.  us, three launches / this: 257 pairs of 8 or 256
// experts 8.1 / 4.5, 512 8.1 / 6.8, 640 8.1 / 8.3 (a thread's rank is a walk over the pairs before it,
// and the line: with one thread for the experts 2048 pairs of 8 or 512 experts in one launch took 50 and 109, three take 8.2 and 8.7)
constexpr int SORT_ONE = 640;

__global__ void __launch_bounds__(SORT_ONE)
moe_sort_one_kernel(const int* __restrict__ ids, int P, int E, int* __restrict__ perm, int* __restrict__ inv_perm, int* __restrict__ offsets,
                    int4* __restrict__ tile_list, int* __restrict__ tile_count, int tile_rows) {
  __shared__ int sa[SORT_ONE], sb[SORT_ONE], first[SORT_ONE];
  __shared__ __align__(16) int sid[SORT_ONE];
  const int i = threadIdx.x, e = i < P ? ids[i] : -1;
  sid[i] = e;
  first[i] = 0;
  __syncthreads();
  if (e >= 0) atomicAdd(&first[e], 1);
  __syncthreads();
  const int mine = first[i];                             // threads past E: none
  const int off = moe_tiles<0>(mine, E, tile_rows, sa, sb, offsets, tile_list, tile_count);
  first[i] = off;
  __syncthreads();
  if (i >= P) return;
  if (e < 0) { if (inv_perm) inv_perm[i] = -1; return; }
  int dst = first[e];
  int j = 0;                                             // earlier pairs of the expert
#pragma unroll 4
  for (; j + 4 <= i; j += 4) {
    const int4 v = *reinterpret_cast<const int4*>(sid + j);
    dst += (v.x == e) + (v.y == e) + (v.z == e) + (v.w == e);
  }
  for (; j < i; ++j) dst += sid[j] == e;
  perm[dst] = i;
  if (inv_perm) inv_perm[i] = dst;
}

// one CTA: exclusive scan over blocks per expert, offsets, tile list
__global__ void __launch_bounds__(1024)
moe_scan_kernel(int* __restrict__ block_hist, int nblocks, int E, int* __restrict__ offsets,
                int4* __restrict__ tile_list, int* __restrict__ tile_count, int tile_rows) {
  __shared__ int sa[1024], sb[1024];
  const int e = threadIdx.x;
  int mine = 0;
  if (e < E) {
    // sixteen counts are asked for before the first is overwritten (one at a time: 40 us for the 320 blocks of 8192 rows, top 10)
    for (int b0 = 0; b0 < nblocks; b0 += 16) {
      int c[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) c[u] = b0 + u < nblocks ? block_hist[static_cast<size_t>(b0 + u) * E + e] : 0;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        if (b0 + u < nblocks) block_hist[static_cast<size_t>(b0 + u) * E + e] = mine;
        mine += c[u];
      }
    }
  }
  moe_tiles<1024>(mine, E, tile_rows, sa, sb, offsets, tile_list, tile_count);
}
__global__ void moe_place_kernel(const int* __restrict__ ids, int P, int E, const int* __restrict__ block_hist,
                                 const int* __restrict__ offsets, int* __restrict__ perm, int* __restrict__ inv_perm) {
  extern __shared__ int sid[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  sid[threadIdx.x] = i < P ? ids[i] : -1;
  __syncthreads();
  if (i >= P) return;
  const int e = sid[threadIdx.x];
  if (e < 0) { if (inv_perm) inv_perm[i] = -1; return; }
  int rank = 0;
  for (int j = 0; j < threadIdx.x; ++j) rank += (sid[j] == e);
  const int dst = offsets[e] + block_hist[static_cast<size_t>(blockIdx.x) * E + e] + rank;
  perm[dst] = i;
  if (inv_perm) inv_perm[i] = dst;
}

// ---------------------------------------------------------------------------------- combine
// res[R,H] += sum_slot w[r,slot] * y[pair_pos(r,slot), :] (+ sg[r] * shared[r,:]).  y fp32 or bf16.
// A thread owns V consecutive columns (one 16-byte load of y per slot; V = 1 where H or an address does not allow it).  The row's slots
// are looked up once per CTA, and a thread's loads of eight slots are issued before the first is widened (a load and its widening in one
// branch per slot waited for every slot by itself).  Added in slot order.  Bound by reading y: 8192 rows of 2048, ten bf16 slots, 82 us
// (110 with a wait per slot, 224 with one column per thread); 2048 rows of 4096, six fp32 slots, 42 (49, 91).
template <int V, typename T> struct CombVec { typedef T type; };
template <> struct CombVec<4, float> { typedef uint4 type; };
template <> struct CombVec<8, __nv_bfloat16> { typedef uint4 type; };
__device__ __forceinline__ void comb_widen(const uint4& r, float (&v)[4]) {
  v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
}
__device__ __forceinline__ void comb_widen(const uint4& r, float (&v)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __bfloat1622float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void comb_widen(const float& r, float (&v)[1]) { v[0] = r; }
__device__ __forceinline__ void comb_widen(const __nv_bfloat16& r, float (&v)[1]) { v[0] = __bfloat162float(r); }

constexpr int COMB_SLOTS = 32, COMB_U = 8;

template <typename TY, int V>
__global__ void __launch_bounds__(256)
moe_combine_kernel(float* __restrict__ res, const TY* __restrict__ y, const int* __restrict__ inv_perm,
                   const float* __restrict__ wts, int top_k, const __nv_bfloat16* __restrict__ shared,
                   const float* __restrict__ sg, int H, __nv_bfloat16* __restrict__ out_bf16,
                   const int* __restrict__ pair_expert) {
  typedef typename CombVec<V, TY>::type Raw;
  __shared__ int row_s[COMB_SLOTS];                           // row of y, -1: the expert lives on another rank
  __shared__ float w_s[COMB_SLOTS];
  const int r = blockIdx.x;
  const float gate = shared && sg ? sg[r] : 1.f;
  const int i = (blockIdx.y * blockDim.x + threadIdx.x) * V;
  float acc[V];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = 0.f;
  for (int s0 = 0; s0 < top_k; s0 += COMB_SLOTS) {
    const int n = min(top_k - s0, COMB_SLOTS);
    if (s0) __syncthreads();
    if (threadIdx.x < n) {
      const int pi = r * top_k + s0 + threadIdx.x;
      row_s[threadIdx.x] = pair_expert && pair_expert[pi] < 0 ? -1 : (inv_perm ? inv_perm[pi] : pi);
      w_s[threadIdx.x] = wts[pi];
    }
    __syncthreads();
    if (i >= H) continue;
    for (int k0 = 0; k0 < n; k0 += COMB_U) {
      Raw raw[COMB_U];
#pragma unroll
      for (int u = 0; u < COMB_U; ++u) {
        const int row = k0 + u < n ? row_s[k0 + u] : -1;
        if (row >= 0) raw[u] = __ldg(reinterpret_cast<const Raw*>(y + static_cast<size_t>(row) * H + i));
      }
#pragma unroll
      for (int u = 0; u < COMB_U; ++u)
        if (k0 + u < n && row_s[k0 + u] >= 0) {
          float v[V];
          comb_widen(raw[u], v);
#pragma unroll
          for (int j = 0; j < V; ++j) acc[j] = fmaf(w_s[k0 + u], v[j], acc[j]);
        }
    }
  }
  if (i >= H) return;
  const size_t o = static_cast<size_t>(r) * H + i;
  if (shared) {
    uint32_t sw[(V + 1) / 2];                                 // V consecutive elements, as one load
    if (V == 8) { const uint4 t = *reinterpret_cast<const uint4*>(shared + o); sw[0] = t.x; sw[1 % ((V + 1) / 2)] = t.y; sw[2 % ((V + 1) / 2)] = t.z; sw[3 % ((V + 1) / 2)] = t.w; }
    else if (V == 4) { const uint2 t = *reinterpret_cast<const uint2*>(shared + o); sw[0] = t.x; sw[1 % ((V + 1) / 2)] = t.y; }
    else sw[0] = reinterpret_cast<const uint16_t*>(shared)[o];
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float s = __uint_as_float(j & 1 ? sw[j >> 1] & 0xffff0000u : sw[j >> 1] << 16);
      acc[j] += sg ? gate * s : s;
    }
  }
  if (res) {
#pragma unroll
    for (int j = 0; j < V; ++j) res[o + j] += acc[j];
  }
  if (out_bf16) {
    if (V == 1) {
      out_bf16[o] = __float2bfloat16(acc[0]);
    } else {
#pragma unroll
      for (int j = 0; j < V; j += 4) {
        const __nv_bfloat162 b0 = __floats2bfloat162_rn(acc[j % V], acc[(j + 1) % V]), b1 = __floats2bfloat162_rn(acc[(j + 2) % V], acc[(j + 3) % V]);
        *reinterpret_cast<uint2*>(out_bf16 + o + j) = make_uint2(*reinterpret_cast<const uint32_t*>(&b0), *reinterpret_cast<const uint32_t*>(&b1));
      }
    }
  }
}

// The same for up to four slots: every thread looks them up itself, with no table to wait for.  us, table / this: 4096 rows of 4096, fp32, one
// slot 51 / 32, two 56 / 38, three 63 / 45, four 71 / 54; single columns, 4096 rows of 2050, four slots 72 / 50 (eight of them this way: 86 / 115);
// 17 rows 2.5 / 2.3.  bf16 vectors of 8 take the same time either way.
template <typename TY, int V>
__global__ void __launch_bounds__(256)
moe_combine_few_kernel(float* __restrict__ res, const TY* __restrict__ y, const int* __restrict__ inv_perm, const float* __restrict__ wts, int top_k,
                       const __nv_bfloat16* __restrict__ shared, const float* __restrict__ sg, int H, __nv_bfloat16* __restrict__ out_bf16,
                       const int* __restrict__ pair_expert) {
  const int r = blockIdx.x, i = (blockIdx.y * blockDim.x + threadIdx.x) * V;
  if (i >= H) return;
  const float gate = shared && sg ? sg[r] : 1.f;
  float acc[V], v[4][V], w[4];
  bool live[4];
#pragma unroll
  for (int j = 0; j < V; ++j) acc[j] = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int pi = r * top_k + min(u, top_k - 1);
    live[u] = u < top_k && !(pair_expert && pair_expert[pi] < 0);                // else: no slot, or the expert lives on another rank
    const int row = inv_perm ? inv_perm[pi] : pi;
    w[u] = wts[pi];
    if (live[u]) comb_widen(__ldg(reinterpret_cast<const typename CombVec<V, TY>::type*>(y + static_cast<size_t>(row) * H + i)), v[u]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (live[u]) {
#pragma unroll
      for (int j = 0; j < V; ++j) acc[j] = fmaf(w[u], v[u][j], acc[j]);
    }
  const size_t o = static_cast<size_t>(r) * H + i;
  if (shared) {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float s = __bfloat162float(shared[o + j]);
      acc[j] += sg ? gate * s : s;
    }
  }
  if (res) {
#pragma unroll
    for (int j = 0; j < V; ++j) res[o + j] += acc[j];
  }
  if (out_bf16) {
    if (V == 4) {
      const __nv_bfloat162 b0 = __floats2bfloat162_rn(acc[0], acc[1 % V]), b1 = __floats2bfloat162_rn(acc[2 % V], acc[3 % V]);
      *reinterpret_cast<uint2*>(out_bf16 + o) = make_uint2(*reinterpret_cast<const uint32_t*>(&b0), *reinterpret_cast<const uint32_t*>(&b1));
    } else {
      out_bf16[o] = __float2bfloat16(acc[0]);
    }
  }
}

template <typename TY, int V>
static void launch_combine(float* res, const void* y, const int* inv_perm, const float* wts, int R, int top_k, const void* shared, const float* sg,
                           int H, void* out, const int* pair_expert, cudaStream_t s) {
  const int per = 256 * V;
  const dim3 grid(R, (H + per - 1) / per);
  if constexpr (V <= 4) {
    if (top_k <= 4) {
      moe_combine_few_kernel<TY, V><<<grid, 256, 0, s>>>(res, (const TY*)y, inv_perm, wts, top_k, (const __nv_bfloat16*)shared, sg, H,
                                                         (__nv_bfloat16*)out, pair_expert);
      return;
    }
  }
  moe_combine_kernel<TY, V><<<grid, 256, 0, s>>>(res, (const TY*)y, inv_perm, wts, top_k, (const __nv_bfloat16*)shared, sg, H, (__nv_bfloat16*)out,
                                                 pair_expert);
}

}  // namespace spark

using namespace spark;

extern "C" int spark_moe_route(const float* logits, int ld, int R, int E, int top_k, int kind, const float* bias,
                               float scale, int shared_gate, float* wts, int* ids, int* pair_row, float* sg,
                               cudaStream_t s, int e_lo, int e_hi, int n_self, float* self_w) {
  if (R <= 0) return 0;
  if (E > ROUTE_MAXE || top_k > 32 || top_k > E || (kind == 3 && !bias)) return -5;
  auto kern = E <= 64 ? moe_route_kernel<2> : E <= 512 ? moe_route_kernel<16> : moe_route_kernel<32>;
  kern<<<(R + ROUTE_ROWS - 1) / ROUTE_ROWS, ROUTE_ROWS * 32, 0, s>>>(logits, ld, R, E, top_k, kind, bias, scale, shared_gate, wts, ids, pair_row, sg,
                                                                   e_lo, e_hi, n_self, self_w);
  return spark_launch_rc(__func__);
}

// Scratch `block_hist` must hold ceil(P/256) * E ints.
// tile_rows 128: tiles {row, end of the expert, expert, 0} of up to 128 rows; another number: even tiles {row, end, expert, rows} of up to that.
extern "C" int spark_moe_sort(const int* ids, int P, int E, int* perm, int* inv_perm, int* offsets, void* tile_list,
                              int* tile_count, int* block_hist, cudaStream_t s, int tile_rows) {
  if (P <= 0) return 0;
  if (E > 1024 || tile_rows < 16 || tile_rows > 192) return -5;                     // one thread per expert in the scan
  if (P <= SORT_ONE && E <= SORT_ONE) {
    const int n = ((P > E ? P : E) + 31) / 32 * 32;
    moe_sort_one_kernel<<<1, n, 0, s>>>(ids, P, E, perm, inv_perm, offsets, (int4*)tile_list, tile_count, tile_rows);
    return spark_launch_rc(__func__);
  }
  const int nb = (P + 255) / 256;
  moe_hist_kernel<<<nb, 256, E * sizeof(int), s>>>(ids, P, E, block_hist);
  moe_scan_kernel<<<1, 1024, 0, s>>>(block_hist, nb, E, offsets, (int4*)tile_list, tile_count, tile_rows);
  moe_place_kernel<<<nb, 256, 256 * sizeof(int), s>>>(ids, P, E, block_hist, offsets, perm, inv_perm);
  return spark_launch_rc(__func__);
}

extern "C" int spark_moe_combine(float* res, const void* y, int y_f32, const int* inv_perm, const float* wts, int R,
                                 int top_k, const void* shared, const float* sg, int H, void* out_bf16, cudaStream_t s,
                                 const int* pair_expert) {
  if (R <= 0) return 0;
  const bool wide = H % 8 == 0 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(out_bf16) | reinterpret_cast<uintptr_t>(shared)) & 15) == 0;
#define SPARK_CMB(T, V) launch_combine<T, V>(res, y, inv_perm, wts, R, top_k, shared, sg, H, out_bf16, pair_expert, s)
  if (y_f32) { if (wide) SPARK_CMB(float, 4); else SPARK_CMB(float, 1); }
  else { if (wide) SPARK_CMB(__nv_bfloat16, 8); else SPARK_CMB(__nv_bfloat16, 1); }
#undef SPARK_CMB
  return spark_launch_rc(__func__);
}

// Fused decode router: see moe_router_topk_kernel.  `logits` scratch [R, ld] fp32 (ld >= E + 1), `counter` one int
// that is zero between launches.  x bf16 [R, K].
extern "C" int spark_moe_router_topk(const void* x, int ldx, const void* Wg, int ldw, float* logits,
                                     int ld, int R, int K, int E, int top_k, int kind, const float* bias, float scale,
                                     int shared_gate, int slots, int shared_expert, int e_lo, int e_hi, int rank, int world,
                                     float* wts, int* ids, int* pair_row, float* sg, int* counter, int n_self, float* self_w,
                                     cudaStream_t s) {
  if (R <= 0) return 0;
  if (R > ROUTER_RB || E > 1024 || top_k > 32 || (K & 7) || slots < top_k || slots > top_k + 1 || ld < E + (shared_gate ? 1 : 0) ||
      top_k > E || (kind == 3 && !bias))
    return -5;
  RouterArgs a;
  a.n_self = n_self; a.self_w = self_w;
  a.x = (const __nv_bfloat16*)x; a.ldx = ldx;
  a.Wg = (const __nv_bfloat16*)Wg; a.ldw = ldw; a.logits = logits; a.ld = ld;
  a.R = R; a.K = K; a.E = E; a.top_k = top_k; a.kind = kind; a.bias = bias; a.scale = scale; a.shared_gate = shared_gate;
  a.slots = slots; a.shared_expert = shared_expert; a.e_lo = e_lo; a.e_hi = e_hi; a.rank = rank; a.world = world < 1 ? 1 : world;
  a.wts = wts; a.ids = ids; a.pair_row = pair_row; a.sg = sg; a.counter = counter;
  const int NE = E + (shared_gate ? 1 : 0);
  // experts per lane: the narrowest form that holds E (a lane's work per choice grows with it)
  auto pick = [&](auto rows, auto knd) {
    constexpr int NR = decltype(rows)::value, KD = decltype(knd)::value;
    return E <= 64 ? moe_router_topk_kernel<2, NR, KD> : E <= 256 ? moe_router_topk_kernel<8, NR, KD>
         : E <= 512 ? moe_router_topk_kernel<16, NR, KD> : moe_router_topk_kernel<32, NR, KD>;
  };
  auto of = [&](auto knd) {
    return R <= 4 ? pick(std::integral_constant<int, 1>{}, knd) : R <= 8 ? pick(std::integral_constant<int, 2>{}, knd)
                  : pick(std::integral_constant<int, 4>{}, knd);
  };
  void (*kern)(RouterArgs) = kind == 0 ? of(std::integral_constant<int, 0>{}) : kind == 1 ? of(std::integral_constant<int, 1>{})
                           : kind == 2 ? of(std::integral_constant<int, 2>{}) : kind == 3 ? of(std::integral_constant<int, 3>{})
                           : kind == 4 ? of(std::integral_constant<int, 4>{}) : of(std::integral_constant<int, 5>{});
  const cudaError_t err = spark_launch_pdl(kern, dim3((NE + ROUTER_COLS - 1) / ROUTER_COLS), dim3(ROUTER_WARPS * 32), 0, s, dim3(1, 1, 1), a);
  return err == cudaSuccess ? 0 : -4;
}

// res fp32 [R, H] (in/out), h bf16 [R, H] out; y fp32 [R * slots, H] in pair order.
extern "C" int spark_moe_combine_norm(const float* y, const float* wts, const int* ids, int R, int slots, int H, float* res,
                                      const float* norm_w, float eps, int one_plus, void* h, const void* shared,
                                      const float* sg, cudaStream_t s) {
  if (R <= 0) return 0;
  int th = H / 4;
  if (H % 128 || th > 2048) return -5;
  if (th > 1024) th = 1024;
  const cudaError_t err = spark_launch_pdl(moe_combine_norm_kernel, dim3(R), dim3(th), 0, s, dim3(1, 1, 1), y, wts, ids, slots, H,
                                           res, norm_w, eps, one_plus, (__nv_bfloat16*)h, (const __nv_bfloat16*)shared, sg);
  return err == cudaSuccess ? 0 : -4;
}
