// Causal GQA attention for prefill segments (bf16 KV cache): streaming softmax on tcgen05.  One CTA = 128 query rows of one q head,
// key/value tiles of 64 tokens.
//   warp 0      TMA: key and value tiles into a ring of four or six slots in the order the products use them (D = 64 / 128: the
//               query tile before them).  A ragged last tile is brought in as boxes of eight rows and plain copies of the rest;
//               its values past the last key are zeroed (a masked probability of 0 times whatever lies there would not be 0)
//   warp 1      issues S = Q K^T one tile ahead of O += P V (P in tensor memory, V as an N-major operand straight from its rows)
//   warps 2..5  softmax, one query row per thread: a row's 64 scores are one tensor-memory load, maximum and sum stay in the thread
//   all warps   the epilogue's gates and stores
// Every weight is taken against the running maximum, so that the heaviest of a row is exactly 1 in bf16 (a reference that lags behind
// the maximum would spare most of the rescaling, and rounds the heavy weights by up to 2^-8): the accumulator is rescaled in 32 bits
// at every tile where a row of the warp has a new maximum.
// The rows of a segment see the committed prefix of their sequence (already in the cache) plus the rows before them in the segment
// (stored by the prep kernel of the same step).  One CTA owns a (row tile, head) from first key to last, so results are run-to-run
// identical.  What bounds it: the softmax, whose exponentials and rescaling are the chain of one warp per scheduler, and L2, from
// which every tile brings 64 KB of keys and values to 128 rows (D = 256).  3999 rows of 16 heads (2 for keys), D = 256, block masks:
// 203 us, 645 TFLOP/s (64-row tiles on warp-level products: 828 us; weights up to 2^8 against a lagging reference, with approximate
// divisions: 165 us).  The rescaling behind the exponentials instead of before them: 20 us less; the epilogue's divisions, chains
// that only other warps hide, over eight warps instead of four: 40 us less.
// Serves: GQA / QSA layers (engine-rs/shim/qwen_qsa.cu attn paths; the reference runs prefill rows through the same per-row kernel
// as decode).
#include "../common/ptx.cuh"

namespace spark {

int make_tmap_bf16(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K, uint64_t ld, int box_rows, int fmt);

constexpr int PF_BM = 128, PF_BN = 64, PF_WARPS = 8, PF_THREADS = PF_WARPS * 32;

// D = 256: the queries are a tensor-memory operand (a product of 64 keys reads 2 KB of shared memory per step instead of 6: 74 -> 25
// cycles of issue each) and the ring has the room; 64 / 128: 256 columns hold everything with the queries in shared memory, and two
// CTAs share an SM
template <int D> struct Pf {
  static constexpr bool QT = D == 256;
  static constexpr int SLOTS = QT ? 6 : 4, SLOT = PF_BN * D * 2, Q_BYTES = QT ? 0 : PF_BM * D * 2;
  static constexpr int SMEM = Q_BYTES + SLOTS * SLOT + 256 + 1024;
  static constexpr int COLS = QT ? 512 : 256, S_COL = 0, P_COL = 64, O_COL = 128, Q_COL = 384;
};

struct PrefillArgs {
  const __nv_bfloat16 *q, *k, *v;                     // [R, Hq, D], [tokens, Hkv, D]
  const long long* row_kv; const int* seg;            // cache row of a sequence's first token per row; [nseg][4]
  const __nv_bfloat16* qkv; int ld, gated;            // gate columns
  __nv_bfloat16* out;
  int Hq, Hkv; float scale_log2;
  const uint32_t* bmask; int mw;                      // MASK: a bit per 4-token key block, mw words per row
  int* status;
};

__device__ __forceinline__ uint32_t pf_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// N-major operand, 128-byte swizzle: 64 n are a 128-byte row per k; chunks of 64 n `chunk` bytes apart, groups of 8 k 1024 bytes
__device__ __forceinline__ uint64_t pf_desc_nmajor(uint32_t addr, uint32_t chunk) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFF) >> 4);
  d |= static_cast<uint64_t>(chunk >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}

// grid (Hq, row tiles, segments)
template <int D, bool MASK>
__global__ void __launch_bounds__(PF_THREADS, D == 256 ? 1 : 2)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmK8,
                    const __grid_constant__ CUtensorMap tmV8, const __grid_constant__ PrefillArgs a) {
  using L = Pf<D>;
  constexpr int CH = D / 64, SLOT = L::SLOT, SLOTS = L::SLOTS, KV_CHUNK = PF_BN * 128, Q_CHUNK = PF_BM * 128;
  constexpr int COLS = L::COLS, O_COL = L::O_COL, LX = D + 1;           // LX: floats of a row in the epilogue
  const int sg = blockIdx.z, h = blockIdx.x;
  const int qt = gridDim.y - 1 - blockIdx.y;                 // longest row tiles (most key tiles) are scheduled first
  const int r0 = a.seg[sg * 4 + 1], n = a.seg[sg * 4 + 2], pos0 = a.seg[sg * 4 + 3];
  if (qt * PF_BM >= n) return;
  const int rows_valid = min(PF_BM, n - qt * PF_BM);
  const int nkeys = pos0 + qt * PF_BM + rows_valid;           // keys visible to the last valid row of the tile
  const int ntiles = (nkeys + PF_BN - 1) / PF_BN;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ring = smem + L::Q_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + SLOTS * SLOT);
  uint64_t* empty = full + SLOTS;
  uint64_t* q_full = empty + SLOTS;
  uint64_t* s_full = q_full + 1;
  uint64_t* s_read = s_full + 1;
  uint64_t* p_full = s_read + 1;
  uint64_t* o_full = p_full + 2;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(o_full + 2);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    if (!L::QT) tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
    for (int s = 0; s < SLOTS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(q_full, L::QT ? 4 : 1); mbar_init(s_full, 1); mbar_init(s_read, 4);
    for (int s = 0; s < 2; ++s) { mbar_init(&p_full[s], 4); mbar_init(&o_full[s], 1); }
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc<COLS>(tmem_ptr); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;

  bool ok = true;
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    const int hk = h / (a.Hq / a.Hkv);
    const int base = static_cast<int>(a.row_kv[r0]);
    int slot = 0; uint32_t ph = 0;
    if (!L::QT && lane == 0) {
      mbar_arrive_expect_tx(q_full, PF_BM * D * 2);
      for (int c = 0; c < CH; ++c) tma_load_2d(smem + c * Q_CHUNK, &tmQ, q_full, h * D + c * 64, r0 + qt * PF_BM);
    }
    const int keep = nkeys - (ntiles - 1) * PF_BN, keep8 = keep & ~7;      // keys of the last tile, in groups of 8
    for (int i = 0; i < 2 * ntiles; ++i) {                    // K0 K1 V0 K2 V1 .. K(n-1) V(n-2) V(n-1)
      const bool is_v = i == 2 * ntiles - 1 || (i >= 2 && !(i & 1));
      const int j = i == 0 ? 0 : i == 2 * ntiles - 1 ? ntiles - 1 : is_v ? i / 2 - 1 : (i + 1) / 2;
      ok = __all_sync(0xffffffffu, mbar_wait(&empty[slot], ph ^ 1));
      if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_EMPTY, blockIdx.x, blockIdx.y, i); break; }
      uint8_t* dst = ring + slot * SLOT;
      if (j < ntiles - 1 || keep == PF_BN) {
        if (lane == 0) {
          mbar_arrive_expect_tx(&full[slot], SLOT);
          for (int c = 0; c < CH; ++c) tma_load_2d(dst + c * KV_CHUNK, is_v ? &tmV : &tmK, &full[slot], hk * D + c * 64, base + j * PF_BN);
        }
      } else {
        // rows keep8 .. keep as plain copies in the swizzle's order, value rows from keep on zero; unread key rows stay as they are
        const __nv_bfloat16* src = is_v ? a.v : a.k;
        const int per = ((is_v ? PF_BN : keep) - keep8) * 8;   // 16-byte units of a chunk
        for (int u = lane; u < CH * per; u += 32) {
          const int c = u / per, row = keep8 + (u - c * per) / 8, x = u & 7;
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (row < keep) v = __ldg(reinterpret_cast<const uint4*>(src + (static_cast<size_t>(base + j * PF_BN + row) * a.Hkv + hk) * D + c * 64) + x);
          *reinterpret_cast<uint4*>(dst + c * KV_CHUNK + row * 128 + ((x ^ (row & 7)) * 16)) = v;
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (keep8 == 0) mbar_arrive(&full[slot]);
          else mbar_arrive_expect_tx(&full[slot], CH * keep8 * 128);
          for (int c = 0; c < CH; ++c)
            for (int r = 0; r < keep8; r += 8)
              tma_load_2d(dst + c * KV_CHUNK + r * 128, is_v ? &tmV8 : &tmK8, &full[slot], hk * D + c * 64, base + j * PF_BN + r);
        }
      }
      __syncwarp();
      if (++slot == SLOTS) { slot = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // (the whole warp walks the loop and one elected lane issues: descriptors stay in uniform registers, where the instructions want
    // them: 48 us less for 4000 rows of 16 heads of 256)
    const uint32_t id_s = make_idesc(1, 1, PF_BM, PF_BN), id_o = make_idesc(1, 1, PF_BM, D) | (1u << 16);
    const uint32_t qs = __shfl_sync(0xffffffffu, smem_u32(smem), 0), rs = qs + L::Q_BYTES, tm = __shfl_sync(0xffffffffu, tmem, 0);
    int slot = 0; uint32_t ph = 0;
    ok = __all_sync(0xffffffffu, mbar_wait(q_full, 0));
    if (!ok) set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, -2);
    for (int j = -1; j < ntiles && ok; ++j) {
      if (j + 1 < ntiles) {
        // the scores have one buffer, free as soon as every warp has loaded those of tile j
        ok = __all_sync(0xffffffffu, mbar_wait(&full[slot], ph) && (j < 0 || mbar_wait(s_read, j & 1)));
        if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, j); break; }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            const uint64_t kd = make_smem_desc_sw128(rs + slot * SLOT + c * KV_CHUNK);
            if (L::QT) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16_ts(tm + L::S_COL, tm + L::Q_COL + c * 32 + k * 8, kd + 2 * k, id_s, (c | k) != 0);
            } else {
              const uint64_t qd = make_smem_desc_sw128(qs + c * Q_CHUNK);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16(tm + L::S_COL, qd + 2 * k, kd + 2 * k, id_s, (c | k) != 0);
            }
          }
          umma_commit(&empty[slot]);
          umma_commit(s_full);
        }
        __syncwarp();
        if (++slot == SLOTS) { slot = 0; ph ^= 1; }
      }
      if (j < 0) continue;
      ok = __all_sync(0xffffffffu, mbar_wait(&full[slot], ph) && mbar_wait(&p_full[j & 1], (j >> 1) & 1));
      if (!ok) { set_status(a.status, ST_TIMEOUT_MBAR_FULL, blockIdx.x, blockIdx.y, j); break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t p = tm + L::P_COL + (j & 1) * 32;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_f16_ts(tm + O_COL, p + k * 8, pf_desc_nmajor(rs + slot * SLOT + k * 2048, KV_CHUNK), id_o, (j | k) != 0);
        umma_commit(&empty[slot]);
        umma_commit(&o_full[j & 1]);
      }
      __syncwarp();
      if (++slot == SLOTS) { slot = 0; ph ^= 1; }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------ softmax, one query row per thread
    const int q = warp & 3, row = q * 32 + lane;
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(q * 32) << 16);
    const int pos = pos0 + qt * PF_BM + min(row, rows_valid - 1);          // padded rows: the last valid row's mask
    const uint32_t* bm = MASK ? a.bmask + static_cast<size_t>(r0 + pos - pos0) * a.mw : nullptr;
    if (L::QT) {                                               // this thread's query: column c holds dimensions 2 c and 2 c + 1
      const uint4* qp = reinterpret_cast<const uint4*>(a.q + (static_cast<size_t>(r0 + qt * PF_BM + min(row, rows_valid - 1)) * a.Hq + h) * D);
#pragma unroll
      for (int c = 0; c < D / 2; c += 32) {
        uint32_t w[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 v = __ldg(qp + c / 4 + i);
          w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
        tmem_st_32x32(t_lane + L::Q_COL + c, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    // the gates are wanted at the end: from DRAM they took longer than the rest of the epilogue, so they are asked into L2 now
    if (a.gated && row < rows_valid) {
      const __nv_bfloat16* gp = a.qkv + static_cast<size_t>(r0 + qt * PF_BM + row) * a.ld + h * 2 * D + D;
#pragma unroll
      for (int c = 0; c < D; c += 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(gp + c));
    }
    float m = -INFINITY, l = 0.f;
    uint32_t word = MASK ? __ldg(bm) : 0u;
    for (int j = 0; j < ntiles; ++j) {
      uint32_t next = 0u;
      if (MASK && (j & 1) && j + 1 < ntiles) next = __ldg(bm + ((j + 1) >> 1));
      ok = __all_sync(0xffffffffu, mbar_wait(s_full, j & 1));
      if (!ok) { set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, j); break; }
      tc_fence_after();
      uint32_t raw[2][32];
      tmem_ld_32x32(t_lane + L::S_COL, raw[0]);
      tmem_ld_32x32(t_lane + L::S_COL + 32, raw[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_read);
      float s[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) s[i] = __uint_as_float(raw[i >> 5][i & 31]);
      const int k0 = j * PF_BN;
      if (MASK) {
        const uint32_t sel = word >> ((j & 1) * 16);           // 16 block bits of this tile (a word covers two tiles)
#pragma unroll
        for (int b = 0; b < 16; ++b) {
          const bool on = (sel >> b) & 1u;
#pragma unroll
          for (int e = 0; e < 4; ++e) s[b * 4 + e] = on ? s[b * 4 + e] : -INFINITY;
        }
        if (j & 1) word = next;
      }
      if (k0 + PF_BN - 1 > pos0 + qt * PF_BM) {                // a tile on the diagonal, or past the last key
        const int seen = pos - k0;
#pragma unroll
        for (int i = 0; i < 64; ++i) s[i] = i <= seen ? s[i] : -INFINITY;
      }
      float mx[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = s[i];
#pragma unroll
      for (int i = 8; i < 64; ++i) mx[i & 7] = fmaxf(mx[i & 7], s[i]);
      const float top = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7]))) * a.scale_log2;
      const bool grow = top > m;                               // m = -inf: this row has seen no key yet
      const bool rescale = j > 0 && __any_sync(0xffffffffu, grow);
      const float c = grow ? exp2f(m - top) : 1.f;
      if (grow) { m = top; l *= c; }
      const float ref = m == -INFINITY ? 0.f : m;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t p[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float e0 = exp2f(fmaf(s[2 * i], a.scale_log2, -ref)), e1 = exp2f(fmaf(s[2 * i + 1], a.scale_log2, -ref));
        sum[i & 1] += e0; sum[2 + (i & 1)] += e1;
        p[i] = pf_pack(e0, e1);
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      // P's buffer: the product of two tiles back has read it
      if (j >= 2) {
        ok = __all_sync(0xffffffffu, mbar_wait(&o_full[j & 1], ((j - 2) >> 1) & 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, j); break; }
      }
      tmem_st_32x32(t_lane + L::P_COL + (j & 1) * 32, p);
      if (rescale) {                                           // behind the exponentials: the product before has finished by now
        ok = __all_sync(0xffffffffu, mbar_wait(&o_full[(j - 1) & 1], ((j - 1) >> 1) & 1));
        if (!ok) { set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, j); break; }
        tc_fence_after();
#pragma unroll 1
        for (int cc = 0; cc < D; cc += 64) {
          uint32_t o[2][32];
          tmem_ld_32x32(t_lane + O_COL + cc, o[0]);
          tmem_ld_32x32(t_lane + O_COL + cc + 32, o[1]);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            o[0][i] = __float_as_uint(__uint_as_float(o[0][i]) * c);
            o[1][i] = __float_as_uint(__uint_as_float(o[1][i]) * c);
          }
          tmem_st_32x32(t_lane + O_COL + cc, o[0]);
          tmem_st_32x32(t_lane + O_COL + cc + 32, o[1]);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j & 1]);
    }
    // ---- epilogue: normalise, through shared memory (queries, keys and values are used up), so that a row's columns are read and
    // written together
    if (ok) {
      ok = __all_sync(0xffffffffu, mbar_wait(&o_full[(ntiles - 1) & 1], ((ntiles - 1) >> 1) & 1));
      if (!ok) set_status(a.status, ST_TIMEOUT_TMEM_FULL, blockIdx.x, blockIdx.y, ntiles);
    }
    if (ok) {
      tc_fence_after();
      float* x = reinterpret_cast<float*>(smem) + row * LX;
      const float inv = 1.f / l;
#pragma unroll 1
      for (int cc = 0; cc < D; cc += 32) {
        uint32_t o[32];
        tmem_ld_32x32(t_lane + O_COL + cc, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) x[cc + i] = __uint_as_float(o[i]) * inv;
      }
    }
  }
  tc_fence_before();
  if (__syncthreads_and(ok)) {
    // ---- gate, store: eight rows of all eight warps at a time (a division is a chain of its own, which only other warps hide), the
    // gates of a group asked for before the first is used
    constexpr int CW = D / 64;                                 // 64-column pieces of a row: a lane has columns 2 lane, 2 lane + 1 of each
    const float* x = reinterpret_cast<const float*>(smem);
    const size_t rw = static_cast<size_t>(r0 + qt * PF_BM);
#pragma unroll 1
    for (int i0 = warp * 8; i0 < rows_valid; i0 += PF_WARPS * 8) {
      uint32_t gate[8][CW];
      if (a.gated) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const __nv_bfloat16* gp = a.qkv + (rw + min(i0 + i, rows_valid - 1)) * a.ld + h * 2 * D + D + 2 * lane;
#pragma unroll
          for (int c = 0; c < CW; ++c) gate[i][c] = __ldg(reinterpret_cast<const uint32_t*>(gp + c * 64));
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (i0 + i >= rows_valid) break;
        __nv_bfloat16* dst = a.out + ((rw + i0 + i) * a.Hq + h) * D + 2 * lane;
#pragma unroll
        for (int c = 0; c < CW; ++c) {
          float v0 = x[(i0 + i) * LX + c * 64 + 2 * lane], v1 = x[(i0 + i) * LX + c * 64 + 2 * lane + 1];
          if (a.gated) {
            const float2 gt = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gate[i][c]));
            v0 = v0 / (1.f + __expf(-gt.x)); v1 = v1 / (1.f + __expf(-gt.y));
          }
          *reinterpret_cast<uint32_t*>(dst + c * 64) = pf_pack(v0, v1);
        }
      }
    }
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc<COLS>(tmem); }
}

template <int D, bool MASK>
static int launch_prefill(int R, long long tokens, int nseg, int max_rows, const PrefillArgs& a, cudaStream_t s) {
  CUtensorMap tq, tk, tv, tk8, tv8;
  const uint64_t wq = static_cast<uint64_t>(a.Hq) * D, wk = static_cast<uint64_t>(a.Hkv) * D;
  if (int r = make_tmap_bf16(&tq, a.q, R, wq, wq, PF_BM, 1)) return r;
  if (int r = make_tmap_bf16(&tk, a.k, tokens, wk, wk, PF_BN, 1)) return r;
  if (int r = make_tmap_bf16(&tv, a.v, tokens, wk, wk, PF_BN, 1)) return r;
  if (int r = make_tmap_bf16(&tk8, a.k, tokens, wk, wk, 8, 1)) return r;
  if (int r = make_tmap_bf16(&tv8, a.v, tokens, wk, wk, 8, 1)) return r;
  auto kern = attn_prefill_kernel<D, MASK>;
  static bool done = false;
  if (!done) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Pf<D>::SMEM); done = true; }
  kern<<<dim3(a.Hq, (max_rows + PF_BM - 1) / PF_BM, nseg), PF_THREADS, Pf<D>::SMEM, s>>>(tq, tk, tv, tk8, tv8, a);
  return spark_launch_rc(__func__);
}

// grid R, 256 threads: the row's selected token list -> one bit per 4-token block (the always-visible tail is part of
// the list, so its blocks are set as well; keys past the row's position are cut by the causal test).
__global__ void __launch_bounds__(256)
sel_blockmask_kernel(const int* __restrict__ sel, const int* __restrict__ sel_n, int sel_ld, uint32_t* __restrict__ bmask,
                     int mw) {
  extern __shared__ uint32_t bits[];
  const int r = blockIdx.x;
  for (int i = threadIdx.x; i < mw; i += blockDim.x) bits[i] = 0u;
  __syncthreads();
  const int n = sel_n[r];
  const int* row = sel + static_cast<size_t>(r) * sel_ld;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int b = row[i] >> 2;
    if ((b >> 5) < mw) atomicOr(&bits[b >> 5], 1u << (b & 31));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < mw; i += blockDim.x) bmask[static_cast<size_t>(r) * mw + i] = bits[i];
}

}  // namespace spark

using namespace spark;

template <bool MASK>
static int prefill(int R, long long tokens, int nseg, int max_rows, int D, const PrefillArgs& a, cudaStream_t s) {
  if (tokens <= 0 || tokens > 0x7fffffffLL || a.Hkv <= 0 || a.Hq % a.Hkv || (a.gated && (a.ld & 1))) return -5;
  if (D == 256) return launch_prefill<256, MASK>(R, tokens, nseg, max_rows, a, s);
  if (D == 128) return launch_prefill<128, MASK>(R, tokens, nseg, max_rows, a, s);
  if (D == 64) return launch_prefill<64, MASK>(R, tokens, nseg, max_rows, a, s);
  return -5;
}

// Dense causal attention over bf16 caches for whole segments.  seg: int [nseg][4] = slot, first row, rows, first position; R: rows of
// qbuf; max_rows = longest segment; tokens: rows of the caches.  No row past the last key of a segment is read (a cache that grows
// on demand may not have it), and none of the bounds is the host's: seg and row_kv may change between replays of a captured launch.
// head_dim 64, 128 or 256.
extern "C" int spark_attn_prefill(const void* qbuf, const void* kc, const void* vc, const long long* row_kv, const int* seg,
                                  int nseg, int max_rows, const void* qkv, int ld, int gated, void* out, int Hq, int Hkv,
                                  int D, float scale, int R, long long tokens, int* status, cudaStream_t s) {
  if (nseg <= 0 || max_rows <= 0 || R <= 0) return 0;
  const PrefillArgs a{(const __nv_bfloat16*)qbuf, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, row_kv, seg, (const __nv_bfloat16*)qkv, ld, gated, (__nv_bfloat16*)out, Hq, Hkv, scale * 1.4426950408889634f,
                      nullptr, 0, status};
  return prefill<false>(R, tokens, nseg, max_rows, D, a, s);
}

// The same tiles for rows with a block-sparse selection (4-token blocks): bmask [R, mw] has a bit per block (mw >= ceil(max context / 128)),
// as spark_topk_mask leaves it; with sel / sel_n (per-row token lists, plan order) it is scratch and made from them.
extern "C" int spark_attn_prefill_masked(const void* qbuf, const void* kc, const void* vc, const long long* row_kv,
                                         const int* seg, int nseg, int max_rows, const void* qkv, int ld, int gated, void* out,
                                         int Hq, int Hkv, int D, float scale, const int* sel, const int* sel_n, int sel_ld,
                                         int R, unsigned* bmask, int mw, long long tokens, int* status, cudaStream_t s) {
  if (nseg <= 0 || max_rows <= 0 || R <= 0) return 0;
  if (mw <= 0 || mw > 8192 || (sel && !sel_n) || !bmask) return -5;
  if (sel) sel_blockmask_kernel<<<R, 256, mw * 4, s>>>(sel, sel_n, sel_ld, bmask, mw);
  const PrefillArgs a{(const __nv_bfloat16*)qbuf, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, row_kv, seg, (const __nv_bfloat16*)qkv, ld, gated, (__nv_bfloat16*)out, Hq, Hkv, scale * 1.4426950408889634f,
                      bmask, mw, status};
  return prefill<true>(R, tokens, nseg, max_rows, D, a, s);
}
