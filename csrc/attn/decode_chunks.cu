// Decode attention in context chunks on the tensor cores: few sequences, all query heads of a KV head at once.
//
// The work is the list of live chunks (`chunk` tokens of one sequence) times KV heads, dealt out in turn to persistent CTAs; lengths are
// read on the device, so the launch fits a CUDA graph whatever they become.  A CTA streams tiles of 64 tokens of K and V (2-D TMA boxes
// of 64 rows x 64 dims with the 128-byte swizzle, a ring of two stages that never drains across items) and its four consumer warps take
// 16 tokens of each tile: S = Q K^T and O += P V as mma.sync m16n8k16 with fp32 sums.  The heads of the group fill rows 0..7 of the
// query tile.  The weights keep all 24 bits of their mantissa: P = hi + mid + lo, three bf16 numbers of 8 bits each, cut off and not rounded, so
// that none is negative and their sum is P exactly.  hi fills rows 0..7 of the second product and mid rows 8..15, which would be empty.  With
// four heads lo has rows 4..7, whose queries are those of rows 0..3 once more; with more it takes a product of its own.  A sequence of one chunk is
// finished here, others leave partials for the merge kernel.
//
// What bounds it is latency (length -> block table -> keys -> scores -> sums), and from about ten sequences the stream of the cache: three
// CTAs per SM (two for groups of more than four, whose third part of the weights takes registers) with 64 KB on their way each.  The dot products
// on the CUDA cores, which this replaces for cache blocks of 64 tokens and more, took longer than the stream: a tile of 64 tokens of four heads needs
// 64 K multiply-adds and 2500 shuffles in a warp.
// Measured with the merge (CUDA cores -> here), 32 / 8 heads: 1 x 3001 tokens 18.6 -> 11.1 us, 13 x 200 .. 2000 34.5 -> 26.8; 64 / 8 heads: 23.1 -> 11.4,
// 58 -> 33.9.  Error of the fp32 partials against 64 bits (CUDA cores -> here): 3001 tokens 8.2e-8 -> 6.3e-8, values without a common direction
// 2.1e-7 -> 1.4e-7, chunks of 1536 tokens 3.8e-7 -> 1.7e-7; of the bf16 result 1.67e-3 both.
#include <algorithm>

#include "../include/decode_common.cuh"
#include "../include/launch.cuh"
#include "../include/mma_sync.cuh"
#include "../include/ptx.cuh"

namespace forge {

constexpr int kCkStages = 2;
__host__ __device__ constexpr int ck_ctas_per_sm(int G) { return G > 4 ? 2 : 3; }

// The parts of a weight: the upper 16 bits of p, of what is left, and of what is left then (at most 8 bits: exact).
__device__ __forceinline__ float ck_upper(float p) { return __uint_as_float(__float_as_uint(p) & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t ck_pack_upper(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }

struct ChunkItem {
  int b, c, kvh, len, chunk;
};

__device__ __forceinline__ int chunk_checked_len(const int* __restrict__ lens, int b, int cap, unsigned* status) {
  int len = lens[b];
  if (len > cap) {                                       // a corrupted length: clamped and reported
    set_status(status, kStatusBadIndex);
    len = cap;
  }
  return max(len, 0);
}

// Item `item`; executed by whole warps.  Direct: of the list [chunk][sequence][KV head] with `most` chunks for every sequence, dead ones have
// c * chunk >= len.  Else of the list [live chunk][KV head].  False: there are not that many.
__device__ __forceinline__ bool chunk_item(const int* __restrict__ lens, int B, int nkv, const DecodeSplit& split, int cap, bool direct, int item,
                                           unsigned* status, ChunkItem& it) {
  const int lane = threadIdx.x & 31;
  int left = item / nkv;
  it.kvh = item - left * nkv;
  if (direct) {
    it.c = left / B;
    it.b = left - it.c * B;
    if (it.c >= split.most) return false;
    it.len = chunk_checked_len(lens, it.b, cap, status);
    it.chunk = decode_chunk_tokens(it.len, split);
    return true;
  }
  for (int b0 = 0; b0 < B; b0 += 32) {
    const int len = b0 + lane < B ? chunk_checked_len(lens, b0 + lane, cap, status) : 0;
    const int chunk = decode_chunk_tokens(len, split), n = (len + chunk - 1) / chunk;
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += u;
    }
    const uint32_t above = __ballot_sync(0xffffffffu, left < sum);
    if (above != 0) {
      const int l = __ffs(above) - 1;
      it.b = b0 + l;
      it.len = __shfl_sync(0xffffffffu, len, l);
      it.chunk = __shfl_sync(0xffffffffu, chunk, l);
      it.c = left - __shfl_sync(0xffffffffu, sum - n, l);
      return true;
    }
    left -= __shfl_sync(0xffffffffu, sum, 31);
  }
  return false;
}

// Sums of a warp that came out as NaN, once more with whole weights, one after the other.  An infinite value under a positive weight is an
// infinite sum, but a part of the weight can be zero, and zero times infinity is not a number; what is NaN here too stays one.  q_rows: the
// heads' queries (shared or global memory); o, m: the warp's sums and maxima.  Executed by a whole warp, rarely, hence not inlined.
__device__ __noinline__ void ck_repair_sums(float* o, const float* m, int heads, const __nv_bfloat16* q_rows, const __nv_bfloat16* k_cache,
                                            const __nv_bfloat16* v_cache, const int* table, int begin, int end, int kvh, int nkv, int block_size,
                                            int num_blocks, float scale_log2, int lane) {
  for (int g = 0; g < heads; ++g) {
    float q[4], sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < 4; ++e) q[e] = __bfloat162float(q_rows[g * kD + 4 * lane + e]);
    const float m_use = m[g] == -INFINITY ? 0.f : m[g];
    for (int tok0 = begin; tok0 < end; tok0 += kTcTile)
      for (int tok = tok0; tok < min(tok0 + 16, end); ++tok) {
        const int blk = table[tok / block_size];
        const size_t off = ((static_cast<size_t>(blk >= 0 && blk < num_blocks ? blk : 0) * nkv + kvh) * block_size + tok % block_size) * kD + 4 * lane;
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) d = fmaf(q[e], __bfloat162float(k_cache[off + e]), d);
#pragma unroll
        for (int i = 16; i > 0; i >>= 1) d += __shfl_xor_sync(0xffffffffu, d, i);
        const float p = exp2f(d * scale_log2 - m_use);
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] = fmaf(p, __bfloat162float(v_cache[off + e]), sum[e]);
      }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (isnan(o[g * kD + 4 * lane + e])) o[g * kD + 4 * lane + e] = sum[e];
  }
}

template <int G>
__global__ void __launch_bounds__(kDecThreads, ck_ctas_per_sm(G)) decode_attn_chunk_kernel(
    const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __nv_bfloat16* __restrict__ q,
    __nv_bfloat16* k_cache, __nv_bfloat16* v_cache, const int* __restrict__ block_tables, const int* __restrict__ context_lens,
    __nv_bfloat16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml, int B, int nq, int nkv, int block_size,
    int table_width, int num_blocks, const DecodeSplit split, int max_chunks, int direct, float scale_log2, unsigned* status, const DecodeFuse fuse) {
  static_assert(G <= 8, "the heads of a group fill the first eight rows of the query tile");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_acc = reinterpret_cast<float*>(smem + kCkStages * 2 * kTcTileBytes);          // merge area
  __nv_bfloat16* s_q = reinterpret_cast<__nv_bfloat16*>(s_acc + decode_merge_floats(G)); // [G][128]
  uint4* s_new = reinterpret_cast<uint4*>(s_q + G * kD); // the newest token: 16 pieces of its key, 16 of its value
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(s_new + 32);
  uint64_t* empty_bar = full_bar + kCkStages;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cap = min(table_width * block_size, max_chunks * split.unit);
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    for (int s = 0; s < kCkStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 4);
    }
    fence_mbar_init();
  }
  __syncthreads();
  pdl_wait();                                           // q, the cache and the step buffer come from predecessors

  ChunkItem it;
  if (warp == 4) {
    // ------------------------------------------------------------------ producer
    int n = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && chunk_item(context_lens, B, nkv, split, cap, direct != 0, item, status, it); item += gridDim.x) {
      if (lane == 0) {
        const int end = min(it.len, (it.c + 1) * it.chunk);
        for (int tok = it.c * it.chunk; tok < end; tok += kTcTile, ++n) {
          const int s = n % kCkStages;
          int blk = block_tables[static_cast<size_t>(it.b) * table_width + tok / block_size];
          if (blk < 0 || blk >= num_blocks) {
            set_status(status, kStatusBadIndex);
            blk = 0;
          }
          const int row = (blk * nkv + it.kvh) * block_size + tok % block_size;
          ok = mbar_wait(&empty_bar[s], ((n / kCkStages) & 1) ^ 1, status);
          if (!ok) break;
          uint8_t* stg = smem + s * 2 * kTcTileBytes;
          mbar_expect_tx(&full_bar[s], 2 * kTcTileBytes);
          tma_load_2d(stg, &tm_k, &full_bar[s], 0, row);
          tma_load_2d(stg + kTcBoxBytes, &tm_k, &full_bar[s], 64, row);
          tma_load_2d(stg + kTcTileBytes, &tm_v, &full_bar[s], 0, row);
          tma_load_2d(stg + kTcTileBytes + kTcBoxBytes, &tm_v, &full_bar[s], 64, row);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
    }
    return;
  }

  // -------------------------------------------------------------------- consumers (warps 0..3): 16 tokens of every tile each
  for (int b = blockIdx.x; b < B; b += gridDim.x)       // padding rows (length 0): defined output
    if (context_lens[b] <= 0)
      for (int i = threadIdx.x; i < nq * kD; i += 128) out[static_cast<size_t>(b) * nq * kD + i] = __float2bfloat16_rn(0.f);
  constexpr bool kLoInRows = G <= 4;                    // rows 4..7 are free for the third part of the weights
  const int row = lane >> 2, quad = lane & 3;           // fragment coordinates: row of the query tile, column pair
  const int head = kLoInRows ? row & 3 : row;           // head of the group
  const bool lo_row = kLoInRows && row >= 4;
  const int mat = lane >> 3, mrow = lane & 7;           // ldmatrix: this lane supplies row `mrow` of matrix `mat`
  int n = 0;
  bool ok = true;                                       // once a wait has run out none is made any more, but every barrier still is
  for (int item = blockIdx.x; chunk_item(context_lens, B, nkv, split, cap, direct != 0, item, nullptr, it); item += gridDim.x) {
    const int qh0 = it.kvh * G, begin = it.c * it.chunk, end = min(it.len, begin + it.chunk);
    if (begin >= end) continue;                         // uniform for the consumers
    // the newest token (position len - 1) is not in the cache yet: the warp that owns its row of its tile prepares it now
    const int newest = it.len - 1, row_new = newest % kTcTile;
    const bool owner = fuse.qkv != nullptr && newest >= begin && newest < end && warp == row_new / 16;
    uint32_t qa[8][2];                                  // rows 0..G-1 = the heads of the group, the others zero (G = 4: again the heads); 8 steps of 16 dims
    if (fuse.qkv != nullptr) {
      const float* cs = fuse.rope != nullptr ? fuse.rope + static_cast<size_t>(min(max(newest, 0), fuse.rope_rows - 1)) * kD : nullptr;
      for (int g = warp; g < G; g += 4) {
        float x[16];
        decode_norm_rope_head(fuse.qkv + static_cast<size_t>(it.b) * fuse.ld_qkv + static_cast<size_t>(qh0 + g) * kD, fuse.q_w, fuse.eps, cs, lane, x);
        if (lane < 8) {
          *reinterpret_cast<uint4*>(s_q + g * kD + 8 * lane) =
              make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
          *reinterpret_cast<uint4*>(s_q + g * kD + 64 + 8 * lane) =
              make_uint4(pack_bf16x2(x[8], x[9]), pack_bf16x2(x[10], x[11]), pack_bf16x2(x[12], x[13]), pack_bf16x2(x[14], x[15]));
        }
      }
      if (owner) {                                      // kept in shared memory: ten registers less across the loop
        const DecodeNewToken fresh = decode_new_token(fuse, it.b, it.kvh, nq, nkv, it.len, lane);
        if (lane < 8) {
          s_new[lane] = fresh.k_lo;
          s_new[8 + lane] = fresh.k_hi;
        }
        reinterpret_cast<uint2*>(s_new + 16)[lane] = fresh.v;
      }
      named_barrier_sync(1, 128);
    }
    {
      const __nv_bfloat16* qp = (fuse.qkv != nullptr ? s_q : q + (static_cast<size_t>(it.b) * nq + qh0) * kD) + head * kD + 2 * quad;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        qa[kk][0] = head < G ? *reinterpret_cast<const uint32_t*>(qp + kk * 16) : 0u;
        qa[kk][1] = head < G ? *reinterpret_cast<const uint32_t*>(qp + kk * 16 + 8) : 0u;
      }
    }
    float m_run = -INFINITY, l_run = 0.f;               // of `head`; l is this lane's share until the end
    float o[16][4];                                     // [..][0, 1]: sums of hi V (lo_row: of lo V), [2, 3]: of mid V (and of lo V), same head and dims
#pragma unroll
    for (int nb = 0; nb < 16; ++nb) o[nb][0] = o[nb][1] = o[nb][2] = o[nb][3] = 0.f;
    for (int tok0 = begin; tok0 < end; tok0 += kTcTile, ++n) {
      const int s = n % kCkStages;
      ok = ok && mbar_wait(&full_bar[s], (n / kCkStages) & 1, status);
      uint8_t* stg = smem + s * 2 * kTcTileBytes;
      const uint32_t Ks = smem_u32(stg), Vs = Ks + kTcTileBytes;
      if (owner && newest - tok0 < kTcTile) {           // its tile: the row is put in place, and into the cache for later steps
        int blk = block_tables[static_cast<size_t>(it.b) * table_width + newest / block_size];
        const bool to_cache = blk >= 0 && blk < num_blocks;
        if (!to_cache) blk = 0;
        const size_t off = ((static_cast<size_t>(blk) * nkv + it.kvh) * block_size + newest % block_size) * kD;
        const uint4 piece = s_new[lane];
        *reinterpret_cast<uint4*>(stg + (tc_tile_addr(lane < 16 ? Ks : Vs, row_new, lane & 15) - Ks)) = piece;
        if (to_cache) *reinterpret_cast<uint4*>((lane < 16 ? k_cache : v_cache) + off + 8 * (lane & 15)) = piece;
        fence_proxy_async_smem();                       // a later copy into this stage comes after these writes
        __syncwarp();
      }
      const int r0 = warp * 16;
      // A product from zero for every 16 dims, added up here, pairs first: a sum that is carried on from product to product is cut off and not
      // rounded at each of them.
      float sc[2][2], part[2][3][2];                    // part: sums of one, two and four products
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t kb[4];
        ldsm_x4(tc_tile_addr(Ks, r0 + (mat >> 1) * 8 + mrow, 2 * kk + (mat & 1)), kb);
        const uint32_t a[4] = {qa[kk][0], 0u, qa[kk][1], 0u};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816(c, a, kb[2 * j], kb[2 * j + 1]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float sum = c[e];
            if (kk % 2 == 1) sum = part[j][0][e] + sum;
            if (kk % 4 == 3) sum = part[j][1][e] + sum;
            if (kk == 7) sc[j][e] = part[j][2][e] + sum;
            else part[j][kk % 2 == 0 ? 0 : kk % 4 == 1 ? 1 : 2][e] = sum;
          }
        }
      }
      // this lane: `head`, tokens r0 + j * 8 + 2 * quad + {0, 1} of the tile
      const int valid = end - tok0;
      float mt = -INFINITY;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (r0 + j * 8 + 2 * quad + e < valid) mt = fmaxf(mt, sc[j][e] * scale_log2);
      mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 1));
      mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, 2));
      const float m_new = fmaxf(m_run, mt);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = exp2f(m_run - m_use);
      float p[2][2], mid[2][2], lo[2][2];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          p[j][e] = r0 + j * 8 + 2 * quad + e < valid ? exp2f(fmaf(sc[j][e], scale_log2, -m_use)) : 0.f;
          mid[j][e] = p[j][e] - ck_upper(p[j][e]);
          lo[j][e] = mid[j][e] - ck_upper(mid[j][e]);
        }
      l_run = fmaf(l_run, alpha, (p[0][0] + p[0][1]) + (p[1][0] + p[1][1]));
      m_run = m_new;
      uint32_t pa[4], pl[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        pa[2 * j] = ck_pack_upper(p[j][0], p[j][1]);
        pa[2 * j + 1] = ck_pack_upper(mid[j][0], mid[j][1]);
        pl[j] = ck_pack_upper(lo[j][0], lo[j][1]);
        if (lo_row) {
          pa[2 * j] = pl[j];
          pa[2 * j + 1] = 0u;
        }
      }
#pragma unroll
      for (int dd = 0; dd < 8; ++dd) {
        uint32_t vb[4];
        ldsm_x4_trans(tc_tile_addr(Vs, r0 + (mat & 1) * 8 + mrow, 2 * dd + (mat >> 1)), vb);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816(c, pa, vb[2 * j], vb[2 * j + 1]);
          if constexpr (!kLoInRows) {
            const uint32_t pb[4] = {0u, pl[0], 0u, pl[1]};
            mma16816(c, pb, vb[2 * j], vb[2 * j + 1]);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) o[2 * dd + j][e] = fmaf(o[2 * dd + j][e], alpha, c[e]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
    }
    // ---- publish the warp's state in the layout decode_merged reads, merge, store
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if constexpr (kLoInRows) {
#pragma unroll
      for (int nb = 0; nb < 16; ++nb)
#pragma unroll
        for (int e = 0; e < 2; ++e) o[nb][2 + e] += __shfl_xor_sync(0xffffffffu, o[nb][e], 16);
    }
    bool repair = false;
    if (row < G) {
      float* dst = s_acc + (warp * G + row) * kD + 2 * quad;
#pragma unroll
      for (int nb = 0; nb < 16; ++nb) {
        const float2 v = make_float2(o[nb][0] + o[nb][2], o[nb][1] + o[nb][3]);
        repair |= isnan(v.x) || isnan(v.y);
        *reinterpret_cast<float2*>(dst + nb * 8) = v;
      }
      if (quad == 0) {
        s_acc[4 * G * kD + warp * G + row] = m_run;
        s_acc[4 * G * kD + 4 * G + warp * G + row] = l_run;
      }
    }
    if (__any_sync(0xffffffffu, repair)) {               // (the newest token is in the cache by now, written by the warp that reads it here)
      __syncwarp();
      ck_repair_sums(s_acc + warp * G * kD, s_acc + 4 * G * kD + warp * G, G, fuse.qkv != nullptr ? s_q : q + (static_cast<size_t>(it.b) * nq + qh0) * kD,
                     k_cache, v_cache, block_tables + static_cast<size_t>(it.b) * table_width, begin + warp * 16, end, it.kvh, nkv, block_size, num_blocks,
                     scale_log2, lane);
    }
    named_barrier_sync(1, 128);
    const int d = threadIdx.x;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float M, L;
      const float ov = decode_merged<G>(s_acc, g, d, M, L);
      if (it.len <= it.chunk) {
        out[(static_cast<size_t>(it.b) * nq + qh0 + g) * kD + d] = __float2bfloat16_rn(ov);
      } else {
        const size_t p = (static_cast<size_t>(it.b) * nq + qh0 + g) * max_chunks + it.c;
        part_o[p * kD + d] = ov;
        if (d == 0) {
          part_ml[p * 2] = M;
          part_ml[p * 2 + 1] = L;
        }
      }
    }
    named_barrier_sync(1, 128);                         // s_acc and s_q are the next item's
  }
}

extern "C" int forge_make_tmap_2d(CUtensorMap* tm, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, int elem_bytes);

template <int G>
static int launch_chunks(const void* q, const void* kc, const void* vc, const int* bt, const int* lens, void* out, float* part_o, float* part_ml, int B,
                         int nq, int nkv, int block_size, int table_width, int num_blocks, const DecodeSplit& split, int max_chunks, float scale_log2, unsigned* status,
                         cudaStream_t stream, const DecodeFuse& fuse) {
  constexpr int smem = kCkStages * 2 * kTcTileBytes + decode_merge_floats(G) * 4 + G * kD * 2 + 512 + 2 * kCkStages * 8 + 1024;
  static_assert(ck_ctas_per_sm(G) * (smem + 1024) <= 228 * 1024, "CTAs per SM");
  auto kern = decode_attn_chunk_kernel<G>;
  FORGE_ENSURE_DYN_SMEM(kern, smem);
  CUtensorMap tm_k, tm_v;
  const uint64_t rows = static_cast<uint64_t>(num_blocks) * nkv * block_size;
  if (forge_make_tmap_2d(&tm_k, kc, rows, kD, kD, kTcTile, 2) != 0 || forge_make_tmap_2d(&tm_v, vc, rows, kD, kD, kTcTile, 2) != 0) return -2;
  // up to two waves of CTAs: one per item, dead ones included (they end at once, and no list is walked); else the live ones over one wave
  const long long most = static_cast<long long>(B) * nkv * split.most;
  const int wave = ck_ctas_per_sm(G) * device_sm_count();
  const int direct = most <= 2 * wave;
  const dim3 grid(static_cast<unsigned>(direct ? most : wave));
  return launch_kernel(kern, grid, dim3(kDecThreads), smem, stream, 0, tm_k, tm_v, static_cast<const __nv_bfloat16*>(q),
                       static_cast<__nv_bfloat16*>(const_cast<void*>(kc)), static_cast<__nv_bfloat16*>(const_cast<void*>(vc)), bt, lens,
                       static_cast<__nv_bfloat16*>(out), part_o, part_ml, B, nq, nkv, block_size, table_width, num_blocks, split, max_chunks,
                       direct, scale_log2, status, fuse) == cudaSuccess ? 0 : -5;
}

// The attention kernel alone (partials of sequences of several chunks are merged by the caller); group = nq / nkv, 4..8.
int launch_decode_chunks(const void* q, const void* kc, const void* vc, const int* bt, const int* lens, void* out, float* part_o, float* part_ml, int B,
                         int nq, int nkv, int block_size, int table_width, int num_blocks, const DecodeSplit& split, int max_chunks, float scale_log2, unsigned* status,
                         cudaStream_t stream, const DecodeFuse& fuse) {
#define FORGE_CK(G)                                                                                                                          \
  case G:                                                                                                                                    \
    return launch_chunks<G>(q, kc, vc, bt, lens, out, part_o, part_ml, B, nq, nkv, block_size, table_width, num_blocks, split, max_chunks, \
                            scale_log2, status, stream, fuse)
  switch (nq / nkv) {
    FORGE_CK(4);
    FORGE_CK(5);
    FORGE_CK(6);
    FORGE_CK(7);
    FORGE_CK(8);
    default: return -1;
  }
#undef FORGE_CK
}

}  // namespace forge
