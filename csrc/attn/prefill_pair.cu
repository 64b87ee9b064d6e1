// Prefill attention on the 5th-generation tensor cores, two query tiles at a time (see prefill_umma.cu for the operands and for
// the kernel of one tile per CTA, and which of them runs).
//
//   S = Q K^T   A = Q tile, B = K tile (128 keys; one tile never straddles a cache block: block_size >= 128), both
//               K-major with the 128-byte swizzle, brought in by TMA, fp32 scores in tensor memory
//   O += P V    A = P, bf16 probabilities that take the place of their scores in tensor memory, B = V tile exactly as
//               TMA delivers it from the cache ([key][head_dim] rows, i.e. MN-major for this product: no transpose pass)
//
// A persistent CTA per SM works on one item at a time: TWO tiles of 128 query rows that share the stream of keys and
// values.  With an even number of q heads per KV head they are the same rows of two heads of a group, otherwise
// consecutive row tiles of one head.  The tensor core serves the tiles in turn, so it multiplies for one of them while
// the softmax warps of the other are at work, and the keys and values are loaded once for both.  Per 128 keys both tiles
// need 2060 clocks of the tensor core, 2048 of the special-function units (one exponential per score) and nearly as many
// of shared memory (P stays out of it for that reason); what bounds the kernel is the chain of a tile: scores, exponentials
// (a row per thread: ~1900 clocks), product with V.
// Measured (one tile per CTA in brackets): 3777 tokens, 32 / 8 heads: 135 us = 0.87 PFLOP/s (197); 28 sequences of 100 .. 1024 tokens, 16 / 8 heads:
// 102 us (188); 8 sequences of 256 tokens behind a prefix of 4096, 32 / 8 heads: 154 us (201); 16000 tokens, 16 / 8 heads: 901 us = 1.16 PFLOP/s (1190).
//
// Warp roles (320 threads): warps 0..3 and 4..7 = softmax of the two tiles, thread = one query row (its TMEM lane), so
// row max and row sum need no shuffles; warp 8 = TMA producer (K and V rings of 2 stages); warp 9 = owner of tensor
// memory and UMMA issuer, in the order  P0 V, Q0 K', P1 V, Q1 K'  (K' = next tile): instructions of one thread execute
// in order, which is what lets the next scores overwrite P and S without a barrier.  The tensor core's queue is short: what the
// issuer does between two products, the core waits for, and on an SM whose schedulers are busy with exponentials every instruction
// of another warp is slow.  So it issues whole groups of products (one asm block each) and waits as rarely as possible.
// The exponentials use a reference maximum that is only raised when the true row maximum has grown by more than 2^8 since it was set
// (exact arithmetic either way: O and the row sum carry the same factor); only then do the softmax warps read O back,
// scale it and store it again, which happens a few times per row instead of once per tile.  Each row decides for itself.  The end of an item (O is normalised and
// stored) overlaps with the first scores of the next one.
//
// Items are dealt out from the last rows of the sequences (the most keys) to the first, forwards and backwards over the
// CTAs in turn, so that long and short ones add up alike; every warp walks the same list by itself from the lengths.
//
// The query rows of a sequence are its LAST q_len positions; with a cached prefix the causal mask is aligned to the
// bottom-right corner: query row i sees keys 0 .. (k_len - q_len + i).  scale > 0 (hidden scores are -inf).  All waits are bounded (ptx.cuh).
#include "../include/launch.cuh"
#include "../include/ptx.cuh"

#include <algorithm>

namespace forge {

constexpr int kWD = 128;                  // head_dim
constexpr int kWM = 128;                  // query rows of a tile
constexpr int kWN = 128;                  // keys per tile
constexpr int kWHalf = 128 * 128;         // bytes of one swizzled box: 128 rows x 64 bf16
constexpr int kWTile = 2 * kWHalf;        // one 128 x 128 bf16 operand
constexpr int kWThreads = 320;
constexpr int kWStages = 2;

// ---- groups of products, issued by one elected lane of a converged warp.  Descriptors advance in units of 16 bytes.
// D = A B^T over 128 entries: two boxes of 64 columns, 32 bytes (16 entries) per instruction; then one arrival on `bar`.
__device__ __forceinline__ void pair_scores(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred e, z, o;\n\t.reg .b64 a, b;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 z, 0, 0;\n\t"
      "setp.eq.b32 o, 0, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, z;\n\t"
      "add.s64 a, %1, 2;\n\tadd.s64 b, %2, 2;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 4;\n\tadd.s64 b, %2, 4;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 6;\n\tadd.s64 b, %2, 6;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 1024;\n\tadd.s64 b, %2, 1024;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 1026;\n\tadd.s64 b, %2, 1026;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 1028;\n\tadd.s64 b, %2, 1028;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "add.s64 a, %1, 1030;\n\tadd.s64 b, %2, 1030;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, o;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%4];\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(bar)
      : "memory");
}
// D (+)= P V over 64 keys: 8 columns of P and 16 rows of V (2048 bytes) per instruction.
__device__ __forceinline__ void pair_values(uint32_t tmem_d, uint32_t tmem_p, uint64_t vdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred e, p, o;\n\t.reg .b64 b;\n\t.reg .b32 a;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.eq.b32 o, 0, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "add.s32 a, %1, 8;\n\tadd.s64 b, %2, 128;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, o;\n\t"
      "add.s32 a, %1, 16;\n\tadd.s64 b, %2, 256;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, o;\n\t"
      "add.s32 a, %1, 24;\n\tadd.s64 b, %2, 384;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, o;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_p), "l"(vdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// p = 2^(s * scale - m_ref) of 32 scores, as pairs of bf16 to tensor memory (16 columns); adds p to the running sums, two sums to a register
// pair: of the four pairs of eight scores, in the order of umma_probs_to_smem.  Two scores per multiply-add and addition.  (A quarter or three eighths of the exponentials as polynomials on the multiply-add
// units instead: slower by 5 to 8 %, the one warp that is active per scheduler issues no faster.)
__device__ __forceinline__ void pair_probs(const uint32_t* v, uint64_t scale2, uint64_t ref2, uint64_t (&sum)[2], uint32_t p_addr) {
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    float p[4];
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[i + e]), __uint_as_float(v[i + e + 1])), scale2, ref2), p[e], p[e + 1]);
      p[e] = ex2_approx(p[e]);
      p[e + 1] = ex2_approx(p[e + 1]);
      pk[(i + e) >> 1] = pack_bf16x2(p[e], p[e + 1]);
    }
    sum[(i >> 2) & 1] = add_f32x2(sum[(i >> 2) & 1], add_f32x2(pack_f32x2(p[0], p[2]), pack_f32x2(p[1], p[3])));
  }
  tmem_st_x16(p_addr, pk);
}

struct PairShape {
  int nq, nkv, block_size, table_width, num_blocks, num_seqs;
  int levels;        // most row blocks of a sequence
  int units;         // items per row block: pairs of heads, or heads
  int head_pairs;    // the tiles of an item are two heads (else consecutive row tiles)
};

// One item of the list: its sequence, and per tile the head, the first row and the number of key tiles (0: no such tile).
struct PairItem {
  int q_begin, q_len, k_len, seq, kvh;
  int h[2], m0[2], n[2];
};

// The list of items: row blocks from the last to the first; within one, the sequences that have it, with all their units.
// Executed by whole warps.
struct PairItems {
  const int* cu;
  const int* lens;
  PairShape s;
  int level, base, count, round;

  __device__ PairItems(const int* cu_, const int* lens_, const PairShape& s_) : cu(cu_), lens(lens_), s(s_), level(s_.levels), base(0), count(0), round(0) {}
  __device__ bool has(int seq) const {
    return seq < s.num_seqs && cu[seq + 1] - cu[seq] > level * (s.head_pairs ? kWM : 2 * kWM);
  }
  __device__ bool next(PairItem& it) {
    const int g = gridDim.x, lane = threadIdx.x & 31;
    const int k = (round & 1) ? (round + 1) * g - 1 - static_cast<int>(blockIdx.x) : round * g + static_cast<int>(blockIdx.x);
    ++round;
    while (k >= base + count * s.units) {
      base += count * s.units;
      if (--level < 0) return false;
      count = 0;
      for (int c = 0; c < s.num_seqs; c += 32) count += __popc(__ballot_sync(0xffffffffu, has(c + lane)));
    }
    int rank = (k - base) / s.units;
    const int unit = (k - base) - rank * s.units;
    int seq = 0;
    for (int c = 0; c < s.num_seqs; c += 32) {
      const bool mine = has(c + lane);
      const uint32_t mask = __ballot_sync(0xffffffffu, mine);
      const int n = __popc(mask);
      if (rank < n) {
        seq = c + __ffs(__ballot_sync(0xffffffffu, mine && __popc(mask & ((1u << lane) - 1)) == rank)) - 1;
        break;
      }
      rank -= n;
    }
    it.seq = seq;
    it.q_begin = cu[seq];
    it.q_len = cu[seq + 1] - it.q_begin;
    it.k_len = lens[seq];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      it.h[i] = s.head_pairs ? 2 * unit + i : unit;
      it.m0[i] = s.head_pairs ? level * kWM : (2 * level + i) * kWM;
      const int kv_end = min(it.k_len, it.k_len - it.q_len + it.m0[i] + kWM);        // keys visible to the last row of the tile
      it.n[i] = it.m0[i] < it.q_len && kv_end > 0 ? (kv_end + kWN - 1) / kWN : 0;
    }
    it.kvh = it.h[0] / (s.nq / s.nkv);
    return true;
  }
};

// tm_q: 2-D view [T, nq * 128] of q, box 128 rows x 64 cols.  tm_k / tm_v: 2-D view [blocks * nkv * block_size, 128]
// of a cache, box 128 rows x 64 cols.
__global__ void __launch_bounds__(kWThreads, 1) prefill_attn_pair_kernel(
    const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
    const int* __restrict__ cu_seqlens_q, const int* __restrict__ context_lens, const int* __restrict__ block_tables,
    __nv_bfloat16* __restrict__ out, const PairShape shape, float scale_log2, unsigned* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                               // [2 tiles]
  uint8_t* sK = sQ + 2 * kWTile;                    // [2 stages]
  uint8_t* sV = sK + kWStages * kWTile;             // [2 stages]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kWStages * kWTile);
  uint64_t* q_full = bars;                          // [2 tiles]
  uint64_t* q_empty = bars + 2;                     // [2 tiles]
  uint64_t* k_full = bars + 4;                      // [2 stages]
  uint64_t* k_empty = bars + 6;                     // [2 stages]
  uint64_t* v_full = bars + 8;                      // [2 stages]
  uint64_t* v_empty = bars + 10;                    // [2 stages]
  uint64_t* s_full = bars + 12;                     // [2 tiles]: scores are there, and all earlier products of the tile in O
  uint64_t* p_full = bars + 14;                     // [2 tiles][2 halves of the keys], one arrival per softmax warp
  uint64_t* o_full = bars + 18;                     // [2 tiles]: the last P V of an item is complete
  uint64_t* o_empty = bars + 20;                    // [2 tiles], one arrival per softmax warp: O has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (warp == 8 && lane == 0) {
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[2 * i], 4);
      mbar_init(&p_full[2 * i + 1], 4);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_empty[i], 4);
    }
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);                         // S0 | S1 | O0 | O1, 128 columns each
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();

  PairItems items(cu_seqlens_q, context_lens, shape);
  PairItem it;
  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    uint32_t t = 0, uses[2] = {0, 0};                   // key tiles so far; items that used each Q buffer
    bool ok = true;
    while (ok && items.next(it)) {
      if (lane == 0) {
        const int n = max(it.n[0], it.n[1]);
        const int* table = block_tables + static_cast<size_t>(it.seq) * shape.table_width;
        for (int j = 0; j < n && ok; ++j, ++t) {
          const int s = t % kWStages;
          const uint32_t ph = (t / kWStages) & 1;
          const int tok = j * kWN;
          int blk = table[min(tok / shape.block_size, shape.table_width - 1)];
          if (blk < 0 || blk >= shape.num_blocks) {
            set_status(status, kStatusBadIndex);
            blk = 0;
          }
          const int row = (blk * shape.nkv + it.kvh) * shape.block_size + (tok % shape.block_size);
          ok = mbar_wait_parked(&k_empty[s], ph ^ 1, status);
          if (!ok) break;
          mbar_expect_tx(&k_full[s], kWTile);
          tma_load_2d(sK + s * kWTile, &tm_k, &k_full[s], 0, row);
          tma_load_2d(sK + s * kWTile + kWHalf, &tm_k, &k_full[s], 64, row);
          if (j == 0) {
            for (int i = 0; i < 2 && ok; ++i) {
              if (it.n[i] == 0) continue;
              ok = mbar_wait_parked(&q_empty[i], (uses[i]++ & 1) ^ 1, status);
              if (!ok) break;
              mbar_expect_tx(&q_full[i], kWTile);
              tma_load_2d(sQ + i * kWTile, &tm_q, &q_full[i], it.h[i] * kWD, it.q_begin + it.m0[i]);
              tma_load_2d(sQ + i * kWTile + kWHalf, &tm_q, &q_full[i], it.h[i] * kWD + 64, it.q_begin + it.m0[i]);
            }
          }
          ok = ok && mbar_wait_parked(&v_empty[s], ph ^ 1, status);
          if (!ok) break;
          mbar_expect_tx(&v_full[s], kWTile);
          tma_load_2d(sV + s * kWTile, &tm_v, &v_full[s], 0, row);
          tma_load_2d(sV + s * kWTile + kWHalf, &tm_v, &v_full[s], 64, row);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ UMMA issuer
    constexpr uint32_t idesc_s = umma_idesc(kWM, kWN, 1, 1);                  // both operands K-major
    constexpr uint32_t idesc_o = umma_idesc(kWM, kWD, 1, 1) | (1u << 16);     // B (= V) MN-major
    const uint64_t q_desc = umma_desc_k_sw128(smem_u32(sQ)), k_desc = umma_desc_k_sw128(smem_u32(sK));
    const uint64_t v_desc = umma_desc_mn_sw128(smem_u32(sV), kWHalf);
    bool ok = true;                                      // once a wait has run out none is made any more
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      if (ok && !mbar_test(bar, parity)) ok = mbar_wait(bar, parity, status);
      __syncwarp();
    };
    uint32_t t = 0, q_phase = 0, p_phase = 0;           // key tiles so far; parities of q_full and of p_full per tile
    while (items.next(it)) {
      const int n = max(it.n[0], it.n[1]);
      for (int j = -1; j < n && n > 0; ++j) {
        // key tile j: its product with V; key tile j + 1: its scores, which take the place of P
        const uint32_t next = t + 1 + j;
        const uint32_t vs = (t + j) % kWStages, ks = next % kWStages;
        if (j + 1 < n) wait(&k_full[ks], (next / kWStages) & 1);
        if (j >= 0) wait(&v_full[vs], ((t + j) / kWStages) & 1);
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const int mine = i == 0 ? it.n[0] : it.n[1];
          const uint32_t s_tmem = tmem_base + i * kWN, o_tmem = tmem_base + 256 + i * kWD;
          if (j >= 0 && j < mine) {
            if (j == 0) wait(&o_empty[i], ((q_phase >> i) & 1) ^ 1);                   // the item before has left O
            const uint64_t vd = v_desc + vs * (kWTile / 16);
            wait(&p_full[2 * i], (p_phase >> i) & 1);
            tcgen05_fence_after();
            pair_values(o_tmem, s_tmem, vd, idesc_o, j);
            wait(&p_full[2 * i + 1], (p_phase >> i) & 1);
            tcgen05_fence_after();
            pair_values(o_tmem, s_tmem + 32, vd + 512, idesc_o, 1);
            p_phase ^= 1u << i;
            if (j + 1 == mine) umma_commit_warp(&o_full[i]);
          }
          if (j + 1 < mine) {
            if (j < 0) {
              wait(&q_full[i], (q_phase >> i) & 1);
              tcgen05_fence_after();
            }
            pair_scores(s_tmem, q_desc + i * (kWTile / 16), k_desc + ks * (kWTile / 16), idesc_s, smem_u32(&s_full[i]));
            if (j + 2 == mine) umma_commit_warp(&q_empty[i]);
          }
        }
        if (j + 1 < n) umma_commit_warp(&k_empty[ks]);
        if (j >= 0) umma_commit_warp(&v_empty[vs]);
      }
      t += n;
      q_phase ^= (it.n[0] > 0 ? 1u : 0u) | (it.n[1] > 0 ? 2u : 0u);
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: thread = query row
    const int i = warp >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;                      // row of the tile == TMEM lane
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_addr + i * kWN, o_addr = tmem_base + lane_addr + 256 + i * kWD;
    const uint64_t scale2 = pack_f32x2(scale_log2, scale_log2);
    uint32_t uses = 0, tiles = 0;
    bool ok = true;
    while (ok && items.next(it)) {
      const int m0 = i == 0 ? it.m0[0] : it.m0[1], n = i == 0 ? it.n[0] : it.n[1], h = i == 0 ? it.h[0] : it.h[1];
      const int limit = min(it.k_len - it.q_len + m0 + r + 1, it.k_len);               // visible keys: [0, limit)
      float m_ref = 0.f, l_run = 0.f;                    // reference maximum of the exponentials (scaled, log2 domain), row sum
      for (int j = 0; j < n; ++j) {
        ok = mbar_wait(&s_full[i], tiles++ & 1, status);
        if (!ok) break;
        tcgen05_fence_after();
        const int kbase = j * kWN;
        if (!__all_sync(0xffffffffu, kbase + kWN <= limit)) {          // the diagonal or the end of the sequence: hidden scores become -inf
#pragma unroll 1
          for (int c = 0; c < kWN; c += 32) {
            uint32_t v[32];
            tmem_ld_x32(s_addr + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = kbase + c + e < limit ? v[e] : 0xff800000u;
            tmem_st_x32(s_addr + c, v);
          }
          tmem_st_wait();
        }
        uint32_t va[32], vb[32];
        float mt;
        {
          uint32_t vc[32], vd[32];
          tmem_ld_x32(s_addr, va);
          tmem_ld_x32(s_addr + 32, vb);
          tmem_ld_x32(s_addr + 64, vc);
          tmem_ld_x32(s_addr + 96, vd);
          tmem_ld_wait();
          float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            m[e & 1] = fmaxf(fmaxf(m[e & 1], __uint_as_float(va[e])), __uint_as_float(vb[e]));
            m[2 + (e & 1)] = fmaxf(fmaxf(m[2 + (e & 1)], __uint_as_float(vc[e])), __uint_as_float(vd[e]));
          }
          mt = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])) * scale_log2;               // scale > 0: max commutes with the scaling
        }
        if (j == 0) {
          m_ref = mt == -INFINITY ? 0.f : mt;            // O is not valid yet: nothing to rescale
        } else if (const bool grow = mt - m_ref > 8.f; __any_sync(0xffffffffu, grow)) {
          // tcgen05.ld / .st are warp-wide: the whole warp rescales, rows whose maximum did not grow by exactly 1 (what a row gives does not
          // depend on its neighbours).  The commit behind s_full covered every earlier P V.
          const float m_new = grow ? mt : m_ref;
          const float alpha = exp2f(m_ref - m_new);
#pragma unroll 1
          for (int c = 0; c < kWD; c += 32) {
            uint32_t o[32];
            tmem_ld_x32(o_addr + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_x32(o_addr + c, o);
          }
          l_run *= alpha;
          m_ref = m_new;
        }
        // P: 32 scores at a time, the next ones on their way from tensor memory meanwhile; P of scores c .. takes columns c / 2 ..,
        // whose scores have been read.  Each half of P is handed over by itself.
        const uint64_t ref2 = pack_f32x2(-m_ref, -m_ref);
        uint64_t sum[2] = {0, 0};
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          pair_probs(va, scale2, ref2, sum, s_addr + half * 32);
          if (half == 0) tmem_ld_x32(s_addr + 64, va);
          pair_probs(vb, scale2, ref2, sum, s_addr + half * 32 + 16);
          tmem_ld_wait();
          if (half == 0) tmem_ld_x32(s_addr + 96, vb);
          tmem_st_wait();
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[2 * i + half]);
          if (half == 0) tmem_ld_wait();
        }
        float l0, l1, l2, l3;
        unpack_f32x2(sum[0], l0, l1);
        unpack_f32x2(sum[1], l2, l3);
        l_run += (l0 + l1) + (l2 + l3);
      }
      // all of O: wait for the last P V, normalise, store (rows that see nothing, and tiles without keys, are zero)
      if (ok && n > 0) ok = mbar_wait(&o_full[i], uses++ & 1, status);
      if (!ok) break;
      if (m0 >= it.q_len) continue;
      tcgen05_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const bool store = m0 + r < it.q_len;
      __nv_bfloat16* dst = out + static_cast<size_t>(it.q_begin + m0 + r) * shape.nq * kWD + h * kWD;
#pragma unroll 1
      for (int c = 0; c < kWD; c += 64) {
        uint32_t o[64];
        if (n > 0) {
          tmem_ld_x32(o_addr + c, o);
          tmem_ld_x32(o_addr + c + 32, o + 32);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 64; ++e) o[e] = 0;
        }
        if (c + 64 == kWD && n > 0) {
          tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_empty[i]);       // O is in registers: the next item may use it
        }
        if (store) {
#pragma unroll
          for (int e = 0; e < 64; e += 8) {
            uint4 pk;
            pk.x = pack_bf16x2(__uint_as_float(o[e]) * inv, __uint_as_float(o[e + 1]) * inv);
            pk.y = pack_bf16x2(__uint_as_float(o[e + 2]) * inv, __uint_as_float(o[e + 3]) * inv);
            pk.z = pack_bf16x2(__uint_as_float(o[e + 4]) * inv, __uint_as_float(o[e + 5]) * inv);
            pk.w = pack_bf16x2(__uint_as_float(o[e + 6]) * inv, __uint_as_float(o[e + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c + e) = pk;
          }
        }
      }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 9) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Tensor maps as above; operands as forge_prefill_attention.
int launch_prefill_attn_pair(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const int* cu_q, const int* lens,
                             const int* bt, void* out, int T, int num_seqs, int max_q, int nq, int nkv, int block_size, int table_width,
                             int num_blocks, float scale_log2, unsigned* status, cudaStream_t stream) {
  constexpr int smem = (2 + 2 * kWStages) * kWTile + 256 + 1024;
  FORGE_ENSURE_DYN_SMEM(prefill_attn_pair_kernel, smem);
  PairShape s;
  s.nq = nq;
  s.nkv = nkv;
  s.block_size = block_size;
  s.table_width = table_width;
  s.num_blocks = num_blocks;
  s.num_seqs = num_seqs;
  s.head_pairs = (nq / nkv) % 2 == 0;
  const int block_rows = s.head_pairs ? kWM : 2 * kWM;
  s.levels = (max_q + block_rows - 1) / block_rows;
  s.units = s.head_pairs ? nq / 2 : nq;
  const long long most = std::min<long long>(static_cast<long long>(num_seqs) * s.levels, T / block_rows + num_seqs) * s.units;
  if (most <= 0) return 0;
  const dim3 grid(static_cast<unsigned>(std::min<long long>(most, device_sm_count())));
  return launch_kernel(prefill_attn_pair_kernel, grid, dim3(kWThreads), smem, stream, 0, tm_q, tm_k, tm_v, cu_q, lens, bt,
                       static_cast<__nv_bfloat16*>(out), s, scale_log2, status) == cudaSuccess ? 0 : -5;
}

}  // namespace forge
