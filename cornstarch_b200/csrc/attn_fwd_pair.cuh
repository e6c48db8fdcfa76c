// Attention forward with two 128-row query tiles per thread block (included by attn_fwd.cu).
//
// The two tiles ("streams") of a block are neighbours of one head and share every K / V tile that is loaded.  Each stream
// has its own softmax group of four warps, ONE thread per query row, its own S buffer and its own accumulator in tensor
// memory (2 x 128 columns of S, 2 x 128 of O).  The MMA warp alternates between the streams:
//
//     S0(0) S1(0) | P0V(0) S0(1)  P1V(0) S1(1) | P0V(1) S0(2)  P1V(1) S1(2) | ...
//
// so that one group computes exponentials while the tensor core works for the other, and the two softmax warps of a
// scheduler are in different phases of a tile.  (With one tile per block both warps of a scheduler load, take maxima and
// store at the same time; the special-function unit and the tensor core then idle in turns.  An MMA warp per stream has the
// same effect: the streams fall into step, 939 us for the case below that takes 833.)  One thread per row takes the maximum
// with three-input instructions and scales and sums in packed pairs; nothing is exchanged between threads.
//
// What bounds it: the chain of a stream, P V and the next S (1024 cycles of the tensor pipe, of which the other stream takes
// as many) and the softmax in between, about 3050 cycles per key tile and pair where the pipe needs 2048; on long runs the
// power cap (990 W at 1.63 GHz).  Before, it was the MMA warp's own instructions: 90 cycles to issue an MMA that takes 64, 550 to
// 1000 per tile for tile classes and waits.  Hence runs of MMAs (umma_f16_run_w), classes as bits in registers and one wait per
// tile for K and V; P goes over in two halves so that P V starts beside the second half's exponentials.
// Measured (B200, 32 / 8 heads of 128, before -> now): 8192 tokens causal 507 -> 460 us (1195 TFLOP/s), full 920 -> 837 to 866 us (1310 to
// 1270 TFLOP/s, by the power cap); 1024 causal 23.4 -> 21.2 us; 4 x 729 tokens, 16 heads of 72: 35.7 -> 35.2 us.  1.2 % of it are two
// waits for soundness: one verdict per warp (mbar_wait_abort_w), and tcgen05.wait::st between a P and its correction.
//
// Hand-overs per stream and tile: s_full (MMA -> softmax) and p_full, one per half of the keys (softmax -> MMA), strictly
// alternating, so no parity wait can be two phases behind.  S(next) of a stream is issued after P V of its current tile, whose
// operand P lives in the columns that S(next) overwrites; s_full of the next tile therefore also says that P V has retired,
// which is what the lazy rescale of O needs.
#pragma once

namespace csb {

// Three warpgroups: TMA, MMA and two spare warps; the softmax warps of stream 0; those of stream 1.  The block is launched
// with 168 registers a thread; the first group hands 80 of them on (88 + 208 + 208 = 3 x 168).
constexpr int PAIR_THREADS = 384;

template <int NCH>
struct PairSmem {
  static constexpr int TILE_BYTES = NCH * CHUNK_BYTES;
  static constexpr int Q_OFF = 0;                          // two query tiles
  static constexpr int K_OFF = Q_OFF + 2 * TILE_BYTES;     // two stages
  static constexpr int V_OFF = K_OFF + 2 * TILE_BYTES;     // two stages
  static constexpr int META_OFF = V_OFF + 2 * TILE_BYTES;  // per softmax warp: key bits int64[128], key positions int[128]
  static constexpr int META_WARP = 128 * 12;
  static constexpr int CLS_OFF = META_OFF + 8 * META_WARP;  // tile classes of both streams
  static constexpr int MAX_NK = AttnSmem<NCH>::MAX_NK;
  static constexpr int BAR_OFF = CLS_OFF + 2 * MAX_NK;
  static constexpr int NBAR = 13;
  static constexpr int TOTAL = BAR_OFF + NBAR * 8 + 16;
  static constexpr int DYN_BYTES = TOTAL + 1024;
};

// Which of the 128 keys of tile j this query row may attend to, as four words of 32 bits (tiles of class 1 only).
// kb_w / kp_w: this warp's staging area for the keys' bits and positions.
__device__ __forceinline__ void tile_mask_words(const AttnFwdParams& p, int b, int j, int q, bool row_valid, const QueryRule& rule,
                                                int lane, int64_t* kb_w, int* kp_w, uint32_t (&w)[4]) {
  const int k0 = j * AT_BN;
  if (mask_by_index(p.mask_mode, p.q_pos, p.k_pos)) {
    int n = p.Sk - k0;  // keys of the tile that exist
    if (p.mask_mode == MASK_CAUSAL) n = min(n, q - k0 + 1);
    if (!row_valid) n = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int m = n - 32 * g;
      w[g] = m >= 32 ? 0xffffffffu : (m <= 0 ? 0u : (1u << m) - 1u);
    }
    return;
  }
  __syncwarp();  // the previous tile's readers are done with the staging area
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = k0 + i * 32 + lane;
    const bool kv = k < p.Sk;
    const int kp = kv ? (p.k_pos ? p.k_pos[(long)b * p.Sk + k] : k) : -1;  // a negative position marks a key that does not exist
    kb_w[i * 32 + lane] = mask_key_bits(p.mask_mode, kp >= 0, (kv && p.k_bits) ? p.k_bits[(long)b * p.Sk + k] : 0);
    kp_w[i * 32 + lane] = kp;
  }
  __syncwarp();
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t m = 0;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) m |= (rule_allows(rule, kb_w[g * 32 + i], kp_w[g * 32 + i]) ? 1u : 0u) << i;
    w[g] = m;
  }
}

template <int NCH>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const AttnFwdParams p) {
  using L = PairSmem<NCH>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* q_full = bars;        // both query tiles and the first K tile
  uint64_t* vk_full = bars + 1;   // [2] V of ring position i and K of position i + 1
  uint64_t* vk_empty = bars + 3;  // [2]
  uint64_t* s_full = bars + 5;    // [2] per stream
  uint64_t* o_full = bars + 7;    // [2] per stream: its last P V has retired
  uint64_t* p_full = bars + 9;    // [2][2] per stream and half of the keys, 128 arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int8_t* cls_s = reinterpret_cast<int8_t*>(smem + L::CLS_OFF);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heaviest (last) query tiles first, over all heads and batch entries, as in attn_fwd_kernel
  const int n_hb = p.Hq * p.B;
  const int n_pairs = (p.nQ + 1) >> 1;
  const int hb = blockIdx.x % n_hb;
  const int qp0 = (n_pairs - 1 - (int)blockIdx.x / n_hb) * 2;  // first query tile of the pair
  const int h = hb % p.Hq, b = hb / p.Hq;
  const int hk = h / (p.Hq / p.Hk);
  const int n_streams = qp0 + 1 < p.nQ ? 2 : 1;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    for (int j = threadIdx.x; j < p.nK; j += blockDim.x)
      cls_s[s * L::MAX_NK + j] = s < n_streams ? tile_class(p, b, qp0 + s, j) : int8_t(0);
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < 9; ++i) mbar_init(&bars[i], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&p_full[i], 128);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_S = tmem_base;        // stream s: columns [128 s, +128); P over the first 64 of them
  const uint32_t tmem_O = tmem_base + 256;  // stream s: columns [128 s, +dk16)
  const int8_t* cls0 = cls_s;
  const int8_t* cls1 = cls_s + L::MAX_NK;
  // next key tile at or after t that either stream needs
  auto next_tile = [&](int t) -> int {
    while (t < p.nK && (cls0[t] | cls1[t]) == 0) ++t;
    return t;
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      auto load = [&](int off, const CUtensorMap* tm, uint64_t* bar, int head, int tile) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) tma_load_4d(smem + off + c * CHUNK_BYTES, tm, bar, c * 64, head, tile * 128, b);
      };
      int t = next_tile(0);
      // Without a key tile (queries that are all padding) nobody waits for the query tiles, so they are not loaded: the block
      // would exit with the copies in flight, into shared memory and barriers that the SM's next block already uses.
      if (t < p.nK) {
        mbar_expect_tx(q_full, (n_streams + 1) * L::TILE_BYTES);
        load(L::Q_OFF, &tm_q, q_full, h, qp0);
        load(L::K_OFF, &tm_k, q_full, hk, t);
        if (n_streams == 2) load(L::Q_OFF + L::TILE_BYTES, &tm_q, q_full, h, qp0 + 1);
      }
      for (uint32_t it = 0; t < p.nK; ++it) {
        const int st = it & 1, tn = next_tile(t + 1);
        // Free are the V stage (P V of position it - 2 is done; the first two are free at the start) and the K stage that position
        // it + 1 takes (S of position it - 1 is done; the first one at the start).  S is issued a position ahead of P V, so one
        // commit after position it - 2 says both; for it = 1 there is one after the first S.
        if (!mbar_wait_abort(&vk_empty[st], ((it >> 1) ^ it ^ 1) & 1, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_EMPTY); *abort_flag = 1; break; }
        mbar_expect_tx(&vk_full[st], (tn < p.nK ? 2 : 1) * L::TILE_BYTES);
        load(L::V_OFF + st * L::TILE_BYTES, &tm_v, &vk_full[st], hk, t);
        if (tn < p.nK) load(L::K_OFF + (st ^ 1) * L::TILE_BYTES, &tm_k, &vk_full[st], hk, tn);
        t = tn;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (whole warp in step, see umma_f16_w)
    const uint32_t idesc_s = make_idesc_bf16(AT_BM, AT_BN, 0, 0);
    const uint32_t idesc_o = make_idesc_bf16(AT_BM, p.dk16, 0, 1);
    const int ksteps_s = p.dk16 / 16;
    const uint64_t q_desc = make_desc_kmajor_sw128(smem_u32(smem + L::Q_OFF));
    const uint64_t k_desc = make_desc_kmajor_sw128(smem_u32(smem + L::K_OFF));
    const uint64_t v_desc = make_desc_mnmajor_sw128(smem_u32(smem + L::V_OFF), CHUNK_BYTES);
    constexpr uint64_t TILE_STEP = L::TILE_BYTES >> 4;  // from one tile to the next, in a descriptor's address field
    bool ok = true;
    auto fail = [&](int code) {
      atomicCAS(p.status, 0, code);
      *abort_flag = 1;
      ok = false;
    };
    // S of stream s = Q_s K^T with the K tile of ring position it
    auto issue_s = [&](int s, uint32_t it) {
      umma_f16_run_w(tmem_S + s * 128, q_desc + s * TILE_STEP, k_desc + (it & 1) * TILE_STEP, CHUNK_BYTES, CHUNK_BYTES, idesc_s, ksteps_s, 0u);
      umma_commit_w(&s_full[s]);
    };
    // Key tiles as bits of 32, per stream: no shared-memory reads on the way from one MMA to the next.
    int base = -32;
    uint32_t bits[2] = {0, 0};
    auto next = [&](uint32_t& who) -> int {  // the next tile that a stream needs (nK at the end); who: bit s = stream s needs it
      while ((bits[0] | bits[1]) == 0) {
        base += 32;
        if (base >= p.nK) {
          who = 0;
          return p.nK;
        }
        const bool in = base + lane < p.nK;
        bits[0] = __ballot_sync(0xffffffffu, in && cls0[base + lane] != 0);
        bits[1] = __ballot_sync(0xffffffffu, in && cls1[base + lane] != 0);
      }
      const uint32_t low = (bits[0] | bits[1]) & (0u - (bits[0] | bits[1]));
      who = ((bits[0] & low) ? 1u : 0u) | ((bits[1] & low) ? 2u : 0u);
      bits[0] &= ~low;
      bits[1] &= ~low;
      return base + __ffs(low) - 1;
    };
    int last[2] = {-1, -1};  // last key tile of each stream
    for (int b0 = 0; b0 < p.nK; b0 += 32) {
      const bool in = b0 + lane < p.nK;
      const uint32_t m0 = __ballot_sync(0xffffffffu, in && cls0[b0 + lane] != 0), m1 = __ballot_sync(0xffffffffu, in && cls1[b0 + lane] != 0);
      if (m0 != 0) last[0] = b0 + 31 - __clz(m0);
      if (m1 != 0) last[1] = b0 + 31 - __clz(m1);
    }
    uint32_t done[2] = {0, 0};  // tiles of each stream whose P V was issued
    uint32_t who, who_next;
    int t = next(who);
    if (t < p.nK) {
      if (!mbar_wait_abort_w(q_full, 0, abort_flag)) fail(ST_TIMEOUT_FULL);
      if (ok) {
        tc_fence_after();
        if (who & 1u) issue_s(0, 0);
        if (who & 2u) issue_s(1, 0);
        umma_commit_w(&vk_empty[1]);
      }
    }
    for (uint32_t it = 0; ok && t < p.nK; ++it) {
      const int tn = next(who_next);
      const int st = it & 1;
      if (!mbar_wait_abort_w(&vk_full[st], (it >> 1) & 1, abort_flag)) { fail(ST_TIMEOUT_FULL); break; }
      tc_fence_after();
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (who & (1u << s)) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (!mbar_wait_abort_w(&p_full[s * 2 + u], done[s] & 1, abort_flag)) { fail(ST_TIMEOUT_MISC); break; }
            tc_fence_after();
            umma_f16_ts_run4_w(tmem_O + s * 128, tmem_S + s * 128 + u * 32,
                               v_desc + st * TILE_STEP + static_cast<uint64_t>((u * 4 * 2048) >> 4), idesc_o, done[s] > 0 || u > 0 ? 1u : 0u);
          }
          if (!ok) break;
          ++done[s];
          if (t == last[s]) umma_commit_w(&o_full[s]);
        }
        if (who_next & (1u << s)) issue_s(s, it + 1);
      }
      if (!ok) break;
      umma_commit_w(&vk_empty[st]);
      t = tn;
      who = who_next;
    }
    __syncwarp();
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    // ------------------------------------------------------------------ softmax / epilogue: one thread per query row
    const int s_id = (warp - 4) >> 2;   // stream
    const int quarter = warp & 3;       // TMEM lane quarter this warp may touch
    const int r = quarter * 32 + lane;  // row inside the tile == TMEM lane
    const int q = (qp0 + s_id) * AT_BM + r;
    const bool row_valid = q < p.Sq;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t_S = tmem_S + s_id * 128 + lane_addr;
    const uint32_t t_O = tmem_O + s_id * 128 + lane_addr;
    const int8_t* cls_row = s_id == 0 ? cls0 : cls1;
    int64_t* kb_w = reinterpret_cast<int64_t*>(smem + L::META_OFF + (warp - 4) * L::META_WARP);
    int* kp_w = reinterpret_cast<int*>(kb_w + 128);
    int64_t qb = 0;
    int qpos = q;
    if (row_valid) {
      if (p.q_bits) qb = p.q_bits[(long)b * p.Sq + q];
      if (p.q_pos) qpos = p.q_pos[(long)b * p.Sq + q];
    }
    const QueryRule rule = make_query_rule(p.mask_mode, row_valid, qb, qpos);
    float m_used = -INFINITY, l_sum = 0.f;
    uint32_t it = 0;
    bool ok = true;
    const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    for (int j = 0; j < p.nK; ++j) {
      const int c = cls_row[j];
      if (c == 0) continue;
      uint32_t w[4] = {0u, 0u, 0u, 0u};
      if (c == 1) tile_mask_words(p, b, j, q, row_valid, rule, lane, kb_w, kp_w, w);  // while S is being computed
      if (!mbar_wait_abort_w(&s_full[s_id], it & 1, abort_flag)) {
        if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int g = 0; g < 4; ++g) tmem_ld_32x32(t_S + g * 32, v[g]);
      tmem_ld_wait();
      if (c == 1) {
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
          for (int i = 0; i < 32; ++i) v[g][i] = ((w[g] >> i) & 1u) ? v[g][i] : 0xff800000u;  // -inf
      }
      uint64_t ls[2] = {0ull, 0ull};
      // exponentials of 64 keys with the maximum that is in use: P over the first 64 columns of S (all of S is in registers)
      auto half_tile = [&](int u) {
        const float m_eff = (m_used == -INFINITY) ? 0.f : m_used * p.scale_log2;
        const uint64_t negm2 = pack_f32x2(-m_eff, -m_eff);
#pragma unroll
        for (int g = 2 * u; g < 2 * u + 2; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const uint64_t y2 = fma_f32x2(pack_u32x2(v[g][2 * i], v[g][2 * i + 1]), scale2, negm2);
            float y0, y1;
            unpack_f32x2(y2, y0, y1);
            const float e0 = fast_exp2(y0), e1 = fast_exp2(y1);
            ls[i & 1] = add_f32x2(ls[i & 1], pack_f32x2(e0, e1));
            pk[i] = pack_bf16x2(e0, e1);
          }
          tmem_st_32x16(t_S + g * 16, pk);
        }
      };
      // The first half's exponentials are taken with the maximum that is in use, beside the search for the tile's, and once more
      // where that has grown by more than 2^8 (a row's first tile, rarely later): the tensor core does not wait for the maximum.
#pragma unroll 1
      for (bool again = false;; again = true) {
        ls[0] = ls[1] = 0ull;
        float mx[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          mx[g] = max3(__uint_as_float(v[g][0]), __uint_as_float(v[g][1]), __uint_as_float(v[g][2]));
#pragma unroll
          for (int i = 3; i + 1 < 32; i += 2) mx[g] = max3(mx[g], __uint_as_float(v[g][i]), __uint_as_float(v[g][i + 1]));
          mx[g] = fmaxf(mx[g], __uint_as_float(v[g][31]));
        }
        half_tile(0);
        if (again) break;
        const float m_new = fmaxf(max3(mx[0], mx[1], mx[2]), fmaxf(mx[3], m_used));
        const bool need = (m_new - m_used) * p.scale_log2 > 8.f;  // also true when m_used is -inf and m_new is finite
        if (!__any_sync(0xffffffffu, need)) break;
        tmem_st_wait();  // stores to one address are in no order without it: P of the new maximum goes over the first one
        if (it > 0) {
          // lazy rescale; s_full of this tile says that the previous P V of this stream has retired
          float alpha = 1.f;
          if (need) alpha = (m_used == -INFINITY) ? 0.f : fast_exp2((m_used - m_new) * p.scale_log2);
#pragma unroll 1
          for (int cc = 0; cc < 4 * NCH; ++cc) {
            uint32_t o[16];
            tmem_ld_32x16(t_O + cc * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x16(t_O + cc * 16, o);
          }
          l_sum *= alpha;
        }
        if (need) m_used = m_new;
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[s_id * 2]);
      half_tile(1);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[s_id * 2 + 1]);
      {
        float a0, a1;
        unpack_f32x2(add_f32x2(ls[0], ls[1]), a0, a1);
        l_sum += a0 + a1;
      }
      ++it;
    }
    // ---- epilogue
    if (ok && it > 0 && !mbar_wait_abort_w(&o_full[s_id], 0, abort_flag)) {
      if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_MISC);
      *abort_flag = 1;
      ok = false;
    }
    if (ok && s_id < n_streams) {
      tc_fence_after();
      const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
      __nv_bfloat16* o_row = p.O + (long)b * p.o_stride_b + (long)q * p.o_stride_s + (long)h * p.D;
#pragma unroll
      for (int cc = 0; cc < 2 * NCH; ++cc) {
        uint32_t o[32];
        if (it > 0) {
          tmem_ld_32x32(t_O + cc * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
        }
        if (row_valid) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int col = cc * 32 + g * 8;
            if (col + 8 <= p.D) {
              float f[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] = it > 0 ? __uint_as_float(o[g * 8 + i]) * inv : 0.f;
              uint4 u;
              u.x = pack_bf16x2(f[0], f[1]);
              u.y = pack_bf16x2(f[2], f[3]);
              u.z = pack_bf16x2(f[4], f[5]);
              u.w = pack_bf16x2(f[6], f[7]);
              *reinterpret_cast<uint4*>(o_row + col) = u;
            }
          }
        }
      }
      if (row_valid)
        p.lse[((long)b * p.Hq + h) * p.Sq + q] = l_sum > 0.f ? m_used * p.scale + logf(l_sum) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace csb
