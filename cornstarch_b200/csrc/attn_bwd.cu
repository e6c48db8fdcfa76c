// Flash-attention backward for sm_100a (bitfield / causal / full masks, GQA, tile skipping).
//
// One CTA owns one 128-row K/V tile of one KV head and keeps dK and dV for it in TMEM for the
// whole kernel, looping over the query heads of the GQA group and over 64-row query tiles:
//
//   S^T  = K  Q^T              M=128(kv) N=64(q)  contraction D     -> TMEM S^T[2] (double buffer)
//   dP^T = V  dO^T             M=128     N=64     contraction D     -> TMEM dP^T
//   P^T  = exp2(S^T*c - LSE),  dS^T = P^T * (dP^T - delta) * scale   (P^T -> bf16 pairs in TMEM over S^T;
//                                                                     dS^T -> bf16 smem tile)
//   dV  += P^T  dO             M=128     N=D      contraction q=64
//   dK  += dS^T Q              M=128     N=D      contraction q=64
//   dQ^T = K^T  dS^T           M=128(d)  N=64(q)  contraction kv=128 -> TMEM dQ^T
//
// dK/dV need no atomics and are bit-reproducible: one CTA handles every query head that shares the KV head, or (small grids)
// several share the list of (query head, query tile) iterations and their fp32 parts are added in a fixed order
// (csb_attn_bwd_splits, attn_dkv_reduce_kernel).  dQ^T tiles are staged in shared memory as [q][d] rows and added into an fp32
// accumulator by TMA reduce-add (one 32 x 64 block per warp), then converted to bf16 by a final pass.
//
// Warp roles (512 threads): warp 0 = MMA issuer of S^T and dP^T, warp 1 = of dV, dK and dQ^T, warps 2 and 3 = query metadata (and
// TMA: K/V once, Q/dO ring of 3 stages), warps 4..7 = dQ^T drain, warps 8..15 = 256 compute threads.  Thread (r, group) owns KV
// row r (TMEM lane r) and 32 of the 64 query columns of S^T / dP^T; a drain thread moves head-dim row r of dQ^T.  The pipeline keeps
// S^T one iteration ahead: while the compute warps turn S^T(i), dP^T(i) into P^T, dS^T, the tensor core already holds S^T(i+1);
// dP^T(i+1) is issued as soon as dP^T(i) has been read, so the next exponentials overlap the dV/dK/dQ^T MMAs of iteration i.
// Per-tile query metadata (LSE, delta, mask rules) is staged in shared memory, a ring stage with Q / dO.
//
// What bounds it: no single unit.  Of the measured 2450 cycles of an iteration the tensor pipe is busy 1676 and the chain of
// the compute warps takes about 2000 without its waits; the MMAs read 192 KB of operands from shared memory and everything else (Q / dO in,
// dS^T, dQ through its staging, statistics) moves about 130 KB, 2500 cycles if reads and writes share a port of 128 B (counters, 4096
// tokens causal: bank reads 35 %, writes 12 %, tensor pipe 53 %, issue slots 34 % of peak).  Long runs are at the power
// cap.  Before, the one MMA warp was: 32 MMAs per iteration at 90 cycles of issue each, 3300 cycles; runs of
// MMAs (umma_f16_run_w) and a second MMA warp, which has work for the pipe while the first waits, took that away.  (dQ^T straight from
// registers by red.global, which spares its two passes through shared memory, takes 65 cycles per warp instruction: 2.0 x the time.)
// Measured with the delta and conversion passes (32 / 8 heads of 128, before -> now): 8192 tokens causal 1679 -> 1411 us (975
// TFLOP/s), full 3190 -> 2632 (1044 TFLOP/s), 4096 causal 476 -> 386, 1024 69 -> 62; 4 x 729 tokens, 16 heads of 72, 88 -> 78.
//
// Replaces cornstarch/kernel/bitfield_attention.py:526-929 (T8, T9: fp32 atomics for dQ, dK and dV)
// and cornstarch/kernel/attention.py:348-852.
#include "host.h"
#include "kv_segments.h"
#include "mask.cuh"
#include "ptx.cuh"

namespace csb {

constexpr int BW_BKV = 128;
constexpr int BW_BQ = 64;
constexpr int KV_CHUNK = 128 * 128;  // 128 rows x 128 B
constexpr int Q_CHUNK = 64 * 128;    // 64 rows x 128 B

struct AttnBwdParams {
  int B, Sq, Sk, Hq, Hk, D, dk16;
  int nQ64, nQ128, nK;
  float scale, scale_log2;
  int mask_mode;
  const int64_t* q_bits;
  const int64_t* k_bits;
  const int* q_pos;
  const int* k_pos;
  const int8_t* cls;  // [B][nQ128][nK], or null: index_tile_class decides
  const float* lse;   // [B][Hq][Sq]
  const float* delta; // [B][Hq][Sq]
  float* dq_acc;      // [B][Sq][Hq][D] fp32, zeroed by attn_delta_kernel
  __nv_bfloat16* dK[CSB_MAX_SEG];  // per key segment: where its dK / dV tiles go (possibly a peer's inbox)
  __nv_bfloat16* dV[CSB_MAX_SEG];
  long dk_stride_b[CSB_MAX_SEG], dk_stride_s[CSB_MAX_SEG], dv_stride_b[CSB_MAX_SEG], dv_stride_s[CSB_MAX_SEG];
  int* status;
  // Several blocks per key block (nsplit > 1, one local segment): block `split` takes an equal share of the iterations and
  // writes its fp32 part of dK and dV to part[0 / 1][split][B][Sk][Hk][D]; attn_dkv_reduce_kernel adds the parts in order.
  int nsplit;
  float* part;
  int kj_slowest;  // block order: 1 = key block slowest (masks that leave key blocks unequal work), 0 = key block fastest
  // dense boolean mask (MASK_DENSE) and additive bias, as in the forward kernel
  const uint8_t* dmask;
  long dm_sb, dm_sq;
  const float* bias;
  long bias_sb, bias_sh, bias_sq;
  float inv_scale;
  SegInfo seg;
};

// Position in a block's list of (query head, query tile) iterations, advanced without divisions (a division and a
// remainder per iteration on the compute warps' chain: 8192 tokens causal 1976 us with, 1903 us without).
struct BwdCursor {
  int h, t, n_valid;
  __device__ __forceinline__ BwdCursor(int it, int n) : h(n > 0 ? it / n : 0), t(n > 0 ? it % n : 0), n_valid(n) {}
  __device__ __forceinline__ void next() {
    if (++t == n_valid) {
      t = 0;
      ++h;
    }
  }
};

struct BwdSmem {
  static constexpr int QSTAGES = 3;
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = K_OFF + 2 * KV_CHUNK;
  static constexpr int Q_OFF = V_OFF + 2 * KV_CHUNK;          // QSTAGES x (2 chunks x 8 KB)
  static constexpr int DO_OFF = Q_OFF + QSTAGES * 2 * Q_CHUNK;
  static constexpr int DST_OFF = DO_OFF + QSTAGES * 2 * Q_CHUNK;  // dS^T [128 kv][64 q] bf16
  static constexpr int DQ_OFF = DST_OFF + KV_CHUNK;           // dQ staging: 4 warps x [64 q][32 d] fp32 (row-major, 8 KB each)
  static constexpr int META_OFF = DQ_OFF + 8 * 4096;          // one buffer per Q stage of: -lse2[64] f32, -delta*scale[64] f32, and the mask rules lim[64] i32, am[64] i64, qe[64] i64
  static constexpr int META_STAGE = 64 * 4 * 3 + 2 * 64 * 8;
  static constexpr int LIST_OFF = META_OFF + QSTAGES * META_STAGE;  // valid 64-row query tiles of this key block: int16 index, int8 class
  static constexpr int MAX_TILES = 1024;                      // sequences up to 65536 tokens
  static constexpr int BAR_OFF = LIST_OFF + MAX_TILES * 4;
  static constexpr int NBAR = 1 + QSTAGES + QSTAGES + 5;
  static constexpr int TOTAL = BAR_OFF + NBAR * 8 + 32;
  static constexpr int DYN_BYTES = TOTAL + 1024;
};

// Eight compute warps: two share a TMEM lane quarter and split the 64 query columns between them.  What does not depend on the
// number of columns (waits, addresses, arrivals of every thread) is on their chain once per warp of a scheduler: sixteen warps of 16
// columns took 1903 us where eight of 32 took 1816 (8192 tokens causal, with the MMA warp as the limit).
struct BwdCfg {
  static constexpr int COMPUTE_THREADS = 8 * 32;
  static constexpr int DRAIN_THREADS = 128;  // four warps that only move dQ^T out (one per TMEM lane quarter)
  static constexpr int THREADS = 128 + DRAIN_THREADS + COMPUTE_THREADS;
  static constexpr int GROUPS = 2;             // column groups
  static constexpr int COLS = BW_BQ / GROUPS;  // query columns of S^T / dP^T per thread
};

// delta[b][h][q] = sum_d O[b][q][h][d] * dO[b][q][h][d].  Sixteen lanes share a row (8 elements each, D <= 128) and take
// DELTA_ROWS queries of one head, so that every thread has 2 x DELTA_ROWS 16-byte loads in flight and the results of a block
// are consecutive.  VEC: rows of both tensors start on 16-byte boundaries.
// The same threads write the zeros that the dQ accumulator starts from: one launch and one fill less in front of each call, which
// small calls are bound by (issued and run one by one: 333 tokens causal, 32 / 8 heads of 128, 54 -> 46 us; 4 x 729 tokens, 16 heads
// of 72, 110 -> 105; long sequences unchanged).
// (A warp per row with 4-byte loads took 13.7 us for the 13 MB of 4 x 729 tokens, 16 heads of 72; the whole backward call went
// from 124 to 112 us with this pass, the conversion below and the statistics warps.)
constexpr int DELTA_ROWS = 4;
template <bool VEC>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ dO, float* __restrict__ delta,
                  float* __restrict__ dq_acc, int Sq, int Hq, int D, long o_sb, long o_ss, long do_sb, long do_ss) {
  const int lane16 = threadIdx.x & 15, row = threadIdx.x >> 4;
  const int n_qb = (Sq + 16 * DELTA_ROWS - 1) / (16 * DELTA_ROWS);
  const int hb = blockIdx.x / n_qb;
  const int h = hb % Hq, b = hb / Hq;
  const int q0 = (blockIdx.x - hb * n_qb) * (16 * DELTA_ROWS) + row;
  const int c = lane16 * 8;
  uint4 uo[DELTA_ROWS], ud[DELTA_ROWS];
#pragma unroll
  for (int i = 0; i < DELTA_ROWS; ++i) {
    const int q = q0 + i * 16;
    uo[i] = ud[i] = make_uint4(0u, 0u, 0u, 0u);
    if (q < Sq && c < D) {
      const __nv_bfloat16* o = O + b * o_sb + (long)q * o_ss + (long)h * D + c;
      const __nv_bfloat16* d = dO + b * do_sb + (long)q * do_ss + (long)h * D + c;
      if constexpr (VEC) {
        uo[i] = *reinterpret_cast<const uint4*>(o);
        ud[i] = *reinterpret_cast<const uint4*>(d);
      } else {
        __align__(16) __nv_bfloat16 to[8], td[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          to[j] = o[j];
          td[j] = d[j];
        }
        uo[i] = *reinterpret_cast<const uint4*>(to);
        ud[i] = *reinterpret_cast<const uint4*>(td);
      }
      float4* z = reinterpret_cast<float4*>(dq_acc + (((long)b * Sq + q) * Hq + h) * D + c);
      z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
#pragma unroll
  for (int i = 0; i < DELTA_ROWS; ++i) {
    const uint32_t wo[4] = {uo[i].x, uo[i].y, uo[i].z, uo[i].w}, wd[4] = {ud[i].x, ud[i].y, ud[i].z, ud[i].w};
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc += __uint_as_float(wo[j] << 16) * __uint_as_float(wd[j] << 16);
      acc += __uint_as_float(wo[j] & 0xffff0000u) * __uint_as_float(wd[j] & 0xffff0000u);
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    const int q = q0 + i * 16;
    if (lane16 == 0 && q < Sq) delta[((long)b * Hq + h) * Sq + q] = acc;
  }
}

// dq (bf16, strided) = dq_acc (fp32, dense [B][Sq][Hq][D]); a thread owns 8 columns (blockIdx.x) and walks the token rows.
// VEC: rows of dq start on 16-byte boundaries (8-byte boundaries otherwise).
template <bool VEC>
__global__ void __launch_bounds__(256)
attn_dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long n_rows, int Sq, int HD, long dq_sb, long dq_ss) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= HD) return;
#pragma unroll 2
  for (long row = blockIdx.y; row < n_rows; row += gridDim.y) {
    const int q = row % Sq;
    const long b = row / Sq;
    const float4 f = __ldcs(reinterpret_cast<const float4*>(acc + row * HD + c));
    const float4 g = __ldcs(reinterpret_cast<const float4*>(acc + row * HD + c + 4));
    uint4 u;
    u.x = pack_bf16x2(f.x, f.y);
    u.y = pack_bf16x2(f.z, f.w);
    u.z = pack_bf16x2(g.x, g.y);
    u.w = pack_bf16x2(g.z, g.w);
    __nv_bfloat16* dst = dq + b * dq_sb + (long)q * dq_ss + c;
    if constexpr (VEC) {
      *reinterpret_cast<uint4*>(dst) = u;
    } else {
      *reinterpret_cast<uint2*>(dst) = make_uint2(u.x, u.y);
      *reinterpret_cast<uint2*>(dst + 4) = make_uint2(u.z, u.w);
    }
  }
}

// EXTRAS: the form with a dense boolean mask and / or an additive bias (their code and registers stay out of the other one).
template <bool EXTRAS>
__global__ void __launch_bounds__(BwdCfg::THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ KvMaps kvm,
                const __grid_constant__ CUtensorMap tm_do, const __grid_constant__ CUtensorMap tm_dq,
                const AttnBwdParams p) {
  using L = BwdSmem;
  using CFG = BwdCfg;
  constexpr int QS = L::QSTAGES;
  constexpr int COLS = CFG::COLS;
  static_assert(COLS == 32, "a thread's columns are one 32-column tensor-memory load");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;            // [QS]  Q + dO stage landed
  uint64_t* q_empty = q_full + QS;        // [QS]  stage consumed by the dV/dK MMAs (and P^T by dV)
  uint64_t* sdp_full = q_empty + QS;      //       S^T and dP^T of an iteration ready in TMEM
  uint64_t* pds_full = sdp_full + 1;      //       P^T and dS^T tiles written (256 arrivals)
  uint64_t* dq_full = pds_full + 1;       //       dQ^T ready in TMEM, P^T and dS^T consumed: the iteration's last MMAs have retired
  uint64_t* dq_free = dq_full + 1;        //       dQ^T drained (128 arrivals)
  uint64_t* dp_read = dq_free + 1;      //       S^T and dP^T of an iteration are in registers (256 arrivals): dP^T may be overwritten
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + L::NBAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* n_valid_slot = reinterpret_cast<int*>(tmem_slot + 2);
  int* peer_ok_slot = reinterpret_cast<int*>(tmem_slot + 3);
  int16_t* tile_idx = reinterpret_cast<int16_t*>(smem + L::LIST_OFF);
  int8_t* tile_cls = reinterpret_cast<int8_t*>(smem + L::LIST_OFF + L::MAX_TILES * 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // One-dimensional grid, key block slowest: under causal masks the first key blocks meet the most query tiles, so
  // the heavy blocks of every head start first and the light ones fill the tail.
  // (With a full mask every block is equally heavy; key block fastest then keeps the Q / dO tiles of few heads in L2.)
  const int n_hb = p.Hk * p.B;
  const int split = blockIdx.x % p.nsplit;
  const int blk = blockIdx.x / p.nsplit;
  const int hb = p.kj_slowest ? blk % n_hb : blk / p.nK;
  const int kj = p.kj_slowest ? blk / n_hb : blk % p.nK;
  const int hk = hb % p.Hk, b = hb / p.Hk;
  const int group = p.Hq / p.Hk;
  const int k0 = kj * BW_BKV;                              // index into k_bits / k_pos (padded gathered space)
  const int sg = seg_of_tile(p.seg, kj);                   // which K/V segment (rank) this key block belongs to
  const int row0 = (kj - p.seg.tile_start[sg]) * BW_BKV;   // first row of the block inside that segment

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < QS; ++i) {
      mbar_init(&q_full[i], 1 + BW_BQ);  // the TMA thread and the 64 metadata threads
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(sdp_full, 1);
    mbar_init(pds_full, CFG::COMPUTE_THREADS);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, CFG::DRAIN_THREADS);
    mbar_init(dp_read, CFG::COMPUTE_THREADS);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    // list of the 64-row query tiles that have at least one allowed pair with this key block (ordered compaction)
    int n = 0;
    for (int base = 0; base < p.nQ64 && n < L::MAX_TILES; base += 32) {
      const int i = base + lane;
      int8_t c = 0;
      if (i < p.nQ64)
        c = p.cls != nullptr ? p.cls[((long)b * p.nQ128 + (i >> 1)) * p.nK + kj]
                             : static_cast<int8_t>(index_tile_class(p.mask_mode, i >> 1, kj, p.Sq, p.Sk));
      const uint32_t m = __ballot_sync(0xffffffffu, c != 0);
      const int pos = n + __popc(m & ((1u << lane) - 1u));
      if (c != 0 && pos < L::MAX_TILES) {
        tile_idx[pos] = static_cast<int16_t>(i);
        tile_cls[pos] = c;
      }
      n += __popc(m);
    }
    if (lane == 0) {
      *n_valid_slot = n < L::MAX_TILES ? n : L::MAX_TILES;
      // A key block of a peer: nothing of this CTA may touch that rank's memory (loads of K/V, stores of dK/dV
      // into its inbox) before the rank has staged its K/V, which also means it is done with its previous inbox.
      int ok = 1;
      if (p.seg.ready_flags != nullptr && sg != p.seg.my_seg) {
        ok = wait_peer_flag(p.seg.ready_flags + sg, p.seg.ready_value) ? 1 : 0;
        if (!ok) atomicCAS(p.status, 0, ST_TIMEOUT_PEER_FLAG);
      }
      *peer_ok_slot = ok;
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_valid = *n_valid_slot;
  const bool peer_ready = *peer_ok_slot != 0;
  // this block's share [it0, it0 + n_iter) of the (query head, query tile) list
  const int n_all = peer_ready ? n_valid * group : 0;
  const int it0 = (int)((long)n_all * split / p.nsplit);
  const int n_iter = (int)((long)n_all * (split + 1) / p.nsplit) - it0;
  // TMEM columns: S^T[0] 0..63, S^T[1] 64..127, dP^T 128..191, dQ^T 192..255, dV 256..383, dK 384..511
  const uint32_t tmem_dPT = tmem_base + 128;
  const uint32_t tmem_dQT = tmem_base + 192;
  const uint32_t tmem_dV = tmem_base + 256;
  const uint32_t tmem_dK = tmem_base + 384;

  // The MMAs come from two warps, so that the pipe has work of one while the other waits for a hand-over: warp 0 issues S^T and dP^T,
  // warp 1 dV, dK and dQ^T.  Whole warps walk this code in step (every lane waits on the barriers; one elected lane issues each run of
  // MMAs and its commit).
  if (warp == 0) {
    // ------------------------------------------------------------------ S^T and dP^T
    const uint32_t idesc_s = make_idesc_bf16(128, BW_BQ, 0, 0);
    const uint64_t k_km = make_desc_kmajor_sw128(smem_u32(smem + L::K_OFF));
    const uint64_t v_km = make_desc_kmajor_sw128(smem_u32(smem + L::V_OFF));
    const uint64_t q_km = make_desc_kmajor_sw128(smem_u32(smem + L::Q_OFF));
    const uint64_t do_km = make_desc_kmajor_sw128(smem_u32(smem + L::DO_OFF));
    constexpr uint64_t STAGE = (2 * Q_CHUNK) >> 4;
    const int ksteps_d = p.dk16 / 16;
    bool ok = n_iter == 0 || mbar_wait_abort_w(kv_full, 0, abort_flag);
    if (!ok) { atomicCAS(p.status, 0, ST_TIMEOUT_FULL); *abort_flag = 1; }
    int s_stage = 0, d_stage = 0;  // ring stages of the next S^T and dP^T
    uint32_t s_phase = 0;
    auto issue_st = [&](int it) -> bool {  // into ST[it & 1]; waits for the Q / dO stage of that iteration
      if (!mbar_wait_abort_w(&q_full[s_stage], s_phase, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_FULL); *abort_flag = 1; return false; }
      tc_fence_after();
      umma_f16_run_w(tmem_base + (it & 1) * 64, k_km, q_km + s_stage * STAGE, KV_CHUNK, Q_CHUNK, idesc_s, ksteps_d, 0u);
      if (++s_stage == QS) { s_stage = 0; s_phase ^= 1u; }
      return true;
    };
    auto issue_dpt = [&]() {  // its commit also covers S^T of the iteration, issued earlier
      umma_f16_run_w(tmem_dPT, v_km, do_km + d_stage * STAGE, KV_CHUNK, Q_CHUNK, idesc_s, ksteps_d, 0u);
      umma_commit_w(sdp_full);
      if (++d_stage == QS) d_stage = 0;
    };
    if (ok && n_iter > 0) {
      ok = issue_st(0);
      if (ok) issue_dpt();
      if (ok && n_iter > 1) ok = issue_st(1);
    }
    int e_stage = 0;  // iteration it's stage and phase
    uint32_t e_phase = 0;
    for (int it = 0; ok && it + 1 < n_iter; ++it) {
      // dP^T(it + 1) as soon as the compute warps hold dP^T(it) in registers, long before they are done with the iteration
      if (!mbar_wait_abort_w(dp_read, it & 1, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_MISC); *abort_flag = 1; break; }
      tc_fence_after();
      issue_dpt();
      if (it + 2 < n_iter) {
        // S^T(it + 2) goes over P^T(it): dV(it) has to have retired, which is what releases the stage of iteration it
        if (!mbar_wait_abort_w(&q_empty[e_stage], e_phase, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_EMPTY); *abort_flag = 1; break; }
        if (++e_stage == QS) { e_stage = 0; e_phase ^= 1u; }
        ok = issue_st(it + 2);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ dV, dK and dQ^T
    const uint32_t idesc_dkv = make_idesc_bf16(128, p.dk16, 0, 1);
    const uint32_t idesc_dq = make_idesc_bf16(128, BW_BQ, 1, 1);
    const uint64_t k_mn = make_desc_mnmajor_sw128(smem_u32(smem + L::K_OFF), KV_CHUNK);
    const uint64_t q_mn = make_desc_mnmajor_sw128(smem_u32(smem + L::Q_OFF), Q_CHUNK);
    const uint64_t do_mn = make_desc_mnmajor_sw128(smem_u32(smem + L::DO_OFF), Q_CHUNK);
    const uint64_t dst_km = make_desc_kmajor_sw128(smem_u32(smem + L::DST_OFF));
    const uint64_t dst_mn = make_desc_mnmajor_sw128(smem_u32(smem + L::DST_OFF), KV_CHUNK);
    constexpr uint64_t STAGE = (2 * Q_CHUNK) >> 4;
    int st = 0;
    uint32_t st_phase = 0;
    bool ok = n_iter == 0 || mbar_wait_abort_w(kv_full, 0, abort_flag);
    if (!ok) { atomicCAS(p.status, 0, ST_TIMEOUT_FULL); *abort_flag = 1; }
    for (int it = 0; ok && it < n_iter; ++it) {
      // (the stage is full long before; the wait orders this warp's MMAs behind the copies)
      if (!mbar_wait_abort_w(&q_full[st], st_phase, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_FULL); *abort_flag = 1; break; }
      if (!mbar_wait_abort_w(pds_full, it & 1, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_MISC); *abort_flag = 1; break; }
      tc_fence_after();
      // dV += P^T dO ; dK += dS^T Q   (contraction over the 64 query rows)
      const uint32_t acc = it > 0 ? 1u : 0u;
      umma_f16_ts_run4_w<COLS>(tmem_dV, tmem_base + (it & 1) * 64, do_mn + st * STAGE, idesc_dkv, acc);
      umma_f16_run4_w<2, 128>(tmem_dK, dst_km, q_mn + st * STAGE, idesc_dkv, acc);  // 16 columns of dS^T, 16 rows of Q a step
      umma_commit_w(&q_empty[st]);
      if (it > 0) {
        if (!mbar_wait_abort_w(dq_free, (it - 1) & 1, abort_flag)) { atomicCAS(p.status, 0, ST_TIMEOUT_TMEM_EMPTY); *abort_flag = 1; break; }
        tc_fence_after();
      }
      // dQ^T = K^T dS^T  (contraction over the 128 key rows)
      umma_f16_run8_w<128, 128>(tmem_dQT, k_mn, dst_mn, idesc_dq, 0u);  // 16 rows of K and of dS^T a step
      umma_commit_w(dq_full);
      if (++st == QS) { st = 0; st_phase ^= 1u; }
    }
    __syncwarp();
  } else if (warp < 4) {
    // ------------------------------------------------------------------ TMA producer and query metadata (warps 2 and 3)
    // Statistics and mask rules of the stage's 64 query rows, one row a thread and one ring stage with its Q / dO tiles, which lane 0
    // of warp 2 loads.  (When two of the compute warps loaded them on the side, every iteration waited for their global loads: 1400 of
    // its 3700 cycles.)
    const float LOG2E = 1.4426950408889634f;
    const int r = (warp - 2) * 32 + lane;
    const bool producer = warp == 2 && lane == 0;
    if (producer) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_do);
      if (n_iter > 0) {  // (a block without iterations only writes zeros)
        mbar_expect_tx(kv_full, 4 * KV_CHUNK);
        for (int c = 0; c < 2; ++c) {
          tma_load_4d(smem + L::K_OFF + c * KV_CHUNK, &kvm.k[sg], kv_full, c * 64, hk, row0, b);
          tma_load_4d(smem + L::V_OFF + c * KV_CHUNK, &kvm.v[sg], kv_full, c * 64, hk, row0, b);
        }
      }
    }
    BwdCursor cur(it0, n_valid);
    int st = 0;
    uint32_t st_phase = 1;
    for (int it = 0; it < n_iter; ++it, cur.next()) {
      const int h = hk * group + cur.h;
      const int qt = tile_idx[cur.t];
      const int q = qt * BW_BQ + r;
      const bool qv = q < p.Sq;
      const long idx = ((long)b * p.Hq + h) * p.Sq + q;
      const float lse = qv ? p.lse[idx] : INFINITY;
      const float delta = qv ? p.delta[idx] : 0.f;
      const int qpos = qv ? (p.q_pos ? p.q_pos[(long)b * p.Sq + q] : q) : 0;
      const int64_t qbits = (qv && p.q_bits) ? p.q_bits[(long)b * p.Sq + q] : 0;
      if (!mbar_wait_abort_w(&q_empty[st], st_phase, abort_flag)) {
        if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_EMPTY);
        *abort_flag = 1;
        break;
      }
      if (producer) {
        mbar_expect_tx(&q_full[st], 4 * Q_CHUNK);
        for (int c = 0; c < 2; ++c) {
          tma_load_4d(smem + L::Q_OFF + (st * 2 + c) * Q_CHUNK, &tm_q, &q_full[st], c * 64, h, qt * BW_BQ, b);
          tma_load_4d(smem + L::DO_OFF + (st * 2 + c) * Q_CHUNK, &tm_do, &q_full[st], c * 64, h, qt * BW_BQ, b);
        }
      }
      __syncwarp();
      const QueryRule rule = make_query_rule(p.mask_mode, qv && qpos >= 0, qbits, qpos);
      float* m = reinterpret_cast<float*>(smem + L::META_OFF + st * L::META_STAGE);
      m[r] = -(lse * LOG2E);  // both negated: their uses are one packed FMA each
      m[64 + r] = -(delta * p.scale);
      reinterpret_cast<int*>(m + 128)[r] = rule.lim;
      reinterpret_cast<int64_t*>(m + 192)[r] = rule.am;
      reinterpret_cast<int64_t*>(m + 320)[r] = rule.qe;
      mbar_arrive(&q_full[st]);
      if (++st == QS) { st = 0; st_phase ^= 1u; }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------------ compute threads (8 warps)
    const int cw = warp - 8;
    const int quarter = warp & 3;       // TMEM lane quarter this warp may touch
    const int half = cw >> 2;           // which group of COLS query columns (of 64) this warp handles
    const int r = quarter * 32 + lane;  // KV row in the tile == TMEM lane; also head-dim row of dQ^T
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int col0 = half * COLS;
    const int kidx = k0 + r;
    const int krow = row0 + r;  // row inside the segment
    const bool k_valid = krow < p.seg.rows[sg];
    const int kpos = k_valid ? (p.k_pos ? p.k_pos[(long)b * p.Sk + kidx] : kidx) : -1;  // negative: a key that does not exist
    const int64_t kb = mask_key_bits(p.mask_mode, kpos >= 0, (k_valid && p.k_bits) ? p.k_bits[(long)b * p.Sk + kidx] : 0);
    const uint64_t scale_log2_2 = pack_f32x2(p.scale_log2, p.scale_log2), scale_2 = pack_f32x2(p.scale, p.scale);
    const bool by_index = mask_by_index(p.mask_mode, p.q_pos, p.k_pos);
    bool ok = true;
    // The statistics and mask rules of iteration it (buffer it % QS) were staged before its Q / dO stage counted as full, so
    // sdp_full(it) covers them too.
    BwdCursor cur(it0, n_valid);
    int stage = 0;  // it % QS
    int c_next = n_iter > 0 ? tile_cls[cur.t] : 0, qt_next = n_iter > 0 ? tile_idx[cur.t] : 0;
    for (int it = 0; it < n_iter && ok; ++it, stage = stage + 1 == QS ? 0 : stage + 1) {
      const int c = c_next, qt = qt_next;
      const int head = cur.h;
      cur.next();  // (of the tile after the last one nothing is used)
      c_next = tile_cls[cur.t];
      qt_next = tile_idx[cur.t];
      float* m_lse = reinterpret_cast<float*>(smem + L::META_OFF + stage * L::META_STAGE);
      float* m_delta = m_lse + 64;
      const int* m_lim = reinterpret_cast<const int*>(m_lse + 128);
      const int64_t* m_am = reinterpret_cast<const int64_t*>(m_lse + 192);
      const int64_t* m_qe = reinterpret_cast<const int64_t*>(m_lse + 320);
      const int q_base = qt * BW_BQ + col0;  // first query row of this thread's columns
      // Mask bytes and biases of this thread's pairs, all loaded before the wait for the scores: rows that do not exist are
      // clamped, not branched around, so that the loads of the COLS columns are in flight together.
      uint32_t mask_word = 0xffffffffu;
      float bias_v[EXTRAS ? COLS : 1];
      if constexpr (EXTRAS) {
        const long q_first = min(q_base, p.Sq - 1), k_at = min(kidx, p.Sk - 1);
        uint32_t mb[COLS];
        const bool masked = c == 1 && p.mask_mode == MASK_DENSE;
        if (masked) {
          const uint8_t* m = p.dmask + (long)b * p.dm_sb + q_first * p.dm_sq + k_at;
#pragma unroll
          for (int x = 0; x < COLS; ++x) {
            mb[x] = __ldg(m);
            m += q_base + x + 1 < p.Sq ? p.dm_sq : 0;
          }
        }
        if (p.bias != nullptr) {
          const float* v = p.bias + (long)b * p.bias_sb + (long)(hk * group + head) * p.bias_sh + q_first * p.bias_sq + k_at;
#pragma unroll
          for (int x = 0; x < COLS; ++x) {
            bias_v[x] = __ldg(v);
            v += q_base + x + 1 < p.Sq ? p.bias_sq : 0;
          }
        }
        if (masked) {
          mask_word = 0u;
#pragma unroll
          for (int x = 0; x < COLS; ++x) mask_word |= (mb[x] != 0u ? 1u : 0u) << x;
        }
      }
      if (!mbar_wait_abort_w(sdp_full, it & 1, abort_flag)) {
        if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t sv[COLS], dv[COLS];
      tmem_ld_32x32(tmem_base + (it & 1) * 64 + col0 + lane_addr, sv);
      if constexpr (EXTRAS) {
        if (p.bias != nullptr) {  // folded in before dP^T is loaded: the biases' registers are free again
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < COLS; ++x)
            sv[x] = __float_as_uint(fmaf(q_base + x < p.Sq && k_valid ? bias_v[x] : 0.f, p.inv_scale, __uint_as_float(sv[x])));
        }
      }
      tmem_ld_32x32(tmem_dPT + col0 + lane_addr, dv);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(dp_read);
      float pv[COLS], ds[COLS];
#pragma unroll
      for (int x4 = 0; x4 < COLS / 4; ++x4) {
        const float4 l4 = *reinterpret_cast<const float4*>(m_lse + col0 + x4 * 4);
        float y0, y1, y2, y3;
        unpack_f32x2(fma_f32x2(pack_u32x2(sv[x4 * 4], sv[x4 * 4 + 1]), scale_log2_2, pack_f32x2(l4.x, l4.y)), y0, y1);
        unpack_f32x2(fma_f32x2(pack_u32x2(sv[x4 * 4 + 2], sv[x4 * 4 + 3]), scale_log2_2, pack_f32x2(l4.z, l4.w)), y2, y3);
        pv[x4 * 4] = fast_exp2(y0);
        pv[x4 * 4 + 1] = fast_exp2(y1);
        pv[x4 * 4 + 2] = fast_exp2(y2);
        pv[x4 * 4 + 3] = fast_exp2(y3);
      }
      if (c == 1) {
        if (EXTRAS && p.mask_mode == MASK_DENSE) {
          const uint32_t allow = k_valid ? mask_word : 0u;
#pragma unroll
          for (int x = 0; x < COLS; ++x) pv[x] = ((allow >> x) & 1u) && q_base + x < p.Sq ? pv[x] : 0.f;
        } else if (by_index) {
          // token indices alone decide (queries beyond Sq already have P = 0 through their statistics)
          const int first = !k_valid ? COLS : (p.mask_mode == MASK_CAUSAL ? kidx - q_base : 0);
#pragma unroll
          for (int x = 0; x < COLS; ++x) pv[x] = x >= first ? pv[x] : 0.f;
        } else {
#pragma unroll
          for (int x = 0; x < COLS; ++x) {
            const int col = col0 + x;
            pv[x] = rule_allows(QueryRule{m_am[col], m_qe[col], m_lim[col]}, kb, kpos) ? pv[x] : 0.f;
          }
        }
      }
      // P^T -> packed bf16 pairs in tensor memory, over this thread's own S^T columns (the first half of them)
      {
        uint32_t pk[COLS / 2];
#pragma unroll
        for (int x = 0; x < COLS / 2; ++x) pk[x] = pack_bf16x2(pv[2 * x], pv[2 * x + 1]);
        tmem_st_32x16(tmem_base + (it & 1) * 64 + col0 + lane_addr, pk);
      }
#pragma unroll
      for (int x4 = 0; x4 < COLS / 4; ++x4) {
        const float4 d4 = *reinterpret_cast<const float4*>(m_delta + col0 + x4 * 4);
        const uint64_t t0 = fma_f32x2(pack_u32x2(dv[x4 * 4], dv[x4 * 4 + 1]), scale_2, pack_f32x2(d4.x, d4.y));
        const uint64_t t1 = fma_f32x2(pack_u32x2(dv[x4 * 4 + 2], dv[x4 * 4 + 3]), scale_2, pack_f32x2(d4.z, d4.w));
        unpack_f32x2(mul_f32x2(pack_f32x2(pv[x4 * 4], pv[x4 * 4 + 1]), t0), ds[x4 * 4], ds[x4 * 4 + 1]);
        unpack_f32x2(mul_f32x2(pack_f32x2(pv[x4 * 4 + 2], pv[x4 * 4 + 3]), t1), ds[x4 * 4 + 2], ds[x4 * 4 + 3]);
      }
      if (it > 0) {
        if (!mbar_wait_abort_w(dq_full, (it - 1) & 1, abort_flag)) {
          if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_MISC);
          *abort_flag = 1;
          ok = false;
          break;
        }
      }
      // dS^T -> bf16 smem tile: row r, this warp's 16-byte pieces (8 query columns each)
#pragma unroll
      for (int pc = 0; pc < COLS / 8; ++pc) {
        uint4 w;
        w.x = pack_bf16x2(ds[pc * 8 + 0], ds[pc * 8 + 1]);
        w.y = pack_bf16x2(ds[pc * 8 + 2], ds[pc * 8 + 3]);
        w.z = pack_bf16x2(ds[pc * 8 + 4], ds[pc * 8 + 5]);
        w.w = pack_bf16x2(ds[pc * 8 + 6], ds[pc * 8 + 7]);
        *reinterpret_cast<uint4*>(smem + L::DST_OFF + sw128_offset(r, half * (COLS / 8) + pc)) = w;
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(pds_full);
    }
    // ---- epilogue: dV and dK tiles (every MMA has retired once the last dS^T was consumed); the warps of a lane quarter split
    //      the head-dim columns
    if (ok && n_iter > 0 && !mbar_wait_abort_w(dq_full, (n_iter - 1) & 1, abort_flag)) {
      if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_MISC);
      *abort_flag = 1;
      ok = false;
    }
    if (ok && peer_ready) {
      tc_fence_after();
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const uint32_t t = which == 0 ? tmem_dV : tmem_dK;
        __nv_bfloat16* base = which == 0
                                  ? p.dV[sg] + (long)b * p.dv_stride_b[sg] + (long)krow * p.dv_stride_s[sg] + (long)hk * p.D
                                  : p.dK[sg] + (long)b * p.dk_stride_b[sg] + (long)krow * p.dk_stride_s[sg] + (long)hk * p.D;
#pragma unroll
        for (int c2 = 0; c2 < 4 / CFG::GROUPS; ++c2) {
          const int cc = half * (4 / CFG::GROUPS) + c2;
          uint32_t v[32];
          if (n_iter > 0) {
            tmem_ld_32x32(t + cc * 32 + lane_addr, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int x = 0; x < 32; ++x) v[x] = 0u;
          }
          if (k_valid && p.nsplit > 1) {
            float* dst = p.part + ((((long)(which == 0 ? 1 : 0) * p.nsplit + split) * p.B + b) * p.Sk + kidx) * p.Hk * p.D + (long)hk * p.D;
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              const int col = cc * 32 + g * 4;
              if (col + 4 <= p.D)
                *reinterpret_cast<float4*>(dst + col) = make_float4(__uint_as_float(v[g * 4]), __uint_as_float(v[g * 4 + 1]),
                                                                    __uint_as_float(v[g * 4 + 2]), __uint_as_float(v[g * 4 + 3]));
            }
          } else if (k_valid) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int col = cc * 32 + g * 8;
              if (col + 8 <= p.D) {
                uint4 u;
                u.x = pack_bf16x2(__uint_as_float(v[g * 8 + 0]), __uint_as_float(v[g * 8 + 1]));
                u.y = pack_bf16x2(__uint_as_float(v[g * 8 + 2]), __uint_as_float(v[g * 8 + 3]));
                u.z = pack_bf16x2(__uint_as_float(v[g * 8 + 4]), __uint_as_float(v[g * 8 + 5]));
                u.w = pack_bf16x2(__uint_as_float(v[g * 8 + 6]), __uint_as_float(v[g * 8 + 7]));
                *reinterpret_cast<uint4*>(base + col) = u;
              }
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dQ^T drain: TMEM -> smem [q][d] rows -> reduce-add
    // Warps of their own, so that the compute warps go straight from dS^T(it) to S^T(it + 1): with the drain in their loop
    // the next exponentials waited for the tensor-memory loads and staging stores of an iteration that was long over.
    const int quarter = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    float* stage = reinterpret_cast<float*>(smem + L::DQ_OFF + quarter * (BW_BQ * 128));
    BwdCursor cur(it0, n_valid);
    for (int it = 0; it < n_iter; ++it, cur.next()) {
      if (!mbar_wait_abort_w(dq_full, it & 1, abort_flag)) {
        if (lane == 0) atomicCAS(p.status, 0, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      if (lane == 0) tma_store_wait_read<0>();  // the previous block has left the staging buffer
      __syncwarp();
      // this warp's [32 d][64 q] block -> shared memory as [q][d] rows of 128 B -> one TMA reduce-add into dq_acc
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t v[32];
        tmem_ld_32x32(tmem_dQT + g * 32 + lane_addr, v);
        tmem_ld_wait();
        if (g == 1) {
          tc_fence_before();
          mbar_arrive(dq_free);
        }
#pragma unroll
        for (int c = 0; c < 32; ++c) stage[(g * 32 + c) * 32 + lane] = __uint_as_float(v[c]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0 && quarter * 32 < p.D) {
        tma_reduce_add_4d(&tm_dq, stage, quarter * 32, hk * group + cur.h, tile_idx[cur.t] * BW_BQ, b);  // box: 32 d x 64 q
        tma_store_commit();
      }
    }
    if (lane == 0) tma_store_wait<0>();  // every reduce-add of this warp has completed
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// dK (blockIdx.z = 0) / dV (1) = sum over the splits, in order, of their fp32 parts [split][rows][HD], rounded to bf16 once.
// A thread owns 8 columns; the parts are dense, the results strided.
__global__ void __launch_bounds__(128)
attn_dkv_reduce_kernel(const float* __restrict__ part, int nsplit, long n_rows, int Sk, int HD, __nv_bfloat16* __restrict__ dk,
                       __nv_bfloat16* __restrict__ dv, long dk_sb, long dk_ss, long dv_sb, long dv_ss) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c >= HD) return;
  const float* src = part + (long)blockIdx.z * nsplit * n_rows * HD;
  for (long row = blockIdx.y; row < n_rows; row += gridDim.y) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int sp = 0; sp < nsplit; ++sp) {
      const float* q = src + ((long)sp * n_rows + row) * HD + c;
      const float4 f = *reinterpret_cast<const float4*>(q), g = *reinterpret_cast<const float4*>(q + 4);
      acc[0] += f.x; acc[1] += f.y; acc[2] += f.z; acc[3] += f.w;
      acc[4] += g.x; acc[5] += g.y; acc[6] += g.z; acc[7] += g.w;
    }
    const long b = row / Sk, k = row - b * Sk;
    __nv_bfloat16* dst = (blockIdx.z == 0 ? dk + b * dk_sb + k * dk_ss : dv + b * dv_sb + k * dv_ss) + c;
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                                                pack_bf16x2(acc[6], acc[7]));
  }
}

static int make_tmap_4d(CUtensorMap* tm, const void* base, int D, int H, int S, int B, long stride_s, long stride_b,
                        int box_rows) {
  uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  uint64_t strides[3] = {(uint64_t)D * 2, (uint64_t)stride_s * 2, (uint64_t)stride_b * 2};
  uint32_t box[4] = {64, 1, (uint32_t)box_rows, 1};
  return make_tmap_nd_bf16(tm, base, 4, dims, strides, box);
}

}  // namespace csb

using namespace csb;

// q / out / dout / dq are [B][Sq][Hq][D] bf16 views (head stride D; token / batch strides in elements); keys and values
// come as segments (kv_segments.h) and the dK / dV tiles of segment r are written to kv->dk[r] / kv->dv[r].
// lse: fp32 [B][Hq][Sq] from the forward; delta: fp32 [B][Hq][Sq] scratch; dq_acc: fp32 dense [B][Sq][Hq][D] scratch
// (16-byte aligned; its contents do not matter).  Sk = padded gathered length; cls: tile classes for 128x128 tiles.
// Optional inputs of the dense-mask / bias form (same layout as in attn_fwd.cu).
struct CsbAttnExtras {
  const unsigned char* dmask;
  long dm_sb, dm_sq;
  const float* bias;
  long bias_sb, bias_sh, bias_sq;
};

static int attn_bwd_seg_impl(const void* q, const CsbKvSegments* kv, const void* out, const void* dout, const float* lse,
                             float* delta, float* dq_acc, void* dq, int B, int Sq, int Sk, int Hq, int Hk, int D, long q_ss,
                             long q_sb, long o_ss, long o_sb, long do_ss, long do_sb, long dq_ss, long dq_sb, float scale,
                             int mask_mode, const long* q_bits, const long* k_bits, const int* q_pos, const int* k_pos,
                             const signed char* cls, int* status, void* stream, const CsbAttnExtras* ex, float* part = nullptr,
                             int nsplit = 1) {
  if (nsplit < 1 || (nsplit > 1 && (part == nullptr || kv == nullptr || kv->n_seg != 1 || kv->ready_flags != nullptr))) return CSB_ERR_BAD_ARG;
  if (D % 8 || D > 128 || D < 16 || Hq % Hk) return CSB_ERR_BAD_ARG;
  if (cls == nullptr && !mask_by_index(mask_mode, q_pos, k_pos)) return CSB_ERR_BAD_ARG;
  if (mask_mode == MASK_DENSE && (ex == nullptr || ex->dmask == nullptr)) return CSB_ERR_BAD_ARG;
  if (kv == nullptr || kv->n_seg < 1 || kv->n_seg > CSB_MAX_SEG) return CSB_ERR_BAD_ARG;
  if ((Sq + BW_BQ - 1) / BW_BQ > BwdSmem::MAX_TILES) return CSB_ERR_TOO_LARGE;
  if ((q_ss % 8) || (do_ss % 8) || (dq_ss % 4)) return CSB_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  {
    const long grid = (long)((Sq + 16 * DELTA_ROWS - 1) / (16 * DELTA_ROWS)) * B * Hq;
    if (grid > 0x7fffffffL) return CSB_ERR_TOO_LARGE;
    const bool vec = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0 && o_ss % 8 == 0 &&
                     o_sb % 8 == 0 && do_ss % 8 == 0 && do_sb % 8 == 0;
    auto kfn = vec ? attn_delta_kernel<true> : attn_delta_kernel<false>;
    kfn<<<(unsigned)grid, 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(out), reinterpret_cast<const __nv_bfloat16*>(dout), delta, dq_acc,
                             Sq, Hq, D, o_sb, o_ss, do_sb, do_ss);
    if (int e = launch_result()) return e;
  }
  AttnBwdParams p;
  p.B = B; p.Sq = Sq; p.Sk = Sk; p.Hq = Hq; p.Hk = Hk; p.D = D;
  p.dk16 = (D + 15) / 16 * 16;
  p.nQ64 = (Sq + BW_BQ - 1) / BW_BQ;
  p.nQ128 = (Sq + 127) / 128;
  p.nK = (Sk + BW_BKV - 1) / BW_BKV;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.mask_mode = mask_mode;
  p.q_bits = reinterpret_cast<const int64_t*>(q_bits);
  p.k_bits = reinterpret_cast<const int64_t*>(k_bits);
  p.q_pos = q_pos; p.k_pos = k_pos;
  p.cls = reinterpret_cast<const int8_t*>(cls);
  p.lse = lse; p.delta = delta; p.dq_acc = dq_acc;
  p.status = status;
  p.dmask = ex ? ex->dmask : nullptr;
  p.dm_sb = ex ? ex->dm_sb : 0; p.dm_sq = ex ? ex->dm_sq : 0;
  p.bias = ex ? ex->bias : nullptr;
  p.bias_sb = ex ? ex->bias_sb : 0; p.bias_sh = ex ? ex->bias_sh : 0; p.bias_sq = ex ? ex->bias_sq : 0;
  p.inv_scale = scale != 0.f ? 1.f / scale : 0.f;
  p.kj_slowest = mask_mode != MASK_FULL;
  p.nsplit = nsplit;
  p.part = part;
  fill_seg_info(&p.seg, kv, BW_BKV);
  if (p.seg.tile_start[kv->n_seg] != p.nK) return CSB_ERR_BAD_ARG;
  CUtensorMap tq, tdo;
  KvMaps kvm;
  int r;
  if ((r = make_tmap_4d(&tq, q, D, Hq, Sq, B, q_ss, q_sb, BW_BQ))) return r;
  if ((r = make_tmap_4d(&tdo, dout, D, Hq, Sq, B, do_ss, do_sb, BW_BQ))) return r;
  for (int i = 0; i < CSB_MAX_SEG; ++i) {
    const int g = i < kv->n_seg ? i : 0;  // unused slots repeat segment 0 (never dereferenced)
    if ((kv->k_stride_s[g] % 8) || (kv->v_stride_s[g] % 8) || (kv->dk_stride_s[g] % 8) || (kv->dv_stride_s[g] % 8)) return CSB_ERR_BAD_ARG;
    if (i < kv->n_seg) {
      if ((r = make_tmap_4d(&kvm.k[i], kv->k[g], D, Hk, kv->rows[g], B, kv->k_stride_s[g], kv->k_stride_b[g], BW_BKV))) return r;
      if ((r = make_tmap_4d(&kvm.v[i], kv->v[g], D, Hk, kv->rows[g], B, kv->v_stride_s[g], kv->v_stride_b[g], BW_BKV))) return r;
    } else {
      kvm.k[i] = kvm.k[0];
      kvm.v[i] = kvm.v[0];
    }
    p.dK[i] = reinterpret_cast<__nv_bfloat16*>(kv->dk[g]);
    p.dV[i] = reinterpret_cast<__nv_bfloat16*>(kv->dv[g]);
    p.dk_stride_s[i] = kv->dk_stride_s[g]; p.dk_stride_b[i] = kv->dk_stride_b[g];
    p.dv_stride_s[i] = kv->dv_stride_s[g]; p.dv_stride_b[i] = kv->dv_stride_b[g];
  }
  CUtensorMap tdq;
  {
    // dq_acc is dense fp32 [B][Sq][Hq][D]; a block is 32 head-dim elements (128 B) x 64 query rows
    uint64_t dims[4] = {(uint64_t)D, (uint64_t)Hq, (uint64_t)Sq, (uint64_t)B};
    uint64_t strides[3] = {(uint64_t)D * 4, (uint64_t)Hq * D * 4, (uint64_t)Sq * Hq * D * 4};
    uint32_t box[4] = {32, 1, (uint32_t)BW_BQ, 1};
    if ((r = make_tmap_nd_f32(&tdq, dq_acc, 4, dims, strides, box))) return r;
  }
  static bool attr = false;
  if (!attr) {
    for (auto kfn : {attn_bwd_kernel<false>, attn_bwd_kernel<true>})
      if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdSmem::DYN_BYTES) != cudaSuccess) return launch_result();
    attr = true;
  }
  const long n_blocks = (long)p.nK * Hk * B * nsplit;
  if (n_blocks > 0x7fffffffL) return CSB_ERR_TOO_LARGE;
  dim3 grid((unsigned)n_blocks);
  auto bwd_kfn = p.dmask != nullptr || p.bias != nullptr ? attn_bwd_kernel<true> : attn_bwd_kernel<false>;
  bwd_kfn<<<grid, BwdCfg::THREADS, BwdSmem::DYN_BYTES, s>>>(tq, kvm, tdo, tdq, p);
  int e = launch_result();
  if (e) return e;
  if (nsplit > 1) {
    const long k_rows = (long)B * Sk;
    const int hd = Hk * D, bx = (hd / 8 + 127) / 128;
    const dim3 rgrid(bx, (unsigned)(k_rows < 2048 ? k_rows : 2048), 2);
    attn_dkv_reduce_kernel<<<rgrid, 128, 0, s>>>(part, nsplit, k_rows, Sk, hd, p.dK[0], p.dV[0], p.dk_stride_b[0], p.dk_stride_s[0],
                                                 p.dv_stride_b[0], p.dv_stride_s[0]);
    if ((e = launch_result())) return e;
  }
  const long n_rows = (long)B * Sq;
  const int HD = Hq * D;
  {
    const int bx = (HD / 8 + 255) / 256;
    long by = ((long)sm_count() * 8 + bx - 1) / bx;
    if (by > n_rows) by = n_rows;
    const bool vec = (reinterpret_cast<uintptr_t>(dq) & 15) == 0 && dq_ss % 8 == 0 && dq_sb % 8 == 0;
    auto kfn = vec ? attn_dq_convert_kernel<true> : attn_dq_convert_kernel<false>;
    kfn<<<dim3(bx, (unsigned)by), 256, 0, s>>>(dq_acc, reinterpret_cast<__nv_bfloat16*>(dq), n_rows, Sq, HD, dq_sb, dq_ss);
  }
  return launch_result();
}

CSB_API int csb_attn_bwd_seg(const void* q, const CsbKvSegments* kv, const void* out, const void* dout, const float* lse,
                             float* delta, float* dq_acc, void* dq, int B, int Sq, int Sk, int Hq, int Hk, int D, long q_ss,
                             long q_sb, long o_ss, long o_sb, long do_ss, long do_sb, long dq_ss, long dq_sb, float scale,
                             int mask_mode, const long* q_bits, const long* k_bits, const int* q_pos, const int* k_pos,
                             const signed char* cls, int* status, void* stream) {
  return attn_bwd_seg_impl(q, kv, out, dout, lse, delta, dq_acc, dq, B, Sq, Sk, Hq, Hk, D, q_ss, q_sb, o_ss, o_sb, do_ss, do_sb,
                           dq_ss, dq_sb, scale, mask_mode, q_bits, k_bits, q_pos, k_pos, cls, status, stream, nullptr);
}

// One local K/V tensor with a dense boolean mask (mask_mode = MASK_DENSE) and / or an additive bias (no bias gradient).
CSB_API int csb_attn_bwd_dense(const void* q, const void* k, const void* v, const void* out, const void* dout,
                               const float* lse, float* delta, float* dq_acc, void* dq, void* dk, void* dv, int B, int Sq,
                               int Sk, int Hq, int Hk, int D, long q_ss, long q_sb, long k_ss, long k_sb, long v_ss, long v_sb,
                               long o_ss, long o_sb, long do_ss, long do_sb, long dq_ss, long dq_sb, long dk_ss, long dk_sb,
                               long dv_ss, long dv_sb, float scale, int mask_mode, const signed char* cls,
                               const CsbAttnExtras* ex, int* status, void* stream) {
  CsbKvSegments kv = {};
  kv.n_seg = 1;
  kv.my_seg = 0;
  kv.rows[0] = Sk;
  kv.k[0] = k; kv.v[0] = v;
  kv.k_stride_s[0] = k_ss; kv.k_stride_b[0] = k_sb; kv.v_stride_s[0] = v_ss; kv.v_stride_b[0] = v_sb;
  kv.dk[0] = dk; kv.dv[0] = dv;
  kv.dk_stride_s[0] = dk_ss; kv.dk_stride_b[0] = dk_sb; kv.dv_stride_s[0] = dv_ss; kv.dv_stride_b[0] = dv_sb;
  kv.ready_flags = nullptr;
  return attn_bwd_seg_impl(q, &kv, out, dout, lse, delta, dq_acc, dq, B, Sq, Sk, Hq, Hk, D, q_ss, q_sb, o_ss, o_sb, do_ss, do_sb,
                           dq_ss, dq_sb, scale, mask_mode, nullptr, nullptr, nullptr, nullptr, cls, status, stream, ex);
}

// Blocks per 128-row key block that csb_attn_bwd should be given for these sizes.  Without a split a key block of one KV head is
// one thread block that walks all query heads of its group: 64 blocks for 1024 tokens and 8 KV heads on 148 SMs, and under a
// causal mask the longest block alone decides.  Each further block costs its set-up and epilogue again and the parts are written
// and read once more.  The count with the smallest predicted time is taken: whole rounds of equal blocks under a full mask, the
// longest block or the average load of the SMs otherwise.  An iteration takes 1.25 to 1.35 us on grids of a single round; the
// constant is larger because more blocks also mean more blocks per SM and more parts.
// One block is kept unless another count is predicted at least 7 % faster (the prediction is no better than that), and the parts
// may take CSB_ATTN_BWD_PART_BYTES at most: long sequences fill the GPU without a split, and must not need gigabytes for the last
// per cents.
// Measured, delta and conversion passes included, one block against the count taken (32 / 8 heads, causal): 256 tokens 34.5 / 24.3 us
// (6 blocks); 333: 45.2 / 28.5 (6); 1024: 99.9 / 61.8 (4); 2048: 191 / 131 (2); 1500 tokens, 8 / 1 heads: 251 / 46.4 (16); full
// mask, 3072 tokens: 529 / 424 (3), 8192: 2828 / 2630 (2, 128 MiB).  Kept whole: 729 tokens, 16 / 16 heads, full: 33.5 us, 45 with
// three blocks; 2 x 900 tokens, 8 / 8 heads: 37, 56 with two; 4096 tokens causal: 390, 410 with two.  The furthest from the best
// count found: 512 tokens causal, 41.1 us with the 6 blocks taken, 33.5 with 4; 1024: 61.8, 58.1 with 3; 6144 tokens, full: 1611 us
// whole, 1552 with three blocks of 151 MB of parts.
constexpr long CSB_ATTN_BWD_PART_BYTES = 128L << 20;
CSB_API int csb_attn_bwd_splits(int mask_mode, int B, int Sq, int Sk, int Hq, int Hk) {
  if (B < 1 || Sq < 1 || Sk < 1 || Hk < 1 || Hq < Hk) return 1;
  const float setup_us = 8.f, tile_us = 1.6f;
  const int sms = sm_count();
  const long blocks = (long)((Sk + BW_BKV - 1) / BW_BKV) * Hk * B;
  const long iters = (long)((Sq + BW_BQ - 1) / BW_BQ) * (Hq / Hk);  // of the longest block
  const long block_bytes = 2L * BW_BKV * 128 * sizeof(float);       // dK and dV parts of a block at the largest head width
  int best = 1;
  float best_us = 0.f;
  for (int n = 1; n <= 16 && (n == 1 || (n <= iters / 2 && n * blocks * block_bytes <= CSB_ATTN_BWD_PART_BYTES)); ++n) {
    const float longest = setup_us + tile_us * iters / n;
    float us;
    if (mask_mode == MASK_FULL) {
      us = longest * ((blocks * n + sms - 1) / sms);
    } else {
      const float average = (blocks * n * setup_us + blocks * (0.5f * iters) * tile_us) / sms;
      us = longest > average ? longest : average;
    }
    if (n == 1) {
      best_us = 0.93f * us;
      continue;
    }
    us += 4.f + 0.052f * n * blocks;  // the parts, written and read
    if (us < best_us) {
      best_us = us;
      best = n;
    }
  }
  return best;
}

// One local K/V tensor ([B][Sk][Hk][D] views) with dK / dV of the same shape.  nsplit > 1: `part` holds 2 * nsplit * B * Sk * Hk
// * D floats of scratch.
CSB_API int csb_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout,
                         const float* lse, float* delta, float* dq_acc, void* dq, void* dk, void* dv, int B, int Sq,
                         int Sk, int Hq, int Hk, int D, long q_ss, long q_sb, long k_ss, long k_sb, long v_ss, long v_sb,
                         long o_ss, long o_sb, long do_ss, long do_sb, long dq_ss, long dq_sb, long dk_ss, long dk_sb,
                         long dv_ss, long dv_sb, float scale, int mask_mode, const long* q_bits, const long* k_bits,
                         const int* q_pos, const int* k_pos, const signed char* cls, int* status, void* stream, float* part,
                         int nsplit) {
  CsbKvSegments kv = {};
  kv.n_seg = 1;
  kv.my_seg = 0;
  kv.rows[0] = Sk;
  kv.k[0] = k; kv.v[0] = v;
  kv.k_stride_s[0] = k_ss; kv.k_stride_b[0] = k_sb; kv.v_stride_s[0] = v_ss; kv.v_stride_b[0] = v_sb;
  kv.dk[0] = dk; kv.dv[0] = dv;
  kv.dk_stride_s[0] = dk_ss; kv.dk_stride_b[0] = dk_sb; kv.dv_stride_s[0] = dv_ss; kv.dv_stride_b[0] = dv_sb;
  kv.ready_flags = nullptr;
  return attn_bwd_seg_impl(q, &kv, out, dout, lse, delta, dq_acc, dq, B, Sq, Sk, Hq, Hk, D, q_ss, q_sb, o_ss, o_sb, do_ss, do_sb,
                           dq_ss, dq_sb, scale, mask_mode, q_bits, k_bits, q_pos, k_pos, cls, status, stream, nullptr, part, nsplit);
}

// --------------------------------------------------------------------------------------------- context-parallel glue
namespace csb {

// Tell every peer that this rank's event counter reached `value` (its K/V are staged, or its dK/dV tiles delivered):
// peer r's flag array has one int per source rank.  Ordered after all earlier work of the stream; the fence makes
// this rank's earlier stores (also those to peer memory) visible before the flag.
__global__ void cp_signal_kernel(int* const* flag_arrays, int world, int me, int value) {
  const int r = threadIdx.x;
  if (r >= world) return;
  __threadfence_system();
  int* f = flag_arrays[r] + me;
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(f), "r"(value) : "memory");
}

// Stream-ordered (bounded) wait until every rank's counter in the local flag array reached `value`.
__global__ void cp_wait_kernel(const int* flags, int world, int value, int* status) {
  if (threadIdx.x != 0) return;
  for (int r = 0; r < world; ++r)
    if (!wait_peer_flag(flags + r, value)) {
      atomicCAS(status, 0, ST_TIMEOUT_PEER_FLAG);
      return;
    }
}

struct CpReduceParams {
  const __nv_bfloat16* src[CSB_MAX_SEG];  // one inbox slot per source rank, all [n] elements
  int world;
  const int* flags;  // local flag array: flags[r] >= value once rank r delivered its tiles
  int value;
  int* status;
};

// out = sum over source ranks of their bf16 partial tiles (fp32 accumulation).
__global__ void __launch_bounds__(256) cp_reduce_kernel(CpReduceParams p, __nv_bfloat16* out, long n8) {
  __shared__ int ok_s;
  if (threadIdx.x == 0) {
    int ok = 1;
    for (int r = 0; r < p.world && ok; ++r)
      if (!wait_peer_flag(p.flags + r, p.value)) ok = 0;
    if (!ok) atomicCAS(p.status, 0, ST_TIMEOUT_PEER_FLAG);
    ok_s = ok;
  }
  __syncthreads();
  if (!ok_s) return;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < p.world; ++r) {
      const uint4 u = reinterpret_cast<const uint4*>(p.src[r])[i];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = __bfloat1622float2(h[k]);
        acc[2 * k] += f.x;
        acc[2 * k + 1] += f.y;
      }
    }
    uint4 o;
    o.x = pack_bf16x2(acc[0], acc[1]);
    o.y = pack_bf16x2(acc[2], acc[3]);
    o.z = pack_bf16x2(acc[4], acc[5]);
    o.w = pack_bf16x2(acc[6], acc[7]);
    reinterpret_cast<uint4*>(out)[i] = o;
  }
}

}  // namespace csb

// flag_arrays: device array of `world` pointers, entry r = rank r's flag array (peer-mapped), each int[world].
CSB_API int csb_cp_signal(void* flag_arrays, int world, int me, int value, void* stream) {
  if (world < 1 || world > CSB_MAX_SEG) return CSB_ERR_BAD_ARG;
  cp_signal_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<int* const*>(flag_arrays), world, me, value);
  return launch_result();
}

CSB_API int csb_cp_wait(const int* flags, int world, int value, int* status, void* stream) {
  if (world < 1 || world > CSB_MAX_SEG) return CSB_ERR_BAD_ARG;
  cp_wait_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(flags, world, value, status);
  return launch_result();
}

// out[n] = sum_r src[r][n] once every rank's counter in `flags` reached `value` (n a multiple of 8).
CSB_API int csb_cp_reduce(const void* const* src, int world, const int* flags, int value, void* out, long n, int* status,
                          void* stream) {
  if (world < 1 || world > CSB_MAX_SEG || (n % 8)) return CSB_ERR_BAD_ARG;
  CpReduceParams p;
  for (int r = 0; r < CSB_MAX_SEG; ++r) p.src[r] = reinterpret_cast<const __nv_bfloat16*>(src[r < world ? r : 0]);
  p.world = world; p.flags = flags; p.value = value; p.status = status;
  const long n8 = n / 8;
  long blocks = (n8 + 255) / 256;
  if (blocks > (long)sm_count() * 8) blocks = (long)sm_count() * 8;
  if (blocks < 1) blocks = 1;
  cp_reduce_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p, reinterpret_cast<__nv_bfloat16*>(out), n8);
  return launch_result();
}

CSB_WAIT_LIMIT_SETTER(attn_bwd)
