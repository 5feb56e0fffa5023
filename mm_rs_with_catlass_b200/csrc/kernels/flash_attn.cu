// Flash attention forward on tcgen05: one CTA per 256 query rows (two tiles of 128) of one (batch, head).
//
//   warps 0..3  softmax of tile 0 : one query row per thread: tcgen05.ld the scores, row maximum, exp2, row sum,
//   warps 4..7  softmax of tile 1   P (operand dtype) written to columns of its own with tcgen05.st, O rescaled in
//                                   TMEM when the running maximum moved by more than 2^8, final O / l and the store
//   warp 8      TMA producer      : both Q tiles once, then K and V blocks of 128 keys through one ring of slots
//   warp 9      MMA issuer        : S_t = Q_t K^T into TMEM, O_t += P_t V with P read from TMEM (the A operand of
//                                   tcgen05.mma may live there); at D = 128 for tile 0, and warp 10 for tile 1
//
// TMEM columns, D = 128: one buffer of scores for both tiles [0, 128), P_0 and P_1 (64 columns of packed 16-bit pairs each) at
// 128 and 192, O_0 and O_1 at 256 and 384. D = 64: S_0, S_1 at 0 and 128, O_0, O_1 at 256 and 320, P_0, P_1 at 384 and 448. The
// scores are read from TMEM once and stay in registers (softmax_row.cuh; a split of the registers between the warpgroups makes
// room), so that a tile's next scores are computed while its softmax works on the present ones.
//
// Bound by the steps of one row: of 2930 cycles a block (D = 128, per tile, cycle counters) 260 go to reading the scores, 300 to
// the maximum, 1840 to the exponentials beside the other tile's (the special-function unit alone: 1024), 400 to waiting for
// the next scores; tensor cores and special-function unit are 65 % busy (1 x 32 x 4096, not causal). With P on top of S_t and one issuer for both tiles, whose
// products waited behind the other tile's softmax, a block took 3490. Causal, 2 x 32 / 8 heads x 8192, D = 128: 855 -> 770 us
// at full clock (operands of zeros), 1040 -> 980 us in a loop, which the power limit holds.
//
// The online-softmax recurrence (m: reference maximum, l: running sum, per row, in the log2 domain):
//   P = exp2(scale S - m),  l' = l a + rowsum(P),  O' = O a + P V,  a = exp2(m - m')
// m follows the running maximum lazily: it moves only when some row of the warp exceeds it by more than 8, i.e.
// P stays below 2^8 (exact in fp32, harmless for a 16-bit P), and then O and l are rescaled. Most blocks skip the
// rescale and its trip through TMEM.
//
// Roles of the reference this kernel plays (different construction, same jobs):
//   3rdparty/catlass/include/catlass/gemm/block/block_mmad_fa_qk.hpp, block_mmad_fa_pv.hpp
//   3rdparty/catlass/include/catlass/epilogue/block/block_epilogue_fa_softmax.hpp, ..._fa_rescale_o.hpp
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <cstring>
#include "catcoc/attn_host.h"
#include "catcoc/capi.h"
#include "catcoc/host_util.h"
#include "catcoc/params.h"
#include "catcoc/ptx.cuh"
#include "catcoc/softmax_row.cuh"

namespace catcoc {
namespace attn {

constexpr int kBQ = 128;          // query rows per tile == TMEM lanes
constexpr int kTiles = 2;         // query tiles per CTA
constexpr int kBKV = 128;         // keys per block
constexpr int kThreads = 384;     // 2 x 4 softmax warps, producer, one or (D = 128) two issuers; the others only complete the warpgroup
// Registers: a softmax thread keeps 128 scores and their probabilities. The block is launched with 168 a thread; the
// third warpgroup gives up what the first two take: 2 x 216 + 72 = 3 x 168.
constexpr int kSoftmaxRegs = 216, kOtherRegs = 72;
constexpr int kProducerWarp = 8, kIssuerWarp = 9;   // + t: a tile's issuer
constexpr int kBlockBytes = 128 * 128;   // one 128-row x 128-byte (64 element) swizzled block
constexpr int kMaxSlots = 8;

struct AttnParams {
  CUtensorMap tm_q, tm_k, tm_v;   // {D, S, B * H} with a {64, 128, 1} box, 128-byte swizzle
  void* out;                      // [B, Hq, Sq, D]
  int B, Hq, Hk, Sq, Sk, D;       // Sq: rows per (batch, query head), or per (batch, KV head) when its heads are packed
  int pos;                        // query positions: row r stands at r % pos
  int causal;                     // key j is visible to position i when j <= i + (Sk - pos)
  int tiles, order_heads;         // CTAs per head; heads that are walked side by side (see the CTA order below)
  float scale_log2;               // softmax scale * log2(e), > 0
  int fmt;                        // FMT_F16 or FMT_BF16
  uint32_t idesc_qk, idesc_pv;
  uint32_t* status;
  uint64_t timeout_ns;
  float* part_o;                  // keys cut into slices: [slice][B * Hq * Sq][D] unnormalised pieces
  float* part_ml;                 // [slice][B * Hq * Sq][2]
  int per;                        // key blocks of a slice
};

struct Bars {
  uint64_t q_full, kv_full[kMaxSlots], kv_empty[kMaxSlots], s_full[kTiles], s_free[kTiles], p_half[kTiles], p_full[kTiles], pv_done[kTiles], o_done[kTiles];
  uint32_t tmem_base, abort_flag;
};

CATCOC_DEVICE void fail(const AttnParams& p, uint32_t what, uint32_t a, uint32_t b) {
  if (atomicCAS(p.status, 0u, static_cast<uint32_t>(STATUS_TIMEOUT_PIPELINE)) == 0u) {
    p.status[1] = 0u; p.status[2] = 100u + what; p.status[3] = a; p.status[4] = b; p.status[5] = 0u;
    p.status[6] = blockIdx.x;
    __threadfence_system();
  }
}

// D: head dimension; FMT: operand and output dtype (compile time: the softmax loop packs 64 pairs per row and block);
// CUT: a CTA takes the key blocks of slice blockIdx.y only and leaves a piece; LATE: a block's softmax waits for the product with V of
// the block before where it needs it, to rescale O or to write P, else ahead of its exponentials (D = 64, see attn_plan)
template <int D, int FMT, bool CUT, bool LATE>
__global__ void __launch_bounds__(kThreads, 1) flash_attn_kernel(const __grid_constant__ AttnParams p) {
  constexpr int kDB = D / 64;                    // 128-byte blocks along the head dimension
  constexpr int kQBytes = kDB * kBlockBytes;     // one Q tile
  constexpr int kSlotBytes = kDB * kBlockBytes;  // one K or V block: 128 keys x D
  constexpr int kSlots = D == 128 ? 4 : 8;       // ring of K / V blocks (K_0 V_0 K_1 V_1 ...)
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kOCol = 256;
  // The probabilities have columns of their own, so that the next scores are computed as soon as the softmax has read the
  // present ones and not behind the second product. At D = 128 that leaves one buffer of scores, which the tiles take in turn.
  // Each tile then has an issuer of its own, so that no tile's products wait behind the other's softmax (one issuer for both: 864
  // us where two take 772, causal 2 x 32 / 8 x 8192 of zeros). At D = 64 one warp issues both tiles' scores, then both products with V,
  // which start on the first half of the keys (two issuers, whole blocks: 728 -> 764 us, 2 x 32 x 8192 of zeros).
  constexpr bool kOneS = D == 128;
  constexpr int kIssuers = kOneS ? 2 : 1;
  constexpr uint32_t kPCol = kOneS ? 128 : 384;    // P_t at kPCol + t * 64
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sq = smem;                            // two Q tiles
  uint8_t* skv = sq + kTiles * kQBytes;
  Bars* bars = reinterpret_cast<Bars*>(skv + kSlots * kSlotBytes);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // CTA order: blocks of `order_heads` heads; inside a block the last (longest, when causal) tiles of all heads first, so
  // that the launch ends with the shortest ones
  const int per_block = p.order_heads * p.tiles;
  const int blk = static_cast<int>(blockIdx.x) / per_block, in_blk = static_cast<int>(blockIdx.x) - blk * per_block;
  const int heads = min(p.order_heads, p.B * p.Hq - blk * p.order_heads);
  const int qt = p.tiles - 1 - in_blk / heads;
  const int q0 = qt * (kTiles * kBQ);
  const int bh = blk * p.order_heads + in_blk % heads;   // b * Hq + h
  const int b = bh / p.Hq, h = bh - b * p.Hq;
  const int bhk = b * p.Hk + h / (p.Hq / p.Hk);    // grouped-query attention: several query heads share one KV head
  const int shift = p.Sk - p.pos;                  // causal diagonal offset
  // positions of a tile's rows: [lo, hi], the whole range when the rows of two packed heads meet in it
  auto tile_lo = [&](int t) { const int r = (q0 + t * kBQ) % p.pos; return r + kBQ > p.pos && p.pos < p.Sq ? 0 : r; };
  auto tile_hi = [&](int t) { const int r = (q0 + t * kBQ) % p.pos; return r + kBQ > p.pos && p.pos < p.Sq ? p.pos - 1 : r + kBQ - 1; };
  // key blocks each tile walks (tile 1 never fewer than tile 0; rows past Sq are computed and not stored)
  int nblk[kTiles];
#pragma unroll
  for (int t = 0; t < kTiles; ++t) {
    const int kv_end = p.causal ? min(p.Sk, tile_hi(t) + 1 + shift) : p.Sk;
    nblk[t] = (kv_end + kBKV - 1) / kBKV;
  }
  // (a slice that some tile sees nothing of is a masked block there: a maximum of -inf, a sum of zero)
  const int j0 = CUT ? static_cast<int>(blockIdx.y) * p.per : 0;
  if constexpr (CUT) {
#pragma unroll
    for (int t = 0; t < kTiles; ++t) nblk[t] = max(1, min(p.per, nblk[t] - j0));
  }
  nblk[1] = max(nblk[0], nblk[1]);
  const int nmax = nblk[1];

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    for (int s = 0; s < kSlots; ++s) { ptx::mbar_init(&bars->kv_full[s], 1); ptx::mbar_init(&bars->kv_empty[s], kIssuers); }
    for (int t = 0; t < kTiles; ++t) {
      ptx::mbar_init(&bars->s_full[t], 1);
      ptx::mbar_init(&bars->s_free[t], 4);
      ptx::mbar_init(&bars->pv_done[t], 1);
      ptx::mbar_init(&bars->p_half[t], 4);         // one arrival per softmax warp: P of the first 64 keys is in TMEM
      ptx::mbar_init(&bars->p_full[t], 4);         // ... of all of them
      ptx::mbar_init(&bars->o_done[t], 1);
    }
    bars->abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tmap(&p.tm_q); ptx::prefetch_tmap(&p.tm_k); ptx::prefetch_tmap(&p.tm_v);
  }
  if (warp == kIssuerWarp) { ptx::tmem_alloc(&bars->tmem_base, kTmemCols); ptx::tmem_relinquish(); }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem = bars->tmem_base;
  ptx::grid_dependency_wait();
  if constexpr (CUT) ptx::launch_dependents();                       // the combine kernel waits for this grid's results by itself

  if (warp >= kProducerWarp) ptx::reg_dec<kOtherRegs>();   // all four warps of the warpgroup at one place
  if (warp == kProducerWarp) {
    // ------------------------------ TMA producer ------------------------------
    if (ptx::elect_one()) {
      ptx::mbar_expect_tx(&bars->q_full, kTiles * kQBytes);
      for (int t = 0; t < kTiles; ++t)
        for (int d = 0; d < kDB; ++d)
          ptx::tma_load_3d(sq + t * kQBytes + d * kBlockBytes, &p.tm_q, &bars->q_full, d * 64, q0 + t * kBQ, bh);
    }
    __syncwarp();
    // item 2 j is K block j, item 2 j + 1 is V block j; item i lives in slot i % kSlots
    for (int item = 0; item < 2 * nmax; ++item) {
      const int slot = item % kSlots;
      const uint32_t use = static_cast<uint32_t>(item / kSlots);
      if (!ptx::mbar_wait(&bars->kv_empty[slot], (use & 1u) ^ 1u, p.timeout_ns, abort_flag)) {
        if (lane == 0) { fail(p, 1u, item, 0u); *abort_flag = 1; }
        break;
      }
      if (ptx::elect_one()) {
        ptx::mbar_expect_tx(&bars->kv_full[slot], kSlotBytes);
        const CUtensorMap* tm = (item & 1) ? &p.tm_v : &p.tm_k;
        for (int d = 0; d < kDB; ++d)
          ptx::tma_load_3d(skv + slot * kSlotBytes + d * kBlockBytes, tm, &bars->kv_full[slot], d * 64, (j0 + (item >> 1)) * kBKV, bhk);
      }
      __syncwarp();
    }
  } else if (warp >= kIssuerWarp && warp < kIssuerWarp + kIssuers) {
    // ------------------------------ MMA issuers ------------------------------
    const uint64_t dq0 = ptx::make_smem_desc_sw128(ptx::smem_u32(sq), 16u, 1024u);
    const uint64_t dk0 = ptx::make_smem_desc_sw128(ptx::smem_u32(skv), 16u, 1024u);
    const uint64_t dv0 = ptx::make_smem_desc_sw128(ptx::smem_u32(skv), static_cast<uint32_t>(kBlockBytes), 1024u);
    // (addresses are in the low words, which no tile or slot carries over into the high ones)
    const uint32_t q_lo = static_cast<uint32_t>(dq0), q_hi = static_cast<uint32_t>(dq0 >> 32);
    const uint32_t k_lo = static_cast<uint32_t>(dk0), k_hi = static_cast<uint32_t>(dk0 >> 32);
    const uint32_t v_lo = static_cast<uint32_t>(dv0), v_hi = static_cast<uint32_t>(dv0 >> 32);
    auto wait_item = [&](int item) {
      return ptx::mbar_wait(&bars->kv_full[item % kSlots], static_cast<uint32_t>(item / kSlots) & 1u, p.timeout_ns, abort_flag);
    };
    // (one warp for both tiles has waited for tile 0's block when it comes to tile 1)
    auto first_use = [&](int t, int j) { return kOneS || t == 0 || j >= nblk[0]; };
    // S_t[128, 128 keys] = Q_t[128, D] K^T of block j, behind the softmax's read of what is in the buffer: both operands
    // K-major (D contiguous), 16 elements of D per MMA
    auto scores = [&](int t, int j) {
      if (first_use(t, j) && !wait_item(2 * j)) return false;
      const int before = !kOneS || t == 0 || j >= nblk[0] ? j - 1 : j;             // the block and the tile that were there
      const int tile = !kOneS ? t : (t == 1 && j < nblk[0] ? 0 : 1);
      if (before >= 0 && !ptx::mbar_wait(&bars->s_free[tile], static_cast<uint32_t>(before & 1), p.timeout_ns, abort_flag)) return false;
      ptx::tcgen05_fence_after();
      const int slot = (2 * j) % kSlots;
      if (ptx::elect_one()) {
        const uint32_t ql = q_lo + static_cast<uint32_t>(t * (kQBytes >> 4)), kl = k_lo + static_cast<uint32_t>(slot * (kSlotBytes >> 4));
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = static_cast<uint32_t>(((kk >> 2) * kBlockBytes + (kk & 3) * 32) >> 4);
          ptx::umma_f16(tmem + (kOneS ? 0 : t * 128), ptx::desc_of(ql + off, q_hi), ptx::desc_of(kl + off, k_hi), p.idesc_qk, kk != 0 ? 1u : 0u);
        }
        ptx::tcgen05_commit(&bars->s_full[t]);
        if (kOneS || t == 1) ptx::tcgen05_commit(&bars->kv_empty[slot]);     // (tile 1 walks no fewer blocks than tile 0)
      }
      __syncwarp();
      return true;
    };
    // O_t[128, D] += P_t[128, 128 keys] V[128 keys, D] of block j: P from TMEM (row = lane, two keys per 32-bit column, 8 columns
    // per MMA), V MN-major (D contiguous): 16 key rows per MMA = 2048 bytes down a block, blocks of 64 head-dim columns 16 KiB
    // apart
    auto values = [&](int t, int j) {
      const int v_item = 2 * j + 1, slot = v_item % kSlots;
      const uint32_t vl = v_lo + static_cast<uint32_t>(slot * (kSlotBytes >> 4));
      if (first_use(t, j) && !wait_item(v_item)) return false;
      constexpr int kParts = kOneS ? 1 : 2, kPerPart = kBKV / 16 / kParts;
#pragma unroll
      for (int part = 0; part < kParts; ++part) {
        if (!ptx::mbar_wait(part + 1 < kParts ? &bars->p_half[t] : &bars->p_full[t], static_cast<uint32_t>(j & 1), p.timeout_ns, abort_flag)) return false;
        ptx::tcgen05_fence_after();
        if (ptx::elect_one()) {
#pragma unroll
          for (int kk = part * kPerPart; kk < (part + 1) * kPerPart; ++kk)
            ptx::umma_f16_ts(tmem + kOCol + t * D, tmem + kPCol + t * 64 + kk * 8, ptx::desc_of(vl + static_cast<uint32_t>((kk * 16 * 128) >> 4), v_hi),
                             p.idesc_pv, (j > 0 || kk != 0) ? 1u : 0u);
          if (part + 1 == kParts) {
            ptx::tcgen05_commit(j + 1 < nblk[t] ? &bars->pv_done[t] : &bars->o_done[t]);
            if (kOneS || t == 1) ptx::tcgen05_commit(&bars->kv_empty[slot]);
          }
        }
        __syncwarp();
      }
      return true;
    };
    bool ok = ptx::mbar_wait(&bars->q_full, 0u, p.timeout_ns, abort_flag);
    if constexpr (kOneS) {
      const int t = warp - kIssuerWarp, nt = nblk[t];
      ok = ok && scores(t, 0);
      for (int j = 0; ok && j < nt; ++j) {
        if (j + 1 < nt) ok = scores(t, j + 1);      // ahead of the product with V, which waits for this block's softmax
        ok = ok && values(t, j);
      }
      // the other tile walks on: its blocks are released for this one too, each when it has arrived
      for (int item = 2 * nt; ok && item < 2 * nmax; ++item) {
        ok = wait_item(item);
        if (ok && lane == 0) ptx::mbar_arrive(&bars->kv_empty[item % kSlots]);
      }
    } else {
      ok = ok && scores(0, 0) && scores(1, 0);
      for (int j = 0; ok && j < nmax; ++j) {
#pragma unroll
        for (int t = 0; t < kTiles; ++t)
          if (j + 1 < nblk[t]) ok = ok && scores(t, j + 1);
#pragma unroll
        for (int t = 0; t < kTiles; ++t)
          if (j < nblk[t]) ok = ok && values(t, j);
      }
    }
    if (!ok && lane == 0) { fail(p, 2u, 0u, 0u); *abort_flag = 1; }
  } else if (warp < kProducerWarp) {
    // ------------------------------ softmax / correction / epilogue ------------------------------
    ptx::reg_inc<kSoftmaxRegs>();
    const int t = warp >> 2;                         // query tile of this warp
    const int qd = warp & 3;                         // TMEM lane quarter of this warp
    const int row = qd * 32 + lane;                  // query row inside the tile
    const int qi = q0 + t * kBQ + row;
    const uint32_t t_s = tmem + (static_cast<uint32_t>(qd * 32) << 16) + (kOneS ? 0 : t * 128);
    const uint32_t t_p = tmem + (static_cast<uint32_t>(qd * 32) << 16) + kPCol + t * 64;
    const uint32_t t_o = tmem + (static_cast<uint32_t>(qd * 32) << 16) + kOCol + t * D;
    const int n_mine = nblk[t];
    const int vis = p.causal ? min(p.Sk, qi % p.pos + shift + 1) : p.Sk;    // keys [0, vis) are visible to this row
    const int vis_tile = p.causal ? min(p.Sk, tile_lo(t) + shift + 1) : p.Sk;   // ... to every row of the tile
    const float sc = p.scale_log2;
    RowState st;
    bool ok = true;
    for (int j = 0; j < n_mine; ++j) {
      if (!ptx::mbar_wait(&bars->s_full[t], static_cast<uint32_t>(j & 1), p.timeout_ns, abort_flag)) { ok = false; break; }
      ptx::tcgen05_fence_after();
      const int key0 = (j0 + j) * kBKV;
      // masked: some row of the tile does not see all of the block
      // P V of block j - 1 has read P, and O is whole
      auto previous = [&] {
        if (j > 0 && !ptx::mbar_wait(&bars->pv_done[t], static_cast<uint32_t>(j - 1) & 1u, p.timeout_ns, abort_flag)) ok = false;
        ptx::tcgen05_fence_after();
      };
      softmax_row_block<FMT>(t_s, t_p, key0 + kBKV > vis_tile, vis - key0, sc, st, [&] {
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->s_free[t]);
      }, [&](bool move, float alpha) {
        if (!LATE || move) previous();
        if (move && j > 0) rescale_o<D>(t_o, alpha);
      }, [&] { if constexpr (LATE) previous(); }, [&] {
        if constexpr (!kOneS) {
          ptx::tcgen05_wait_st();
          ptx::tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&bars->p_half[t]);
        }
      });
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ptx::tcgen05_wait_st();
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->p_full[t]);
    }
    if (ok) ok = ptx::mbar_wait(&bars->o_done[t], 0u, p.timeout_ns, abort_flag);
    if (!ok) {
      if (lane == 0) { fail(p, 3u, t, 0u); *abort_flag = 1; }
    } else {
      ptx::tcgen05_fence_after();
      const float inv = (st.l > 0.0f) ? 1.0f / st.l : 0.0f;
      uint8_t* orow = static_cast<uint8_t*>(p.out) + (static_cast<int64_t>(bh) * p.Sq + qi) * D * 2;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(t_o + c * 32, v);
        ptx::tcgen05_wait_ld();
        if (CUT && qi < p.Sq) {
          const int64_t prow = (static_cast<int64_t>(blockIdx.y) * p.B * p.Hq + bh) * p.Sq + qi;
#pragma unroll
          for (int u = 0; u < 8; ++u) ptx::st_global_v4(p.part_o + prow * D + c * 32 + u * 4, make_uint4(v[u * 4], v[u * 4 + 1], v[u * 4 + 2], v[u * 4 + 3]));
          if (c == 0) *reinterpret_cast<float2*>(p.part_ml + prow * 2) = make_float2(st.m, st.l);
        } else if (qi < p.Sq) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack16<FMT>(__uint_as_float(v[u * 8 + 2 * e]) * inv, __uint_as_float(v[u * 8 + 2 * e + 1]) * inv);
            ptx::st_global_v4(orow + c * 64 + u * 16, make_uint4(w[0], w[1], w[2], w[3]));
          }
        }
      }
    }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  if (warp == kIssuerWarp) ptx::tmem_dealloc(tmem, kTmemCols);
}

// The slices of a row, a warp each; every row has a slice that it sees something of unless it sees nothing at all. A slice of which
// the row sees nothing is left out, not weighed with zero: its piece is zero times values that the row's tile may not see either, where
// an infinity makes a NaN. (A sum that is not zero, a NaN, is no such slice.)
template <int D, int FMT>
__global__ void __launch_bounds__(128) flash_slices_kernel(const float* part_o, const float* part_ml, void* out, int64_t rows, int slices) {
  constexpr int kPer = D / 32;                     // columns per lane
  const int64_t r = static_cast<int64_t>(blockIdx.x) * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  ptx::grid_dependency_wait();
  if (r >= rows) return;
  const float2 ml = lane < slices ? *reinterpret_cast<const float2*>(part_ml + (lane * rows + r) * 2) : make_float2(-INFINITY, 0.0f);
  float mx = ml.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float w = ml.x == -INFINITY ? 0.0f : ptx::ex2_approx(ml.x - mx);
  const uint32_t seen = __ballot_sync(0xffffffffu, !(ml.x == -INFINITY && ml.y == 0.0f));
  float l = w * ml.y, acc[kPer];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
  for (int e = 0; e < kPer; ++e) acc[e] = 0.0f;
#pragma unroll 4
  for (int c = 0; c < slices; ++c) {
    const float wc = __shfl_sync(0xffffffffu, w, c);
    const float* src = part_o + (c * rows + r) * D + lane * kPer;
    float o[kPer] = {};
    if ((seen >> c) & 1u) {
      if constexpr (kPer == 4) *reinterpret_cast<float4*>(o) = *reinterpret_cast<const float4*>(src);
      else *reinterpret_cast<float2*>(o) = *reinterpret_cast<const float2*>(src);
    }
#pragma unroll
    for (int e = 0; e < kPer; ++e) acc[e] += wc * o[e];
  }
  const float inv = l > 0.0f ? 1.0f / l : 0.0f;
  uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(out) + (r * D + lane * kPer) * 2);
#pragma unroll
  for (int e = 0; e < kPer / 2; ++e) dst[e] = pack16<FMT>(acc[2 * e] * inv, acc[2 * e + 1] * inv);
}

}  // namespace attn
}  // namespace catcoc

using namespace catcoc;
using namespace catcoc::host;

namespace {
// D = 64: does a softmax wait for the product before late? That is the faster form while the two tiles of a CTA are out of step, from
// its start on (10 blocks of keys: 2 x 32 / 8 heads x 300 over 1200 keys 22.1 -> 20.1 us) and where the mask gives them different numbers
// of blocks, at least a third of the keys (load 17, 3 x 600 over 1200: 40.6 -> 39.8; 22, 4 x 32 / 4 x 500 over 1500: 43.7 -> 41.6; 35,
// 2 x 2048: 65.9 -> 64.8). In step the other one is: load 22, 8 x 300 over 1200 59.2 -> 61.0; 46, 6 x 1000, not causal, 96.5 -> 102.6; 57,
// 1 x 32 x 4096 105 -> 107; 221, 2 x 4096, not causal, 349 -> 367. `load`: key blocks of the busiest SM.
bool late_wait(double load, int64_t ctas, int causal, int pos, int Sk) {
  return load <= (causal && 3ll * pos >= Sk ? 35.0 : ctas <= 148 ? 16.0 : 0.0);
}

struct AttnPlan {
  int Hq, Sq;          // as the kernel sees them (the query heads of a KV head may be packed)
  int tiles;
  int slices, per;     // keys cut into slices of `per` blocks
  double load;         // key blocks of the busiest SM
};

AttnPlan attn_plan(int B, int Hq, int Hk, int Sq, int Sk, int causal, bool cut) {
  const int group = Hq / Hk, rows_cta = attn::kTiles * attn::kBQ, pos = Sq;
  auto blocks = [&](int hi) { return static_cast<double>((causal ? std::min<int64_t>(Sk, static_cast<int64_t>(hi) + Sk - pos) : Sk) + 127) / 128; };
  const double longest = blocks(pos);
  AttnPlan d{Hq, Sq, (Sq + rows_cta - 1) / rows_cta, 1, 0, 0.0}, packed = d;
  double plain = 0.0;
  for (int i = 0; i < d.tiles; ++i) plain += blocks(std::min((i + 1) * rows_cta, pos));
  d.load = std::max(longest, static_cast<double>(B) * Hq * plain / 148.0);
  bool pack = false;
  // A call of few query positions: the query heads of a KV head are contiguous rows, so they can fill tiles together. It
  // costs the keys that a head's early tiles would have skipped; in units of (CTA, 128-key block), a launch takes its
  // total over the SMs or its longest CTA. 16 x 32 / 4 heads x 100 positions over 2000 keys: 154 -> 71 us,
  // 16 x 32 / 8 x 64 over 1000 (D = 64): 78 -> 20 us.
  if (group > 1 && static_cast<int64_t>(group) * Sq <= (1 << 24)) {
    packed.Sq = group * Sq;
    packed.Hq = Hk;
    packed.tiles = (packed.Sq + rows_cta - 1) / rows_cta;
    pack = true;
    packed.load = std::max(longest, static_cast<double>(B) * Hk * packed.tiles * longest / 148.0);
    if (packed.load < 0.95 * d.load) d = packed;
  }
  // Few tiles over many keys leave SMs idle: the keys are then cut into slices, which a second kernel merges. In us, a CTA takes 5
  // and 1.55 a block of keys, the merge 4 and its bytes at 3 TB/s. In a loop, D = 128: 32 heads x 131 positions over 3404 keys 46 ->
  // 26 us, 256 over 4096 54 -> 26, 8 heads x 512 over 16384 199 -> 40, 4 x 4096 causal 54 -> 39. Below 14 blocks a call waits
  // for its host work, which the second launch makes longer (8 blocks 17.0 -> 20.0 us, 12 blocks 22.9 -> 24.0).
  const int nblk = (Sk + 127) / 128;
  if (!cut || longest < 14.0) return d;
  double best = 0.85 * (5.0 + 1.55 * longest);
  const AttnPlan forms[2] = {d, packed};
  for (int f = 0; f < (pack ? 2 : 1); ++f) {
    const AttnPlan& x = forms[f];
    const int64_t ctas = static_cast<int64_t>(B) * x.Hq * x.tiles, rows = static_cast<int64_t>(B) * x.Hq * x.Sq;
    for (int n = 2; n <= 16 && ctas * n <= 148 && 2 * n <= nblk; ++n) {
      const int per = (nblk + n - 1) / n, slices = (nblk + per - 1) / per;
      const double t = 9.0 + 1.55 * per + static_cast<double>(slices) * rows * 128 * 8 / 3e6;
      if (t < best) { best = t; d = x; d.slices = slices; d.per = per; }
    }
  }
  return d;
}
}  // namespace

// Scratch of a call whose keys are cut into slices, else 0
extern "C" int64_t catcoc_flash_attention_workspace_bytes(int B, int Hq, int Hk, int Sq, int Sk, int D, int causal) {
  if (B <= 0 || Hq <= 0 || Hk <= 0 || Sq <= 0 || Sk <= 0 || Hq % Hk != 0 || (D != 64 && D != 128)) return 0;
  const AttnPlan d = attn_plan(B, Hq, Hk, Sq, Sk, causal, true);
  return d.slices > 1 ? static_cast<int64_t>(d.slices) * B * Hq * Sq * (D + 2) * static_cast<int64_t>(sizeof(float)) : 0;
}

extern "C" int64_t catcoc_attention_route(int B, int Hq, int Hk, int Sq, int Sk, int D, int causal) {
  const int64_t decode = catcoc_flash_decode_workspace_bytes(B, Hq, Hk, Sq, Sk, D);
  return decode >= 0 ? decode : -1 - catcoc_flash_attention_workspace_bytes(B, Hq, Hk, Sq, Sk, D, causal);
}

extern "C" int catcoc_flash_attention(const void* q, const void* k, const void* v, void* out, int B, int Hq, int Hk,
                                      int Sq, int Sk, int D, int fmt, int causal, float scale, uint32_t* status,
                                      uint64_t timeout_ns, void* stream) {
  return catcoc_flash_attention_cut(q, k, v, out, nullptr, B, Hq, Hk, Sq, Sk, D, fmt, causal, scale, status, timeout_ns, stream);
}

extern "C" int catcoc_flash_attention_cut(const void* q, const void* k, const void* v, void* out, void* workspace, int B, int Hq, int Hk,
                                          int Sq, int Sk, int D, int fmt, int causal, float scale, uint32_t* status,
                                          uint64_t timeout_ns, void* stream) {
  if (!q || !k || !v || !out || !status || B <= 0 || Hq <= 0 || Hk <= 0 || Sq <= 0 || Sk <= 0) {
    set_error("flash_attention: bad arguments");
    return CATCOC_E_BAD_ARG;
  }
  if (D != 64 && D != 128) { set_error("flash_attention: head dimension %d (64 and 128 are built)", D); return CATCOC_E_UNSUPPORTED; }
  if (Hq % Hk != 0) { set_error("flash_attention: %d query heads do not divide over %d key / value heads", Hq, Hk); return CATCOC_E_BAD_ARG; }
  if (fmt != CATCOC_FMT_F16 && fmt != CATCOC_FMT_BF16) { set_error("flash_attention takes fp16 / bf16"); return CATCOC_E_UNSUPPORTED; }
  if (causal && Sk < Sq) { set_error("causal attention needs Sk >= Sq"); return CATCOC_E_BAD_ARG; }
  if (!(scale > 0.0f)) { set_error("flash_attention: the softmax scale must be positive (the row maximum is taken before scaling)"); return CATCOC_E_UNSUPPORTED; }
  const int rows_cta = attn::kTiles * attn::kBQ, pos = Sq;
  const AttnPlan d = attn_plan(B, Hq, Hk, Sq, Sk, causal, workspace != nullptr);
  Hq = d.Hq;
  Sq = d.Sq;
  attn::AttnParams p;
  memset(&p, 0, sizeof(p));
  const CUtensorMapDataType dt = fmt == CATCOC_FMT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  int rc = encode_bsd(&p.tm_q, q, dt, static_cast<int64_t>(B) * Hq, Sq, D);
  if (rc == 0) rc = encode_bsd(&p.tm_k, k, dt, static_cast<int64_t>(B) * Hk, Sk, D);
  if (rc == 0) rc = encode_bsd(&p.tm_v, v, dt, static_cast<int64_t>(B) * Hk, Sk, D);
  if (rc != 0) return rc;
  p.out = out;
  const int64_t rows = static_cast<int64_t>(B) * Hq * Sq;
  p.part_o = static_cast<float*>(workspace);
  p.part_ml = workspace != nullptr ? p.part_o + d.slices * rows * D : nullptr;
  p.per = d.per;
  p.B = B; p.Hq = Hq; p.Hk = Hk; p.Sq = Sq; p.Sk = Sk; p.D = D; p.pos = pos;
  const int64_t ctas = static_cast<int64_t>(B) * Hq * ((Sq + rows_cta - 1) / rows_cta);
  if (ctas > 0x7fffffff) { set_error("flash_attention: too many query tiles"); return CATCOC_E_TOO_LARGE; }
  p.tiles = d.tiles;
  // Causal tiles differ in length, and with one head after the other the launch ended with the long tiles of its last
  // heads (in a loop, causal 2 x 32 x 8192: 1065 -> 1036 us, 1 x 32 x 4096: 183 -> 150). Heads side by side share the L2, so their keys and values must fit it.
  const int64_t kv_bytes = static_cast<int64_t>(Sk) * D * 4;
  p.order_heads = causal ? static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(static_cast<int64_t>(B) * Hq, (72ll << 20) / kv_bytes * (Hq / Hk)))) : 1;
  p.causal = causal ? 1 : 0;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.fmt = fmt;
  const uint32_t f = fmt == CATCOC_FMT_BF16 ? 1u : 0u;
  p.idesc_qk = ptx::make_instr_desc(1u, f, f, 0u, 0u, 128u, 128u);
  p.idesc_pv = ptx::make_instr_desc(1u, f, f, 0u, 1u, 128u, static_cast<uint32_t>(D));
  p.status = status;
  p.timeout_ns = timeout_ns ? timeout_ns : 10000000000ull;
  const dim3 grid(static_cast<unsigned>(ctas), static_cast<unsigned>(d.slices));
  const int db = D / 64;
  const int slots = D == 128 ? 4 : 8;
  const size_t smem = static_cast<size_t>(attn::kTiles * db + slots * db) * attn::kBlockBytes + sizeof(attn::Bars) + 1024 + 64;
  cudaError_t e;
  auto launch = [&](auto kernel) -> int {
    // (one attribute call per launch: it is cheap and keeps the four instantiations in one place)
    cudaError_t a = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (a != cudaSuccess) { set_error("cudaFuncSetAttribute failed: %s", cudaGetErrorString(a)); return -1000 - static_cast<int>(a); }
    a = launch_overlapped(kernel, grid, dim3(attn::kThreads), smem, static_cast<cudaStream_t>(stream), p);
    if (a != cudaSuccess) { set_error("flash_attention launch failed: %s", cudaGetErrorString(a)); return -1000 - static_cast<int>(a); }
    return 0;
  };
  auto merge = [&](auto kernel) -> int {
    CATCOC_CUDA_OK(launch_overlapped(kernel, dim3(static_cast<unsigned>((rows + 3) / 4)), dim3(128), 0, static_cast<cudaStream_t>(stream), p.part_o, p.part_ml, out,
                                     rows, d.slices));
    return 0;
  };
  const bool bf = fmt == CATCOC_FMT_BF16;
  int lrc;
  if (d.slices > 1) {
    if (D == 128) lrc = bf ? launch(attn::flash_attn_kernel<128, FMT_BF16, true, true>) : launch(attn::flash_attn_kernel<128, FMT_F16, true, true>);
    else lrc = bf ? launch(attn::flash_attn_kernel<64, FMT_BF16, true, true>) : launch(attn::flash_attn_kernel<64, FMT_F16, true, true>);
    if (lrc == 0 && D == 128) lrc = bf ? merge(attn::flash_slices_kernel<128, FMT_BF16>) : merge(attn::flash_slices_kernel<128, FMT_F16>);
    else if (lrc == 0) lrc = bf ? merge(attn::flash_slices_kernel<64, FMT_BF16>) : merge(attn::flash_slices_kernel<64, FMT_F16>);
  } else if (D == 128) {
    lrc = bf ? launch(attn::flash_attn_kernel<128, FMT_BF16, false, true>) : launch(attn::flash_attn_kernel<128, FMT_F16, false, true>);
  } else if (late_wait(d.load, ctas, causal, pos, Sk)) {
    lrc = bf ? launch(attn::flash_attn_kernel<64, FMT_BF16, false, true>) : launch(attn::flash_attn_kernel<64, FMT_F16, false, true>);
  } else {
    lrc = bf ? launch(attn::flash_attn_kernel<64, FMT_BF16, false, false>) : launch(attn::flash_attn_kernel<64, FMT_F16, false, false>);
  }
  if (lrc != 0) return lrc;
  e = cudaGetLastError();
  if (e != cudaSuccess) { set_error("flash_attention launch failed: %s", cudaGetErrorString(e)); return -1000 - static_cast<int>(e); }
  return CATCOC_OK;
}
