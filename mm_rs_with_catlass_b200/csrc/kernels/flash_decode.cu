// Flash attention for few query rows per key / value head: decode steps and short prefills over a cache.
//
// The query heads that share a key / value head are one tile: rows = (Hq / Hk) * Sq <= 128, contiguous in
// [B, Hq, Sq, D], so that every key and value is fetched once for all of them. What is left is a stream of K and V
// at HBM speed, and the work is dealt out by bytes: the key blocks of all (batch, KV head) pairs form one list, cut
// into equal runs of `per` blocks, one run per CTA. A run may end inside a sequence; the pieces of a sequence that
// was cut go to a workspace as (O, m, l) and flash_combine_kernel merges them, a sequence that lies in one run is
// finished in place.
//
//   warps 0..3  softmax of the even blocks of the run, one query row per thread (warps whose rows do not exist idle)
//   warps 4..7  softmax of the odd blocks: its own maximum, sum and O accumulator, merged at the end of a sequence
//   warp 8      TMA producer : Q per sequence (two buffers), K and V blocks in the order the issuer consumes them
//   warp 9      MMA issuer   : S_t = Q K^T into TMEM, O_t += P_t V with P in TMEM; t = block parity, so that the tensor
//                              core and the copies never wait for one softmax chain
//
// Bound by HBM: batch 16, 8 KV heads of 128, 4096 keys (268 MB of K and V, 4 query heads each): 276 us with one CTA
// per query head and 256 rows per CTA, 54 us here (4.9 TB/s).
//
// Roles of the reference this kernel plays (different construction, same jobs):
//   3rdparty/catlass/include/catlass/gemm/block/block_mmad_fa_qk.hpp, block_mmad_fa_pv.hpp
//   3rdparty/catlass/include/catlass/epilogue/block/block_epilogue_fa_softmax.hpp, ..._fa_rescale_o.hpp
#include <cstring>
#include "catcoc/attn_host.h"
#include "catcoc/capi.h"
#include "catcoc/host_util.h"
#include "catcoc/params.h"
#include "catcoc/ptx.cuh"
#include "catcoc/sched.h"
#include "catcoc/softmax_row.cuh"

namespace catcoc {
namespace decode {

using attn::RowState;
using attn::pack16;

constexpr int kRows = 128;        // query rows of a tile == TMEM lanes
constexpr int kBKV = 128;         // keys per block
constexpr int kThreads = 320;
constexpr int kProducerWarp = 8, kIssuerWarp = 9;
constexpr int kBlockBytes = 128 * 128;   // one 128-row x 128-byte (64 element) swizzled block
constexpr int kMaxSlots = 10;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kOCol = 256;

struct DecodeParams {
  CUtensorMap tm_q;               // {D, rows, B * Hk} with a {64, 128, 1} box: rows past the tile's read as zeros
  CUtensorMap tm_k, tm_v;         // {D, Sk, B * Hk}, the same box
  void* out;                      // [B * Hk, rows, D]
  float* part_o;                  // [cta + bh][rows][D] unnormalised pieces
  float* part_ml;                 // [cta + bh][rows][2]
  int BH, rows, Sq, Sk;
  int nb;                         // key blocks per sequence
  int per;                        // key blocks per CTA
  int causal;                     // key j is visible to row r when j <= r % Sq + (Sk - Sq)
  float scale_log2;               // softmax scale * log2(e), > 0
  uint32_t idesc_qk, idesc_pv;
  uint32_t* status;
  uint64_t timeout_ns;
};

struct Bars {
  uint64_t q_full[2], q_empty[2], kv_full[kMaxSlots], kv_empty[kMaxSlots], s_full[2], p_full[2], o_done, o_free, ml_full;
  uint32_t tmem_base, abort_flag;
  float2 ml[2][2][kRows];         // [sequence parity][block parity][row]: (m, l)
};

CATCOC_DEVICE void fail(const DecodeParams& p, uint32_t what, uint32_t a, uint32_t b) {
  if (atomicCAS(p.status, 0u, static_cast<uint32_t>(STATUS_TIMEOUT_PIPELINE)) == 0u) {
    p.status[1] = 0u; p.status[2] = 300u + what; p.status[3] = a; p.status[4] = b; p.status[5] = 0u;
    p.status[6] = blockIdx.x;
    __threadfence_system();
  }
}

// Position of a K or V block in the order the issuer consumes them: K0 K1 V0 K2 V1 ... K(n-1) V(n-2) V(n-1), the
// scores running one block ahead of the second product.
CATCOC_HD int item_of_k(int i) { return i == 0 ? 0 : 2 * i - 1; }
CATCOC_HD int item_of_v(int i, int n) { return i + 1 < n ? 2 * i + 2 : 2 * n - 1; }

template <int D, int FMT>
__global__ void __launch_bounds__(kThreads, 1) flash_decode_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int kDB = D / 64;                    // 128-byte blocks along the head dimension
  constexpr int kQBytes = kDB * kBlockBytes;
  constexpr int kSlotBytes = kDB * kBlockBytes;  // one K or V block: 128 keys x D
  constexpr int kSlots = D == 128 ? 4 : 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sq = smem;                            // two Q buffers
  uint8_t* skv = sq + 2 * kQBytes;
  Bars* bars = reinterpret_cast<Bars*>(skv + kSlots * kSlotBytes);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = p.BH * p.nb;
  const int g_begin = blockIdx.x * p.per;                       // this CTA's run of the block list
  const int n_run = min(total, g_begin + p.per) - g_begin;      // > 0: the grid covers the list exactly
  const int row_warps = (p.rows + 31) / 32;                     // softmax warps per group that own rows

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&bars->q_full[i], 1);
      ptx::mbar_init(&bars->q_empty[i], 1);
      ptx::mbar_init(&bars->s_full[i], 1);
      ptx::mbar_init(&bars->p_full[i], row_warps);
    }
    for (int s = 0; s < kSlots; ++s) { ptx::mbar_init(&bars->kv_full[s], 1); ptx::mbar_init(&bars->kv_empty[s], 1); }
    ptx::mbar_init(&bars->o_done, 1);
    ptx::mbar_init(&bars->o_free, 2 * row_warps);
    ptx::mbar_init(&bars->ml_full, 2 * row_warps);
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
  ptx::launch_dependents();                      // the combine kernel waits for this grid's results by itself

  if (warp == kProducerWarp) {
    // ------------------------------ TMA producer ------------------------------
    bool ok = true;
    int loaded_seqs = 0, seq_end = 0;            // sequences whose Q was requested; first run block past the latest one
    for (int item = 0; ok && item < 2 * n_run; ++item) {
      // K0 K1 V0 K2 V1 ... V(n-1)
      const bool is_k = item == 0 || ((item & 1) != 0 && item != 2 * n_run - 1);
      const int i = is_k ? (item + 1) >> 1 : (item == 2 * n_run - 1 ? n_run - 1 : (item >> 1) - 1);
      const int g = g_begin + i;
      const int bh = g / p.nb, blk = g - bh * p.nb;
      if (is_k && i == seq_end) {
        const int qb = loaded_seqs & 1;
        if (!ptx::mbar_wait(&bars->q_empty[qb], (static_cast<uint32_t>(loaded_seqs >> 1) & 1u) ^ 1u, p.timeout_ns, abort_flag)) { ok = false; break; }
        if (ptx::elect_one()) {
          ptx::mbar_expect_tx(&bars->q_full[qb], kQBytes);
          for (int d = 0; d < kDB; ++d)
            ptx::tma_load_3d(sq + qb * kQBytes + d * kBlockBytes, &p.tm_q, &bars->q_full[qb], d * 64, 0, bh);
        }
        __syncwarp();
        ++loaded_seqs;
        seq_end = i + p.nb - blk;
      }
      const int slot = item % kSlots;
      if (!ptx::mbar_wait(&bars->kv_empty[slot], (static_cast<uint32_t>(item / kSlots) & 1u) ^ 1u, p.timeout_ns, abort_flag)) { ok = false; break; }
      if (ptx::elect_one()) {
        ptx::mbar_expect_tx(&bars->kv_full[slot], kSlotBytes);
        for (int d = 0; d < kDB; ++d)
          ptx::tma_load_3d(skv + slot * kSlotBytes + d * kBlockBytes, is_k ? &p.tm_k : &p.tm_v, &bars->kv_full[slot], d * 64, blk * kBKV, bh);
      }
      __syncwarp();
    }
    if (!ok && lane == 0) { fail(p, 1u, 0u, 0u); *abort_flag = 1; }
  } else if (warp == kIssuerWarp) {
    // ------------------------------ MMA issuer ------------------------------
    auto wait_item = [&](int item) {
      return ptx::mbar_wait(&bars->kv_full[item % kSlots], static_cast<uint32_t>(item / kSlots) & 1u, p.timeout_ns, abort_flag);
    };
    // scores of run block i; a sequence's first block waits for its Q, its last one hands the buffer back
    int qk_seq = -1, qk_end = 0;
    auto scores = [&](int i) {
      const int g = g_begin + i, blk = g % p.nb;
      if (i == qk_end) {
        ++qk_seq;
        qk_end = i + p.nb - blk;
        if (!ptx::mbar_wait(&bars->q_full[qk_seq & 1], static_cast<uint32_t>(qk_seq >> 1) & 1u, p.timeout_ns, abort_flag)) return false;
      }
      const int item = item_of_k(i);
      if (!wait_item(item)) return false;
      ptx::tcgen05_fence_after();
      if (ptx::elect_one()) {
        const uint64_t dq = ptx::make_smem_desc_sw128(ptx::smem_u32(sq + (qk_seq & 1) * kQBytes), 16u, 1024u);
        const uint64_t dk = ptx::make_smem_desc_sw128(ptx::smem_u32(skv + (item % kSlots) * kSlotBytes), 16u, 1024u);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint64_t off = static_cast<uint64_t>(((kk >> 2) * kBlockBytes + (kk & 3) * 32) >> 4);
          ptx::umma_f16(tmem + (i & 1) * 128, dq + off, dk + off, p.idesc_qk, kk != 0 ? 1u : 0u);
        }
        ptx::tcgen05_commit(&bars->s_full[i & 1]);
        ptx::tcgen05_commit(&bars->kv_empty[item % kSlots]);
        if (i + 1 == qk_end || i + 1 == n_run) ptx::tcgen05_commit(&bars->q_empty[qk_seq & 1]);
      }
      __syncwarp();
      return true;
    };
    bool ok = scores(0);
    if (ok && n_run > 1) ok = scores(1);
    int pv_seq = -1, pv_end = 0, pv_begin = 0;
    for (int i = 0; ok && i < n_run; ++i) {
      if (i == pv_end) {
        // first block of a sequence: both accumulators have been read
        ++pv_seq;
        pv_begin = i;
        pv_end = min(n_run, i + p.nb - (g_begin + i) % p.nb);
        ok = ptx::mbar_wait(&bars->o_free, (static_cast<uint32_t>(pv_seq) & 1u) ^ 1u, p.timeout_ns, abort_flag);
        if (!ok) break;
      }
      const int t = i & 1, item = item_of_v(i, n_run);
      ok = wait_item(item) && ptx::mbar_wait(&bars->p_full[t], static_cast<uint32_t>(i >> 1) & 1u, p.timeout_ns, abort_flag);
      if (!ok) break;
      ptx::tcgen05_fence_after();
      if (ptx::elect_one()) {
        // O_t[128, D] += P_t[128, 128 keys] V[128 keys, D]: P from TMEM, V MN-major (D contiguous)
        const uint64_t dv = ptx::make_smem_desc_sw128(ptx::smem_u32(skv + (item % kSlots) * kSlotBytes),
                                                      static_cast<uint32_t>(kBlockBytes), 1024u);
        const bool accumulate = i - pv_begin >= 2;
#pragma unroll
        for (int kk = 0; kk < kBKV / 16; ++kk) {
          const uint64_t offb = static_cast<uint64_t>((kk * 16 * 128) >> 4);
          ptx::umma_f16_ts(tmem + kOCol + t * D, tmem + t * 128 + kk * 8, dv + offb, p.idesc_pv, (accumulate || kk != 0) ? 1u : 0u);
        }
        ptx::tcgen05_commit(&bars->kv_empty[item % kSlots]);
        if (i + 1 == pv_end) ptx::tcgen05_commit(&bars->o_done);
      }
      __syncwarp();
      if (i + 2 < n_run) ok = scores(i + 2);       // lands on P_t(i): behind the product that reads it, in issue order
    }
    if (!ok && lane == 0) { fail(p, 2u, 0u, 0u); *abort_flag = 1; }
  } else if ((warp & 3) < row_warps) {
    // ------------------------------ softmax / merge / output ------------------------------
    const int t = warp >> 2;                       // block parity of this warp
    const int qd = warp & 3;                       // TMEM lane quarter of this warp
    const int row = qd * 32 + lane;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(qd * 32) << 16);
    const uint32_t t_s = lanes + t * 128;
    const uint32_t t_o = lanes + kOCol + t * D;
    const int shift = p.Sk - p.Sq;
    const int vis = p.causal ? min(p.Sk, row % p.Sq + shift + 1) : p.Sk;   // keys [0, vis) are visible to this row
    const int vis_all = p.causal ? min(p.Sk, shift + 1) : p.Sk;            // ... to every row
    bool ok = true;
    int seq = 0;
    for (int i0 = 0; ok && i0 < n_run; ++seq) {
      const int bh = (g_begin + i0) / p.nb;
      const int blk0 = (g_begin + i0) - bh * p.nb;
      const int i1 = min(n_run, i0 + p.nb - blk0);
      RowState st;
      const int mine0 = i0 + ((i0 ^ t) & 1);       // first block of this parity in the sequence
      for (int i = mine0; i < i1; i += 2) {
        if (!ptx::mbar_wait(&bars->s_full[t], static_cast<uint32_t>(i >> 1) & 1u, p.timeout_ns, abort_flag)) { ok = false; break; }
        ptx::tcgen05_fence_after();
        const int key0 = (blk0 + i - i0) * kBKV;
        attn::softmax_row_block<FMT>(t_s, t_s, key0 + kBKV > vis_all, vis - key0, p.scale_log2, st, [] {}, [&](bool move, float alpha) {
          // s_full(i) was committed behind the second product of this parity's previous block, so O_t is whole
          if (move && i > mine0) attn::rescale_o<D>(t_o, alpha);
        }, [] {}, [] {});
        ptx::tcgen05_wait_st();
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->p_full[t]);
      }
      if (!ok) break;
      // merge the two parities: both warps of a lane quarter see both maxima and sums, each finishes half of the columns
      bars->ml[seq & 1][t][row] = make_float2(st.m, st.l);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->ml_full);
      ok = ptx::mbar_wait(&bars->ml_full, static_cast<uint32_t>(seq) & 1u, p.timeout_ns, abort_flag) &&
           ptx::mbar_wait(&bars->o_done, static_cast<uint32_t>(seq) & 1u, p.timeout_ns, abort_flag);
      if (!ok) break;
      ptx::tcgen05_fence_after();
      const float2 other = bars->ml[seq & 1][t ^ 1][row];
      const bool both = i1 - i0 > 1;               // one block: only its parity's accumulator was written
      const bool any0 = both || (i0 & 1) == 0, any1 = both || (i0 & 1) == 1;
      const float m0 = t == 0 ? st.m : other.x, l0 = t == 0 ? st.l : other.y;
      const float m1 = t == 0 ? other.x : st.m, l1 = t == 0 ? other.y : st.l;
      const float m = fmaxf(m0, m1);
      const float a0 = m0 == -INFINITY ? 0.0f : ptx::ex2_approx(m0 - m);
      const float a1 = m1 == -INFINITY ? 0.0f : ptx::ex2_approx(m1 - m);
      const float l = a0 * l0 + a1 * l1;
      const bool whole = i1 - i0 == p.nb;
      const float inv = !whole ? 1.0f : (l > 0.0f ? 1.0f / l : 0.0f);
      const bool store = row < p.rows;
      const int64_t orow = static_cast<int64_t>(bh) * p.rows + row;
      const int64_t prow = (static_cast<int64_t>(blockIdx.x) + bh) * p.rows + row;
      if (!whole && store && t == 0) *reinterpret_cast<float2*>(p.part_ml + prow * 2) = make_float2(m, l);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) {
        const int col = t * (D / 2) + c * 32;
        uint32_t v0[32], v1[32];
        ptx::tmem_ld_32x32b_x32(lanes + kOCol + col, v0);
        ptx::tmem_ld_32x32b_x32(lanes + kOCol + D + col, v1);
        ptx::tcgen05_wait_ld();
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e)
          o[e] = ((any0 ? a0 * __uint_as_float(v0[e]) : 0.0f) + (any1 ? a1 * __uint_as_float(v1[e]) : 0.0f)) * inv;
        if (store && whole) {
          uint8_t* dst = static_cast<uint8_t*>(p.out) + (orow * D + col) * 2;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = pack16<FMT>(o[u * 8 + 2 * e], o[u * 8 + 2 * e + 1]);
            ptx::st_global_v4(dst + u * 16, make_uint4(w[0], w[1], w[2], w[3]));
          }
        } else if (store) {
          float* dst = p.part_o + prow * D + col;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            *reinterpret_cast<float4*>(dst + u * 4) = make_float4(o[u * 4], o[u * 4 + 1], o[u * 4 + 2], o[u * 4 + 3]);
        }
      }
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&bars->o_free);
      i0 = i1;
    }
    if (!ok && lane == 0) { fail(p, 3u, t, 0u); *abort_flag = 1; }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  if (warp == kIssuerWarp) ptx::tmem_dealloc(tmem, kTmemCols);
}

// Merges the pieces of the sequences that were cut: out = sum_c 2^(m_c - m) O_c / sum_c 2^(m_c - m) l_c. One warp per row,
// 32 pieces at a time: a lane takes the maximum and the weight of one piece, then all lanes add up its columns.
// Started early by the main kernel, whose results it waits for.
template <int D, int FMT>
__global__ void __launch_bounds__(128) flash_combine_kernel(const float* part_o, const float* part_ml, void* out, int rows, int nb, int per) {
  constexpr int kPer = D / 32;                     // columns per lane
  const int bh = blockIdx.x, r = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  ptx::grid_dependency_wait();
  const int c0 = bh * nb / per, c1 = ((bh + 1) * nb - 1) / per;
  if (r >= rows) return;
  if (c0 == c1) return;                            // written by its CTA
  float m = -INFINITY, l = 0.0f, acc[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) acc[e] = 0.0f;
  for (int base = c0; base <= c1; base += 32) {
    const int count = min(32, c1 + 1 - base);
    const int64_t pr = (static_cast<int64_t>(base) + bh) * rows + r;        // piece c: + c * rows
    const float2 ml = lane < count ? *reinterpret_cast<const float2*>(part_ml + (pr + static_cast<int64_t>(lane) * rows) * 2)
                                   : make_float2(-INFINITY, 0.0f);
    float mx = fmaxf(m, ml.x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float old = m == -INFINITY ? 0.0f : ptx::ex2_approx(m - mx);
    const float w = ml.x == -INFINITY ? 0.0f : ptx::ex2_approx(ml.x - mx);
    float wl = w * ml.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) wl += __shfl_xor_sync(0xffffffffu, wl, o);
    m = mx;
    l = l * old + wl;
#pragma unroll
    for (int e = 0; e < kPer; ++e) acc[e] *= old;
#pragma unroll 8
    for (int c = 0; c < count; ++c) {
      const float wc = __shfl_sync(0xffffffffu, w, c);
      const float* src = part_o + (pr + static_cast<int64_t>(c) * rows) * D + lane * kPer;
      float o[kPer];
      if constexpr (kPer == 4) *reinterpret_cast<float4*>(o) = *reinterpret_cast<const float4*>(src);
      else *reinterpret_cast<float2*>(o) = *reinterpret_cast<const float2*>(src);
#pragma unroll
      for (int e = 0; e < kPer; ++e) acc[e] += wc * o[e];
    }
  }
  const float inv = l > 0.0f ? 1.0f / l : 0.0f;
  uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(out) + ((static_cast<int64_t>(bh) * rows + r) * D + lane * kPer) * 2);
#pragma unroll
  for (int e = 0; e < kPer / 2; ++e) dst[e] = pack16<FMT>(acc[2 * e] * inv, acc[2 * e + 1] * inv);
}

}  // namespace decode
}  // namespace catcoc

using namespace catcoc;
using namespace catcoc::host;

namespace {
struct DecodePlan {
  int rows = 0, nb = 0, per = 0, ctas = 0;
  bool cut = false;              // some sequence is spread over several CTAs
};

// Runs of equal length over all SMs. A run is a whole number of sequences where that costs no more than two blocks
// (a block is about 1.4 us of one SM's share of the bandwidth, the second kernel and its workspace about two of them), or where
// the whole run is short: a second launch costs the caller more than the blocks (8 x 4 KV heads, 2 tokens, 700 keys 20.7 -> 15.7
// us, 4 x 4, 1 token, 576 keys 19.8 -> 15.8 with D = 64).
DecodePlan decode_plan(int B, int Hq, int Hk, int Sq, int Sk, int sms) {
  DecodePlan d;
  const int64_t bh = static_cast<int64_t>(B) * Hk;
  d.rows = Hq / Hk * Sq;
  d.nb = (Sk + decode::kBKV - 1) / decode::kBKV;
  const int64_t total = bh * d.nb;
  int64_t per = (total + sms - 1) / sms;
  if (per < 2) per = 2;                                     // both softmax groups have work
  const int64_t aligned = (bh + sms - 1) / sms * d.nb;
  if (aligned <= per + 2 || aligned <= 6) per = aligned;
  d.per = static_cast<int>(per);
  d.ctas = static_cast<int>((total + per - 1) / per);
  d.cut = per % d.nb != 0;
  return d;
}

int device_sms() {
  int device = 0;
  cudaGetDevice(&device);
  return catcoc_num_sms(device);
}
}  // namespace

// Does the few-rows kernel take this call, and with how much workspace? (-1: no)
extern "C" int64_t catcoc_flash_decode_workspace_bytes(int B, int Hq, int Hk, int Sq, int Sk, int D) {
  if (B <= 0 || Hq <= 0 || Hk <= 0 || Sq <= 0 || Sk <= 0 || Hq % Hk != 0 || (D != 64 && D != 128)) return -1;
  // The query rows of a KV head fill at most one tile of 128: the general kernel spends two tiles per query HEAD on them.
  if (static_cast<int64_t>(Hq / Hk) * Sq > decode::kRows) return -1;
  if (static_cast<int64_t>(B) * Hk * ((Sk + decode::kBKV - 1) / decode::kBKV) > (1ll << 30)) return -1;
  const DecodePlan d = decode_plan(B, Hq, Hk, Sq, Sk, device_sms());
  if (!d.cut) return 0;
  return (static_cast<int64_t>(d.ctas) + static_cast<int64_t>(B) * Hk) * d.rows * (D + 2) * static_cast<int64_t>(sizeof(float));
}

extern "C" int catcoc_flash_decode(const void* q, const void* k, const void* v, void* out, void* workspace, int B, int Hq,
                                   int Hk, int Sq, int Sk, int D, int fmt, int causal, float scale, uint32_t* status,
                                   uint64_t timeout_ns, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int64_t need = catcoc_flash_decode_workspace_bytes(B, Hq, Hk, Sq, Sk, D);
  if (!q || !k || !v || !out || !status || need < 0 || (need > 0 && workspace == nullptr)) {
    set_error("flash_decode: bad arguments");
    return CATCOC_E_BAD_ARG;
  }
  if (fmt != CATCOC_FMT_F16 && fmt != CATCOC_FMT_BF16) { set_error("flash_attention takes fp16 / bf16"); return CATCOC_E_UNSUPPORTED; }
  if (causal && Sk < Sq) { set_error("causal attention needs Sk >= Sq"); return CATCOC_E_BAD_ARG; }
  if (!(scale > 0.0f)) { set_error("flash_attention: the softmax scale must be positive (the row maximum is taken before scaling)"); return CATCOC_E_UNSUPPORTED; }
  const DecodePlan d = decode_plan(B, Hq, Hk, Sq, Sk, device_sms());
  decode::DecodeParams p;
  memset(&p, 0, sizeof(p));
  const CUtensorMapDataType dt = fmt == CATCOC_FMT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int64_t bh = static_cast<int64_t>(B) * Hk;
  int rc = encode_bsd(&p.tm_q, q, dt, bh, d.rows, D);
  if (rc == 0) rc = encode_bsd(&p.tm_k, k, dt, bh, Sk, D);
  if (rc == 0) rc = encode_bsd(&p.tm_v, v, dt, bh, Sk, D);
  if (rc != 0) return rc;
  p.out = out;
  p.BH = static_cast<int>(bh); p.rows = d.rows; p.Sq = Sq; p.Sk = Sk; p.nb = d.nb; p.per = d.per;
  if (d.cut) {
    p.part_o = static_cast<float*>(workspace);
    p.part_ml = p.part_o + (static_cast<int64_t>(d.ctas) + bh) * d.rows * D;
  }
  p.causal = causal ? 1 : 0;
  p.scale_log2 = scale * 1.4426950408889634f;
  const uint32_t f = fmt == CATCOC_FMT_BF16 ? 1u : 0u;
  p.idesc_qk = ptx::make_instr_desc(1u, f, f, 0u, 0u, 128u, 128u);
  p.idesc_pv = ptx::make_instr_desc(1u, f, f, 0u, 1u, 128u, static_cast<uint32_t>(D));
  p.status = status;
  p.timeout_ns = timeout_ns ? timeout_ns : 10000000000ull;
  const int db = D / 64;
  const int slots = D == 128 ? 4 : 8;
  const size_t smem = static_cast<size_t>(2 + slots) * db * decode::kBlockBytes + sizeof(decode::Bars) + 1024;
  auto launch = [&](auto main_kernel, auto combine_kernel) -> int {
    CATCOC_CUDA_OK(cudaFuncSetAttribute(main_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CATCOC_CUDA_OK(launch_overlapped(main_kernel, dim3(static_cast<unsigned>(d.ctas)), dim3(decode::kThreads), smem, stream, p));
    if (!d.cut) return CATCOC_OK;
    const dim3 grid(static_cast<unsigned>(bh), static_cast<unsigned>((d.rows + 3) / 4), 1);
    CATCOC_CUDA_OK(launch_overlapped(combine_kernel, grid, dim3(128), 0, stream, p.part_o, p.part_ml, out, p.rows, p.nb, p.per));
    return CATCOC_OK;
  };
  if (D == 128) {
    return fmt == CATCOC_FMT_BF16 ? launch(decode::flash_decode_kernel<128, FMT_BF16>, decode::flash_combine_kernel<128, FMT_BF16>)
                                  : launch(decode::flash_decode_kernel<128, FMT_F16>, decode::flash_combine_kernel<128, FMT_F16>);
  }
  return fmt == CATCOC_FMT_BF16 ? launch(decode::flash_decode_kernel<64, FMT_BF16>, decode::flash_combine_kernel<64, FMT_BF16>)
                                : launch(decode::flash_decode_kernel<64, FMT_F16>, decode::flash_combine_kernel<64, FMT_F16>);
}
