// Multi-head latent attention, decode step over a paged latent cache, for the query rows on the N side, on tcgen05.
//
// A decode step with 16 or 32 heads is a stream of the cache: 1152 bytes a key, one read for all heads. mla_decode.cu
// makes the query rows the M side of the products (128 lanes, mostly padding) and splits the 512 output columns over
// two CTAs, each of which fetches every key. Here the KEYS are the M side and the query rows the N side:
//
//   S^T[128 keys, N] = K[128, 576] Q^T      O^T[512, N] += V^T[512, 128 keys] P^T      N = 16, 32 or 64 rows
//
// so that one CTA holds all 512 output columns (four accumulators of N columns) and nothing is fetched twice. The
// first product reads a page as it lies (K-major), the second reads the same bytes MN-major; P^T goes through shared
// memory. A thread of the softmax owns one key: the row maxima run across threads, so they are only taken when some
// score exceeds its row's reference maximum by more than 2^8 (one vote of the warpgroup per block says so); in the
// other blocks the step is N exponentials a thread.
//
// The pages of all sequences form one list, cut into equal runs over the SMs (lengths are device data: every CTA sums
// them itself); pieces of a sequence that was cut go to a workspace and mla_rows_combine_kernel merges them.
//
//   warps 0..3 (64 rows: 0..7, 32 rows to a warpgroup)  softmax, rescale, output      then one warp each  TMA producer, MMA issuer
//
// Shared memory: Q, P, one or two rotary blocks (16 KiB) and five slots of two latent blocks (32 KiB): a page needs
// four, and a slot is free again as soon as its quarter of the second product is done. 64 rows leave room for four slots, and P
// lies where the page's rotary block was.
//
// Bound by HBM and the depth of the slots: batch 32, 16 heads, 2048 to 4096 keys (113 MB), in a loop: 82 us in mla_decode.cu,
// 31 us here (3.7 TB/s); with 12288 keys on average 232 -> 81 us (5.6 TB/s). Straight-line code is kept short on purpose: a run is a few
// pages, and with everything unrolled the instruction fetch of a cold launch cost up to 50 us.
//
// The reference carries this computation as 3rdparty/catlass/examples/19_mla/mla_kernel.cpp.
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
namespace mlar {

constexpr int kDV = 512, kDR = 64;
constexpr int kPage = 128;                   // keys per page == TMEM lanes of S^T
constexpr int kBlockBytes = kPage * 128;     // 128 keys x 64 columns
constexpr int kPairBytes = 2 * kBlockBytes;
constexpr int kPairs = kDV / 128;            // pairs of latent blocks per page
using attn::kLazyRescale;

template <int N> struct Geo {
  // 64 rows: P^T of a page (16 KiB) lies where its rotary block was, which the scores have read by then
  static constexpr bool kShared = N == 64;
  static constexpr int kRopeSlots = N == 16 ? 2 : 1, kPairSlots = kShared ? 4 : 5;
  static constexpr uint32_t kOCol = N < 32 ? 32 : N, kTmemCols = N == 64 ? 512 : 256;
  static constexpr int kW = N < 32 ? N : 32;           // rows of a softmax thread: 64 rows have two warpgroups
  static constexpr int kSoftWarps = 4 * N / kW, kProducerWarp = kSoftWarps, kIssuerWarp = kSoftWarps + 1, kThreads = 32 * (kSoftWarps + 2);
  static constexpr int kQChunk = N * 128;              // N rows x 64 columns
  static constexpr int kQBytes = 9 * kQChunk;
  static constexpr int kPBytes = 2 * N * 128;          // N rows x 128 keys, two blocks of 64 keys
  static constexpr int kTail = kQBytes + (kShared ? 0 : kPBytes) + kRopeSlots * kBlockBytes + kPairSlots * kPairBytes;
  static_assert(!kShared || kPBytes <= kBlockBytes);
};

struct RowsParams {
  CUtensorMap tm_qn, tm_qr;       // q_nope {64, rows, 8}, box {64, N, 8} / q_rope {64, rows}, box {64, N}
  CUtensorMap tm_kn, tm_kr;       // latent {64, 128, 8, pages}, box {64, 128, 2, 1} / rotary {64, 128, pages}, box {64, 128, 1}
  const int* block_table;         // [B, max_pages]
  const int* kv_lens;             // [B]
  void* out;                      // [B * rows_per_item, 512]
  float* part_o;                  // [2 * run + (0: first piece of the run, 1: last)][chunk][N][512]
  float* part_ml;                 // the same without the columns, (m, l)
  int2* place;                    // [B] of a sequence with pages: where its first page stands in the list, pages per run
  int B, q_len, H, max_pages, num_pages, rows_per_item, chunks;
  int causal;
  float scale_log2;
  uint32_t idesc_qk, idesc_pv;
  uint32_t* status;
  uint64_t timeout_ns;
};

struct Bars {
  uint64_t q_full, q_empty, rope_full[2], rope_empty[2], pair_full[5], pair_empty[5], s_full, p_full, pv_done;
  uint32_t tmem_base, abort_flag;
  float wmax[4][64], lsum[4][64], m[64], alpha[64];
};

CATCOC_DEVICE void fail(const RowsParams& p, uint32_t what, uint32_t a) {
  if (atomicCAS(p.status, 0u, static_cast<uint32_t>(STATUS_TIMEOUT_PIPELINE)) == 0u) {
    p.status[1] = 0u; p.status[2] = 400u + what; p.status[3] = a; p.status[4] = 0u; p.status[5] = 0u;
    p.status[6] = blockIdx.x;
    __threadfence_system();
  }
}

CATCOC_DEVICE int item_len(const int* kv_lens, int max_pages, int item) { return min(max(0, kv_lens[item]), max_pages * kPage); }
CATCOC_DEVICE int item_pages(const int* kv_lens, int max_pages, int item) { return (item_len(kv_lens, max_pages, item) + kPage - 1) / kPage; }

// Equal runs; from 33 pages on at least two each (128 pieces of one page take longer to merge than a second page to read)
CATCOC_DEVICE int pages_per_run(int total, int runs) { return max(total > 32 ? 2 : 1, (total + runs - 1) / runs); }

// This CTA's run of the page list (computed by every warp for itself)
struct Run {
  int n;            // pages of the run
  int begin, per;   // where it starts in the page list, pages per run
  int item, page;   // where it starts
  CATCOC_DEVICE Run(const RowsParams& p, int lane) {
    int sum = 0;
    for (int i = lane; i < p.B; i += 32) sum += item_pages(p.kv_lens, p.max_pages, i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    per = pages_per_run(sum, static_cast<int>(gridDim.x));
    begin = static_cast<int>(blockIdx.x) * per;
    n = min(sum, begin + per) - begin;
    item = 0; page = 0;
    if (n <= 0) { n = 0; return; }
    int before = 0;
    for (int base = 0; base < p.B; base += 32) {
      const int mine = base + lane < p.B ? item_pages(p.kv_lens, p.max_pages, base + lane) : 0;
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const int lo = before + incl - mine;
      const uint32_t hit = __ballot_sync(0xffffffffu, begin >= lo && begin < lo + mine);
      if (hit != 0u) {
        const int l = __ffs(hit) - 1;
        item = base + l;
        page = begin - __shfl_sync(0xffffffffu, lo, l);
        return;
      }
      before += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
};

// Pieces of a run, one per sequence it touches
struct Piece {
  int i0, i1;            // run indexes
  int item, page0, pages;
  CATCOC_DEVICE Piece(const RowsParams& p, const Run& r) : i0(0), item(r.item), page0(r.page) { open(p, r); }
  CATCOC_DEVICE void open(const RowsParams& p, const Run& r) {
    pages = item_pages(p.kv_lens, p.max_pages, item);
    i1 = min(r.n, i0 + pages - page0);
  }
  CATCOC_DEVICE void next(const RowsParams& p, const Run& r) {
    i0 = i1;
    page0 = 0;
    if (i0 >= r.n) return;
    do ++item; while (item + 1 < p.B && item_pages(p.kv_lens, p.max_pages, item) == 0);
    open(p, r);
  }
};

CATCOC_DEVICE bool vote_any(int bar, bool pred) {          // of the 128 threads of a softmax warpgroup
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r) : "r"(static_cast<uint32_t>(pred)), "r"(bar) : "memory");
  return r != 0u;
}
CATCOC_DEVICE float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
template <int W> CATCOC_DEVICE void tmem_ld_n(uint32_t taddr, uint32_t (&r)[W]) {
  if constexpr (W == 32) ptx::tmem_ld_32x32b_x32(taddr, r);
  else ptx::tmem_ld_32x32b_x16(taddr, r);
}
template <int W> CATCOC_DEVICE void tmem_st_n(uint32_t taddr, const uint32_t (&r)[W]) {
  if constexpr (W == 32) ptx::tmem_st_32x32b_x32(taddr, r);
  else ptx::tmem_st_32x32b_x16(taddr, r);
}
template <int FMT> CATCOC_DEVICE uint16_t cvt16(float x) {
  if constexpr (FMT == FMT_BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(x));
  else return __half_as_ushort(__float2half_rn(x));
}

template <int N, int FMT>
__global__ void __launch_bounds__(Geo<N>::kThreads, 1) mla_rows_kernel(const __grid_constant__ RowsParams p) {
  using G = Geo<N>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* sq = smem;
  uint8_t* sp = sq + G::kQBytes;
  uint8_t* srope = G::kShared ? sp : sp + G::kPBytes;
  uint8_t* spair = srope + G::kRopeSlots * kBlockBytes;
  Bars* bars = reinterpret_cast<Bars*>(smem + G::kTail);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunk = blockIdx.y;                     // N query rows of every sequence

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    ptx::mbar_init(&bars->q_empty, 1);
    for (int s = 0; s < 2; ++s) { ptx::mbar_init(&bars->rope_full[s], 1); ptx::mbar_init(&bars->rope_empty[s], 1); }
    for (int s = 0; s < G::kPairSlots; ++s) { ptx::mbar_init(&bars->pair_full[s], 1); ptx::mbar_init(&bars->pair_empty[s], 1); }
    ptx::mbar_init(&bars->s_full, 1);
    ptx::mbar_init(&bars->p_full, G::kSoftWarps);
    ptx::mbar_init(&bars->pv_done, 1);
    bars->abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tmap(&p.tm_qn); ptx::prefetch_tmap(&p.tm_qr); ptx::prefetch_tmap(&p.tm_kn); ptx::prefetch_tmap(&p.tm_kr);
  }
  if (warp == G::kIssuerWarp) { ptx::tmem_alloc(&bars->tmem_base, G::kTmemCols); ptx::tmem_relinquish(); }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem = bars->tmem_base;
  ptx::grid_dependency_wait();
  ptx::launch_dependents();                         // the combine kernel waits for this grid's results by itself
  const Run run(p, lane);

  if (run.n == 0) {
    // nothing for this CTA
  } else if (warp == G::kProducerWarp) {
    // ------------------------------ TMA producer ------------------------------
    bool ok = true;
    int seq = 0;
    for (Piece pc(p, run); ok && pc.i0 < run.n; pc.next(p, run), ++seq) {
      const int* table = p.block_table + static_cast<int64_t>(pc.item) * p.max_pages;
      int page_next = table[pc.page0];
      for (int i = pc.i0; ok && i < pc.i1; ++i) {
        // a bad entry reads a wrong page, never outside the cache
        const int page = min(max(page_next, 0), p.num_pages - 1);
        if (i + 1 < pc.i1) page_next = table[pc.page0 + (i + 1 - pc.i0)];
        const int rs = i % G::kRopeSlots;
        auto rotary = [&] {
          ok = ptx::mbar_wait(&bars->rope_empty[rs], (static_cast<uint32_t>(i / G::kRopeSlots) & 1u) ^ 1u, p.timeout_ns, abort_flag);
          if (ok && ptx::elect_one()) {
            ptx::mbar_expect_tx(&bars->rope_full[rs], kBlockBytes);
            ptx::tma_load_3d(srope + rs * kBlockBytes, &p.tm_kr, &bars->rope_full[rs], 0, 0, page);
          }
          __syncwarp();
        };
        if (!G::kShared) rotary();
        for (int c = 0; ok && c < kPairs; ++c) {
          const int it = i * kPairs + c, slot = it % G::kPairSlots;
          ok = ptx::mbar_wait(&bars->pair_empty[slot], (static_cast<uint32_t>(it / G::kPairSlots) & 1u) ^ 1u, p.timeout_ns, abort_flag);
          if (!ok) break;
          if (ptx::elect_one()) {
            ptx::mbar_expect_tx(&bars->pair_full[slot], kPairBytes);
            ptx::tma_load_4d(spair + slot * kPairBytes, &p.tm_kn, &bars->pair_full[slot], 0, 0, 2 * c, page);
          }
          __syncwarp();
          if (c == 0 && i == pc.i0) {
            // the rows of this sequence, behind the copies that the free slots take anyway
            ok = ptx::mbar_wait(&bars->q_empty, (static_cast<uint32_t>(seq) & 1u) ^ 1u, p.timeout_ns, abort_flag);
            if (!ok) break;
            if (ptx::elect_one()) {
              const int grow0 = pc.item * p.rows_per_item + chunk * N;
              ptx::mbar_expect_tx(&bars->q_full, G::kQBytes);
              ptx::tma_load_3d(sq, &p.tm_qn, &bars->q_full, 0, grow0, 0);
              ptx::tma_load_2d(sq + 8 * G::kQChunk, &p.tm_qr, &bars->q_full, 0, grow0);
            }
            __syncwarp();
          }
        }
        if (G::kShared && ok) rotary();   // free only behind the whole second product of the page before
      }
    }
    if (!ok && lane == 0) { fail(p, 1u, 0u); *abort_flag = 1; }
  } else if (warp == G::kIssuerWarp) {
    // ------------------------------ MMA issuer ------------------------------
    bool ok = true;
    int seq = 0;
    for (Piece pc(p, run); ok && pc.i0 < run.n; pc.next(p, run), ++seq) {
      ok = ptx::mbar_wait(&bars->q_full, static_cast<uint32_t>(seq) & 1u, p.timeout_ns, abort_flag);
      const int kv_len = item_len(p.kv_lens, p.max_pages, pc.item);
      for (int i = pc.i0; ok && i < pc.i1; ++i) {
        // S^T = K Q^T, 64 columns of the keys at a time: the rotary block, then the latent ones (as they arrive: where the rotary
        // block shares its place with P, the other way around)
        const int rs = i % G::kRopeSlots;
        auto scores64 = [&](const uint8_t* kblk, int qchunk, bool first) {
          const uint64_t dk = ptx::make_smem_desc_sw128(ptx::smem_u32(kblk), 16u, 1024u);
          const uint64_t dq = ptx::make_smem_desc_sw128(ptx::smem_u32(sq + qchunk * G::kQChunk), 16u, 1024u);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            ptx::umma_f16(tmem, dk + static_cast<uint64_t>(kk * 2), dq + static_cast<uint64_t>(kk * 2), p.idesc_qk,
                          (first && kk == 0) ? 0u : 1u);
        };
        auto last = [&] {
          ptx::tcgen05_commit(&bars->s_full);
          if (i + 1 == pc.i1) ptx::tcgen05_commit(&bars->q_empty);
        };
        auto rotary = [&] {
          ok = ptx::mbar_wait(&bars->rope_full[rs], static_cast<uint32_t>(i / G::kRopeSlots) & 1u, p.timeout_ns, abort_flag);
          ptx::tcgen05_fence_after();
          if (ok && ptx::elect_one()) {
            scores64(srope + rs * kBlockBytes, 8, !G::kShared);
            if (G::kShared) last();
            else ptx::tcgen05_commit(&bars->rope_empty[rs]);
          }
          __syncwarp();
        };
        if (!G::kShared) rotary();
        for (int c = 0; ok && c < kPairs; ++c) {
          const int it = i * kPairs + c, slot = it % G::kPairSlots;
          ok = ptx::mbar_wait(&bars->pair_full[slot], static_cast<uint32_t>(it / G::kPairSlots) & 1u, p.timeout_ns, abort_flag);
          if (!ok) break;
          ptx::tcgen05_fence_after();
          if (ptx::elect_one()) {
            scores64(spair + slot * kPairBytes, 2 * c, G::kShared && c == 0);
            scores64(spair + slot * kPairBytes + kBlockBytes, 2 * c + 1, false);
            if (!G::kShared && c == kPairs - 1) last();
          }
          __syncwarp();
        }
        if (G::kShared && ok) rotary();
        if (!ok) break;
        // O^T += V^T P^T, 128 output columns (one slot) at a time. Only keys of the sequence, 16 at a time: what lies behind
        // them in its last page has probability zero, but may hold anything, and zero times an infinity is a NaN
        const int steps = min(kPage, kv_len - (pc.page0 + i - pc.i0) * kPage + 15) / 16;
        ok = ptx::mbar_wait(&bars->p_full, static_cast<uint32_t>(i) & 1u, p.timeout_ns, abort_flag);
        if (!ok) break;
        ptx::tcgen05_fence_after();
        if (ptx::elect_one()) {
#pragma unroll
          for (int c = 0; c < kPairs; ++c) {
            const int slot = (i * kPairs + c) % G::kPairSlots;
            const uint64_t dv = ptx::make_smem_desc_sw128(ptx::smem_u32(spair + slot * kPairBytes), static_cast<uint32_t>(kBlockBytes), 1024u);
#pragma unroll
            for (int kk = 0; kk < kPage / 16; ++kk) {
              if (kk >= steps) break;
              const uint64_t dp = ptx::make_smem_desc_sw128(ptx::smem_u32(sp + (kk >> 2) * N * 128), 16u, 1024u) + static_cast<uint64_t>((kk & 3) * 2);
              ptx::umma_f16(tmem + G::kOCol + c * N, dv + static_cast<uint64_t>((kk * 2048) >> 4), dp, p.idesc_pv,
                            (i > pc.i0 || kk != 0) ? 1u : 0u);
            }
            ptx::tcgen05_commit(&bars->pair_empty[slot]);
          }
          if (G::kShared) ptx::tcgen05_commit(&bars->rope_empty[rs]);
          ptx::tcgen05_commit(&bars->pv_done);
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) { fail(p, 2u, 0u); *abort_flag = 1; }
  } else {
    // ------------------------------ softmax / rescale / output ------------------------------
    // A wait that failed is carried into the next vote, so that the four warps of a warpgroup leave the loop together.
    constexpr int W = G::kW;
    const int sw = warp & 3, g = (warp >> 2) * W, bar = 1 + (warp >> 2), tid = threadIdx.x & 127;   // rows [g, g + W) of the chunk
    const int key = sw * 32 + lane;                // key of the page == TMEM lane; also a column of 128 in the output
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(sw * 32) << 16);
    uint8_t* p_key = sp + (key >> 6) * N * 128 + g * 128 + (key & 7) * 2;   // P^T row g + r: + r * 128 + ((unit ^ (r & 7)) << 4)
    const int p_unit = (key & 63) >> 3;
    const float sc = p.scale_log2;
    bool bad = false;
    for (Piece pc(p, run); !bad && pc.i0 < run.n; pc.next(p, run)) {
      if (chunk == 0 && threadIdx.x == 0 && pc.page0 == 0) p.place[pc.item] = make_int2(run.begin + pc.i0, run.per);
      const int kv_len = item_len(p.kv_lens, p.max_pages, pc.item);
      const int vis_all = p.causal ? max(0, kv_len - (p.q_len - 1)) : kv_len;   // keys every row sees
      // lane r: the keys that row g + r of this chunk sees (with the causal mask a new token does not see those behind it)
      const int vis_lane = p.causal ? kv_len - (p.q_len - 1 - min((chunk * N + g + lane) / p.H, p.q_len - 1)) : kv_len;
      float nm[W], l[W];                             // minus the reference maximum (log2 domain), this key's share of the sum
#pragma unroll
      for (int r = 0; r < W; ++r) { nm[r] = INFINITY; l[r] = 0.0f; }
      if (tid < W) bars->m[g + tid] = -INFINITY;     // read behind the first block's barriers
      for (int i = pc.i0; i < pc.i1; ++i) {
        bad = !ptx::mbar_wait(&bars->s_full, static_cast<uint32_t>(i) & 1u, p.timeout_ns, abort_flag);
        ptx::tcgen05_fence_after();
        uint32_t v[W];
        tmem_ld_n<W>(t_lane + g, v);
        ptx::tcgen05_wait_ld();
        const int key0 = (pc.page0 + i - pc.i0) * kPage;
        if (key0 + kPage > vis_all) {
#pragma unroll
          for (int r = 0; r < W; ++r)
            if (key0 + key >= __shfl_sync(0xffffffffu, vis_lane, r)) v[r] = 0xff800000u;
        }
        bool over = bad;
#pragma unroll
        for (int r = 0; r < W; ++r) over = over || fmaf(__uint_as_float(v[r]), sc, nm[r]) > kLazyRescale;
        // the second product of the block before has read P, and O holds it
        if (i > 0 && !ptx::mbar_wait(&bars->pv_done, static_cast<uint32_t>(i - 1) & 1u, p.timeout_ns, abort_flag)) { bad = true; over = true; }
        if (vote_any(bar, over)) {
          bad = vote_any(bar, bad);
          if (bad) break;
          float mine = -INFINITY;
#pragma unroll
          for (int r = 0; r < W; ++r) {
            const float w = warp_max(__uint_as_float(v[r]));
            if (lane == r) mine = w;
          }
          if (lane < W) bars->wmax[sw][g + lane] = mine;
          ptx::named_bar_sync(bar, 128);
          if (tid < W) {
            const int r = g + tid;
            const float m_old = bars->m[r];
            const float m_new = fmaxf(m_old, fmaxf(fmaxf(bars->wmax[0][r], bars->wmax[1][r]), fmaxf(bars->wmax[2][r], bars->wmax[3][r])) * sc);
            bars->m[r] = m_new;
            bars->alpha[r] = m_old == -INFINITY ? 0.0f : ptx::ex2_approx(m_old - m_new);
          }
          ptx::named_bar_sync(bar, 128);
#pragma unroll
          for (int r = 0; r < W; ++r) { nm[r] = -bars->m[g + r]; l[r] *= bars->alpha[g + r]; }
          if (i > pc.i0) {
            ptx::tcgen05_fence_after();
#pragma unroll 1
            for (int c = 0; c < kPairs; ++c) {
              uint32_t o[W];
              tmem_ld_n<W>(t_lane + G::kOCol + c * N + g, o);
              ptx::tcgen05_wait_ld();
#pragma unroll
              for (int r = 0; r < W; ++r) o[r] = __float_as_uint(__uint_as_float(o[r]) * bars->alpha[g + r]);
              tmem_st_n<W>(t_lane + G::kOCol + c * N + g, o);
            }
            ptx::tcgen05_wait_st();
          }
        }
#pragma unroll
        for (int r = 0; r < W; ++r) {
          const float e = ptx::ex2_approx(fmaf(__uint_as_float(v[r]), sc, nm[r] == INFINITY ? 0.0f : nm[r]));   // a row that sees nothing yet
          l[r] += e;
          *reinterpret_cast<uint16_t*>(p_key + r * 128 + ((p_unit ^ (r & 7)) << 4)) = cvt16<FMT>(e);
        }
        ptx::fence_proxy_async_smem();
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&bars->p_full);
      }
      if (bad) break;
      // end of the sequence's piece: sums over the keys (lane r ends with the sum of row g + r over its warp), then O
#pragma unroll
      for (int step = W / 2; step > 0; step >>= 1) {
        const bool up = (lane & step) != 0;
#pragma unroll
        for (int r = 0; r < step; ++r) {
          const float give = up ? l[r] : l[r + step], keep = up ? l[r + step] : l[r];
          l[r] = keep + __shfl_xor_sync(0xffffffffu, give, step);
        }
      }
      if constexpr (N == 16) l[0] += __shfl_xor_sync(0xffffffffu, l[0], 16);
      if (lane < W) bars->lsum[sw][g + lane] = l[0];
      bad = !ptx::mbar_wait(&bars->pv_done, static_cast<uint32_t>(pc.i1 - 1) & 1u, p.timeout_ns, abort_flag);
      bad = vote_any(bar, bad);
      if (bad) break;
      ptx::tcgen05_fence_after();
      const int rows = min(W, p.rows_per_item - chunk * N - g);      // of this warpgroup (none: 0 or less)
      const bool whole = pc.i1 - pc.i0 == pc.pages;
      const int64_t row0 = static_cast<int64_t>(pc.item) * p.rows_per_item + chunk * N + g;
      const int64_t part0 = ((static_cast<int64_t>(blockIdx.x) * 2 + (pc.i0 == 0 ? 0 : 1)) * p.chunks + chunk) * N + g;
      const int lr = g + (lane & (W - 1));
      const float l_row = (bars->lsum[0][lr] + bars->lsum[1][lr]) + (bars->lsum[2][lr] + bars->lsum[3][lr]);
      if (!whole && key < rows) *reinterpret_cast<float2*>(p.part_ml + (part0 + key) * 2) = make_float2(bars->m[g + key], l_row);
      const float inv_row = l_row > 0.0f ? 1.0f / l_row : 0.0f;
#pragma unroll 1
      for (int c = 0; c < kPairs; ++c) {
        uint32_t o[W];
        tmem_ld_n<W>(t_lane + G::kOCol + c * N + g, o);
        ptx::tcgen05_wait_ld();
        if (whole) {
          uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + row0 * kDV + c * 128 + key;
#pragma unroll
          for (int r = 0; r < W; ++r) {
            const float x = __uint_as_float(o[r]) * __shfl_sync(0xffffffffu, inv_row, r);
            if (r < rows) dst[r * kDV] = cvt16<FMT>(x);
          }
        } else {
          float* dst = p.part_o + part0 * kDV + c * 128 + key;
#pragma unroll
          for (int r = 0; r < W; ++r)
            if (r < rows) dst[r * kDV] = __uint_as_float(o[r]);
        }
      }
      ptx::tcgen05_fence_before();
      // m and lsum have been read by everyone before the next piece writes them
      bad = vote_any(bar, false);
    }
    if (bad && lane == 0) { fail(p, 3u, 0u); *abort_flag = 1; }
  }

  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  if (warp == G::kIssuerWarp) ptx::tmem_dealloc(tmem, G::kTmemCols);
}

// Merges the pieces of the sequences that were cut, and zeroes the rows of empty sequences. One block per (row, sequence).
template <int FMT>
__global__ void __launch_bounds__(128) mla_rows_combine_kernel(const float* part_o, const float* part_ml, const int2* place, void* out,
                                                               const int* kv_lens, int max_pages, int rows_per_item, int chunks, int n, int runs) {
  constexpr int kPieces = 8;                       // loads in flight per thread
  __shared__ float s_max[4], s_w[128], s_wl[128];
  const int item = blockIdx.y, row = blockIdx.x;
  ptx::grid_dependency_wait();
  const int pages = item_pages(kv_lens, max_pages, item);
  // not written for a sequence without pages, nor behind a wait that ran out: whatever it holds, the pieces read are the workspace's
  const int2 at = place[item];
  const int before = min(max(0, at.x), 1 << 24), per = max(1, at.y);
  const int c0 = min(before / per, runs - 1), c1 = min((before + pages - 1) / per, runs - 1);
  if (pages > 0 && c0 == c1) return;               // written by its CTA
  const int col = threadIdx.x * 4;
  const int chunk = row / n, r = row - chunk * n;
  // a sequence is the first piece of every run but the one it starts in, where it is the last unless it starts the run
  auto index = [&](int c) { return ((static_cast<int64_t>(c) * 2 + (before > c * per ? 1 : 0)) * chunks + chunk) * n + r; };
  // 128 pieces at a time: their maxima and weights side by side, one per thread, then their O
  float m = -INFINITY, l = 0.0f;
  float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int base = c0; pages > 0 && base <= c1; base += 128) {
    const int count = min(128, c1 + 1 - base);
    // O of the first pieces is on its way while their weights are worked out
    float4 o[kPieces];
    auto fetch = [&](int c) {
#pragma unroll
      for (int e = 0; e < kPieces; ++e)
        o[e] = c + e < count ? *reinterpret_cast<const float4*>(part_o + index(base + c + e) * kDV + col) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    fetch(0);
    const float2 ml = static_cast<int>(threadIdx.x) < count ? *reinterpret_cast<const float2*>(part_ml + index(base + threadIdx.x) * 2)
                                                            : make_float2(-INFINITY, 0.0f);
    float mx = warp_max(ml.x);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(m, fmaxf(s_max[0], s_max[1])), fmaxf(s_max[2], s_max[3]));
    const float old = m == -INFINITY ? 0.0f : ptx::ex2_approx(m - mx);
    const float w = ml.x == -INFINITY ? 0.0f : ptx::ex2_approx(ml.x - mx);
    s_w[threadIdx.x] = w;
    s_wl[threadIdx.x] = w * ml.y;
    __syncthreads();
    m = mx;
    l *= old;
    acc.x *= old; acc.y *= old; acc.z *= old; acc.w *= old;
    for (int c = 0; c < count; c += kPieces) {
      if (c > 0) fetch(c);
#pragma unroll
      for (int e = 0; e < kPieces; ++e) {          // (past the last piece: weights of zero)
        const float wc = s_w[c + e];
        l += s_wl[c + e];
        acc.x += wc * o[e].x; acc.y += wc * o[e].y; acc.z += wc * o[e].z; acc.w += wc * o[e].w;
      }
    }
  }
  const float inv = l > 0.0f ? 1.0f / l : 0.0f;
  uint2 packed;
  packed.x = attn::pack16<FMT>(acc.x * inv, acc.y * inv);
  packed.y = attn::pack16<FMT>(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(static_cast<uint8_t*>(out) + ((static_cast<int64_t>(item) * rows_per_item + row) * kDV + col) * 2) = packed;
}

}  // namespace mlar
}  // namespace catcoc

using namespace catcoc;
using namespace catcoc::host;

namespace {
struct RowsPlan {
  int n = 0, chunks = 0, runs = 0;
};
// Rows of a CTA. 64 rows read every page half as often, but the page's slots are its only ones: the loads of the next page wait
// for the second product, a pass takes 1.3 to 1.5 times as long, and a piece leaves twice the partial sums. In a loop, bf16,
// chunks of 32 -> of 64 rows, by the passes of 32 rows over a page that an SM makes:
//   an even number of chunks, four or more: 2 to 5 passes 22.5 -> 24.2 us, 27.7 -> 29.5; 6 passes 26.6 -> 27.9; 7 passes 27.7 -> 27.3, 28.0 -> 27.2; 11 passes 46.6 -> 48.4; 14
//     passes 44.6 -> 40.9, 43.7 -> 38.4; 55 passes 135 -> 104; 221 passes 507 -> 344
//   two: 5 passes 31.2 -> 34.0, 14 passes 48.9 -> 50.1, 28 passes 80.2 -> 71.7; 110 passes 335 -> 262
//   three (a quarter of the rows is padding): 10 passes 34.9 -> 38.6, 21 passes 64.5 -> 68.3, 41 passes 105 -> 101
int chunk_rows(int rows_per_item, int64_t page_slots, int sms) {
  if (rows_per_item <= 32) return rows_per_item <= 16 ? 16 : 32;
  const int chunks = (rows_per_item + 31) / 32;
  const int64_t line = chunks >= 4 && chunks % 2 == 0 ? 12 : 24;
  return page_slots * chunks > line * sms ? 64 : 32;
}
RowsPlan rows_plan(int rows_per_item, int64_t page_slots) {
  RowsPlan d;
  int device = 0;
  cudaGetDevice(&device);
  const int sms = catcoc_num_sms(device);
  d.n = chunk_rows(rows_per_item, page_slots, sms);
  d.chunks = (rows_per_item + d.n - 1) / d.n;
  d.runs = sms / d.chunks;
  if (d.runs < 1) d.runs = 1;
  return d;
}

int encode_map(CUtensorMap* tm, const void* base, CUtensorMapDataType dt, int rank, const cuuint64_t* gdim, const cuuint64_t* gstride,
               const cuuint32_t* box) {
  static EncodeTiledFn fn = driver_fn<EncodeTiledFn>("cuTensorMapEncodeTiled");
  if (fn == nullptr) return CATCOC_E_DRIVER;
  if (reinterpret_cast<uintptr_t>(base) & 15) { set_error("mla_decode operands must be 16-byte aligned"); return CATCOC_E_ALIGNMENT; }
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(tm, dt, static_cast<cuuint32_t>(rank), const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled (mla) failed: CUresult %d", static_cast<int>(r)); return CATCOC_E_DRIVER; }
  return CATCOC_OK;
}
}  // namespace

// Scratch of the few-rows kernel, or -1 when the general one takes the call.
extern "C" int64_t catcoc_mla_rows_workspace_bytes(int B, int q_len, int H, int max_pages) {
  if (B <= 0 || q_len < 1 || q_len > 4 || H <= 0 || max_pages <= 0) return -1;
  const int64_t rows = static_cast<int64_t>(q_len) * H;
  // The chunks of a sequence's rows read a page side by side (from L2 but for the first). Measured against mla_decode.cu in a
  // loop, batch 32, sequences of 2048 to 4096 keys, bf16: 16 rows 83 -> 29 us, 32 rows 83 -> 33, 64 rows 87 -> 47, 128 rows
  // 148 -> 67, 192 rows 264 -> 87, 512 rows 445 -> 194; 128 sequences of up to 300 keys, 512 rows 150 -> 136. Up to 1024 rows,
  // 16 chunks of 64: that many runs side by side are still nine pieces of the page list.
  if (rows > 1024) return -1;
  if (B > 65535 || static_cast<int64_t>(B) * max_pages > (1 << 24)) return -1;
  // One page a sequence: the general kernel is a single launch, which is what such a call waits for (batch 1 to 128, 16 to 128
  // rows, back to back: 19 to 21 us against 24). Larger batches are several waves of its CTAs.
  if (max_pages == 1 && B <= 128) return -1;
  // Short sequences of more than 128 rows: the general kernel takes 8.3 us and 6.1 us a page for each 148 of its CTAs (at least
  // for one such set), this one about 17 us and 3.3 us for every pass of 32 rows over a page that an SM makes. 37 sequences of 256
  // rows, 2 to 6 pages: 20 to 45 us against 32 to 47; 64 of 512 rows: 68 against 77 at two pages, 91 against 83 at three.
  if (rows > 128 && max_pages <= 6) {
    int device = 0;
    cudaGetDevice(&device);
    const int64_t sms = catcoc_num_sms(device), ctas = 2 * B * ((rows + 127) / 128), passes = static_cast<int64_t>(B) * max_pages * ((rows + 31) / 32);
    if (max_pages <= 2 || std::max(sms, ctas) * (83 + 61 * max_pages) < sms * 170 + passes * 33) return -1;
  }
  const RowsPlan d = rows_plan(static_cast<int>(rows), static_cast<int64_t>(B) * max_pages);
  return static_cast<int64_t>(d.runs) * 2 * d.chunks * d.n * (mlar::kDV + 2) * static_cast<int64_t>(sizeof(float)) + B * static_cast<int64_t>(sizeof(int2));
}

extern "C" int catcoc_mla_rows(const void* q_nope, const void* q_rope, const void* ckv, const void* krope, const int* block_table,
                               const int* kv_lens, void* out, void* workspace, int B, int q_len, int H, int num_pages, int max_pages,
                               int fmt, int causal, float scale, uint32_t* status, uint64_t timeout_ns, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (!q_nope || !q_rope || !ckv || !krope || !block_table || !kv_lens || !out || !status || !workspace || num_pages <= 0 ||
      catcoc_mla_rows_workspace_bytes(B, q_len, H, max_pages) < 0) {
    set_error("mla_decode: bad arguments");
    return CATCOC_E_BAD_ARG;
  }
  if (fmt != CATCOC_FMT_F16 && fmt != CATCOC_FMT_BF16) { set_error("mla_decode takes fp16 / bf16"); return CATCOC_E_UNSUPPORTED; }
  if (!(scale > 0.0f)) { set_error("mla_decode: the softmax scale must be positive"); return CATCOC_E_UNSUPPORTED; }
  const int rows_per_item = q_len * H;
  const RowsPlan d = rows_plan(rows_per_item, static_cast<int64_t>(B) * max_pages);
  mlar::RowsParams p;
  memset(&p, 0, sizeof(p));
  const CUtensorMapDataType dt = fmt == CATCOC_FMT_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const cuuint64_t rows = static_cast<cuuint64_t>(B) * rows_per_item, pages = static_cast<cuuint64_t>(num_pages);
  const cuuint32_t n = static_cast<cuuint32_t>(d.n);
  // the 512 latent columns as eight blocks of 64 behind the rows: one copy lays the blocks out one after the other
  const cuuint64_t qn_dim[3] = {64, rows, 8}, qn_str[2] = {mlar::kDV * 2, 128};
  const cuuint32_t qn_box[3] = {64, n, 8};
  const cuuint64_t qr_dim[2] = {64, rows}, qr_str[1] = {mlar::kDR * 2};
  const cuuint32_t qr_box[2] = {64, n};
  const cuuint64_t kn_dim[4] = {64, mlar::kPage, 8, pages}, kn_str[3] = {mlar::kDV * 2, 128, mlar::kPage * mlar::kDV * 2};
  const cuuint32_t kn_box[4] = {64, mlar::kPage, 2, 1};
  const cuuint64_t kr_dim[3] = {64, mlar::kPage, pages}, kr_str[2] = {mlar::kDR * 2, mlar::kPage * mlar::kDR * 2};
  const cuuint32_t kr_box[3] = {64, mlar::kPage, 1};
  int rc = encode_map(&p.tm_qn, q_nope, dt, 3, qn_dim, qn_str, qn_box);
  if (rc == 0) rc = encode_map(&p.tm_qr, q_rope, dt, 2, qr_dim, qr_str, qr_box);
  if (rc == 0) rc = encode_map(&p.tm_kn, ckv, dt, 4, kn_dim, kn_str, kn_box);
  if (rc == 0) rc = encode_map(&p.tm_kr, krope, dt, 3, kr_dim, kr_str, kr_box);
  if (rc != 0) return rc;
  p.block_table = block_table; p.kv_lens = kv_lens; p.out = out;
  p.part_o = static_cast<float*>(workspace);
  p.part_ml = p.part_o + static_cast<int64_t>(d.runs) * 2 * d.chunks * d.n * mlar::kDV;
  p.place = reinterpret_cast<int2*>(p.part_ml + static_cast<int64_t>(d.runs) * 2 * d.chunks * d.n * 2);
  p.B = B; p.q_len = q_len; p.H = H; p.max_pages = max_pages; p.num_pages = num_pages;
  p.rows_per_item = rows_per_item; p.chunks = d.chunks;
  p.causal = causal ? 1 : 0;
  p.scale_log2 = scale * 1.4426950408889634f;
  const uint32_t f = fmt == CATCOC_FMT_BF16 ? 1u : 0u;
  p.idesc_qk = ptx::make_instr_desc(1u, f, f, 0u, 0u, 128u, n);
  p.idesc_pv = ptx::make_instr_desc(1u, f, f, 1u, 0u, 128u, n);
  p.status = status;
  p.timeout_ns = timeout_ns ? timeout_ns : 10000000000ull;
  auto launch = [&](auto main_kernel, auto combine_kernel, int tail, int threads) -> int {
    const int smem = tail + static_cast<int>(sizeof(mlar::Bars)) + 1024;
    CATCOC_CUDA_OK(cudaFuncSetAttribute(main_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    CATCOC_CUDA_OK(launch_overlapped(main_kernel, dim3(static_cast<unsigned>(d.runs), static_cast<unsigned>(d.chunks)), dim3(static_cast<unsigned>(threads)),
                                     smem, stream, p));
    CATCOC_CUDA_OK(launch_overlapped(combine_kernel, dim3(static_cast<unsigned>(rows_per_item), static_cast<unsigned>(B)), dim3(128), 0,
                                     stream, p.part_o, p.part_ml, p.place, out, kv_lens, max_pages, rows_per_item, d.chunks, d.n, d.runs));
    return CATCOC_OK;
  };
  const bool bf = fmt == CATCOC_FMT_BF16;
  if (d.n == 16)
    return bf ? launch(mlar::mla_rows_kernel<16, FMT_BF16>, mlar::mla_rows_combine_kernel<FMT_BF16>, mlar::Geo<16>::kTail, mlar::Geo<16>::kThreads)
              : launch(mlar::mla_rows_kernel<16, FMT_F16>, mlar::mla_rows_combine_kernel<FMT_F16>, mlar::Geo<16>::kTail, mlar::Geo<16>::kThreads);
  if (d.n == 64)
    return bf ? launch(mlar::mla_rows_kernel<64, FMT_BF16>, mlar::mla_rows_combine_kernel<FMT_BF16>, mlar::Geo<64>::kTail, mlar::Geo<64>::kThreads)
              : launch(mlar::mla_rows_kernel<64, FMT_F16>, mlar::mla_rows_combine_kernel<FMT_F16>, mlar::Geo<64>::kTail, mlar::Geo<64>::kThreads);
  return bf ? launch(mlar::mla_rows_kernel<32, FMT_BF16>, mlar::mla_rows_combine_kernel<FMT_BF16>, mlar::Geo<32>::kTail, mlar::Geo<32>::kThreads)
            : launch(mlar::mla_rows_kernel<32, FMT_F16>, mlar::mla_rows_combine_kernel<FMT_F16>, mlar::Geo<32>::kTail, mlar::Geo<32>::kThreads);
}
