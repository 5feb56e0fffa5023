// Local products on double tiles: a CTA pair owns TWO accumulators of one 256 x 2 bn output tile at a time, each bn columns.
//
// What bounds the 256 x 256 pair tile of fused_gemm.cuh is shared memory: a K block brings 32 KiB into each CTA per 512 cycles
// of MMAs and the MMAs read 64 bytes per cycle of it, 128 bytes per cycle together, which is all there is. A double tile takes
// in 48 KiB per 1024 cycles, and its products come in pairs that share their A: the second takes it from the tensor core's
// collector buffer. What is read from L2 and HBM falls with the intake, which counts where the power limit sets the clock.
// bf16 8192 x 28672 x 8192: 2076 -> 1848 us at full clock (operands of zeros), 3020 -> 2860 us under the power limit.
//
// All 512 columns of TMEM hold one tile, so that nothing is double-buffered. Instead the halves are kept out of phase: at
// either end of a tile half 0 runs `lead` K blocks ahead of half 1. Its accumulator is finished, drained and free again while
// the tensor core still works on half 1, and the other way round. Each half has four epilogue warps of its own.
//
//   warp 0      TMA producer A          warps 2..5   epilogue of half 0
//   warp 1      MMA issuer (leader)     warps 8..11  epilogue of half 1
//   warp 6      TMA producer B          warp 7       idle
//
// Roles, barriers, bounded waits and the status block are those of fused_gemm.cuh.
#pragma once
#include "catcoc/fused_gemm.cuh"

namespace catcoc {
namespace dtile {

constexpr int kThreads = 384;
constexpr int kRingBytes = 192 * 1024;
constexpr int kLead = 2;
constexpr int kSmemBytes = kRingBytes + 2 * kEpiWarps * kEpiWinBytes + 256 /*barriers*/ + 8 * kMaxTokenGroups + 1024 /*align slack*/;
static_assert(sizeof(SmemTail) <= 256 && kSmemBytes <= 227 * 1024, "shared memory of a CTA");
constexpr uint32_t kMxBN = 192;                  // block-scaled: two accumulators of 192 columns, the scales behind them
constexpr uint32_t kMxSfCol = 2 * kMxBN;         // + slot * 16: SFA (4 columns), SFB of the tile's 384 columns (12)
constexpr int kMxSfBytes = 4 * 512;              // in a stage: one block of SFA, three of SFB

template <int KIND>
CATCOC_DEVICE void umma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
  if (KIND == KIND_F16) ptx::umma_f16_pair(d, a, b, idesc, accum);
  else if (KIND == KIND_I8) ptx::umma_i8_pair(d, a, b, idesc, accum);
  else ptx::umma_f8f6f4_pair(d, a, b, idesc, accum);
}

// The same A for both halves of a tile of two column halves: read from shared memory once
template <int KIND>
CATCOC_DEVICE void umma_pair_both(uint32_t d0, uint32_t d1, uint64_t a, uint64_t b0, uint64_t b1, uint32_t idesc, uint32_t idesc1, uint32_t accum) {
  if (KIND == KIND_F16) { ptx::umma_f16_pair_fill(d0, a, b0, idesc, accum); ptx::umma_f16_pair_use(d1, a, b1, idesc1, accum); }
  else if (KIND == KIND_I8) { ptx::umma_i8_pair_fill(d0, a, b0, idesc, accum); ptx::umma_i8_pair_use(d1, a, b1, idesc1, accum); }
  else { ptx::umma_f8f6f4_pair_fill(d0, a, b0, idesc, accum); ptx::umma_f8f6f4_pair_use(d1, a, b1, idesc1, accum); }
}

// Scales, int32 bias, alpha / beta / C / fp32 bias and activation on 32 columns of one row, in the order of the fused kernel:
// accumulators in, fp32 values out. `grow` is the row in the whole output, `n` the first column, `nv` the group's vectors.
template <int KIND>
CATCOC_DEVICE void finish_columns(const FusedParams& p, uint32_t (&v)[32], float (&f)[32], float row_scale, int grow, bool row_ok, int n, int nv, int st_fmt) {
  const int cvalid = min(32, p.sched.N - n);
  if (KIND == KIND_I8) {
    if (p.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < cvalid) v[j] += static_cast<uint32_t>(p.bias[nv + n + j]);
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = static_cast<float>(static_cast<int32_t>(v[j]));
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
  }
  if (p.scale_n != nullptr) {
    const float* scol = p.scale_n + nv + n;
    if (vec_cols(scol, cvalid == 32)) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float4 s = reinterpret_cast<const float4*>(scol)[u];
        f[u * 4] = f[u * 4] * s.x * row_scale; f[u * 4 + 1] = f[u * 4 + 1] * s.y * row_scale;
        f[u * 4 + 2] = f[u * 4 + 2] * s.z * row_scale; f[u * 4 + 3] = f[u * 4 + 3] * s.w * row_scale;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) f[j] = f[j] * (j < cvalid ? scol[j] : 1.0f) * row_scale;
    }
  } else if (p.scale_m != nullptr) {
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = f[j] * row_scale;
  }
  if (p.affine) {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      float x = p.alpha * f[j];
      if (p.bias_f != nullptr && j < cvalid) x += p.bias_f[nv + n + j];
      f[j] = x;
    }
    if (p.c_src != nullptr && row_ok) {
      const int64_t c0 = static_cast<int64_t>(grow) * p.ldc_src + n;
      if (st_fmt == FMT_F32) {
        const float* c = static_cast<const float*>(p.c_src) + c0;
#pragma unroll
        for (int j = 0; j < 32; ++j) if (j < cvalid) f[j] += p.beta * c[j];
      } else {
        const uint16_t* c = static_cast<const uint16_t*>(p.c_src) + c0;
        if (cvalid == 32 && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint4 w = ptx::ld_global_v4(c + u * 8);
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 c2 = unpack2(ww[e], st_fmt);
              f[u * 8 + e * 2] += p.beta * c2.x;
              f[u * 8 + e * 2 + 1] += p.beta * c2.y;
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) if (j < cvalid) f[j] += p.beta * unpack2(c[j], st_fmt).x;
        }
      }
    }
  }
  if (p.act != ACT_NONE) activate32(f, p.act);
}

// The same for swapped roles: 32 tokens of one feature. `feature` is the lane's own (nv: its place in the per-feature vectors).
template <int KIND>
CATCOC_DEVICE void finish_tokens(const FusedParams& p, uint32_t (&v)[32], float (&f)[32], int token, int tokens, int feature, int nv, bool feature_ok) {
  if (KIND == KIND_I8) {
    const uint32_t b = (p.bias != nullptr && feature_ok) ? static_cast<uint32_t>(p.bias[nv + feature]) : 0u;
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = static_cast<float>(static_cast<int32_t>(v[j] + b));
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
  }
  if (p.scale_n != nullptr || p.scale_m != nullptr) {
    const float sn = (p.scale_n != nullptr && feature_ok) ? p.scale_n[nv + feature] : 1.0f;
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = f[j] * sn * (p.scale_m != nullptr && j < tokens ? p.scale_m[token + j] : 1.0f);
  }
  if (p.affine) {
    const float b = (p.bias_f != nullptr && feature_ok) ? p.bias_f[nv + feature] : 0.0f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const float x = p.alpha * f[j];
      f[j] = p.bias_f != nullptr ? x + b : x;
    }
  }
  if (p.act != ACT_NONE) activate32(f, p.act);
}

// Rows of a staged window (unswizzled, `row_bytes` each: 64 or 128) to global memory: `rows` rows, `n` values of each. A word a
// lane where the output's pitch or the row's end is no multiple of 16 bytes, as in flush_staged.
CATCOC_DEVICE void flush_rows(uint32_t stg, int lane, int row_bytes, uint8_t* base, int64_t pitch, int rows, int n, int elt, bool vec_ok) {
  if (vec_ok && n * elt % 16 == 0) {
    const int units = row_bytes / 16, b0 = (lane % units) * 16;
    for (int r = lane / units; r < rows; r += 32 / units)
      if (b0 < n * elt) ptx::st_global_v4(base + r * pitch + b0, ptx::ld_shared_v4(stg + r * row_bytes + b0));
    return;
  }
  const int width = row_bytes / 4;
  store_rows_by_word(lane, width, base, pitch, rows, n, elt, [&](int r) { return ptx::ld_shared_u32(stg + r * row_bytes + (lane & (width - 1)) * 4); });
}

template <int KIND, bool FULL, bool SWAP, class Params>
__global__ void __launch_bounds__(kThreads, 1) double_tile_kernel(const __grid_constant__ Params p) {
  constexpr bool kGk = std::is_same<Params, FusedParamsGk>::value;   // every group has a K range of its own
  constexpr bool kTok = std::is_same<Params, FusedParamsTok>::value; // ragged groups of tokens along the columns
  constexpr bool kMx = KIND == KIND_MX;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* epi_stage = smem + kRingBytes;
  SmemTail* tail = reinterpret_cast<SmemTail*>(epi_stage + 2 * kEpiWarps * kEpiWinBytes);
  volatile uint32_t* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TileSched& sched = p.sched;
  const DoubleTile& dt = p.dt;
  const int sub = static_cast<int>(ptx::cluster_ctarank());    // this CTA's 128 of every 256 rows
  const bool leader = sub == 0;
  const int worker = static_cast<int>(blockIdx.x >> 1), num_workers = static_cast<int>(gridDim.x >> 1);
  const int num_stages = dt.stages;
  constexpr uint32_t acc_stride = kMx ? kMxBN : static_cast<uint32_t>(kMaxBN);
  const bool grouped = p.num_groups > 0;
  if (grouped) ptx::grid_dependency_wait();   // the group list may be the predecessor's result
  int total_tiles = 0;
  TokenGroup* tok_groups = reinterpret_cast<TokenGroup*>(reinterpret_cast<uint8_t*>(tail) + 256);
  if constexpr (kTok) {
    // the groups by falling width of their tiles: extents as in group_walk_tile (clamped, never decreasing) by a scan of one warp,
    // then every group counts those in front of it
    TokenGroup* found = reinterpret_cast<TokenGroup*>(epi_stage);
    if (warp == 0) {
      int before = 0;
      for (int g0 = 0; g0 < p.num_groups; g0 += 32) {
        const int g = g0 + lane;
        int e = g < p.num_groups ? group_end_row(p.group_ends, p.group_rows, sched.N, g) : 0;
        int most = e;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, most, o);
          if (lane >= o) most = max(most, x);
        }
        const int prev = __shfl_up_sync(0xffffffffu, most, 1);
        const int begin = lane == 0 ? before : max(before, prev);
        if (g < p.num_groups) found[g] = TokenGroup{begin, max(0, e - begin) << 7 | g};
        before = max(before, __shfl_sync(0xffffffffu, most, 31));
      }
    }
    __syncthreads();
    if (threadIdx.x < p.num_groups) {
      const int g = threadIdx.x, mine = token_width(found[g].rows_g >> 7);
      int rank = 0;
      for (int o = 0; o < p.num_groups; ++o) {
        const int w = token_width(found[o].rows_g >> 7);
        rank += w > mine || (w == mine && o < g) ? 1 : 0;
      }
      tok_groups[rank] = found[g];
    }
    __syncthreads();
    for (int g = lane; g < p.num_groups; g += 32) total_tiles += token_tiles(tok_groups[g].rows_g >> 7) * sched.seg_mt;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total_tiles += __shfl_xor_sync(0xffffffffu, total_tiles, o);
  } else if (grouped) {
    total_tiles = grouped_total_tiles(p, lane);
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < num_stages; ++s) {
      ptx::mbar_init(&tail->full[s], 2);      // A producer + B producer
      ptx::mbar_init(&tail->empty[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      ptx::mbar_init(&tail->acc_full[h], 1);
      ptx::mbar_init(&tail->acc_empty[h], 2 * kEpiWarps);   // the half's epilogue warps of both CTAs
    }
    ptx::mbar_init(&tail->drain, 1);
    tail->abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::prefetch_tmap(&p.tm_a);
    ptx::prefetch_tmap(&p.tm_b);
    if (p.out_tma) ptx::prefetch_tmap(&p.tm_out);
  }
  if (warp == 1) {
    ptx::tmem_alloc_pair(&tail->tmem_base, kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();   // the peer's barriers exist before anyone signals them
  ptx::tcgen05_fence_after();
  const uint32_t tmem_base = tail->tmem_base;
  ptx::grid_dependency_wait();   // nothing above touches global memory
  const long long cta_t0 = (p.trace != nullptr) ? ptx::clock_cycles() : 0;

  // The i-th item of this pair: a tile, its number of halves (a single unit takes one accumulator, in turn) and their columns,
  // its K range and, for a slice of a cut unit, its plane (else -1)
  struct Item { TileInfo ti; int bn, bn1, parts, half, k_off, k_len, plane; };
  struct TokenWalk { int g, tile_base; };
  using Walk = typename std::conditional<kTok, TokenWalk, GroupWalk>::type;
  auto event_id = [&](int i) { return static_cast<uint32_t>(worker + i * num_workers); };
  auto walk_begin = [&]() {
    if constexpr (kTok) return TokenWalk{0, 0};
    else return group_walk_begin(p);
  };
  auto get_item = [&](int i, Walk& walk, Item& it) {
    it.bn = it.bn1 = dt.bn; it.parts = 2; it.half = 0; it.k_off = 0; it.k_len = p.K; it.plane = -1;
    if constexpr (kTok) {
      const int t = i * num_workers + ((i & 1) ? num_workers - 1 - worker : worker);
      if (t >= total_tiles) return false;
      int tiles = token_tiles(tok_groups[walk.g].rows_g >> 7) * sched.seg_mt;
      while (t >= walk.tile_base + tiles) {
        walk.tile_base += tiles;
        tiles = token_tiles(tok_groups[++walk.g].rows_g >> 7) * sched.seg_mt;
      }
      const int local = t - walk.tile_base;
      const TokenTile tt = token_tile(tok_groups[walk.g], local / sched.seg_mt);
      it.ti.seg = tt.group;
      it.ti.mi = local % sched.seg_mt;
      it.ti.m0 = it.ti.mi * 2 * kBM;
      it.ti.rows = min(2 * kBM, sched.M - it.ti.m0);
      it.ti.n0 = tt.n0;
      it.ti.cols = tt.valid;
      it.bn = token_half0(tt.width);
      it.bn1 = tt.width - it.bn;
      if (it.bn1 == 0) { it.parts = 1; it.half = i & 1; }
      return true;
    } else if (grouped) {
      const int t = worker + i * num_workers;
      if (t >= total_tiles) return false;
      it.ti = walk_tile(p, t, walk);
      if constexpr (kGk) {
        const int2 r = p.gk_range[it.ti.seg];
        it.k_off = r.x;
        it.k_len = r.y - r.x;
      }
      return true;
    }
    if constexpr (!kGk && !kTok) {
      const DoubleItem d = double_item(dt.plan, worker, i);
      if (d.kind == 0) return false;
      if (d.kind == 1) {
        it.ti = double_tile_extent(sched, d.index);
      } else {
        it.ti = double_unit_extent(sched, dt.plan, dt.bn, d.index);
        it.parts = 1;
        it.half = i & 1;
        if (d.kind == 3) {
          it.k_off = d.slice * dt.plan.slice_k;
          it.k_len = min(dt.plan.slice_k, p.K - it.k_off);
          it.plane = (d.index - dt.plan.singles) * dt.plan.slices + d.slice;
        }
      }
      return true;
    }
    return false;
  };

  if (warp == 0 || warp == 6) {
    // =============================== TMA producers ===============================
    const bool is_a = warp == 0;
    const bool mn = is_a ? p.a_mn_major != 0 : p.b_mn_major != 0;
    const int smem_off = is_a ? 0 : kABytes;
    const int per_box = 128 / p.elt_bytes_a;
    int stage = 0;
    uint32_t phase = 0, issued_mask = 0, issued_parity = 0;
    bool ok = true;
    const bool tr = (p.trace != nullptr) && lane == 0 && is_a;
    unsigned long long c_wait = 0, c_issue = 0;
    Tick tick(tr);
    Walk walk = walk_begin();
    Item it;
    for (int i = 0; ok && get_item(i, walk, it); ++i) {
      if (is_a && lane == 0) emit_event(p, EV_PRODUCER, EV_BEGIN, event_id(i));
      const TileInfo& ti = it.ti;
      const int parts = is_a ? 1 : it.parts;                        // each half has a block of B of its own
      int k_off = it.k_off;
      const int bytes = is_a ? kABytes : kTok ? (it.bn + (parts == 2 ? it.bn1 : 0)) * 64 : parts * dt.b_half;
      int mn0 = is_a ? ti.m0 + sub * kBM : ti.n0;
      if (grouped) {
        // (with swapped roles the operand under A is the groups' weights)
        const bool weights = is_a == SWAP;
        mn0 += weights ? ti.seg * p.g_b_row : -ti.seg * p.g_a_row_back;
        k_off += ti.seg * (weights ? p.g_b_k : p.g_a_k);
      }
      const CUtensorMap* tm = is_a ? &p.tm_a : &p.tm_b;
      bool map_3d = is_a ? p.a_3d != 0 : p.b_3d != 0;
      if (!is_a && p.b_3d == 2 && mn0 + (parts - 1) * it.bn + sub * it.bn / 2 + it.bn / 2 > sched.N / per_box * per_box) { map_3d = false; tm = &p.tm_a_gath[1]; }
      if constexpr (kGk) tm = &p.gk_map[2 * ti.seg + (is_a ? 0 : 1)];
      const int tile_kb = ceil_div(it.k_len, p.bk);
      for (int kb = 0; kb < tile_kb; ++kb) {
        tick.lap(c_issue);
        const bool got = ptx::mbar_wait(&tail->empty[stage], phase ^ 1u, p.timeout_ns, abort_flag);
        tick.lap(c_wait);
        if (!got) {
          if (lane == 0) {
            report_status(p, STATUS_TIMEOUT_PIPELINE, is_a ? 0u : 4u, static_cast<uint32_t>(i), static_cast<uint32_t>(kb), 0u);
            *abort_flag = 1;
          }
          ok = false;
          break;
        }
        if (ptx::elect_one()) {
          // both CTAs' copies are credited to the leader's barrier; only the leader arms it, with the bytes of the pair
          const uint32_t bar = ptx::map_to_cta(ptx::smem_u32(&tail->full[stage]), 0u);
          if (leader) ptx::mbar_expect_tx(&tail->full[stage], 2u * (bytes + (!kMx ? 0 : is_a ? 512 : 1536)));
          uint8_t* base = smem + stage * dt.stage_bytes;
          const int k0 = kb * p.bk + k_off;
          if (kMx) {
            // 512-byte blocks of scales: of this CTA's 128 rows, or of all of the tile's columns (three blocks, wherever it starts)
            ptx::tma_load_3d_pair(base + dt.sf_off + (is_a ? 0 : 512), &p.tm_a_gath[is_a ? 0 : 1], bar, 0, (it.k_off / p.bk + kb) * 4,
                                  is_a ? mn0 / kBM : ti.n0 / 128);
          }
          for (int h = 0; h < parts; ++h) {
            uint8_t* dst = base + smem_off + h * dt.b_half;
            const int bn = h == 0 ? it.bn : it.bn1;
            const int c0 = is_a ? mn0 : mn0 + h * it.bn + sub * (bn / 2);
            if constexpr (kTok) { if (!is_a) tm = &p.tok_map[bn / 32 - 1]; }
            if (!mn) {
              ptx::tma_load_2d_pair(dst, tm, bar, k0, c0);
            } else if (map_3d) {
              ptx::tma_load_3d_pair(dst, tm, bar, 0, k0, c0 / per_box);
            } else {
              for (int b = 0; b * per_box < (is_a ? kBM : bn / 2); ++b) ptx::tma_load_2d_pair(dst + b * (p.bk * 128), tm, bar, c0 + b * per_box, k0);
            }
          }
        }
        __syncwarp();
        issued_mask |= 1u << stage;
        issued_parity = (issued_parity & ~(1u << stage)) | (phase << stage);
        if (++stage == num_stages) { stage = 0; phase ^= 1u; }
      }
    }
    if (tr) { atomicAdd(p.trace + 0, c_wait); atomicAdd(p.trace + 1, c_issue); }
    if (*abort_flag && lane == 0 && leader && is_a) {
      // let every bulk copy that is under way land before the CTA's shared memory goes away
      volatile uint32_t never = 0;
      for (int s = 0; s < num_stages; ++s)
        if (issued_mask & (1u << s)) ptx::mbar_wait(&tail->full[s], (issued_parity >> s) & 1u, 2000000ull, &never);
    }
  } else if (warp == 1) {
    // =============================== MMA issuer ===============================
    if (leader) {
      int stage0 = 0, stage1 = 0;       // next stage of each half
      uint32_t full_phase = 0, acc_phase = 0;   // (acc_phase: bit h for accumulator h)
      bool ok = true, probed = false;
      const uint32_t a_lbo = p.a_mn_major ? static_cast<uint32_t>(p.bk) * 128u : 16u;
      const uint32_t b_lbo = p.b_mn_major ? static_cast<uint32_t>(p.bk) * 128u : 16u;
      const uint32_t a_kinc = (p.a_mn_major ? static_cast<uint32_t>(p.umma_k) * 128u : 32u) >> 4;
      const uint32_t b_kinc = (p.b_mn_major ? static_cast<uint32_t>(p.umma_k) * 128u : 32u) >> 4;
      const uint32_t stage_inc = static_cast<uint32_t>(dt.stage_bytes) >> 4;
      const uint64_t da0 = ptx::make_smem_desc_sw128(ptx::smem_u32(smem), a_lbo, 1024u);
      const uint64_t db0 = ptx::make_smem_desc_sw128(ptx::smem_u32(smem) + kABytes, b_lbo, 1024u);
      // (addresses are in the low words, which no stage carries over into the high ones)
      const uint32_t a_lo = static_cast<uint32_t>(da0), a_hi = static_cast<uint32_t>(da0 >> 32);
      const uint32_t b_lo = static_cast<uint32_t>(db0), b_hi = static_cast<uint32_t>(db0 >> 32);
      const uint32_t b_half = static_cast<uint32_t>(dt.b_half) >> 4;
      uint32_t idesc = p.idesc, idesc1 = p.idesc;
      const bool tr = (p.trace != nullptr) && lane == 0;
      unsigned long long c_full = 0, c_acc = 0, c_issue = 0;
      Tick tick(tr);
      uint32_t slot0 = 0, slot1 = 0;    // K blocks so far: slot of the scales (block-scaled)
      Walk walk = walk_begin();
      Item it;
      for (int i = 0; ok && get_item(i, walk, it); ++i) {
        const int tile_kb = ceil_div(it.k_len, p.bk), k_mmas = ceil_div(it.k_len, p.umma_k);
        if (tile_kb <= 0) continue;
        if constexpr (kTok) {   // the halves' own widths
          idesc = (p.idesc & ~(0x3Fu << 17)) | static_cast<uint32_t>(it.bn >> 3) << 17;
          idesc1 = (p.idesc & ~(0x3Fu << 17)) | static_cast<uint32_t>(it.bn1 >> 3) << 17;
        }
        const uint32_t sfb0 = 4u + (static_cast<uint32_t>(it.ti.n0 & 127) >> 5);   // block-scaled: a tile may start inside a block
        // Waits for the stage under half 0's cursor. `probed` is the answer of a probe made before the previous stage's products
        // were issued: a stage that was ready by then costs nothing here.
        auto wait_full = [&](int kb) {
          tick.lap(c_issue);
          const bool got = probed || ptx::mbar_wait(&tail->full[stage0], full_phase, p.timeout_ns, abort_flag);
          tick.lap(c_full);
          if (!got) {
            if (lane == 0) {
              report_status(p, STATUS_TIMEOUT_PIPELINE, 2u, static_cast<uint32_t>(i), static_cast<uint32_t>(kb), 0u);
              *abort_flag = 1;
            }
            ok = false;
            return;
          }
          ptx::tcgen05_fence_after();
          const bool wrap = stage0 + 1 == num_stages;
          probed = ptx::mbar_test_wait(&tail->full[wrap ? 0 : stage0 + 1], wrap ? full_phase ^ 1u : full_phase);
        };
        // One K block of half 0, half 1, both (product by product in turn) or a single unit (whose B is in half 0's place) into
        // accumulator `acc`; by one lane. A whole block, all but the last one, is four products without a test between them: the
        // issue of narrow ones is what bounds them.
        auto products = [&](auto mode, int kb, int acc) {
          constexpr int m = decltype(mode)::value;
          const int st = m == 1 ? stage1 : stage0;
          const uint32_t off = static_cast<uint32_t>(st) * stage_inc;
          const uint32_t al = a_lo + off, bl = b_lo + off + (m == 1 ? b_half : 0u);
          const uint32_t d = tmem_base + static_cast<uint32_t>(acc) * acc_stride;
          uint32_t sf = 0;
          if constexpr (kMx) {
            // eight slots of scales: a copy never overwrites columns that an earlier, still running MMA may read
            sf = tmem_base + kMxSfCol + ((m == 1 ? slot1 : slot0) & 7u) * 16u;
            if (m != 1) {
              const uint32_t sf_smem = ptx::smem_u32(smem + st * dt.stage_bytes + dt.sf_off);
#pragma unroll
              for (int b = 0; b < 4; ++b)
                ptx::tmem_cp_32x128b_warpx4_pair(sf + 4u * b, ptx::make_smem_desc_noswizzle(sf_smem + 512u * b, 128u, 128u));
            }
          }
          auto step = [&](int k, uint32_t accum) {
            const uint64_t da = ptx::desc_of(al + k * a_kinc, a_hi), db = ptx::desc_of(bl + k * b_kinc, b_hi);
            if constexpr (kMx) {
              const uint32_t sel = static_cast<uint32_t>(k) << 30, id = ptx::with_sf_ids(idesc, k, k);
              const uint32_t sfb = sf + sfb0 + (m == 1 ? kMxBN / 32 : 0u);
              if (m == 2) {
                ptx::umma_mxf8_pair_fill(d, da, db, id, sf | sel, sfb | sel, accum);
                ptx::umma_mxf8_pair_use(d + acc_stride, da, ptx::desc_of(bl + b_half + k * b_kinc, b_hi), id, sf | sel, (sfb + kMxBN / 32) | sel, accum);
              } else {
                ptx::umma_mxf8_pair(d, da, db, id, sf | sel, sfb | sel, accum);
              }
            } else if (m == 2) {
              umma_pair_both<KIND>(d, d + acc_stride, da, db, ptx::desc_of(bl + b_half + k * b_kinc, b_hi), idesc, idesc1, accum);
            } else {
              umma_pair<KIND>(d, da, db, m == 1 ? idesc1 : idesc, accum);
            }
          };
          const int left = k_mmas - kb * 4;
          step(0, kb != 0 ? 1u : 0u);
          if (left >= 4) {
            step(1, 1u); step(2, 1u); step(3, 1u);
          } else {
            if (left > 1) step(1, 1u);
            if (left > 2) step(2, 1u);
          }
          if (m != 0) ptx::tcgen05_commit_pair(&tail->empty[st], 3);     // the stage is not needed any more
          if (kb == tile_kb - 1) {
            ptx::tcgen05_commit_pair(&tail->acc_full[acc], 3);
            if (m == 2) ptx::tcgen05_commit_pair(&tail->acc_full[1], 3);
          }
        };
        auto next0 = [&]() { ++slot0; if (++stage0 == num_stages) { stage0 = 0; full_phase ^= 1u; } };
        auto next1 = [&]() { ++slot1; if (++stage1 == num_stages) stage1 = 0; };
        auto wait_acc = [&](int h) {
          tick.lap(c_issue);
          const bool got = ptx::mbar_wait(&tail->acc_empty[h], ((acc_phase >> h) & 1u) ^ 1u, p.timeout_ns, abort_flag);
          tick.lap(c_acc);
          if (!got) {
            if (lane == 0) {
              report_status(p, STATUS_TIMEOUT_PIPELINE, 1u, static_cast<uint32_t>(i), static_cast<uint32_t>(h), 0u);
              *abort_flag = 1;
            }
            ok = false;
            return;
          }
          acc_phase ^= 1u << h;
          ptx::tcgen05_fence_after();
        };
        if (it.parts == 1) {
          wait_acc(it.half);
          if (ok && lane == 0) emit_event(p, EV_MMA, EV_BEGIN, event_id(i));
          for (int kb = 0; ok && kb < tile_kb; ++kb) {
            wait_full(kb);
            if (!ok) break;
            if (ptx::elect_one()) products(std::integral_constant<int, 3>(), kb, it.half);
            __syncwarp();
            next0(); next1();
          }
          if (ok && lane == 0) emit_event(p, EV_MMA, EV_END, event_id(i));
          continue;
        }
        // half 0 leads at both ends of the tile; in between the halves take turns and a stage is free after one block of each
        const int lead0 = min(dt.lead, (tile_kb + 1) / 2), lead1 = min(dt.lead, tile_kb - lead0);
        for (int kb = 0; ok && kb < tile_kb;) {
          const int count = kb == 0 ? lead0 : (kb + lead1 >= tile_kb ? lead1 : 1);
          if (kb > 0 && count == 1) {
            wait_full(kb);
            if (!ok) break;
            if (ptx::elect_one()) products(std::integral_constant<int, 2>(), kb, 0);
            __syncwarp();
            next0(); next1();
            ++kb;
            continue;
          }
          if (kb == 0) {
            wait_acc(0);
            if (ok && lane == 0) emit_event(p, EV_MMA, EV_BEGIN, event_id(i));
          }
          for (int j = 0; ok && j < count; ++j) {
            wait_full(kb + j);
            if (!ok) break;
            if (ptx::elect_one()) products(std::integral_constant<int, 0>(), kb + j, 0);
            __syncwarp();
            next0();
          }
          if (kb == 0 && ok) wait_acc(1);
          for (int j = 0; ok && j < count; ++j) {
            if (ptx::elect_one()) products(std::integral_constant<int, 1>(), kb + j, 1);
            __syncwarp();
            next1();
          }
          kb += count;
        }
        if (ok && lane == 0) emit_event(p, EV_MMA, EV_END, event_id(i));
      }
      tick.lap(c_issue);
      if (tr) { atomicAdd(p.trace + 2, c_full); atomicAdd(p.trace + 3, c_acc); atomicAdd(p.trace + 4, c_issue); }
      if (*abort_flag && lane == 0) {
        // wait (bounded) for the tensor core to retire what was issued before TMEM is freed: a barrier nobody waits on any more
        volatile uint32_t never = 0;
        ptx::tcgen05_commit_pair(&tail->drain, 1);
        ptx::mbar_wait(&tail->drain, 0u, 2000000ull, &never);
      }
    }
  } else if (warp != 7) {
    // =============================== epilogue ===============================
    // Four warps per half, which never synchronise with each other: warp q owns 32 of the CTA's 128 rows end to end.
    const int h = warp >= 8 ? 1 : 0;
    const int q = warp & 3;                 // TMEM lane quarter this warp may read
    const uint32_t stg = ptx::smem_u32(epi_stage + (h * kEpiWarps + q) * kEpiWinBytes);
    const int row_base = sub * kBM + q * 32;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(h) * acc_stride;
    uint32_t acc_phase = 0;
    bool ok = true, prev_tma = false;       // the last window left by a TMA store, which may still read the buffer
    const bool tr = (p.trace != nullptr) && lane == 0 && q == 0;
    unsigned long long c_full = 0, c_work = 0;
    Tick tick(tr);
    Walk walk = walk_begin();
    Item it;
    for (int i = 0; ok && get_item(i, walk, it); ++i) {
      if (it.k_len <= 0 || (it.parts == 1 && it.half != h)) continue;
      const TileInfo& ti = it.ti;
      const bool raw = it.plane >= 0;         // a slice's accumulator goes to its plane whole, as it is
      const int st_fmt = raw ? (KIND == KIND_I8 ? FMT_S32 : FMT_F32) : p.out_fmt, st_elt = fmt_bytes(st_fmt);
      const int bn = it.parts == 2 && h == 1 ? it.bn1 : it.bn, col_base = it.parts == 2 ? h * it.bn : 0;
      const int rows_valid = raw ? 32 : max(0, min(32, ti.rows - row_base));   // (swapped roles: features, and tokens below)
      const int cols = raw ? bn : max(0, min(bn, ti.cols - col_base));
      const int n0 = ti.n0 + col_base;
      const int grow = ti.m0 + row_base + lane;
      const int nv = grouped ? ti.seg * p.g_nvec : 0;
      float row_scale = 1.0f;
      if (FULL && !SWAP && !raw && p.scale_m != nullptr && lane < rows_valid) row_scale = p.scale_m[grow];
      tick.lap(c_work);
      const bool got = ptx::mbar_wait(&tail->acc_full[h], acc_phase, p.timeout_ns, abort_flag);
      tick.lap(c_full);
      if (!got) {
        if (lane == 0) {
          report_status(p, STATUS_TIMEOUT_PIPELINE, 3u, static_cast<uint32_t>(i), static_cast<uint32_t>(h), 0u);
          *abort_flag = 1;
        }
        break;
      }
      acc_phase ^= 1u;
      ptx::tcgen05_fence_after();
      if (lane == 0 && q == 0) emit_event(p, h == 0 ? EV_EPILOGUE : EV_EPILOGUE_2, EV_BEGIN, event_id(i));
      const int64_t pitch = p.ldc * st_elt;
      if constexpr (SWAP) {
        // The accumulator's lanes are features, its columns tokens. 32-bit values are staged token by token, 32 features of a
        // warp to a row; 16-bit ones after neighbouring lanes have exchanged every other token, two features to a word. A
        // window of 64 (32-bit: 32) tokens leaves by one TMA store, rows of 64 (128) bytes.
        const int f0 = ti.m0 + row_base;
        uint8_t* base = static_cast<uint8_t*>(p.out) + (static_cast<int64_t>(n0) * p.ldc + f0) * st_elt;
        const int per_win = 128 / st_elt, row_bytes = 32 * st_elt;
        const int nwin = rows_valid > 0 ? ceil_div(cols, per_win) : 0;
        bool dst_ok = true;
#if defined(CATCOC_CHECKED)
        if (raw)
          dst_ok = CATCOC_BOUND_ABS(p, SITE_PUSH_SLAB, it.plane * bn + cols, dt.plan.cut * dt.plan.slices * bn);
        else if (rows_valid > 0 && cols > 0)
          dst_ok = CATCOC_BOUND(p, SITE_OUT_STORE, (base - static_cast<uint8_t*>(p.out)) + static_cast<int64_t>(cols - 1) * pitch +
                                                       static_cast<int64_t>(rows_valid) * st_elt, LIM_OUT);
#endif
        for (int win = 0; win < nwin; ++win) {
          const int c0 = win * per_win, tokens = min(per_win, cols - c0);
          const int groups = tokens > 32 ? 2 : 1;
          uint32_t v[2][32];
          if (CATCOC_BOUND_ABS(p, SITE_TMEM, h * acc_stride + c0 + groups * 32, kTmemCols)) {
            ptx::tmem_ld_32x32b_x32(taddr + static_cast<uint32_t>(c0), v[0]);
            if (groups == 2) ptx::tmem_ld_32x32b_x32(taddr + static_cast<uint32_t>(c0 + 32), v[1]);
            ptx::tcgen05_wait_ld();
          }
          if (win == nwin - 1) {
            // every TMEM read of this half is done: hand the accumulator back to the MMA warp
            ptx::tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&tail->acc_empty[h]), 0u));
          }
          if (!dst_ok) continue;
          if (prev_tma) {
            if (lane == 0) ptx::bulk_wait_group_read<0>();   // the window before this one has left the buffer
            __syncwarp();
            prev_tma = false;
          }
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (g >= groups) break;
            float f[32];
            if (FULL && !raw) {
              finish_tokens<KIND>(p, v[g], f, n0 + c0 + g * 32, tokens - g * 32, f0 + lane, nv, lane < rows_valid);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) f[j] = (KIND == KIND_I8 && st_elt == 2) ? static_cast<float>(static_cast<int32_t>(v[g][j])) : __uint_as_float(v[g][j]);
            }
            if (st_elt == 4) {
              if (FULL && !raw && st_fmt == FMT_S32) {
                const uint32_t b = (KIND == KIND_I8 && p.bias != nullptr && lane < rows_valid) ? static_cast<uint32_t>(p.bias[nv + f0 + lane]) : 0u;
#pragma unroll
                for (int j = 0; j < 32; ++j) ptx::st_shared_u32(stg + j * 128 + lane * 4, v[g][j] + b);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) ptx::st_shared_u32(stg + j * 128 + lane * 4, __float_as_uint(f[j]));
              }
            } else {
              const bool odd = (lane & 1) != 0;
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float other = __shfl_xor_sync(0xffffffffu, odd ? f[2 * j] : f[2 * j + 1], 1);
                const float lo = odd ? other : f[2 * j], hi = odd ? f[2 * j + 1] : other;
                ptx::st_shared_u32(stg + (g * 32 + 2 * j + (lane & 1)) * 64 + (lane >> 1) * 4, pack2(lo, hi, st_fmt));
              }
            }
          }
          // whole windows (and half ones, by a map of their own) and what the output's edge clips
          const bool whole = p.out_tma != 0 && (tokens == per_win || (!kTok && n0 + cols == sched.N));
          const bool half_win = p.out_tma != 0 && st_elt == 2 && tokens == 32;
          if (raw || whole || half_win) {
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (raw) ptx::tma_store_2d(&p.tm_part[0], stg, row_base, it.plane * bn + c0);
              else ptx::tma_store_2d(whole ? &p.tm_out : &p.tm_part[1], stg, f0, n0 + c0);
              ptx::bulk_commit_group();
            }
            prev_tma = true;
          } else {
            __syncwarp();
            flush_rows(stg, lane, row_bytes, base + static_cast<int64_t>(c0) * pitch, pitch, tokens, rows_valid, st_elt, p.out_vec_ok != 0);
          }
          __syncwarp();
        }
        if (nwin == 0) {
          ptx::tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&tail->acc_empty[h]), 0u));
        }
        if (lane == 0 && q == 0) emit_event(p, h == 0 ? EV_EPILOGUE : EV_EPILOGUE_2, EV_END, event_id(i));
        continue;
      }
      uint8_t* base = static_cast<uint8_t*>(p.out) + (static_cast<int64_t>(ti.m0 + row_base) * p.ldc + n0) * st_elt;
      const bool vec_ok = p.out_vec_ok != 0 && (n0 * st_elt) % 16 == 0;
      bool dst_ok = true;
#if defined(CATCOC_CHECKED)
      if (raw)
        dst_ok = CATCOC_BOUND_ABS(p, SITE_PUSH_SLAB, it.plane * 2 * kBM + row_base + 32, dt.plan.cut * dt.plan.slices * 2 * kBM);
      else if (rows_valid > 0 && cols > 0)
        dst_ok = CATCOC_BOUND(p, SITE_OUT_STORE, (base - static_cast<uint8_t*>(p.out)) + static_cast<int64_t>(rows_valid - 1) * pitch +
                                                     static_cast<int64_t>(cols) * st_elt, LIM_OUT);
#endif
      // TMA clips at the output's edges only: rows that end inside it (a group's last) and a window that ends inside it (an
      // accumulator of 32 modulo 64 columns) leave by plain stores
      const bool rows_tma = raw || (p.out_tma != 0 && (rows_valid == 32 || !grouped));
      const bool row_direct = !rows_tma && st_elt == 2 && (cols & 31) == 0 &&
                              ((reinterpret_cast<uintptr_t>(base) | static_cast<uintptr_t>(pitch)) & 31) == 0;
      const int per_win = 128 / st_elt, nwin = rows_valid > 0 ? ceil_div(cols, per_win) : 0;
      for (int win = 0; win < nwin; ++win) {
        const int c0 = win * per_win;
        const int groups = min(per_win, cols - c0) > 32 ? 2 : 1;
        uint32_t v[2][32];
        if (CATCOC_BOUND_ABS(p, SITE_TMEM, h * acc_stride + c0 + groups * 32, kMx ? static_cast<int>(kMxSfCol) : kTmemCols)) {
          ptx::tmem_ld_32x32b_x32(taddr + static_cast<uint32_t>(c0), v[0]);
          if (groups == 2) ptx::tmem_ld_32x32b_x32(taddr + static_cast<uint32_t>(c0 + 32), v[1]);
          ptx::tcgen05_wait_ld();
        }
        if (win == nwin - 1) {
          // every TMEM read of this half is done: hand the accumulator back to the MMA warp
          ptx::tcgen05_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&tail->acc_empty[h]), 0u));
        }
        if (!dst_ok) continue;
        const bool win_tma = rows_tma && (c0 + per_win <= cols || n0 + cols >= sched.N);
        if (prev_tma && !row_direct) {
          if (lane == 0) ptx::bulk_wait_group_read<0>();   // the window before this one has left the buffer
          __syncwarp();
          prev_tma = false;
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          if (g >= groups) break;
          if (st_elt == 4) {
            if (FULL && !raw && st_fmt == FMT_F32) {
              float f[32];
              finish_columns<KIND>(p, v[g], f, row_scale, grow, lane < rows_valid, n0 + c0, nv, st_fmt);
#pragma unroll
              for (int j = 0; j < 32; ++j) v[g][j] = __float_as_uint(f[j]);
            } else if (FULL && !raw && KIND == KIND_I8 && p.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) if (n0 + c0 + j < sched.N) v[g][j] += static_cast<uint32_t>(p.bias[nv + n0 + c0 + j]);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) stage_write(stg, lane, u, make_uint4(v[g][u * 4], v[g][u * 4 + 1], v[g][u * 4 + 2], v[g][u * 4 + 3]));
          } else {
            float f[32];
            if (FULL) {
              finish_columns<KIND>(p, v[g], f, row_scale, grow, lane < rows_valid, n0 + c0 + g * 32, nv, st_fmt);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) f[j] = KIND == KIND_I8 ? static_cast<float>(static_cast<int32_t>(v[g][j])) : __uint_as_float(v[g][j]);
            }
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e] = pack2(f[2 * e], f[2 * e + 1], st_fmt);
            if (row_direct) {
              if (lane < rows_valid) {
                uint8_t* o = base + static_cast<int64_t>(lane) * pitch + (c0 + g * 32) * 2;
                const uint32_t lo[8] = {w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7]}, hi[8] = {w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15]};
                ptx::st_global_v8(o, lo);
                ptx::st_global_v8(o + 32, hi);
              }
            } else {
#pragma unroll
              for (int u = 0; u < 4; ++u) stage_write(stg, lane, g * 4 + u, make_uint4(w[u * 4], w[u * 4 + 1], w[u * 4 + 2], w[u * 4 + 3]));
            }
          }
        }
        if (row_direct) continue;
        if (win_tma) {
          ptx::fence_proxy_async_smem();   // the staged bytes become visible to the TMA unit
          __syncwarp();
          if (lane == 0) {
            if (raw) ptx::tma_store_2d(&p.tm_part[0], stg, c0, it.plane * 2 * kBM + row_base);
            else ptx::tma_store_2d(&p.tm_out, stg, n0 + c0, ti.m0 + row_base);
            ptx::bulk_commit_group();
          }
          prev_tma = true;
        } else {
          __syncwarp();
          flush_staged<false>(stg, lane, base + static_cast<int64_t>(win) * 128, pitch, rows_valid, min(per_win, cols - c0), st_elt, vec_ok, nullptr, nullptr, 0, 0, 1);
        }
        __syncwarp();
      }
      if (nwin == 0) {   // nothing of this half lies inside the output: still return the accumulator
        ptx::tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive_cluster(ptx::map_to_cta(ptx::smem_u32(&tail->acc_empty[h]), 0u));
      }
      if (lane == 0 && q == 0) emit_event(p, h == 0 ? EV_EPILOGUE : EV_EPILOGUE_2, EV_END, event_id(i));
    }
    if (lane == 0) ptx::bulk_wait_group_all();   // every TMA store of this warp is performed before the kernel ends
    __syncwarp();
    tick.lap(c_work);
    if (tr) { atomicAdd(p.trace + 5 + 9 * h, c_full); atomicAdd(p.trace + 6 + 9 * h, c_work); }
  }

  // =============================== teardown ===============================
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::cluster_sync_all();   // neither CTA of a pair leaves while the other may touch it
  ptx::tcgen05_fence_after();
  if (warp == 1) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
  if (p.trace != nullptr && threadIdx.x == 0) atomicAdd(p.trace + 8, static_cast<unsigned long long>(ptx::clock_cycles() - cta_t0));
}

}  // namespace dtile
}  // namespace catcoc
