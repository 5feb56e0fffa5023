// One query row's share of an online-softmax step, for the attention kernels whose scores and probabilities live in
// TMEM (one row per lane, 128 keys per block).
//
// All 128 scores of the row are read ONCE into registers (four 32-column tcgen05.ld in flight together) and stay
// there for the maximum, the exponentials and the sum; a second read would put the TMEM latency into every block's
// serial chain again. Scale, shift and sum run on register pairs (fma / add .f32x2) and the maximum takes three
// operands per instruction, so that the special-function unit (32 lanes of ex2 take 8 cycles on a scheduler) and not
// instruction issue is the longest of the warp's pipes.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "catcoc/params.h"
#include "catcoc/ptx.cuh"

namespace catcoc {
namespace attn {

constexpr int kRowKeys = 128;            // keys per block
constexpr float kLazyRescale = 8.0f;     // log2 units the running maximum may exceed the reference by

template <int FMT>
CATCOC_DEVICE uint32_t pack16(float lo, float hi) {
  if constexpr (FMT == FMT_BF16) { __nv_bfloat162 hh = __floats2bfloat162_rn(lo, hi); return *reinterpret_cast<uint32_t*>(&hh); }
  else { __half2 hh = __floats2half2_rn(lo, hi); return *reinterpret_cast<uint32_t*>(&hh); }
}

// m: reference maximum (log2 domain), l: running sum
struct RowState {
  float m = -INFINITY, l = 0.0f;
};

// O *= alpha, one row of D fp32 columns in TMEM
template <int D>
CATCOC_DEVICE void rescale_o(uint32_t t_o, float alpha) {
#pragma unroll
  for (int c = 0; c < D / 16; ++c) {
    uint32_t v[16];
    ptx::tmem_ld_32x32b_x16(t_o + c * 16, v);
    ptx::tcgen05_wait_ld();
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
    ptx::tmem_st_32x32b_x16(t_o + c * 16, v);
  }
}

// Reads 128 scores at TMEM address `t_s`, writes the packed probabilities (64 columns) to `t_p`, which may be the same
// place, and updates the state. `loaded()` is called when the scores are in registers, `before(move, alpha)` ahead of the
// first probability: with `move` (the same in all lanes) the reference maximum of some row of the warp moved and O has to
// be multiplied by alpha; `ready()` ahead of the first store of probabilities, `half()` behind
// it (those of the first 64 keys). `vis_left`: keys of this block the row sees (used when `masked`).
//
// Tried and not kept: a quarter of the exponentials as a degree-5 polynomial on the FMA pipe (D = 128, causal 4 % faster, not causal 2
// to 6 % slower, D = 64 slower), the two warps of a scheduler taking their exponentials strictly in turn (4 % slower).
template <int FMT, class Loaded, class Before, class Ready, class Half>
CATCOC_DEVICE void softmax_row_block(uint32_t t_s, uint32_t t_p, bool masked, int vis_left, float sc, RowState& st, Loaded&& loaded,
                                     Before&& before, Ready&& ready, Half&& half) {
  uint32_t v[4][32];
#pragma unroll
  for (int c = 0; c < 4; ++c) ptx::tmem_ld_32x32b_x32(t_s + c * 32, v[c]);
  ptx::tcgen05_wait_ld();
  loaded();
  if (masked) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (c * 32 + i >= vis_left) v[c][i] = 0xff800000u;   // -inf: its probability is exactly zero
  }
  float mx[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    mx[c] = fmaxf(__uint_as_float(v[c][0]), __uint_as_float(v[c][1]));
#pragma unroll
    for (int i = 2; i < 32; i += 2) mx[c] = ptx::max3(mx[c], __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
  }
  const float m_new = fmaxf(st.m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sc);
  const bool move = __any_sync(0xffffffffu, m_new > st.m + kLazyRescale);   // -inf + 8 = -inf: the first block moves
  const float m_use = move ? m_new : st.m;
  const float m_safe = (m_use == -INFINITY) ? 0.0f : m_use;      // a row that sees nothing yet
  const float alpha = !move ? 1.0f : ((st.m == -INFINITY) ? 0.0f : ptx::ex2_approx(st.m - m_safe));
  before(move, alpha);
  const uint64_t sc2 = ptx::pack_f32x2(sc, sc), nm2 = ptx::pack_f32x2(-m_safe, -m_safe);
  uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t w[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int c = 2 * h + (i >> 4), e = (i & 15) * 2;
      float e0, e1;
      ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(__uint_as_float(v[c][e]), __uint_as_float(v[c][e + 1])), sc2, nm2), e0, e1);
      e0 = ptx::ex2_approx(e0);
      e1 = ptx::ex2_approx(e1);
      sum2[i & 1] = ptx::add_f32x2(sum2[i & 1], ptx::pack_f32x2(e0, e1));
      w[i] = pack16<FMT>(e0, e1);
    }
    if (h == 0) ready();
    ptx::tmem_st_32x32b_x32(t_p + h * 32, w);
    if (h == 0) half();
  }
  float s0, s1;
  ptx::unpack_f32x2(ptx::add_f32x2(sum2[0], sum2[1]), s0, s1);
  st.l = st.l * alpha + (s0 + s1);
  st.m = m_use;
}

}  // namespace attn
}  // namespace catcoc
