// LDPC normalised min-sum with FP16 messages, packed: two frames per lane, 64 frames
// per warp.
//
// The decoder of ldpc_lanes.cu (BpDecoderImpl, src/detail/BpDecoder/BpDecoderImpl.cpp:37-179,
// min-sum boxplus src/detail/LlrMetrics.h:184-191) in FP16 message passing with FP32
// bit-node sums.  Lane l of group g holds frames 64 g + l (the .x halves) and
// 64 g + 32 + l (the .y halves):
//     chan[g][n][32], app[g][n][32]  float2 (FP32 bit-node values of the two frames)
//     c2v[g][e][32]                  half2  (the two frames' check-to-bit messages)
// so every warp access is 256 (float2) or 128 (half2) contiguous bytes, and one
// packed instruction serves two frames:
//   check  v = app - c2v in FP32 (packed f32x2), rounded to FP16; |v|, the two
//          smallest magnitudes (m2 = min(m2, max(m1, |v|)), m1 = min(m1, |v|)) and
//          the sign parity in half2; edge j gets m2 where |v_j| == m1, else m1, its
//          sign, times the scaling, as one half2 store;
//   bit    app = chan + sum of c2v in edge order, FP32 (packed f32x2 adds).
// Ties are exact: two equal minima give m2 == m1.  The syndrome stop, the retirement
// of frames and the waves are those of ldpc_lanes.cu, with a pair of lane masks per
// group (.x frames, .y frames).
//
// Narrow groups.  The per-pass kernels also take groups of W = 2, 4, 8 or 16 lanes
// (2 W frames):
// chan / app [g][n][W] and c2v [g][e][W], a warp serving 32 / W rows (or bits) of its
// group at once, lane l on row (or bit) l / W and frame pair l % W.  A batch of a few
// frames then runs as many warps per pass as its frames need (one frame of a 64800-bit
// code: 64800 / 16 warps per bit pass with W = 2, against 64800 with W = 32), with the
// same arithmetic per frame, so the results do not depend on W.
//
// Hard-decision decodes keep no a-posteriori values: the bit pass (flow_bit) turns each of
// its messages c in place into v = app - c, rounded as the check pass would, and leaves the
// signs of app as words of frame bits; the check pass (flow_check) then reads a row's messages
// one after the other, without column indices or a gather, writes the new ones over them, and
// takes the row's syndrome as the xor of the sign words of its bits.  The passes are bound by
// L2 traffic and its latency: 16 bytes per edge and lane and 8 per bit, against 20 and 16 with
// the a-posteriori values stored, three dependent loads less per check row, and 46 MB instead of 62
// MB per group of DVB-S2 normal frames, so that a wave holds two.  The values are the same
// bit for bit.  DVB-S2 normal r=3/4 x 512, <= 50 iterations: 5.4 ms against 8.7.  Groups of 2 or 4
// lanes, and some batches in groups of 8 (keeps_app), keep the a-posteriori values.
#include <cuda_fp16.h>
#include <math.h>

#include "common.cuh"
#include "grid_sync.cuh"
#include "kernels.hpp"

namespace fecl {
namespace {

constexpr int kLanes = 32;
constexpr int kWarps = 8;
constexpr uint32_t kSigns = 0x80008000u;

__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 from_bits(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }

// (v.x, v.y) rounded to nearest FP16, overflow saturated to +-65504, as one
// conversion: the same bits as rounding and then clamping to [-65504, 65504] for
// every finite or infinite input.  The PTX operand order puts the first source in
// the upper half.
__device__ __forceinline__ __half2 half2_satfinite(float2 v) {
  uint32_t r;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  return from_bits(r);
}

// active[it & 1][g][2] and fail[it & 1][g][2]: .x and .y frame masks.
__device__ __forceinline__ uint32_t* active_of(const LdpcLanesParams& p, int it) { return p.active + (it & 1) * 2 * p.groups; }
__device__ __forceinline__ uint32_t* fail_of(const LdpcLanesParams& p, int it) { return p.fail + (it & 1) * 2 * p.groups; }

template <int DMAX>
struct Row {
  uint32_t e0;
  int d;
  __half2 v[DMAX];
  unsigned px, py;  // parity of the hard decisions of the previous APP
};

template <int DMAX, int W = kLanes>
__device__ __forceinline__ void load_row(const LdpcLanesParams& p, int g, int r, int sub, Row<DMAX>& w) {
  const __half2* c2v = static_cast<const __half2*>(p.c2v);
  const float2* app = reinterpret_cast<const float2*>(p.app);
  w.e0 = __ldg(p.row_ptr + r);
  w.d = int(__ldg(p.row_ptr + r + 1) - w.e0);
  const __half2* cg = c2v + (int64_t(g) * p.E + w.e0) * W + sub;
  const float2* ag = app + int64_t(g) * p.N * W + sub;
  w.px = w.py = 0;
#pragma unroll
  for (int j = 0; j < DMAX; ++j) {
    if (j < w.d) {
      const uint32_t col = __ldg(p.col_idx + w.e0 + j);
      const float2 a = ag[int64_t(col) * W];
      const float2 c = __half22float2(cg[j * W]);
      w.px ^= unsigned(a.x >= 0.0f);
      w.py ^= unsigned(a.y >= 0.0f);
      // a - c in FP32, rounded to FP16 and kept finite (saturated at +-65504)
      w.v[j] = half2_satfinite(__ffma2_rn(c, make_float2(-1.0f, -1.0f), a));
    }
  }
}

template <int DMAX, int W = kLanes>
__device__ __forceinline__ void store_row(const LdpcLanesParams& p, int g, int sub, const Row<DMAX>& w, __half2 sf2,
                                          bool mine_x, bool mine_y, bool keep_all) {
  __half2* c2v = static_cast<__half2*>(p.c2v);
  const __half2 inf2 = __floats2half2_rn(INFINITY, INFINITY);
  __half2 m1 = inf2, m2 = inf2;
  uint32_t sg = 0;
#pragma unroll
  for (int j = 0; j < DMAX; ++j) {
    if (j < w.d) {
      const __half2 a = __habs2(w.v[j]);
      m2 = __hmin2(m2, __hmax2(m1, a));
      m1 = __hmin2(m1, a);
      sg ^= bits(w.v[j]);
    }
  }
  // d - 1 inputs per output: the sign is (d - 2) xor the parity of the others' signs.
  sg = (sg & kSigns) ^ (((w.d - 2) & 1) ? kSigns : 0u);
  // Lanes whose frames are not decoding keep their messages where the soft outputs,
  // which are sums of these messages, are wanted; a hard-decision decode reads only
  // the a-posteriori values, which the bit pass freezes for retired frames.
  const uint32_t keep = keep_all ? (mine_x ? 0u : 0x0000ffffu) | (mine_y ? 0u : 0xffff0000u) : 0u;
  __half2* cg = c2v + (int64_t(g) * p.E + w.e0) * W + sub;
  // The scaling is applied to the two magnitudes once per row: rounding to nearest is
  // symmetric, so (-m) * s is -(m * s) bit for bit and the edge's sign can be xored
  // into the scaled magnitude.
  if constexpr (DMAX > 16) {
    // Rows of degree > 16 also take the row's sign parity into the two magnitudes,
    // leaving each edge its own sign bit (one operation fewer per edge; measured
    // faster for these rows, slower for the rows of degree <= 16 below).
    const uint32_t b1 = bits(__hmul2(m1, sf2)) ^ sg, b2 = bits(__hmul2(m2, sf2)) ^ sg;
#pragma unroll
    for (int j = 0; j < DMAX; ++j) {
      if (j < w.d) {
        const uint32_t eq = __heq2_mask(__habs2(w.v[j]), m1);
        const __half2 out = from_bits(((b2 & eq) | (b1 & ~eq)) ^ (bits(w.v[j]) & kSigns));
        if (keep == 0u) {
          cg[j * W] = out;
        } else if (keep != 0xffffffffu) {
          const uint32_t old = bits(cg[j * W]);
          cg[j * W] = from_bits((bits(out) & ~keep) | (old & keep));
        }
      }
    }
    return;
  }
  const uint32_t b1 = bits(__hmul2(m1, sf2)), b2 = bits(__hmul2(m2, sf2));
#pragma unroll
  for (int j = 0; j < DMAX; ++j) {
    if (j < w.d) {
      const uint32_t eq = __heq2_mask(__habs2(w.v[j]), m1);
      const uint32_t mag = (b2 & eq) | (b1 & ~eq);
      const uint32_t sign = (sg ^ bits(w.v[j])) & kSigns;
      const __half2 out = from_bits(mag ^ sign);
      if (keep == 0u) {
        cg[j * W] = out;
      } else if (keep != 0xffffffffu) {
        const uint32_t old = bits(cg[j * W]);
        cg[j * W] = from_bits((bits(out) & ~keep) | (old & keep));
      }
    }
  }
}

// The lanes of a W-lane group whose bit is set in a warp ballot (lane l standing for
// frame pair l % W).
template <int W>
__device__ __forceinline__ uint32_t fold_lanes(uint32_t b) {
  if constexpr (W == 32) {
    return b;
  } else {
#pragma unroll
    for (int s = W; s < 32; s *= 2) b |= b >> s;
    return b & ((1u << W) - 1u);
  }
}

// Rows per lane: two for rows of degree <= 8 (more loads in flight per warp), except
// in groups of 2 or 4 lanes, whose batches of a few frames want warps, not loads per
// warp (one DVB-S2 normal r=1/2 frame, 50 iterations: 0.50 ms against 0.57 with two;
// with 8 or 16 lanes two rows measured faster, 1.00 against 1.13 ms for 12 frames).
template <int DMAX, int W>
constexpr int rows_per_lane() { return DMAX <= 8 && W >= 8 ? 2 : 1; }

// Rows r .. r + kRows - 1 of group g at iteration `it` (kRows = rows_per_lane; r is
// this lane's, rows past the last are skipped): the row updates; bx / by collect the
// lanes whose syndrome bit is set.  Every lane of the warp calls it.
template <int DMAX, int W = kLanes>
__device__ __forceinline__ void check_rows(const LdpcLanesParams& p, int it, int g, int r, int sub, bool mx, bool my,
                                           bool keep_all, bool check_syndrome, uint32_t& bx, uint32_t& by) {
  constexpr int kRows = rows_per_lane<DMAX, W>();
  Row<DMAX> w[kRows];
#pragma unroll
  for (int q = 0; q < kRows; ++q) {
    w[q].d = 0;
    if (r + q < p.M) load_row<DMAX, W>(p, g, r + q, sub, w[q]);
  }
#pragma unroll
  for (int q = 0; q < kRows; ++q) {
    if (check_syndrome) {
      bx |= fold_lanes<W>(__ballot_sync(0xffffffffu, w[q].d > 0 && w[q].px != 0));
      by |= fold_lanes<W>(__ballot_sync(0xffffffffu, w[q].d > 0 && w[q].py != 0));
    }
    if (w[q].d > 0) {
      // the scaling of rows of this degree (constant across iterations on this path)
      const float s = p.sf[size_t(it % p.n_sf) * p.sf_stride + (w[q].d >= 2 ? w[q].d - 2 : 0)];
      store_row<DMAX, W>(p, g, sub, w[q], __float2half2_rn(s), mx, my, keep_all);
    }
  }
}

template <int DMAX, int W>
__global__ void __launch_bounds__(kWarps * 32) h2_check(LdpcLanesParams p, int it, int g0) {
  pdl_enter();
  constexpr int kRows = rows_per_lane<DMAX, W>();
  constexpr int kSlots = 32 / W;  // rows (or row pairs) per warp step
  const int lane = threadIdx.x & 31;
  const int sub = lane % W, slot = lane / W;
  const int warps = int(gridDim.x) * kWarps;
  const bool check_syndrome = it > 0 && !p.fixed_iterations;
  const int g = g0 + int(blockIdx.y);
  const uint32_t ax = active_of(p, it)[2 * g], ay = active_of(p, it)[2 * g + 1];
  if ((ax | ay) == 0) return;
  const bool mx = (ax >> sub) & 1, my = (ay >> sub) & 1;
  const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
  uint32_t bx = 0, by = 0;
  const int w0 = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  for (int r = w0 * kSlots * kRows; r < p.M; r += warps * kSlots * kRows)
    check_rows<DMAX, W>(p, it, g, r + slot * kRows, sub, mx, my, keep_all, check_syndrome, bx, by);
  bx &= ax;
  by &= ay;
  if (lane == 0) {
    if (bx) atomicOr(fail_of(p, it) + 2 * g, bx);
    if (by) atomicOr(fail_of(p, it) + 2 * g + 1, by);
  }
}

// Retirement of the .x (h = 0) or .y (h = 1) frames of group g after the check pass of
// iteration `it`, and their masks for iteration it + 1.
template <int W = kLanes>
__device__ __forceinline__ void retire_half(const LdpcLanesParams& p, int it, int g, int h) {
  const uint32_t a = active_of(p, it)[2 * g + h];
  uint32_t done = 0;
  if (it == p.iterations - 1) done = a;
  else if (it > 0 && !p.fixed_iterations) done = a & ~fail_of(p, it)[2 * g + h];
  for (uint32_t m = done; m; m &= m - 1) p.iters_ws[int64_t(g) * 2 * W + h * W + (__ffs(m) - 1)] = it + 1;
  active_of(p, it + 1)[2 * g + h] = a & ~done;
  fail_of(p, it + 1)[2 * g + h] = 0;
}

// app = chan + sum of c2v over bit b's edges (edge order, FP32) for this lane's two
// frames; a retired frame's value stays.  The edges go in runs of 8 (one run for most
// bits): every edge id of a run is loaded, then every message, then they are added in
// order, so a bit costs three dependent loads rather than two per edge.
template <int W = kLanes>
__device__ __forceinline__ void bit_one(const LdpcLanesParams& p, int g, int b, int sub, bool mx, bool my) {
  constexpr uint32_t kRun = 8;
  const __half2* cg = static_cast<const __half2*>(p.c2v) + int64_t(g) * p.E * W + sub;
  const float2* chan = reinterpret_cast<const float2*>(p.chan);
  float2* app = reinterpret_cast<float2*>(p.app);
  const int64_t base = (int64_t(g) * p.N + b) * W + sub;
  const uint32_t k0 = __ldg(p.col_ptr + b), k1 = __ldg(p.col_ptr + b + 1);
  float2 acc = chan[base];
  for (uint32_t k = k0; k < k1; k += kRun) {
    uint32_t e[kRun];
    __half2 x[kRun];
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j) e[j] = k + j < k1 ? __ldg(p.col_edges + k + j) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j) x[j] = k + j < k1 ? cg[int64_t(e[j]) * W] : __half2{};
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j)
      if (k + j < k1) acc = __fadd2_rn(acc, __half22float2(x[j]));
  }
  if (mx && my) {
    app[base] = acc;
  } else {  // one of the lane's frames has retired: its APP stays
    float2 out = app[base];
    if (mx) out.x = acc.x;
    if (my) out.y = acc.y;
    app[base] = out;
  }
}

// Bit pass; with it < 0 the initial APP for every lane.  Block (0, y) retires frames
// and writes the group's masks for iteration it + 1.
template <int W>
__global__ void __launch_bounds__(kWarps * 32) h2_bit(LdpcLanesParams p, int it, int g0) {
  pdl_enter();
  constexpr int kSlots = 32 / W;
  const int lane = threadIdx.x & 31;
  const int sub = lane % W, slot = lane / W;
  const int warps = int(gridDim.x) * kWarps;
  const int g = g0 + int(blockIdx.y);
  const uint32_t ax = it < 0 ? 0xffffffffu : active_of(p, it)[2 * g];
  const uint32_t ay = it < 0 ? 0xffffffffu : active_of(p, it)[2 * g + 1];
  if (it >= 0 && blockIdx.x == 0 && threadIdx.x < 2) retire_half<W>(p, it, g, threadIdx.x);
  const bool mx = (ax >> sub) & 1, my = (ay >> sub) & 1;
  if (!mx && !my) return;
  for (int b = (int(blockIdx.x) * kWarps + (threadIdx.x >> 5)) * kSlots + slot; b < p.N; b += warps * kSlots)
    bit_one<W>(p, g, b, sub, mx, my);
}

// ---- hard decisions: messages in place ---------------------------------------------

// The sign words of bit b of group g: bit l of .x (.y) is set where the a-posteriori value
// of the .x (.y) frame of lane l is >= 0.  They take the place of the a-posteriori values.
__device__ __forceinline__ uint2* signs_of(const LdpcLanesParams& p, int g) {
  return reinterpret_cast<uint2*>(p.app) + int64_t(g) * p.N;
}

// The xor of the sign words of a row's bits, for the W lanes that hold the row (every lane of
// the warp calls it; d = 0: no row).
template <int DMAX, int W>
__device__ __forceinline__ uint2 row_syndrome(const LdpcLanesParams& p, const uint2* signs, uint32_t e0, int d, int sub) {
  uint2 w = make_uint2(0u, 0u);
  if constexpr (W == 32) {
    if (sub < d) w = signs[__ldg(p.col_idx + e0 + sub)];
    w.x = __reduce_xor_sync(0xffffffffu, w.x);
    w.y = __reduce_xor_sync(0xffffffffu, w.y);
  } else {
    constexpr int kPer = (DMAX + W - 1) / W;  // all indices, then all words: two loads deep
    uint32_t col[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) col[q] = sub + q * W < d ? __ldg(p.col_idx + e0 + sub + q * W) : 0u;
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (sub + q * W < d) {
        const uint2 v = signs[col[q]];
        w.x ^= v.x;
        w.y ^= v.y;
      }
#pragma unroll
    for (int o = W / 2; o > 0; o /= 2) {
      w.x ^= __shfl_xor_sync(0xffffffffu, w.x, o);
      w.y ^= __shfl_xor_sync(0xffffffffu, w.y, o);
    }
  }
  return w;
}

template <int DMAX, int W>
__global__ void __launch_bounds__(kWarps * 32) flow_check(LdpcLanesParams p, int it, int g0) {
  pdl_enter();
  constexpr int kRows = rows_per_lane<DMAX, W>();
  constexpr int kSlots = 32 / W;
  const int lane = threadIdx.x & 31;
  const int sub = lane % W, slot = lane / W;
  const int warps = int(gridDim.x) * kWarps;
  const bool check_syndrome = it > 0 && !p.fixed_iterations;
  const int g = g0 + int(blockIdx.y);
  const uint32_t ax = active_of(p, it)[2 * g], ay = active_of(p, it)[2 * g + 1];
  if ((ax | ay) == 0) return;
  const uint2* signs = signs_of(p, g);
  const __half2* cg = static_cast<const __half2*>(p.c2v) + int64_t(g) * p.E * W + sub;
  const float* sf = p.sf + size_t(it % p.n_sf) * p.sf_stride;
  uint32_t bx = 0, by = 0;
  const int w0 = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  for (int r0 = w0 * kSlots * kRows; r0 < p.M; r0 += warps * kSlots * kRows) {
    Row<DMAX> w[kRows];
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      const int r = r0 + slot * kRows + q;
      w[q].e0 = 0;
      w[q].d = 0;
      if (r < p.M) {
        w[q].e0 = __ldg(p.row_ptr + r);
        w[q].d = int(__ldg(p.row_ptr + r + 1) - w[q].e0);
      }
      const __half2* row = cg + int64_t(w[q].e0) * W;
#pragma unroll
      for (int j = 0; j < DMAX; ++j)
        if (j < w[q].d) w[q].v[j] = row[j * W];
    }
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      if (check_syndrome) {
        const uint2 bad = row_syndrome<DMAX, W>(p, signs, w[q].e0, w[q].d, sub);
        bx |= bad.x;
        by |= bad.y;
      }
      if (w[q].d > 0)
        store_row<DMAX, W>(p, g, sub, w[q], __float2half2_rn(sf[w[q].d >= 2 ? w[q].d - 2 : 0]), true, true, false);
    }
  }
  if (!check_syndrome) return;
  if constexpr (W < 32) {  // the rows of the warp's slots
    bx = __reduce_or_sync(0xffffffffu, bx);
    by = __reduce_or_sync(0xffffffffu, by);
  }
  bx &= ax;
  by &= ay;
  if (lane == 0) {
    if (bx) atomicOr(fail_of(p, it) + 2 * g, bx);
    if (by) atomicOr(fail_of(p, it) + 2 * g + 1, by);
  }
}

// v = app - c as the check pass takes it: FP32, rounded to FP16 and kept finite.
__device__ __forceinline__ __half2 to_check(float2 app, __half2 c) {
  return half2_satfinite(__ffma2_rn(__half22float2(c), make_float2(-1.0f, -1.0f), app));
}

// B neighbouring bits of D edges each, the same for every lane of the warp (their edges lie one
// after the other): their a-posteriori values, their messages turned around where `go_on`.
// zero: the first pass, whose messages are all 0.
template <int D, int B>
__device__ __forceinline__ void flow_bits_d(__half2* cg, const uint32_t* edges, float2 (&acc)[B], bool zero, bool go_on) {
  uint32_t e[B * D];
  __half2 x[B * D];
#pragma unroll
  for (int j = 0; j < B * D; ++j) e[j] = __ldg(edges + j);
#pragma unroll
  for (int j = 0; j < B * D; ++j) x[j] = zero ? __half2{} : cg[int64_t(e[j]) * kLanes];
#pragma unroll
  for (int i = 0; i < B; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) acc[i] = __fadd2_rn(acc[i], __half22float2(x[i * D + j]));
  if (go_on) {
#pragma unroll
    for (int j = 0; j < B * D; ++j) cg[int64_t(e[j]) * kLanes] = to_check(acc[j / D], x[j]);
  }
}

// Any degree, which lanes of different slots need not share: runs of 8 edges, as bit_one.
template <int W>
__device__ __forceinline__ float2 flow_bit_any(__half2* cg, const uint32_t* edges, uint32_t deg, float2 ch, bool zero,
                                               bool go_on) {
  constexpr uint32_t kRun = 8;
  uint32_t e[kRun];
  __half2 x[kRun];
  float2 acc = ch;
  auto load = [&](uint32_t k) {
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j) e[j] = k + j < deg ? __ldg(edges + k + j) : 0u;
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j) x[j] = k + j < deg && !zero ? cg[int64_t(e[j]) * W] : __half2{};
  };
  for (uint32_t k = 0; k < deg; k += kRun) {
    load(k);
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j)
      if (k + j < deg) acc = __fadd2_rn(acc, __half22float2(x[j]));
  }
  if (!go_on) return acc;
  for (uint32_t k = 0; k < deg; k += kRun) {
    if (deg > kRun) load(k);
#pragma unroll
    for (uint32_t j = 0; j < kRun; ++j)
      if (k + j < deg) cg[int64_t(e[j]) * W] = to_check(acc, x[j]);
  }
  return acc;
}

constexpr int kFlowBits = 2;

// Bit pass after the check pass of iteration `it`, or with it < 0 the first one.  Block (0, y)
// retires frames, as in h2_bit; a group none of whose frames goes on keeps its messages.
// Four blocks per SM: the compiler alone took 66 registers with whole warps per bit, three
// blocks (64 DVB-S2 normal r=1/2 frames 1318 and 1204 us, 512 of r=3/4 5.73 and 5.34 ms; five
// blocks cost r=9/10 5 %).  Narrower groups need 40.
template <int W>
__global__ void __launch_bounds__(kWarps * 32, W == 32 ? 4 : 0) flow_bit(LdpcLanesParams p, int it, int g0) {
  pdl_enter();
  constexpr int kSlots = 32 / W;
  constexpr uint32_t kAll = W == 32 ? 0xffffffffu : (1u << W) - 1u;
  const int lane = threadIdx.x & 31;
  const int sub = lane % W, slot = lane / W;
  const int warps = int(gridDim.x) * kWarps;
  const int g = g0 + int(blockIdx.y);
  const bool first = it < 0;
  const uint32_t ax = first ? kAll : active_of(p, it)[2 * g], ay = first ? kAll : active_of(p, it)[2 * g + 1];
  bool go_on = true;
  if (!first) {
    const bool test = it > 0 && !p.fixed_iterations;
    const uint32_t on_x = test ? ax & fail_of(p, it)[2 * g] : ax, on_y = test ? ay & fail_of(p, it)[2 * g + 1] : ay;
    go_on = it != p.iterations - 1 && (on_x | on_y) != 0;
    if (blockIdx.x == 0 && threadIdx.x < 2) retire_half<W>(p, it, g, threadIdx.x);
  }
  if ((ax | ay) == 0) return;
  uint2* signs = signs_of(p, g);
  const bool whole = ax == kAll && ay == kAll;  // no retired frame, whose sign stays
  __half2* cg = static_cast<__half2*>(p.c2v) + int64_t(g) * p.E * W + sub;
  const float2* chan = reinterpret_cast<const float2*>(p.chan) + int64_t(g) * p.N * W + sub;
  const int w0 = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if constexpr (W == 32) {
    // kFlowBits neighbouring bits per warp and step, whose loads are in flight together where
    // they have the same degree
    for (int b0 = w0 * kFlowBits; b0 < p.N; b0 += warps * kFlowBits) {
      const int n = min(kFlowBits, p.N - b0);
      uint32_t k[kFlowBits + 1];
      float2 acc[kFlowBits];
      uint2 old[kFlowBits];
#pragma unroll
      for (int i = 0; i <= kFlowBits; ++i) k[i] = __ldg(p.col_ptr + b0 + min(i, n));
#pragma unroll
      for (int i = 0; i < kFlowBits; ++i) {
        acc[i] = i < n ? chan[int64_t(b0 + i) * W] : make_float2(0.0f, 0.0f);
        old[i] = make_uint2(0u, 0u);
        if (!whole && lane == 0 && i < n) old[i] = signs[b0 + i];
      }
      const uint32_t deg = k[1] - k[0];
      bool same = n == kFlowBits;
#pragma unroll
      for (int i = 1; i < kFlowBits; ++i) same = same && k[i + 1] - k[i] == deg;
      const uint32_t* edges = p.col_edges + k[0];
      switch (same ? deg : 0u) {
        case 1: flow_bits_d<1, kFlowBits>(cg, edges, acc, first, go_on); break;
        case 2: flow_bits_d<2, kFlowBits>(cg, edges, acc, first, go_on); break;
        case 3: flow_bits_d<3, kFlowBits>(cg, edges, acc, first, go_on); break;
        case 4: flow_bits_d<4, kFlowBits>(cg, edges, acc, first, go_on); break;
        default:
#pragma unroll
          for (int i = 0; i < kFlowBits; ++i)
            acc[i] = flow_bit_any<W>(cg, p.col_edges + k[i], k[i + 1] - k[i], acc[i], first, go_on);
      }
#pragma unroll
      for (int i = 0; i < kFlowBits; ++i) {
        const uint32_t wx = __ballot_sync(0xffffffffu, acc[i].x >= 0.0f), wy = __ballot_sync(0xffffffffu, acc[i].y >= 0.0f);
        if (i < n && lane == 0)
          signs[b0 + i] = make_uint2((old[i].x & ~ax) | (wx & ax), (old[i].y & ~ay) | (wy & ay));
      }
    }
  } else {
    for (int b0 = w0 * kSlots; b0 < p.N; b0 += warps * kSlots) {
      const int b = b0 + slot;
      float2 acc = make_float2(0.0f, 0.0f);
      uint2 old = make_uint2(0u, 0u);
      if (b < p.N) {
        const uint32_t k0 = __ldg(p.col_ptr + b), deg = __ldg(p.col_ptr + b + 1) - k0;
        if (!whole && sub == 0) old = signs[b];
        acc = flow_bit_any<W>(cg, p.col_edges + k0, deg, chan[int64_t(b) * W], first, go_on);
      }
      const uint32_t wx = __ballot_sync(0xffffffffu, acc.x >= 0.0f) >> (slot * W) & kAll;
      const uint32_t wy = __ballot_sync(0xffffffffu, acc.y >= 0.0f) >> (slot * W) & kAll;
      if (b < p.N && sub == 0) signs[b] = make_uint2((old.x & ~ax) | (wx & ax), (old.y & ~ay) | (wy & ay));
    }
  }
}

// Persistent decoder for a small batch (at most kPersistGroups groups of 64 frames,
// one wave): one launch runs the initial APP and every iteration, the passes of all
// groups spread over the whole grid and separated by grid barriers.  It computes
// exactly the rows, bits and retirements of h2_check / h2_bit.  A barrier that gives
// up marks every frame's iteration count -1 (not decoded).
constexpr int kPersistGroups = 16;

template <int DMAX>
__global__ void __launch_bounds__(kWarps * 32) h2_persist(LdpcLanesParams p) {
  constexpr int kRows = DMAX <= 8 ? 2 : 1;
  __shared__ uint32_t s_bad[2 * kPersistGroups];
  const int lane = threadIdx.x & 31;
  const int warp = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  const int warps = int(gridDim.x) * kWarps;
  const int ng = p.groups;
  const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
  unsigned epoch = 0;
  for (int64_t u = warp; u < int64_t(ng) * p.N; u += warps) bit_one(p, int(u / p.N), int(u % p.N), lane, true, true);
  bool ok = grid_barrier(p.barrier, p.barrier + 1, epoch);
  const int rows = (p.M + kRows - 1) / kRows;
  for (int it = 0; ok && it < p.iterations; ++it) {
    const bool check_syndrome = it > 0 && !p.fixed_iterations;
    if (threadIdx.x < 2 * kPersistGroups) s_bad[threadIdx.x] = 0;
    __syncthreads();
    int g_cur = -1;
    uint32_t bx = 0, by = 0, ax = 0, ay = 0;
    for (int64_t u = warp; u < int64_t(ng) * rows; u += warps) {
      const int g = int(u / rows);
      if (g != g_cur) {
        if (lane == 0 && (bx & ax)) atomicOr(&s_bad[2 * g_cur], bx & ax);
        if (lane == 0 && (by & ay)) atomicOr(&s_bad[2 * g_cur + 1], by & ay);
        g_cur = g;
        bx = by = 0;
        ax = active_of(p, it)[2 * g];
        ay = active_of(p, it)[2 * g + 1];
      }
      if ((ax | ay) == 0) continue;
      check_rows<DMAX>(p, it, g, int(u % rows) * kRows, lane, (ax >> lane) & 1, (ay >> lane) & 1, keep_all,
                       check_syndrome, bx, by);
    }
    if (lane == 0 && g_cur >= 0 && (bx & ax)) atomicOr(&s_bad[2 * g_cur], bx & ax);
    if (lane == 0 && g_cur >= 0 && (by & ay)) atomicOr(&s_bad[2 * g_cur + 1], by & ay);
    __syncthreads();
    if (threadIdx.x < 2 * ng && s_bad[threadIdx.x]) atomicOr(fail_of(p, it) + threadIdx.x, s_bad[threadIdx.x]);
    if (!(ok = grid_barrier(p.barrier, p.barrier + 1, epoch))) break;
    if (blockIdx.x == 0 && threadIdx.x < 2 * ng) retire_half(p, it, threadIdx.x >> 1, threadIdx.x & 1);
    g_cur = -1;
    for (int64_t u = warp; u < int64_t(ng) * p.N; u += warps) {
      const int g = int(u / p.N);
      if (g != g_cur) {
        g_cur = g;
        ax = active_of(p, it)[2 * g];
        ay = active_of(p, it)[2 * g + 1];
      }
      const bool mx = (ax >> lane) & 1, my = (ay >> lane) & 1;
      if (mx || my) bit_one(p, g, int(u % p.N), lane, mx, my);
    }
    if (!(ok = grid_barrier(p.barrier, p.barrier + 1, epoch))) break;
    uint32_t left = 0;
    for (int i = 0; i < 2 * ng; ++i) left |= active_of(p, it + 1)[i];
    if (left == 0) break;
  }
  if (!ok && blockIdx.x == 0)
    for (int i = threadIdx.x; i < ng * 64; i += blockDim.x) p.iters_ws[i] = -1;
}

// h2_persist for one narrow group (at most 16 frames).  Its passes are a few microseconds each
// and a launch per pass is bound by the launches, those after the last frame has
// retired included; here a pass costs a grid barrier and the kernel ends with the last
// frame.  A warp works on the same rows and bits in every pass, so their index lists stay in
// shared memory, a task's lists side by side over its slots, and a pass waits for one
// load from L2 instead of three.  `rows` and `bits`: tasks (32 / W rows or bits) per warp.
// One DVB-S2 short r=2/3 frame in the waterfall: 168 us a call against 232 (persists_alone has more).
constexpr int kNarrowThreads = 512;

__host__ __device__ inline size_t narrow_words_per_warp(int d_max, int c_max, int W, int rows, int bits) {
  return size_t(32 / W) * (size_t(rows) * (2 + d_max) + size_t(bits) * (1 + c_max));
}

template <int DMAX, int W>
__global__ void __launch_bounds__(kNarrowThreads) h2_persist_narrow(LdpcLanesParams p, int rows, int bits) {
  constexpr int kSlots = 32 / W, kRun = 8;
  extern __shared__ uint32_t lists[];
  const int lane = threadIdx.x & 31, sub = lane % W, slot = lane / W;
  const int warp = int(blockIdx.x) * (kNarrowThreads / 32) + (threadIdx.x >> 5);
  const int warps = int(gridDim.x) * (kNarrowThreads / 32);
  const int rstep = (2 + p.d_max) * kSlots, bstep = (1 + p.c_max) * kSlots;
  uint32_t* rl = lists + (threadIdx.x >> 5) * (rows * rstep + bits * bstep) + slot;  // e0, degree, columns
  uint32_t* bl = rl + rows * rstep;                                                  // degree, edges
  for (int k = 0; k < rows; ++k) {
    const int r = (warp + k * warps) * kSlots + slot;
    const uint32_t e0 = r < p.M ? p.row_ptr[r] : 0u, d = r < p.M ? p.row_ptr[r + 1] - e0 : 0u;
    uint32_t* q = rl + k * rstep;
    if (sub == 0) q[0] = e0;
    if (sub == 0) q[kSlots] = d;
    for (uint32_t i = sub; i < d; i += W) q[(2 + i) * kSlots] = p.col_idx[e0 + i];
  }
  for (int k = 0; k < bits; ++k) {
    const int b = (warp + k * warps) * kSlots + slot;
    const uint32_t e0 = b < p.N ? p.col_ptr[b] : 0u, d = b < p.N ? p.col_ptr[b + 1] - e0 : 0u;
    uint32_t* q = bl + k * bstep;
    if (sub == 0) q[0] = d;
    for (uint32_t i = sub; i < d; i += W) q[(1 + i) * kSlots] = p.col_edges[e0 + i];
  }
  __syncwarp();

  __half2* cg = static_cast<__half2*>(p.c2v) + sub;
  float2* app = reinterpret_cast<float2*>(p.app) + sub;
  const float2* chan = reinterpret_cast<const float2*>(p.chan) + sub;
  const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
  // bit_one over this warp's bits
  auto bit_pass = [&](bool mx, bool my) {
    for (int k = 0; k < bits; ++k) {
      const int64_t at = int64_t((warp + k * warps) * kSlots + slot) * W;
      if ((warp + k * warps) * kSlots + slot >= p.N) continue;
      const uint32_t* q = bl + k * bstep;
      const int deg = int(q[0]);
      float2 acc = chan[at];
      for (int i0 = 0; i0 < deg; i0 += kRun) {
        __half2 x[kRun];
#pragma unroll
        for (int i = 0; i < kRun; ++i) x[i] = i0 + i < deg ? cg[int64_t(q[(1 + i0 + i) * kSlots]) * W] : __half2{};
#pragma unroll
        for (int i = 0; i < kRun; ++i)
          if (i0 + i < deg) acc = __fadd2_rn(acc, __half22float2(x[i]));
      }
      if (mx && my) {
        app[at] = acc;
      } else {
        float2 out = app[at];
        if (mx) out.x = acc.x;
        if (my) out.y = acc.y;
        app[at] = out;
      }
    }
  };
  unsigned epoch = 0;
  const unsigned long long limit = p.barrier_us ? 1000ull * p.barrier_us : kBarrierNs;
  auto together = [&] { return grid_barrier(p.barrier, p.barrier + 1, epoch, limit, p.barrier_missing); };
  bit_pass(true, true);
  // every thread follows the masks: those of the next iteration come from these and the failures
  uint32_t ax = active_of(p, 0)[0], ay = active_of(p, 0)[1];
  bool ok = together();
  for (int it = 0; ok && it < p.iterations; ++it) {
    const bool check_syndrome = it > 0 && !p.fixed_iterations;
    const bool mx = (ax >> sub) & 1, my = (ay >> sub) & 1;
    const float* sf = p.sf + size_t(it % p.n_sf) * p.sf_stride;
    uint32_t bx = 0, by = 0;
    // check_rows over this warp's rows
    for (int k = 0; k < rows; ++k) {
      const uint32_t* q = rl + k * rstep;
      Row<DMAX> w;
      w.e0 = q[0];
      w.d = int(q[kSlots]);
      w.px = w.py = 0;
      const float s = sf[w.d >= 2 ? w.d - 2 : 0];
      const __half2* row = cg + int64_t(w.e0) * W;
      float2 a[DMAX];
#pragma unroll
      for (int i = 0; i < DMAX; ++i)
        if (i < w.d) {
          a[i] = app[int64_t(q[(2 + i) * kSlots]) * W];
          w.v[i] = row[i * W];
        }
#pragma unroll
      for (int i = 0; i < DMAX; ++i) {
        if (i < w.d) {
          w.px ^= unsigned(a[i].x >= 0.0f);
          w.py ^= unsigned(a[i].y >= 0.0f);
          w.v[i] = half2_satfinite(__ffma2_rn(__half22float2(w.v[i]), make_float2(-1.0f, -1.0f), a[i]));
        }
      }
      if (check_syndrome) {
        bx |= fold_lanes<W>(__ballot_sync(0xffffffffu, w.d > 0 && w.px != 0));
        by |= fold_lanes<W>(__ballot_sync(0xffffffffu, w.d > 0 && w.py != 0));
      }
      if (w.d > 0) store_row<DMAX, W>(p, 0, sub, w, __float2half2_rn(s), mx, my, keep_all);
    }
    if (lane == 0 && (bx & ax)) atomicOr(fail_of(p, it), bx & ax);
    if (lane == 0 && (by & ay)) atomicOr(fail_of(p, it) + 1, by & ay);
    if (!(ok = together())) break;
    uint32_t on_x = ax, on_y = ay;
    if (it == p.iterations - 1) on_x = on_y = 0;
    else if (check_syndrome) {
      on_x &= fail_of(p, it)[0];
      on_y &= fail_of(p, it)[1];
    }
    if (blockIdx.x == 0 && threadIdx.x < 2) retire_half<W>(p, it, 0, threadIdx.x);
    if (mx || my) bit_pass(mx, my);
    ax = on_x;
    ay = on_y;
    if ((ax | ay) == 0) break;
    if (!(ok = together())) break;
  }
}  // a barrier that gave up leaves p.barrier[1] set: h2_finish_narrow decodes

// ---- several codes in one launch ------------------------------------------------

// The groups of every job of a mixed batch (each job one code, its own scratch) whose
// check degrees are at most DMAX (8, 16 or 32) in one persistent launch: waves of
// groups, from any codes, whose working sets fit in L2 together; per wave the initial
// APP and every iteration, each pass spreading every group's rows (or bits) over the
// whole grid, passes separated by grid barriers.  A group runs exactly the rows, bits
// and retirements of h2_check / h2_bit with its own code's tables, scaling and
// iteration limit, so every frame's result is that of its job decoded alone.  A
// barrier that gives up marks the iteration counts of every frame -1 (not decoded).
__device__ __forceinline__ bool wave_left(const LdpcMultiParams& m, const LdpcLanesParams* codes, int q0, int q1,
                                          int it) {
  uint32_t left = 0;
  for (int q = q0; q < q1; ++q) {
    const LdpcMultiGroup gr = m.groups[q];
    const LdpcLanesParams& p = codes[gr.code];
    left |= active_of(p, it)[2 * gr.group] | active_of(p, it)[2 * gr.group + 1];
  }
  return left != 0;
}

template <int DMAX>
__global__ void __launch_bounds__(kWarps * 32, DMAX <= 16 ? 3 : 2) h2_multi(LdpcMultiParams m) {
  constexpr int kRows = DMAX <= 8 ? 2 : 1;
  __shared__ LdpcLanesParams s_codes[kMultiMaxCodes];
  __shared__ uint32_t s_bad[2 * kMultiMaxWaveGroups];
  {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(m.codes);
    uint32_t* dst = reinterpret_cast<uint32_t*>(s_codes);
    const int words = int(m.ncodes * sizeof(LdpcLanesParams) / 4);
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  const int warps = int(gridDim.x) * kWarps;
  unsigned epoch = 0;
  bool ok = true;
  for (int w = 0; ok && w < m.nwaves; ++w) {
    const int q0 = m.wave_ptr[w], q1 = m.wave_ptr[w + 1];
    int max_it = 0;
    for (int q = q0; q < q1; ++q) max_it = max(max_it, s_codes[m.groups[q].code].iterations);
    for (int q = q0; q < q1; ++q) {
      const LdpcMultiGroup gr = m.groups[q];
      const LdpcLanesParams& p = s_codes[gr.code];
      for (int b = warp; b < p.N; b += warps) bit_one(p, gr.group, b, lane, true, true);
    }
    ok = grid_barrier(m.barrier, m.barrier + 1, epoch);
    for (int it = 0; ok && it < max_it; ++it) {
      if (threadIdx.x < 2 * kMultiMaxWaveGroups) s_bad[threadIdx.x] = 0;
      __syncthreads();
      for (int q = q0; q < q1; ++q) {
        const LdpcMultiGroup gr = m.groups[q];
        const LdpcLanesParams& p = s_codes[gr.code];
        const uint32_t ax = active_of(p, it)[2 * gr.group], ay = active_of(p, it)[2 * gr.group + 1];
        if ((ax | ay) == 0) continue;
        const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
        const bool check_syndrome = it > 0 && !p.fixed_iterations;
        uint32_t bx = 0, by = 0;
        for (int r = warp * kRows; r < p.M; r += warps * kRows)
          check_rows<DMAX>(p, it, gr.group, r, lane, (ax >> lane) & 1, (ay >> lane) & 1, keep_all, check_syndrome, bx,
                           by);
        if (lane == 0 && (bx & ax)) atomicOr(&s_bad[2 * (q - q0)], bx & ax);
        if (lane == 0 && (by & ay)) atomicOr(&s_bad[2 * (q - q0) + 1], by & ay);
      }
      __syncthreads();
      if (threadIdx.x < 2 * (q1 - q0) && s_bad[threadIdx.x]) {
        const LdpcMultiGroup gr = m.groups[q0 + (threadIdx.x >> 1)];
        atomicOr(fail_of(s_codes[gr.code], it) + 2 * gr.group + (threadIdx.x & 1), s_bad[threadIdx.x]);
      }
      if (!(ok = grid_barrier(m.barrier, m.barrier + 1, epoch))) break;
      if (blockIdx.x == 0 && threadIdx.x < 2 * (q1 - q0)) {
        const LdpcMultiGroup gr = m.groups[q0 + (threadIdx.x >> 1)];
        retire_half(s_codes[gr.code], it, gr.group, threadIdx.x & 1);
      }
      for (int q = q0; q < q1; ++q) {
        const LdpcMultiGroup gr = m.groups[q];
        const LdpcLanesParams& p = s_codes[gr.code];
        const uint32_t ax = active_of(p, it)[2 * gr.group], ay = active_of(p, it)[2 * gr.group + 1];
        const bool mx = (ax >> lane) & 1, my = (ay >> lane) & 1;
        if (!mx && !my) continue;
        for (int b = warp; b < p.N; b += warps) bit_one(p, gr.group, b, lane, mx, my);
      }
      if (!(ok = grid_barrier(m.barrier, m.barrier + 1, epoch))) break;
      if (!wave_left(m, s_codes, q0, q1, it + 1)) break;
    }
  }
  if (!ok && blockIdx.x == 0)
    for (int c = 0; c < m.ncodes; ++c)
      for (int i = threadIdx.x; i < s_codes[c].groups * 64; i += blockDim.x) s_codes[c].iters_ws[i] = -1;
}

// Frame f of a W-lane group g sits in lane f % W, half (f / W) % 2.
template <int W>
__device__ __forceinline__ int64_t frame_of(int g, int sub, int h) { return int64_t(g) * 2 * W + h * W + sub; }

template <int W>
__global__ void h2_stage(LdpcLanesParams p) {
  float2* chan = reinterpret_cast<float2*>(p.chan);
  __half2* c2v = static_cast<__half2*>(p.c2v);
  const int g = int(blockIdx.y);
  const int stride = int(gridDim.x) * blockDim.x;
  const int t0 = int(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int i = t0; i < p.N * W; i += stride) {
    const int sub = i % W, b = i / W;
    float v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t f = frame_of<W>(g, sub, h);
      v[h] = 0.0f;
      if (f < p.nframes) {
        v[h] = load_llr(p.llr, p.llr_dtype, f * p.N + b);
        if (p.syst_in && b < p.msg) v[h] += load_llr(p.syst_in, p.llr_dtype, f * p.msg + b);
      }
    }
    chan[int64_t(g) * p.N * W + i] = make_float2(v[0], v[1]);
  }
  for (int64_t i = t0; i < p.E * W; i += stride) c2v[int64_t(g) * p.E * W + i] = __floats2half2_rn(0.0f, 0.0f);
  if (t0 == 0) {
    constexpr uint32_t kAll = W == 32 ? 0xffffffffu : (1u << W) - 1u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t left = p.nframes - int64_t(g) * 2 * W - h * W;
      p.active[2 * g + h] = left >= W ? kAll : (left > 0 ? ((1u << left) - 1u) : 0u);
      p.active[2 * p.groups + 2 * g + h] = 0;
      p.fail[2 * g + h] = 0;
      p.fail[2 * p.groups + 2 * g + h] = 0;
    }
  }
}

// Staging for the hard-decision passes: a tile of bits of a group's 2 W frames goes through
// shared memory, so that both the frame-major reads and the lane-minor writes are
// contiguous.  Block (0, y) writes the group's masks.
constexpr int kTile = 2048;  // elements of a tile: kTile / 2 W bits
template <int W>
__global__ void __launch_bounds__(256) flow_stage(LdpcLanesParams p) {
  constexpr int kBits = kTile / (2 * W);
  __shared__ float tile[2 * W][kBits + 1];
  const int g = int(blockIdx.y), b0 = int(blockIdx.x) * kBits;
#pragma unroll
  for (int q = 0; q < kTile / 256; ++q) {
    const int i = q * 256 + threadIdx.x, frame = i / kBits, bit = i % kBits;
    const int64_t f = int64_t(g) * 2 * W + frame;
    tile[frame][bit] = f < p.nframes && b0 + bit < p.N ? load_llr(p.llr, p.llr_dtype, f * p.N + b0 + bit) : 0.0f;
  }
  __syncthreads();
  float2* chan = reinterpret_cast<float2*>(p.chan) + (int64_t(g) * p.N + b0) * W;
#pragma unroll
  for (int q = 0; q < kTile / 512; ++q) {
    const int i = q * 256 + threadIdx.x, sub = i % W, bit = i / W;
    if (b0 + bit < p.N) chan[i] = make_float2(tile[sub][bit], tile[W + sub][bit]);
  }
  if (blockIdx.x == 0 && threadIdx.x < 2) {
    constexpr uint32_t kAll = W == 32 ? 0xffffffffu : (1u << W) - 1u;
    const int h = threadIdx.x;
    const int64_t left = p.nframes - int64_t(g) * 2 * W - h * W;
    p.active[2 * g + h] = left >= W ? kAll : (left > 0 ? ((1u << left) - 1u) : 0u);
    p.active[2 * p.groups + 2 * g + h] = 0;
    p.fail[2 * g + h] = 0;
    p.fail[2 * p.groups + 2 * g + h] = 0;
  }
}

// The decisions of group blockIdx.y from the sign words: V consecutive bits per thread, the
// group's frames one after the other (blockIdx.z takes every gridDim.z-th), so that a
// warp's stores are contiguous.
template <int W, int V>
__global__ void __launch_bounds__(256) flow_finish(LdpcLanesParams p) {
  const int g = int(blockIdx.y);
  const uint2* signs = signs_of(p, g);
  for (int b = (int(blockIdx.x) * 256 + threadIdx.x) * V; b < p.msg; b += int(gridDim.x) * 256 * V) {
    uint2 w[V];
#pragma unroll
    for (int i = 0; i < V; ++i) w[i] = signs[b + i];
    for (int frame = blockIdx.z; frame < 2 * W; frame += gridDim.z) {
      const int64_t f = int64_t(g) * 2 * W + frame;
      if (f >= p.nframes) break;
      uint32_t v = 0;
#pragma unroll
      for (int i = 0; i < V; ++i) v |= ((frame < W ? w[i].x >> frame : w[i].y >> (frame - W)) & 1u) << (8 * i);
      if constexpr (V == 4) *reinterpret_cast<uint32_t*>(p.hard + f * p.msg + b) = v;
      else p.hard[f * p.msg + b] = uint8_t(v);
    }
  }
  if (p.iters && blockIdx.x == 0 && blockIdx.z == 0 && threadIdx.x < 2 * W) {
    const int64_t f = int64_t(g) * 2 * W + threadIdx.x;
    if (f < p.nframes) p.iters[f] = p.iters_ws[f];
  }
}

// The outputs of group g, by block `block` of `blocks`.
template <int W>
__device__ __forceinline__ void finish_group(const LdpcLanesParams& p, int g, int block, int blocks) {
  const float2* chan = reinterpret_cast<const float2*>(p.chan);
  const float2* app = reinterpret_cast<const float2*>(p.app);
  const __half2* c2v = static_cast<const __half2*>(p.c2v);
  const int stride = blocks * int(blockDim.x);
  const int t0 = block * int(blockDim.x) + int(threadIdx.x);
  const bool soft = p.msg_out || p.syst_out || p.parity_out;
  const __half2* cg = c2v + int64_t(g) * p.E * W;
  for (int i = t0; i < p.N * W; i += stride) {
    const int sub = i % W, b = i / W;
    const int64_t at = int64_t(g) * p.N * W + i;
    const float2 a = app[at];
    float2 ext = make_float2(0.0f, 0.0f);
    if (soft)
      for (uint32_t k = __ldg(p.col_ptr + b); k < __ldg(p.col_ptr + b + 1); ++k)
        ext = __fadd2_rn(ext, __half22float2(cg[int64_t(__ldg(p.col_edges + k)) * W + sub]));
    const float2 ch = chan[at];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t f = frame_of<W>(g, sub, h);
      if (f >= p.nframes) continue;
      const float av = h ? a.y : a.x, ev = h ? ext.y : ext.x, cv = h ? ch.y : ch.x;
      if (p.hard && b < p.msg) p.hard[f * p.msg + b] = uint8_t(av >= 0.0f);
      if (soft) {
        if (p.parity_out) store_llr(p.parity_out, p.out_dtype, f * p.N + b, ev);
        if (b < p.msg) {
          if (p.syst_out) store_llr(p.syst_out, p.out_dtype, f * p.msg + b, ev);
          if (p.msg_out) store_llr(p.msg_out, p.out_dtype, f * p.msg + b, cv + ev);
        }
      }
    }
  }
  if (p.state_out) {
    for (int64_t i = t0; i < p.E * W; i += stride) {
      const int sub = int(i % W);
      const int64_t e = i / W;
      const float2 c = __half22float2(cg[i]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t f = frame_of<W>(g, sub, h);
        if (f < p.nframes) store_llr(p.state_out, p.out_dtype, f * p.E + e, h ? c.y : c.x);
      }
    }
  }
  if (p.iters && t0 < 2 * W) {
    const int64_t f = int64_t(g) * 2 * W + t0;
    if (f < p.nframes) p.iters[f] = p.iters_ws[f];
  }
}

template <int W>
__global__ void h2_finish(LdpcLanesParams p) {
  finish_group<W>(p, int(blockIdx.y), int(blockIdx.x), int(gridDim.x));
}

// The decode of h2_persist_narrow by one block, from the staged L-values: for a launch whose
// grid barrier gave up.  Slow (one SM), and as good as never needed.
template <int DMAX, int W>
__device__ __noinline__ void decode_by_block(const LdpcLanesParams& p) {
  constexpr int kSlots = 32 / W, kRows = rows_per_lane<DMAX, W>();
  const int lane = threadIdx.x & 31, sub = lane % W, slot = lane / W;
  const int warp = threadIdx.x >> 5, warps = int(blockDim.x) >> 5;
  const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
  __half2* c2v = static_cast<__half2*>(p.c2v);
  for (int64_t i = threadIdx.x; i < p.E * W; i += blockDim.x) c2v[i] = __floats2half2_rn(0.0f, 0.0f);
  if (threadIdx.x < 2) {
    const int64_t left = p.nframes - int64_t(threadIdx.x) * W;
    p.active[threadIdx.x] = left >= W ? (1u << W) - 1u : (left > 0 ? (1u << left) - 1u : 0u);
    p.fail[threadIdx.x] = 0;
    p.fail[2 + threadIdx.x] = 0;
  }
  auto bits = [&](bool mx, bool my) {
    for (int b = warp * kSlots + slot; b < p.N; b += warps * kSlots) bit_one<W>(p, 0, b, sub, mx, my);
  };
  __syncthreads();
  bits(true, true);
  __syncthreads();
  for (int it = 0; it < p.iterations; ++it) {
    const uint32_t ax = active_of(p, it)[0], ay = active_of(p, it)[1];
    if ((ax | ay) == 0) break;
    const bool check_syndrome = it > 0 && !p.fixed_iterations, mx = (ax >> sub) & 1, my = (ay >> sub) & 1;
    uint32_t bx = 0, by = 0;
    for (int r0 = warp * kSlots * kRows; r0 < p.M; r0 += warps * kSlots * kRows)
      check_rows<DMAX, W>(p, it, 0, r0 + slot * kRows, sub, mx, my, keep_all, check_syndrome, bx, by);
    if (lane == 0 && (bx & ax)) atomicOr(fail_of(p, it), bx & ax);
    if (lane == 0 && (by & ay)) atomicOr(fail_of(p, it) + 1, by & ay);
    __syncthreads();
    if (threadIdx.x < 2) retire_half<W>(p, it, 0, threadIdx.x);
    bits(mx, my);
    __syncthreads();
  }
}

// h2_finish after h2_persist_narrow.
template <int DMAX, int W>
__global__ void __launch_bounds__(256) h2_finish_narrow(LdpcLanesParams p) {
  if (p.barrier[1] == 0u) {
    finish_group<W>(p, 0, int(blockIdx.x), int(gridDim.x));
  } else if (blockIdx.x == 0) {
    decode_by_block<DMAX, W>(p);
    finish_group<W>(p, 0, 0, 1);
  }
}

dim3 grid_for(int64_t per_group, int groups) {
  const int64_t need = (per_group + kWarps - 1) / kWarps;
  const int64_t share = (148 * 16 + groups - 1) / groups;
  const int64_t x = need < share ? need : share;
  return dim3(unsigned(x > 0 ? x : 1), unsigned(groups));
}

// Waves as in ldpc_lanes.cu: the most groups whose working set fits in kWaveCap (one
// packed group of DVB-S2 normal frames is 62 MB: one group per wave ran 15 % faster
// than two).
constexpr int64_t kWaveCap = 96ll << 20;

// ---- several codes, one launch per pass ---------------------------------------

// The passes of h2_check / h2_bit over the groups [q0, q0 + gridDim.y) of a group
// table spanning several codes (each group's code parameters copied to shared memory
// by its blocks), so that one check launch per check-degree class and one bit launch
// serve every code of a batch in an iteration.  A block's rows (or bits) are those of
// h2_check / h2_bit for its group, so every frame gets exactly its own code's passes;
// blocks past their group's rows return at once.
__device__ __forceinline__ void load_group_params(const LdpcMultiParams& m, int q, LdpcLanesParams& sp, int& g) {
  const LdpcMultiGroup gr = m.groups[q];
  const uint32_t* src = reinterpret_cast<const uint32_t*>(m.codes + gr.code);
  uint32_t* dst = reinterpret_cast<uint32_t*>(&sp);
  for (int i = threadIdx.x; i < int(sizeof(LdpcLanesParams) / 4); i += blockDim.x) dst[i] = src[i];
  g = gr.group;
  __syncthreads();
}

// The rows of group g spread over the x blocks of its grid row (a warp per row or row
// pair), the lanes whose syndrome failed accumulated in bx / by.
template <int DMAX>
__device__ __forceinline__ void check_group(const LdpcLanesParams& p, int it, int g, int lane, bool mx, bool my,
                                            bool keep_all, bool check_syndrome, uint32_t& bx, uint32_t& by) {
  constexpr int kRows = DMAX <= 8 ? 2 : 1;
  const int warps = int(gridDim.x) * kWarps;
  const int w0 = int(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  for (int r = w0 * kRows; r < p.M; r += warps * kRows)
    check_rows<DMAX>(p, it, g, r, lane, mx, my, keep_all, check_syndrome, bx, by);
}

// DMAX = 0: groups of every check-degree class in one launch, each block taking its
// group's class (blocks of a grid row share a group, so the choice is uniform).
template <int DMAX>
__global__ void __launch_bounds__(kWarps * 32) h2_check_many(LdpcMultiParams m, int it, int q0) {
  pdl_enter();
  __shared__ LdpcLanesParams sp;
  int g;
  load_group_params(m, q0 + int(blockIdx.y), sp, g);
  const LdpcLanesParams& p = sp;
  if (it >= p.iterations) return;
  const int lane = threadIdx.x & 31;
  const bool check_syndrome = it > 0 && !p.fixed_iterations;
  const uint32_t ax = active_of(p, it)[2 * g], ay = active_of(p, it)[2 * g + 1];
  if ((ax | ay) == 0) return;
  const bool mx = (ax >> lane) & 1, my = (ay >> lane) & 1;
  const bool keep_all = p.msg_out || p.syst_out || p.parity_out || p.state_out;
  uint32_t bx = 0, by = 0;
  const int cls = DMAX ? DMAX : (p.d_max <= 8 ? 8 : (p.d_max <= 16 ? 16 : 32));
  if (cls == 8) check_group<8>(p, it, g, lane, mx, my, keep_all, check_syndrome, bx, by);
  else if (cls == 16) check_group<16>(p, it, g, lane, mx, my, keep_all, check_syndrome, bx, by);
  else check_group<32>(p, it, g, lane, mx, my, keep_all, check_syndrome, bx, by);
  bx &= ax;
  by &= ay;
  if (lane == 0) {
    if (bx) atomicOr(fail_of(p, it) + 2 * g, bx);
    if (by) atomicOr(fail_of(p, it) + 2 * g + 1, by);
  }
}

__global__ void __launch_bounds__(kWarps * 32) h2_bit_many(LdpcMultiParams m, int it, int q0) {
  pdl_enter();
  __shared__ LdpcLanesParams sp;
  int g;
  load_group_params(m, q0 + int(blockIdx.y), sp, g);
  const LdpcLanesParams& p = sp;
  if (it >= p.iterations) return;
  const int lane = threadIdx.x & 31;
  const int warps = int(gridDim.x) * kWarps;
  const uint32_t ax = it < 0 ? 0xffffffffu : active_of(p, it)[2 * g];
  const uint32_t ay = it < 0 ? 0xffffffffu : active_of(p, it)[2 * g + 1];
  if (it >= 0 && blockIdx.x == 0 && threadIdx.x < 2) retire_half(p, it, g, threadIdx.x);
  const bool mx = (ax >> lane) & 1, my = (ay >> lane) & 1;
  if (!mx && !my) return;
  for (int b = int(blockIdx.x) * kWarps + (threadIdx.x >> 5); b < p.N; b += warps) bit_one(p, g, b, lane, mx, my);
}

// The persistent launches: for batches of at most kPersistGroups groups, all in one wave, on a
// stream that is not capturing.  Where asked for (persist == 1) they take full groups of 32 lanes
// or one narrow group; by themselves the narrow groups of persists_alone.

// One narrow group of a code of at most kPersistBits bits takes the persistent launch by itself
// where its call decodes nothing else beside it (`alone`) and no persistent launch of another stream is under
// way (ldpc_persist_launch): 1 to 16 DVB-S2 short frames, 50 iterations allowed,
// took 80 to 105 us against 230 a dB above the waterfall (8 iterations), 175 to 220 against
// 250 to 305 in it (18), and as long with frames that never converge (437 to 481 against 433 to
// 535).  Frames of 64800 bits gained as much when they converged early but ran 8 to 20 %
// longer when they did not, so they keep a launch per pass.  Groups of 2 lanes are widened
// to 4, which touch whole sectors of app (457 us against 438).
constexpr int kPersistBits = 20000;

bool persists_alone(const LdpcLanesParams& p) {
  return p.alone && p.persist == 0 && p.nframes <= 16 && p.N <= kPersistBits;
}

bool use_persistent(const LdpcLanesParams& p, int64_t wave, bool narrow, cudaStream_t s) {
  if ((p.persist <= 0 && !narrow) || p.groups > kPersistGroups || wave < p.groups) return false;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return false;
  }
  return true;
}

template <int DMAX>
cudaError_t launch_persistent(LdpcLanesParams p, cudaStream_t s) {
  auto kern = h2_persist<DMAX>;
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWarps * 32, 0)) != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  constexpr int kRows = DMAX <= 8 ? 2 : 1;
  const int64_t rows = (p.M + kRows - 1) / kRows;
  const int64_t units = int64_t(p.groups) * (int64_t(p.N) > rows ? int64_t(p.N) : rows);
  int64_t blocks = (units + kWarps - 1) / kWarps;
  if (blocks > int64_t(per_sm) * sms) blocks = int64_t(per_sm) * sms;
  if (blocks < 1) return cudaErrorInvalidConfiguration;
  if ((e = cudaMemsetAsync(p.barrier, 0, 2 * sizeof(unsigned), s)) != cudaSuccess) return e;
  void* args[] = {&p};
  return ldpc_persist_launch(s, reinterpret_cast<const void*>(kern), unsigned(blocks), kWarps * 32, 0, args, true);
}

// One block per SM at most; cudaErrorInvalidConfiguration where the index lists do not fit.
template <int DMAX, int W>
cudaError_t launch_narrow(LdpcLanesParams p, cudaStream_t s) {
  constexpr int kSlots = 32 / W, kBlockWarps = kNarrowThreads / 32;
  int dev = 0, sms = 0, limit = 0;
  cudaError_t e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  const int row_tasks = (p.M + kSlots - 1) / kSlots, bit_tasks = (p.N + kSlots - 1) / kSlots;
  const int need = ((row_tasks > bit_tasks ? row_tasks : bit_tasks) + kBlockWarps - 1) / kBlockWarps;
  const int blocks = need < sms ? need : sms, warps = blocks * kBlockWarps;
  int rows = (row_tasks + warps - 1) / warps, bits = (bit_tasks + warps - 1) / warps;
  const size_t smem = kBlockWarps * narrow_words_per_warp(p.d_max, p.c_max, W, rows, bits) * 4;
  if (blocks < 1 || smem + 1024 > size_t(limit)) return cudaErrorInvalidConfiguration;
  auto kern = h2_persist_narrow<DMAX, W>;
  if ((e = allow_shared_memory(kern)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(p.barrier, 0, 2 * sizeof(unsigned), s)) != cudaSuccess) return e;
  void* args[] = {&p, &rows, &bits};
  return ldpc_persist_launch(s, reinterpret_cast<const void*>(kern), unsigned(blocks), kNarrowThreads, smem, args, p.persist > 0);
}

// The grid of the staging and finishing kernels: 256 threads per block over the
// larger of a group's bit and edge slots, at most about eight blocks per SM in all.
dim3 stage_grid(const LdpcLanesParams& p, int W) {
  const int64_t need = ((p.N > p.E ? int64_t(p.N) : p.E) * W + 255) / 256;
  const int64_t share = (148 * 8 + p.groups - 1) / p.groups;
  const int64_t x = need < share ? need : share;
  return dim3(unsigned(x > 0 ? x : 1), unsigned(p.groups));
}

// A hard-decision decode: flow_stage, the first bit pass, flow_check and flow_bit per
// iteration, flow_finish; waves as below, of the smaller working set.
template <int DMAX, int W>
cudaError_t run_flow(const LdpcLanesParams& p, cudaStream_t s) {
  static_assert(W >= 8);
  constexpr int kSlots = 32 / W, kBits = kTile / (2 * W), kRows = rows_per_lane<DMAX, W>();
  const int64_t gb = int64_t(W) * (8 * int64_t(p.N) + 4 * p.E) + 8 * int64_t(p.N);
  int64_t wave = p.wave_groups > 0 ? p.wave_groups : kWaveCap / gb;
  if (wave < 1) wave = 1;
  if (wave > p.groups) wave = p.groups;
  flow_stage<W><<<dim3(unsigned((p.N + kBits - 1) / kBits), unsigned(p.groups)), 256, 0, s>>>(p);
  for (int w0 = 0; w0 < p.groups; w0 += int(wave)) {
    const int nw = p.groups - w0 < wave ? p.groups - w0 : int(wave);
    constexpr int kPerWarp = W == 32 ? kFlowBits : kSlots;
    const dim3 gbit = grid_for((p.N + kPerWarp - 1) / kPerWarp, nw);
    const dim3 gchk = grid_for((p.M + kRows * kSlots - 1) / (kRows * kSlots), nw);
    cudaError_t e = launch_pdl(flow_bit<W>, gbit, dim3(kWarps * 32), s, p, -1, w0);
    for (int it = 0; e == cudaSuccess && it < p.iterations; ++it) {
      e = launch_pdl(flow_check<DMAX, W>, gchk, dim3(kWarps * 32), s, p, it, w0);
      if (e == cudaSuccess) e = launch_pdl(flow_bit<W>, gbit, dim3(kWarps * 32), s, p, it, w0);
    }
    if (e != cudaSuccess) return e;
  }
  const bool quads = p.msg % 4 == 0 && reinterpret_cast<uintptr_t>(p.hard) % 4 == 0;
  const int per = 256 * (quads ? 4 : 1), parts = 4;
  const dim3 gf(unsigned((p.msg + per - 1) / per), unsigned(p.groups), unsigned(parts));
  if (quads) flow_finish<W, 4><<<gf, 256, 0, s>>>(p);
  else flow_finish<W, 1><<<gf, 256, 0, s>>>(p);
  return cudaGetLastError();
}

// Groups of 8 lanes, a sector per access, with rows of up to 16 edges keep the a-posteriori values
// where they fit in L2: the in-place bit pass's scattered stores then cost more than the gathers they
// save.  20 iterations on noise, values kept and in place: DVB-S2 short r=1/2 (rows of 7) x 48 290
// and 310 us, x 112 561 and 583, but in its waterfall 5 % the other way from there, so the line lies
// at 20 MB; r=3/5 x 112 699 and 776; normal r=3/5 x 48 1152 and 1273, x 80 1496 and 1610, x 112, beyond
// L2, 2168 and 2052; a single group of normal frames 0 to 13 % slower with the values kept.  Rows of
// more than 16 edges gain in place at every size (short r=8/9 x 48 338 and 278), and so do the jobs
// of a mixed batch, which share L2.
template <int DMAX, int W>
bool keeps_app(const LdpcLanesParams& p) {
  if (W > 8 || DMAX > 16 || !p.alone) return false;
  const int64_t bytes = int64_t(p.groups) * W * (2 * 8 * int64_t(p.N) + 4 * p.E);
  if (DMAX <= 8) return p.groups > 1 && bytes <= 20000000;
  return (p.groups > 1 || p.N <= kPersistBits) && bytes <= kWaveCap;
}

template <int DMAX, int W>
cudaError_t run(const LdpcLanesParams& p, cudaStream_t s) {
  if (p.groups > 65535) return cudaErrorInvalidValue;
  // Hard decisions alone, in launches per pass: messages in place.  Groups of 2 or 4 lanes keep
  // the a-posteriori values: with less than a sector per access the in-place bit pass's
  // scattered stores cost more than the gathers they save (one DVB-S2 short frame: 0.33 ms
  // against 0.25).
  if constexpr (W >= 8)
    if (!persists_alone(p) && !keeps_app<DMAX, W>(p) && p.hard && !p.msg_out && !p.syst_out && !p.parity_out && !p.state_out && !p.syst_in && p.persist <= 0)
      return run_flow<DMAX, W>(p, s);
  constexpr int kSlots = 32 / W;
  const int64_t gb = int64_t(W) * (2 * 8 * int64_t(p.N) + 4 * p.E);
  int64_t wave = p.wave_groups > 0 ? p.wave_groups : kWaveCap / gb;
  if (wave < 1) wave = 1;
  if (wave > p.groups) wave = p.groups;
  const dim3 gs = stage_grid(p, W);
  h2_stage<W><<<gs, 256, 0, s>>>(p);
  bool done = false;
  const bool narrow = W < kLanes && p.groups == 1 && persists_alone(p);
  if ((W == kLanes || p.groups == 1) && use_persistent(p, wave, narrow, s)) {
    cudaError_t e;
    if constexpr (W == kLanes) e = launch_persistent<DMAX>(p, s);
    else e = launch_narrow<DMAX, W>(p, s);
    if (e == cudaSuccess) done = true;
    else if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported && e != cudaErrorInvalidConfiguration &&
             e != cudaErrorNotReady)
      return e;
    else cudaGetLastError();
  }
  for (int w0 = 0; !done && w0 < p.groups; w0 += int(wave)) {
    const int nw = p.groups - w0 < wave ? p.groups - w0 : int(wave);
    constexpr int kRows = rows_per_lane<DMAX, W>();
    const dim3 gbit = grid_for((p.N + kSlots - 1) / kSlots, nw);
    const dim3 gchk = grid_for((p.M + kRows * kSlots - 1) / (kRows * kSlots), nw);
    cudaError_t e = launch_pdl(h2_bit<W>, gbit, dim3(kWarps * 32), s, p, -1, w0);
    for (int it = 0; e == cudaSuccess && it < p.iterations; ++it) {
      e = launch_pdl(h2_check<DMAX, W>, gchk, dim3(kWarps * 32), s, p, it, w0);
      if (e == cudaSuccess) e = launch_pdl(h2_bit<W>, gbit, dim3(kWarps * 32), s, p, it, w0);
    }
    if (e != cudaSuccess) return e;
  }
  if constexpr (W < kLanes) {
    if (done) {
      // a thread per bit and lane: fewer blocks than stage_grid's, whose many rounds of a kernel with
      // decode_by_block's registers took 4 us more (177 and 173 us a call)
      h2_finish_narrow<DMAX, W><<<unsigned((int64_t(p.N) * W + 255) / 256), 256, 0, s>>>(p);
      return cudaGetLastError();
    }
  }
  h2_finish<W><<<gs, 256, 0, s>>>(p);
  return cudaGetLastError();
}

template <int DMAX>
cudaError_t run_width(const LdpcLanesParams& p, int W, cudaStream_t s) {
  switch (W) {
    case 2: return run<DMAX, 2>(p, s);
    case 4: return run<DMAX, 4>(p, s);
    case 8: return run<DMAX, 8>(p, s);
    case 16: return run<DMAX, 16>(p, s);
    default: return run<DMAX, kLanes>(p, s);
  }
}

template <int DMAX>
int multi_blocks() {
  int per_sm = 0, dev = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, h2_multi<DMAX>, kWarps * 32, 0) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm * sms;
}

template <int DMAX>
cudaError_t launch_multi(LdpcMultiParams m, cudaStream_t s) {
  const int blocks = multi_blocks<DMAX>();
  if (blocks <= 0) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaMemsetAsync(m.barrier, 0, 2 * sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  // A cooperative launch (all blocks resident, so the grid barriers are safe).  Outside
  // a stream capture it is ordered after the device's previous persistent launch;
  // under capture it goes through cudaLaunchKernelEx, which records a cooperative
  // graph node.
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if ((e = cudaStreamIsCapturing(s, &cs)) != cudaSuccess) return e;
  if (cs == cudaStreamCaptureStatusNone) {
    void* args[] = {&m};
    return ldpc_persist_launch(s, reinterpret_cast<const void*>(h2_multi<DMAX>), unsigned(blocks), kWarps * 32, 0, args, true);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, h2_multi<DMAX>, m);
}

}  // namespace

size_t ldpc_lanes_h2_scratch_bytes(int64_t N, int64_t E, int64_t nframes) {
  const int64_t groups = (nframes + 63) / 64;
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  return al(size_t(groups) * N * kLanes * 8) * 2 + al(size_t(groups) * E * kLanes * 4) + al(size_t(groups) * 32) +
         al(size_t(groups) * 64 * 4) + al(2 * sizeof(unsigned));
}

void ldpc_lanes_h2_layout(LdpcLanesParams& p, void* scratch, int W) {
  p.groups = int32_t((p.nframes + 2 * W - 1) / (2 * W));
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  char* q = static_cast<char*>(scratch);
  p.chan = reinterpret_cast<float*>(q);
  q += al(size_t(p.groups) * p.N * W * 8);
  p.app = reinterpret_cast<float*>(q);
  q += al(size_t(p.groups) * p.N * W * 8);
  p.c2v = q;
  q += al(size_t(p.groups) * p.E * W * 4);
  p.active = reinterpret_cast<uint32_t*>(q);  // [2][groups][2]
  p.fail = p.active + 4 * p.groups;          // [2][groups][2]
  q += al(size_t(p.groups) * 32);
  p.iters_ws = reinterpret_cast<int32_t*>(q);
  q += al(size_t(p.groups) * 2 * W * 4);
  p.barrier = reinterpret_cast<unsigned*>(q);
}

// Lanes per group for a batch of n frames.  Up to 16 frames: the narrowest power of
// two from 2 to 8 whose group (2 W frames) holds the batch.  Beyond: 32, 16 or 8
// lanes, whichever leaves the fewest idle frame slots in the last group, the wider
// unless a narrower one saves more than n / 16 of them -- groups of 8 lanes and up
// still use every 32-byte sector they touch, narrower ones would not.
int ldpc_lanes_h2_width(int64_t nframes) {
  if (nframes <= 16) {
    int W = 2;
    while (2 * W < nframes) W *= 2;
    return W;
  }
  auto idle = [&](int64_t w) { return (nframes + 2 * w - 1) / (2 * w) * (2 * w) - nframes; };
  int best = kLanes;
  for (int W : {16, 8})
    if (idle(best) - idle(W) > nframes / 16) best = W;
  return best;
}

int64_t ldpc_lanes_h2_group_bytes(int64_t N, int64_t E) { return int64_t(kLanes) * (2 * 8 * N + 4 * E); }

cudaError_t launch_ldpc_h2_stage(const LdpcLanesParams& p, cudaStream_t s) {
  if (p.groups <= 0) return cudaSuccess;
  h2_stage<kLanes><<<dim3((148 * 8 + p.groups - 1) / p.groups, p.groups), 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_ldpc_h2_finish(const LdpcLanesParams& p, cudaStream_t s) {
  if (p.groups <= 0) return cudaSuccess;
  h2_finish<kLanes><<<dim3((148 * 8 + p.groups - 1) / p.groups, p.groups), 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_ldpc_h2_many(const LdpcMultiParams& m, const LdpcManyWave& w, int d_max, cudaStream_t s) {
  if (w.groups <= 0 || w.groups > 65535) return w.groups == 0 ? cudaSuccess : cudaErrorInvalidValue;
  const dim3 gbit = grid_for(w.max_bits, w.groups);
  const int kRows = d_max > 0 && d_max <= 8 ? 2 : 1;
  const dim3 gchk = grid_for((w.max_rows + kRows - 1) / kRows, w.groups);
  cudaError_t e = launch_pdl(h2_bit_many, gbit, dim3(kWarps * 32), s, m, -1, w.q0);
  for (int it = 0; e == cudaSuccess && it < w.iterations; ++it) {
    if (d_max <= 0) e = launch_pdl(h2_check_many<0>, gchk, dim3(kWarps * 32), s, m, it, w.q0);
    else if (d_max <= 8) e = launch_pdl(h2_check_many<8>, gchk, dim3(kWarps * 32), s, m, it, w.q0);
    else if (d_max <= 16) e = launch_pdl(h2_check_many<16>, gchk, dim3(kWarps * 32), s, m, it, w.q0);
    else e = launch_pdl(h2_check_many<32>, gchk, dim3(kWarps * 32), s, m, it, w.q0);
    if (e == cudaSuccess) e = launch_pdl(h2_bit_many, gbit, dim3(kWarps * 32), s, m, it, w.q0);
  }
  return e;
}

cudaError_t launch_ldpc_h2_multi(LdpcMultiParams m, int d_max, cudaStream_t s) {
  if (m.nwaves <= 0) return cudaSuccess;
  if (m.ncodes <= 0 || m.ncodes > kMultiMaxCodes) return cudaErrorInvalidValue;
  if (d_max <= 8) return launch_multi<8>(m, s);
  if (d_max <= 16) return launch_multi<16>(m, s);
  if (d_max <= 32) return launch_multi<32>(m, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_ldpc_lanes_h2(LdpcLanesParams p, void* scratch, cudaStream_t s) {
  if (p.nframes <= 0) return cudaSuccess;
  if (p.state_in || p.algorithm != 2) return cudaErrorInvalidValue;
  int W = ldpc_lanes_h2_width(p.nframes);
  if (W < 4 && persists_alone(p)) W = 4;
  ldpc_lanes_h2_layout(p, scratch, W);
  if (p.d_max <= 8) return run_width<8>(p, W, s);
  if (p.d_max <= 16) return run_width<16>(p, W, s);
  if (p.d_max <= 32) return run_width<32>(p, W, s);
  return cudaErrorInvalidValue;
}

}  // namespace fecl
