// Viterbi decoding of the convolutional codec (Convolutional::decodeBlocks ->
// ViterbiDecoderImpl::decodeBlock, src/detail/ViterbiDecoder/ViterbiDecoderImpl.cpp).
//
// Path metrics start at [0, -inf, ...]; per trellis step the branch metrics are the
// correlations of each output word with the step's L-values; every (state, input)
// pair is compared in state-then-input order and the later one wins ties (>=),
// recording its state and input for the traceback; no normalisation.  Tail termination
// traces back from state 0, Truncate from the first state of largest metric.  The
// metrics are FP64, as the reference's (FloatLlrMetrics::Type is double), so the
// survivors -- and the decisions -- are the reference's bit for bit.
//
// viterbi_warp takes every trellis whose states all have as many predecessors as there
// are inputs, 2 or 4 (every shift-register trellis): the states of a frame lie across the
// lanes of a warp.  viterbi_kernel, a thread per frame walking the reference's loops,
// takes the others.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.hpp"
#include "trellis_encode.cuh"

namespace fecl {
namespace {

constexpr int kMaxStates = 64;
constexpr int kMaxOutputs = 64;

__global__ void __launch_bounds__(64) viterbi_kernel(TurboDeviceConstituent k, ViterbiRun r) {
  const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= r.nframes) return;
  const int S = k.state_count, U = k.input_count, O = 1 << k.output_size;
  const int T = k.length + k.tail;
  const int64_t P = k.parity_size;
  uint8_t* st = r.trace + f * int64_t(T) * S * 2;  // [T][S] states, then [T][S] inputs
  uint8_t* in = st + int64_t(T) * S;
  double pm[kMaxStates], nm[kMaxStates], bm[kMaxOutputs];
  pm[0] = 0.0;
  for (int s = 1; s < S; ++s) pm[s] = -INFINITY;
  for (int t = 0; t < T; ++t) {
    for (int o = 0; o < O; ++o) {
      double x = 0.0;
      for (int b = 0; b < k.output_size; ++b)
        if ((o >> b) & 1) x += double(load_llr(r.llr, r.llr_dtype, f * P + int64_t(t) * k.output_size + b));
      bm[o] = x;
    }
    for (int s = 0; s < S; ++s) nm[s] = -INFINITY;
    uint8_t* srow = st + int64_t(t) * S;
    uint8_t* irow = in + int64_t(t) * S;
    for (int j = 0; j < S; ++j)
      for (int u = 0; u < U; ++u) {
        const int n = int(k.next_state[j * U + u]);
        const double c = pm[j] + bm[k.output[j * U + u]];
        if (c >= nm[n]) {
          srow[n] = uint8_t(j);
          irow[n] = uint8_t(u);
          nm[n] = c;
        }
      }
    for (int s = 0; s < S; ++s) pm[s] = nm[s];
  }
  int best = 0;
  if (k.termination != 0)
    for (int s = 0; s < S; ++s)
      if (pm[s] > pm[best]) best = s;
  for (int t = T - 1; t >= 0; --t) {
    if (t < k.length) {
      const int u = in[int64_t(t) * S + best];
      for (int j = 0; j < k.input_size; ++j) r.hard[f * k.msg_size + int64_t(t) * k.input_size + j] = uint8_t((u >> j) & 1);
    }
    best = st[int64_t(t) * S + best];
  }
}

// A warp decodes 32 / G frames, G lanes each, SPL states per lane; P predecessors per
// state, in the reference's (state, input) order.
// Bound by the latency of a step (fetch the predecessors' metrics, add, compare, select):
// time cannot be split, since the FP64 sums run in order.  With one state per lane the
// metrics travel by shuffle.  With two, a shift register that drops its lowest bit (PAIR:
// predecessor i of every state is odd or even as i is) puts states 2 l and 2 l + 1 in lane
// l, so that predecessor i lies in slot i and a shuffle fetches it too; other trellises put
// state l + 32 s in slot s and pass the metrics through shared memory.  A block of 32
// steps' branch metrics is made at once in shared memory, from L-values loaded one block
// ahead.
//
// Decisions are kept as warp ballots (P = 2: one bit per state and step).  The traceback
// gives every lane of a frame a chunk of the steps: a lane starts `overlap` steps behind its
// chunk from state 0 -- the survivors of all states have mostly met by then -- and the state it
// reaches at the chunk's end is compared with the one the lane of the later chunk came
// out at; where they differ the chunk is walked again from that one, until all agree with
// the last chunk, which starts from the frame's final state.
// The constraint-length-7 code, 256 frames of 1024 bits: 104 us (about 100 ns a step)
// against 29.2 ms with a thread per frame, whose metrics and decisions went through local
// and global memory.  Carrying each state's origin along for the traceback instead cost
// 10 instructions a step (152 us through shared memory, 241 us by shuffle).
constexpr int kStep = 32;  // steps per block

struct ViterbiShape {
  int lanes, frames_per_warp, words, chunk, overlap;  // words: ballots per step; chunk: steps per lane
  size_t bm, pm, bytes;                               // shared memory: offsets of the doubles, total
};

ViterbiShape viterbi_shape(const TurboDeviceConstituent& k) {
  ViterbiShape v;
  const int O = 1 << k.output_size, T = k.length + k.tail;
  v.lanes = k.state_count <= 4 ? 4 : k.state_count <= 8 ? 8 : k.state_count <= 16 ? 16 : 32;
  while (v.lanes < 32 && 32 / v.lanes * O > 64) v.lanes *= 2;  // the branch metrics' shared memory
  v.frames_per_warp = 32 / v.lanes;
  v.words = (k.state_count > 32 ? 2 : 1) * (k.input_count > 2 ? 2 : 1);
  v.chunk = (T + v.lanes - 1) / v.lanes;
  int bits = 1;
  while ((1 << bits) < k.state_count) ++bits;
  v.overlap = 16 * (bits + 1);
  v.bm = size_t(v.frames_per_warp) * kStep * k.output_size;
  v.pm = v.bm + size_t(v.frames_per_warp) * kStep * O;
  v.bytes = (v.pm + 2 * 64) * sizeof(double) + size_t(k.state_count) * k.input_count * 4;
  return v;
}

template <int G, int SPL, int P, bool PAIR = false>
__global__ void __launch_bounds__(32) viterbi_warp(TurboDeviceConstituent k, ViterbiRun r, ViterbiShape v) {
  constexpr int kFrames = 32 / G, kBits = P > 2 ? 2 : 1, kWords = SPL * kBits;
  constexpr int kPre = 2 * kStep / G;         // L-values per lane loaded ahead: a block of two per step
  constexpr bool kShared = SPL > 1 && !PAIR;  // metrics through shared memory
  // the state in slot s of this lane; the lane (of its frame's group) and slot of a state
  auto state_at = [](int sub, int s) { return PAIR ? 2 * sub + s : sub + 32 * s; };
  auto lane_of = [](int st) { return PAIR ? st >> 1 : SPL > 1 ? st & 31 : st; };
  auto slot_of = [](int st) { return PAIR ? st & 1 : SPL > 1 ? st >> 5 : 0; };
  extern __shared__ __align__(16) double sh[];
  double* pms = sh + v.pm;                                     // [2][64] metrics
  uint32_t* pred = reinterpret_cast<uint32_t*>(pms + 2 * 64);  // [S][P] state | input << 8 | output << 16
  const int lane = threadIdx.x, sub = lane % G, fr = lane / G;
  const int S = k.state_count, os = k.output_size, O = 1 << os, T = k.length + k.tail;
  const int64_t f = int64_t(blockIdx.x) * kFrames + fr;
  const int64_t in0 = (f < r.nframes ? f : r.nframes - 1) * int64_t(k.parity_size);
  uint32_t* trace = reinterpret_cast<uint32_t*>(r.trace) + int64_t(blockIdx.x) * T * kWords;
  const int per_block = kStep * os, total = T * os;
  double* rw = sh + fr * per_block;       // this block's L-values
  double* b = sh + v.bm + fr * kStep * O; // and branch metrics

  for (int i = lane; i < S * P; i += 32) pred[i] = k.pred[i];
  __syncwarp();
  int src[SPL][P], out[SPL][P];
  double pm[SPL];
#pragma unroll
  for (int s = 0; s < SPL; ++s) {
    const int st = state_at(sub, s);
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const uint32_t e = st < S ? pred[st * P + p] : 0u;
      src[s][p] = kShared ? int(e & 0xffu) : lane_of(int(e & 0xffu));
      out[s][p] = int(e >> 16);
    }
    pm[s] = st == 0 ? 0.0 : -INFINITY;
    if (kShared) pms[st] = pm[s];
  }
  double pre[kPre];
  auto load_ahead = [&](int t0) {
#pragma unroll
    for (int q = 0; q < kPre; ++q) {
      const int i = q * G + sub, at = t0 * os + i;
      pre[q] = 0.0;
      if (i < per_block && at < total) pre[q] = double(load_llr(r.llr, r.llr_dtype, size_t(in0 + at)));
    }
  };
  int cur = 0;
  uint32_t kept[kWords];
  // Step t of a block.  NAN_ONLY_LOSES: an infinite L-value was seen, so that a candidate
  // may be NaN (against an unreached state); the reference starts from -inf, which every
  // number replaces and NaN does not.
  auto step = [&](int t, auto nan_only_loses) {
    double best[SPL];
    int d[SPL];
#pragma unroll
    for (int s = 0; s < SPL; ++s) {
      best[s] = 0.0;
      d[s] = 0;
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const double a = kShared ? pms[64 * cur + src[s][p]] : __shfl_sync(0xffffffffu, pm[PAIR ? p : 0], src[s][p], G);
        const double c = a + b[t * O + out[s][p]];
        const bool take = p == 0 || c >= best[s] || (nan_only_loses && best[s] != best[s]);
        best[s] = take ? c : best[s];
        d[s] = take ? p : d[s];
      }
    }
#pragma unroll
    for (int s = 0; s < SPL; ++s) {
      pm[s] = best[s];
      if (kShared) pms[64 * (cur ^ 1) + sub + 32 * s] = best[s];
#pragma unroll
      for (int q = 0; q < kBits; ++q) {
        const uint32_t w = __ballot_sync(0xffffffffu, (d[s] >> q) & 1);
        kept[s * kBits + q] = lane == t ? w : kept[s * kBits + q];
      }
    }
    if (kShared) {
      cur ^= 1;
      __syncwarp();
    }
  };

  load_ahead(0);
  bool infinite = false;
  for (int t0 = 0; t0 < T; t0 += kStep) {
    bool odd = false;
#pragma unroll
    for (int q = 0; q < kPre; ++q) {
      if (q * G + sub < per_block) rw[q * G + sub] = pre[q];
      odd = odd || !isfinite(pre[q]);
    }
    for (int i = kPre * G + sub; i < per_block; i += G) {
      const int at = t0 * os + i;
      const double x = at < total ? double(load_llr(r.llr, r.llr_dtype, size_t(in0 + at))) : 0.0;
      rw[i] = x;
      odd = odd || !isfinite(x);
    }
    infinite = __any_sync(0xffffffffu, odd) || infinite;
    __syncwarp();  // the block's L-values, other lanes' among them (a vote does not order memory)
    for (int e = sub; e < kStep * O; e += G) {
      const int t = e >> os, o = e & (O - 1);
      double x = 0.0;
      for (int j = 0; j < os; ++j)
        if ((o >> j) & 1) x += rw[t * os + j];
      b[e] = x;
    }
    if (t0 + kStep < T) load_ahead(t0 + kStep);
    __syncwarp();
    const int n = min(kStep, T - t0);
#pragma unroll
    for (int w = 0; w < kWords; ++w) kept[w] = 0;
    if (n == kStep && !infinite) {
#pragma unroll 8
      for (int t = 0; t < kStep; ++t) step(t, std::false_type{});
    } else {
#pragma unroll 1
      for (int t = 0; t < n; ++t) step(t, std::true_type{});
    }
    if (lane < n) {
#pragma unroll
      for (int w = 0; w < kWords; ++w) trace[int64_t(t0 + lane) * kWords + w] = kept[w];
    }
    __syncwarp();
  }

  // final state: 0 (Tail) or the first of largest metric
  double* fin = kShared ? pms + 64 * cur : pms;  // [frames][S]
  if (!kShared) {
#pragma unroll
    for (int s = 0; s < SPL; ++s) fin[fr * G + state_at(sub, s)] = pm[s];
  }
  __syncwarp();
  int last = 0;
  if (k.termination != 0) {
    const double* q = fin + fr * G;
    for (int s = 1; s < S; ++s)
      if (q[s] > q[last] || (q[last] != q[last] && q[s] > -INFINITY)) last = s;
  }

  // traceback
  const int t_lo = min(T, sub * v.chunk), t_hi = min(T, t_lo + v.chunk);
  uint8_t* hard = f < r.nframes ? r.hard + f * k.msg_size : nullptr;
  // Walks from the state after step t - 1 down to the state before step lo, writing the
  // inputs of steps below `upto`; the ballots of 8 steps are loaded at once.
  auto walk = [&](int state, int t, int lo, int upto) {
    for (--t; t >= lo; t -= 8) {
      uint32_t w[8][kWords];
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int x = 0; x < kWords; ++x) w[j][x] = t - j >= lo ? trace[int64_t(t - j) * kWords + x] : 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (t - j < lo) continue;
        const int bit = fr * G + lane_of(state), hi = slot_of(state);
        uint32_t d = ((hi ? w[j][(SPL - 1) * kBits] : w[j][0]) >> bit) & 1u;
        if (kBits > 1) d |= (((hi ? w[j][(SPL - 1) * kBits + kBits - 1] : w[j][kBits - 1]) >> bit) & 1u) << 1;
        const uint32_t e = pred[state * P + d];
        state = int(e & 0xffu);
        if (t - j < upto && hard) {
          const uint32_t u = (e >> 8) & 0xffu;
          for (int i = 0; i < k.input_size; ++i) hard[int64_t(t - j) * k.input_size + i] = uint8_t((u >> i) & 1u);
        }
      }
    }
    return state;
  };
  const int t_from = min(T, t_hi + v.overlap);
  int at_hi = walk(t_from == T ? last : 0, t_from, t_hi, 0);
  bool again = t_lo < t_hi;
  int at_lo = at_hi;
  do {
    if (again) at_lo = walk(at_hi, t_hi, t_lo, k.length);
    else if (t_lo >= t_hi) at_lo = last;
    __syncwarp();
    const int want = __shfl_down_sync(0xffffffffu, at_lo, 1, G);
    again = t_hi < T && at_hi != want;
    at_hi = again ? want : at_hi;
  } while (__any_sync(0xffffffffu, again));
}

__global__ void __launch_bounds__(kEncodeThreads) conv_encode_cta(const __grid_constant__ TurboDeviceConstituent c,
                                                                  const uint8_t* msg, uint8_t* parity) {
  __shared__ EncodeShared sh;
  extern __shared__ __align__(16) uint8_t s[];
  const int64_t f = blockIdx.x;
  encode_constituent(c, msg + f * c.msg_size, nullptr, parity + f * c.parity_size, nullptr, sh, s);
}

// A thread per frame, for trellises and lengths beyond conv_encode_cta's and for many short messages
// (encode_cta_us).
__global__ void conv_encode_kernel(TurboDeviceConstituent c, const uint8_t* msg, uint8_t* parity, int64_t nframes) {
  const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= nframes) return;
  const uint8_t* m = msg + f * c.msg_size;
  uint8_t* out = parity + f * c.parity_size;
  uint32_t state = 0;
  for (int s = 0; s < c.length; ++s) {
    uint32_t u = 0;
    for (int k = 0; k < c.input_size; ++k) u |= uint32_t(m[s * c.input_size + k] & 1) << k;
    const uint32_t o = c.output[state * c.input_count + u];
    state = c.next_state[state * c.input_count + u];
    for (int k = 0; k < c.output_size; ++k) out[s * c.output_size + k] = uint8_t((o >> k) & 1);
  }
  // greedy termination (src/detail/Convolutional.cpp:189-211)
  for (int s = 0; s < c.tail; ++s) {
    int best_count = -1;
    uint32_t best = 0;
    for (int u = 0; u < c.input_count; ++u) {
      const int count = __popc(state) - __popc(c.next_state[state * c.input_count + u]);
      if (count > best_count) {
        best_count = count;
        best = uint32_t(u);
      }
    }
    const uint32_t o = c.output[state * c.input_count + best];
    for (int k = 0; k < c.output_size; ++k) out[(c.length + s) * c.output_size + k] = uint8_t((o >> k) & 1);
    state = c.next_state[state * c.input_count + best];
  }
}

}  // namespace

// Whether the trellis takes viterbi_warp: a predecessor table with one entry per input.
static bool viterbi_lanes_ok(const TurboDeviceConstituent& k) {
  return k.pred && (k.input_count == 2 || k.input_count == 4) && k.length + k.tail > 0;
}

size_t viterbi_scratch_bytes(const TurboDeviceConstituent& k, int64_t nframes) {
  const size_t T = size_t(k.length + k.tail);
  if (!viterbi_lanes_ok(k)) return size_t(nframes) * T * size_t(k.state_count) * 2 + 256;
  const ViterbiShape v = viterbi_shape(k);
  return size_t((nframes + v.frames_per_warp - 1) / v.frames_per_warp) * T * size_t(v.words) * 4 + 256;
}

template <int G, int SPL>
static cudaError_t run_viterbi(const TurboDeviceConstituent& k, const ViterbiRun& r, const ViterbiShape& v, cudaStream_t s) {
  const int64_t blocks = (r.nframes + v.frames_per_warp - 1) / v.frames_per_warp;
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  if constexpr (SPL > 1) {
    if (k.pred_paired) {
      viterbi_warp<G, SPL, 2, true><<<unsigned(blocks), 32, v.bytes, s>>>(k, r, v);
      return cudaGetLastError();
    }
  }
  if (k.input_count == 2) viterbi_warp<G, SPL, 2><<<unsigned(blocks), 32, v.bytes, s>>>(k, r, v);
  else viterbi_warp<G, SPL, 4><<<unsigned(blocks), 32, v.bytes, s>>>(k, r, v);
  return cudaGetLastError();
}

cudaError_t launch_viterbi(const TurboDeviceConstituent& k, const ViterbiRun& r, cudaStream_t s) {
  if (r.nframes <= 0) return cudaSuccess;
  if (k.state_count > kMaxStates || k.output_size > 6 || k.input_count > 256) return cudaErrorInvalidValue;
  if (viterbi_lanes_ok(k)) {
    const ViterbiShape v = viterbi_shape(k);
    if (k.state_count > 32) return run_viterbi<32, 2>(k, r, v, s);
    switch (v.lanes) {
      case 4: return run_viterbi<4, 1>(k, r, v, s);
      case 8: return run_viterbi<8, 1>(k, r, v, s);
      case 16: return run_viterbi<16, 1>(k, r, v, s);
      default: return run_viterbi<32, 1>(k, r, v, s);
    }
  }
  viterbi_kernel<<<unsigned((r.nframes + 63) / 64), 64, 0, s>>>(k, r);
  return cudaGetLastError();
}

cudaError_t launch_conv_encode(const TurboDeviceConstituent& c, const uint8_t* msg, uint8_t* parity, int64_t nframes,
                               cudaStream_t s) {
  if (nframes <= 0) return cudaSuccess;
  if (encode_by_cta(c) && nframes <= 0x7fffffff && encode_cta_us(c, nframes) <= encode_thread_us(c, nframes, 200.0)) {
    const cudaError_t e = allow_shared_memory(conv_encode_cta, kEncodeFixed);
    if (e != cudaSuccess) return e;
    conv_encode_cta<<<unsigned(nframes), kEncodeThreads, size_t(c.length), s>>>(c, msg, parity);
    return cudaGetLastError();
  }
  conv_encode_kernel<<<unsigned((nframes + 63) / 64), 64, 0, s>>>(c, msg, parity, nframes);
  return cudaGetLastError();
}

}  // namespace fecl
