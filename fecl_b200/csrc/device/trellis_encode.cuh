// Encoding of one constituent of a trellis code by a CTA (the turbo and the convolutional
// device encoders).
//
// A thread walking a frame's trellis alone takes a chain of dependent loads per step.  Here the
// message is cut into a chunk per thread: each thread finds the state its chunk ends in for
// every state it may start in, one thread composes those maps from state 0, and every
// thread then walks its chunk from its true start, leaving the output words in shared
// memory, from where the bits go out contiguously.  The states and words are those of one walk.
#pragma once

#include <stdint.h>

#include "kernels.hpp"

namespace fecl {

constexpr int kEncodeThreads = 128;
constexpr int kEncodeStates = 64;   // states of a trellis encoded this way
constexpr int kEncodeSteps = 200 << 10;  // steps: a byte of shared memory each

inline bool encode_by_cta(const TurboDeviceConstituent& c) {
  return c.state_count <= kEncodeStates && c.input_count <= 4 && c.length <= kEncodeSteps && c.length > 0;
}

// Estimated microseconds of a CTA per message and of a thread per message (step_ns a step: 200 for
// a convolutional code, 400 through an interleaver), to within a third from 4 to 64 states, 1 to
// 6144 steps and 1 to 5000 messages: CTAs queue on the SMs and pay for their maps, threads all
// run at once up to a full chip.  So many short messages go a thread each (5000 of 40
// steps, CTA and thread: 64 states 96 and 15 us, 4 states 22 and 15; 8000 constituents of K=40
// 45 and 24), all others a CTA each (1024 steps of 64 states: 183 and 292).
inline double encode_cta_us(const TurboDeviceConstituent& c, int64_t messages) {
  return 1e-3 * double(messages) * (2.5 + 0.23 * c.state_count + c.length * (0.003 + 0.0003 * c.state_count));
}
inline double encode_thread_us(const TurboDeviceConstituent& c, int64_t messages, double step_ns) {
  const double chip = 148 * 2048, full = messages > chip ? messages / chip : 1.0;
  return 1e-3 * full * (3000.0 + step_ns * c.length);
}

struct EncodeShared {
  uint16_t branch[kEncodeStates * 4];  // next state | output word << 8
  uint8_t map[kEncodeThreads][kEncodeStates];
  uint8_t start[kEncodeThreads + 1];
};
constexpr size_t kEncodeFixed = sizeof(EncodeShared) + 1024;
static_assert(kEncodeFixed + kEncodeSteps <= 227 << 10);

// Message m (through the interleaver where perm is given) into the parity bits at par and,
// where tail_out is given, the termination's input bits there.  steps: c.length bytes of shared memory.
__device__ __forceinline__ void encode_constituent(const TurboDeviceConstituent& c, const uint8_t* m, const uint32_t* perm,
                                                   uint8_t* par, uint8_t* tail_out, EncodeShared& sh, uint8_t* steps) {
  const int S = c.state_count, U = c.input_count, is = c.input_size, os = c.output_size, L = c.length;
  const int tid = threadIdx.x;
  for (int i = tid; i < S * U; i += kEncodeThreads) sh.branch[i] = uint16_t(c.next_state[i] | (c.output[i] << 8));
  for (int t = tid; t < L; t += kEncodeThreads) {
    uint32_t u = 0;
    for (int k = 0; k < is; ++k) {
      const int i = t * is + k;
      u |= uint32_t(m[perm ? perm[i] : uint32_t(i)] & 1) << k;
    }
    steps[t] = uint8_t(u);
  }
  __syncthreads();
  const int len = (L + kEncodeThreads - 1) / kEncodeThreads;
  const int t0 = min(L, tid * len), t1 = min(L, t0 + len);
  for (int s0 = 0; s0 < S; s0 += 4) {  // four starts at a time, whose chains overlap
    uint32_t s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = uint32_t(min(s0 + q, S - 1));
    for (int t = t0; t < t1; ++t) {
      const uint32_t u = steps[t];
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] = sh.branch[s[q] * U + u] & 0xffu;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (s0 + q < S) sh.map[tid][s0 + q] = uint8_t(s[q]);
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t s = 0;
    for (int i = 0; i < kEncodeThreads; ++i) {
      sh.start[i] = uint8_t(s);
      s = sh.map[i][s];
    }
    sh.start[kEncodeThreads] = uint8_t(s);
  }
  __syncthreads();
  uint32_t state = sh.start[tid];
  for (int t = t0; t < t1; ++t) {
    const uint32_t b = sh.branch[state * U + steps[t]];
    steps[t] = uint8_t(b >> 8);
    state = b & 0xffu;
  }
  // greedy termination (src/detail/Convolutional.cpp:189-211)
  if (tid == kEncodeThreads - 1) {
    state = sh.start[kEncodeThreads];
    for (int s = 0; s < c.tail; ++s) {
      int best_count = -1;
      uint32_t best = 0;
      for (int u = 0; u < U; ++u) {
        const int count = __popc(state) - __popc(sh.branch[state * U + u] & 0xffu);
        if (count > best_count) {
          best_count = count;
          best = uint32_t(u);
        }
      }
      const uint32_t b = sh.branch[state * U + best];
      for (int k = 0; k < os; ++k) par[int64_t(L + s) * os + k] = uint8_t((b >> (8 + k)) & 1u);
      if (tail_out)
        for (int k = 0; k < is; ++k) tail_out[s * is + k] = uint8_t((best >> k) & 1u);
      state = b & 0xffu;
    }
  }
  __syncthreads();
  if (os == 1) {
    for (int t = tid; t < L; t += kEncodeThreads) par[t] = steps[t] & 1u;
  } else {
    for (int64_t i = tid; i < int64_t(L) * os; i += kEncodeThreads) {
      const int t = int(i / os);
      par[i] = (steps[t] >> int(i - int64_t(t) * os)) & 1u;
    }
  }
}

}  // namespace fecl
