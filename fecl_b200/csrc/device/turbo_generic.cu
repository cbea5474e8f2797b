// Generic turbo decoder, FP32 metrics: any number of constituents, any small
// trellis, Tail or Truncate, Serial or Parallel exchange, all three algorithms.
//
// Every value is computed by the reference's sequence of operations, in FP32:
//   TurboDecoderImpl::decodeBlock / soDecodeBlock (src/detail/TurboDecoder/TurboDecoderImpl.cpp:31-150)
//   serialTransferUpdate / parallelTransferUpdate / aPosterioriUpdate (:152-250)
//   MapDecoderImpl branch/forward/backward/aPosteriori updates
//     (src/detail/MapDecoder/MapDecoderImpl.cpp:80-410), with the log-sum policies of
//     src/detail/LlrMetrics.h:48-121.
// This is the kernel used for arbitrary codes; the LTE code has its own windowed kernel.
//
// turbo_generic_cta decodes a frame with a CTA.  A MAP pass runs the forward recursion in
// one warp and the backward one in another, a state (two beyond 32 states) per lane, while two
// more warps make the branch metrics of the next block of steps; then every
// thread forms the outputs of steps of its own from the stored metrics.  Within a state
// and within an output the sums run in the reference's order -- they are not associative
// under the Linear and Exact algorithms -- so the values are those of one thread walking the
// reference's loops, as turbo_generic_f32 does for the codes that keep it (states with unequal
// numbers of predecessors, interleavers with repeated indices) and for thousands of short
// frames (map_cta_us).  Bound by the latency of the
// recursions' steps (shuffle, add, table sum, warp maximum; about 85 ns in Linear with the
// step's outputs): 128 frames of a K = 1024 two-constituent code, 6 iterations, take 1.22 ms
// against 263 ms with a thread per frame, and 3.45 ms before the number of branches was a
// compile-time constant and the shuffles ran beside the maximum.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.hpp"

namespace fecl {
namespace {

constexpr int kExact = 0, kLinear = 1, kApproximate = 2;
constexpr int kMaxS = 64;  // states
constexpr int kMaxU = 4;   // branches per state
constexpr float kNegInf = -INFINITY;

__constant__ LinearLut c_lut;
__constant__ LinearPairs c_pairs;

// Recursive log-sum (MaxLogSum / LinearLogSum) of two metrics.
template <int ALG>
__device__ __forceinline__ float lsum(float a, float b) {
  if (ALG == kApproximate) return fmaxf(a, b);
  if (a == b) return a;  // LinearLogSum::sum, src/detail/LlrMetrics.h:107-112
  return fmaxf(a, b) + lut_log1pexpm(c_lut, fabsf(a - b));
}

// Exact (LogSum) prior(x, max): 1 when x == max, exp(x - max) otherwise.
__device__ __forceinline__ float eprior(float x, float mx) { return (x == mx) ? 1.0f : expf(x - mx); }

struct Frame {
  float* pin;   // parityIn_  [parity]
  float* pout;  // parityOut_ [parity]
  float* ext;   // extrinsic_ [state]
  float* extb;  // extrinsicBuffer_ [state]
  float* alpha;
};

__device__ __forceinline__ float gamma_of(const TurboDeviceConstituent& k, const float* par, const float* sys, int t,
                                          int s, int u) {
  // correlation of the branch output with the parity L-values, then of the input
  // with the a-priori L-values (MapDecoderImpl.cpp:86-108)
  const uint32_t out = k.output[s * k.input_count + u];
  float g = 0.0f;
  for (int b = 0; b < k.output_size; ++b)
    if ((out >> b) & 1) g += par[t * k.output_size + b];
  float h = 0.0f;
  for (int b = 0; b < k.input_size; ++b)
    if ((u >> b) & 1) h += sys[t * k.input_size + b];
  return g + h;
}

// One MAP pass of constituent k.  sys: a-priori in, extrinsic out (in place).
// par: the constituent's parity L-values.  parity_out: optional parity extrinsic.
// app_out (optional): sf * L of the message steps' input bits (the convolutional
// codec's msg output, MapDecoderImpl.cpp:197-212).
template <int ALG>
__device__ void map_pass(const TurboDeviceConstituent& k, const float* par, float* sys, float* parity_out, float sf,
                         float* alpha, float* app_out = nullptr) {
  const int S = k.state_count, U = k.input_count;
  const int T = k.length + k.tail;
  if (T == 0) return;  // a truncated code of no bits: no step, no metrics
  // forward, MapDecoderImpl.cpp:117-139 (recursive) and :237-274 (LogSum)
  alpha[0] = 0.0f;
  for (int s = 1; s < S; ++s) alpha[s] = kNegInf;
  for (int t = 0; t + 1 < T; ++t) {
    const float* a = alpha + t * S;
    float* an = alpha + (t + 1) * S;
    if (ALG == kExact) {
      float mx[kMaxS], acc[kMaxS];
      for (int s = 0; s < S; ++s) mx[s] = kNegInf;
      for (int s = 0; s < S; ++s)
        for (int u = 0; u < U; ++u) {
          const int n = k.next_state[s * U + u];
          mx[n] = fmaxf(a[s] + gamma_of(k, par, sys, t, s, u), mx[n]);
        }
      for (int s = 0; s < S; ++s) acc[s] = 0.0f;
      for (int s = 0; s < S; ++s)
        for (int u = 0; u < U; ++u) {
          const int n = k.next_state[s * U + u];
          acc[n] = eprior(a[s] + gamma_of(k, par, sys, t, s, u), mx[n]) + acc[n];
        }
      for (int s = 0; s < S; ++s) an[s] = logf(acc[s]) + mx[s];
    } else {
      for (int s = 0; s < S; ++s) an[s] = kNegInf;
      for (int s = 0; s < S; ++s)
        for (int u = 0; u < U; ++u) {
          const int n = k.next_state[s * U + u];
          an[n] = lsum<ALG>(an[n], a[s] + gamma_of(k, par, sys, t, s, u));
        }
    }
    float m = kNegInf;
    for (int s = 0; s < S; ++s) m = fmaxf(an[s], m);
    for (int s = 0; s < S; ++s) an[s] -= m;
  }
  // backward + a-posteriori, MapDecoderImpl.cpp:141-235
  float beta[kMaxS], bprev[kMaxS];
  if (k.termination == 0) {
    beta[0] = 0.0f;
    for (int s = 1; s < S; ++s) beta[s] = kNegInf;
  } else {
    for (int s = 0; s < S; ++s) beta[s] = 0.0f;
  }
  for (int t = T - 1; t >= 0; --t) {
    const float* a = alpha + t * S;
    // delta[s][u] = gamma + alpha + beta(next)
    float delta[kMaxS * kMaxU];
    for (int s = 0; s < S; ++s)
      for (int u = 0; u < U; ++u)
        delta[s * U + u] = gamma_of(k, par, sys, t, s, u) + a[s] + beta[k.next_state[s * U + u]];
    // input bits
    float lin[4];
    for (int j = 0; j < k.input_size; ++j) {
      float r;
      if (ALG == kExact) {
        float mx0 = kNegInf, mx1 = kNegInf, m0 = 0.0f, m1 = 0.0f;
        for (int s = 0; s < S; ++s)
          for (int u = 0; u < U; ++u) {
            if ((u >> j) & 1) mx1 = fmaxf(delta[s * U + u], mx1);
            else mx0 = fmaxf(delta[s * U + u], mx0);
          }
        for (int s = 0; s < S; ++s)
          for (int u = 0; u < U; ++u) {
            if ((u >> j) & 1) m1 = eprior(delta[s * U + u], mx1) + m1;
            else m0 = eprior(delta[s * U + u], mx0) + m0;
          }
        r = (logf(m1) + mx1) - (logf(m0) + mx0);
      } else {
        float m0 = kNegInf, m1 = kNegInf;
        for (int s = 0; s < S; ++s)
          for (int u = 0; u < U; ++u) {
            if ((u >> j) & 1) m1 = lsum<ALG>(m1, delta[s * U + u]);
            else m0 = lsum<ALG>(m0, delta[s * U + u]);
          }
        r = m1 - m0;
      }
      lin[j] = r;
    }
    // parity bits (only when requested)
    if (parity_out) {
      for (int j = 0; j < k.output_size; ++j) {
        float r;
        if (ALG == kExact) {
          float mx0 = kNegInf, mx1 = kNegInf, m0 = 0.0f, m1 = 0.0f;
          for (int s = 0; s < S; ++s)
            for (int u = 0; u < U; ++u) {
              const bool b = (k.output[s * U + u] >> j) & 1;
              if (b) mx1 = fmaxf(delta[s * U + u], mx1);
              else mx0 = fmaxf(delta[s * U + u], mx0);
            }
          for (int s = 0; s < S; ++s)
            for (int u = 0; u < U; ++u) {
              const bool b = (k.output[s * U + u] >> j) & 1;
              if (b) m1 = eprior(delta[s * U + u], mx1) + m1;
              else m0 = eprior(delta[s * U + u], mx0) + m0;
            }
          r = (logf(m1) + mx1) - (logf(m0) + mx0);
        } else {
          float m0 = kNegInf, m1 = kNegInf;
          for (int s = 0; s < S; ++s)
            for (int u = 0; u < U; ++u) {
              const bool b = (k.output[s * U + u] >> j) & 1;
              if (b) m1 = lsum<ALG>(m1, delta[s * U + u]);
              else m0 = lsum<ALG>(m0, delta[s * U + u]);
            }
          r = m1 - m0;
        }
        parity_out[t * k.output_size + j] = sf * (r - par[t * k.output_size + j]);
      }
    }
    // next beta (state after step t-1) from beta and gamma_t
    if (t > 0) {
      if (ALG == kExact) {
        for (int s = 0; s < S; ++s) {
          float mx = kNegInf;
          float buf[kMaxU];
          for (int u = 0; u < U; ++u) {
            buf[u] = beta[k.next_state[s * U + u]] + gamma_of(k, par, sys, t, s, u);
            mx = fmaxf(buf[u], mx);
          }
          float acc = 0.0f;
          for (int u = 0; u < U; ++u) acc = eprior(buf[u], mx) + acc;
          bprev[s] = logf(acc) + mx;
        }
      } else {
        for (int s = 0; s < S; ++s) {
          float acc = kNegInf;
          for (int u = 0; u < U; ++u)
            acc = lsum<ALG>(acc, beta[k.next_state[s * U + u]] + gamma_of(k, par, sys, t, s, u));
          bprev[s] = acc;
        }
      }
      float m = kNegInf;
      for (int s = 0; s < S; ++s) m = fmaxf(bprev[s], m);
      for (int s = 0; s < S; ++s) beta[s] = bprev[s] - m;
    }
    // extrinsic on the input bits, written over the a-priori of this step
    for (int j = 0; j < k.input_size; ++j) {
      const int idx = t * k.input_size + j;
      if (app_out && t < k.length) app_out[idx] = sf * lin[j];
      sys[idx] = sf * (lin[j] - sys[idx]);
    }
  }
}

__device__ void serial_transfer(const TurboDeviceCode& c, Frame& fr, int i) {
  // TurboDecoderImpl::serialTransferUpdate, TurboDecoderImpl.cpp:225-250
  float* syst = fr.pout;
  for (int k = 0; k < c.msg; ++k) syst[k] = fr.pin[k];
  const float* systTail = fr.pin + c.msg;
  float* ext = fr.ext;
  for (int j = 0; j < i; ++j) {
    for (int k = 0; k < c.c[j].msg_size; ++k) syst[c.c[j].perm[k]] += ext[k];
    ext += c.c[j].syst_size;
    systTail += c.c[j].syst_tail_size;
  }
  float* slot = ext;
  ext += c.c[i].msg_size;
  for (int k = 0; k < c.c[i].syst_tail_size; ++k) ext[k] = systTail[k];
  ext += c.c[i].syst_tail_size;
  for (int j = i + 1; j < c.n; ++j) {
    for (int k = 0; k < c.c[j].msg_size; ++k) syst[c.c[j].perm[k]] += ext[k];
    ext += c.c[j].syst_size;
  }
  for (int k = 0; k < c.c[i].msg_size; ++k) slot[k] = syst[c.c[i].perm[k]];
}

__device__ void parallel_transfer(const TurboDeviceCode& c, Frame& fr) {
  // TurboDecoderImpl::parallelTransferUpdate, TurboDecoderImpl.cpp:191-223
  float* ext = fr.ext;
  float* tmp = fr.extb;
  const float* systTail = fr.pin + c.msg;
  float* syst = fr.pout;
  for (int k = 0; k < c.msg; ++k) syst[k] = 0.0f;
  for (int j = 0; j < c.n; ++j) {
    const TurboDeviceConstituent& q = c.c[j];
    for (int k = 0; k < q.msg_size; ++k) {
      tmp[k] = ext[k];
      ext[k] = syst[q.perm[k]];
      syst[q.perm[k]] += tmp[k];
    }
    ext += q.msg_size;
    tmp += q.msg_size;
    for (int k = 0; k < q.syst_tail_size; ++k) ext[k] = systTail[k];
    ext += q.syst_tail_size;
    systTail += q.syst_tail_size;
  }
  for (int k = 0; k < c.msg; ++k) syst[k] = fr.pin[k];
  for (int j = c.n - 1; j >= 0; --j) {
    const TurboDeviceConstituent& q = c.c[j];
    ext -= q.syst_size;
    tmp -= q.msg_size;
    for (int k = 0; k < q.msg_size; ++k) {
      ext[k] += syst[q.perm[k]];
      syst[q.perm[k]] += tmp[k];
    }
  }
}

// Membership in a sorted constituent list [lo, hi), advanced monotonically like the
// reference's iterator walks.
__device__ __forceinline__ bool take(const int32_t* list, int& at, int hi, int j) {
  while (at < hi && list[at] < j) ++at;
  return at < hi && list[at] == j;
}

// TurboDecoderImpl::customTransferUpdate, TurboDecoderImpl.cpp:252-289: the a-priori
// input of activation a (constituent i) is the channel systematic plus the
// de-interleaved extrinsic values of the listed constituents, interleaved into the
// buffer's slot of constituent i; the systematic tail is copied into the live
// extrinsic array (as the reference does), not into the buffer.
__device__ void custom_transfer(const TurboDeviceCode& c, Frame& fr, int a) {
  const int i = c.act_con[a];
  const int t_hi = c.act_tptr[a + 1];
  int at = c.act_tptr[a];
  float* syst = fr.pout;
  for (int k = 0; k < c.msg; ++k) syst[k] = fr.pin[k];
  const float* ext = fr.ext;
  float* tmp = fr.extb;
  const float* systTail = fr.pin + c.msg;
  for (int j = 0; j < i; ++j) {
    if (take(c.transfer, at, t_hi, j))
      for (int k = 0; k < c.c[j].msg_size; ++k) syst[c.c[j].perm[k]] += ext[k];
    ext += c.c[j].syst_size;
    tmp += c.c[j].syst_size;
    systTail += c.c[j].syst_tail_size;
  }
  float* slot = tmp;
  float* tail_dst = fr.ext + (ext - fr.ext) + c.c[i].msg_size;
  for (int k = 0; k < c.c[i].syst_tail_size; ++k) tail_dst[k] = systTail[k];
  ext += c.c[i].syst_size;
  for (int j = i + 1; j < c.n; ++j) {
    if (take(c.transfer, at, t_hi, j)) {
      for (int k = 0; k < c.c[j].msg_size; ++k) syst[c.c[j].perm[k]] += ext[k];
    } else if (at >= t_hi) {
      break;
    }
    ext += c.c[j].syst_size;
  }
  for (int k = 0; k < c.c[i].msg_size; ++k) slot[k] = syst[c.c[i].perm[k]];
}

// TurboDecoderImpl::customActivationUpdate, TurboDecoderImpl.cpp:170-189: the stage's
// constituents, in increasing order, each with the scaling of (iteration, constituent)
// -- in decode and soDecode alike.
template <int ALG>
__device__ void custom_activation(const TurboDeviceCode& c, Frame& fr, int it, int stage) {
  const int hi = c.stage_ptr[stage + 1];
  int at = c.stage_ptr[stage];
  const float* par = fr.pin + c.syst;
  float* ext = fr.ext;
  for (int j = 0; j < c.n; ++j) {
    if (take(c.act_con, at, hi, j)) map_pass<ALG>(c.c[j], par, ext, nullptr, c.sf[j * c.iterations + it], fr.alpha);
    else if (at >= hi) break;
    ext += c.c[j].syst_size;
    par += c.c[j].parity_size;
  }
}

__device__ void aposteriori(const TurboDeviceCode& c, Frame& fr) {
  // TurboDecoderImpl::aPosterioriUpdate, TurboDecoderImpl.cpp:152-168
  const float* ext = fr.ext;
  float* systTail = fr.pout + c.msg;
  float* syst = fr.pout;
  for (int j = 0; j < c.n; ++j) {
    const TurboDeviceConstituent& q = c.c[j];
    for (int k = 0; k < q.msg_size; ++k) syst[q.perm[k]] += ext[k];
    ext += q.msg_size;
    for (int k = 0; k < q.syst_tail_size; ++k) systTail[k] += ext[k];
    ext += q.syst_tail_size;
    systTail += q.syst_tail_size;
  }
}

// CRC stop (an extension): the decisions the frame would end with after this
// iteration -- channel systematic plus every constituent's extrinsic values, as at
// the end of decodeBlock -- and whether their CRC syndrome, the xor of the table
// entries of the bits that are 1, is zero.  Uses the systematic part of parity_buf,
// which every transfer rewrites before it reads it.
__device__ bool crc_passes(const TurboDeviceCode& c, Frame& fr, const uint32_t* crc) {
  for (int k = 0; k < c.msg; ++k) fr.pout[k] = fr.pin[k];
  aposteriori(c, fr);
  uint32_t syn = 0;
  for (int k = 0; k < c.msg; ++k)
    if (fr.pout[k] > 0.0f) syn ^= __ldg(crc + k);
  return syn == 0;
}

template <int ALG>
__global__ void __launch_bounds__(64) turbo_generic_f32(TurboDeviceCode c, TurboRun p) {
  const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= p.nframes) return;
  Frame fr;
  fr.pin = p.parity_in + f * c.parity;
  fr.pout = p.parity_buf + f * c.parity;
  fr.ext = p.ext + f * c.state;
  fr.extb = p.ext_buf + f * c.state;
  fr.alpha = p.alpha + f * int64_t(c.max_steps) * c.max_states;

  for (int k = 0; k < c.parity; ++k) fr.pin[k] = load_llr(p.llr, p.llr_dtype, f * c.parity + k);
  if (p.syst_in)
    for (int k = 0; k < c.syst; ++k) fr.pin[k] += load_llr(p.syst_in, p.llr_dtype, f * c.syst + k);
  for (int k = 0; k < c.state; ++k) fr.ext[k] = p.state_in ? load_llr(p.state_in, p.llr_dtype, f * c.state + k) : 0.0f;
  for (int k = 0; k < c.parity; ++k) fr.pout[k] = 0.0f;

  const bool want_parity = p.soft && p.parity_out;
  if (p.soft && c.iterations == 0 && want_parity)
    for (int k = c.syst; k < c.parity; ++k) fr.pout[k] = 0.0f;

  int ran = c.iterations;
  for (int i = 0; i < c.iterations; ++i) {
    if (c.scheduling == 2) {
      for (int st = 0; st < c.n_stages; ++st) {
        for (int k = 0; k < c.state; ++k) fr.extb[k] = fr.ext[k];
        for (int a = c.stage_ptr[st]; a < c.stage_ptr[st + 1]; ++a) custom_transfer(c, fr, a);
        float* t = fr.ext;
        fr.ext = fr.extb;
        fr.extb = t;
        custom_activation<ALG>(c, fr, i, st);
      }
    } else {
      if (c.scheduling == 1) parallel_transfer(c, fr);
      const float* par = fr.pin + c.syst;
      float* pout = fr.pout + c.syst;
      float* ext = fr.ext;
      for (int j = 0; j < c.n; ++j) {
        if (c.scheduling == 0) serial_transfer(c, fr, j);
        const float sf = p.soft ? 1.0f : c.sf[j * c.iterations + i];
        const bool last = (i == c.iterations - 1);
        map_pass<ALG>(c.c[j], par, ext, (want_parity && last) ? pout : nullptr, sf, fr.alpha);
        ext += c.c[j].syst_size;
        par += c.c[j].parity_size;
        pout += c.c[j].parity_size;
      }
    }
    if (!p.soft && p.crc && i + 1 < c.iterations && crc_passes(c, fr, p.crc)) {
      ran = i + 1;
      break;
    }
  }

  if (!p.soft) {
    for (int k = 0; k < c.msg; ++k) fr.pout[k] = fr.pin[k];
    aposteriori(c, fr);
    for (int k = 0; k < c.msg; ++k) p.hard[f * c.msg + k] = uint8_t(fr.pout[k] > 0.0f);
  } else {
    for (int k = 0; k < c.syst; ++k) fr.pout[k] = 0.0f;
    aposteriori(c, fr);
    if (p.syst_out)
      for (int k = 0; k < c.syst; ++k) store_llr(p.syst_out, p.out_dtype, f * c.syst + k, fr.pout[k]);
    if (p.parity_out)
      for (int k = 0; k < c.parity; ++k) store_llr(p.parity_out, p.out_dtype, f * c.parity + k, fr.pout[k]);
    if (p.state_out)
      for (int k = 0; k < c.state; ++k) store_llr(p.state_out, p.out_dtype, f * c.state + k, fr.ext[k]);
    if (p.msg_out)
      for (int k = 0; k < c.msg; ++k) store_llr(p.msg_out, p.out_dtype, f * c.msg + k, fr.pin[k] + fr.pout[k]);
  }
  if (p.iters) p.iters[f] = ran;
}

// ---- a CTA per frame ---------------------------------------------------------------

constexpr int kMapThreads = 128;
constexpr int kTable = 1024;  // branch metrics of a block of steps

struct MapShared {
  float gam[2][2][kTable];  // [direction][buffer] branch metrics by step, input and output word
  uint32_t branch[kMaxS * kMaxU];  // next state | branch metric << 8 of every (state, input)
  float2 pairs[8];          // the Linear table
  uint32_t part[kMapThreads / 32];
};

template <int ALG>
__device__ __forceinline__ float log_sum(const MapShared& sh, float a, float b) {
  return ALG == kApproximate ? fmaxf(a, b) : linear_sum(sh.pairs, a, b);
}

// The largest value over the warp (sm_100: one instruction).
__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// Steps per block: as many as the table holds branch metrics for, at most 32.
__device__ __forceinline__ int block_steps(const TurboDeviceConstituent& k) {
  const int n = kTable / (k.input_count << k.output_size);
  return n < 32 ? n : 32;
}

// Branch metrics of the steps [t0, t0 + n) into tab[step][input][output word], `stride` apart
// per step: the sums of gamma_of, by `threads` threads.
__device__ __forceinline__ void fill_gammas(const TurboDeviceConstituent& k, const float* par, const float* sys, int t0,
                                            int n, float* tab, int thread, int threads, int stride) {
  const int os = k.output_size, is = k.input_size, bits = os + is;
  for (int e = thread; e < n << bits; e += threads) {
    const int tt = e >> bits, q = e & ((1 << bits) - 1), o = q & ((1 << os) - 1), u = q >> os, t = t0 + tt;
    float g = 0.0f, h = 0.0f;
    for (int b = 0; b < os; ++b)
      if ((o >> b) & 1) g += par[t * os + b];
    for (int b = 0; b < is; ++b)
      if ((u >> b) & 1) h += sys[t * is + b];
    tab[tt * stride + q] = g + h;
  }
}

// The forward (dir 0, warp 0) or backward (dir 1, warp 1) recursion of one MAP pass, with
// warp 2 + dir filling the next block's branch metrics: alpha[t][s], the metrics before
// step t, or beta[t][s], those after it.  P branches per state.
template <int ALG, int SPL, int P>
__device__ __forceinline__ void recurse(const TurboDeviceConstituent& k, const float* par, const float* sys, float* store,
                                        int dir, MapShared& sh) {
  const int S = k.state_count, os = k.output_size, Q = P << os, T = k.length + k.tail;
  const int lane = threadIdx.x & 31, C = block_steps(k), blocks = (T + C - 1) / C;
  const bool walker = (threadIdx.x >> 5) < 2;
  auto block_of = [&](int i) { return dir ? blocks - 1 - i : i; };
  auto fill = [&](int i) {
    const int t0 = block_of(i) * C;
    fill_gammas(k, par, sys, t0, min(C, T - t0), sh.gam[dir][i & 1], threadIdx.x & 31, 32, Q);
  };
  if (!walker) {
    fill(0);
    for (int i = 0; i < blocks; ++i) {
      pair_sync(1 + dir);  // table i is there, table i - 1 is free
      if (i + 1 < blocks) fill(i + 1);
    }
    return;
  }
  // the branches of each state: into it (forward) or out of it (backward), in the
  // reference's order
  int src[SPL][P], type[SPL][P];
  // The metrics before their normalisation, and its maximum: v - m travels as v and m, so
  // that a step's shuffles need not wait for the maximum.
  float v[SPL], m = 0.0f;
  bool mine[SPL];
#pragma unroll
  for (int s = 0; s < SPL; ++s) {
    const int st = lane + 32 * s;
    mine[s] = st < S;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      src[s][p] = st;
      type[s][p] = 0;
      if (st < S) {
        if (dir == 0) {
          const uint32_t e = k.pred[st * P + p];
          src[s][p] = int(e & 0xffu);
          type[s][p] = (int((e >> 8) & 0xffu) << os) + int(e >> 16);
        } else {
          src[s][p] = int(k.next_state[st * P + p]);
          type[s][p] = (p << os) + int(k.output[st * P + p]);
        }
      }
    }
    const bool known = dir == 0 || k.termination == 0;  // the trellis starts (ends) in state 0
    v[s] = !mine[s] || (known && st != 0) ? kNegInf : 0.0f;
    if (mine[s]) store[int64_t(dir ? T - 1 : 0) * S + st] = v[s];
  }
  for (int i = 0; i < blocks; ++i) {
    pair_sync(1 + dir);
    const int t0 = block_of(i) * C, n = min(C, T - t0), by = dir ? -1 : 1;
    // the last forward step and the first one backward lead out of the frame
    const int from = dir ? n - 1 : 0, steps = (dir ? t0 == 0 : t0 + n == T) ? n - 1 : n;
    const float* tab = sh.gam[dir][i & 1] + from * Q;
    float* out = store + int64_t(t0 + from + by) * S + lane;
    for (int q = 0; q < steps; ++q, tab += by * Q, out += by * S) {
      float next[SPL];
#pragma unroll
      for (int s = 0; s < SPL; ++s) {
        float x[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
          float a = __shfl_sync(0xffffffffu, v[0], src[s][p] & 31);
          if (SPL > 1) {
            const float hi = __shfl_sync(0xffffffffu, v[SPL - 1], src[s][p] & 31);
            a = src[s][p] & 32 ? hi : a;
          }
          x[p] = (a - m) + tab[type[s][p]];
        }
        if (ALG == kExact) {
          float mx = kNegInf, acc = 0.0f;
#pragma unroll
          for (int p = 0; p < P; ++p) mx = fmaxf(x[p], mx);
#pragma unroll
          for (int p = 0; p < P; ++p) acc = eprior(x[p], mx) + acc;
          next[s] = logf(acc) + mx;
        } else {
          next[s] = ALG == kApproximate ? fmaxf(kNegInf, x[0]) : x[0];
#pragma unroll
          for (int p = 1; p < P; ++p) next[s] = log_sum<ALG>(sh, next[s], x[p]);
        }
      }
#pragma unroll
      for (int s = 0; s < SPL; ++s) v[s] = mine[s] ? next[s] : kNegInf;
      m = warp_max(SPL > 1 ? fmaxf(v[0], v[SPL - 1]) : v[0]);
#pragma unroll
      for (int s = 0; s < SPL; ++s)
        if (mine[s]) out[32 * s] = v[s] - m;
    }
  }
}

// L of the branches in a set against the others, of the step whose branch metrics, forward
// and backward metrics are tab, a and be (`one`: whether branch (s, u), number i, is in the set).
template <int ALG, int P, class F>
__device__ __forceinline__ float branch_llr(const MapShared& sh, int S, const float* tab, const float* a, const float* be,
                                            F&& one) {
  auto each = [&](auto&& f) {
    for (int s = 0, i = 0; s < S; ++s) {
      const float as = a[s];
#pragma unroll
      for (int u = 0; u < P; ++u, ++i) {
        const uint32_t b = sh.branch[i];
        f(tab[b >> 8] + as + be[b & 0xffu], one(i, u));
      }
    }
  };
  float mx[2] = {kNegInf, kNegInf};
  if (ALG == kExact) {
    each([&](float d, bool in) {
      if (in) mx[1] = fmaxf(d, mx[1]);
      else mx[0] = fmaxf(d, mx[0]);
    });
    float m0 = 0.0f, m1 = 0.0f;
    each([&](float d, bool in) {
      if (in) m1 = eprior(d, mx[1]) + m1;
      else m0 = eprior(d, mx[0]) + m0;
    });
    return (logf(m1) + mx[1]) - (logf(m0) + mx[0]);
  }
  each([&](float d, bool in) {
    if (in) mx[1] = log_sum<ALG>(sh, mx[1], d);
    else mx[0] = log_sum<ALG>(sh, mx[0], d);
  });
  return mx[1] - mx[0];
}

// One MAP pass of constituent k by the CTA: map_pass, its recursions and outputs spread over
// the threads.
template <int ALG, int SPL, int P>
__device__ __forceinline__ void map_pass_p(const TurboDeviceConstituent& k, const float* par, float* sys, float* parity_out,
                                           float sf, float* alpha, float* beta, float* app_out, MapShared& sh) {
  constexpr int kBits = P > 2 ? 2 : 1;  // input bits
  const int S = k.state_count, os = k.output_size, Q = P << os, T = k.length + k.tail;
  const int dir = (threadIdx.x >> 5) & 1;
  for (int i = threadIdx.x; i < S * P; i += kMapThreads)
    sh.branch[i] = k.next_state[i] | (((uint32_t(i % P) << os) + k.output[i]) << 8);
  recurse<ALG, SPL, P>(k, par, sys, dir ? beta : alpha, dir, sh);
  __syncthreads();
  // a thread per step; a step's branch metrics at an odd stride
  float* table = &sh.gam[0][0][0];
  const int stride = Q | 1, tile = min(kMapThreads, 4 * kTable / stride);
  for (int t0 = 0; t0 < T; t0 += tile) {
    const int n = min(tile, T - t0), t = t0 + int(threadIdx.x);
    fill_gammas(k, par, sys, t0, n, table, threadIdx.x, kMapThreads, stride);
    __syncthreads();
    if (int(threadIdx.x) < n) {
      const float* a = alpha + int64_t(t) * S;
      const float* be = beta + int64_t(t) * S;
      const float* tab = table + threadIdx.x * stride;
      if (parity_out)
        for (int j = 0; j < os; ++j) {
          const float r = branch_llr<ALG, P>(sh, S, tab, a, be, [&](int i, int) { return (k.output[i] >> j) & 1; });
          parity_out[t * os + j] = sf * (r - par[t * os + j]);
        }
#pragma unroll
      for (int j = 0; j < kBits; ++j) {
        const float lin = branch_llr<ALG, P>(sh, S, tab, a, be, [&](int, int u) { return (u >> j) & 1; });
        const int idx = t * kBits + j;
        if (app_out && t < k.length) app_out[idx] = sf * lin;
        sys[idx] = sf * (lin - sys[idx]);
      }
    }
    __syncthreads();
  }
}

template <int ALG, int SPL>
__device__ __noinline__ void map_pass_cta(const TurboDeviceConstituent& k, const float* par, float* sys, float* parity_out,
                                          float sf, float* alpha, float* beta, float* app_out, MapShared& sh) {
  if (k.input_count == 2) map_pass_p<ALG, SPL, 2>(k, par, sys, parity_out, sf, alpha, beta, app_out, sh);
  else map_pass_p<ALG, SPL, 4>(k, par, sys, parity_out, sf, alpha, beta, app_out, sh);
}

#define FECL_EACH(k, n) for (int k = threadIdx.x; k < (n); k += kMapThreads)

// The exchange steps of serial_transfer, parallel_transfer, custom_transfer and aposteriori:
// an interleaver's indices are distinct here, so within one constituent the elements are
// independent, and the constituents follow one another.
__device__ void add_interleaved(const TurboDeviceConstituent& q, const float* ext, float* syst) {
  FECL_EACH(k, q.msg_size) syst[q.perm[k]] += ext[k];
  __syncthreads();
}

__device__ void serial_transfer_cta(const TurboDeviceCode& c, Frame& fr, int i) {
  float* syst = fr.pout;
  FECL_EACH(k, c.msg) syst[k] = fr.pin[k];
  __syncthreads();
  const float* tail = fr.pin + c.msg;
  float* ext = fr.ext;
  float* slot = nullptr;
  for (int j = 0; j < c.n; ++j) {
    if (j == i) {
      slot = ext;
      FECL_EACH(k, c.c[i].syst_tail_size) ext[c.c[i].msg_size + k] = tail[k];
    } else {
      add_interleaved(c.c[j], ext, syst);
    }
    ext += c.c[j].syst_size;
    tail += c.c[j].syst_tail_size;
  }
  FECL_EACH(k, c.c[i].msg_size) slot[k] = syst[c.c[i].perm[k]];
  __syncthreads();
}

__device__ void parallel_transfer_cta(const TurboDeviceCode& c, Frame& fr) {
  float* ext = fr.ext;
  float* tmp = fr.extb;
  const float* tail = fr.pin + c.msg;
  float* syst = fr.pout;
  FECL_EACH(k, c.msg) syst[k] = 0.0f;
  __syncthreads();
  for (int j = 0; j < c.n; ++j) {
    const TurboDeviceConstituent& q = c.c[j];
    FECL_EACH(k, q.msg_size) {
      const float e = ext[k], s = syst[q.perm[k]];
      tmp[k] = e;
      ext[k] = s;
      syst[q.perm[k]] = s + e;
    }
    FECL_EACH(k, q.syst_tail_size) ext[q.msg_size + k] = tail[k];
    __syncthreads();
    ext += q.syst_size;
    tmp += q.msg_size;
    tail += q.syst_tail_size;
  }
  FECL_EACH(k, c.msg) syst[k] = fr.pin[k];
  __syncthreads();
  for (int j = c.n - 1; j >= 0; --j) {
    const TurboDeviceConstituent& q = c.c[j];
    ext -= q.syst_size;
    tmp -= q.msg_size;
    FECL_EACH(k, q.msg_size) {
      const float s = syst[q.perm[k]];
      ext[k] += s;
      syst[q.perm[k]] = s + tmp[k];
    }
    __syncthreads();
  }
}

__device__ void custom_transfer_cta(const TurboDeviceCode& c, Frame& fr, int a) {
  const int i = c.act_con[a], t_hi = c.act_tptr[a + 1];
  int at = c.act_tptr[a];
  float* syst = fr.pout;
  FECL_EACH(k, c.msg) syst[k] = fr.pin[k];
  __syncthreads();
  float* ext = fr.ext;
  float* tmp = fr.extb;
  const float* tail = fr.pin + c.msg;
  for (int j = 0; j < i; ++j) {
    if (take(c.transfer, at, t_hi, j)) add_interleaved(c.c[j], ext, syst);
    ext += c.c[j].syst_size;
    tmp += c.c[j].syst_size;
    tail += c.c[j].syst_tail_size;
  }
  FECL_EACH(k, c.c[i].syst_tail_size) ext[c.c[i].msg_size + k] = tail[k];
  ext += c.c[i].syst_size;
  for (int j = i + 1; j < c.n; ++j) {
    if (take(c.transfer, at, t_hi, j)) add_interleaved(c.c[j], ext, syst);
    else if (at >= t_hi) break;
    ext += c.c[j].syst_size;
  }
  FECL_EACH(k, c.c[i].msg_size) tmp[k] = syst[c.c[i].perm[k]];
  __syncthreads();
}

__device__ void aposteriori_cta(const TurboDeviceCode& c, Frame& fr) {
  const float* ext = fr.ext;
  float* tail = fr.pout + c.msg;
  for (int j = 0; j < c.n; ++j) {
    const TurboDeviceConstituent& q = c.c[j];
    FECL_EACH(k, q.syst_tail_size) tail[k] += ext[q.msg_size + k];
    add_interleaved(q, ext, fr.pout);
    ext += q.syst_size;
    tail += q.syst_tail_size;
  }
}

__device__ bool crc_passes_cta(const TurboDeviceCode& c, Frame& fr, const uint32_t* crc, MapShared& sh) {
  FECL_EACH(k, c.msg) fr.pout[k] = fr.pin[k];
  __syncthreads();
  aposteriori_cta(c, fr);
  uint32_t syn = 0;
  FECL_EACH(k, c.msg) if (fr.pout[k] > 0.0f) syn ^= __ldg(crc + k);
  syn = __reduce_xor_sync(0xffffffffu, syn);
  if ((threadIdx.x & 31) == 0) sh.part[threadIdx.x >> 5] = syn;
  __syncthreads();
  syn = sh.part[0] ^ sh.part[1] ^ sh.part[2] ^ sh.part[3];
  __syncthreads();
  return syn == 0;
}

// turbo_generic_f32 with a CTA per frame, for frames [f0, f0 + gridDim.x); alpha holds the
// slices' forward and backward metrics.
template <int ALG, int SPL>
__global__ void __launch_bounds__(kMapThreads) turbo_generic_cta(const __grid_constant__ TurboDeviceCode c,
                                                                 const __grid_constant__ TurboRun p, int64_t f0) {
  __shared__ MapShared sh;
  const int64_t f = f0 + blockIdx.x;
  Frame fr;
  fr.pin = p.parity_in + f * c.parity;
  fr.pout = p.parity_buf + f * c.parity;
  fr.ext = p.ext + f * c.state;
  fr.extb = p.ext_buf + f * c.state;
  const int64_t steps = int64_t(c.max_steps) * c.max_states;
  fr.alpha = p.alpha + blockIdx.x * 2 * steps;
  float* beta = fr.alpha + steps;
  if (threadIdx.x < 8) sh.pairs[threadIdx.x] = c_pairs.v[threadIdx.x];

  FECL_EACH(k, c.parity) {
    float x = load_llr(p.llr, p.llr_dtype, f * c.parity + k);
    if (p.syst_in && k < c.syst) x += load_llr(p.syst_in, p.llr_dtype, f * c.syst + k);
    fr.pin[k] = x;
    fr.pout[k] = 0.0f;
  }
  FECL_EACH(k, c.state) fr.ext[k] = p.state_in ? load_llr(p.state_in, p.llr_dtype, f * c.state + k) : 0.0f;
  __syncthreads();

  const bool want_parity = p.soft && p.parity_out;
  int ran = c.iterations;
  for (int i = 0; i < c.iterations; ++i) {
    if (c.scheduling == 2) {
      for (int st = 0; st < c.n_stages; ++st) {
        FECL_EACH(k, c.state) fr.extb[k] = fr.ext[k];
        __syncthreads();
        for (int a = c.stage_ptr[st]; a < c.stage_ptr[st + 1]; ++a) custom_transfer_cta(c, fr, a);
        float* t = fr.ext;
        fr.ext = fr.extb;
        fr.extb = t;
        // custom_activation
        const int hi = c.stage_ptr[st + 1];
        int at = c.stage_ptr[st];
        const float* par = fr.pin + c.syst;
        float* ext = fr.ext;
        for (int j = 0; j < c.n; ++j) {
          if (take(c.act_con, at, hi, j))
            map_pass_cta<ALG, SPL>(c.c[j], par, ext, nullptr, c.sf[j * c.iterations + i], fr.alpha, beta, nullptr, sh);
          else if (at >= hi) break;
          ext += c.c[j].syst_size;
          par += c.c[j].parity_size;
        }
      }
    } else {
      if (c.scheduling == 1) parallel_transfer_cta(c, fr);
      const float* par = fr.pin + c.syst;
      float* pout = fr.pout + c.syst;
      float* ext = fr.ext;
      for (int j = 0; j < c.n; ++j) {
        if (c.scheduling == 0) serial_transfer_cta(c, fr, j);
        const float sf = p.soft ? 1.0f : c.sf[j * c.iterations + i];
        const bool last = (i == c.iterations - 1);
        map_pass_cta<ALG, SPL>(c.c[j], par, ext, (want_parity && last) ? pout : nullptr, sf, fr.alpha, beta, nullptr, sh);
        ext += c.c[j].syst_size;
        par += c.c[j].parity_size;
        pout += c.c[j].parity_size;
      }
    }
    if (!p.soft && p.crc && i + 1 < c.iterations && crc_passes_cta(c, fr, p.crc, sh)) {
      ran = i + 1;
      break;
    }
  }

  FECL_EACH(k, p.soft ? c.syst : c.msg) fr.pout[k] = p.soft ? 0.0f : fr.pin[k];
  __syncthreads();
  aposteriori_cta(c, fr);
  if (!p.soft) {
    FECL_EACH(k, c.msg) p.hard[f * c.msg + k] = uint8_t(fr.pout[k] > 0.0f);
  } else {
    if (p.syst_out) FECL_EACH(k, c.syst) store_llr(p.syst_out, p.out_dtype, f * c.syst + k, fr.pout[k]);
    if (p.parity_out) FECL_EACH(k, c.parity) store_llr(p.parity_out, p.out_dtype, f * c.parity + k, fr.pout[k]);
    if (p.state_out) FECL_EACH(k, c.state) store_llr(p.state_out, p.out_dtype, f * c.state + k, fr.ext[k]);
    if (p.msg_out) FECL_EACH(k, c.msg) store_llr(p.msg_out, p.out_dtype, f * c.msg + k, fr.pin[k] + fr.pout[k]);
  }
  if (p.iters && threadIdx.x == 0) p.iters[f] = ran;
}

// conv_map_f32 with a CTA per frame, for frames [f0, f0 + gridDim.x).
template <int ALG, int SPL>
__global__ void __launch_bounds__(kMapThreads) conv_map_cta(const __grid_constant__ TurboDeviceConstituent k,
                                                            const __grid_constant__ ConvMapRun r, int64_t f0) {
  __shared__ MapShared sh;
  const int64_t f = f0 + blockIdx.x;
  const int P = k.parity_size, Sy = k.syst_size, M = k.msg_size;
  const int64_t steps = int64_t(k.length + k.tail) * k.state_count;
  float* par = r.par + f * P;
  float* sys = r.sys + f * Sy;
  float* pout = r.parity_out ? r.pout + f * P : nullptr;
  float* app = r.app + f * M;
  float* alpha = r.alpha + blockIdx.x * 2 * steps;
  if (threadIdx.x < 8) sh.pairs[threadIdx.x] = c_pairs.v[threadIdx.x];
  FECL_EACH(i, P) par[i] = load_llr(r.llr, r.llr_dtype, f * P + i);
  FECL_EACH(i, Sy) sys[i] = r.syst_in ? load_llr(r.syst_in, r.llr_dtype, f * Sy + i) : 0.0f;
  __syncthreads();
  map_pass_cta<ALG, SPL>(k, par, sys, pout, r.sf, alpha, alpha + steps, app, sh);
  if (r.msg_out) FECL_EACH(i, M) store_llr(r.msg_out, r.out_dtype, f * M + i, app[i]);
  if (r.syst_out) FECL_EACH(i, Sy) store_llr(r.syst_out, r.out_dtype, f * Sy + i, sys[i]);
  if (r.parity_out) FECL_EACH(i, P) store_llr(r.parity_out, r.out_dtype, f * P + i, pout[i]);
}

#undef FECL_EACH

// The convolutional codec's soDecode (Convolutional::soDecodeBlocks ->
// MapDecoderImpl::soDecodeBlock, src/detail/MapDecoder/MapDecoderImpl.cpp:56-78,
// :174-235): one MAP pass over the trellis per frame, one thread per frame.
template <int ALG>
__global__ void __launch_bounds__(64) conv_map_f32(TurboDeviceConstituent k, ConvMapRun r) {
  const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= r.nframes) return;
  const int P = k.parity_size, Sy = k.syst_size, M = k.msg_size;
  const int T = k.length + k.tail;
  float* par = r.par + f * P;
  float* sys = r.sys + f * Sy;
  float* pout = r.parity_out ? r.pout + f * P : nullptr;
  float* app = r.app + f * M;
  float* alpha = r.alpha + f * int64_t(T) * k.state_count;
  for (int i = 0; i < P; ++i) par[i] = load_llr(r.llr, r.llr_dtype, f * P + i);
  for (int i = 0; i < Sy; ++i) sys[i] = r.syst_in ? load_llr(r.syst_in, r.llr_dtype, f * Sy + i) : 0.0f;
  map_pass<ALG>(k, par, sys, pout, r.sf, alpha, app);
  if (r.msg_out)
    for (int i = 0; i < M; ++i) store_llr(r.msg_out, r.out_dtype, f * M + i, app[i]);
  if (r.syst_out)
    for (int i = 0; i < Sy; ++i) store_llr(r.syst_out, r.out_dtype, f * Sy + i, sys[i]);
  if (r.parity_out)
    for (int i = 0; i < P; ++i) store_llr(r.parity_out, r.out_dtype, f * P + i, pout[i]);
}

}  // namespace

cudaError_t turbo_generic_init() {
  static std::atomic<unsigned long long> done{0};
  return once_per_device(done, [] {
    const LinearLut l = make_linear_lut();
    const LinearPairs t = make_linear_pairs();
    const cudaError_t e = cudaMemcpyToSymbol(c_pairs, &t, sizeof(t));
    return e != cudaSuccess ? e : cudaMemcpyToSymbol(c_lut, &l, sizeof(l));
  });
}

// Frames that a CTA-per-frame launch of `nframes` holds the metrics of at once, `steps` bytes forward
// and as many backward each: all of them up to 4096, but half the batch where they take more
// than 4 GiB, so that a batch of long frames that fits with its forward metrics alone, as a
// thread per frame needs them, still fits.  4 GiB hold 167 frames of 50000 steps of 64 states: halves
// that leave SMs idle belong to longer frames only.
static int64_t slice_of(size_t steps, int64_t nframes) {
  constexpr size_t kRoom = size_t(4) << 30;
  const int64_t fit = int64_t(kRoom / (2 * steps));
  const int64_t half = (nframes + 1) / 2;
  int64_t n = half > fit ? half : fit;
  if (n > 4096) n = 4096;
  return n < nframes ? n : nframes;
}

// Microseconds of one MAP pass over `nframes` frames of k with a CTA and with a thread per frame, to
// within a quarter from 4 to 64 states, 3 to 130 steps and 1 to 50000 frames.  A CTA's warps
// share a frame's steps but pay for its start; threads all run at once, each through a chain of
// dependent steps.  So thousands of short frames go a thread each, in Linear (CTA and thread): 4 states, 3
// steps x 50000 frames 375 and 52 us, x 5000 59 and 46, x 1000 30 and 45; 8 states, 11 steps x
// 50000 461 and 345, x 20000 200 and 246; all trellises of more than 32 states a CTA (7 steps of 64 states x 50000
// 988 and 2262).
static double map_cta_us(const TurboDeviceConstituent& k, int algorithm, int64_t nframes) {
  const double T = double(k.length + k.tail), step = (k.state_count > 32 ? 1.25 : 0.27) * (algorithm == kExact ? 2.0 : 1.0);
  return 25.0 + 1e-3 * double(nframes) * ((k.state_count > 32 ? 11.0 : 6.3) + step * T);
}
static double map_thread_us(const TurboDeviceConstituent& k, int algorithm, int64_t nframes) {
  const double work = double(k.length + k.tail) * k.state_count;
  return 10.0 + work * (2.2 * (algorithm == kExact ? 1.25 : algorithm == kLinear ? 1.0 : 0.85) + 4e-5 * double(nframes));
}

static size_t steps_bytes(int64_t steps, int64_t states) { return size_t(steps) * size_t(states) * sizeof(float); }

// Room for either form, so that a batch never takes more than a larger one, whichever they run.
static size_t metrics_bytes(bool cta_ok, size_t steps, int64_t nframes) {
  const size_t thread = size_t(nframes) * steps, cta = size_t(slice_of(steps, nframes)) * 2 * steps;
  return cta_ok && cta > thread ? cta : thread;
}

size_t turbo_generic_metrics_bytes(const TurboDeviceCode& c, int64_t nframes) {
  const size_t steps = steps_bytes(c.max_steps, c.max_states);
  return metrics_bytes(c.cta_ok != 0, steps, nframes);
}

cudaError_t launch_turbo_generic(const TurboDeviceCode& c, const TurboRun& p, cudaStream_t s) {
  cudaError_t e0 = turbo_generic_init();
  if (e0 != cudaSuccess) return e0;
  if (p.nframes <= 0) return cudaSuccess;
  if (c.max_states > kMaxS) return cudaErrorInvalidValue;
  for (int j = 0; j < c.n; ++j)
    if (c.c[j].input_count > kMaxU || c.c[j].input_size > 4) return cudaErrorInvalidValue;
  double cta = 0.0, thread = 0.0;
  for (int j = 0; j < c.n; ++j) {
    cta += map_cta_us(c.c[j], c.algorithm, p.nframes);
    thread += map_thread_us(c.c[j], c.algorithm, p.nframes);
  }
  if (c.cta_ok && cta <= thread) {  // 2 or 4 inputs
    auto pick = [&](auto spl) -> void (*)(TurboDeviceCode, TurboRun, int64_t) {
      constexpr int kSpl = decltype(spl)::value;
      if (c.algorithm == kExact) return turbo_generic_cta<kExact, kSpl>;
      if (c.algorithm == kLinear) return turbo_generic_cta<kLinear, kSpl>;
      return turbo_generic_cta<kApproximate, kSpl>;
    };
    auto kern = c.max_states > 32 ? pick(std::integral_constant<int, 2>{}) : pick(std::integral_constant<int, 1>{});
    const int64_t slice = slice_of(steps_bytes(c.max_steps, c.max_states), p.nframes);
    for (int64_t f0 = 0; f0 < p.nframes; f0 += slice) {
      const int64_t n = p.nframes - f0 < slice ? p.nframes - f0 : slice;
      kern<<<unsigned(n), kMapThreads, 0, s>>>(c, p, f0);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const dim3 block(64), grid(unsigned((p.nframes + 63) / 64));
  switch (c.algorithm) {
    case kExact: turbo_generic_f32<kExact><<<grid, block, 0, s>>>(c, p); break;
    case kLinear: turbo_generic_f32<kLinear><<<grid, block, 0, s>>>(c, p); break;
    default: turbo_generic_f32<kApproximate><<<grid, block, 0, s>>>(c, p); break;
  }
  return cudaGetLastError();
}

// Whether conv_map_cta takes the trellis.
static bool map_by_cta(const TurboDeviceConstituent& k) { return k.pred && (k.input_count == 2 || k.input_count == 4); }

size_t conv_map_scratch_bytes(const TurboDeviceConstituent& k, int64_t nframes) {
  const size_t steps = steps_bytes(int64_t(k.length) + k.tail, k.state_count);
  return size_t(nframes) * size_t(2 * k.parity_size + k.syst_size + k.msg_size) * sizeof(float) +
         metrics_bytes(map_by_cta(k), steps, nframes) + 1024;
}

cudaError_t launch_conv_map(const TurboDeviceConstituent& k, ConvMapRun r, void* scratch, cudaStream_t s) {
  cudaError_t e = turbo_generic_init();
  if (e != cudaSuccess) return e;
  if (r.nframes <= 0) return cudaSuccess;
  if (k.state_count > kMaxS || k.input_count > kMaxU) return cudaErrorInvalidValue;
  float* q = static_cast<float*>(scratch);
  r.par = q;
  q += r.nframes * k.parity_size;
  r.pout = q;
  q += r.nframes * k.parity_size;
  r.sys = q;
  q += r.nframes * k.syst_size;
  r.app = q;
  q += r.nframes * k.msg_size;
  r.alpha = q;
  if (map_by_cta(k) && map_cta_us(k, r.algorithm, r.nframes) <= map_thread_us(k, r.algorithm, r.nframes)) {
    auto pick = [&](auto spl) -> void (*)(TurboDeviceConstituent, ConvMapRun, int64_t) {
      constexpr int kSpl = decltype(spl)::value;
      if (r.algorithm == kExact) return conv_map_cta<kExact, kSpl>;
      if (r.algorithm == kLinear) return conv_map_cta<kLinear, kSpl>;
      return conv_map_cta<kApproximate, kSpl>;
    };
    auto kern = k.state_count > 32 ? pick(std::integral_constant<int, 2>{}) : pick(std::integral_constant<int, 1>{});
    const int64_t slice = slice_of(steps_bytes(int64_t(k.length) + k.tail, k.state_count), r.nframes);
    for (int64_t f0 = 0; f0 < r.nframes; f0 += slice) {
      const int64_t n = r.nframes - f0 < slice ? r.nframes - f0 : slice;
      kern<<<unsigned(n), kMapThreads, 0, s>>>(k, r, f0);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const unsigned blocks = unsigned((r.nframes + 63) / 64);
  switch (r.algorithm) {
    case kExact: conv_map_f32<kExact><<<blocks, 64, 0, s>>>(k, r); break;
    case kLinear: conv_map_f32<kLinear><<<blocks, 64, 0, s>>>(k, r); break;
    default: conv_map_f32<kApproximate><<<blocks, 64, 0, s>>>(k, r); break;
  }
  return cudaGetLastError();
}

}  // namespace fecl
