// Windowed turbo decoder for two 8-state rate-1/2 constituents with Tail
// termination (the LTE code of 3GPP TS 36.212 and every code of that shape),
// serial scheduling, hard-decision decode, FP32 metrics.
//
// What it computes is the reference's full-frame BCJR (MapDecoderImpl,
// src/detail/MapDecoder/MapDecoderImpl.cpp:80-235) inside the serial turbo loop
// (TurboDecoderImpl::decodeBlock, src/detail/TurboDecoder/TurboDecoderImpl.cpp:31-72);
// how it computes it is B200-shaped:
//
//   One CTA of 2 * SEGS threads decodes one frame for all iterations.  The frame's
//   two exchange arrays live in shared memory by natural bit index (LteMap::pos):
//     X[k] = Ls[k] + e0[k]          (a-priori of constituent 1 before interleaving;
//                                    also the partial a-posteriori sum)
//     Y[k] = e1 at natural index k  (constituent 1 writes e1(t) to Y[pi(t)])
//   so constituent 0 reads Ls + Y contiguously and constituent 1 gathers X[pi(t)].
//
//   Per half-iteration:
//   A. SEGS forward and SEGS backward segments run concurrently (one thread each).
//      A segment starts from metrics obtained by a training run of G steps from a
//      flat start, walks its steps and leaves metric checkpoints every 8 steps in
//      global memory (L2) plus its end metrics in shared memory.
//   A2. Verification.  Segment 0 (forward) and the last segment (backward) start
//      from the exact trellis termination.  The training start of segment w is
//      accepted when it matches, within FP32 rounding (close8), the end metrics
//      that segment w-1 computed from its own accepted start; otherwise segment w
//      is walked again from that end, until its metrics reproduce a checkpoint of
//      the earlier walk.  Rounds repeat until every boundary is accepted, so every
//      checkpoint equals the full-frame recursion up to rounding.  (Max-log and
//      log-MAP forget their start exponentially fast; training merely makes
//      fix-ups rare.)
//   B. Every 8-step block is then independent: a thread reloads the forward
//      checkpoint at the block start and the backward checkpoint at its end,
//      recomputes the 8 forward vectors in registers and walks backward emitting
//      the extrinsic values, scaled, minus the a-priori (MapDecoderImpl.cpp:203-212).
//
// The recursions subtract the largest state metric once per 8-step chunk (at every
// checkpoint) rather than after every step as the reference does: the subtraction
// cancels in every difference the decoder takes, so this changes FP32 rounding only,
// and it removes the eight-way maximum and the subtractions from seven steps of
// eight.  Global loads of the next chunk are issued one chunk ahead.
//
// Inputs are first converted into an FP32 scratch layout in which the walkers of a warp
// read neighbouring 16-byte pieces (LteMap).
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.hpp"

namespace fecl {
namespace {

constexpr int kExact = 0, kLinear = 1, kApproximate = 2;
constexpr int kBlk = 8;  // checkpoint spacing / APP block length
constexpr float kNegInf = -INFINITY;
// Boundary acceptance: |x - y| <= abs + rel * max(|x|, |y|).  Two walks that have
// forgotten their starts differ by the rounding of the steps since, which grows with
// the metrics' magnitude (strong a-priori values late in a decode).  An accepted
// difference reaches the extrinsic values at most doubled, so soDecode, whose soft
// outputs must stay within 1e-4 relative of the reference, accepts only differences
// two orders of magnitude below that; decode, which outputs hard decisions, accepts
// 1e-3 (+ 1e-5 relative), which saves fix-up walks.
struct Tol {
  float abs, rel;
};
constexpr Tol kDecodeTol = {1e-3f, 1e-5f};
constexpr Tol kSoftTol = {1e-6f, 1e-6f};
constexpr int kDefaultSegs = 64;

__constant__ LinearPairs c_lut;
__shared__ float2 s_lut[8];

// The LTE RSC, Trellis({4}, {{015}}, {013}) (src/Trellis.cpp:76-143): with state bits
// s0 s1 s2, the feedback bit is u ^ s0 ^ s1, the next state shifts it in at the top
// and the parity output is u ^ s1 ^ s2.  Compile-time tables keep every metric in
// registers.
__host__ __device__ constexpr int lte_next(int s, int u) { return (s >> 1) | (((u ^ s ^ (s >> 1)) & 1) << 2); }
__host__ __device__ constexpr int lte_out(int s, int u) { return (u ^ (s >> 1) ^ (s >> 2)) & 1; }

template <int ALG>
__device__ __forceinline__ float lsum(float a, float b) {
  return ALG == kApproximate ? fmaxf(a, b) : linear_sum(s_lut, a, b);
}

// max(a, b, c) in one instruction (the three-input form of max.f32, sm_100): the same
// value as fmaxf(fmaxf(a, b), c), a maximum being exact.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// v[s] -= max(v), with the subtraction as four packed f32x2 adds of -m (x - m is
// x + (-m) exactly).
__device__ __forceinline__ void normalize8(float v[8]) {
  const float m = fmax3(fmax3(v[0], v[1], v[2]), fmax3(v[3], v[4], v[5]), fmaxf(v[6], v[7]));
  const float2 nm = make_float2(-m, -m);
#pragma unroll
  for (int s = 0; s < 8; s += 2) {
    const float2 r = __fadd2_rn(make_float2(v[s], v[s + 1]), nm);
    v[s] = r.x;
    v[s + 1] = r.y;
  }
}

// Two-term log-sum in the Exact (LogSum) form: max, then exp-sum, then log.  The
// exponentials take arguments <= 0 and the logarithm arguments in [1, 16], where the
// hardware approximations (__expf, __logf) are within about 2^-22 relative and 2^-21
// absolute: every metric and extrinsic value moves by less than 1e-6 absolute per
// step, far inside the soft-output rule (1e-4 relative, 1e-4 absolute below 1), at a
// few instructions each instead of the accurate functions' range reductions.
__device__ __forceinline__ float esum2(float x0, float x1) {
  const float m = fmaxf(x0, x1);
  const float a = (x0 == m) ? 1.0f : __expf(x0 - m);
  const float b = (x1 == m) ? 1.0f : __expf(x1 - m);
  return __logf(a + b) + m;
}

struct Gam {
  float g[4];  // index (u << 1) | p : 0, Lp, La, La + Lp
  __device__ __forceinline__ void set(float la, float lp) {
    g[0] = 0.0f;
    g[1] = lp;
    g[2] = la;
    g[3] = lp + la;
  }
  // x + gamma(s, u).  In max-log the branch with no 1 bits adds nothing: x + 0 is x for
  // every metric but -0, and a -0 metric (x == 0) only ever meets +0 in a maximum or a
  // difference, which treat both alike; the other algorithms keep the reference's adds.
  template <int ALG>
  __device__ __forceinline__ float plus(float x, int s, int u) const {
    const int i = (u << 1) | lte_out(s, u);
    if (ALG == kApproximate && i == 0) return x;
    return x + g[i];
  }
};

// The log-MAP recursions keep the reference's normalisation after every step (max-log
// normalises once per chunk, see above): their table and exp/log corrections are not
// translation-invariant in FP32, so this keeps their rounding that of the reference.
template <int ALG>
__device__ __forceinline__ void normalize_step(float v[8]) {
  if constexpr (ALG != kApproximate) {
    float m = kNegInf;
#pragma unroll
    for (int s = 0; s < 8; ++s) m = fmaxf(v[s], m);
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = v[s] - m;
  }
}

// alpha_{t+1} from alpha_t (MapDecoderImpl.cpp:117-139, :237-274); normalised here only
// by the log-MAP algorithms.
template <int ALG>
__device__ __forceinline__ void fwd_step(float a[8], const Gam& g) {
  float c0[8], c1[8];
  bool first[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) first[s] = true;
#pragma unroll
  for (int s = 0; s < 8; ++s)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int d = lte_next(s, u);
      const float v = g.plus<ALG>(a[s], s, u);
      if (first[d]) {
        c0[d] = v;
        first[d] = false;
      } else {
        c1[d] = v;
      }
    }
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    if (ALG == kExact) a[s] = esum2(c0[s], c1[s]);
    else if (ALG == kApproximate) a[s] = fmaxf(c0[s], c1[s]);
    // Linear: the reference's accumulation starts from -inf, and lsum(-inf, c) is c
    // (the table gives 0 beyond 3.5), so it is left out; only a -0 metric would come
    // out as +0, which every later maximum and difference treats alike
    else a[s] = lsum<ALG>(c0[s], c1[s]);
  }
  normalize_step<ALG>(a);
}

// beta_t from beta_{t+1} (MapDecoderImpl.cpp:141-172, :276-329); normalised here only by
// the log-MAP algorithms.
template <int ALG>
__device__ __forceinline__ void bwd_step(float b[8], const Gam& g) {
  float n[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const float x0 = g.plus<ALG>(b[lte_next(s, 0)], s, 0);
    const float x1 = g.plus<ALG>(b[lte_next(s, 1)], s, 1);
    if (ALG == kExact) n[s] = esum2(x0, x1);
    else if (ALG == kApproximate) n[s] = fmaxf(x0, x1);
    else n[s] = lsum<ALG>(x0, x1);  // as in fwd_step
  }
#pragma unroll
  for (int s = 0; s < 8; ++s) b[s] = n[s];
  normalize_step<ALG>(b);
}

// Extrinsic value of one step, L(u) - La (msgUpdateImpl, MapDecoderImpl.cpp:331-376).
// Max-log: L(u=1) = La + max_s(a[s] + b[next(s,1)] + p(s,1) Lp) and L(u=0) =
// max_s(a[s] + b[next(s,0)] + p(s,0) Lp), so the a-priori value cancels and each
// maximum splits by parity bit: the states with p(s,0) = 1 are 2..5 (and with
// p(s,1) = 1 the others), so Lp is added once per maximum instead of once per state.
template <int ALG>
__device__ __forceinline__ float ext_step(const float a[8], const float b[8], const Gam& g) {
  if constexpr (ALG == kApproximate) {
    float w0[8], w1[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      w0[s] = a[s] + b[lte_next(s, 0)];
      w1[s] = a[s] + b[lte_next(s, 1)];
    }
    const float lp = g.g[1];
    // u = 0: parity 0 at s in {0,1,6,7}, parity 1 at {2,3,4,5}; u = 1 the reverse.
    const float m0p0 = fmax3(fmaxf(w0[0], w0[1]), w0[6], w0[7]);
    const float m0p1 = fmax3(fmaxf(w0[2], w0[3]), w0[4], w0[5]);
    const float m1p0 = fmax3(fmaxf(w1[2], w1[3]), w1[4], w1[5]);
    const float m1p1 = fmax3(fmaxf(w1[0], w1[1]), w1[6], w1[7]);
    const float m0 = fmaxf(m0p0, m0p1 + lp);
    const float m1 = fmaxf(m1p0, m1p1 + lp);
    return m1 - m0;
  } else {
    float d[16];
#pragma unroll
    for (int s = 0; s < 8; ++s)
#pragma unroll
      for (int u = 0; u < 2; ++u) d[s * 2 + u] = g.plus<ALG>(a[s], s, u) + b[lte_next(s, u)];
    float l;
    if (ALG == kExact) {
      float mx0 = kNegInf, mx1 = kNegInf;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        mx0 = fmaxf(d[s * 2], mx0);
        mx1 = fmaxf(d[s * 2 + 1], mx1);
      }
      float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        m0 = ((d[s * 2] == mx0) ? 1.0f : __expf(d[s * 2] - mx0)) + m0;
        m1 = ((d[s * 2 + 1] == mx1) ? 1.0f : __expf(d[s * 2 + 1] - mx1)) + m1;
      }
      l = (__logf(m1) + mx1) - (__logf(m0) + mx0);  // esum2's approximations
    } else {
      float m0 = kNegInf, m1 = kNegInf;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        m0 = lsum<ALG>(m0, d[s * 2]);
        m1 = lsum<ALG>(m1, d[s * 2 + 1]);
      }
      l = m1 - m0;
    }
    return l - g.g[2];
  }
}

// Parity extrinsic value of one step, L(p) - Lp (parityUpdate, MapDecoderImpl.cpp:
// 376-410), for soDecode's parity output.  Max-log: the branches with p = 1 are
// (s in 2..5, u = 0) and (s in {0,1,6,7}, u = 1); Lp cancels and La is added once per
// maximum.
template <int ALG>
__device__ __forceinline__ float par_step(const float a[8], const float b[8], const Gam& g) {
  if constexpr (ALG == kApproximate) {
    float w0[8], w1[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      w0[s] = a[s] + b[lte_next(s, 0)];
      w1[s] = a[s] + b[lte_next(s, 1)];
    }
    const float la = g.g[2];
    const float m0p0 = fmax3(fmaxf(w0[0], w0[1]), w0[6], w0[7]);
    const float m0p1 = fmax3(fmaxf(w0[2], w0[3]), w0[4], w0[5]);
    const float m1p0 = fmax3(fmaxf(w1[2], w1[3]), w1[4], w1[5]);
    const float m1p1 = fmax3(fmaxf(w1[0], w1[1]), w1[6], w1[7]);
    return fmaxf(m0p1, m1p1 + la) - fmaxf(m0p0, m1p0 + la);
  } else {
    float d[16];
#pragma unroll
    for (int s = 0; s < 8; ++s)
#pragma unroll
      for (int u = 0; u < 2; ++u) d[s * 2 + u] = g.plus<ALG>(a[s], s, u) + b[lte_next(s, u)];
    float l;
    if (ALG == kExact) {
      float mx0 = kNegInf, mx1 = kNegInf;
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (lte_out(s, u)) mx1 = fmaxf(d[s * 2 + u], mx1);
          else mx0 = fmaxf(d[s * 2 + u], mx0);
        }
      float m0 = 0.0f, m1 = 0.0f;
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float x = d[s * 2 + u];
          if (lte_out(s, u)) m1 = ((x == mx1) ? 1.0f : __expf(x - mx1)) + m1;
          else m0 = ((x == mx0) ? 1.0f : __expf(x - mx0)) + m0;
        }
      l = (__logf(m1) + mx1) - (__logf(m0) + mx0);  // esum2's approximations
    } else {
      float m0 = kNegInf, m1 = kNegInf;
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (lte_out(s, u)) m1 = lsum<ALG>(m1, d[s * 2 + u]);
          else m0 = lsum<ALG>(m0, d[s * 2 + u]);
        }
      l = m1 - m0;
    }
    return l - g.g[1];
  }
}

// Where a frame's values lie.  A frame is cut into S segments of Lc chunks of 8 steps; the
// walkers of a warp stand at the same chunk k of neighbouring segments w, so every staged
// array holds its chunks by k and then by w: chunk c = w Lc + k at slot k Sp + w, as two
// planes of 4 floats per slot.  A warp's load of one plane is then contiguous (with the
// chunks in time order it touched one line per lane, and the L1 pipe, at 73 % of its
// peak, bound the kernel).  The exchange arrays in shared memory are in time order with the
// halves of every other group of 4 chunks swapped: a chunk is two 16-byte accesses, which
// for an odd number of chunks per segment fall into distinct banks over the lanes, and
// interleaved positions (a QPP interleaver maps steps that differ by a multiple of 8 to
// positions that do) into 8 banks instead of 4.  One plane per step modulo 8 had no
// conflicts at all, but took 13 instructions more per chunk, and instructions bound the kernel.
struct LteMap {
  int Lc, S, Sp, slots, nblk;
  __device__ __forceinline__ int slot_of(int c) const { return (c % Lc) * Sp + c / Lc; }
  __device__ __forceinline__ static int pos(int t) { return t ^ ((t >> 3) & 4); }
};

struct Frame {
  LteMap m;
  const float* Ls;    // [2][slots][4] systematic L-values, then constituent 0's tail
  const float* Lp0;   // [2][slots][4] parity (with tail parity) of constituent 0
  const float* Lp1;   // [2][slots][4]
  const float* ts;    // [8]  tail systematic of constituent 0 (3) then 1 (3)
  const uint4* perm;  // [slots] byte offset of each step's interleaved element, 16 bits each
  float* cka;         // [2][slots][4] forward metrics before each chunk
  float* ckb;         // [2][slots][4] backward metrics before each chunk (chunk nblk: the end)
};

// A segment's boundary vectors: a forward segment's start (after training) is its
// first checkpoint and a backward segment's end its last, so those two stay in the
// checkpoint arrays (global memory); the other two are kept here.
template <int SEGS>
struct Shared {
  float bwd_start[8][SEGS];  // backward segment w's metrics at its end a1 after training
  float fwd_end[8][SEGS];    // forward segment w's metrics at a1
  uint32_t crc_part[2 * SEGS / 32];  // per-warp CRC syndromes
};

// The global loads of one 8-step chunk: the parity L-values and either the systematic
// L-values (constituent 0) or the 8 interleaved positions (constituent 1, in q0).
struct RawChunk {
  float4 p0, p1;  // parity
  uint4 q0, q1;   // systematic (as bits) or interleaved positions
};

__device__ __forceinline__ void load_raw(int j, int slot, const Frame& fr, RawChunk& r) {
  // plain loads: a small batch's CTAs stage their frames themselves
  const float4* Lp = reinterpret_cast<const float4*>(j == 0 ? fr.Lp0 : fr.Lp1) + slot;
  r.p0 = Lp[0];
  r.p1 = Lp[fr.m.slots];
  if (j == 0) {
    const uint4* q = reinterpret_cast<const uint4*>(fr.Ls) + slot;
    r.q0 = q[0];
    r.q1 = q[fr.m.slots];
  } else {
    r.q0 = fr.perm[slot];
  }
}

// Entry i of the 8 16-bit offsets of a chunk.
__device__ __forceinline__ uint32_t offset_of(const uint4& q, int i) {
  const uint32_t w = i < 2 ? q.x : i < 4 ? q.y : i < 6 ? q.z : q.w;
  return (i & 1) ? w >> 16 : w & 0xffffu;
}

// The two halves of chunk c in an exchange array (in 4-float units): steps 0 to 3 and 4 to 7.
__device__ __forceinline__ int half_of(int c, int h) { return 2 * c + (h ^ ((c >> 2) & 1)); }

// A chunk's a-priori and parity L-values.
struct Chunk {
  float la[kBlk];
  float lp[kBlk];
};

// The CTA's dynamic shared memory; the exchange arrays X and Y start at 0 and at Kp.
extern __shared__ __align__(16) float lte_smem[];

// The tail steps need no case of their own: constituent 0's tail bits follow the systematic
// values, with zeros in Y, and constituent 1's wait in X behind the message, where the
// offsets of its tail steps point (a select per step before: K=6144 x 1024 900 us, now 836;
// K=40 x 1 65.6, now 57.6; Linear soft K=1024 x 64 531, now 552).
__device__ __forceinline__ void resolve(int j, int c, int Kp, const RawChunk& r, Chunk& ch) {
  ch.lp[0] = r.p0.x; ch.lp[1] = r.p0.y; ch.lp[2] = r.p0.z; ch.lp[3] = r.p0.w;
  ch.lp[4] = r.p1.x; ch.lp[5] = r.p1.y; ch.lp[6] = r.p1.z; ch.lp[7] = r.p1.w;
  if (j == 0) {
    const float ls[kBlk] = {__uint_as_float(r.q0.x), __uint_as_float(r.q0.y), __uint_as_float(r.q0.z),
                            __uint_as_float(r.q0.w), __uint_as_float(r.q1.x), __uint_as_float(r.q1.y),
                            __uint_as_float(r.q1.z), __uint_as_float(r.q1.w)};
    const float4* y = reinterpret_cast<const float4*>(lte_smem + Kp);
    const float4 y0 = y[half_of(c, 0)], y1 = y[half_of(c, 1)];
    const float yv[kBlk] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
#pragma unroll
    for (int i = 0; i < kBlk; ++i) ch.la[i] = ls[i] + yv[i];
  } else {
#pragma unroll
    for (int i = 0; i < kBlk; ++i) ch.la[i] = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(lte_smem) + offset_of(r.q0, i));
  }
}

__device__ __forceinline__ void store_ck(float* ck, int slots, int slot, const float v[8]) {
  float4* q = reinterpret_cast<float4*>(ck) + slot;
  q[0] = make_float4(v[0], v[1], v[2], v[3]);
  q[slots] = make_float4(v[4], v[5], v[6], v[7]);
}

__device__ __forceinline__ void load_ck(const float* ck, int slots, int slot, float v[8]) {
  const float4* q = reinterpret_cast<const float4*>(ck) + slot;
  const float4 c0 = q[0], c1 = q[slots];
  v[0] = c0.x; v[1] = c0.y; v[2] = c0.z; v[3] = c0.w;
  v[4] = c1.x; v[5] = c1.y; v[6] = c1.z; v[7] = c1.w;
}

__device__ __forceinline__ bool close8(const float x[8], const float y[8], Tol t) {
  bool ok = true;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const float tol = t.abs + t.rel * fmaxf(fabsf(x[s]), fabsf(y[s]));
    ok = ok && ((x[s] == y[s]) || fabsf(x[s] - y[s]) <= tol);
  }
  return ok;
}

// One segment walk of constituent j, forward (fwd != 0) or backward, of segment w from the
// metrics v.  Training chunks outside the segment run first without checkpoints -- forward
// over the `lead` chunks before it, backward over those behind it, cut short at the frame's
// ends -- then the segment's own chunks run, leaving a checkpoint before each (and at T for
// the last backward segment).  The metrics at the segment's end go to vbound (forward), or
// those at its boundary after training (backward), [8][segs].  Walkers with a full training
// stand at the same chunk of their segments, those that start at the frame's end at the
// same chunk of the frame, so a warp's loads stay contiguous or equal.  Metrics are
// normalised at the end of every chunk, so every checkpoint and both boundary vectors
// have their largest state at 0.  The global loads of the next chunk are issued before a
// chunk runs.  A fix-up walk (`refine`) starts from a corrected boundary over checkpoints
// an earlier walk of the same segment left; it stops at the first checkpoint its metrics
// reproduce (close8): from there on the earlier walk is the same recursion, so its
// checkpoints and end stand.  Kept out of line so that Phase A and the fix-up rounds share
// one copy of the code.
template <int ALG>
__device__ __noinline__ void segment_walk(int fwd, int j, int w, int lead, float4 va, float4 vb, int bound, int segs,
                                          int K, int T, Frame fr, int Kp, bool refine, Tol tol) {
  // out of line, the address spaces are not known
  __builtin_assume(__isGlobal(fr.Ls) && __isGlobal(fr.Lp0) && __isGlobal(fr.Lp1));
  __builtin_assume(__isGlobal(fr.perm) && __isGlobal(fr.cka) && __isGlobal(fr.ckb));
  float* vbound = lte_smem + bound;
  float v[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
  const int Lc = fr.m.Lc, Sp = fr.m.Sp, slots = fr.m.slots, nblk = fr.m.nblk;
  const int turn = (Lc - 1) * Sp - 1;  // from a segment's last slot back to the next one's first
  const int c_own = w * Lc;
  if (fwd) {
    const int c_end = min(nblk, c_own + Lc);
    int c = max(0, c_own - lead), kk = c % Lc;
    int slot = kk * Sp + c / Lc;
    RawChunk nxt;
    load_raw(j, slot, fr, nxt);
    for (; c < c_end; ++c) {
      const int here = slot;
      const RawChunk cur = nxt;
      if (++kk == Lc) {
        kk = 0;
        slot -= turn;
      } else {
        slot += Sp;
      }
      if (c + 1 < c_end) load_raw(j, slot, fr, nxt);
      Chunk ch;
      resolve(j, c, Kp, cur, ch);
      if (c >= c_own) {
        if (refine && c > c_own) {
          float old[8];
          load_ck(fr.cka, slots, here, old);
          if (close8(v, old, tol)) return;
        }
        store_ck(fr.cka, slots, here, v);
      }
      const int n = min(kBlk, T - c * kBlk);
      if (n == kBlk) {  // every chunk but the frame's last, whose few steps run in a loop
#pragma unroll
        for (int i = 0; i < kBlk; ++i) {
          Gam g;
          g.set(ch.la[i], ch.lp[i]);
          fwd_step<ALG>(v, g);
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < n; ++i) {
          Gam g;
          g.set(ch.la[0], ch.lp[0]);
          fwd_step<ALG>(v, g);
#pragma unroll
          for (int q = 0; q + 1 < kBlk; ++q) {
            ch.la[q] = ch.la[q + 1];
            ch.lp[q] = ch.lp[q + 1];
          }
        }
      }
      normalize8(v);
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) vbound[s * segs + w] = v[s];
  } else {
    int c = min(nblk, c_own + Lc + lead) - 1, kk = c % Lc;
    int slot = kk * Sp + c / Lc;
    if (lead == 0 || w == fr.m.S - 1) {
#pragma unroll
      for (int s = 0; s < 8; ++s) vbound[s * segs + w] = v[s];
      if (w == fr.m.S - 1) store_ck(fr.ckb, slots, fr.m.slot_of(nblk), v);
    }
    RawChunk nxt;
    load_raw(j, slot, fr, nxt);
    for (; c >= c_own; --c) {
      const int here = slot;
      const RawChunk cur = nxt;
      if (--kk < 0) {
        kk = Lc - 1;
        slot += turn;
      } else {
        slot -= Sp;
      }
      if (c > c_own) load_raw(j, slot, fr, nxt);
      Chunk ch;
      resolve(j, c, Kp, cur, ch);
      const int hi = min(kBlk, T - c * kBlk);
      if (hi == kBlk) {  // as in the forward walk
#pragma unroll
        for (int i = kBlk - 1; i >= 0; --i) {
          Gam g;
          g.set(ch.la[i], ch.lp[i]);
          bwd_step<ALG>(v, g);
        }
      } else {
#pragma unroll 1
        for (int i = kBlk - 1; i >= 0; --i) {
          if (i < hi) {
            Gam g;
            g.set(ch.la[kBlk - 1], ch.lp[kBlk - 1]);
            bwd_step<ALG>(v, g);
          }
#pragma unroll
          for (int q = kBlk - 1; q > 0; --q) {
            ch.la[q] = ch.la[q - 1];
            ch.lp[q] = ch.lp[q - 1];
          }
        }
      }
      normalize8(v);
      // v now holds the metrics before chunk c
      if (c == c_own + Lc) {
#pragma unroll
        for (int s = 0; s < 8; ++s) vbound[s * segs + w] = v[s];
      }
      if (c < c_own + Lc) {
        if (refine) {
          float old[8];
          load_ck(fr.ckb, slots, here, old);
          if (close8(v, old, tol)) return;
        }
        store_ck(fr.ckb, slots, here, v);
      }
    }
  }
}

// Where soDecode's last iteration leaves its values: the constituent's extrinsic values
// of every trellis step (tail included) in its own order, and its parity extrinsic
// values (nullable) at element offset par0 of par, of type dtype.
struct SoftSink {
  float* ext = nullptr;  // [T]
  void* par = nullptr;
  int64_t par0 = 0;
  int32_t dtype = 1;
};

// Phase B for one 8-step block b of constituent j: reload the forward checkpoint at
// the block start and the backward one at its end, recompute the block's forward
// vectors in registers, walk backward emitting sf * extrinsic into out (X: Ls + e at
// t, Y: e at pi(t)).  FULL: all 8 steps are message steps (no per-step tests).  SOFT:
// soDecode's last iteration, which also records every step's extrinsic value (tail
// steps too) and parity extrinsic value in `sink`.
template <int ALG, bool FULL, bool SOFT>
__device__ __forceinline__ void ext_block(int j, int k, int w, int K, int T, const Frame& fr, int Kp, float sf, float* out, const SoftSink& sink) {
  const int b = w * fr.m.Lc + k, slot = k * fr.m.Sp + w, slots = fr.m.slots;
  const int after = k + 1 < fr.m.Lc ? slot + fr.m.Sp : w + 1;  // chunk b + 1
  const int t0 = b * kBlk;
  const int n = FULL ? kBlk : min(kBlk, T - t0);
  RawChunk raw;
  load_raw(j, slot, fr, raw);
  float al[kBlk][8];
  load_ck(fr.cka, slots, slot, al[0]);
  float be[8];
  load_ck(fr.ckb, slots, after, be);
  Chunk in;
  resolve(j, b, Kp, raw, in);
#pragma unroll
  for (int i = 1; i < kBlk; ++i) {
    if (FULL || i < n) {
#pragma unroll
      for (int s = 0; s < 8; ++s) al[i][s] = al[i - 1][s];
      Gam g;
      g.set(in.la[i - 1], in.lp[i - 1]);
      fwd_step<ALG>(al[i], g);
    }
  }
  const float ls[kBlk] = {__uint_as_float(raw.q0.x), __uint_as_float(raw.q0.y), __uint_as_float(raw.q0.z),
                          __uint_as_float(raw.q0.w), __uint_as_float(raw.q1.x), __uint_as_float(raw.q1.y),
                          __uint_as_float(raw.q1.z), __uint_as_float(raw.q1.w)};
  float x[kBlk] = {};
#pragma unroll
  for (int i = kBlk - 1; i >= 0; --i) {
    if (FULL || i < n) {
      Gam g;
      g.set(in.la[i], in.lp[i]);
      const float e = sf * ext_step<ALG>(al[i], be, g);
      if (FULL && j == 0) x[i] = ls[i] + e;
      else if (FULL || t0 + i < K) {
        if (j == 0) out[fr.m.pos(t0 + i)] = ls[i] + e;
        else *reinterpret_cast<float*>(reinterpret_cast<char*>(out) + offset_of(raw.q0, i)) = e;
      }
      if (SOFT && sink.ext) {
        sink.ext[t0 + i] = e;
        if (sink.par) store_llr(sink.par, sink.dtype, sink.par0 + t0 + i, par_step<ALG>(al[i], be, g));
      }
      if (i > 0) bwd_step<ALG>(be, g);
    }
  }
  if (FULL && j == 0) {
    float4* o = reinterpret_cast<float4*>(out);
    o[half_of(b, 0)] = make_float4(x[0], x[1], x[2], x[3]);
    o[half_of(b, 1)] = make_float4(x[4], x[5], x[6], x[7]);
  }
}

// The same block for the log-MAP algorithms, step by step: their steps are long (dozens of
// instructions per log-sum), and 8 of them unrolled three times over ran from the
// instruction cache's misses.  The forward vectors wait in local memory.
template <int ALG, bool SOFT>
__device__ __forceinline__ void ext_steps(int j, int k, int w, int K, int T, const Frame& fr, int Kp, float sf, float* out, const SoftSink& sink) {
  const int b = w * fr.m.Lc + k, slot = k * fr.m.Sp + w, slots = fr.m.slots;
  const int after = k + 1 < fr.m.Lc ? slot + fr.m.Sp : w + 1;  // chunk b + 1
  const int t0 = b * kBlk, n = min(kBlk, T - t0);
  RawChunk raw;
  load_raw(j, slot, fr, raw);
  float v[8], be[8];
  load_ck(fr.cka, slots, slot, v);
  load_ck(fr.ckb, slots, after, be);
  Chunk in;
  resolve(j, b, Kp, raw, in);
  float4 al[kBlk][2];
#pragma unroll 1
  for (int i = 0;; ++i) {
    al[i][0] = make_float4(v[0], v[1], v[2], v[3]);
    al[i][1] = make_float4(v[4], v[5], v[6], v[7]);
    if (i + 1 >= n) break;
    Gam g;
    g.set(in.la[i], in.lp[i]);
    fwd_step<ALG>(v, g);
  }
  const uint32_t q[kBlk] = {raw.q0.x, raw.q0.y, raw.q0.z, raw.q0.w, raw.q1.x, raw.q1.y, raw.q1.z, raw.q1.w};
#pragma unroll 1
  for (int i = n - 1; i >= 0; --i) {
    const float4 a0 = al[i][0], a1 = al[i][1];
    const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    Gam g;
    g.set(in.la[i], in.lp[i]);
    const float e = sf * ext_step<ALG>(a, be, g);
    if (t0 + i < K) {
      if (j == 0) out[fr.m.pos(t0 + i)] = __uint_as_float(q[i]) + e;
      else *reinterpret_cast<float*>(reinterpret_cast<char*>(out) + ((i & 1) ? q[i >> 1] >> 16 : q[i >> 1] & 0xffffu)) = e;
    }
    if (SOFT && sink.ext) {
      sink.ext[t0 + i] = e;
      if (sink.par) store_llr(sink.par, sink.dtype, sink.par0 + t0 + i, par_step<ALG>(a, be, g));
    }
    if (i > 0) bwd_step<ALG>(be, g);
  }
}

// Segment w and chunk k of block i in the order phase B takes the first n blocks: by k, and
// within a k by w, so that the lanes of a warp read neighbouring slots.
__device__ __forceinline__ void block_at(int i, int n, const LteMap& m, int& k, int& w) {
  const int rem = n - (m.S - 1) * m.Lc;  // blocks of the last segment; the others have Lc
  if (i < rem * m.S) {
    k = i / m.S;
    w = i - k * m.S;
  } else {
    const int q = (i - rem * m.S) / (m.S - 1);
    k = rem + q;
    w = i - rem * m.S - q * (m.S - 1);
  }
}

// One frame's geometry and buffers, as the decode loop below sees them.
struct LteJob {
  int32_t K = 0, Kp = 0, Tp = 0, train = 0, iterations = 0;
  LteMap map;
  const float* sf = nullptr;            // [2][iterations]
  const float* scratch = nullptr;       // staged L-values: Ls | Lp0 | Lp1 [8 slots] each | tail [8]
  const uint4* perm = nullptr;          // staged interleaved positions [slots]
  float* ck = nullptr;                  // checkpoints [2][8 slots]
  uint8_t* hard = nullptr;              // [K]
  int32_t* iters = nullptr;             // nullable
  unsigned long long* stats = nullptr;  // nullable
  const uint32_t* crc = nullptr;        // [K] x^(K-1-i) mod g: stop when the decisions' CRC checks (nullable)
  // Parallel scheduling: constituent 1 runs first and leaves its extrinsic values in
  // ynew, copied into Y once constituent 0, which reads the old ones, is done.
  int32_t parallel = 0;
  float* ynew = nullptr;  // [Kp]
  // soDecode (decode_lte_frame<.., SOFT = true>): this frame's inputs and outputs in
  // FeCl's turbo layouts, as element offsets into the caller's buffers.
  float* soft_ext = nullptr;  // [2][Tp] scratch: each constituent's last extrinsic values by step
  const void* state_in = nullptr;
  int32_t in_dtype = 1, out_dtype = 1;
  void *msg_out = nullptr, *syst_out = nullptr, *parity_out = nullptr, *state_out = nullptr;
  int64_t frame = 0;  // frame index within the caller's buffers
};

// Segment length for a frame of T steps split into `segs` segments: a multiple of
// the checkpoint spacing, so every segment boundary is a checkpoint.
__host__ __device__ inline int lte_seg_len(int T, int segs) {
  const int L = (T + segs - 1) / segs;
  return (L + kBlk - 1) / kBlk * kBlk;
}

// Decodes one frame with the whole CTA; lte_smem holds 2 * Kp floats + Shared<SEGS>.
// SOFT: soDecode (TurboDecoderImpl::soDecodeBlock, TurboDecoderImpl.cpp:75-150).
// WHOLE: K is a multiple of 8, as every LTE size is (the max-log kernels have a form for each,
// so that none carries both: their code has to stay in the instruction cache).
template <int ALG, int SEGS, bool SOFT, bool WHOLE>
__device__ __forceinline__ void decode_lte_frame(const LteJob& q) {
  constexpr int kThreads = 2 * SEGS;
  const int K = q.K, T = q.K + 3;
  const LteMap& m = q.map;
  const int nblk = m.nblk;
  const int nblk_msg = (K + kBlk - 1) / kBlk;
  float* X = lte_smem;
  float* Y = lte_smem + q.Kp;
  Shared<SEGS>& sh = *reinterpret_cast<Shared<SEGS>*>(lte_smem + 2 * q.Kp);
  Frame fr;
  fr.m = m;
  fr.Ls = q.scratch;
  fr.Lp0 = q.scratch + 8 * m.slots;
  fr.Lp1 = q.scratch + 16 * m.slots;
  fr.ts = q.scratch + 24 * m.slots;
  fr.perm = q.perm;
  fr.cka = q.ck;
  fr.ckb = q.ck + 8 * m.slots;
  const int tid = threadIdx.x;
  const int Lc = m.Lc, S = m.S;
  const Tol tol = SOFT ? kSoftTol : kDecodeTol;

  if (ALG == kLinear && tid < 8) s_lut[tid] = c_lut.v[tid];
  // X = Ls + e0 with e0 = 0 (constituent 1 reads it first under Parallel scheduling)
  for (int i = tid; i < nblk; i += kThreads) {
    int k, w;
    block_at(i, nblk, m, k, w);
    const float4* l = reinterpret_cast<const float4*>(fr.Ls) + k * m.Sp + w;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      reinterpret_cast<float4*>(X)[half_of(w * Lc + k, h)] = l[h * m.slots];
      reinterpret_cast<float4*>(Y)[half_of(w * Lc + k, h)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  // Tail: the trellis starts and ends in state 0; training starts from all states equal
  const float4 flat = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const float4 term_a = make_float4(0.0f, kNegInf, kNegInf, kNegInf);
  const float4 term_b = make_float4(kNegInf, kNegInf, kNegInf, kNegInf);
  __syncthreads();
  if (tid < 3) X[m.pos(K + tid)] = fr.ts[3 + tid];  // constituent 1's tail (resolve)
  __syncthreads();
  if (SOFT && q.state_in) {
    // the initial extrinsic values: X = Ls + e0, Y[pi(t)] = e1(t) (tail values are
    // replaced by the channel's tail bits before every pass, as in the reference)
    const int64_t s0 = q.frame * int64_t(2 * (K + 3));
    const uint16_t* perm = reinterpret_cast<const uint16_t*>(fr.perm);
    for (int k = tid; k < K; k += kThreads) {
      X[m.pos(k)] = X[m.pos(k)] + load_llr(q.state_in, q.in_dtype, s0 + k);
      Y[perm[m.slot_of(k >> 3) * 8 + (k & 7)] / 4] = load_llr(q.state_in, q.in_dtype, s0 + K + 3 + k);
    }
    __syncthreads();
  }

  int ran = q.iterations;
  for (int it = 0; it < q.iterations; ++it) {
    const bool last_soft = SOFT && it == q.iterations - 1;
#pragma unroll 1
    for (int jj = 0; jj < 2; ++jj) {
      const int j = q.parallel ? 1 - jj : jj;  // parallel: constituent 1 first, on the old X
      const bool fwd = tid < SEGS;
      const int w = fwd ? tid : tid - SEGS;
      const int lead = q.train / kBlk;
      // ---- A: segments with training starts
      {
        // the trellis's own start (end) where the training would reach it
        const bool exact = fwd ? (w == 0 || w * Lc - lead <= 0) : (w == S - 1 || ((w + 1) * Lc + lead) * kBlk >= T);
        // a forward start is the checkpoint at a0, a backward end the one at a0
        if (w < S)
          segment_walk<ALG>(fwd, j, w, lead, exact ? term_a : flat, exact ? term_b : flat,
                            int((fwd ? &sh.fwd_end[0][0] : &sh.bwd_start[0][0]) - lte_smem), SEGS, K, T, fr, q.Kp, false, tol);
      }
      __syncthreads();
      // ---- A2: verify boundaries; walk again the segments whose start disagrees.
      // One barrier both publishes and combines the checks; a round with a rejected
      // boundary adds two more.
      int rounds = 0;
      for (int round = 0; round < S; ++round) {
        bool bad = false;
        // forward: this segment's start (its checkpoint at a0) against the previous
        // segment's end; backward: this segment's start at a1 against the next
        // segment's end (its checkpoint at a1).  `right` is the neighbour's end.
        float right[8] = {};
        if (w < S && (fwd ? w > 0 : w < S - 1)) {
          float mine[8];
          if (fwd) {
            load_ck(fr.cka, m.slots, w, mine);
#pragma unroll
            for (int s = 0; s < 8; ++s) right[s] = sh.fwd_end[s][w - 1];
          } else {
            load_ck(fr.ckb, m.slots, w + 1, right);
#pragma unroll
            for (int s = 0; s < 8; ++s) mine[s] = sh.bwd_start[s][w];
          }
          bad = !close8(mine, right, tol);
        }
        // The end is in registers before the barrier and becomes the segment's start
        // after it, so a neighbour that is itself being walked again is read in its
        // old state; the next round checks the boundary again.
        if (!__syncthreads_or(bad)) break;
        ++rounds;
        if (bad) {
          if (q.stats) atomicAdd(q.stats + 2, 1ull);
          segment_walk<ALG>(fwd, j, w, 0, make_float4(right[0], right[1], right[2], right[3]),
                            make_float4(right[4], right[5], right[6], right[7]),
                            int((fwd ? &sh.fwd_end[0][0] : &sh.bwd_start[0][0]) - lte_smem), SEGS, K, T, fr, q.Kp, true, tol);
        }
        __syncthreads();
      }
      if (q.stats && tid == 0) {
        atomicAdd(q.stats + 0, 1ull);
        atomicAdd(q.stats + 1, (unsigned long long)rounds);
      }
      // ---- B: 8-step blocks, extrinsic output.  Only blocks holding message steps
      // run: the tail steps' a-priori values are the channel's tail bits, so their
      // extrinsic values are never read (with K a multiple of 8, as every LTE size
      // is, the last block is all tail).
      // soDecode does not scale the extrinsic values (TurboDecoderImpl.cpp:75-150)
      const float sf = SOFT ? 1.0f : q.sf[j * q.iterations + it];
      float* out = j == 0 ? X : (q.parallel ? q.ynew : Y);
      // soDecode's last iteration runs every block, tail blocks too, and records the
      // extrinsic and parity extrinsic values
      const int blocks = last_soft ? nblk : nblk_msg;
      SoftSink sink;
      if (last_soft) {
        sink.ext = q.soft_ext + j * q.Tp;
        sink.par = q.parity_out;
        sink.par0 = q.frame * int64_t(3 * K + 12) + K + 6 + j * (K + 3);
        sink.dtype = q.out_dtype;
      }
      for (int i = tid; i < blocks; i += kThreads) {
        int kb, wb;
        block_at(i, blocks, m, kb, wb);
        // WHOLE: every message block has 8 message steps, and runs without per-step tests, in
        // soDecode up to the last iteration (one K=6144 frame 259 us, 286 with the tests in every one)
        if constexpr (ALG == kApproximate && WHOLE && SOFT) {
          if (last_soft) ext_block<ALG, false, true>(j, kb, wb, K, T, fr, q.Kp, sf, out, sink);
          else ext_block<ALG, true, false>(j, kb, wb, K, T, fr, q.Kp, sf, out, sink);
        } else if constexpr (ALG == kApproximate) ext_block<ALG, WHOLE, SOFT>(j, kb, wb, K, T, fr, q.Kp, sf, out, sink);
        else ext_steps<ALG, SOFT>(j, kb, wb, K, T, fr, q.Kp, sf, out, sink);
      }
      __syncthreads();
    }
    if (q.parallel) {
      for (int k = tid; k < K; k += kThreads) Y[m.pos(k)] = q.ynew[m.pos(k)];
      __syncthreads();
    }
    // CRC stop (an extension; LTE transport blocks end with a CRC-24): the decisions
    // after this iteration are those the frame would end with; the CRC syndrome of the
    // K decided bits is the xor of the table entries of the bits that are 1.
    if (q.crc) {
      uint32_t syn = 0;
#pragma unroll 1
      for (int k = tid; k < K; k += kThreads)
        if ((X[m.pos(k)] + Y[m.pos(k)]) > 0.0f) syn ^= __ldg(q.crc + k);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) syn ^= __shfl_xor_sync(0xffffffffu, syn, o);
      if ((tid & 31) == 0) sh.crc_part[tid >> 5] = syn;
      __syncthreads();
      uint32_t all = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) all ^= sh.crc_part[w];
      __syncthreads();
      if (all == 0) {
        ran = it + 1;
        break;
      }
    }
  }
  if constexpr (SOFT) {
    // aPosterioriUpdate (TurboDecoderImpl.cpp:152-168) and the soDecode outputs: syst =
    // (0 + e0) + e1 at natural positions, the tails' extrinsic values after them;
    // parity = syst | both constituents' parity extrinsic values (written above);
    // msg = channel (+ a-priori) + syst; state = e0 | e1 in each constituent's order.
    const float* e0 = q.soft_ext;
    const float* e1 = q.soft_ext + q.Tp;
    const int64_t f = q.frame;
    for (int k = tid; k < K + 6; k += kThreads) {
      float v;
      if (k < K) v = e0[k] + Y[m.pos(k)];
      else v = k < K + 3 ? e0[k] : e1[k - 3];
      if (q.syst_out) store_llr(q.syst_out, q.out_dtype, f * int64_t(K + 6) + k, v);
      if (q.parity_out) store_llr(q.parity_out, q.out_dtype, f * int64_t(3 * K + 12) + k, v);
      if (q.msg_out && k < K) {
        const float ls = fr.Ls[((k >> 2) & 1) * 4 * m.slots + m.slot_of(k >> 3) * 4 + (k & 3)];
        store_llr(q.msg_out, q.out_dtype, f * int64_t(K) + k, ls + v);
      }
    }
    if (q.state_out)
      for (int t = tid; t < 2 * (K + 3); t += kThreads) {
        const float v = t < K + 3 ? e0[t] : e1[t - (K + 3)];
        store_llr(q.state_out, q.out_dtype, f * int64_t(2 * (K + 3)) + t, v);
      }
  } else {
    // a-posteriori and hard decision, TurboDecoderImpl.cpp:64-71
    if (K % 8 == 0 && reinterpret_cast<uintptr_t>(q.hard) % 8 == 0) {
#pragma unroll 1
      for (int b = tid; b < K / 8; b += kThreads) {
        uint32_t bits[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 x = reinterpret_cast<const float4*>(X)[half_of(b, h)], y = reinterpret_cast<const float4*>(Y)[half_of(b, h)];
          bits[h] = uint32_t((x.x + y.x) > 0.0f) | uint32_t((x.y + y.y) > 0.0f) << 8 | uint32_t((x.z + y.z) > 0.0f) << 16 |
                    uint32_t((x.w + y.w) > 0.0f) << 24;
        }
        reinterpret_cast<uint2*>(q.hard)[b] = make_uint2(bits[0], bits[1]);
      }
    } else {
#pragma unroll 1
      for (int k = tid; k < K; k += kThreads) q.hard[k] = uint8_t((X[m.pos(k)] + Y[m.pos(k)]) > 0.0f);
    }
    if (q.iters && tid == 0) *q.iters = ran;
  }
}

template <typename T>
__device__ __forceinline__ float to_f32(T v) { return float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

// Slots of chunks with the quotient by Lc (chunk numbers below 2^11) as a multiplication.
struct SlotOf {
  int Lc, Sp, plane;
  uint32_t inv;
  __device__ __forceinline__ explicit SlotOf(const LteMap& m)
      : Lc(m.Lc), Sp(m.Sp), plane(4 * m.slots), inv(m.Lc > 1 ? 0xffffffffu / uint32_t(m.Lc) + 1u : 0u) {}
  __device__ __forceinline__ int slot(int c) const {
    if (Lc == 1) return c;
    const int w = int(__umulhi(uint32_t(c), inv));
    return (c - w * Lc) * Sp + w;
  }
  // where step t's element of a staged array lies
  __device__ __forceinline__ int element(int t) const { return ((t >> 2) & 1) * plane + slot(t >> 3) * 4 + (t & 3); }
};

// One frame's input [3K+12] in FeCl's turbo layout | msg [K] | systTail1 [3] | systTail2 [3] |
// parity1 [K+3] | parity2 [K+3] | -> FP32 scratch in slot order: the regions are copied by
// loops of their own, and the element type is fixed per launch.  soDecode's a-priori input is added
// to the channel's systematic values and tails (TurboDecoderImpl.cpp:77-82).
template <typename T>
__device__ __forceinline__ void stage_frame(const T* in, const T* sys, float* out, int K, int Tp, const LteMap& m) {
  const SlotOf where(m);
  // four elements per thread and step, all loaded before any is stored, so that each
  // thread keeps four loads in flight (load latency, not bandwidth, bounds the copy)
  constexpr int kU = 4;
  const int step = int(blockDim.x);
  for (int i0 = threadIdx.x; i0 < Tp; i0 += kU * step) {
    float v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int i = i0 + u * step;
      v[u] = i < K + 3 ? (sys ? to_f32(in[i]) + to_f32(sys[i]) : to_f32(in[i])) : 0.0f;  // tail 1 follows the message
    }
#pragma unroll
    for (int u = 0; u < kU; ++u)
      if (i0 + u * step < Tp) out[where.element(i0 + u * step)] = v[u];
  }
  for (int c = 0; c < 2; ++c) {
    const T* src = in + K + 6 + c * (K + 3);  // parity (with its tail) of constituent c
    float* dst = out + (1 + c) * 8 * m.slots;
    for (int t0 = threadIdx.x; t0 < Tp; t0 += kU * step) {
      float v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int t = t0 + u * step;
        v[u] = t < K + 3 ? to_f32(src[t]) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (t0 + u * step < Tp) dst[where.element(t0 + u * step)] = v[u];
    }
  }
  if (threadIdx.x < 8) {
    float v = 0.0f;
    if (threadIdx.x < 6) v = sys ? to_f32(in[K + threadIdx.x]) + to_f32(sys[K + threadIdx.x]) : to_f32(in[K + threadIdx.x]);
    out[24 * m.slots + threadIdx.x] = v;
  }
}

// The byte offset of every step's interleaved element (LteMap::pos; K <= 12288: 16 bits), in
// slot order; the tail steps read behind the message, steps past them the first.
__device__ __forceinline__ void stage_positions(const uint32_t* perm, uint16_t* out, int K, int Tp, const LteMap& m,
                                                int first, int step) {
  const SlotOf where(m);
#pragma unroll 4
  for (int t = first; t < Tp; t += step) out[where.slot(t >> 3) * 8 + (t & 7)] = t < K + 3 ? uint16_t(4 * m.pos(t < K ? int(__ldg(perm + t)) : t)) : 0;
}

// A CTA's own staging of its frame and of positions for it alone (launches of at most one frame
// per SM, which this saves the staging launch; kStageHere).
__device__ __noinline__ void stage_here(const TurboLteParams& p, int64_t f, float* out, uint16_t* positions, LteMap m) {
  const int K = p.K;
  const int64_t in0 = f * int64_t(3 * K + 12), sys0 = f * int64_t(K + 6);
  const SlotOf where(m);
#pragma unroll 4
  for (int i = threadIdx.x; i < 3 * p.Tp; i += blockDim.x) {
    const int c = i < p.Tp ? 0 : i < 2 * p.Tp ? 1 : 2, t = i - c * p.Tp;  // systematic, parity 1, parity 2
    float v = 0.0f;
    if (t < K + 3) {  // tail 1 follows the message
      v = load_llr(p.llr, p.llr_dtype, size_t(in0 + (c ? K + 6 + (c - 1) * (K + 3) : 0) + t));
      if (c == 0 && p.syst_in) v += load_llr(p.syst_in, p.llr_dtype, size_t(sys0 + t));
    }
    out[c * 8 * m.slots + where.element(t)] = v;
  }
  if (threadIdx.x < 8) {
    float v = 0.0f;
    if (threadIdx.x < 6) {
      v = load_llr(p.llr, p.llr_dtype, size_t(in0 + K + threadIdx.x));
      if (p.syst_in) v += load_llr(p.syst_in, p.llr_dtype, size_t(sys0 + K + threadIdx.x));
    }
    out[24 * m.slots + threadIdx.x] = v;
  }
  stage_positions(p.perm[1], positions, K, p.Tp, m, threadIdx.x, blockDim.x);
  __syncthreads();
}

template <int ALG, int SEGS, bool SOFT, bool WHOLE>
__global__ void __launch_bounds__(2 * SEGS, SEGS == 32 ? 4 : (SEGS == 128 ? 1 : 3)) turbo_lte_kernel(const __grid_constant__ TurboLteParams p) {
  const int64_t f = p.frame0 + blockIdx.x;
  LteJob q;
  q.K = p.K;
  q.Kp = p.Kp;
  q.Tp = p.Tp;
  q.map = LteMap{p.seg_len / kBlk, p.segments, p.seg_stride, p.slots, p.Tp / kBlk};
  q.train = p.train;
  q.iterations = p.iterations;
  q.sf = p.sf;
  q.perm = p.perm_pos;
  q.scratch = p.scratch + int64_t(blockIdx.x) * p.frame_stride;
  if (p.stage_here) {
    q.perm = p.perm_pos + int64_t(blockIdx.x) * p.slots;
    stage_here(p, f, p.scratch + int64_t(blockIdx.x) * p.frame_stride,
               reinterpret_cast<uint16_t*>(p.perm_pos + int64_t(blockIdx.x) * p.slots), q.map);
  }
  q.ck = p.ck + int64_t(blockIdx.x) * (16 * p.slots);
  q.hard = p.hard + f * p.K;
  q.iters = p.iters ? p.iters + f : nullptr;
  q.stats = p.stats;
  q.crc = p.crc;
  q.parallel = p.parallel;
  if (p.ynew) {  // per frame: ynew [Tp] | soft_ext [2][Tp]
    q.ynew = p.ynew + int64_t(blockIdx.x) * (3 * p.Tp);
    q.soft_ext = q.ynew + p.Tp;
  }
  q.state_in = p.state_in;
  q.in_dtype = p.llr_dtype;
  q.out_dtype = p.out_dtype;
  q.msg_out = p.msg_out;
  q.syst_out = p.syst_out;
  q.parity_out = p.parity_out;
  q.state_out = p.state_out;
  q.frame = f;
  decode_lte_frame<ALG, SEGS, SOFT, WHOLE>(q);
}


// Geometry of a frame of K message bits: T trellis steps, nblk 8-step chunks, the padded
// length Kp = Tp of the exchange arrays, and the staged layout of `segs` forward and `segs`
// backward segments (LteMap).  Sp is one more than S (the checkpoint at T may open a segment
// of its own) and even, so that rows of slots start on 32-byte sectors.
struct LteGeometry {
  int T, nblk, Tp, Kp, seg_len, S, Sp, slots;
  __host__ __device__ LteGeometry(int K, int segs) {
    T = K + 3;
    nblk = (T + kBlk - 1) / kBlk;
    Tp = nblk * kBlk;
    Kp = Tp;
    seg_len = lte_seg_len(T, segs);
    S = (T + seg_len - 1) / seg_len;
    Sp = (S + 2) & ~1;
    slots = seg_len / kBlk * Sp;
  }
  __host__ __device__ LteMap map() const { return LteMap{seg_len / kBlk, S, Sp, slots, nblk}; }
  __host__ __device__ int staged_floats() const { return 24 * slots + 8; }
  __host__ __device__ int ck_floats() const { return 16 * slots; }
  __host__ __device__ int perm_floats() const { return 4 * slots; }
  // One frame of the mixed-K batch: staged inputs, checkpoints, positions, rounded to 128
  // bytes so frames share no cache line.
  __host__ __device__ int frame_floats() const { return (staged_floats() + ck_floats() + perm_floats() + 31) & ~31; }
};

// Staging of a launch's frames (grid-strided) and, by the last block, of its positions.
template <typename T>
__global__ void turbo_lte_stage(TurboLteParams p) {
  const LteMap m{p.seg_len / kBlk, p.segments, p.seg_stride, p.slots, p.Tp / kBlk};
  if (blockIdx.x == gridDim.x - 1) {
    stage_positions(p.perm[1], reinterpret_cast<uint16_t*>(p.perm_pos), p.K, p.Tp, m, threadIdx.x, blockDim.x);
    return;
  }
  const T* llr = static_cast<const T*>(p.llr);
  for (int64_t i = blockIdx.x; i < p.nframes; i += gridDim.x - 1) {
    const int64_t f = p.frame0 + i;
    const T* sys = p.syst_in ? static_cast<const T*>(p.syst_in) + f * int64_t(p.K + 6) : nullptr;
    stage_frame(llr + f * int64_t(3 * p.K + 12), sys, p.scratch + i * p.frame_stride, p.K, p.Tp, m);
  }
}

// Mixed-K batch, staging: one block per frame (grid-strided).
__global__ void turbo_lte_batch_stage(TurboLteBatchParams p) {
  for (int64_t f = blockIdx.x; f < p.nframes; f += gridDim.x) {
    const TurboLteBatchFrame d = p.frames[f];
    const LteGeometry g(d.K, kDefaultSegs);
    const LteMap m = g.map();
    switch (d.llr_dtype) {
      case kF64: stage_frame(static_cast<const double*>(d.llr), static_cast<const double*>(nullptr), d.scratch, d.K, g.Tp, m); break;
      case kF16: stage_frame(static_cast<const __half*>(d.llr), static_cast<const __half*>(nullptr), d.scratch, d.K, g.Tp, m); break;
      default: stage_frame(static_cast<const float*>(d.llr), static_cast<const float*>(nullptr), d.scratch, d.K, g.Tp, m); break;
    }
    stage_positions(d.perm, reinterpret_cast<uint16_t*>(d.scratch + g.staged_floats() + g.ck_floats()), d.K, g.Tp, m,
                    threadIdx.x, blockDim.x);
  }
}

// Mixed-K batch, decoding: persistent CTAs take frames from a counter in the order
// of the descriptor table (longest first), so frames of every size share one launch
// and the long ones do not trail behind.  Shared memory is sized for the largest K.
template <int ALG, int SEGS, bool WHOLE>
__global__ void __launch_bounds__(2 * SEGS, SEGS == 32 ? 4 : 3) turbo_lte_batch_kernel(TurboLteBatchParams p) {
  __shared__ int next;
  for (;;) {
    __syncthreads();  // every thread has read `next` (and finished the last frame)
    if (threadIdx.x == 0) next = atomicAdd(p.counter, 1);
    __syncthreads();
    const int64_t f = next;
    if (f >= p.nframes) break;
    const TurboLteBatchFrame d = p.frames[f];
    const LteGeometry g(d.K, SEGS);
    LteJob q;
    q.K = d.K;
    q.Kp = g.Kp;
    q.Tp = g.Tp;
    q.map = g.map();
    q.train = p.train;
    q.iterations = d.iterations;
    q.sf = d.sf;
    q.scratch = d.scratch;
    q.ck = d.scratch + g.staged_floats();
    q.perm = reinterpret_cast<const uint4*>(d.scratch + g.staged_floats() + g.ck_floats());
    q.hard = d.hard;
    q.iters = d.iters;
    q.stats = p.stats;
    q.crc = d.crc;
    decode_lte_frame<ALG, SEGS, false, WHOLE>(q);
  }
}

template <int SEGS>
size_t lte_smem_bytes(int max_K) {
  return size_t(2 * LteGeometry(max_K, SEGS).Kp) * sizeof(float) + sizeof(Shared<SEGS>);
}

// Frames that CTAs may stage themselves (one per SM of a 148-SM GPU), with at most so many elements
// per thread: longer frames are staged by a launch of their own, which keeps more loads in flight than
// the few threads of a decoding CTA.  Itself and by a launch, max-log: K=2112 decode (25 a thread) 125.8 and 123.7 us,
// K=6144 (72) 174.8 and 167.4, K=1024 (12) the same either way; soDecode with its 128 threads K=1024
// (24) 124.7 and 124.4, K=2112 (50) 165.7 and 157.7, K=6144 (144) 314.9 and 285.4.
constexpr int64_t kStageHere = 148;
constexpr int kStageElements = 24;

int resolve_segs(int segs) { return segs == 32 || segs == 64 || segs == 128 ? segs : kDefaultSegs; }

// Streaming multiprocessors of the current device (0 if the query fails).
int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms;
}

// Training steps before each segment when the caller leaves them to the launcher.
// Max-log: 80 (K=6144 x 1024 at 0.7 dB: 1.10 ms against 1.13 ms with 96, the same
// decisions; 4x more segments are walked again, but a walk again stops at the first
// checkpoint it reproduces).  The log-MAP algorithms: 96, since their fix-up walks
// cost more than the training they save (Exact 54.8 ms with 80 against 40.7 ms).
int default_train(int algorithm) { return algorithm == kApproximate ? 80 : 96; }

// CTAs of `smem` bytes resident on an SM, at most `most` (their registers).
int64_t ctas_per_sm(size_t smem, int64_t most) {
  const int64_t fit = int64_t((228 << 10) / ((smem + 1024 + 127) / 128 * 128));
  return fit < most ? fit : most;
}

// Frames (from the first) that the 32-segment shape decodes when the segment count
// is left to the launcher; the rest take the 64-segment shape.  A CTA decodes one
// frame start to end, so n frames take ceil(n / resident) rounds of about equal time
// and a last round holding a few frames leaves most of the GPU idle for a whole
// frame's decode.  When the 64-segment shape (fewer resident CTAs: 3 per SM against
// 4, register-bound) would end on a round less than half full, whole rounds of the
// 32-segment shape go first so that the 64-segment rounds are full or nearly so:
// K=6144 x 1024 frames on 148 SMs is 592 + 432 frames in two rounds instead of
// 444 + 444 + 136 in three.  Which frames take which shape decides the FP32 rounding of
// their window boundaries, so the rule is fixed arithmetic.
int64_t split_frames(int K, int64_t nframes, int sms) {
  const int64_t r64 = sms * ctas_per_sm(lte_smem_bytes<64>(K), 3), r32 = sms * ctas_per_sm(lte_smem_bytes<32>(K), 4);
  if (r64 <= 0 || r32 <= 0 || nframes <= r64) return 0;
  auto rounds = [](int64_t n, int64_t r) { return (n + r - 1) / r; };
  auto tail_ok = [&](int64_t n) { return n % r64 == 0 || 2 * (n % r64) >= r64; };
  if (tail_ok(nframes)) return 0;
  for (int64_t n32 = r32; n32 < nframes; n32 += r32) {
    const int64_t rest = nframes - n32;
    if (tail_ok(rest) && rounds(n32, r32) + rounds(rest, r64) <= rounds(nframes, r64)) return n32;
  }
  return 0;
}

}  // namespace

cudaError_t turbo_lte_init() {
  static std::atomic<unsigned long long> done{0};
  return once_per_device(done, [] {
    const LinearPairs t = make_linear_pairs();
    return cudaMemcpyToSymbol(c_lut, &t, sizeof(t));
  });
}

size_t turbo_lte_scratch_bytes(int K, int64_t nframes, bool extra) {
  // whichever shapes the launcher takes: the largest frame of the three, and positions for two
  // launches or for every frame of a small batch
  int frame = 0, positions = 0;
  for (int segs : {32, 64, 128}) {
    const LteGeometry g(K, segs);
    frame = std::max(frame, g.staged_floats() + g.ck_floats());
    positions = std::max(positions, g.perm_floats());
  }
  const int Tp = LteGeometry(K, kDefaultSegs).Tp;
  auto need = [&](int64_t n) {
    return (size_t(n) * (size_t(frame) + (extra ? size_t(3 * Tp) : 0)) +
            size_t(n <= kStageHere ? n + 1 : 2) * size_t(positions)) *
           sizeof(float);
  };
  // never less than a smaller batch takes: a host call's chunks share the plan of the longest, and
  // a last one of at most kStageHere frames holds positions for each (148 frames of K = 6144
  // take more than 149)
  return std::max(need(nframes), need(std::min(nframes, kStageHere)));
}

cudaError_t launch_turbo_lte(TurboLteParams p, cudaStream_t s) {
  cudaError_t e0 = turbo_lte_init();
  if (e0 != cudaSuccess) return e0;
  if (p.nframes <= 0) return cudaSuccess;
  int segs = resolve_segs(p.segs);
  // A batch of at most one frame per SM decodes in one round whose time is one
  // frame's latency: with the segment count left to the launcher it takes the
  // 128-segment shape (one CTA of 256 threads per frame: half as many phase B blocks
  // per thread and shorter segment walks than with 64), as does an explicit 128.
  // soDecode always uses 64.
  const int sms = device_sms();
  if (p.soft) segs = 64;
  else if (p.segs == 0 && p.nframes <= sms) segs = 128;
  // Short frames: the fewest threads whose segments are the same (K <= 248: 8 steps each in
  // every shape; warps without a segment only lengthen the barriers).
  auto narrowest = [&](int segs) {
    while (!p.soft && segs > 32 && lte_seg_len(p.K + 3, segs / 2) == lte_seg_len(p.K + 3, segs)) segs /= 2;
    return segs;
  };
  segs = narrowest(segs);
  if (p.soft) p.crc = nullptr;
  if (p.train < 0) p.train = default_train(p.algorithm);
  float* at = p.scratch;
  // frames [first, first + n) with `segs` segments: staging, then the decoder
  auto decode = [&](int64_t first, int64_t n, int segs, auto kern, size_t smem) -> cudaError_t {
    const LteGeometry g(p.K, segs);
    TurboLteParams q = p;
    q.frame0 = first;
    q.nframes = n;
    q.Tp = g.Tp;
    q.Kp = g.Kp;  // the exchange arrays are padded like the parity
    q.seg_len = g.seg_len;
    q.segments = g.S;
    q.seg_stride = g.Sp;
    q.slots = g.slots;
    q.frame_stride = g.staged_floats();
    q.scratch = at;
    q.ck = q.scratch + n * q.frame_stride;
    at = q.ck + n * int64_t(g.ck_floats());
    // parallel scheduling and soDecode: per frame ynew [Tp] | soft_ext [2][Tp] after the
    // checkpoints (turbo_lte_scratch_bytes(K, n, true))
    q.ynew = (p.parallel || p.soft) ? at : nullptr;
    if (q.ynew) at += n * int64_t(3 * g.Tp);
    q.perm_pos = reinterpret_cast<uint4*>(at);
    q.stage_here = p.nframes <= kStageHere && p.nframes <= sms && 3 * g.Tp <= kStageElements * 2 * segs;
    at += (q.stage_here ? n : 1) * int64_t(g.perm_floats());
    const unsigned blocks = unsigned(n < 148 * 8 ? n : 148 * 8) + 1;
    if (!q.stage_here) switch (p.llr_dtype) {
      case kF64: turbo_lte_stage<double><<<blocks, 256, 0, s>>>(q); break;
      case kF16: turbo_lte_stage<__half><<<blocks, 256, 0, s>>>(q); break;
      default: turbo_lte_stage<float><<<blocks, 256, 0, s>>>(q); break;
    }
    cudaError_t err = allow_shared_memory(kern);
    if (err != cudaSuccess) return err;
    kern<<<unsigned(n), 2 * segs, smem, s>>>(q);
    return cudaGetLastError();
  };
  // the kernel of a shape for the algorithm and, in max-log, for K % 8
  const bool whole = p.K % kBlk == 0;
  auto pick = [&](auto shape, auto soft) -> void (*)(TurboLteParams) {
    constexpr int kSegs = decltype(shape)::value;
    constexpr bool kSoft = decltype(soft)::value;
    if (p.algorithm == kExact) return turbo_lte_kernel<kExact, kSegs, kSoft, true>;
    if (p.algorithm == kLinear) return turbo_lte_kernel<kLinear, kSegs, kSoft, true>;
    if (whole) return turbo_lte_kernel<kApproximate, kSegs, kSoft, true>;
    return turbo_lte_kernel<kApproximate, kSegs, kSoft, false>;
  };
  using S32 = std::integral_constant<int, 32>;
  using S64 = std::integral_constant<int, 64>;
  using S128 = std::integral_constant<int, 128>;
  if (p.soft) return decode(0, p.nframes, 64, pick(S64{}, std::true_type{}), lte_smem_bytes<64>(p.K));
  if (segs == 32) return decode(0, p.nframes, 32, pick(S32{}, std::false_type{}), lte_smem_bytes<32>(p.K));
  if (segs == 128) return decode(0, p.nframes, 128, pick(S128{}, std::false_type{}), lte_smem_bytes<128>(p.K));
  // the launcher's choice: whole rounds of the 32-segment shape first where that fills
  // the rounds better (split_frames)
  const int64_t n32 = p.segs == 0 && segs == 64 ? split_frames(p.K, p.nframes, sms) : 0;
  if (n32 > 0) {
    const cudaError_t err = decode(0, n32, 32, pick(S32{}, std::false_type{}), lte_smem_bytes<32>(p.K));
    if (err != cudaSuccess) return err;
  }
  return decode(n32, p.nframes - n32, 64, pick(S64{}, std::false_type{}), lte_smem_bytes<64>(p.K));
}

// The mixed-K kernel for the algorithm and, in max-log, for batches whose K are all
// multiples of 8.
static void (*batch_kernel(int algorithm, bool whole))(TurboLteBatchParams) {
  if (algorithm == kExact) return turbo_lte_batch_kernel<kExact, kDefaultSegs, true>;
  if (algorithm == kLinear) return turbo_lte_batch_kernel<kLinear, kDefaultSegs, true>;
  if (whole) return turbo_lte_batch_kernel<kApproximate, kDefaultSegs, true>;
  return turbo_lte_batch_kernel<kApproximate, kDefaultSegs, false>;
}

size_t turbo_lte_frame_floats(int K) { return size_t(LteGeometry(K, kDefaultSegs).frame_floats()); }

int turbo_lte_batch_max_ctas(int max_K, int algorithm, bool whole) {
  const size_t smem = lte_smem_bytes<kDefaultSegs>(max_K);
  int per_sm = 0, sms = 0, dev = 0;
  auto kern = batch_kernel(algorithm, whole);
  if (allow_shared_memory(kern) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 2 * kDefaultSegs, smem) != cudaSuccess) {
    cudaGetLastError();
    per_sm = 0;
  }
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per_sm * sms;
}

cudaError_t launch_turbo_lte_batch(const TurboLteBatchParams& p, cudaStream_t s) {
  cudaError_t e = turbo_lte_init();
  if (e != cudaSuccess) return e;
  if (p.nframes <= 0) return cudaSuccess;
  if (p.max_K <= 0 || p.max_K > 12288) return cudaErrorInvalidValue;
  TurboLteBatchParams q = p;
  if (q.train < 0) q.train = default_train(q.algorithm);
  e = cudaMemsetAsync(q.counter, 0, sizeof(int32_t), s);
  if (e != cudaSuccess) return e;
  const unsigned stage_blocks = unsigned(q.nframes < 148 * 8 ? q.nframes : 148 * 8);
  turbo_lte_batch_stage<<<stage_blocks, 256, 0, s>>>(q);
  const size_t smem = lte_smem_bytes<kDefaultSegs>(q.max_K);
  int ctas = q.ctas > 0 ? q.ctas : turbo_lte_batch_max_ctas(q.max_K, q.algorithm, q.whole != 0);
  if (ctas <= 0) return cudaErrorInvalidConfiguration;
  if (int64_t(ctas) > q.nframes) ctas = int(q.nframes);
  auto kern = batch_kernel(q.algorithm, q.whole != 0);
  e = allow_shared_memory(kern);
  if (e != cudaSuccess) return e;
  kern<<<unsigned(ctas), 2 * kDefaultSegs, smem, s>>>(q);
  return cudaGetLastError();
}

}  // namespace fecl
