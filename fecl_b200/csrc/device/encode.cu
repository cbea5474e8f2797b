// Device encoders and the BPSK/AWGN channel.
//
// The encoders run the reference's encoding steps, so their output is bit-exact with
// LdpcCode::encode / TurboCode::encode and the reference they restate:
//   LDPC  systematic copy, then the sparse XOR steps of Ldpc::Structure::encode
//         (src/detail/Ldpc.cpp:180-209): gap parity from the message (DC), the
//         B correction, the message part of the T rows (A), and the back
//         substitution through T;
//   turbo systematic copy, then per constituent the interleaved message through the
//         trellis and the greedy tail of Convolutional::Structure::encode
//         (src/detail/Convolutional.cpp:167-221), in Turbo::Structure::encode's
//         layout (src/detail/Turbo.cpp:155-170).
// The channel maps bit b to x = 2b - 1, adds N(0, sigma^2) noise with
// sigma^2 = 1 / (2 Es/N0) and returns L = 2 y / sigma^2 (the model of the bench and
// of the reference's test channel).  Its normal variates come from Philox-4x32-10
// (Salmon, Moraes, Dror, Shaw: "Parallel random numbers: as easy as 1, 2, 3",
// SC 2011), counter = (element / 4, seed), and the Box-Muller transform.
#include <math.h>

#include "common.cuh"
#include "kernels.hpp"
#include "trellis_encode.cuh"

#include <algorithm>

namespace fecl {
namespace {

// LDPC encoding, a CTA per `per` (at most 8) frames with the whole code word in shared
// memory: byte i holds bit i of the CTA's frames, frame f in its bit f, so one byte xor
// serves all of them and the code's tables are read once per CTA.  Bound by the gathers
// of the T-part rows (one shared byte per edge and CTA); a thread per row, its entries
// interleaved over the 32 rows of a warp so that their loads are contiguous.  The
// accumulator of the DVB-S2 codes is a prefix xor: each thread folds an odd number of
// words (so that the threads' strides fall into different banks), the threads' totals
// are scanned over the block, and the words are written back with their carries.  Other
// T parts are solved level by level.  V: bytes per access of the caller's buffers.
// 512 DVB-S2 normal r=1/2 frames: 35 us a call (1.4 TB/s of bits in and out) against
// 44.6 ms with a thread per frame, whose single chain of dependent loads left the GPU
// idle; 79 us before a warp's entry lines were streamed.
template <int V>
struct EncodeVec;
template <>
struct EncodeVec<16> {
  uint4 v;
};
template <>
struct EncodeVec<8> {
  uint2 v;
};
template <>
struct EncodeVec<4> {
  uint32_t v;
};
template <>
struct EncodeVec<1> {
  uint8_t v;
};

constexpr int kEncodeFrames = 8;  // frames per CTA at most: the bits of a byte

// Bit f of every byte, and the frames' bits folded into one byte each.
__device__ __forceinline__ uint32_t bit_of(uint32_t w, int f) { return (w >> f) & 0x01010101u; }
__device__ __forceinline__ uint4 bit_of(uint4 w, int f) {
  return make_uint4(bit_of(w.x, f), bit_of(w.y, f), bit_of(w.z, f), bit_of(w.w, f));
}
__device__ __forceinline__ uint2 bit_of(uint2 w, int f) { return make_uint2(bit_of(w.x, f), bit_of(w.y, f)); }
__device__ __forceinline__ uint8_t bit_of(uint8_t w, int f) { return uint8_t((w >> f) & 1); }
__device__ __forceinline__ void fold(uint32_t& a, uint32_t w, int f) { a |= w << f; }
__device__ __forceinline__ void fold(uint4& a, uint4 w, int f) {
  fold(a.x, w.x, f);
  fold(a.y, w.y, f);
  fold(a.z, w.z, f);
  fold(a.w, w.w, f);
}
__device__ __forceinline__ void fold(uint2& a, uint2 w, int f) {
  fold(a.x, w.x, f);
  fold(a.y, w.y, f);
}
__device__ __forceinline__ void fold(uint8_t& a, uint8_t w, int f) { a = uint8_t(a | (w << f)); }

// Writes bits [0, n) of s to position `at` of each of the nf frames' code words.
template <int V>
__device__ __forceinline__ void put_bits(const uint8_t* s, int n, uint8_t* parity, int64_t N, int64_t at, int nf) {
  using T = decltype(EncodeVec<V>::v);
  for (int i = int(threadIdx.x) * V; i < n; i += int(blockDim.x) * V) {
    const T w = *reinterpret_cast<const T*>(s + i);
#pragma unroll
    for (int f = 0; f < kEncodeFrames; ++f)
      if (f < nf) *reinterpret_cast<T*>(parity + f * N + at + i) = bit_of(w, f);
  }
}

template <int V>
__global__ void __launch_bounds__(1024) ldpc_encode_kernel(LdpcEncodeTables t, const uint8_t* msg, uint8_t* parity,
                                                           int64_t nframes, int per) {
  using T = decltype(EncodeVec<V>::v);
  extern __shared__ __align__(16) uint8_t s[];
  __shared__ uint32_t part[32];
  const int tid = int(threadIdx.x), threads = int(blockDim.x), lane = tid & 31, warp = tid >> 5, warps = threads >> 5;
  const int64_t f0 = int64_t(blockIdx.x) * per;
  const int nf = int(nframes - f0 < per ? nframes - f0 : per);
  const uint8_t* m = msg + f0 * t.K;
  uint8_t* c = parity + f0 * t.N;

  // the message: copied to the code words and folded into shared memory
  for (int i = tid * V; i < t.K; i += threads * V) {
    T w[kEncodeFrames];
#pragma unroll
    for (int f = 0; f < kEncodeFrames; ++f)
      if (f < nf) w[f] = bit_of(*reinterpret_cast<const T*>(m + int64_t(f) * t.K + i), 0);
    T acc = {};
#pragma unroll
    for (int f = 0; f < kEncodeFrames; ++f)
      if (f < nf) {
        *reinterpret_cast<T*>(c + int64_t(f) * t.N + i) = w[f];
        fold(acc, w[f], f);
      }
    *reinterpret_cast<T*>(s + i) = acc;
  }
  if (tid == 0) s[t.zero_at] = 0;
  __syncthreads();

  // gap parity from the message: dense rows, a warp each
  uint8_t* gap = s + t.off_gap;
  for (int r = warp; r < t.gap; r += warps) {
    uint32_t v = 0;
    for (uint32_t e = t.dc_ptr[r] + lane; e < t.dc_ptr[r + 1]; e += 32) v ^= s[t.dc_idx[e]];
    v = __reduce_xor_sync(0xffffffffu, v);
    if (lane == 0) gap[r] = uint8_t(v);
  }
  if (t.gap) __syncthreads();

  // T-part rows: the message (A) and gap (B) columns.  A warp takes a run of blocks and
  // streams their entry lines, kAhead lines loaded while the kAhead before are gathered;
  // lane l holds the end of the run's block l.
  uint8_t* p = s + t.off_t;
  constexpr int kAhead = 8;
  const int blocks = (t.rows + 31) / 32, run = (blocks + warps - 1) / warps;
  const int b_end = min(blocks, (warp + 1) * run);
  for (int b = warp * run; b < b_end; b += 32) {
    const int nb = min(32, b_end - b);
    const uint32_t ends = t.row_ptr[min(b + lane + 1, blocks)];
    uint32_t e = t.row_ptr[b];
    const uint32_t last = __shfl_sync(0xffffffffu, ends, nb - 1);
    uint32_t next[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) next[j] = e + 32 * j < last ? __ldg(t.row_idx + e + 32 * j + lane) : t.zero_at;
    uint32_t v = 0, end = __shfl_sync(0xffffffffu, ends, 0);
    int cur = 0;
    for (; e < last; e += 32 * kAhead) {
      uint32_t idx[kAhead];
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        idx[j] = next[j];
        const uint32_t a = e + 32 * (kAhead + j);
        next[j] = a < last ? __ldg(t.row_idx + a + lane) : t.zero_at;
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        while (cur < nb && end == e + 32 * j) {  // block cur is complete (or has no entries)
          const int r = (b + cur) * 32 + lane;
          if (r < t.rows) p[r] = uint8_t(v);
          v = 0;
          if (++cur < nb) end = __shfl_sync(0xffffffffu, ends, cur);
        }
        v ^= s[idx[j]];
      }
    }
    for (; cur < nb; ++cur) {  // the last block with entries, and empty ones after it
      const int r = (b + cur) * 32 + lane;
      if (r < t.rows) p[r] = uint8_t(v);
      v = 0;
    }
  }
  __syncthreads();

  // back substitution through T
  if (t.chain) {
    uint32_t* w = reinterpret_cast<uint32_t*>(p);
    const int words = (t.rows + 3) / 4;
    if (tid < words * 4 - t.rows) p[t.rows + tid] = 0;
    const int each = ((words + threads - 1) / threads) | 1;
    const int w0 = tid * each, w1 = min(words, w0 + each);
    __syncthreads();
    uint32_t x = 0;
    for (int i = w0; i < w1; ++i) x ^= w[i];
    x ^= x >> 16;
    x = (x ^ (x >> 8)) & 0xffu;
    uint32_t upto = x;  // inclusive scan over the warp
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto ^= y;
    }
    if (lane == 31) part[warp] = upto;
    __syncthreads();
    uint32_t carry = upto ^ x;
    for (int q = 0; q < warp; ++q) carry ^= part[q];
    for (int i = w0; i < w1; ++i) {
      uint32_t v = w[i];
      v ^= v << 8;
      v ^= v << 16;
      v ^= carry * 0x01010101u;
      w[i] = v;
      carry = v >> 24;
    }
    __syncthreads();
  } else {
    for (int l = 0; l < t.levels; ++l) {
      for (uint32_t q = t.level_ptr[l] + tid; q < t.level_ptr[l + 1]; q += threads) {
        const uint32_t r = t.level_rows[q];
        uint32_t v = p[r];
        for (uint32_t e = t.src_ptr[q]; e < t.src_ptr[q + 1]; ++e) v ^= p[t.src_idx[e]];
        p[r] = uint8_t(v);
      }
      __syncthreads();
    }
  }
  put_bits<V>(gap, t.gap, c, t.N, t.K, nf);
  put_bits<V>(p, t.rows, c, t.N, int64_t(t.K) + t.gap, nf);
}

// The same steps with one thread per frame, for code words beyond shared memory.
__global__ void ldpc_encode_long_kernel(LdpcEncodeTables t, const uint8_t* msg, uint8_t* parity, int64_t nframes) {
  const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= nframes) return;
  const uint8_t* m = msg + f * t.K;
  uint8_t* c = parity + f * t.N;
  for (int i = 0; i < t.K; ++i) c[i] = m[i] & 1;
  for (int i = t.K; i < t.N; ++i) c[i] = 0;
  uint8_t* p = c + t.K;
  for (int r = 0; r < t.dc_rows; ++r) {
    uint8_t v = p[r];
    for (uint32_t e = t.dc_ptr[r]; e < t.dc_ptr[r + 1]; ++e) v ^= m[t.dc_idx[e]] & 1;
    p[r] = v;
  }
  for (int r = 0; r < t.b_rows; ++r) {
    uint8_t v = p[t.gap + r];
    for (uint32_t e = t.b_ptr[r]; e < t.b_ptr[r + 1]; ++e) v ^= p[t.b_idx[e]];
    p[t.gap + r] = v;
  }
  uint8_t* p2 = p + t.gap;
  for (int r = 0; r < t.a_rows; ++r) {
    uint8_t v = p2[r];
    for (uint32_t e = t.a_ptr[r]; e < t.a_ptr[r + 1]; ++e) v ^= m[t.a_idx[e]] & 1;
    p2[r] = v;
  }
  for (int r = 0; r < t.t_rows; ++r) {
    const uint8_t v = p2[r];
    if (v)
      for (uint32_t e = t.t_ptr[r] + 1; e < t.t_ptr[r + 1]; ++e) p2[t.t_idx[e]] ^= 1;
  }
}

__device__ __forceinline__ int popc(uint32_t x) { return __popc(x); }

// CTA (frame, constituent j); constituent 0's CTA also copies the message.
// K=6144 x 1024 frames: 97 us a call against 2.97 ms with a thread per frame and constituent.
__global__ void __launch_bounds__(kEncodeThreads) turbo_encode_cta(const __grid_constant__ TurboDeviceCode code,
                                                                   const uint8_t* msg, uint8_t* parity) {
  __shared__ EncodeShared sh;
  extern __shared__ __align__(16) uint8_t s[];
  const int64_t f = blockIdx.x / code.n;
  const int j = int(blockIdx.x - f * code.n);
  const uint8_t* m = msg + f * code.msg;
  uint8_t* out = parity + f * code.parity;
  if (j == 0)
    for (int i = threadIdx.x; i < code.msg; i += kEncodeThreads) out[i] = m[i] & 1;
  int tail = code.msg, par = code.syst;
  for (int q = 0; q < j; ++q) {
    tail += code.c[q].syst_tail_size;
    par += code.c[q].parity_size;
  }
  encode_constituent(code.c[j], m, code.c[j].perm, out + par, out + tail, sh, s);
}

// Thread (frame, constituent j), for trellises and lengths beyond turbo_encode_cta's and for many
// short messages (encode_cta_us);
// constituent 0's thread also copies the message.
__global__ void turbo_encode_kernel(TurboDeviceCode code, const uint8_t* msg, uint8_t* parity, int64_t nframes) {
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t f = t / code.n;
  const int j = int(t - f * code.n);
  if (f >= nframes) return;
  const uint8_t* m = msg + f * code.msg;
  uint8_t* out = parity + f * code.parity;
  if (j == 0)
    for (int i = 0; i < code.msg; ++i) out[i] = m[i] & 1;
  int syst_tail = code.msg, par = code.syst;
  for (int q = 0; q < j; ++q) {
    syst_tail += code.c[q].syst_tail_size;
    par += code.c[q].parity_size;
  }
  const TurboDeviceConstituent& c = code.c[j];
  uint32_t state = 0;
  for (int s = 0; s < c.length; ++s) {
    uint32_t in = 0;
    for (int k = 0; k < c.input_size; ++k) {
      const int i = s * c.input_size + k;
      in |= uint32_t(m[c.perm[i]] & 1) << k;
    }
    const uint32_t o = c.output[state * c.input_count + in];
    state = c.next_state[state * c.input_count + in];
    for (int k = 0; k < c.output_size; ++k) out[par + s * c.output_size + k] = uint8_t((o >> k) & 1);
  }
  int po = par + c.length * c.output_size, to = syst_tail;
  for (int s = 0; s < c.tail; ++s) {
    int best_count = -1;
    uint32_t best = 0;
    for (int u = 0; u < c.input_count; ++u) {
      const int count = popc(state) - popc(c.next_state[state * c.input_count + u]);
      if (count > best_count) {
        best_count = count;
        best = uint32_t(u);
      }
    }
    const uint32_t o = c.output[state * c.input_count + best];
    for (int k = 0; k < c.output_size; ++k) out[po + k] = uint8_t((o >> k) & 1);
    for (int k = 0; k < c.input_size; ++k) out[to + k] = uint8_t((best >> k) & 1);
    po += c.output_size;
    to += c.input_size;
    state = c.next_state[state * c.input_count + best];
  }
}

// Philox-4x32 with 10 rounds (Salmon et al. 2011, Section 4.2): a round multiplies
// the two even words by the round constants, swaps and xors the high halves with the
// odd words and the key; the key is bumped by the Weyl constants between rounds.
struct U4 {
  uint32_t x, y, z, w;
};
__device__ __forceinline__ U4 philox10(U4 ctr, uint32_t k0, uint32_t k1) {
  constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = U4{hi1 ^ ctr.y ^ k0, lo1, hi0 ^ ctr.w ^ k1, lo0};
    k0 += W0;
    k1 += W1;
  }
  return ctr;
}

// A uniform in (0, 1] from 32 random bits.
__device__ __forceinline__ float unit(uint32_t v) { return (float(v) + 1.0f) * 2.3283064365386963e-10f; }

__global__ void awgn_kernel(const uint8_t* bits, int64_t n, float sigma, float scale, uint64_t seed, int dtype, void* out) {
  const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;  // one Philox block = 4 elements
  if (q * 4 >= n) return;
  const U4 r = philox10(U4{uint32_t(q), uint32_t(uint64_t(q) >> 32), 0x46654331u, 0u}, uint32_t(seed),
                        uint32_t(seed >> 32));
  float z[4];
  {
    const float rad = sqrtf(-2.0f * logf(unit(r.x)));
    float s, c;
    sincospif(2.0f * unit(r.y), &s, &c);
    z[0] = rad * c;
    z[1] = rad * s;
  }
  {
    const float rad = sqrtf(-2.0f * logf(unit(r.z)));
    float s, c;
    sincospif(2.0f * unit(r.w), &s, &c);
    z[2] = rad * c;
    z[3] = rad * s;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = q * 4 + k;
    if (i < n) {
      const float x = (bits[i] & 1) ? 1.0f : -1.0f;
      store_llr(out, dtype, size_t(i), scale * (x + sigma * z[k]));
    }
  }
}

unsigned blocks_for(int64_t threads, int per_block) {
  const int64_t b = (threads + per_block - 1) / per_block;
  return unsigned(b > 0 ? b : 1);
}

}  // namespace

cudaError_t launch_ldpc_encode(const LdpcEncodeTables& t, const uint8_t* msg, uint8_t* parity, int64_t nframes,
                               cudaStream_t s) {
  if (nframes <= 0) return cudaSuccess;
  if (!t.bytes) {
    ldpc_encode_long_kernel<<<blocks_for(nframes, 64), 64, 0, s>>>(t, msg, parity, nframes);
    return cudaGetLastError();
  }
  // Frames per CTA: as few as let one round of CTAs, one per SM, take the batch (the row
  // gathers cost the same for 1 and for 8 frames), at most the 8 bits of a byte.
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  int64_t per = (nframes + sms - 1) / sms;
  if (per > kEncodeFrames) per = kEncodeFrames;
  const int64_t blocks = (nframes + per - 1) / per;
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
  const int threads = t.N >= 8192 ? 1024 : 256;
  // the widest access that divides the parts of a code word and both buffers' alignment
  const uintptr_t parts = uintptr_t(t.K) | uintptr_t(t.N) | uintptr_t(t.gap) | reinterpret_cast<uintptr_t>(msg) |
                          reinterpret_cast<uintptr_t>(parity);
  auto run = [&](auto kern) -> cudaError_t {
    cudaError_t err = allow_shared_memory(kern);
    if (err != cudaSuccess) return err;
    kern<<<unsigned(blocks), threads, t.bytes, s>>>(t, msg, parity, nframes, int(per));
    return cudaGetLastError();
  };
  if (parts % 16 == 0) return run(ldpc_encode_kernel<16>);
  if (parts % 8 == 0) return run(ldpc_encode_kernel<8>);
  if (parts % 4 == 0) return run(ldpc_encode_kernel<4>);
  return run(ldpc_encode_kernel<1>);
}

cudaError_t launch_turbo_encode(const TurboDeviceCode& code, const uint8_t* msg, uint8_t* parity, int64_t nframes,
                                cudaStream_t s) {
  if (nframes <= 0) return cudaSuccess;
  bool by_cta = nframes * code.n <= 0x7fffffff;
  int longest = 0;
  double cta = 0.0, thread = 0.0;
  for (int j = 0; j < code.n; ++j) {
    by_cta = by_cta && encode_by_cta(code.c[j]);
    cta += encode_cta_us(code.c[j], nframes);
    thread = std::max(thread, encode_thread_us(code.c[j], nframes * code.n, 400.0));
    longest = code.c[j].length > longest ? code.c[j].length : longest;
  }
  if (by_cta && cta <= thread) {
    const cudaError_t e = allow_shared_memory(turbo_encode_cta, kEncodeFixed);
    if (e != cudaSuccess) return e;
    turbo_encode_cta<<<unsigned(nframes * code.n), kEncodeThreads, size_t(longest), s>>>(code, msg, parity);
    return cudaGetLastError();
  }
  turbo_encode_kernel<<<blocks_for(nframes * code.n, 64), 64, 0, s>>>(code, msg, parity, nframes);
  return cudaGetLastError();
}

cudaError_t launch_awgn(const uint8_t* bits, int64_t n, double esn0, uint64_t seed, int dtype, void* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const double sigma2 = 1.0 / (2.0 * esn0);
  awgn_kernel<<<blocks_for((n + 3) / 4, 256), 256, 0, s>>>(bits, n, float(sqrt(sigma2)), float(2.0 / sigma2), seed,
                                                            dtype, out);
  return cudaGetLastError();
}

}  // namespace fecl
