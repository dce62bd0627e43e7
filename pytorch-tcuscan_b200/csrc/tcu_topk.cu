// tcu_topk.cu -- top-k of 16-bit keys on B200.
//
// Reference: run_topk_int16 / run_topk_fp16 (src/torch/torch_topk.h:86-211,
// src/kernels/kernel_topk.h:35-140) bisect the value range with repeated
// stable splits.  The set returned is every element above the k-th largest
// key t plus the lowest-positioned elements equal to t; here it is written in
// input order (the reference emits it band by band).
//
// Three forms, chosen by size and k (topk_t):
//   sampled     x is read from HBM once.  topk_collect_kernel: every CTA takes
//               the same 1024 stratified samples of x and their r-th largest
//               key lo (r so far above the k / n quantile that fewer than k
//               elements >= lo is a ~6-sigma event), then streams its part of
//               x: one candidate bit per element (key >= lo) and a shared
//               histogram of the candidates' keys.  The last CTA finds t in
//               the summed histogram.
//   histograms  k beyond n / 32, small n, and what the sampled form hands
//               over (samples full of one value, t outside the histogram,
//               fewer than k candidates): two full histograms (high byte, then
//               low byte inside the chosen high byte, topk_hist_kernel<0/1>),
//               each picking its byte in its last CTA.
//   one CTA     n <= kTkSmall: the same two histograms and the output in one
//               launch (topk_small_kernel).
// The first two share topk_count_kernel (elements above and equal to t per
// warp and per CTA, and the final bits key >= t) and topk_emit_kernel (each
// CTA's output offset from the totals before it, then its elements in order).
// The sampled form launches the histogram kernels too; after a collect pass
// that found t they return at once.  No kernel waits on another CTA: "last
// CTA" is the one whose arrival completes the count.
//
// Bound by instructions, then by the latency of five dependent launches: the
// reads alone would take 6.5 us for 20 Mi fp16 (42 MB).  Measured on B200, a
// whole call, U[0,1) fp16 (before: two shared-atomic histograms, count,
// offsets and emit passes over x): n = 4096 17 us (43), n = 2^20, k = 1024
// 27 us (46), n = 20 Mi - 10, k = 4579 46 us (146), k = n / 8 104 us (168),
// k = n - 1 123 us (327); sorted input, k = 4579 84 us (119).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "tcu_host.h"

namespace tcu {

constexpr int kTkThreads = 256;
constexpr int kTkWarps = kTkThreads / 32;
constexpr int kTkStep = 256;       // elements of one warp step: 8 (16 bytes) per lane
constexpr int kTkUnroll = 4;       // warp steps in flight
constexpr int kTkBins = 8192;      // candidate histogram: keys lo .. lo + 8190, the last bin takes all above
constexpr int kTkSamples = 1024;
constexpr int kTkCtasPerSm = 4;
constexpr int kTkHistCtasPerSm = 3;  // 64 KB of counters each
constexpr int kTkSmallThreads = 512;
// One CTA holds 64 keys per thread and their 128 KB of byte counters: 17 us a
// call at 4096 elements, where the launches of the other forms take 25 us.
constexpr int kTkSmall = kTkSmallThreads * 64;

// The selection key merges -0 with +0 and maps every NaN to the largest key:
// the reference compares values (x <= pivot is false for NaN, so NaNs always
// rank above the pivot).
enum TopkCodec { kTopkInt16 = 1, kTopkFp16 = 2, kTopkBf16 = 3 };

template <int CODEC>
__device__ __forceinline__ uint32_t topk_key(uint32_t b) {  // b < 65536
  if constexpr (CODEC == kTopkInt16) {
    return b ^ 0x8000u;
  } else {
    const uint32_t inf = CODEC == kTopkFp16 ? 0x7C00u : 0x7F80u;
    const uint32_t mag = b & 0x7FFFu;
    if (mag > inf) return 0xFFFFu;  // NaN
    return (b & 0x8000u) ? 0x8000u - mag : 0x8000u + mag;
  }
}

// Keys of the two halves of a word (5 instructions for two floats where the
// scalar form takes about 8 for each).
template <int CODEC>
__device__ __forceinline__ uint32_t topk_key2(uint32_t w) {
  if constexpr (CODEC == kTopkInt16) {
    return w ^ 0x80008000u;
  } else {
    uint32_t neg;  // 0xFFFF in every negative half
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(neg) : "r"(w));
    const uint32_t k = (w ^ (neg | 0x80008000u)) + (neg & 0x00010001u);
    if constexpr (CODEC == kTopkFp16) {
      const __half2 h = *reinterpret_cast<const __half2*>(&w);
      return k | __hneu2_mask(h, h);
    } else {
      const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w);
      return k | __hneu2_mask(h, h);
    }
  }
}

// Input bits of a key that is no NaN (both halves).
template <int CODEC>
__device__ __forceinline__ uint32_t topk_unkey2(uint32_t key) {
  uint32_t b;
  if constexpr (CODEC == kTopkInt16) b = key ^ 0x8000u;
  else b = key >= 0x8000u ? key - 0x8000u : 0x8000u | (0x8000u - key);
  return b | (b << 16);
}

// Bit i: key i of the 8 packed in kw >= the key in both halves of t2.
__device__ __forceinline__ uint32_t tk_ge8(const uint32_t (&kw)[4], uint32_t t2) {
  uint32_t acc = 0;
#pragma unroll
  for (int w = 3; w >= 0; --w) acc = (acc << 2) | __vminu2(__vmaxu2(kw[w], t2) ^ kw[w], 0x00010001u);
  return ~(acc | (acc >> 15)) & 0xFFu;
}

// The same straight from the input bits, for a pivot that is no NaN (NaN
// inputs compare as above it).
template <int CODEC>
__device__ __forceinline__ uint32_t tk_ge8_raw(const uint4& v, uint32_t piv2) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if constexpr (CODEC == kTopkInt16) {
    const uint32_t kw[4] = {topk_key2<CODEC>(w[0]), topk_key2<CODEC>(w[1]), topk_key2<CODEC>(w[2]),
                            topk_key2<CODEC>(w[3])};
    return tk_ge8(kw, topk_key2<CODEC>(piv2));
  } else {
    uint32_t acc = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t m;
      if constexpr (CODEC == kTopkFp16)
        m = __hgeu2_mask(*reinterpret_cast<const __half2*>(&w[i]), *reinterpret_cast<const __half2*>(&piv2));
      else
        m = __hgeu2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[i]),
                         *reinterpret_cast<const __nv_bfloat162*>(&piv2));
      acc |= m & (0x00020001u << (2 * i));
    }
    return (acc | (acc >> 16)) & 0xFFu;
  }
}

struct TopkState {
  int robust;          // the histograms decide t (zero after a collect pass that found it)
  int hi;              // high byte of t (histogram form)
  int krem;            // elements still to take inside that high byte
  int thr;             // t
  int ties;            // elements equal to t to take (lowest positions first)
  unsigned arrived[3];  // CTAs finished: collect, histogram 0, histogram 1
};

struct TopkParams {
  const uint16_t* x;
  int64_t n;
  int64_t k;
  int64_t steps;      // ceil(n / kTkStep)
  int64_t cta_steps;  // steps of one CTA of the collect / count / emit grid
  int warp_steps;     // steps of one warp of that grid
  int rank;           // collect: the sample rank that gives lo
  int force_robust;   // no collect pass ran
  TopkState* st;
  unsigned* bins;     // [kTkBins] candidate keys, then [2][256] bytes; zero on entry
  uint32_t* mask;     // one bit per element
  int2* warp_cnt;     // (above, equal) per warp
  int2* cta_cnt;      // and per CTA
  uint16_t* out;
  int* idx_out;
};

// Inclusive block sum of one int; *total gets the block's.  sw: WARPS ints.
template <int WARPS>
__device__ __forceinline__ int tk_block_incl(int v, int* sw, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += o;
  }
  if (lane == 31) sw[w] = v;
  __syncthreads();
  int pre = 0, tot = 0;
#pragma unroll
  for (int k = 0; k < WARPS; ++k) {
    const int s = sw[k];
    pre += k < w ? s : 0;
    tot += s;
  }
  __syncthreads();
  *total = tot;
  return pre + v;
}

// True for the CTA whose arrival completes the grid; its reads of what the
// other CTAs wrote before arriving follow the fence.
__device__ __forceinline__ bool tk_last_cta(unsigned* arrived, int* s_flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *s_flag = atomicAdd(arrived, 1u) == gridDim.x - 1;
  __syncthreads();
  const bool last = *s_flag != 0;
  if (last) __threadfence();
  return last;
}

// 8 consecutive elements from e0 as packed words (zero past the end).
template <bool VEC>
__device__ __forceinline__ uint4 tk_load8(const uint16_t* __restrict__ x, int64_t e0, int64_t n) {
  if (VEC && e0 + 8 <= n) return __ldg(reinterpret_cast<const uint4*>(x + e0));
  uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (e0 + i < n) w[i >> 1] |= (uint32_t)x[e0 + i] << (16 * (i & 1));
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Elements of [e0, e0 + 8) inside the input, as a bit mask.
__device__ __forceinline__ uint32_t tk_in(int64_t e0, int64_t n) {
  return e0 + 8 <= n ? 0xFFu : (e0 >= n ? 0u : (1u << (int)(n - e0)) - 1u);
}

// Byte counters: every thread counts 256 digits in 64 words of its own, all in
// the thread's shared-memory bank, so counting needs no atomics and has no
// bank conflicts whatever the distribution.  No digit may be counted more than
// 255 times by a thread between two flushes.
template <int THREADS>
struct TkCounters {
  uint8_t* mine;
  uint32_t* words;  // [64][THREADS]
  __device__ __forceinline__ explicit TkCounters(uint8_t* s)
      : mine(s + threadIdx.x * 4), words(reinterpret_cast<uint32_t*>(s)) {}
  __device__ __forceinline__ void zero() {
#pragma unroll 16
    for (int i = 0; i < 64; ++i) words[i * THREADS + threadIdx.x] = 0u;
  }
  // dig: the digit in bits 8-15, anything elsewhere
  __device__ __forceinline__ void add(uint32_t dig) {
    constexpr uint32_t ROW = THREADS * 4 / 1024;  // row bytes over the digit's place value
    mine[(dig & 0xFC00u) * ROW + ((dig >> 8) & 3u)]++;
  }
  // Returns the block's count of digit threadIdx.x (threads below 256).
  __device__ __forceinline__ int flush() {
    constexpr int TPR = THREADS / 64;      // threads per row of four digits
    constexpr int WPT = THREADS / TPR;     // words of each of them
    __syncthreads();
    const int row = threadIdx.x / TPR, q = threadIdx.x % TPR, lane = threadIdx.x & 31;
    uint32_t a02 = 0, a13 = 0;  // 16-bit sums of bytes 0 / 2 and 1 / 3
#pragma unroll 8
    for (int i = 0; i < WPT; ++i) {  // rotated: a warp's reads spread over the banks
      const uint32_t v = words[row * THREADS + q * WPT + ((i + lane) & (WPT - 1))];
      a02 += v & 0x00FF00FFu;
      a13 += (v >> 8) & 0x00FF00FFu;
    }
    __syncthreads();  // the counters may be reused
    uint32_t c0 = a02 & 0xFFFFu, c1 = a13 & 0xFFFFu, c2 = a02 >> 16, c3 = a13 >> 16;
#pragma unroll
    for (int d = 1; d < TPR; d <<= 1) {
      c0 += __shfl_xor_sync(0xffffffffu, c0, d);
      c1 += __shfl_xor_sync(0xffffffffu, c1, d);
      c2 += __shfl_xor_sync(0xffffffffu, c2, d);
      c3 += __shfl_xor_sync(0xffffffffu, c3, d);
    }
    if (q == 0) {
      uint32_t* o = words + 4 * row;
      o[0] = c0;
      o[1] = c1;
      o[2] = c2;
      o[3] = c3;
    }
    __syncthreads();
    const int c = threadIdx.x < 256 ? (int)words[threadIdx.x] : 0;
    __syncthreads();
    return c;
  }
};

// Counts the keys of 8 packed elements by their high byte (LEVEL 0), or by
// the low byte among those whose high byte is hi (LEVEL 1).
template <int LEVEL, int THREADS>
__device__ __forceinline__ void tk_count8(TkCounters<THREADS>& cnt, const uint32_t (&kw)[4], uint32_t in, uint32_t hi) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t k = (i & 1) ? kw[i >> 1] >> 16 : kw[i >> 1] & 0xFFFFu;
    if (((in >> i) & 1u) && (!LEVEL || (k >> 8) == hi)) cnt.add(LEVEL ? k << 8 : k);
  }
}

// The digit holding the want-th largest key, from the counts of digits in s_c
// (256 ints): s_pick gets the digit and the keys above it.  All threads.
template <int WARPS>
__device__ __forceinline__ void tk_pick(const int* s_c, int want, int* sw, int* s_pick) {
  const int d = 255 - (int)threadIdx.x;
  const int c = d >= 0 ? s_c[d] : 0;
  int tot;
  const int incl = tk_block_incl<WARPS>(c, sw, &tot);
  if (incl >= want && incl - c < want) {
    s_pick[0] = d;
    s_pick[1] = incl - c;
  }
  __syncthreads();
}

// The r-th largest of the block's 4 sample keys per thread; *at_least gets
// the number of samples not below it.  s_h: 256 ints.
__device__ __forceinline__ uint32_t tk_sample_rank(const uint32_t (&key)[4], int r, int* s_h, int* sw, int* s_pick,
                                                   int* at_least) {
  uint32_t hi = 0;
  int want = r, got = 0;
#pragma unroll
  for (int level = 0; level < 2; ++level) {
    s_h[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (level == 0 || (key[i] >> 8) == hi) atomicAdd(&s_h[level == 0 ? key[i] >> 8 : key[i] & 0xFFu], 1);
    __syncthreads();
    tk_pick<kTkWarps>(s_h, want, sw, s_pick);
    const uint32_t dig = (uint32_t)s_pick[0];
    want -= s_pick[1];
    got += s_pick[1];
    if (level == 0) {
      hi = dig;
    } else {
      *at_least = got + s_h[dig];
      hi = (hi << 8) | dig;
    }
    __syncthreads();
  }
  return hi;
}

// The published integer hash "lowbias32" (C. Wellons, hash-prospector).
__device__ __forceinline__ uint32_t tk_hash(uint32_t v) {
  v ^= v >> 16;
  v *= 0x7FEB352Du;
  v ^= v >> 15;
  v *= 0x846CA68Bu;
  return v ^ (v >> 16);
}

// The collect pass (see the file comment).  Candidate bits and not candidate
// lists, because bits need no capacity: an input whose samples mislead only
// sets more of them.  22 us for 20 Mi fp16 from a cold cache (13 instructions
// per element); 36 us with a scalar key and eight predicated histogram updates
// per vector (25 per element).
template <int CODEC, bool VEC>
__global__ void __launch_bounds__(kTkThreads, kTkCtasPerSm) topk_collect_kernel(const TopkParams p) {
  __shared__ int s_h[kTkBins];
  __shared__ int sw[kTkWarps], s_pick[2], s_flag;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t n = p.n;
  uint32_t skey[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // one element of every 1024th part of x
    const uint32_t j = threadIdx.x * 4 + i;
    const int64_t a = (int64_t)((uint64_t)n * j / kTkSamples), b = (int64_t)((uint64_t)n * (j + 1) / kTkSamples);
    const int64_t e = a + (int64_t)(((uint64_t)tk_hash(j) * (uint64_t)(b - a)) >> 32);
    skey[i] = topk_key<CODEC>(__ldg(p.x + e));
  }
  int at_least;
  const uint32_t lo = tk_sample_rank(skey, p.rank, s_h, sw, s_pick, &at_least);
  // one value holds a large part of the samples: nearly all of x could be
  // candidates with one counter, so the byte histograms take over (the same
  // decision in every CTA)
  if (at_least > 2 * p.rank + 64 || lo == 0xFFFFu) {
    if (blockIdx.x == 0 && threadIdx.x == 0) p.st->robust = 1;
    return;
  }
#pragma unroll
  for (int i = 0; i < kTkBins / kTkThreads; ++i) s_h[i * kTkThreads + threadIdx.x] = 0;
  __syncthreads();

  const uint32_t piv2 = topk_unkey2<CODEC>(lo);
  uint8_t* mask8 = reinterpret_cast<uint8_t*>(p.mask);
  const int64_t full = n / kTkStep;  // whole steps
  const int64_t s_end = min((blockIdx.x + 1) * p.cta_steps, p.steps);
  const int64_t s0 = blockIdx.x * p.cta_steps + (int64_t)w * p.warp_steps;
  const int64_t s1 = min(s0 + p.warp_steps, s_end);
  for (int64_t s = s0; s < s1; s += kTkUnroll) {
    uint4 v[kTkUnroll];
#pragma unroll
    for (int u = 0; u < kTkUnroll; ++u)
      if (s + u < s1) v[u] = tk_load8<VEC>(p.x, (s + u) * kTkStep + lane * 8, n);
#pragma unroll
    for (int u = 0; u < kTkUnroll; ++u) {
      if (s + u >= s1) break;  // warp-uniform
      uint32_t bits = tk_ge8_raw<CODEC>(v[u], piv2);
      if (s + u >= full) bits &= tk_in((s + u) * kTkStep + lane * 8, n);
      mask8[(s + u) * 32 + lane] = (uint8_t)bits;
      while (bits) {
        const int i = __ffs(bits) - 1;
        bits &= bits - 1;
        const uint32_t a = (i & 2) ? v[u].y : v[u].x, b = (i & 2) ? v[u].w : v[u].z;
        const uint32_t wd = (i & 4) ? b : a;
        const uint32_t key = topk_key<CODEC>((i & 1) ? wd >> 16 : wd & 0xFFFFu);
        atomicAdd(&s_h[min(key - lo, (uint32_t)(kTkBins - 1))], 1);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kTkBins / kTkThreads; ++i) {
    const int c = s_h[i * kTkThreads + threadIdx.x];
    if (c) atomicAdd(&p.bins[i * kTkThreads + threadIdx.x], (unsigned)c);
  }
  if (!tk_last_cta(&p.st->arrived[0], &s_flag)) return;
  // the bin of the k-th largest key, from the top: a thread owns 32 bins
  constexpr int PER = kTkBins / kTkThreads;
  const int b0 = (kTkThreads - 1 - (int)threadIdx.x) * PER;
  int b[PER], c = 0;
#pragma unroll
  for (int i = 0; i < PER; i += 4) {
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(p.bins + b0 + i));
    b[i] = (int)q.x;
    b[i + 1] = (int)q.y;
    b[i + 2] = (int)q.z;
    b[i + 3] = (int)q.w;
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) c += b[i];
  int tot;
  const int incl = tk_block_incl<kTkWarps>(c, sw, &tot);
  if (threadIdx.x == 0 && tot < p.k) p.st->robust = 1;
  int above = incl - c;
  if (incl >= p.k && above < p.k) {
#pragma unroll
    for (int i = PER - 1; i >= 0; --i) {
      if (above < p.k && above + b[i] >= p.k) {
        if (b0 + i == kTkBins - 1) p.st->robust = 1;  // t lies among the keys that share the last bin
        p.st->thr = (int)lo + b0 + i;
        p.st->ties = (int)p.k - above;
      }
      above += b[i];
    }
  }
}

// 256-bin histogram of the key's high byte (LEVEL 0), or of the low byte of
// the keys whose high byte is st->hi (LEVEL 1); the last CTA picks the bin of
// the k-th largest.  22 / 24 us for 20 Mi fp16 U[0,1) and no other for any
// other distribution; shared atomics on four copies per warp took 30 / 33 us
// (four high bytes hold half of those keys) and serialised on equal keys.
template <int CODEC, int LEVEL, bool VEC>
__global__ void __launch_bounds__(kTkThreads, kTkHistCtasPerSm) topk_hist_kernel(const TopkParams p) {
  extern __shared__ __align__(16) uint8_t s_cnt[];
  __shared__ int s_c[256];
  __shared__ int sw[kTkWarps], s_pick[2], s_flag;
  if (!p.force_robust && !p.st->robust) return;
  const uint32_t hi = LEVEL ? (uint32_t)p.st->hi : 0u;
  TkCounters<kTkThreads> cnt(s_cnt);
  int acc = 0;
  cnt.zero();  // each thread clears the words it counts in
  constexpr int PER = 4 * 8;  // keys per thread and round
  constexpr int64_t ROUND = (int64_t)kTkThreads * PER;
  int done = 0;
  for (int64_t b = blockIdx.x * ROUND; b < p.n; b += gridDim.x * ROUND) {  // block-uniform
    if (done + PER > 255) {
      acc += cnt.flush();
      cnt.zero();
      done = 0;
    }
    uint4 v[4];
    const int64_t e0 = b + threadIdx.x * 8;
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = tk_load8<VEC>(p.x, e0 + u * kTkThreads * 8, p.n);
    const bool whole = b + ROUND <= p.n;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t kw[4] = {topk_key2<CODEC>(v[u].x), topk_key2<CODEC>(v[u].y), topk_key2<CODEC>(v[u].z),
                              topk_key2<CODEC>(v[u].w)};
      if (whole) tk_count8<LEVEL>(cnt, kw, 0xFFu, hi);
      else tk_count8<LEVEL>(cnt, kw, tk_in(e0 + u * kTkThreads * 8, p.n), hi);
    }
    done += PER;
  }
  acc += cnt.flush();
  unsigned* bins = p.bins + kTkBins + LEVEL * 256;
  if (acc) atomicAdd(&bins[threadIdx.x], (unsigned)acc);
  if (!tk_last_cta(&p.st->arrived[1 + LEVEL], &s_flag)) return;
  s_c[threadIdx.x] = (int)__ldcg(&bins[threadIdx.x]);
  const int want = LEVEL ? p.st->krem : (int)p.k;
  __syncthreads();
  tk_pick<kTkWarps>(s_c, want, sw, s_pick);
  if (threadIdx.x == 0) {
    if (LEVEL == 0) {
      p.st->hi = s_pick[0];
      p.st->krem = want - s_pick[1];
    } else {
      p.st->thr = (int)((hi << 8) | (uint32_t)s_pick[0]);
      p.st->ties = want - s_pick[1];
    }
  }
}

// Elements above and equal to t per warp and per CTA, and the bits key >= t.
// After a collect pass only the candidates are looked at; otherwise all of x
// is read.
template <int CODEC, bool VEC>
__global__ void __launch_bounds__(kTkThreads, kTkCtasPerSm) topk_count_kernel(const TopkParams p) {
  __shared__ int2 s_c[kTkWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t thr = (uint32_t)p.st->thr;
  const int64_t s_end = min((blockIdx.x + 1) * p.cta_steps, p.steps);
  const int64_t s0 = blockIdx.x * p.cta_steps + (int64_t)w * p.warp_steps;
  const int64_t s1 = min(s0 + p.warp_steps, s_end);
  int a = 0, ge = 0;
  if (p.force_robust || p.st->robust) {
    uint8_t* mask8 = reinterpret_cast<uint8_t*>(p.mask);
    const uint32_t t2 = thr | (thr << 16);
    const uint32_t u2 = thr < 0xFFFFu ? t2 + 0x00010001u : t2;
    const uint32_t gt_on = thr < 0xFFFFu ? 0xFFu : 0u;
    for (int64_t s = s0; s < s1; s += kTkUnroll) {
      uint4 v[kTkUnroll];
#pragma unroll
      for (int u = 0; u < kTkUnroll; ++u)
        if (s + u < s1) v[u] = tk_load8<VEC>(p.x, (s + u) * kTkStep + lane * 8, p.n);
#pragma unroll
      for (int u = 0; u < kTkUnroll; ++u) {
        if (s + u >= s1) break;  // warp-uniform
        const uint32_t in = tk_in((s + u) * kTkStep + lane * 8, p.n);
        const uint32_t kw[4] = {topk_key2<CODEC>(v[u].x), topk_key2<CODEC>(v[u].y), topk_key2<CODEC>(v[u].z),
                                topk_key2<CODEC>(v[u].w)};
        const uint32_t g = tk_ge8(kw, t2) & in;
        mask8[(s + u) * 32 + lane] = (uint8_t)g;
        ge += __popc(g);
        a += __popc(tk_ge8(kw, u2) & in & gt_on);
      }
    }
  } else {
    const int64_t w1 = s1 * 8;
#pragma unroll 4
    for (int64_t i = s0 * 8 + lane; i < w1; i += 32) {
      const uint32_t m0 = p.mask[i];
      uint32_t m = m0, keep = 0;
      while (m) {
        const int j = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t key = topk_key<CODEC>(__ldg(p.x + i * 32 + j));
        a += key > thr;
        keep |= (uint32_t)(key >= thr) << j;
      }
      if (keep != m0) p.mask[i] = keep;
      ge += __popc(keep);
    }
  }
  a = warp_sum_any(a);
  ge = warp_sum_any(ge);
  if (lane == 0) {
    s_c[w] = make_int2(a, ge - a);
    p.warp_cnt[blockIdx.x * kTkWarps + w] = make_int2(a, ge - a);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 t = s_c[0];
#pragma unroll
    for (int k = 1; k < kTkWarps; ++k) {
      t.x += s_c[k].x;
      t.y += s_c[k].y;
    }
    p.cta_cnt[blockIdx.x] = t;
  }
}

// Writes the selected elements in input order (values and int32 positions).
// 32 mask words (1024 elements) at a time: where they hold few elements each
// lane walks the bits of its own word; where they hold many the warp takes one
// word after another, a lane per element, so the stores are consecutive.
template <int CODEC>
__global__ void __launch_bounds__(kTkThreads, kTkCtasPerSm) topk_emit_kernel(const TopkParams p) {
  constexpr int kDense = 128;  // elements in 32 words
  __shared__ int s_a[kTkWarps], s_q[kTkWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int2 own = p.cta_cnt[blockIdx.x];
  if (own.x + own.y == 0) return;  // block-uniform
  const uint32_t thr = (uint32_t)p.st->thr;
  const int ties = p.st->ties;
  int a = 0, q = 0;  // elements above / equal before this warp
  for (int c = threadIdx.x; c < (int)blockIdx.x; c += kTkThreads) {
    const int2 t = p.cta_cnt[c];
    a += t.x;
    q += t.y;
  }
  a = warp_sum_any(a);
  q = warp_sum_any(q);
  if (lane == 0) {
    s_a[w] = a;
    s_q[w] = q;
  }
  __syncthreads();
  a = q = 0;
#pragma unroll
  for (int k = 0; k < kTkWarps; ++k) {
    a += s_a[k];
    q += s_q[k];
  }
  for (int k = 0; k < w; ++k) {
    const int2 t = p.warp_cnt[blockIdx.x * kTkWarps + k];
    a += t.x;
    q += t.y;
  }
  const int2 mine = p.warp_cnt[blockIdx.x * kTkWarps + w];
  if (mine.x + mine.y == 0 || (mine.x == 0 && q >= ties)) return;  // warp-uniform, no barrier follows
  const unsigned lt = (1u << lane) - 1u;
  const int64_t s_end = min((blockIdx.x + 1) * p.cta_steps, p.steps);
  const int64_t s0 = blockIdx.x * p.cta_steps + (int64_t)w * p.warp_steps;
  const int64_t w1 = min(s0 + p.warp_steps, s_end) * 8;
  for (int64_t i0 = s0 * 8; i0 < w1; i0 += 32) {
    const uint32_t m = i0 + lane < w1 ? p.mask[i0 + lane] : 0u;
    const int held = warp_sum_any(__popc(m));
    if (held == 0) continue;
    if (held <= kDense) {
      const int e0 = (int)(i0 + lane) * 32;
      uint32_t am = 0;
      for (uint32_t b = m; b; b &= b - 1) {
        const int j = __ffs(b) - 1;
        am |= (uint32_t)(topk_key<CODEC>(__ldg(p.x + e0 + j)) > thr) << j;
      }
      const int c = __popc(am) | (__popc(m ^ am) << 16);
      int inc = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      const int tot = __shfl_sync(0xffffffffu, inc, 31);
      int la = a + ((inc - c) & 0xFFFF), lq = q + ((inc - c) >> 16);
      a += tot & 0xFFFF;
      q += tot >> 16;
      for (uint32_t b = m; b; b &= b - 1) {
        const int j = __ffs(b) - 1;
        const bool above = (am >> j) & 1u;
        if (above || lq < ties) {
          const int o = la + (lq < ties ? lq : ties);
          p.out[o] = p.x[e0 + j];
          p.idx_out[o] = e0 + j;
        }
        la += above;
        lq += !above;
      }
    } else {
#pragma unroll 1
      for (int g = 0; g < 32; g += 8) {
        uint32_t mw[8], xv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          mw[u] = __shfl_sync(0xffffffffu, m, g + u);
          xv[u] = ((mw[u] >> lane) & 1u) ? (uint32_t)__ldg(p.x + (i0 + g + u) * 32 + lane) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const bool on = (mw[u] >> lane) & 1u;
          const bool above = on && topk_key<CODEC>(xv[u]) > thr;
          const unsigned am = __ballot_sync(0xffffffffu, above);
          const unsigned qm = mw[u] & ~am;
          const int lq = q + __popc(qm & lt);
          if (on && (above || lq < ties)) {
            const int o = a + __popc(am & lt) + (lq < ties ? lq : ties);
            p.out[o] = (uint16_t)xv[u];
            p.idx_out[o] = (int)(i0 + g + u) * 32 + lane;
          }
          a += __popc(am);
          q += __popc(qm);
        }
      }
    }
  }
}

// n <= kTkSmall in one launch: each thread holds 64 consecutive elements, the
// two byte histograms give t, block scans give the positions.
template <int CODEC, bool VEC>
__global__ void __launch_bounds__(kTkSmallThreads, 1) topk_small_kernel(const uint16_t* __restrict__ x, int n, int k,
                                                                        uint16_t* __restrict__ out,
                                                                        int* __restrict__ idx_out) {
  extern __shared__ __align__(16) uint8_t s_cnt[];
  constexpr int WARPS = kTkSmallThreads / 32;
  __shared__ int s_c[256];
  __shared__ int sw[WARPS], s_pick[2];
  const int per = ((n + kTkSmallThreads - 1) / kTkSmallThreads + 7) & ~7;  // elements per thread, <= 64
  const int e0 = threadIdx.x * per;
  const int nv = per / 8;
  uint4 v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = u < nv ? tk_load8<VEC>(x, e0 + u * 8, n) : make_uint4(0u, 0u, 0u, 0u);
  TkCounters<kTkSmallThreads> cnt(s_cnt);
  uint32_t thr = 0;
  int ties = k;
#pragma unroll
  for (int level = 0; level < 2; ++level) {
    cnt.zero();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (u >= nv) break;  // block-uniform
      const uint32_t kw[4] = {topk_key2<CODEC>(v[u].x), topk_key2<CODEC>(v[u].y), topk_key2<CODEC>(v[u].z),
                              topk_key2<CODEC>(v[u].w)};
      const uint32_t in = tk_in(e0 + u * 8, n);
      if (level == 0) tk_count8<0>(cnt, kw, in, 0u);
      else tk_count8<1>(cnt, kw, in, thr);
    }
    const int c = cnt.flush();
    if (threadIdx.x < 256) s_c[threadIdx.x] = c;
    __syncthreads();
    tk_pick<WARPS>(s_c, ties, sw, s_pick);
    thr = (thr << 8) | (uint32_t)s_pick[0];
    ties -= s_pick[1];
    __syncthreads();
  }
  unsigned long long am = 0, qm = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const uint32_t kw[4] = {topk_key2<CODEC>(v[u].x), topk_key2<CODEC>(v[u].y), topk_key2<CODEC>(v[u].z),
                            topk_key2<CODEC>(v[u].w)};
    const uint32_t in = u < nv ? tk_in(e0 + u * 8, n) : 0u;
    const uint32_t t2 = thr | (thr << 16);
    const uint32_t ge = tk_ge8(kw, t2) & in;
    const uint32_t gt = thr < 0xFFFFu ? tk_ge8(kw, t2 + 0x00010001u) & in : 0u;
    am |= (unsigned long long)gt << (8 * u);
    qm |= (unsigned long long)(ge ^ gt) << (8 * u);
  }
  int tot;
  const int ca = __popcll(am), cq = __popcll(qm);
  const int ia = tk_block_incl<WARPS>(ca, sw, &tot);
  int lq = tk_block_incl<WARPS>(cq, sw, &tot) - cq, la = ia - ca;
  unsigned long long m = am | qm;
  while (m) {
    const int j = __ffsll((long long)m) - 1;
    m &= m - 1;
    const bool above = (am >> j) & 1ull;
    if (above || lq < ties) {
      const int o = la + (lq < ties ? lq : ties);
      out[o] = x[e0 + j];
      idx_out[o] = e0 + j;
    }
    la += above;
    lq += !above;
  }
}

// ---------------------------------------------------------------------------
// Host side.
static size_t tk_align(size_t b) { return (b + 255) & ~(size_t)255; }

struct TopkPlan {
  int64_t steps;
  int ctas;
  int64_t cta_steps;
  int warp_steps;
  bool collect;
  int rank;
  size_t off_mask, off_warp, off_cta, bytes;
};

constexpr int64_t kTkCollectMin = 1 << 18;
constexpr size_t kTkHead = 256 + (kTkBins + 512) * sizeof(unsigned);  // state and bins, zeroed for every call

static TopkPlan tk_plan(int64_t n, int64_t k) {
  TopkPlan t{};
  t.steps = (n + kTkStep - 1) / kTkStep;
  int64_t c = (int64_t)sm_count() * kTkCtasPerSm;
  const int64_t need = (t.steps + kTkWarps * kTkUnroll - 1) / (kTkWarps * kTkUnroll);
  if (need < c) c = need < 1 ? 1 : need;
  t.cta_steps = (t.steps + c - 1) / c;
  t.warp_steps = (int)((t.cta_steps + kTkWarps - 1) / kTkWarps);
  t.ctas = (int)((t.steps + t.cta_steps - 1) / t.cta_steps);
  t.off_mask = tk_align(kTkHead);
  t.off_warp = t.off_mask + tk_align((size_t)t.steps * 32);
  t.off_cta = t.off_warp + tk_align((size_t)t.ctas * kTkWarps * sizeof(int2));
  t.bytes = t.off_cta + tk_align((size_t)t.ctas * sizeof(int2));
  // The sample bounds t when k is a small part of n: at k = n / 32 about 7 %
  // of x are candidates and the sampled form takes 60 us at 20 Mi elements
  // against 104 us for the histograms at k = n / 8.  Below kTkCollectMin both
  // forms are bound by their launches (30 us at 2^18).
  const double mu = (double)kTkSamples * (double)k / (double)n;
  t.collect = n >= kTkCollectMin && k <= n / 32;
  double s = 1.0;  // sqrt(mu) from above by Newton's steps (mu <= 32)
  for (int i = 0; i < 12; ++i) s = 0.5 * (s + mu / s);
  t.rank = (int)(mu + 6.0 * s + 8.0);
  return t;
}

template <int CODEC, bool VEC>
static tcu_status_t topk_run(TopkParams p, const TopkPlan& t, cudaStream_t st) {
  static DeviceSet opted;
  cudaError_t e = allow_smem(opted, 65536, topk_hist_kernel<CODEC, 0, VEC>, topk_hist_kernel<CODEC, 1, VEC>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(topk)");
  e = cudaMemsetAsync(p.st, 0, kTkHead, st);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(topk state)");
  int64_t hist = (int64_t)sm_count() * kTkHistCtasPerSm;
  const int64_t need = (p.n + kTkThreads * 32 - 1) / (kTkThreads * 32);
  if (need < hist) hist = need;
  if (t.collect) topk_collect_kernel<CODEC, VEC><<<t.ctas, kTkThreads, 0, st>>>(p);
  topk_hist_kernel<CODEC, 0, VEC><<<(int)hist, kTkThreads, 65536, st>>>(p);
  topk_hist_kernel<CODEC, 1, VEC><<<(int)hist, kTkThreads, 65536, st>>>(p);
  topk_count_kernel<CODEC, VEC><<<t.ctas, kTkThreads, 0, st>>>(p);
  topk_emit_kernel<CODEC><<<t.ctas, kTkThreads, 0, st>>>(p);
  e = cudaGetLastError();
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "topk launch");
}

template <int CODEC, bool VEC>
static tcu_status_t topk_small(const uint16_t* x, int n, int k, uint16_t* out, int* idx_out, cudaStream_t st) {
  constexpr int smem = kTkSmallThreads * 256;
  static DeviceSet opted;
  cudaError_t e = allow_smem(opted, smem, topk_small_kernel<CODEC, VEC>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(topk)");
  topk_small_kernel<CODEC, VEC><<<1, kTkSmallThreads, smem, st>>>(x, n, k, out, idx_out);
  e = cudaGetLastError();
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "topk launch");
}

template <int CODEC>
static tcu_status_t topk_t(const uint16_t* x, int64_t n, int64_t k, uint16_t* out, int* idx_out, uint8_t* tmp,
                           cudaStream_t st) {
  if (n <= kTkSmall)
    return aligned16(x) ? topk_small<CODEC, true>(x, (int)n, (int)k, out, idx_out, st)
                        : topk_small<CODEC, false>(x, (int)n, (int)k, out, idx_out, st);
  const TopkPlan t = tk_plan(n, k);
  TopkParams p{};
  p.x = x;
  p.n = n;
  p.k = k;
  p.steps = t.steps;
  p.cta_steps = t.cta_steps;
  p.warp_steps = t.warp_steps;
  p.rank = t.rank;
  p.force_robust = t.collect ? 0 : 1;
  p.st = reinterpret_cast<TopkState*>(tmp);
  p.bins = reinterpret_cast<unsigned*>(tmp + 256);
  p.mask = reinterpret_cast<uint32_t*>(tmp + t.off_mask);
  p.warp_cnt = reinterpret_cast<int2*>(tmp + t.off_warp);
  p.cta_cnt = reinterpret_cast<int2*>(tmp + t.off_cta);
  p.out = out;
  p.idx_out = idx_out;
  return aligned16(x) ? topk_run<CODEC, true>(p, t, st) : topk_run<CODEC, false>(p, t, st);
}

}  // namespace tcu

using namespace tcu;

extern "C" {

size_t tcu_topk_tmp_bytes(int64_t n) { return n <= 0 ? 0 : tk_plan(n, 1).bytes; }

tcu_status_t tcu_topk(const void* x, tcu_dtype_t dtype, int64_t n, int64_t k, void* out, int32_t* idx_out, void* tmp,
                      size_t tmp_bytes, void* stream) {
  if (n < 0 || n > 0x7FFFFFFFLL || k < 0 || k > n) return TCU_ERR_ARG;
  if (dtype != TCU_INT16 && dtype != TCU_FLOAT16 && dtype != TCU_BFLOAT16) return TCU_ERR_DTYPE;
  if (k == 0) return TCU_OK;
  if (!x || !out || !idx_out) return TCU_ERR_ARG;
  if (!tmp || tmp_bytes < tcu_topk_tmp_bytes(n)) return TCU_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(tmp) & 255u) || (reinterpret_cast<uintptr_t>(idx_out) & 3u) ||
      (reinterpret_cast<uintptr_t>(x) & 1u) || (reinterpret_cast<uintptr_t>(out) & 1u))
    return TCU_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  const uint16_t* xs = static_cast<const uint16_t*>(x);
  uint16_t* o = static_cast<uint16_t*>(out);
  uint8_t* t = static_cast<uint8_t*>(tmp);
  if (dtype == TCU_INT16) return topk_t<kTopkInt16>(xs, n, k, o, idx_out, t, st);
  if (dtype == TCU_FLOAT16) return topk_t<kTopkFp16>(xs, n, k, o, idx_out, t, st);
  return topk_t<kTopkBf16>(xs, n, k, o, idx_out, t, st);
}

}  // extern "C"
