// tcu_compress.cu -- stream compaction on B200.
//
// Reference: run_compress / run_compress_pos / run_compress_ind /
// run_compress_ind_no_arange (src/torch/torch_compress.h:41-309) count the
// mask per block with reduce_tiles, read the total back to the host, then
// gather with the vector GatherMask instruction (kernel_compress.h:97-208).
//
// Compaction is byte/integer work bound by HBM, so it stays on the SIMT cores
// (no tensor-core reshaping).  Three launches, each a pure stream with no
// waiting between CTAs:
//   cmp_count_kernel    four 2048-element tiles per warp: the selected elements,
//                       each tile's offset inside its group of 32 tiles and
//                       the group's total -- and, where the caller gave scratch
//                       for it, the mask as one bit per element;
//   cmp_groups_kernel   one CTA: the exclusive int64 scan of the group totals;
//   compact_kernel      one warp per tile: 16-byte loads of the values, the
//                       selection bits, a warp scan, the selected elements
//                       compacted in the warp's own shared memory and written
//                       with 16-byte stores.  No barrier wider than a warp.
// The compaction reads bits and not mask bytes where it can: the 2^28-element
// mask is 268 MB and its bits 34 MB, which stay in L2 between the passes.
// run_compress needs the count on the host before it can size its output, so
// the count pass is work it has to do anyway; a single-pass look-back variant
// was measured slower (every tile waited on its predecessors' counts).
//
// Measured on B200, mask Bernoulli(0.3), count read back included, 2^28
// elements (before: TMA-staged tiles of 64-element rows, one persistent CTA per
// SM, mask bytes read twice): fp16 208 us (288), fp16 positions 320 us (372),
// fp16 split 265 us (430).  The compaction takes 9 instructions per 32 fp16
// elements (14 before, at half the issue rate) and moves its 732 MB at about
// 5.4 TB/s; the count reads the mask at about 5.5 TB/s.
//
// Without bit scratch (the entry points that take a look-back workspace) the
// counts and offsets live in the workspace's descriptor region and are zeroed
// after use: the region must hold only look-back descriptors or zeros between
// launches.
#include <cuda_runtime.h>

#include <cstdio>

#include "tcu_host.h"

namespace tcu {

constexpr int kCmpTile = 2048;                // elements of one warp
constexpr int kCmpWarps = 8;                  // warps per CTA
constexpr int kCmpGroup = 4 * kCmpWarps;      // tiles of a group: one CTA of the count, one total to scan
constexpr int kCmpThreads = 32 * kCmpWarps;
constexpr int kCmpStage = 8192;               // bytes of staged elements per warp, at most

template <int EB>
struct ElemT;
template <>
struct ElemT<1> { using T = uint8_t; };
template <>
struct ElemT<2> { using T = uint16_t; };
template <>
struct ElemT<4> { using T = uint32_t; };
template <>
struct ElemT<8> { using T = unsigned long long; };

struct CompactParams {
  const void* x;
  const int8_t* mask;    // read when there are no bits
  const uint8_t* bits;   // bit e of byte e / 8
  const void* idx_in;    // gathered indices (IDX 1)
  void* out;
  void* idx_out;
  int64_t n;
  int64_t capacity;      // elements the outputs can hold (compress_pos output_len)
  int64_t groups;
  const long long* group_off;  // [groups + 1], the total last
  const int* tile_off;         // inside the group
};

// A warp takes its tile in parts of SUB elements: U vectors of 16 bytes per
// lane, as many as fit the staging area and, with gathered indices, about 10
// vectors of values and indices in registers.
template <int EB, int IDX, int IB, bool SPLIT>
struct CmpCfg {
  static constexpr int EPV = 16 / EB;  // elements of a vector
  static constexpr int IBX = IDX ? IB : 0;
  static constexpr int fit(int u) {
    return u > 1 && (u * 32 * EPV > kCmpTile || u * 32 * EPV * (EB + IBX) > kCmpStage ||
                     (IDX == 1 && u * (EB + IB) > 10 * EB))
               ? fit(u / 2)
               : u;
  }
  static constexpr int U = fit(8);
  static constexpr int SUB = U * 32 * EPV;
  // 16-byte aligned areas; a run starts up to 15 bytes in, so that it lies in
  // shared memory as it does in the output
  static constexpr int X_BYTES = SUB * EB + 64;
  static constexpr int I_BYTES = IBX ? SUB * IBX + 64 : 0;
  static constexpr int SMEM = kCmpWarps * (X_BYTES + I_BYTES);
  // Values alone run faster with 64 registers and four CTAs per SM than with
  // the 63 to 109 they ask for, spills of up to 100 bytes included (512 MB of
  // values, mask 0.3, the compaction kernel alone): 2 bytes 131 against 135 us
  // and split 203 against 213, 4 bytes 109 against 128 and split 179 against
  // 193, 8 bytes 107 against 110; at mask 0.9 195 against 194, 160 against 176
  // and 163 against 162.  The 8-byte split does not (183 against 173 us), nor
  // do one-byte values (162 -> 172 us for a whole call) and most forms with
  // indices (fp32 positions: 395 -> 450 us): they take the registers they ask for.
  static constexpr int MIN_CTAS = IDX == 0 && EB >= 2 && !(EB == 8 && SPLIT) ? 4 : 0;  // 0: no bound
  static_assert(kCmpTile % SUB == 0, "parts of a tile");
};

// Element j of a run of 16-byte vectors held in registers (constant j after
// unrolling, so the extraction is shifts and selects).
template <int EB>
__device__ __forceinline__ typename ElemT<EB>::T vec_elem(const uint4* v, int j) {
  constexpr int PER = 16 / EB;
  const uint4 w = v[j / PER];
  const int b = (j % PER) * EB;  // byte offset inside the vector
  const uint32_t word = (b < 4) ? w.x : (b < 8) ? w.y : (b < 12) ? w.z : w.w;
  if constexpr (EB == 8) {
    const uint32_t hi = (b < 8) ? w.y : w.w;
    return ((unsigned long long)hi << 32) | word;
  } else if constexpr (EB == 4) {
    return word;
  } else {
    return (typename ElemT<EB>::T)(word >> (8 * (b % 4)));
  }
}

// Pushes the selection bits of 4 mask bytes under acc: acc * 16 + bits.  The
// nonzero bytes' top bits meet in the product's upper four bits (no two of its
// terms share a bit), and the funnel shift takes them along: 5 instructions.
__device__ __forceinline__ uint32_t push_sel4(uint32_t acc, uint32_t w) {
  const uint32_t t = (((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) & 0x80808080u;
  return __funnelshift_l(t * 0x00204081u, acc, 4);
}

// Mask bytes -> selection bits: 2, 4, 8 or 16 elements from e (aligned to
// their count).
template <int EPV>
__device__ __forceinline__ uint32_t mask_bits(const int8_t* __restrict__ mask, int64_t e) {
  if constexpr (EPV == 16) {
    const uint4 m = __ldg(reinterpret_cast<const uint4*>(mask + e));
    return push_sel4(push_sel4(push_sel4(push_sel4(0u, m.w), m.z), m.y), m.x);
  } else if constexpr (EPV == 8) {
    const uint2 m = __ldg(reinterpret_cast<const uint2*>(mask + e));
    return push_sel4(push_sel4(0u, m.y), m.x);
  } else if constexpr (EPV == 4) {
    return push_sel4(0u, __ldg(reinterpret_cast<const uint32_t*>(mask + e)));
  } else {
    return push_sel4(0u, (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(mask + e)));
  }
}
// The same from the mask's bits; e is a multiple of EPV.
template <int EPV>
__device__ __forceinline__ uint32_t stored_bits(const uint8_t* __restrict__ bits, int64_t e) {
  if constexpr (EPV == 16) return __ldg(reinterpret_cast<const uint16_t*>(bits + (e >> 3)));
  else if constexpr (EPV == 8) return __ldg(bits + (e >> 3));
  else return ((uint32_t)__ldg(bits + (e >> 3)) >> ((int)e & 7)) & ((1u << EPV) - 1u);
}

// Writes the run s[shift .. shift + len) to dst[g0 .. g0 + len) (positions
// below cap only), one warp.  vec: dst is 16-byte aligned and shift leaves
// g0's remainder modulo a vector, so whole vectors move as such; the few
// elements before the first and behind the last whole vector take one step,
// the first 16 lanes one element each on either side.
template <typename E>
__device__ __forceinline__ void store_run(const E* s, int shift, int len, E* dst, long long g0, long long cap,
                                          bool vec, int lane) {
  constexpr int V = 16 / (int)sizeof(E);
  if (g0 + len > cap) len = cap > g0 ? (int)(cap - g0) : 0;
  if (!vec) {
    for (int i = lane; i < len; i += 32) dst[g0 + i] = s[shift + i];
    return;
  }
  const int end = shift + len;
  dst += g0 - shift;
  const int v0 = (shift + V - 1) & ~(V - 1), v1 = end & ~(V - 1);  // whole vectors: [v0, v1)
  for (int i = v0 + lane * V; i < v1; i += 32 * V)
    *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(s + i);
  const int i = lane < 16 ? (shift & ~(V - 1)) + lane : v1 + lane - 16;
  const bool head = lane < 16 && i >= shift && i < (v0 < end ? v0 : end);
  const bool tail = lane >= 16 && i >= v0 && i < end;
  if (head || tail) dst[i] = s[i];
}

// Where bit j of b is set: stores v at the shared address and moves it on.
// Three instructions an element (test, store, add); the compiler's form of the
// same loop took about nine.
template <typename E>
__device__ __forceinline__ void push_if(uint32_t b, uint32_t bit, uint32_t& addr, E v) {
  if constexpr (sizeof(E) == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u8 [%0], %1;\n\t@p add.u32 %0, %0, 1;\n\t}"
        : "+r"(addr) : "r"((uint32_t)v), "r"(b & bit) : "memory");
  else if constexpr (sizeof(E) == 2)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u16 [%0], %1;\n\t@p add.u32 %0, %0, 2;\n\t}"
        : "+r"(addr) : "h"((uint16_t)v), "r"(b & bit) : "memory");
  else if constexpr (sizeof(E) == 4)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u32 [%0], %1;\n\t@p add.u32 %0, %0, 4;\n\t}"
        : "+r"(addr) : "r"((uint32_t)v), "r"(b & bit) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.u64 [%0], %1;\n\t@p add.u32 %0, %0, 8;\n\t}"
        : "+r"(addr) : "l"((unsigned long long)v), "r"(b & bit) : "memory");
}

// IDX: 0 none, 1 gather idx_in (IB bytes), 2 positions (int32 when IB == 4,
// int64 when IB == 8).  SPLIT: stable partition instead of compaction -- every
// element is written, the selected ones at their compaction offsets and the
// others after all selected ones (at total + the unselected elements before
// them), so a part writes two runs.  Bound by HBM: see the file comment.
template <int EB, int IDX, int IB, bool SPLIT, bool BITS>
__global__ void __launch_bounds__(kCmpThreads, (CmpCfg<EB, IDX, IB, SPLIT>::MIN_CTAS)) compact_kernel(const CompactParams p) {
  using C = CmpCfg<EB, IDX, IB, SPLIT>;
  using T = typename ElemT<EB>::T;
  using I = typename ElemT<(IB > 0 ? IB : 4)>::T;
  constexpr int EPV = C::EPV, U = C::U, SUB = C::SUB, V = 16 / EB, VI = 16 / (int)sizeof(I);
  constexpr int IW = IDX == 1 ? EPV * IB / 4 : 1;  // index words of a vector
  extern __shared__ __align__(16) uint8_t smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t tile = (int64_t)blockIdx.x * kCmpWarps + w;
  const int64_t tile0 = tile * kCmpTile;
  if (tile0 >= p.n) return;  // warp-uniform; the warps of a CTA never meet
  T* sx = reinterpret_cast<T*>(smem + w * (C::X_BYTES + C::I_BYTES));
  I* si = reinterpret_cast<I*>(smem + w * (C::X_BYTES + C::I_BYTES) + C::X_BYTES);
  const T* x = static_cast<const T*>(p.x);
  T* out = static_cast<T*>(p.out);
  I* iout = static_cast<I*>(p.idx_out);
  const bool ivec = IDX != 0 && (reinterpret_cast<uintptr_t>(iout) & 15u) == 0;
  long long pre = p.group_off[tile / kCmpGroup] + p.tile_off[tile];  // selected elements before this part
  const long long all = SPLIT ? p.group_off[p.groups] : 0;
#pragma unroll 1
  for (int64_t s0 = tile0; s0 < tile0 + kCmpTile && s0 < p.n; s0 += SUB) {
    uint32_t b[U];
    uint4 v[U];
    uint32_t iw[U][IW];
    const int64_t e0 = s0 + lane * EPV;  // element 0 of vector 0; vector u is 32 * EPV * u further
    const int room = p.n - s0 < SUB ? (int)(p.n - s0) : SUB;
    if (room == SUB) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t e = e0 + u * 32 * EPV;
        b[u] = BITS ? stored_bits<EPV>(p.bits, e) : mask_bits<EPV>(p.mask, e);
        v[u] = __ldg(reinterpret_cast<const uint4*>(x + e));
        if constexpr (IDX == 1) {
          if constexpr (IW >= 4) {
#pragma unroll
            for (int k = 0; k < IW / 4; ++k) {
              const uint4 q = __ldg(reinterpret_cast<const uint4*>(static_cast<const I*>(p.idx_in) + e) + k);
              iw[u][4 * k] = q.x;
              iw[u][4 * k + 1] = q.y;
              iw[u][4 * k + 2] = q.z;
              iw[u][4 * k + 3] = q.w;
            }
          } else {
            const uint2 q = __ldg(reinterpret_cast<const uint2*>(static_cast<const I*>(p.idx_in) + e));
            iw[u][0] = q.x;
            iw[u][1] = q.y;
          }
        }
      }
    } else {  // the ragged end of the input: element loads
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t e = e0 + u * 32 * EPV;
        uint32_t wd[4] = {0u, 0u, 0u, 0u};
        b[u] = 0;
#pragma unroll
        for (int k = 0; k < IW; ++k) iw[u][k] = 0;
#pragma unroll
        for (int j = 0; j < EPV; ++j) {
          if (e + j < p.n) {
            const bool on = BITS ? (p.bits[(e + j) >> 3] >> (int)((e + j) & 7)) & 1 : p.mask[e + j] != 0;
            b[u] |= (uint32_t)on << j;
            const T t = x[e + j];
            if constexpr (EB == 8) {
              wd[2 * j] = (uint32_t)t;
              wd[2 * j + 1] = (uint32_t)(t >> 32);
            } else {
              wd[j * EB / 4] |= (uint32_t)t << (8 * (j * EB % 4));
            }
            if constexpr (IDX == 1) {
              const I t2 = static_cast<const I*>(p.idx_in)[e + j];
              if constexpr (IB == 8) {
                iw[u][2 * j] = (uint32_t)t2;
                iw[u][2 * j + 1] = (uint32_t)(t2 >> 32);
              } else {
                iw[u][j] = (uint32_t)t2;
              }
            }
          }
        }
        v[u] = make_uint4(wd[0], wd[1], wd[2], wd[3]);
      }
    }
    // ---- offsets of every lane's vectors inside the part: warp scans of the
    // counts, up to three vectors to a register (10 bits each: at most 512) ----
    int off[U], total = 0;
    constexpr int PK = EPV == 16 ? 2 : 3, SH = EPV == 16 ? 16 : 10;
#pragma unroll
    for (int u0 = 0; u0 < U; u0 += PK) {
      uint32_t c = 0;
#pragma unroll
      for (int k = 0; k < PK; ++k)
        if (u0 + k < U) c |= (uint32_t)__popc(b[u0 + k < U ? u0 + k : 0]) << (SH * k);
      uint32_t inc = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
      inc -= c;
#pragma unroll
      for (int k = 0; k < PK; ++k) {
        if (u0 + k < U) {
          off[u0 + k < U ? u0 + k : 0] = total + (int)((inc >> (SH * k)) & ((1u << SH) - 1u));
          total += (int)((tot >> (SH * k)) & ((1u << SH) - 1u));
        }
      }
    }
    // ---- where the runs start in shared memory ----
    const long long ug0 = all + s0 - pre;  // SPLIT: the part's first unselected element in the output
    const int xs = (int)(pre & (V - 1)), is = ivec ? (int)(pre & (VI - 1)) : 0;
    const int xu = SPLIT ? ((xs + total + V - 1) & ~(V - 1)) + (int)(ug0 & (V - 1)) : 0;
    const int iu = SPLIT ? ((is + total + VI - 1) & ~(VI - 1)) + (ivec ? (int)(ug0 & (VI - 1)) : 0) : 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l0 = u * 32 * EPV + lane * EPV;  // the vector's first element in the part
      uint32_t ax = smem_u32(sx + xs + off[u]), ai = smem_u32(si + is + off[u]);
      [[maybe_unused]] uint32_t cx = smem_u32(sx + xu + l0 - off[u]), ci = smem_u32(si + iu + l0 - off[u]);
      // SPLIT: the unselected elements inside the input
      [[maybe_unused]] const uint32_t nb =
          ~b[u] & (l0 + EPV <= room ? 0xFFFFu : (l0 >= room ? 0u : (1u << (room - l0)) - 1u));
#pragma unroll
      for (int j = 0; j < EPV; ++j) {
        const T t = vec_elem<EB>(&v[u], j);
        push_if<T>(b[u], 1u << j, ax, t);
        if constexpr (SPLIT) push_if<T>(nb, 1u << j, cx, t);
        if constexpr (IDX != 0) {
          I i;
          if constexpr (IDX == 2) i = (I)(s0 + l0 + j);
          else if constexpr (IB == 8) i = ((unsigned long long)iw[u][2 * j + 1] << 32) | iw[u][2 * j];
          else i = iw[u][j];
          push_if<I>(b[u], 1u << j, ai, i);
          if constexpr (SPLIT) push_if<I>(nb, 1u << j, ci, i);
        }
      }
    }
    __syncwarp();
    store_run<T>(sx, xs, total, out, pre, p.capacity, true, lane);
    if constexpr (IDX != 0) store_run<I>(si, is, total, iout, pre, p.capacity, ivec, lane);
    if constexpr (SPLIT) {
      store_run<T>(sx, xu, room - total, out, ug0, p.capacity, true, lane);
      if constexpr (IDX != 0) store_run<I>(si, iu, room - total, iout, ug0, p.capacity, ivec, lane);
    }
    __syncwarp();  // the staging area is reused
    pre += total;
  }
}

// Selected elements of every tile (mask != 0): the tile's offset inside its
// group (one CTA), the group's total, and the mask's bits (bits != nullptr;
// zero past the end).
__global__ void __launch_bounds__(kCmpThreads) cmp_count_kernel(const int8_t* __restrict__ mask, int64_t n,
                                                                int64_t tiles, int* __restrict__ tile_off,
                                                                long long* __restrict__ group_tot,
                                                                uint16_t* __restrict__ bits) {
  __shared__ int s_c[kCmpGroup];
  constexpr int NV = kCmpTile / 512;  // 16-byte vectors per lane
  constexpr int TPW = kCmpGroup / kCmpWarps;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t t0 = (int64_t)blockIdx.x * kCmpGroup;
#pragma unroll
  for (int k0 = 0; k0 < TPW; k0 += 2) {  // two tiles in flight
    const int64_t e0 = (t0 + w * TPW + k0) * kCmpTile;
    uint32_t b[2 * NV];
    if (e0 + 2 * kCmpTile <= n) {  // warp-uniform
#pragma unroll
      for (int v = 0; v < 2 * NV; ++v) b[v] = mask_bits<16>(mask, e0 + (v * 32 + lane) * 16);
    } else {
#pragma unroll
      for (int v = 0; v < 2 * NV; ++v) {
        b[v] = 0;
        const int64_t e = e0 + (v * 32 + lane) * 16;
        for (int j = 0; j < 16; ++j)
          if (e + j < n) b[v] |= (uint32_t)(mask[e + j] != 0) << j;
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      int c = 0;
#pragma unroll
      for (int v = 0; v < NV; v += 2) c += __popc(b[k * NV + v] | (b[k * NV + v + 1] << 16));
      if (bits && e0 + k * kCmpTile < n) {
#pragma unroll
        for (int v = 0; v < NV; ++v) bits[((e0 + k * kCmpTile) >> 4) + v * 32 + lane] = (uint16_t)b[k * NV + v];
      }
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) s_c[w * TPW + k0 + k] = c;
    }
  }
  __syncthreads();
  if (w == 0) {  // kCmpGroup == 32: one tile per lane
    const int c = s_c[lane];
    int inc = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    if (t0 + lane < tiles) tile_off[t0 + lane] = inc - c;
    if (lane == 31) group_tot[blockIdx.x] = inc;
  }
}
static_assert(kCmpGroup == 32, "a lane per tile of the group");

// Exclusive scan of the group totals in place (one CTA; 4096 groups at 2^28
// elements), the total behind them and, when given, in *count_out.
__global__ void __launch_bounds__(1024) cmp_groups_kernel(long long* __restrict__ group_off, int64_t groups,
                                                          long long* count_out) {
  __shared__ long long s_w[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  long long carry = 0;
  constexpr int PER = 4;
  for (int64_t b = 0; b < groups; b += 1024 * PER) {  // block-uniform
    const int64_t i0 = b + (int64_t)threadIdx.x * PER;
    long long v[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      v[i] = i0 + i < groups ? group_off[i0 + i] : 0;
      sum += v[i];
    }
    long long inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const long long o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    if (lane == 31) s_w[wid] = inc;
    __syncthreads();
    long long ws = s_w[lane], winc = ws;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const long long o = __shfl_up_sync(0xffffffffu, winc, d);
      if (lane >= d) winc += o;
    }
    long long run = carry + __shfl_sync(0xffffffffu, winc - ws, wid) + inc - sum;
    carry += __shfl_sync(0xffffffffu, winc, 31);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (i0 + i < groups) group_off[i0 + i] = run;
      run += v[i];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    group_off[groups] = carry;
    if (count_out) *count_out = carry;
  }
}

// Output position of every segment start: the number of selected elements
// before it = the offset of its tile + the selected elements between the tile
// start and the segment start.  One warp per segment start.
__global__ void __launch_bounds__(256) seg_positions_kernel(const int8_t* __restrict__ mask, int64_t n,
                                                            const long long* __restrict__ starts, int64_t nseg,
                                                            const long long* __restrict__ group_off,
                                                            const int* __restrict__ tile_off, int64_t tiles,
                                                            int64_t groups, long long* __restrict__ pos) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (i >= nseg) return;  // warp-uniform
  long long s = starts[i];
  s = s < 0 ? 0 : (s > n ? n : s);
  const int64_t t = s / kCmpTile;
  const long long base = t < tiles ? group_off[t / kCmpGroup] + tile_off[t] : group_off[groups];
  const int64_t e0 = t * kCmpTile;
  const int64_t len = s - e0;
  const int64_t nv = len / 16;
  const uint4* mv = reinterpret_cast<const uint4*>(mask + e0);
  unsigned long long c = 0;
  for (int64_t v = lane; v < nv; v += 32) {
    const uint4 w = __ldg(mv + v);
    c += __popc(sel4(w.x) | (sel4(w.y) << 4) | (sel4(w.z) << 8) | (sel4(w.w) << 12));
  }
  for (int64_t e = nv * 16 + lane; e < len; e += 32) c += mask[e0 + e] != 0;
  c = warp_sum_any(c);
  if (lane == 0) pos[i] = base + (long long)c;
}

// Count of mask != 0 (the reference's reduce_tiles + .sum() used to size the
// output, src/torch/torch_compress.h:62-64).  *count must be zero on entry.
__global__ void __launch_bounds__(256) mask_count_kernel(const int8_t* mask, int64_t n, unsigned long long* count) {
  unsigned long long c = 0;
  const int64_t nv = n / 16;
  const uint4* mv = reinterpret_cast<const uint4*>(mask);
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
    const uint4 w = __ldg(mv + v);
    c += __popc(sel4(w.x) | (sel4(w.y) << 4) | (sel4(w.z) << 8) | (sel4(w.w) << 12));
  }
  if (blockIdx.x == 0) {
    for (int64_t i = nv * 16 + threadIdx.x; i < n; i += blockDim.x) c += mask[i] != 0;
  }
  c = warp_sum_any(c);
  __shared__ unsigned long long s[8];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tsum = 0;
    for (int k = 0; k < (int)(blockDim.x / 32); ++k) tsum += s[k];
    if (tsum) atomicAdd(count, tsum);
  }
}

// ---------------------------------------------------------------------------
// Host side.  Scratch: group_off[groups + 1] (int64), tile_off[tiles] (int32)
// and, in caller-given scratch only, the mask bits of whole tiles.
struct CmpScratch {
  long long* group_off;
  int* tile_off;
  uint8_t* bits;  // or nullptr
  int64_t tiles;
  int64_t groups;
  size_t bytes;
};

static void cmp_layout(int64_t n, bool bits, uint8_t* base, CmpScratch* sc) {
  sc->tiles = (n + kCmpTile - 1) / kCmpTile;
  sc->groups = (sc->tiles + kCmpGroup - 1) / kCmpGroup;
  const size_t tile_at = (size_t)(sc->groups + 1) * 8;
  const size_t bits_at = (tile_at + (size_t)sc->tiles * 4 + 15) & ~(size_t)15;
  sc->bytes = bits ? bits_at + (size_t)sc->tiles * (kCmpTile / 8) : bits_at;
  sc->group_off = reinterpret_cast<long long*>(base);
  sc->tile_off = reinterpret_cast<int*>(base + tile_at);
  sc->bits = bits ? base + bits_at : nullptr;
}

// Counts and offsets in a look-back workspace.
static tcu_status_t cmp_scratch(void* ws, size_t ws_bytes, int64_t n, CmpScratch* sc) {
  if (!ws) return TCU_ERR_WORKSPACE;
  cmp_layout(n, false, reinterpret_cast<uint8_t*>(ws_descs(ws)), sc);
  if (ws_bytes < 128 + sc->bytes || ws_capacity(ws_bytes) * 16 < (int64_t)sc->bytes) return TCU_ERR_WORKSPACE;
  return TCU_OK;
}

// Counts, offsets and bits in scratch of tcu_compact_tmp_bytes(n) bytes.
static tcu_status_t cmp_tmp(void* tmp, size_t tmp_bytes, int64_t n, CmpScratch* sc) {
  if (!tmp) return TCU_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(tmp) & 15u) return TCU_ERR_ALIGN;
  cmp_layout(n, true, static_cast<uint8_t*>(tmp), sc);
  return tmp_bytes < sc->bytes ? TCU_ERR_WORKSPACE : TCU_OK;
}

static tcu_status_t cmp_clear(void* ws, const CmpScratch& sc, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(ws_descs(ws), 0, sc.bytes, st);
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "cudaMemsetAsync(compress scratch)");
}

static tcu_status_t cmp_count(const int8_t* mask, int64_t n, const CmpScratch& sc, long long* count_out,
                              cudaStream_t st) {
  if (sc.groups > 0x7FFFFFFF) return TCU_ERR_ARG;
  cmp_count_kernel<<<(unsigned)sc.groups, kCmpThreads, 0, st>>>(mask, n, sc.tiles, sc.tile_off, sc.group_off,
                                                               reinterpret_cast<uint16_t*>(sc.bits));
  cmp_groups_kernel<<<1, 1024, 0, st>>>(sc.group_off, sc.groups, count_out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "compress count launch");
}

template <int EB, int IDX, int IB, bool SPLIT, bool BITS>
static tcu_status_t launch_compact(const CompactParams& p, cudaStream_t st) {
  using C = CmpCfg<EB, IDX, IB, SPLIT>;
  auto kern = compact_kernel<EB, IDX, IB, SPLIT, BITS>;
  static DeviceSet opted;
  cudaError_t e = allow_smem(opted, C::SMEM, kern);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(compress)");
  const int64_t ctas = ((p.n + kCmpTile - 1) / kCmpTile + kCmpWarps - 1) / kCmpWarps;
  if (ctas > 0x7FFFFFFF) return TCU_ERR_ARG;
  kern<<<(unsigned)ctas, kCmpThreads, C::SMEM, st>>>(p);
  e = cudaGetLastError();
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "compact_kernel launch");
}

static tcu_status_t cmp_check(const void* x, int elem_bytes, const void* mask, const void* idx_in, int idx_bytes,
                              int idx_mode, const void* out, const void* idx_out) {
  if (!x || !mask || !out) return TCU_ERR_ARG;
  if (!aligned16(x) || !aligned16(mask) || !aligned16(out)) return TCU_ERR_ALIGN;
  if (idx_mode < 0 || idx_mode > 2) return TCU_ERR_ARG;
  if (idx_mode != 0 && (!idx_out || (idx_bytes != 4 && idx_bytes != 8))) return TCU_ERR_ARG;
  if (idx_mode == 1 && (!idx_in || !aligned16(idx_in))) return idx_in ? TCU_ERR_ALIGN : TCU_ERR_ARG;
  if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return TCU_ERR_DTYPE;
  return TCU_OK;
}

template <int EB, bool BITS>
static tcu_status_t compact_elem(const CompactParams& p, int idx_bytes, int idx_mode, bool split, cudaStream_t st) {
  if (split) {  // stable partition: values only or with gathered indices
    if (idx_mode == 0) return launch_compact<EB, 0, 0, true, BITS>(p, st);
    if (idx_mode == 2) return TCU_ERR_ARG;
    return idx_bytes == 4 ? launch_compact<EB, 1, 4, true, BITS>(p, st) : launch_compact<EB, 1, 8, true, BITS>(p, st);
  }
  if (idx_mode == 0) return launch_compact<EB, 0, 0, false, BITS>(p, st);
  if (idx_mode == 1)
    return idx_bytes == 4 ? launch_compact<EB, 1, 4, false, BITS>(p, st) : launch_compact<EB, 1, 8, false, BITS>(p, st);
  return idx_bytes == 4 ? launch_compact<EB, 2, 4, false, BITS>(p, st) : launch_compact<EB, 2, 8, false, BITS>(p, st);
}

template <bool BITS>
static tcu_status_t compact_dispatch(const CompactParams& p, int elem_bytes, int idx_bytes, int idx_mode, bool split,
                                     cudaStream_t st) {
  switch (elem_bytes) {
    case 1: return compact_elem<1, BITS>(p, idx_bytes, idx_mode, split, st);
    case 2: return compact_elem<2, BITS>(p, idx_bytes, idx_mode, split, st);
    case 4: return compact_elem<4, BITS>(p, idx_bytes, idx_mode, split, st);
    default: return compact_elem<8, BITS>(p, idx_bytes, idx_mode, split, st);
  }
}

// The compaction pass, with the counts and offsets already in the scratch.
static tcu_status_t cmp_run(const void* x, int elem_bytes, const int8_t* mask, int64_t n, const void* idx_in,
                            int idx_bytes, int idx_mode, void* out, void* idx_out, int64_t capacity,
                            const CmpScratch& sc, cudaStream_t st, bool split = false) {
  CompactParams p{};
  p.x = x;
  p.mask = mask;
  p.bits = sc.bits;
  p.idx_in = idx_in;
  p.out = out;
  p.idx_out = idx_out;
  p.n = n;
  p.capacity = capacity;
  p.groups = sc.groups;
  p.group_off = sc.group_off;
  p.tile_off = sc.tile_off;
  if (sc.groups > 0x7FFFFFFF) return TCU_ERR_ARG;
  return sc.bits ? compact_dispatch<true>(p, elem_bytes, idx_bytes, idx_mode, split, st)
                 : compact_dispatch<false>(p, elem_bytes, idx_bytes, idx_mode, split, st);
}

static tcu_status_t zero_count(void* count_dev, cudaStream_t st) {
  if (!count_dev) return TCU_OK;
  cudaError_t e = cudaMemsetAsync(count_dev, 0, sizeof(long long), st);
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "cudaMemsetAsync(count)");
}

}  // namespace tcu

using namespace tcu;

extern "C" {

tcu_status_t tcu_mask_count(const int8_t* mask, int64_t n, void* count_dev, void* stream) {
  if (n < 0 || !count_dev) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(count_dev, 0, sizeof(unsigned long long), st);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(count)");
  if (n == 0) return TCU_OK;
  if (!mask || !aligned16(mask) || !aligned16(count_dev)) return mask ? TCU_ERR_ALIGN : TCU_ERR_ARG;
  int64_t blocks = (n / 16 + 255) / 256;
  const int64_t cap = (int64_t)sm_count() * 4;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  mask_count_kernel<<<(int)blocks, 256, 0, st>>>(mask, n, static_cast<unsigned long long*>(count_dev));
  e = cudaGetLastError();
  return e == cudaSuccess ? TCU_OK : cuda_fail(e, "mask_count_kernel launch");
}

tcu_status_t tcu_compress_count(const int8_t* mask, int64_t n, int elem_bytes, int idx_mode, int idx_bytes,
                                void* count_dev, void* ws, size_t ws_bytes, void* stream) {
  if (n < 0) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) return zero_count(count_dev, st);
  if (!mask) return TCU_ERR_ARG;
  if (!aligned16(mask) || (reinterpret_cast<uintptr_t>(count_dev) & 7u)) return TCU_ERR_ALIGN;
  if (elem_bytes != 1 && elem_bytes != 2 && elem_bytes != 4 && elem_bytes != 8) return TCU_ERR_DTYPE;
  CmpScratch sc;
  tcu_status_t s = cmp_scratch(ws, ws_bytes, n, &sc);
  if (s != TCU_OK) return s;
  return cmp_count(mask, n, sc, static_cast<long long*>(count_dev), st);
}

tcu_status_t tcu_compress_counted(const void* x, int elem_bytes, const int8_t* mask, int64_t n, const void* idx_in,
                                  int idx_bytes, int idx_mode, void* out, void* idx_out, int64_t capacity, void* ws,
                                  size_t ws_bytes, void* stream) {
  if (n < 0 || capacity < 0) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) return TCU_OK;
  tcu_status_t s = cmp_check(x, elem_bytes, mask, idx_in, idx_bytes, idx_mode, out, idx_out);
  if (s != TCU_OK) return s;
  CmpScratch sc;
  s = cmp_scratch(ws, ws_bytes, n, &sc);
  if (s != TCU_OK) return s;
  s = cmp_run(x, elem_bytes, mask, n, idx_in, idx_bytes, idx_mode, out, idx_out, capacity, sc, st);
  if (s != TCU_OK) return s;
  return cmp_clear(ws, sc, st);
}

tcu_status_t tcu_compress(const void* x, int elem_bytes, const int8_t* mask, int64_t n, const void* idx_in,
                          int idx_bytes, int idx_mode, void* out, void* idx_out, int64_t capacity, void* count_dev,
                          void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || capacity < 0) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) return zero_count(count_dev, st);
  tcu_status_t s = cmp_check(x, elem_bytes, mask, idx_in, idx_bytes, idx_mode, out, idx_out);
  if (s != TCU_OK) return s;
  if (reinterpret_cast<uintptr_t>(count_dev) & 7u) return TCU_ERR_ALIGN;
  CmpScratch sc;
  s = cmp_scratch(ws, ws_bytes, n, &sc);
  if (s == TCU_OK) s = cmp_count(mask, n, sc, static_cast<long long*>(count_dev), st);
  if (s == TCU_OK) s = cmp_run(x, elem_bytes, mask, n, idx_in, idx_bytes, idx_mode, out, idx_out, capacity, sc, st);
  if (s != TCU_OK) return s;
  return cmp_clear(ws, sc, st);
}

tcu_status_t tcu_compress_segments(const void* x, int elem_bytes, const int8_t* mask, int64_t n,
                                   const int64_t* seg_starts, int64_t nseg, void* out, int64_t capacity,
                                   int64_t* seg_pos, void* ws, size_t ws_bytes, void* stream) {
  if (n < 0 || nseg < 0 || capacity < 0 || !seg_pos || (nseg > 0 && !seg_starts)) return TCU_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(seg_pos) & 7u) || (reinterpret_cast<uintptr_t>(seg_starts) & 7u))
    return TCU_ERR_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) {
    cudaError_t e = cudaMemsetAsync(seg_pos, 0, (size_t)(nseg + 1) * sizeof(int64_t), st);
    return e == cudaSuccess ? TCU_OK : cuda_fail(e, "cudaMemsetAsync(seg_pos)");
  }
  tcu_status_t s = cmp_check(x, elem_bytes, mask, nullptr, 0, 0, out, nullptr);
  if (s != TCU_OK) return s;
  CmpScratch sc;
  s = cmp_scratch(ws, ws_bytes, n, &sc);
  if (s == TCU_OK) s = cmp_count(mask, n, sc, reinterpret_cast<long long*>(seg_pos + nseg), st);
  if (s == TCU_OK) s = cmp_run(x, elem_bytes, mask, n, nullptr, 0, 0, out, nullptr, capacity, sc, st);
  if (s != TCU_OK) return s;
  if (nseg > 0) {
    const int64_t blocks = (nseg * 32 + 255) / 256;
    if (blocks > 0x7FFFFFFF) return TCU_ERR_ARG;
    seg_positions_kernel<<<(unsigned)blocks, 256, 0, st>>>(mask, n, reinterpret_cast<const long long*>(seg_starts),
                                                           nseg, sc.group_off, sc.tile_off, sc.tiles, sc.groups,
                                                           reinterpret_cast<long long*>(seg_pos));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "seg_positions_kernel launch");
  }
  return cmp_clear(ws, sc, st);
}

size_t tcu_compact_tmp_bytes(int64_t n) {
  if (n <= 0) return 16;
  CmpScratch sc;
  cmp_layout(n, true, nullptr, &sc);
  return sc.bytes;
}

tcu_status_t tcu_compact_count(const int8_t* mask, int64_t n, void* count_dev, void* tmp, size_t tmp_bytes,
                               void* stream) {
  if (n < 0) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (reinterpret_cast<uintptr_t>(count_dev) & 7u) return TCU_ERR_ALIGN;
  if (n == 0) return zero_count(count_dev, st);
  if (!mask) return TCU_ERR_ARG;
  if (!aligned16(mask)) return TCU_ERR_ALIGN;
  CmpScratch sc;
  tcu_status_t s = cmp_tmp(tmp, tmp_bytes, n, &sc);
  if (s != TCU_OK) return s;
  return cmp_count(mask, n, sc, static_cast<long long*>(count_dev), st);
}

tcu_status_t tcu_compact_counted(const void* x, int elem_bytes, int64_t n, const void* idx_in, int idx_bytes,
                                 int idx_mode, int split, void* out, void* idx_out, int64_t capacity, void* tmp,
                                 size_t tmp_bytes, void* stream) {
  if (n < 0 || capacity < 0 || (split && idx_mode == 2)) return TCU_ERR_ARG;
  if (n == 0) return TCU_OK;
  CmpScratch sc;
  tcu_status_t s = cmp_tmp(tmp, tmp_bytes, n, &sc);
  if (s == TCU_OK) s = cmp_check(x, elem_bytes, tmp, idx_in, idx_bytes, idx_mode, out, idx_out);
  if (s != TCU_OK) return s;
  return cmp_run(x, elem_bytes, nullptr, n, idx_in, idx_bytes, idx_mode, out, idx_out, split ? n : capacity, sc,
                 (cudaStream_t)stream, split != 0);
}

// Stable partition (the reference's run_split / run_split_ind,
// src/torch/torch_split.h:33-79 and :91-142): out[0, k) = x[mask != 0],
// out[k, n) = x[mask == 0], both in input order; with idx_mode 1 the same
// permutation is applied to idx_in.  One count pass, one offset scan, one
// streaming pass that writes both runs of every tile.
tcu_status_t tcu_split(const void* x, int elem_bytes, const int8_t* mask, int64_t n, const void* idx_in, int idx_bytes,
                       int idx_mode, void* out, void* idx_out, void* count_dev, void* ws, size_t ws_bytes,
                       void* stream) {
  if (n < 0) return TCU_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) return zero_count(count_dev, st);
  if (idx_mode != 0 && idx_mode != 1) return TCU_ERR_ARG;
  tcu_status_t s = cmp_check(x, elem_bytes, mask, idx_in, idx_bytes, idx_mode, out, idx_out);
  if (s != TCU_OK) return s;
  if (reinterpret_cast<uintptr_t>(count_dev) & 7u) return TCU_ERR_ALIGN;
  CmpScratch sc;
  s = cmp_scratch(ws, ws_bytes, n, &sc);
  if (s == TCU_OK) s = cmp_count(mask, n, sc, static_cast<long long*>(count_dev), st);
  if (s == TCU_OK) s = cmp_run(x, elem_bytes, mask, n, idx_in, idx_bytes, idx_mode, out, idx_out, n, sc, st, true);
  if (s != TCU_OK) return s;
  return cmp_clear(ws, sc, st);
}

}  // extern "C"
