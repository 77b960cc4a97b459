// Bit-plane passes of the wavelet-tree build (alphabets of up to 2^16 codes).
//
// The level-j order is the text stably sorted by the top j bits of every
// symbol's L-bit code; level j holds bit L-1-j of the codes in that order.
// The build keeps an order as bit planes: plane j of the level-a order is
// the bit array of code bit L-1-j in that order, so plane a of it is level
// a itself.  A pass takes the planes a .. L-1 of the level-a order and
// writes levels a+1 .. a+k (k <= 4), plus the deeper planes of those orders
// that something reads later (the next pass, the group query levels):
//
//   1. ingest_planes_kernel: text -> the planes of the level-0 order (a
//      32 x 8 bit transpose in registers) and the code counts of every tile
//      of the first pass, in one read of the text;
//   2. plane_counts_kernel (later passes, and passes that start with many
//      nodes): the digit counts of every tile from the planes, a digit being
//      the k bits below the node;
//   3. range_totals / digit_starts / chunk_starts kernels: where every
//      digit class starts, and the digits of a node before every chunk of
//      tiles;
//   4. plane_pass_kernel: every tile k times stably partitioned, as bit
//      planes, in shared memory.
//
// Why planes: a stable partition of 32 symbols by one bit moves every plane
// with the same five masked swaps (below), so a plane costs about one thread
// instruction per symbol and level and 1/8 byte of shared memory, where
// moving the symbols as bytes took about 20 instructions and a byte store per
// symbol and level.  6 Gi uint8 symbols, sigma 256 (one GB300): passes 38.6 ->
// 19.6 ms, digit counts 3.6 -> 1.2 ms, whole build 57.6 -> 31.4 ms.
//
// The partition of one slot (128 or 256 consecutive positions of one class)
// by its mask m: an inverse butterfly of stages of distance 1, 2, 4, .. brings
// the elements with m = 1 to the low end in their order and those with m = 0
// to the high end in reversed order.  A stage of distance h swaps
// position q of the left with position q of the right half of each block of
// 2h where bit q of  rotl(1^h 0^h, M) mod 2h  is set, M being the ones of m
// before the right half: the ones take consecutive residues mod 2h starting
// at the number of ones before the block, the zeros the residues below it,
// downwards.  Zeros thus change their direction at every level: the order
// of a class is stored reversed when the number of zero bits in its path
// is odd, and the words are bit-reversed only where they are written out.
//
// The reference re-sorts the whole text with a radix sort per level and
// fills each level from it (wavelet_tree.cuh:806-818, 2422-2493); the bits
// written here are identical.  Words shared by two runs are combined with
// atomicOr, cleared beforehand (clear_edges_kernel); all writes are
// bounds-checked.
#pragma once

#include <algorithm>
#include <functional>
#include <vector>

#include "internal.cuh"

namespace ewt {
namespace {

constexpr uint32_t kMaxPlanes = 16;  // code bits
constexpr uint32_t kMaxPassK = 4;    // levels per pass
constexpr uint32_t kMaxDigits = 16;  // digits of a tile count (up to 4 bits)

// The tiles of one pass: every node [starts[N], starts[N+1]) of the level-a
// order is cut into tiles of `tile` symbols, `ct` consecutive tiles of a
// node make a chunk (the unit a CTA takes), and `rc` consecutive chunks of a
// node a range (a warp's work in the scan of the digit counts).
struct TileGrid {
  uint64_t n;
  uint32_t nodes, D, tile, ct, rc;
  uint32_t halves;          // 1: starts_next has two entries per digit (below)
  uint64_t* starts;         // nodes + 1
  uint32_t* tile_first;     // nodes + 1
  uint32_t* chunk_first;    // nodes + 1
  uint32_t* range_first;    // nodes + 1
  uint16_t* tile_cnt;       // [tile][1 << D]
  uint64_t* chunk_pre;      // [chunk][1 << D]: the digit in the node before
  uint64_t* range_tot;      // [range][1 << D]
  uint64_t* starts_next;    // (nodes << D << halves) + 1
};

// Where digit d of node N starts.  The last pass's digits are the classes of
// the last level, of which plane_pass_kernel counts the ones on its way: the
// second entry of a digit, the start of its ones, begins as the digit's end
// and is lowered by them.  (Counting digits of one bit more beforehand, a
// popcount for each of twice as many classes: digit counts of 6 Gi symbols of
// 256 2.63 -> 1.66 ms, 1.19 since they run as one wave.)
__device__ __forceinline__ uint64_t* digit_start(TileGrid const& g, uint32_t N, uint32_t d) {
  return g.starts_next + ((uint64_t(N) << g.D | d) << g.halves);
}

// The node owning entry i of a non-decreasing table first[0 .. nodes]: the
// last one whose first entry is <= i.
__device__ __forceinline__ uint32_t owner_node(uint32_t const* first, uint32_t nodes,
                                               uint32_t i) {
  uint32_t lo = 0, hi = nodes - 1;
  while (lo < hi) {
    uint32_t const mid = (lo + hi + 1) >> 1;
    if (first[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The tables of a single node, the whole order.
__device__ __forceinline__ void single_node_tables(TileGrid const& g) {
  uint32_t const tiles = static_cast<uint32_t>((g.n + g.tile - 1) / g.tile);
  g.starts[0] = 0;
  g.starts[1] = g.n;
  uint32_t const chunks = (tiles + g.ct - 1) / g.ct;
  g.tile_first[0] = g.chunk_first[0] = g.range_first[0] = 0;
  g.tile_first[1] = tiles;
  g.chunk_first[1] = chunks;
  g.range_first[1] = (chunks + g.rc - 1) / g.rc;
}

// Tiles, chunks and ranges before every node (one CTA).
__global__ void __launch_bounds__(1024)
tile_table_kernel(TileGrid g) {
  __shared__ uint32_t warp_sum[3][32];
  __shared__ uint32_t carry[3];
  uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t* const first[3] = {g.tile_first, g.chunk_first, g.range_first};
  if (tid < 3) carry[tid] = 0;
  __syncthreads();
  for (uint32_t base = 0; base < g.nodes; base += 1024) {
    uint32_t const N = base + tid;
    uint32_t x[3] = {0, 0, 0}, inc[3];
    if (N < g.nodes) {
      uint64_t const len = g.starts[N + 1] - g.starts[N];
      x[0] = static_cast<uint32_t>((len + g.tile - 1) / g.tile);
      x[1] = (x[0] + g.ct - 1) / g.ct;
      x[2] = (x[1] + g.rc - 1) / g.rc;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      uint32_t y = x[i];
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
        uint32_t const z = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) y += z;
      }
      inc[i] = y;
      if (lane == 31) warp_sum[i][wid] = y;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      uint32_t const before =
          carry[i] + __reduce_add_sync(0xffffffffu, lane < wid ? warp_sum[i][lane] : 0u);
      if (N < g.nodes) first[i][N] = before + inc[i] - x[i];
      if (N == g.nodes - 1) first[i][g.nodes] = before + inc[i];
      inc[i] += before;
    }
    __syncthreads();
    if (tid == 1023)
#pragma unroll
      for (int i = 0; i < 3; ++i) carry[i] = inc[i];
    __syncthreads();
  }
}

// Inclusive warp scan (a shuffle's predicate says whether its source lane
// exists).
__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    asm volatile(
        "{ .reg .pred p; .reg .u32 y;\n"
        "shfl.sync.up.b32 y|p, %0, %1, 0, 0xffffffff;\n"
        "@p add.u32 %0, %0, y; }"
        : "+r"(x)
        : "r"(o));
  return x;
}

// ---- transposes ------------------------------------------------------------

// Four words (a, b, c, d): out[i] = byte i of each, in that order.
__device__ __forceinline__ void transpose4(uint32_t a, uint32_t b, uint32_t c,
                                           uint32_t d, uint32_t* out, int stride) {
  uint32_t const t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
  uint32_t const u0 = __byte_perm(c, d, 0x5140), u1 = __byte_perm(c, d, 0x7362);
  out[0] = __byte_perm(t0, u0, 0x5410);
  out[stride] = __byte_perm(t0, u0, 0x7632);
  out[2 * stride] = __byte_perm(t1, u1, 0x5410);
  out[3 * stride] = __byte_perm(t1, u1, 0x7632);
}

// 8 x 8 bit transpose in each of the four byte columns of w[0..7]: bit b of
// byte h of w[i] and bit i of byte h of w[b] change places.
__device__ __forceinline__ void transpose_bits(uint32_t (&w)[8]) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    int const s = 1 << t;
    uint32_t const m = t == 0 ? 0x55555555u : t == 1 ? 0x33333333u : 0x0F0F0F0Fu;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i & s) continue;
      uint32_t const x = ((w[i] >> s) ^ w[i + s]) & m;
      w[i + s] ^= x;
      w[i] ^= x << s;
    }
  }
}

// Digit counters: counter d of lane x at word d * 32 + x (its own bank);
// dw holds a digit in each byte.
__device__ __forceinline__ void count_digits(uint32_t base, uint32_t lane4,
                                             uint32_t dw) {
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    uint32_t const a = (h == 0 ? dw << 7 : dw >> (8 * h - 7)) & 0x7F80u;
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(base + (a | lane4)) : "memory");
  }
}

// A warp writes the counters of 1 << D digits to a row and clears them.
__device__ __forceinline__ void flush_digits(uint32_t* cnt, uint32_t D,
                                             uint16_t* __restrict__ row) {
  uint32_t const lane = threadIdx.x & 31, digits = 1u << D;
  uint32_t keep = 0;
  for (uint32_t i = 0; i < digits; ++i) {
    uint32_t const v = cnt[i * 32 + lane];
    cnt[i * 32 + lane] = 0;
    uint32_t const s = __reduce_add_sync(0xffffffffu, v);
    if (lane == i) keep = s;
  }
  if (lane < digits) row[lane] = static_cast<uint16_t>(keep);
}

// ---- 1. text -> planes -------------------------------------------------------

struct IngestArgs {
  uint64_t n;
  uint64_t first, last;        // tiles to read
  uint32_t L, D, tile;         // code bits, digit bits of the counts, tile symbols
  uint32_t* plane[kMaxPlanes]; // plane j: code bit L - 1 - j
  uint16_t const* lut;         // symbol -> code, for symbols up to max_symbol
  uint32_t max_symbol;
  uint16_t* tile_cnt;          // null: no counts
  uint32_t* err;               // bit 0: a symbol outside the alphabet
  TileGrid g;                  // of the first pass, when it has one node
};

constexpr uint32_t kIngestThreads = 256;

// One CTA per tile in turn, 32 symbols per thread and step: two (u8) or four
// (u16) 16-byte loads, a byte transpose, the 8 x 8 bit transposes, one word
// of every plane out (128 bytes per warp and plane).  Map: codes come from a
// table (256 entries in shared memory for bytes).
template <class T, bool Map>
__global__ void __launch_bounds__(kIngestThreads, sizeof(T) == 1 ? 6 : 2)
ingest_planes_kernel(T const* __restrict__ text, IngestArgs a) {
  __shared__ uint32_t cnt[kMaxDigits * 32];
  __shared__ uint16_t lut_s[Map && sizeof(T) == 1 ? 256 : 1];
  uint32_t const tid = threadIdx.x, lane4 = (tid & 31) * 4;
  bool const counted = a.tile_cnt != nullptr;
  if (counted && blockIdx.x == 0 && tid == 0) single_node_tables(a.g);
  for (uint32_t i = tid; i < kMaxDigits * 32; i += kIngestThreads) cnt[i] = 0;
  if constexpr (Map && sizeof(T) == 1)
    for (uint32_t i = tid; i < 256; i += kIngestThreads) lut_s[i] = a.lut[i];
  __syncthreads();
  uint32_t const base = static_cast<uint32_t>(__cvta_generic_to_shared(cnt));
  uint32_t const sh = a.L - a.D, dmask = ((1u << a.D) - 1u) * 0x01010101u;
  uint32_t const lo_mask = 0x01010101u * (0xFFu >> min(sh, 8u));
  // bits at or above L in a symbol
  uint32_t const over_lo = a.L >= 8 ? 0u : 0x01010101u * ((0xFFu << a.L) & 0xFFu);
  uint32_t const over_hi = a.L >= 16 ? 0u
                           : a.L <= 8 ? ~0u
                                      : 0x01010101u * ((0xFFu << (a.L - 8)) & 0xFFu);
  uint32_t bad = 0;
  for (uint64_t ti = a.first + blockIdx.x; ti < a.last; ti += gridDim.x) {
    uint64_t const s = ti * a.tile;
    uint32_t const len = static_cast<uint32_t>(min(uint64_t(a.tile), a.n - s));
    for (uint32_t w = tid; w * 32 < len; w += kIngestThreads) {
      uint64_t const p0 = s + uint64_t(w) * 32;
      uint32_t const valid = min(32u, len - w * 32);
      constexpr int kX = 8 * sizeof(T);
      uint32_t x[kX];
      if (valid == 32) {
        uint4 const* v = reinterpret_cast<uint4 const*>(text + p0);
#pragma unroll
        for (int i = 0; i < kX / 4; ++i) {
          uint4 const q = __ldg(v + i);
          x[4 * i] = q.x;
          x[4 * i + 1] = q.y;
          x[4 * i + 2] = q.z;
          x[4 * i + 3] = q.w;
        }
      } else {
#pragma unroll
        for (int i = 0; i < kX; ++i) {
          x[i] = 0;
#pragma unroll
          for (uint32_t h = 0; h < 4 / sizeof(T); ++h) {
            uint32_t const at = i * (4 / sizeof(T)) + h;
            // past the end: a symbol of the alphabet (its plane bits are
            // cleared below)
            T const c = text[p0 + min(at, valid - 1)];
            x[i] |= uint32_t(c) << (8 * sizeof(T) * h);
          }
        }
      }
      // byte h of lo[i] (hi[i]): the low (high) byte of symbol 8 h + i
      uint32_t lo[8], hi[8];
      if constexpr (sizeof(T) == 1) {
        transpose4(x[0], x[2], x[4], x[6], lo, 1);
        transpose4(x[1], x[3], x[5], x[7], lo + 4, 1);
#pragma unroll
        for (int i = 0; i < 8; ++i) hi[i] = 0;
      } else {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          uint32_t t[4];
          transpose4(x[p], x[4 + p], x[8 + p], x[12 + p], t, 1);
          lo[2 * p] = t[0];
          hi[2 * p] = t[1];
          lo[2 * p + 1] = t[2];
          hi[2 * p + 1] = t[3];
        }
      }
      if constexpr (Map) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint32_t nl = 0, nh = 0;
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t c = (lo[i] >> (8 * h)) & 0xFFu;
            if constexpr (sizeof(T) == 2) c |= ((hi[i] >> (8 * h)) & 0xFFu) << 8;
            bad |= c > a.max_symbol;
            c = sizeof(T) == 1 ? uint32_t(lut_s[c & 0xFFu]) : uint32_t(__ldg(a.lut + c));
            nl |= (c & 0xFFu) << (8 * h);
            nh |= (c >> 8) << (8 * h);
          }
          lo[i] = nl;
          hi[i] = nh;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) bad |= (lo[i] & over_lo) | (hi[i] & over_hi);
      }
      if (counted) {
        if (valid == 32) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            uint32_t dw;
            if (sh >= 8) dw = (hi[i] >> (sh - 8)) & dmask;
            else dw = ((hi[i] << (8 - sh)) | ((lo[i] >> sh) & lo_mask)) & dmask;
            count_digits(base, lane4, dw);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int h = 0; h < 4; ++h)
              if (8 * h + i < valid) {
                uint32_t const c = ((lo[i] >> (8 * h)) & 0xFFu) |
                                   (((hi[i] >> (8 * h)) & 0xFFu) << 8);
                uint32_t const d = (c >> sh) & ((1u << a.D) - 1u);
                atomicAdd(&cnt[d * 32 + (tid & 31)], 1u);
              }
        }
      }
      uint32_t const vm = valid == 32 ? ~0u : (1u << valid) - 1u;
      uint64_t const wi = p0 >> 5;
      transpose_bits(lo);
#pragma unroll
      for (uint32_t b = 0; b < 8; ++b)
        if (b < a.L) a.plane[a.L - 1 - b][wi] = lo[b] & vm;
      if (a.L > 8) {
        transpose_bits(hi);
#pragma unroll
        for (uint32_t b = 0; b < 8; ++b)
          if (b + 8 < a.L) a.plane[a.L - 9 - b][wi] = hi[b] & vm;
      }
    }
    if (counted) {
      __syncthreads();
      if (tid < 32) flush_digits(cnt, a.D, a.tile_cnt + (ti << a.D));
      __syncthreads();
    }
  }
  if (bad) atomicOr(a.err, 1u);
}

// ---- 2. digit counts from planes --------------------------------------------

struct PlaneSources {
  uint32_t const* p[kMaxPlanes];
};

// 32 bits of an array from bit q on, of which `valid` (>= 1) are wanted: no
// word behind the last wanted bit is read.
__device__ __forceinline__ uint32_t plane_bits32(uint32_t const* __restrict__ w,
                                                 uint64_t q, uint32_t valid) {
  uint64_t const i = q >> 5;
  uint32_t const s = static_cast<uint32_t>(q) & 31u;
  uint32_t const a = __ldg(w + i);
  uint32_t const b = s + valid > 32 ? __ldg(w + i + 1) : 0u;
  return __funnelshift_r(a, b, s);
}

// Adds, for every inner node I of the digit tree (root 1, children 2 I for a
// zero and 2 I + 1 for a one bit), the positions of m whose next bit is one.
template <int I, int J, int D>
__device__ __forceinline__ void tally(uint32_t m, uint32_t const (&x)[D],
                                      uint32_t (&acc)[1 << D]) {
  if constexpr (J < D) {
    uint32_t const one = m & x[J];
    acc[I] += __popc(one);
    tally<2 * I + 1, J + 1, D>(one, x, acc);
    tally<2 * I, J + 1, D>(m & ~x[J], x, acc);
  }
}

// Tile counts of the D-bit digits held by planes src.p[0 .. D-1], the first
// the highest bit: a CTA per tile in turn, one word of every plane per thread
// and step, one popcount per inner node of the digit tree (2^D - 1 for 32
// symbols; counting digits one by one took four times the instructions).  One
// wave: twelve CTAs per SM, of which ten fit for D = 4, took 1.67 ms at 6 Gi
// symbols, ten 1.19.
constexpr uint32_t kCountThreads = 128;

template <int D>
__global__ void __launch_bounds__(kCountThreads, 10)
plane_counts_kernel(const __grid_constant__ PlaneSources src, TileGrid g) {
  __shared__ uint32_t sum[1 << D];
  uint32_t const tid = threadIdx.x, lane = tid & 31;
  if (tid < (1u << D)) sum[tid] = 0;
  uint32_t const tiles = g.tile_first[g.nodes];
  for (uint32_t ti = blockIdx.x; ti < tiles; ti += gridDim.x) {
    uint32_t const N = owner_node(g.tile_first, g.nodes, ti);
    uint64_t const s = g.starts[N] + uint64_t(ti - g.tile_first[N]) * g.tile;
    uint64_t const e = g.starts[N + 1];
    uint32_t const len = s < e ? static_cast<uint32_t>(min(uint64_t(g.tile), e - s)) : 0u;
    uint32_t acc[1 << D];
#pragma unroll
    for (int i = 0; i < (1 << D); ++i) acc[i] = 0;
#pragma unroll 1
    for (uint32_t w = tid; w * 32 < len; w += kCountThreads) {
      uint64_t const p0 = s + uint64_t(w) * 32;
      uint32_t const valid = min(32u, len - w * 32);
      uint32_t x[D];
#pragma unroll
      for (int b = 0; b < D; ++b) x[b] = plane_bits32(src.p[b], p0, valid);
      tally<1, 0, D>(valid == 32 ? ~0u : (1u << valid) - 1u, x, acc);
    }
    __syncthreads();  // sum is clear
#pragma unroll
    for (int i = 1; i < (1 << D); ++i) {
      uint32_t const v = __reduce_add_sync(0xffffffffu, acc[i]);
      if (lane == 0) atomicAdd(&sum[i], v);
    }
    __syncthreads();
    if (tid < (1u << D)) {  // digit tid: down the tree from the root's `len`
      uint32_t c = len, i = 1;
#pragma unroll
      for (int j = 0; j < D; ++j) {
        uint32_t const bit = (tid >> (D - 1 - j)) & 1u, one = sum[i];
        c = bit ? one : c - one;
        i = 2 * i + bit;
      }
      g.tile_cnt[(uint64_t(ti) << D) + tid] = static_cast<uint16_t>(c);
    }
    __syncthreads();
    if (tid < (1u << D)) sum[tid] = 0;
  }
}

// ---- 3. scans ------------------------------------------------------------------

// One pass: its tiles, input planes and outputs.
struct PlanePass {
  TileGrid g;
  uint32_t k, np;                        // levels written; planes behind plane a
  uint32_t const* src[kMaxPlanes];       // src[j]: plane a + j, j = 0 .. np
  uint32_t* out[kMaxPassK + 1];          // out[r]: level a + r, r = 1 .. k
  uint64_t out_words[kMaxPassK + 1];
  uint32_t* ext[kMaxPassK + 1][kMaxPlanes];  // plane a + j in level-(a+r) order
  uint32_t ext_mask[kMaxPassK + 1];      // bit j: ext[r][j] is wanted
  uint64_t ext_words;
};

// Clears word w of level a + r and of the deeper planes of its order.
__device__ __forceinline__ void clear_word(PlanePass const& p, uint32_t r, uint64_t w) {
  if (w < p.out_words[r]) p.out[r][w] = 0;
  for (uint32_t mask = p.ext_mask[r]; mask; mask &= mask - 1)
    if (w < p.ext_words) p.ext[r][__ffs(mask) - 1][w] = 0;
}

// The words of a pass's outputs that two runs may share, into which the pass
// ORs, are cleared first: every word that holds the start of a tile's class
// run, and the arrays' ends (all other words are written whole by one
// thread).  A warp takes tiles t0 .. t1 - 1 of a node, lane per digit: the
// digit positions (start: the digit's own, pre: the node's before t0), stepped
// from tile to tile and added up per class.  (Clearing the outputs whole took
// 1.4 ms per build of 6 Gi symbols of 256.)
__device__ __forceinline__ void clear_tile_edges(PlanePass const& p, uint64_t start,
                                                 uint64_t pre, uint32_t t0, uint32_t t1) {
  uint32_t const lane = threadIdx.x & 31, D = p.g.D;
  bool const on = lane < (1u << D);
  for (uint32_t t = t0; t < t1; ++t) {
    uint64_t sum = pre;  // of the lane's class
    for (uint32_t r = D; r > 0; --r) {
      uint32_t const h = 1u << (D - r);  // digits of a level-r class
      if (h > 1) sum += __shfl_xor_sync(0xffffffffu, sum, h >> 1);
      if (r <= p.k && on && (lane & (h - 1)) == 0) clear_word(p, r, (start + sum) >> 5);
    }
    if (on) pre += p.g.tile_cnt[(uint64_t(t) << D) + lane];
  }
}
__device__ __forceinline__ void clear_ends(PlanePass const& p) {
  for (uint32_t r = 1; r <= p.k; ++r) {
    uint64_t const lim = max(p.out_words[r], p.ext_mask[r] ? p.ext_words : uint64_t(0));
    for (uint64_t w = (p.g.n >> 5) + threadIdx.x; w < lim; w += blockDim.x) clear_word(p, r, w);
  }
}

// ... a warp per chunk.
__global__ void __launch_bounds__(128)
clear_edges_kernel(const __grid_constant__ PlanePass p) {
  uint32_t const lane = threadIdx.x & 31, D = p.g.D;
  uint32_t const chunks = p.g.chunk_first[p.g.nodes];
  bool const on = lane < (1u << D);
  if (blockIdx.x == 0) clear_ends(p);
  for (uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5); c < chunks; c += gridDim.x * 4) {
    uint32_t const N = owner_node(p.g.chunk_first, p.g.nodes, c);
    uint32_t const t0 = p.g.tile_first[N] + (c - p.g.chunk_first[N]) * p.g.ct;
    clear_tile_edges(p, on ? *digit_start(p.g, N, lane) : 0,
                     on ? p.g.chunk_pre[(uint64_t(c) << D) + lane] : 0, t0,
                     min(t0 + p.g.ct, p.g.tile_first[N + 1]));
  }
}

// Range r: its node and tiles [t0, t1) (whole chunks).
__device__ __forceinline__ uint32_t range_tiles(TileGrid const& g, uint32_t r, uint32_t* t0,
                                                uint32_t* t1) {
  uint32_t const N = owner_node(g.range_first, g.nodes, r);
  uint32_t const f = g.tile_first[N], e = g.tile_first[N + 1];
  *t0 = min(e, f + (r - g.range_first[N]) * g.rc * g.ct);
  *t1 = min(e, *t0 + g.rc * g.ct);
  return N;
}

constexpr uint32_t kRangeWarps = 4;

// Digit totals of every range (a warp each, lane per digit).
__global__ void __launch_bounds__(kRangeWarps * 32)
range_totals_kernel(TileGrid g) {
  uint32_t const d = threadIdx.x & 31, r = blockIdx.x * kRangeWarps + (threadIdx.x >> 5);
  if (r >= g.range_first[g.nodes] || d >= (1u << g.D)) return;
  uint32_t t0, t1;
  range_tiles(g, r, &t0, &t1);
  uint64_t sum = 0;
  uint16_t const* c = g.tile_cnt + d;
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) sum += c[uint64_t(t) << g.D];
  g.range_tot[(uint64_t(r) << g.D) + d] = sum;
}

// Warp w of the CTA holds the digit totals `own` (lane = digit) of the w-th
// stretch of node N: returns the digits before the stretch and writes every
// digit's start position (node start + smaller digits).
__device__ __forceinline__ uint64_t node_digit_starts(TileGrid const& g, uint32_t N,
                                                      uint64_t own) {
  __shared__ uint64_t part[32][32];
  uint32_t const lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  part[wid][lane] = own;
  __syncthreads();
  uint64_t before = 0, tot = 0;
  for (uint32_t w = 0; w < warps; ++w) {
    if (w == wid) before = tot;
    tot += part[w][lane];
  }
  if (wid == 0) {
    uint64_t inc = tot;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      uint64_t const y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane < (1u << g.D)) {
      uint64_t const at = g.starts[N] + inc - tot;
      uint64_t* const s = digit_start(g, N, lane);
      s[0] = at;
      if (g.halves || (N == g.nodes - 1 && lane == (1u << g.D) - 1)) s[1] = at + tot;
      if (g.halves && N == g.nodes - 1 && lane == (1u << g.D) - 1) s[2] = at + tot;
    }
  }
  return before;
}

// Per node: the range totals become counts before the range, and every
// digit's start position (a CTA per node, lane per digit, a stretch of
// ranges per warp).
__global__ void __launch_bounds__(1024)
digit_starts_kernel(TileGrid g) {
  uint32_t const d = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint32_t const N = blockIdx.x;
  bool const on = d < (1u << g.D);
  uint32_t const f = g.range_first[N], ranges = g.range_first[N + 1] - f;
  uint32_t const per = (ranges + warps - 1) / warps;
  uint32_t const r0 = min(ranges, wid * per), r1 = min(ranges, r0 + per);
  uint64_t* const p = g.range_tot + (uint64_t(f) << g.D) + d;
  uint64_t own = 0;
#pragma unroll 8
  for (uint32_t r = r0; r < r1; ++r) own += on ? p[uint64_t(r) << g.D] : 0;
  uint64_t run = node_digit_starts(g, N, own);
#pragma unroll 8
  for (uint32_t r = r0; r < r1; ++r) {
    uint64_t const x = on ? p[uint64_t(r) << g.D] : 0;
    if (on) p[uint64_t(r) << g.D] = run;
    run += x;
  }
}

// All of the scan in one launch for orders of few tiles: a CTA per node, lane
// per digit, a stretch of chunks per warp.  With p.k > 0 the outputs' shared
// words are cleared as well; with next.nodes > 0 (a single node) the next
// pass's tables are made.
__global__ void __launch_bounds__(1024)
node_scan_kernel(const __grid_constant__ PlanePass p, const __grid_constant__ TileGrid next) {
  TileGrid const& g = p.g;
  uint32_t const d = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint32_t const N = blockIdx.x;
  bool const on = d < (1u << g.D);
  uint32_t const f = g.tile_first[N], e = g.tile_first[N + 1], c0 = g.chunk_first[N];
  uint32_t const chunks = (e - f + g.ct - 1) / g.ct;
  uint32_t const per = (chunks + warps - 1) / warps * g.ct;
  uint32_t const t0 = min(e, f + wid * per), t1 = min(e, t0 + per);
  uint16_t const* c = g.tile_cnt + d;
  uint64_t own = 0;
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) own += on ? c[uint64_t(t) << g.D] : 0;
  uint64_t const before = node_digit_starts(g, N, own);
  uint64_t run = before;
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) {
    if (on && (t - f) % g.ct == 0)
      g.chunk_pre[(uint64_t(c0 + (t - f) / g.ct) << g.D) + d] = run;
    run += on ? c[uint64_t(t) << g.D] : 0;
  }
  __syncthreads();  // the digit starts are written
  if (p.k) {
    if (N == 0) clear_ends(p);
    clear_tile_edges(p, on ? *digit_start(g, N, d) : 0, before, t0, t1);
  }
  if (next.nodes && wid == 0) {  // as many as this pass has digits
    uint32_t x[3] = {0, 0, 0};
    if (on) {
      uint64_t const len = g.starts_next[d + 1] - g.starts_next[d];
      x[0] = static_cast<uint32_t>((len + next.tile - 1) / next.tile);
      x[1] = (x[0] + next.ct - 1) / next.ct;
      x[2] = (x[1] + next.rc - 1) / next.rc;
    }
    uint32_t* const first[3] = {next.tile_first, next.chunk_first, next.range_first};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      uint32_t const inc = warp_inclusive(x[i]);
      if (on) first[i][d] = inc - x[i];
      if (on && d == next.nodes - 1) first[i][next.nodes] = inc;
    }
  }
}

// The digits of the node before every chunk (a warp per range).
__global__ void __launch_bounds__(kRangeWarps * 32)
chunk_starts_kernel(TileGrid g) {
  uint32_t const d = threadIdx.x & 31, r = blockIdx.x * kRangeWarps + (threadIdx.x >> 5);
  if (r >= g.range_first[g.nodes] || d >= (1u << g.D)) return;
  uint32_t t0, t1;
  uint32_t const N = range_tiles(g, r, &t0, &t1);
  uint64_t run = g.range_tot[(uint64_t(r) << g.D) + d];
  uint32_t const f = g.tile_first[N], c0 = g.chunk_first[N];
  uint16_t const* c = g.tile_cnt + d;
#pragma unroll 8
  for (uint32_t t = t0; t < t1; ++t) {
    if ((t - f) % g.ct == 0)
      g.chunk_pre[(uint64_t(c0 + (t - f) / g.ct) << g.D) + d] = run;
    run += c[uint64_t(t) << g.D];
  }
}

// ---- 4. the pass ------------------------------------------------------------------


// Swap masks of the five in-word stages for one word of the mask plane with
// r0 ones before it in the slot: c[s] holds the positions q of the left
// halves (blocks of 2^(s+1)) that change places with q + 2^s.  The counts
// come from one SWAR popcount (pairs, nibbles, bytes) and its byte prefix.
struct SwapMasks {
  uint32_t c[5];
};

__host__ __device__ __forceinline__ uint32_t rotl32(uint32_t x, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(x, x, s);
#else
  s &= 31;
  return s ? x << s | x >> (32 - s) : x;
#endif
}

__host__ __device__ __forceinline__ SwapMasks swap_masks(uint32_t m, uint32_t r0) {
  SwapMasks k;
  uint32_t const v1 = m - ((m >> 1) & 0x55555555u);                  // pairs
  uint32_t const v2 = (v1 & 0x33333333u) + ((v1 >> 2) & 0x33333333u);  // nibbles
  uint32_t const v3 = (v2 + (v2 >> 4)) & 0x0F0F0F0Fu;                // bytes
  // byte j of P: r0 + the ones of bytes 0 .. j; of PE: before byte j
  uint32_t const P = (v3 + r0) * 0x01010101u;
  uint32_t const PE = (P << 8) | r0;
  uint32_t const Q = PE + (v2 & 0x0F0F0F0Fu);  // before the byte's high nibble
  k.c[4] = rotl32(0x0000FFFFu, P >> 8) & 0x0000FFFFu;
  k.c[3] = (rotl32(0x00FF00FFu, P) & 0x000000FFu) |
           (rotl32(0x00FF00FFu, P >> 16) & 0x00FF0000u);
  {  // four byte lanes at once: 1111 << (Q mod 4), inverted when bit 2 of Q is set
    uint32_t const t1 = (Q & 0x01010101u) * 15u + 0x0F0F0F0Fu;
    uint32_t const t2 = (t1 & (((Q >> 1) & 0x01010101u) * 255u)) * 3u + t1;
    k.c[2] = (t2 & 0x0F0F0F0Fu) ^ (((Q >> 2) & 0x01010101u) * 15u);
  }
  // ones before every nibble (X) and before its upper pair (Y), mod 4
  uint32_t const X = (PE & 0x03030303u) | ((Q & 0x03030303u) << 4);
  uint32_t const Y = X + (v1 & 0x33333333u);
  k.c[1] = ~(Y ^ ((Y >> 1) & 0x11111111u)) & 0x33333333u;
  uint32_t const U = (X & 0x11111111u) | ((Y & 0x11111111u) << 2);  // parity before a pair
  k.c[0] = ~(U ^ m) & 0x55555555u;
  return k;
}

__host__ __device__ __forceinline__ uint32_t swap_stages(uint32_t x, SwapMasks const& k) {
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    uint32_t const t = ((x >> (1 << s)) ^ x) & k.c[s];
    x ^= t * ((1u << (1 << s)) + 1u);  // t and t << 2^s share no bit
  }
  return x;
}

__device__ __forceinline__ void red_or_shared(uint32_t addr, uint32_t v) {
  asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// A slot is W 32-bit words of a class run, one thread's work.  A class run of
// len symbols starts at a bit offset of at most 31 in its first slot (that of
// its output words), so it takes at most (len + 31 + 32 W - 1) / (32 W) slots
// and a level of 2^k classes at most tile / (32 W) + 1.25 * 2^k (W >= 4).
__host__ __device__ constexpr uint32_t pass_tile(uint32_t slots, uint32_t W, uint32_t k) {
  return (slots - ((5u << k) + 3) / 4) * 32 * W;
}
// A plane's words in a buffer (slots and two words' pad at least that only
// words without bits of a run are ORed into).
__host__ __device__ constexpr uint32_t plane_stride(uint32_t slots, uint32_t W) {
  return slots * W + 8;
}
__host__ __device__ constexpr uint32_t buffer_words(uint32_t slots, uint32_t W, uint32_t np) {
  return np * plane_stride(slots, W) + 8;
}
__host__ __device__ constexpr size_t pass_smem(uint32_t slots, uint32_t W, uint32_t np) {
  return size_t(2) * buffer_words(slots, W, np) * 4;
}

// Bits at or above position c of word i (all when c is below it).
__host__ __device__ __forceinline__ uint32_t bits_from(uint32_t c, uint32_t i) {
  return c <= 32 * i ? ~0u : c >= 32 * i + 32 ? 0u : ~0u << (c - 32 * i);
}

// The stages across words: stage t swaps word u of the left with word u of
// the right half of each block of 2^(t+1) words under mask m[..], in the
// order the stages run; ones[i] = ones of the slot before word i.
template <uint32_t W>
struct WordSwaps {
  static constexpr uint32_t kCount = W == 4 ? 4 : 12;
  uint32_t m[kCount];
};
template <uint32_t W>
__host__ __device__ __forceinline__ WordSwaps<W> word_swaps(uint32_t const* ones) {
  WordSwaps<W> s;
  uint32_t at = 0;
#pragma unroll
  for (uint32_t h = 1; h < W; h *= 2)
#pragma unroll
    for (uint32_t b = 0; b < W; b += 2 * h) {
      // ring of 64 h positions: positions at or above M mod 32 h, inverted in
      // its upper half
      uint32_t const M = ones[b + h] & (64 * h - 1);
      uint32_t const inv = M >= 32 * h ? ~0u : 0u;
#pragma unroll
      for (uint32_t u = 0; u < h; ++u) s.m[at++] = bits_from(M & (32 * h - 1), u) ^ inv;
    }
  return s;
}
template <uint32_t W>
__host__ __device__ __forceinline__ void swap_words(uint32_t* x, WordSwaps<W> const& s) {
  uint32_t at = 0;
#pragma unroll
  for (uint32_t h = 1; h < W; h *= 2)
#pragma unroll
    for (uint32_t b = 0; b < W; b += 2 * h)
#pragma unroll
      for (uint32_t u = 0; u < h; ++u) {
        uint32_t const t = (x[b + u] ^ x[b + h + u]) & s.m[at++];
        x[b + u] ^= t;
        x[b + h + u] ^= t;
      }
}

template <uint32_t W>
__device__ __forceinline__ void load_slot(uint32_t const* p, uint32_t* y) {
  uint4 const* v = reinterpret_cast<uint4 const*>(p);
#pragma unroll
  for (uint32_t i = 0; i < W / 4; ++i) {
    uint4 const x = v[i];
    y[4 * i] = x.x;
    y[4 * i + 1] = x.y;
    y[4 * i + 2] = x.z;
    y[4 * i + 3] = x.w;
  }
}
template <uint32_t W>
__device__ __forceinline__ void store_slot(uint32_t* p, uint32_t const* y) {
  uint4* v = reinterpret_cast<uint4*>(p);
#pragma unroll
  for (uint32_t i = 0; i < W / 4; ++i)
    v[i] = make_uint4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
}

// Persistent CTAs of one thread per slot; CTA b takes chunks b, b + G, ...,
// a chunk's tiles in order (the run positions carry from tile to tile).
// Per tile: class tables of all levels from the tile's digit counts (warp r
// builds level r's); then per level r: every slot finds its class and writes
// its 128 bits of level a+r (and of the wanted deeper planes) out, a scan of
// the slots' zero counts gives each slot's place in its class's two
// children, and every deeper plane is swapped and ORed into the next order's
// buffer.
//
// Bound by the ALU pipe (73 % busy, 62 % of the issue slots used; 3 CTAs of
// 256 threads per SM by shared memory).  128-bit slots: a
// slot's bookkeeping costs about as much as three plane moves, so 64-bit
// slots took 28 % more instructions; 256-bit slots leave 3 warps per
// scheduler (18 % slower).  Passes of at most 4 levels: with 128 classes
// (one pass of 7 levels) runs waste a third of the slots, 36 against 20 ms.
// A class run is laid out at the bit offset of its place in the
// level's words, so that going out is a copy of whole words.
template <uint32_t NT, uint32_t W, class Index>
__global__ void __launch_bounds__(NT, NT == 256 ? 3 : 4)
plane_pass_kernel(const __grid_constant__ PlanePass p) {
  using Words = std::make_unsigned_t<Index>;
  constexpr uint32_t kWarps = NT / 32, kSlotBits = 32 * W;
  extern __shared__ __align__(16) uint32_t buf[];
  __shared__ __align__(16) uint2 rec[2 << kMaxPassK];  // class q of level r at (1 << r) + q:
                                       // {first slot | length << 16, zeros in classes before | bit offset << 16}
  __shared__ uint64_t gpos[2 << kMaxPassK];        // its run's next bit
  __shared__ uint64_t pre_s[kMaxDigits + 1];
  __shared__ uint32_t dig_s[kMaxDigits + 1];       // tile symbols with a smaller digit
  __shared__ uint32_t flags[kMaxPassK + 1][kWarps];  // slots that begin a class
  __shared__ uint8_t first_cls[kMaxPassK + 1][NT];   // ... and which
  __shared__ uint8_t warp_cls[kMaxPassK + 1][kWarps];  // class of a warp's first slot
  __shared__ uint32_t nslots[kMaxPassK + 1];
  __shared__ uint32_t warp_tot[kWarps];
  __shared__ uint32_t half_ones[1 << kMaxPassK];  // last pass: ones of every class, last plane
  __shared__ uint64_t ck_start;
  __shared__ uint32_t ck_node, ck_tile, ck_len;

  uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t const k = p.k, np = p.np, D = p.g.D, digits = 1u << D;
  uint32_t const chunks = p.g.chunk_first[p.g.nodes];
  uint64_t const chunk_syms = uint64_t(p.g.tile) * p.g.ct;
  constexpr uint32_t kPS = plane_stride(NT, W);
  // plane j of buffer x, slot s: buf[x * half + 8 + (j - 1) * kPS + s * W]
  uint32_t const half = buffer_words(NT, W, np);

  for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    // ---- the chunk: its symbols, and every class run's position
    if (tid == 0) {
      uint32_t const N = owner_node(p.g.chunk_first, p.g.nodes, c);
      uint32_t const j = c - p.g.chunk_first[N];
      uint64_t const s = p.g.starts[N] + j * chunk_syms, e = p.g.starts[N + 1];
      ck_node = N;
      ck_start = s;
      ck_tile = p.g.tile_first[N] + j * p.g.ct;
      ck_len = s < e ? static_cast<uint32_t>(min(chunk_syms, e - s)) : 0u;
    }
    if (wid == 1) {  // digits of the node before the chunk, as a prefix over digits
      uint64_t const own = lane < digits ? p.g.chunk_pre[(uint64_t(c) << D) + lane] : 0;
      uint64_t inc = own;
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
        uint64_t const y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane < digits) pre_s[lane + 1] = inc;
      if (lane == 0) pre_s[0] = 0;
    }
    __syncthreads();
    for (uint32_t i = 2 + tid; i < (2u << k); i += NT) {
      uint32_t const r = 31 - __clz(i), q = i - (1u << r);
      uint32_t const d0 = q << (D - r), d1 = (q + 1) << (D - r);
      gpos[i] = *digit_start(p.g, ck_node, d0) + pre_s[d1] - pre_s[d0];
    }
    if (tid < (1u << kMaxPassK)) half_ones[tid] = 0;
    uint32_t const len_c = ck_len;
    uint32_t const tiles = (len_c + p.g.tile - 1) / p.g.tile;
    for (uint32_t ti = 0; ti < tiles; ++ti) {
      uint64_t const ts = ck_start + uint64_t(ti) * p.g.tile;
      uint32_t const tcnt = min(p.g.tile, len_c - ti * p.g.tile);
      // ---- planes of the tile: slot tid's 128 positions of each; the first
      //      level's target zeroed
      uint32_t m[W];
      uint32_t const zero[W] = {};
      {
        uint64_t const q = ts + uint64_t(tid) * kSlotBits;
        uint32_t const v = tid * kSlotBits < tcnt ? min(kSlotBits, tcnt - tid * kSlotBits) : 0u;
        uint64_t const i = q >> 5;
        uint32_t const s = static_cast<uint32_t>(q) & 31u;
        auto load = [&](uint32_t const* __restrict__ w, uint32_t* y) {
          w += i;
          uint32_t x[W + 1];
#pragma unroll
          for (uint32_t u = 0; u <= W; ++u)
            x[u] = v && s + v > 32 * u ? __ldg(w + u) : 0u;
#pragma unroll
          for (uint32_t u = 0; u < W; ++u)
            y[u] = __funnelshift_r(x[u], x[u + 1], s) & ~bits_from(v, u);
        };
        load(p.src[0], m);
#pragma unroll 2
        for (uint32_t j = 1; j <= np; ++j) {
          uint32_t y[W];
          load(p.src[j], y);
          store_slot<W>(buf + half + 8 + (j - 1) * kPS + tid * W, y);
          store_slot<W>(buf + 8 + (j - 1) * kPS + tid * W, zero);
        }
      }
      // the chunk's next tile, on its way to L2 (1.7 % of the pass)
      if (ti + 1 < tiles && (ti + 1) * p.g.tile + tid * kSlotBits < len_c) {
        uint64_t const at = (ts + p.g.tile + uint64_t(tid) * kSlotBits) >> 5;
        for (uint32_t j = 0; j <= np; ++j)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.src[j] + at));
      }
      // ---- class tables
      if (wid == 0) {  // prefix of the tile's digit counts
        uint32_t const own =
            lane < digits ? p.g.tile_cnt[(uint64_t(ck_tile + ti) << D) + lane] : 0u;
        uint32_t const inc = warp_inclusive(own);
        if (lane < digits) dig_s[lane + 1] = inc;
        if (lane == 0) dig_s[0] = 0;
      } else {
        for (uint32_t i = tid - 32; i < (kMaxPassK + 1) * kWarps; i += NT - 32)
          (&flags[0][0])[i] = 0;
      }
      __syncthreads();
      for (uint32_t r = wid; r <= k; r += kWarps) {  // lane q: class q of level r
        uint32_t const nc = 1u << r, sh = D - r, q = lane;
        uint32_t len = 0, off = 0, zeros = 0;
        if (q < nc) {
          uint32_t const a = dig_s[q << sh];
          len = dig_s[(q + 1) << sh] - a;
          if (r < k) zeros = dig_s[(2 * q + 1) << (sh - 1)] - a;
          if (r) {  // the offset of the run's first (stored reversed: last)
                    // bit in its output word
            uint32_t const g = static_cast<uint32_t>(gpos[nc + q]);
            off = (__popc(~q & (nc - 1)) & 1 ? ~(g + len - 1) : g) & 31u;
          }
        }
        uint32_t const ns = len ? (off + len + kSlotBits - 1) / kSlotBits : 0u;
        uint32_t const own = ns << 16 | zeros;
        uint32_t const inc = warp_inclusive(own);
        if (lane == 31) nslots[r] = min(inc >> 16, NT);
        uint32_t const first = (inc - own) >> 16;
        if (q < nc) rec[nc + q] = make_uint2(first | (len << 16), ((inc - own) & 0xFFFFu) | (off << 16));
        if (len && first + ns <= NT) {
          atomicOr(&flags[r][first >> 5], 1u << (first & 31));
          first_cls[r][first] = static_cast<uint8_t>(q);
          for (uint32_t w = (first + 31) / 32; w * 32 < first + ns; ++w)
            warp_cls[r][w] = static_cast<uint8_t>(q);
        }
      }
      __syncthreads();
      // ---- levels
      for (uint32_t r = 0;; ++r) {
        // planes r+1 .. np in level-(a+r) order
        uint32_t const* const cur = buf + 8 + tid * W + ((r & 1) ? 0u : half);
        // the slot's class q, its run's bits [off, end) counted from its
        // first slot, this slot's [b0, b0 + 32 W)
        uint32_t q = 0, off = 0, end = 0, zcum = 0, b0 = 0, v = 0;
        bool const act = tid < nslots[r];
        if (act) {
          uint32_t const f = flags[r][wid] & (0xFFFFFFFFu >> (31 - lane));
          q = f ? first_cls[r][(wid << 5) + 31 - __clz(f)] : warp_cls[r][wid];
          uint2 const rc = rec[(1u << r) + q];
          off = rc.y >> 16;
          end = off + (rc.x >> 16);
          zcum = rc.y & 0xFFFFu;
          b0 = (tid - (rc.x & 0xFFFFu)) * kSlotBits;
          v = min(end, b0 + kSlotBits) - max(off, b0);
          if (r) load_slot<W>(cur + (r - 1) * kPS, m);
        } else {
#pragma unroll
          for (uint32_t u = 0; u < W; ++u) m[u] = 0;
        }
        // -- out: level a+r and the wanted planes of its order
        if (r && act) {
          bool const rev = __popc(~q & ((1u << r) - 1u)) & 1;
          uint64_t const gs = gpos[(1u << r) + q];
          // the W output words base .. base + W - 1, of which those in
          // [w0, w1) are the run's own and whole; a slot's part of the run's
          // first (before w0) and last word (at w1) is ORed (rev: the other
          // way round)
          Words const base = rev ? static_cast<Words>((gs + end - 1) >> 5) - (b0 >> 5) - (W - 1)
                                 : static_cast<Words>((gs - off) >> 5) + (b0 >> 5);
          uint32_t const f0 = b0 < off ? 1u : 0u, f1 = min(W, (end - b0) / 32);
          bool const tail = f1 < W && b0 + 32 * f1 < end;
          uint32_t const w0 = rev ? W - f1 : f0, w1 = rev ? W - f0 : f1;
          uint32_t const ua = rev ? W - 1 : 0, ub = rev ? W - 1 - f1 : f1;
          auto put = [&](uint32_t const* y, uint32_t* __restrict__ o, Words nw) {
            uint32_t x[W];
#pragma unroll
            for (uint32_t u = 0; u < W; ++u) x[u] = rev ? __brev(y[W - 1 - u]) : y[u];
            o += static_cast<Index>(base);  // rev: may start before the array
            int const lim = static_cast<int>(
                min(static_cast<Index>(w1), static_cast<Index>(nw - base)));
#pragma unroll
            for (uint32_t u = 0; u < W; ++u)
              if (u >= w0 && static_cast<int>(u) < lim) o[u] = x[u];
            if (f0 && base + ua < nw) atomicOr(o + ua, rev ? x[W - 1] : x[0]);
            if (tail && base + ub < nw) {
              uint32_t e = x[0];
#pragma unroll
              for (uint32_t u = 1; u < W; ++u) e = ub == u ? x[u] : e;
              atomicOr(o + ub, e);
            }
          };
          put(m, p.out[r], static_cast<Words>(p.out_words[r]));
          for (uint32_t mask = p.ext_mask[r]; mask; mask &= mask - 1) {
            uint32_t const j = __ffs(mask) - 1;
            uint32_t y[W];
            load_slot<W>(cur + (j - 1) * kPS, y);
            put(y, p.ext[r][j], static_cast<Words>(p.ext_words));
          }
        }
        if (r == k) {
          if (p.g.halves && act) {
            uint32_t c = 0;
#pragma unroll
            for (uint32_t u = 0; u < W; ++u) c += __popc(m[u]);
            atomicAdd(&half_ones[q], c);
          }
          break;
        }
        // -- zeros before every slot in its class
        uint32_t ones[W];  // of the slot, before word u
        uint32_t c = 0;
#pragma unroll
        for (uint32_t u = 0; u < W; ++u) {
          ones[u] = c;
          c += __popc(m[u]);
        }
        uint32_t const zc = v - c;
        uint32_t const inc = warp_inclusive(zc);
        if (lane == 31) warp_tot[wid] = inc;
        uint32_t* const dst = buf + 8 + ((r & 1) ? half : 0u);
        if (r && tid < nslots[r + 1])  // level r's target (level r-1's source until now)
#pragma unroll 2
          for (uint32_t j = r + 1; j <= np; ++j)
            store_slot<W>(dst + (j - 1) * kPS + tid * W, zero);
        __syncthreads();
        if ((wid << 5) < nslots[r]) {
          uint32_t const before =
              __reduce_add_sync(0xffffffffu, lane < wid ? warp_tot[lane] : 0u);
          uint32_t const lead = b0 < off ? off : 0u;  // slot bits before the run
          uint32_t const Z = before + inc - zc - zcum;
          uint32_t const O = (b0 > off ? b0 - off : 0u) - Z;
          uint4 const ch = *reinterpret_cast<uint4 const*>(&rec[(2u << r) + 2 * q]);
          // ones: bits ob .. ob + c - 1; zeros (reversed) end at the zero
          // child's end less the zeros before: the swapped slot's bit x
          // lands at zb + x (bits before the run count as its first zeros)
          uint32_t const ob = (ch.z & 0xFFFFu) * kSlotBits + (ch.w >> 16) + O;
          int const zb = static_cast<int>((ch.x & 0xFFFFu) * kSlotBits + (ch.y >> 16) +
                                          (ch.x >> 16) - Z + lead) -
                         static_cast<int>(kSlotBits);
          uint32_t const so = ob & 31u, sz = static_cast<uint32_t>(zb) & 31u;
          // never outside the plane's slots and the words before and after
          uint32_t const wo = min(ob >> 5, W * NT - 1);
          int const wz = max(-static_cast<int>(W), min(zb >> 5, static_cast<int>(W * NT - 1)));
          // words that hold ones (zeros) of any of the warp's slots: the
          // first n_one (from n_zero on) of the W + 1
          uint32_t const n_one =
              __reduce_max_sync(0xffffffffu, act && c ? (so + c + 31) / 32 : 0u);
          uint32_t const n_zero = __reduce_min_sync(
              0xffffffffu, act && zc ? (sz + kSlotBits - zc - lead) / 32 : W + 1);
          if (act) {
            uint32_t zm[W];  // bits at or above c: not ones
#pragma unroll
            for (uint32_t u = 0; u < W; ++u) zm[u] = bits_from(c, u);
            SwapMasks in_word[W];
#pragma unroll
            for (uint32_t u = 0; u < W; ++u) in_word[u] = swap_masks(m[u], ones[u]);
            WordSwaps<W> const across = word_swaps<W>(ones);
            uint32_t const db =
                static_cast<uint32_t>(__cvta_generic_to_shared(dst)) + r * (kPS * 4);
            uint32_t po = db + wo * 4, pz = db + static_cast<uint32_t>(wz) * 4;
            uint32_t const* from = cur + r * kPS;
            // two planes side by side: 1 Gi symbols 3405 -> 3345 us
#pragma unroll 2
            for (uint32_t j = np - r; j > 0; --j) {
              uint32_t x[W];
              load_slot<W>(from, x);
#pragma unroll
              for (uint32_t u = 0; u < W; ++u) x[u] = swap_stages(x[u], in_word[u]);
              swap_words<W>(x, across);
              // words without bits of the run are ORed all the same: a
              // branch per lane costs more than the shared-memory access
              uint32_t a = 0;
#pragma unroll
              for (uint32_t u = 0; u <= W; ++u) {
                uint32_t const b = u < W ? x[u < W ? u : 0] & ~zm[u < W ? u : 0] : 0u;
                if (u <= W / 2 + 1 || u < n_one)
                  red_or_shared(po + 4 * u, __funnelshift_l(a, b, so));
                a = b;
              }
              a = 0;
#pragma unroll
              for (uint32_t u = 0; u <= W; ++u) {
                uint32_t const b = u < W ? x[u < W ? u : 0] & zm[u < W ? u : 0] : 0u;
                if (u >= W / 2 - 1 || u >= n_zero)
                  red_or_shared(pz + 4 * u, __funnelshift_l(a, b, sz));
                a = b;
              }
              from += kPS;
              po += kPS * 4;
              pz += kPS * 4;
            }
          }
        }
        __syncthreads();
      }
      __syncthreads();  // the tile is out
      for (uint32_t i = 2 + tid; i < (2u << k); i += NT) gpos[i] += rec[i].x >> 16;
    }
    if (p.g.halves && tid < (1u << k) && half_ones[tid])
      atomicAdd(reinterpret_cast<unsigned long long*>(digit_start(p.g, ck_node, tid) + 1),
                0ull - half_ones[tid]);
    __syncthreads();  // gpos and the chunk's words are rewritten next
  }
}

// ---- the pipeline ---------------------------------------------------------------

// Deeper planes of one level's order: plane(j), first <= j < first + count, is
// code bit L - 1 - j in level `level`'s order.  The first `kept` of them
// outlive the pass that reads the order; the first `front` are in `mem`.
struct OrderPlanes {
  uint32_t level = 0, first = 0, count = 0, kept = 0, front = 0;
  uint64_t stride = 0;  // words per plane
  DevBuf mem, rest;
  uint32_t* plane(uint32_t j) const {
    uint32_t const i = j - first;
    return i < front ? mem.as<uint32_t>() + uint64_t(i) * stride
                     : rest.as<uint32_t>() + uint64_t(i - front) * stride;
  }
};

// Orders of more bytes than this hold the planes that go with their pass in
// an allocation of their own, so that they make room for the group levels (6
// Gi symbols of 256: 3.8 bytes per symbol at the peak instead of 4.7).  The
// pool gives such pieces back in other pieces than it gave them out, which
// costs more than it saves where memory is not short (6 Gi: 2.7 ms).
constexpr uint64_t kSplitOrderBytes = uint64_t(32) << 30;

// Where the forms for large texts begin (tests take them at small sizes): orders
// of more than split_bytes in two allocations, levels of wide_words 32-bit words
// with 64-bit word indices (2^36 symbols).
struct PlaneLimits {
  uint64_t split_bytes = kSplitOrderBytes;
  uint64_t wide_words = INT32_MAX;
};

// Levels per pass: as few passes of at most 4 levels as cover the L - 1 below
// level 0; the first of 3 where that takes no pass more (a group level's
// planes start at level 3, and the first pass carries the most planes), the
// others of near-equal size.
inline std::vector<uint32_t> plan_plane_passes(uint32_t L) {
  uint32_t rest = L - 1;
  std::vector<uint32_t> ks;
  if (rest <= kMaxPassK) return {rest};
  if ((rest - 3 + kMaxPassK - 1) / kMaxPassK + 1 == (rest + kMaxPassK - 1) / kMaxPassK) {
    ks.push_back(3);
    rest -= 3;
  }
  uint32_t const np = (rest + kMaxPassK - 1) / kMaxPassK;
  for (uint32_t i = 0; i < np; ++i) ks.push_back(rest / np + (i < rest % np ? 1u : 0u));
  return ks;
}

constexpr uint32_t kSlotWords = 4;  // words of a slot: a thread's work

// The largest CTA of which three fit an SM's shared memory (128: four, three
// from 14 planes on).
inline uint32_t pass_slots(uint32_t np) { return np <= 8 ? 256 : 128; }

// One wave of CTAs for `items` that kernel `k` deals out by CTA number: a CTA that
// started when others had ended would have its share done on a nearly empty GPU.
template <class Kernel>
uint32_t one_wave(Kernel k, uint32_t threads, size_t smem, uint64_t items) {
  int per_sm = 0;
  EWT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem));
  return static_cast<uint32_t>(std::max<uint64_t>(
      1, std::min<uint64_t>(items, uint64_t(sm_count()) * std::max(per_sm, 1))));
}

template <uint32_t NT, class Index>
void launch_plane_pass_as(PlanePass const& p, uint64_t max_chunks, cudaStream_t st) {
  auto kern = plane_pass_kernel<NT, kSlotWords, Index>;
  set_smem_limit(kern, static_cast<int>(pass_smem(NT, kSlotWords, NT == 256 ? 8 : 15)));
  size_t const smem = pass_smem(NT, kSlotWords, p.np);
  // (four CTAs per SM where three fit: 256 Mi uint16 symbols of 65,536 6.28 ms,
  // 6.10 so)
  uint32_t const grid = one_wave(kern, NT, smem, max_chunks);
  kern<<<grid, NT, smem, st>>>(p);
  EWT_LAUNCHED();
}

inline void launch_plane_pass(PlanePass const& p, uint32_t slots, uint64_t max_chunks,
                              uint64_t wide_words, cudaStream_t st) {
  bool const narrow = p.ext_words < wide_words;
  if (slots == 256 && narrow) launch_plane_pass_as<256, int32_t>(p, max_chunks, st);
  else if (slots == 256) launch_plane_pass_as<256, int64_t>(p, max_chunks, st);
  else if (narrow) launch_plane_pass_as<128, int32_t>(p, max_chunks, st);
  else launch_plane_pass_as<128, int64_t>(p, max_chunks, st);
}

// The text of a build (or the concatenated texts of a batch, one node each).
template <class T>
struct PlaneText {
  T const* sym = nullptr;      // 16-byte aligned; device memory, or readable host memory
  uint64_t n = 0;
  uint32_t L = 0;              // code bits, <= 16
  uint16_t const* lut = nullptr;  // symbol -> code (device); null: the symbol
  uint32_t max_symbol = 0;     // largest symbol with a code (lut)
  // A text in parts of about part_symbols (sym is null): part(begin, len) puts
  // the symbols from begin on at a 16-byte aligned address, in the stream's
  // order, where they stay until the next call.
  std::function<T const*(uint64_t begin, uint64_t len)> part;
  uint64_t part_symbols = 0;
  uint32_t nodes = 1;
  uint64_t* starts = nullptr;  // device, nodes + 1 (nodes > 1)
  int ingest_phase = EWT_PHASE_FILL;
};

// Levels 0 .. L-1 of a text: level l at words[l] (word_count[l] words, zero
// past the text's end on levels above 0), and starts_out, (nodes << L) + 1 entries: the
// start of every code's symbols.  `wanted`: (level, planes) pairs, the planes
// that many levels below `level` in its order are kept and returned.
template <class T>
std::vector<OrderPlanes> run_plane_passes(
    PlaneText<T> const& x, uint32_t* const* words, uint64_t const* word_count,
    uint64_t* starts_out, std::vector<std::pair<uint32_t, uint32_t>> const& wanted,
    uint32_t* err, cudaStream_t st, PlaneLimits const& limits = {}) {
  uint64_t const n = x.n;
  uint32_t const L = x.L;
  EWT_REQUIRE(L >= 1 && L <= kMaxPlanes, EWT_ERR_UNSUPPORTED, "too many levels for plane passes");
  uint32_t const sms = static_cast<uint32_t>(sm_count());
  std::vector<uint32_t> const ks = plan_plane_passes(L);
  uint64_t const stride = ceil_div(ceil_div(n, 32), 32) * 32 + 32;
  auto wants = [&](uint32_t level) -> uint32_t {
    for (auto const& w : wanted)
      if (w.first == level) return w.second;
    return 0;
  };
  std::vector<OrderPlanes> kept;
  auto make_order = [&](uint32_t level, uint32_t count) {
    OrderPlanes o;
    o.level = level;
    o.first = level + 1;
    o.count = count;
    o.kept = std::min(wants(level), count);
    o.front = count * stride * 4 > limits.split_bytes ? o.kept : count;
    o.stride = stride;
    if (o.front) o.mem.alloc(o.front * stride * 4);
    if (count > o.front) o.rest.alloc((count - o.front) * stride * 4);
    return o;
  };
  OrderPlanes cur = make_order(0, L - 1);
  DevBuf starts_buf[2], scratch;
  uint32_t nodes = x.nodes;
  uint64_t* starts = x.starts;
  if (nodes == 1) {
    starts_buf[0].alloc(16);
    starts = starts_buf[0].as<uint64_t>();
  }
  // ---- every pass's tiles, and one allocation for the nodes' tables
  std::vector<TileGrid> grids(ks.size());
  DevBuf tables;
  {
    size_t bytes = 0;
    std::vector<size_t> at;
    uint64_t nd = nodes;
    for (size_t i = 0, a = 0; i < ks.size(); a += ks[i], nd <<= ks[i], ++i) {
      TileGrid& g = grids[i];
      g.n = n;
      g.nodes = static_cast<uint32_t>(nd);
      g.halves = i + 1 == ks.size() && ks[i];
      g.D = std::max(ks[i], 1u);
      g.tile = pass_tile(pass_slots(static_cast<uint32_t>(L - 1 - a)), kSlotWords, ks[i]);
      // chunks of up to 8 tiles while every CTA still gets several
      g.ct = static_cast<uint32_t>(std::min<uint64_t>(
          8, std::max<uint64_t>(1, n / g.tile / (uint64_t(sms) * 12))));
      g.rc = ceil_div(64, g.ct);  // 64 tiles a range
      at.push_back(bytes);
      bytes += 3 * ((nd + 1) * 4 + 255) / 256 * 256;
    }
    tables.alloc(bytes);
    for (size_t i = 0; i < grids.size(); ++i) {
      uint32_t* const first = reinterpret_cast<uint32_t*>(tables.as<unsigned char>() + at[i]);
      grids[i].tile_first = first;
      grids[i].chunk_first = first + grids[i].nodes + 1;
      grids[i].range_first = first + 2 * (uint64_t(grids[i].nodes) + 1);
    }
  }
  uint32_t a = 0;
  bool tables_made = false;  // of this pass, by the one before
  for (size_t i = 0; i < ks.size(); ++i) {
    uint32_t const k = ks[i], b = a + k, np = L - 1 - a;
    bool const final = i + 1 == ks.size();
    uint32_t const slots = pass_slots(np);
    TileGrid& g = grids[i];
    uint64_t const max_tiles = n / g.tile + nodes;
    uint64_t const max_chunks = n / (uint64_t(g.tile) * g.ct) + nodes;
    EWT_REQUIRE(max_tiles < INT32_MAX, EWT_ERR_UNSUPPORTED, "text too long");
    uint64_t const max_ranges = max_chunks / g.rc + nodes;
    // one allocation for the pass's counts
    size_t bytes = 0;
    auto room = [&](uint64_t b) {
      size_t const at = bytes;
      bytes += (b + 255) / 256 * 256;
      return at;
    };
    size_t const at_cnt = room((max_tiles << g.D) * 2), at_pre = room((max_chunks << g.D) * 8),
                 at_tot = room((max_ranges << g.D) * 8);
    scratch.alloc(bytes);
    unsigned char* const base = scratch.as<unsigned char>();
    uint64_t* next_starts = starts_out;
    if (!final) {
      DevBuf& sb = starts_buf[(i + 1) & 1];
      sb.alloc(((uint64_t(nodes) << g.D) + 1) * 8);
      next_starts = sb.as<uint64_t>();
    }
    g.starts = starts;
    g.tile_cnt = reinterpret_cast<uint16_t*>(base + at_cnt);
    g.chunk_pre = reinterpret_cast<uint64_t*>(base + at_pre);
    g.range_tot = reinterpret_cast<uint64_t*>(base + at_tot);
    g.starts_next = next_starts;
    uint32_t const scan_grid = static_cast<uint32_t>(
        std::min<uint64_t>(max_tiles, uint64_t(sms) * 6));
    if (i == 0) {
      PhaseTimer pt(x.ingest_phase, st);
      IngestArgs ia{};
      ia.n = n;
      ia.L = L;
      ia.D = g.D;
      ia.tile = g.tile;
      ia.plane[0] = words[0];
      for (uint32_t j = 1; j < L; ++j) ia.plane[j] = cur.plane(j);
      ia.lut = x.lut;
      ia.max_symbol = x.max_symbol;
      ia.tile_cnt = nodes == 1 ? g.tile_cnt : nullptr;
      ia.err = err;
      ia.g = g;
      auto kern = x.lut ? ingest_planes_kernel<T, true> : ingest_planes_kernel<T, false>;
      uint64_t const tiles = ceil_div(n, g.tile);
      // (whole tiles of a multiple of eight symbols: parts stay aligned)
      uint64_t const step = x.part ? std::max<uint64_t>(1, x.part_symbols / g.tile) : tiles;
      for (ia.first = 0; ia.first < tiles; ia.first = ia.last) {
        ia.last = std::min(tiles, ia.first + step);
        uint64_t const begin = ia.first * g.tile;
        T const* const text =
            x.part ? x.part(begin, std::min(n, ia.last * g.tile) - begin) - begin : x.sym;
        kern<<<scan_grid, kIngestThreads, 0, st>>>(text, ia);
        EWT_LAUNCHED();
      }
    }
    // ---- the pass's outputs
    PlanePass p{};
    p.g = g;
    p.k = k;
    p.np = np;
    p.ext_words = stride;
    p.src[0] = words[a];
    for (uint32_t j = 1; j <= np; ++j) p.src[j] = cur.plane(a + j);
    OrderPlanes next;
    for (uint32_t r = 1; r <= k; ++r) {
      p.out[r] = words[a + r];
      p.out_words[r] = word_count[a + r];
      bool const whole = r == k && !final;  // the next pass's input
      uint32_t const count = whole ? np - k : std::min(wants(a + r), np - r);
      if (!count) continue;
      OrderPlanes o = make_order(a + r, count);
      for (uint32_t j = 1; j <= count; ++j) {
        p.ext[r][r + j] = o.plane(a + r + j);
        p.ext_mask[r] |= 1u << (r + j);
      }
      if (whole) next = std::move(o);
      else kept.push_back(std::move(o));
    }
    bool const few_tiles = max_tiles <= 2048;
    bool const clears = few_tiles && k && n / g.tile <= 256;
    {
      PhaseTimer pt(EWT_PHASE_HIST, st);
      if (nodes > 1 && !tables_made) {
        tile_table_kernel<<<1, 1024, 0, st>>>(g);
        EWT_LAUNCHED();
      }
      if (i > 0 || nodes > 1) {
        PlaneSources src{};
        src.p[0] = words[a];
        for (uint32_t j = 1; j < g.D; ++j) src.p[j] = cur.plane(a + j);
        auto kern = g.D == 1   ? plane_counts_kernel<1>
                    : g.D == 2 ? plane_counts_kernel<2>
                    : g.D == 3 ? plane_counts_kernel<3>
                               : plane_counts_kernel<4>;
        kern<<<one_wave(kern, kCountThreads, 0, max_tiles), kCountThreads, 0, st>>>(src, g);
        EWT_LAUNCHED();
      }
      // One launch while the tiles are few enough for the warps of one CTA,
      // should a single node hold them all (16 Mi symbols, 520 tiles: 7 us
      // against 17 us by three launches); it clears the outputs' shared words
      // up to eight tiles a warp (about 3 us, as long as a launch takes).
      uint32_t const range_grid = static_cast<uint32_t>(ceil_div(max_ranges, kRangeWarps));
      tables_made = few_tiles && nodes == 1 && !final;
      if (few_tiles) {
        PlanePass scanned = p;
        scanned.k = clears ? k : 0;
        TileGrid following{};
        if (tables_made) following = grids[i + 1];
        node_scan_kernel<<<nodes, nodes == 1 ? 1024 : nodes <= 64 ? 512 : 128, 0, st>>>(
            scanned, following);
        EWT_LAUNCHED();
      } else {
        range_totals_kernel<<<range_grid, kRangeWarps * 32, 0, st>>>(g);
        EWT_LAUNCHED();
        digit_starts_kernel<<<nodes, nodes <= 64 ? 1024 : 128, 0, st>>>(g);
        EWT_LAUNCHED();
        if (k) {
          chunk_starts_kernel<<<range_grid, kRangeWarps * 32, 0, st>>>(g);
          EWT_LAUNCHED();
        }
      }
    }
    if (k == 0) break;
    {
      PhaseTimer pt(EWT_PHASE_SPLIT, st);
      if (!clears) {
        clear_edges_kernel<<<static_cast<uint32_t>(std::min<uint64_t>(
                                 ceil_div(max_chunks, 4), uint64_t(sms) * 8)),
                             128, 0, st>>>(p);
        EWT_LAUNCHED();
      }
      launch_plane_pass(p, slots, max_chunks, limits.wide_words, st);
    }
    if (cur.kept) {  // the rest makes room for what is built next
      cur.rest.reset();
      cur.count = cur.kept;
      kept.push_back(std::move(cur));
    }
    cur = std::move(next);
    starts = next_starts;
    nodes <<= k;
    a = b;
  }
  return kept;
}

}  // namespace
}  // namespace ewt
