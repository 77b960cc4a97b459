// Group query levels: runs of w = 2 (quad) or 3
// (octal) consecutive binary levels l .. l+w-1 become one level of w-bit
// digits in level-l order, so a query resolves w binary levels per
// dependent DRAM access.  The plan covers all L levels: as many octal
// groups as fit, then one or two quad groups (L = 8: 3 + 3 + 2).  No
// reference counterpart; the binary levels and their RankSelect stay the
// source of truth for exports.
//
// Over an alphabet of no power of two they hold the minimal codes padded with
// zero bits to L bits, for every position of the text on every level (the
// passes carry ended codes to the end of the later orders), so the walks are
// those of a power-of-two tree of 2^L codes.
//
// A digit's bits are the planes l .. l+w-1 of the level-l order: plane l is
// the binary level l, the deeper ones come from the pass that wrote that
// order (planes.cuh; the per-level split of larger alphabets extracts them
// from the symbols of its level orders).  Per group level:
//   1. group_counts_kernel (warp per superblock): its digit counts, by
//      popcounts of the planes and of their intersections;
//   2. group_scan_*: counts before every superblock (chunked scan);
//   3. group_level_kernel (CTA per superblock, thread per block): block
//      headers from a CTA scan, blocks and dense select samples written;
//      the superblock's totals are checked against pass 1, the level's
//      against the count table.
// Node ranks (digit counts before every node) and digit totals come from
// the count table on the host.
#include <algorithm>
#include <vector>

#include "internal.cuh"

namespace ewt {

using ecl::detail::GroupShape;
using ecl::detail::kQuadDigits;
using ecl::detail::kQuadSbBlocks;
using ecl::detail::kQuadSbDigits;
using ecl::detail::GroupLevel;
using ecl::detail::GroupView;

constexpr uint32_t kOctDigits = GroupShape<3>::kDigits;
constexpr uint32_t kOctSbBlocks = GroupShape<3>::kSbBlocks;
constexpr uint64_t kOctSbDigits = uint64_t(kOctDigits) * kOctSbBlocks;

namespace {

constexpr uint32_t kScanChunk = 4096;   // superblock entries per scan CTA

// Bits 2k of the result take bit k of x (k < 16).
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

// Block-wide exclusive scan of a uint64 (blockDim.x a multiple of 32, at
// most 1024); *total receives the sum.
__device__ __forceinline__ uint64_t cta_exclusive_scan(uint64_t x, uint64_t* total) {
  __shared__ uint64_t warp_sums[32];
  uint32_t const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t inc = x;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    uint64_t const y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warp_sums[wid] = inc;
  __syncthreads();
  uint32_t const nwarps = blockDim.x >> 5;
  if (wid == 0) {
    uint64_t t = lane < nwarps ? warp_sums[lane] : 0;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      uint64_t const y = __shfl_up_sync(0xFFFFFFFFu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nwarps) warp_sums[lane] = t;  // inclusive over warps
  }
  __syncthreads();
  uint64_t const before = wid ? warp_sums[wid - 1] : 0;
  *total = warp_sums[nwarps - 1];
  __syncthreads();
  return before + inc - x;
}

// Scan 1: per chunk of kScanChunk superblock entries (S digits each), the
// S sums.
template <uint32_t S>
__global__ void __launch_bounds__(256)
group_scan_partial_kernel(uint64_t const* __restrict__ sb, uint64_t count,
                          uint64_t* __restrict__ chunk) {
  uint64_t const first = uint64_t(blockIdx.x) * kScanChunk;
  uint64_t c[S];
#pragma unroll
  for (uint32_t d = 0; d < S; ++d) c[d] = 0;
  for (uint64_t i = first + threadIdx.x; i < min(count, first + kScanChunk);
       i += blockDim.x)
#pragma unroll
    for (uint32_t d = 0; d < S; ++d) c[d] += sb[i * S + d];
#pragma unroll
  for (uint32_t d = 0; d < S; ++d) {
    uint64_t tot = 0;
    cta_exclusive_scan(c[d], &tot);
    if (threadIdx.x == 0) chunk[blockIdx.x * S + d] = tot;
  }
}

// Scan 2: exclusive prefix of the chunk sums (one thread per digit).
template <uint32_t S>
__global__ void group_scan_chunks_kernel(uint64_t* __restrict__ chunk,
                                         uint64_t chunks) {
  uint32_t const d = threadIdx.x;
  if (d >= S) return;
  uint64_t run = 0;
  for (uint64_t i = 0; i < chunks; ++i) {
    uint64_t const x = chunk[i * S + d];
    chunk[i * S + d] = run;
    run += x;
  }
}

// Scan 3: exclusive prefix of every entry, in place (1024 threads; two
// digits packed per 64-bit scan: every entry is below 2^16, a round's sums
// below 2^32).
template <uint32_t S>
__global__ void __launch_bounds__(1024)
group_scan_apply_kernel(uint64_t* __restrict__ sb, uint64_t count,
                        uint64_t const* __restrict__ chunk) {
  uint64_t const first = uint64_t(blockIdx.x) * kScanChunk;
  uint64_t const end = min(count, first + kScanChunk);
  uint64_t carry[S];
  for (uint32_t d = 0; d < S; ++d) carry[d] = chunk ? chunk[blockIdx.x * S + d] : 0;
  for (uint64_t base = first; base < end; base += blockDim.x) {
    uint64_t const i = base + threadIdx.x;
    bool const in = i < end;
#pragma unroll
    for (uint32_t k = 0; k < S / 2; ++k) {
      uint4 const a = in ? reinterpret_cast<uint4 const*>(sb + i * S)[k]
                         : make_uint4(0, 0, 0, 0);
      uint64_t tot = 0;
      uint64_t const e = cta_exclusive_scan(uint64_t(a.x) | (uint64_t(a.z) << 32), &tot);
      if (in) {
        sb[i * S + 2 * k] = carry[2 * k] + (e & 0xFFFFFFFFu);
        sb[i * S + 2 * k + 1] = carry[2 * k + 1] + (e >> 32);
      }
      carry[2 * k] += tot & 0xFFFFFFFFu;
      carry[2 * k + 1] += tot >> 32;
    }
  }
}

// Counts before every superblock of one level's table (nsb + 1 entries of
// S digits, the last one zero before and the totals after).
template <uint32_t S>
void scan_superblocks(uint64_t* sb, uint64_t entries, DevBuf& chunk, cudaStream_t st) {
  uint64_t const chunks = ceil_div(entries, kScanChunk);
  if (chunks > 1) {
    group_scan_partial_kernel<S><<<static_cast<uint32_t>(chunks), 256, 0, st>>>(
        sb, entries, chunk.as<uint64_t>());
    EWT_LAUNCHED();
    group_scan_chunks_kernel<S><<<1, 32, 0, st>>>(chunk.as<uint64_t>(), chunks);
    EWT_LAUNCHED();
  }
  group_scan_apply_kernel<S><<<static_cast<uint32_t>(chunks), 1024, 0, st>>>(
      sb, entries, chunks > 1 ? chunk.as<uint64_t>() : nullptr);
  EWT_LAUNCHED();
}

// Dense samples of one block: entry k of digit d names the block holding
// its (k * R + 1)-th occurrence, R = 2^sel_shift <= 2^16; before/c =
// occurrences before / in it (S = 2^width digits).  The first multiple of R
// at or after `before` is before + ((R - before) mod R): an entry lies in the
// block iff that offset is below c (32-bit test; 64-bit work only then).
template <uint32_t S>
__device__ __forceinline__ void put_group_samples(uint32_t* __restrict__ ds,
                                                  GroupLevel const& ql, uint64_t blk,
                                                  uint64_t const before[S],
                                                  uint32_t const c[S]) {
  uint32_t const sh = ql.sel_shift;
  uint32_t const rm = (1u << sh) - 1u;
#pragma unroll
  for (uint32_t d = 0; d < S; ++d) {
    uint32_t const off = (0u - static_cast<uint32_t>(before[d])) & rm;
    if (off >= c[d]) continue;  // the common case: no entry here
    uint32_t* S_ = ds + ql.ds_off[d];
    uint64_t k = (before[d] + off) >> sh;
    for (uint32_t o = off; o < c[d]; o += rm + 1, ++k) S_[k] = static_cast<uint32_t>(blk);
  }
}

// 64 bits of a plane from bit q on (the arrays have slack behind their end).
__device__ __forceinline__ uint64_t bits64(uint32_t const* __restrict__ w, uint64_t q) {
  uint64_t const i = q >> 5;
  uint32_t const s = static_cast<uint32_t>(q) & 31u;
  uint32_t const a = __ldg(w + i), b = __ldg(w + i + 1), c = __ldg(w + i + 2);
  return uint64_t(__funnelshift_r(a, b, s)) | (uint64_t(__funnelshift_r(b, c, s)) << 32);
}

// The planes of a group level, the digit's highest bit first.
struct GroupPlanes {
  uint32_t const* p[3];
};

// Digit counts from the popcounts of the planes and their intersections:
// for W = 3 {h, m, b, hm, hb, mb, hmb}, for W = 2 {h, b, hb}; n positions.
template <int W>
__device__ __forceinline__ void digit_counts(uint32_t const* s, uint32_t n, uint32_t* c) {
  if constexpr (W == 2) {
    c[3] = s[2];
    c[2] = s[0] - s[2];
    c[1] = s[1] - s[2];
    c[0] = n - s[0] - c[1];
  } else {
    c[7] = s[6];
    c[6] = s[3] - s[6];
    c[5] = s[4] - s[6];
    c[3] = s[5] - s[6];
    c[4] = s[0] - c[7] - c[6] - c[5];
    c[2] = s[1] - c[7] - c[6] - c[3];
    c[1] = s[2] - c[7] - c[5] - c[3];
    c[0] = n - s[0] - c[3] - c[2] - c[1];
  }
}

// Pass 1: digit counts of every superblock (a warp each; whole words).  The
// planes hold zeros past position n.  Bound by reading the planes once.
template <int W>
__global__ void __launch_bounds__(256)
group_counts_kernel(GroupPlanes g, uint64_t n, uint64_t nsb, uint64_t* __restrict__ sb) {
  constexpr uint32_t S = 1u << W, K = S - 1;
  constexpr uint32_t kWords = GroupShape<W>::kDigits * GroupShape<W>::kSbBlocks / 32;
  uint64_t const s = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  uint32_t const lane = threadIdx.x & 31;
  if (s > nsb) return;
  uint32_t acc[K];
#pragma unroll
  for (uint32_t i = 0; i < K; ++i) acc[i] = 0;
  uint64_t const first = s * kWords * 32;
  uint32_t const total =
      s < nsb && first < n ? static_cast<uint32_t>(min(uint64_t(kWords) * 32, n - first)) : 0u;
#pragma unroll 4
  for (uint32_t i = lane; i * 32 < total; i += 32) {
    uint64_t const w = s * kWords + i;
    uint32_t const h = __ldg(g.p[0] + w), m = __ldg(g.p[1] + w);
    acc[0] += __popc(h);
    acc[1] += __popc(m);
    if constexpr (W == 2) {
      acc[2] += __popc(h & m);
    } else {
      uint32_t const b = __ldg(g.p[2] + w);
      acc[2] += __popc(b);
      acc[3] += __popc(h & m);
      acc[4] += __popc(h & b);
      acc[5] += __popc(m & b);
      acc[6] += __popc(h & m & b);
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < K; ++i) acc[i] = __reduce_add_sync(0xFFFFFFFFu, acc[i]);
  uint32_t c[S];
  digit_counts<W>(acc, total, c);
#pragma unroll
  for (uint32_t d = 0; d < S; ++d)
    if (lane == d) sb[s * S + d] = c[d];  // entry nsb: zeros
}

// Exclusive scan of four uint32 over a CTA of 512 threads.
__device__ __forceinline__ uint4 cta_exclusive_scan4(uint4 x, uint4* total) {
  __shared__ uint4 ws[16];
  uint32_t const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint4 inc = x;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    uint32_t const a = __shfl_up_sync(0xFFFFFFFFu, inc.x, o);
    uint32_t const b = __shfl_up_sync(0xFFFFFFFFu, inc.y, o);
    uint32_t const c = __shfl_up_sync(0xFFFFFFFFu, inc.z, o);
    uint32_t const d = __shfl_up_sync(0xFFFFFFFFu, inc.w, o);
    if (lane >= o) { inc.x += a; inc.y += b; inc.z += c; inc.w += d; }
  }
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    uint4 t = lane < 16 ? ws[lane] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t o = 1; o < 16; o <<= 1) {
      uint32_t const a = __shfl_up_sync(0xFFFFFFFFu, t.x, o);
      uint32_t const b = __shfl_up_sync(0xFFFFFFFFu, t.y, o);
      uint32_t const c = __shfl_up_sync(0xFFFFFFFFu, t.z, o);
      uint32_t const d = __shfl_up_sync(0xFFFFFFFFu, t.w, o);
      if (lane >= o) { t.x += a; t.y += b; t.z += c; t.w += d; }
    }
    if (lane < 16) ws[lane] = t;
  }
  __syncthreads();
  uint4 const before = wid ? ws[wid - 1] : make_uint4(0, 0, 0, 0);
  *total = ws[15];
  return make_uint4(before.x + inc.x - x.x, before.y + inc.y - x.y,
                    before.z + inc.z - x.z, before.w + inc.w - x.w);
}

// Pass 3: a CTA of 512 threads per superblock, thread t its block t: the
// block's bits of every plane, digit counts by popcounts, the header from a
// CTA scan of them (two 16-bit counts per word: a superblock holds fewer
// than 2^16 digits), and the dense samples.
template <int W>
__global__ void __launch_bounds__(512, 3)
group_level_kernel(GroupPlanes g, uint64_t n, GroupLevel ql, uint4* __restrict__ blocks,
                   uint64_t const* __restrict__ sb, uint64_t nsb,
                   uint32_t* __restrict__ ds, uint32_t* __restrict__ err) {
  constexpr uint32_t S = 1u << W, kD = GroupShape<W>::kDigits, kSb = GroupShape<W>::kSbBlocks;
  uint64_t const sbi = blockIdx.x;
  uint32_t const t = threadIdx.x;
  uint64_t const blk = sbi * kSb + t;
  bool const mine = blk < ql.num_blocks;
  uint64_t const p = blk * kD;
  uint32_t const valid =
      mine && p < n ? static_cast<uint32_t>(min(uint64_t(kD), n - p)) : 0u;
  uint32_t c[S];
  uint64_t H = 0, M = 0, B = 0;          // octal: 42 bits of each plane
  uint32_t h[3] = {0, 0, 0}, b[3] = {0, 0, 0};  // quad: three words of each
  if constexpr (W == 3) {
    if (valid) {
      uint64_t const vm = (1ull << valid) - 1;
      H = bits64(g.p[0], p) & vm;
      M = bits64(g.p[1], p) & vm;
      B = bits64(g.p[2], p) & vm;
    }
    uint32_t const s[7] = {uint32_t(__popcll(H)),     uint32_t(__popcll(M)),
                           uint32_t(__popcll(B)),     uint32_t(__popcll(H & M)),
                           uint32_t(__popcll(H & B)), uint32_t(__popcll(M & B)),
                           uint32_t(__popcll(H & M & B))};
    digit_counts<3>(s, valid, c);
  } else {
    uint32_t s[3] = {0, 0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) {
      uint32_t const v = valid > 32 * k ? min(32u, valid - 32 * k) : 0u;
      if (v) {
        uint32_t const vm = v == 32 ? ~0u : (1u << v) - 1u;
        h[k] = __ldg(g.p[0] + blk * 3 + k) & vm;
        b[k] = __ldg(g.p[1] + blk * 3 + k) & vm;
      }
      s[0] += __popc(h[k]);
      s[1] += __popc(b[k]);
      s[2] += __popc(h[k] & b[k]);
    }
    digit_counts<2>(s, valid, c);
  }
  uint4 x = make_uint4(c[0] | (c[1] << 16), c[2] | (c[3] << 16), 0, 0);
  if constexpr (W == 3) {
    x.z = c[4] | (c[5] << 16);
    x.w = c[6] | (c[7] << 16);
  }
  uint4 tot;
  uint4 const e = cta_exclusive_scan4(x, &tot);
  uint64_t const* sbe = sb + sbi * S;
  if (t < S) {  // pass 1's counts must agree, and the level's totals
    uint32_t const w4[4] = {tot.x, tot.y, tot.z, tot.w};
    uint32_t const own = (w4[t >> 1] >> (16 * (t & 1))) & 0xFFFFu;
    if (sbe[S + t] - sbe[t] != own) atomicOr(err, 2u);
    if (sbi == 0 && sb[nsb * S + t] != ql.total[t]) atomicOr(err, 4u);
  }
  if (!mine) return;
  uint4* out = blocks + blk * 2;
  if constexpr (W == 3) {
    // planes H, M, B in words 1..3, counts of digits 4..6 above them
    uint64_t const w1 = H | (uint64_t(e.z & 0xFFFFu) << 42);
    uint64_t const w2 = M | (uint64_t(e.z >> 16) << 42);
    uint64_t const w3 = B | (uint64_t(e.w & 0xFFFFu) << 42);
    out[0] = make_uint4(e.x, e.y, static_cast<uint32_t>(w1), static_cast<uint32_t>(w1 >> 32));
    out[1] = make_uint4(static_cast<uint32_t>(w2), static_cast<uint32_t>(w2 >> 32),
                        static_cast<uint32_t>(w3), static_cast<uint32_t>(w3 >> 32));
  } else {
    uint32_t dw[6];
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) {
      dw[2 * k] = spread16(b[k]) | (spread16(h[k]) << 1);
      dw[2 * k + 1] = spread16(b[k] >> 16) | (spread16(h[k] >> 16) << 1);
    }
    out[0] = make_uint4(e.x, e.y & 0xFFFFu, dw[0], dw[1]);
    out[1] = make_uint4(dw[2], dw[3], dw[4], dw[5]);
  }
  if (ds && ql.sel_shift) {
    uint32_t const hd[8] = {e.x & 0xFFFFu, e.x >> 16, e.y & 0xFFFFu, e.y >> 16,
                            e.z & 0xFFFFu, e.z >> 16, e.w & 0xFFFFu, e.w >> 16};
    uint64_t before[S];
#pragma unroll
    for (uint32_t d = 0; d < S; ++d) before[d] = sbe[d] + hd[d];
    put_group_samples<S>(ds, ql, blk, before, c);
  }
}

// Dense samples of one group level from its finished blocks and scanned
// superblock table (samples at another rate; a build's are written with the
// blocks).
template <int W>
__global__ void __launch_bounds__(256)
group_samples_kernel(uint4 const* __restrict__ blocks, uint64_t const* __restrict__ sb,
                     uint64_t n, GroupLevel ql, uint32_t* __restrict__ ds) {
  constexpr uint32_t S = 1u << W;
  constexpr uint32_t kD = GroupShape<W>::kDigits, kSb = GroupShape<W>::kSbBlocks;
  uint64_t const b = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (!ds || ql.sel_shift == 0 || b >= ql.num_blocks) return;
  uint4 const x = blocks[b * 2], y = blocks[b * 2 + 1];
  uint64_t q[4];
  ecl::detail::quad_words(x, y, q);
  uint64_t const first = b * kD;
  uint32_t const valid = first < n ? static_cast<uint32_t>(min(uint64_t(kD), n - first)) : 0u;
  uint4 const* sb4 = reinterpret_cast<uint4 const*>(sb + (b / kSb) * S);
  uint64_t sbv[S];
#pragma unroll
  for (uint32_t k = 0; k < S / 2; ++k) {
    uint4 const e = sb4[k];
    sbv[2 * k] = uint64_t(e.y) << 32 | e.x;
    sbv[2 * k + 1] = uint64_t(e.w) << 32 | e.z;
  }
  uint64_t before[S];
  uint32_t c[S];
  if constexpr (W == 3) {  // headers parsed once, counts from the planes
    uint64_t const vm = (1ull << valid) - 1;
    uint64_t const H = q[1] & vm, M = q[2] & vm, B = q[3] & vm;
    uint32_t h[8];
    h[0] = static_cast<uint32_t>(q[0]) & 0xFFFFu;
    h[1] = static_cast<uint32_t>(q[0] >> 16) & 0xFFFFu;
    h[2] = static_cast<uint32_t>(q[0] >> 32) & 0xFFFFu;
    h[3] = static_cast<uint32_t>(q[0] >> 48);
    h[4] = static_cast<uint32_t>(q[1] >> 42) & 0xFFFFu;
    h[5] = static_cast<uint32_t>(q[2] >> 42) & 0xFFFFu;
    h[6] = static_cast<uint32_t>(q[3] >> 42) & 0xFFFFu;
    h[7] = static_cast<uint32_t>(b % kSb) * kD - h[0] - h[1] - h[2] - h[3] - h[4] -
           h[5] - h[6];
#pragma unroll
    for (uint32_t d = 0; d < S; ++d) {
      c[d] = __popcll((d & 4 ? H : ~H) & (d & 2 ? M : ~M) & (d & 1 ? B : ~B) & vm);
      before[d] = sbv[d] + h[d];
    }
  } else {
#pragma unroll
    for (uint32_t d = 0; d < S; ++d) {
      c[d] = ecl::detail::group_count<W>(q, d, valid);
      before[d] = ecl::detail::group_before<W>(q, sbv[d], d, b);
    }
  }
  put_group_samples<S>(ds, ql, b, before, c);
}

// Sample shift of a group level for the tree-wide rate 2^shift: octal
// digits are about half as frequent and blocks hold 42 instead of 96, and
// the interpolated block is off by more blocks at equal bracket width, so
// octal levels sample 8 times as densely.
uint32_t level_shift(uint32_t width, uint32_t shift) {
  if (shift == 0) return 0;
  return width == 3 ? std::max<uint32_t>(shift, 7) - 3 : shift;
}

// Lays out the dense samples of every group level at rate 2^shift.
void layout_group_samples(GroupStore& qs, uint32_t shift) {
  qs.ds.reset();
  qs.sel_shift = shift;
  uint64_t total = 0;
  for (auto& ql : qs.levels) {
    ql.sel_shift = level_shift(ql.width, shift);
    for (uint32_t d = 0; d < 8; ++d) ql.ds_off[d] = 0;
    if (!ql.sel_shift) continue;
    for (uint32_t d = 0; d < (1u << ql.width); ++d) {
      ql.ds_off[d] = total;
      total += ceil_div(ql.total[d], uint64_t(1) << ql.sel_shift);
    }
  }
  if (shift) qs.ds.alloc(std::max<uint64_t>(total, 1) * 4);
}

void run_group_samples(GroupStore& qs, uint64_t n, cudaStream_t st) {
  if (!qs.ds.get()) return;
  for (auto const& ql : qs.levels) {
    uint32_t* const ds = qs.ds.get() ? qs.ds.as<uint32_t>() : nullptr;
    uint32_t const grid = static_cast<uint32_t>(ceil_div(ql.num_blocks, 256));
    uint4 const* const blocks = qs.blocks.as<uint4>() + ql.blk_off * 2;
    uint64_t const* const sb = qs.sb.as<uint64_t>() + ql.sb_off;
    if (ql.width == 3)
      group_samples_kernel<3><<<grid, 256, 0, st>>>(blocks, sb, n, ql, ds);
    else
      group_samples_kernel<2><<<grid, 256, 0, st>>>(blocks, sb, n, ql, ds);
    EWT_LAUNCHED();
  }
}

void upload_levels(GroupStore& qs, cudaStream_t st) {
  qs.levels_d.alloc(std::max<size_t>(qs.levels.size(), 1) * sizeof(GroupLevel));
  if (!qs.levels.empty())
    EWT_CUDA(cudaMemcpyAsync(qs.levels_d.get(), qs.levels.data(),
                             qs.levels.size() * sizeof(GroupLevel),
                             cudaMemcpyHostToDevice, st));
}

}  // namespace

std::vector<uint32_t> group_widths(uint32_t L) {
  std::vector<uint32_t> w;
  if (L < 2) return w;
  uint32_t const quads = L % 3 == 0 ? 0 : L % 3 == 2 ? 1 : 2;
  for (uint32_t i = 0; i < (L - 2 * quads) / 3; ++i) w.push_back(3);
  for (uint32_t i = 0; i < quads; ++i) w.push_back(2);
  return w;
}

GroupView GroupStore::view() const {
  GroupView v{};
  if (levels.empty() || !blocks.get()) return v;
  v.blocks = blocks.as<uint4>();
  v.sb = sb.as<uint64_t>();
  v.ds = sel_shift && ds.get() ? ds.as<uint32_t>() : nullptr;
  v.node_ranks = node_ranks.as<uint64_t>();
  v.levels = levels_d.as<GroupLevel>();
  v.num = static_cast<uint32_t>(levels.size());
  uint32_t covered = 0;
  for (auto const& ql : levels) covered += ql.width;
  v.covered = covered;
  v.counts = counts.as<uint64_t>();
  v.code = code.as<uint16_t>();
  v.symbol = symbol.as<uint16_t>();
  return v;
}

bool groups_eligible(ewt_tree const& t) {
  return (t.pow2 || t.L <= 16) && t.L >= 2 && t.n >= 1;
}

std::vector<uint64_t> code_counts(ewt_tree const& t) {
  std::vector<uint64_t> C((uint64_t(1) << t.L) + 1, 0);
  for (uint64_t i = 0; i < t.sigma; ++i) C[padded_code(t, i) + 1] = t.occ[i];
  for (size_t i = 1; i < C.size(); ++i) C[i] += C[i - 1];
  return C;
}

void upload_group_codes(ewt_tree& t, std::vector<uint64_t> const& C, cudaStream_t st) {
  if (t.pow2) return;
  std::vector<uint16_t> code(t.sigma), symbol(C.size() - 1, 0);
  for (uint64_t i = 0; i < t.sigma; ++i) {
    uint64_t const c = padded_code(t, i);
    code[i] = static_cast<uint16_t>(c);
    symbol[c] = static_cast<uint16_t>(i);
  }
  GroupStore& qs = t.groups;
  qs.counts.alloc(C.size() * 8);
  qs.code.alloc(code.size() * 2);
  qs.symbol.alloc(symbol.size() * 2);
  EWT_CUDA(cudaMemcpyAsync(qs.counts.get(), C.data(), C.size() * 8, cudaMemcpyHostToDevice, st));
  EWT_CUDA(cudaMemcpyAsync(qs.code.get(), code.data(), code.size() * 2,
                           cudaMemcpyHostToDevice, st));
  EWT_CUDA(cudaMemcpyAsync(qs.symbol.get(), symbol.data(), symbol.size() * 2,
                           cudaMemcpyHostToDevice, st));
  EWT_CUDA(cudaStreamSynchronize(st));  // the host tables leave scope
}

namespace {

// Block, superblock-table and level layout of a tree's group levels (needs n
// and L only); allocates the blocks and tables.
void layout_groups(ewt_tree& t) {
  GroupStore& qs = t.groups;
  uint64_t const n = t.n;
  std::vector<uint32_t> const widths = group_widths(t.L);
  uint64_t blk = 0, sbw = 0;
  qs.levels.assign(widths.size(), GroupLevel{});
  uint32_t l = 0;
  for (size_t j = 0; j < widths.size(); ++j) {
    uint32_t const w = widths[j];
    GroupLevel& ql = qs.levels[j];
    ql.width = w;
    ql.start = l;
    uint32_t const kD = w == 3 ? kOctDigits : kQuadDigits;
    uint32_t const kSb = w == 3 ? kOctSbBlocks : kQuadSbBlocks;
    ql.num_blocks = n / kD + 1;
    ql.blk_off = blk;
    ql.sb_off = sbw;
    blk += ql.num_blocks;
    sbw += (ceil_div(ql.num_blocks, uint64_t(kSb)) + 1) << w;  // + the totals entry
    l += w;
  }
  qs.blocks.alloc(blk * 32);
  qs.sb.alloc(sbw * 8);
}

template <int W>
void build_group_level(GroupStore& qs, GroupLevel const& ql, GroupPlanes const& g, uint64_t n,
                       DevBuf& chunk, uint32_t* err, cudaStream_t st) {
  uint64_t const nsb = ceil_div(ql.num_blocks, uint64_t(GroupShape<W>::kSbBlocks));
  uint64_t* const sb = qs.sb.as<uint64_t>() + ql.sb_off;
  group_counts_kernel<W><<<static_cast<uint32_t>(ceil_div(nsb + 1, 8)), 256, 0, st>>>(
      g, n, nsb, sb);
  EWT_LAUNCHED();
  scan_superblocks<(1u << W)>(sb, nsb + 1, chunk, st);
  group_level_kernel<W><<<static_cast<uint32_t>(nsb), 512, 0, st>>>(
      g, n, ql, qs.blocks.as<uint4>() + ql.blk_off * 2, sb, nsb,
      qs.ds.get() ? qs.ds.as<uint32_t>() : nullptr, err);
  EWT_LAUNCHED();
}

}  // namespace

std::vector<std::pair<uint32_t, uint32_t>> group_planes(uint32_t L) {
  std::vector<std::pair<uint32_t, uint32_t>> v;
  uint32_t l = 0;
  for (uint32_t w : group_widths(L)) {
    v.emplace_back(l, w - 1);
    l += w;
  }
  return v;
}

void build_groups(ewt_tree& t, std::vector<uint64_t> const& C,
                  std::vector<std::vector<uint32_t const*>> const& planes, cudaStream_t st) {
  GroupStore& qs = t.groups;
  qs.levels.clear();
  qs.blocks.reset();
  if (!groups_eligible(t)) return;
  PhaseTimer pt(EWT_PHASE_QUAD, st);
  uint32_t const L = t.L;
  uint64_t const n = t.n;
  EWT_REQUIRE(C.size() == (uint64_t(1) << L) + 1 && C.back() == n, EWT_ERR_CUDA,
              "count table inconsistent");
  upload_group_codes(t, C, st);
  layout_groups(t);
  EWT_REQUIRE(planes.size() == qs.levels.size(), EWT_ERR_CUDA, "group planes missing");
  // host: digit totals, node ranks
  std::vector<uint64_t> nr;
  uint64_t max_sb = 0;
  for (auto& ql : qs.levels) {
    uint32_t const w = ql.width, S = 1u << w, l = ql.start;
    ql.nr_off = nr.size();
    max_sb = std::max(max_sb, ceil_div(ql.num_blocks, uint64_t(w == 3 ? kOctSbBlocks
                                                                     : kQuadSbBlocks)));
    uint32_t const sh = L - l;  // symbols under a level-l node: 2^sh
    uint64_t const nodes = uint64_t(1) << l;
    uint64_t run[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint64_t g = 0; g < nodes; ++g)
      for (uint32_t d = 0; d < S; ++d) {
        nr.push_back(run[d]);
        uint64_t const pre = (g << w) | d;  // prefix of l + w bits
        run[d] += C[(pre + 1) << (sh - w)] - C[pre << (sh - w)];
      }
    for (uint32_t d = 0; d < S; ++d) ql.total[d] = run[d];
  }
  qs.node_ranks.alloc(nr.size() * 8);
  EWT_CUDA(cudaMemcpyAsync(qs.node_ranks.get(), nr.data(), nr.size() * 8,
                           cudaMemcpyHostToDevice, st));
  layout_group_samples(qs, qs.sel_shift);
  upload_levels(qs, st);
  DevBuf err_d(4);
  EWT_CUDA(cudaMemsetAsync(err_d.get(), 0, 4, st));
  DevBuf chunk(ceil_div(max_sb + 1, kScanChunk) * 8 * 8);
  for (size_t gi = 0; gi < qs.levels.size(); ++gi) {
    GroupLevel const& ql = qs.levels[gi];
    EWT_REQUIRE(planes[gi].size() == ql.width, EWT_ERR_CUDA, "group planes missing");
    GroupPlanes g{};
    for (uint32_t j = 0; j < ql.width; ++j) g.p[j] = planes[gi][j];
    if (ql.width == 3)
      build_group_level<3>(qs, ql, g, n, chunk, err_d.as<uint32_t>(), st);
    else
      build_group_level<2>(qs, ql, g, n, chunk, err_d.as<uint32_t>(), st);
  }
  uint32_t bad = 0;
  EWT_CUDA(cudaMemcpyAsync(&bad, err_d.get(), 4, cudaMemcpyDeviceToHost, st));
  EWT_CUDA(cudaStreamSynchronize(st));
  EWT_REQUIRE(bad == 0, EWT_ERR_CUDA,
              "internal consistency check failed (group levels, kind " +
                  std::to_string(bad) + ")");
}

void set_select_rate(ewt_tree& t, uint32_t shift, cudaStream_t st) {
  build_dense_samples(t.rs, shift, st);
  build_group_samples(t, shift, st);
  t.view.rs = t.rs.view();
  t.view.groups = t.groups.view();
}

void build_group_samples(ewt_tree& t, uint32_t shift, cudaStream_t st) {
  GroupStore& qs = t.groups;
  if (qs.levels.empty()) return;
  EWT_CUDA(cudaStreamSynchronize(st));  // no query may read the old samples
  layout_group_samples(qs, shift);
  upload_levels(qs, st);
  run_group_samples(qs, t.n, st);
  EWT_CUDA(cudaStreamSynchronize(st));
}

}  // namespace ewt
