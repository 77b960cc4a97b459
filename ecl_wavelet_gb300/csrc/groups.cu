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
//      popcounts of the planes and of their intersections, added up per chunk
//      of superblocks as well;
//   2. group_scan_kernel: counts before every superblock (CTA per chunk);
//   3. group_level_kernel (CTA per superblock, thread per two blocks): block
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

constexpr uint32_t kScanChunk = 512;   // superblock entries per scan CTA

// Bits 2k of the result take bit k of x (k < 16).
__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

// A block in one 32-byte store.
__device__ __forceinline__ void store_block(uint4* p, uint4 a, uint4 b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x),
               "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w));
}

// Inclusive warp scan.
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

// Pass 2: counts before every superblock, in place (a thread per entry of S
// digits, each below 2^16; chunk[c] = the digits of chunk c).  A CTA adds up
// the chunks before its own, so the scan is one launch: 6 Gi symbols have 586
// chunks.  (Three launches over chunks of 4,096 entries took 53 us a level at
// 2^28 symbols, this one 6 us.)
template <uint32_t S>
__global__ void __launch_bounds__(kScanChunk)
group_scan_kernel(uint64_t* __restrict__ sb, uint64_t count,
                  uint64_t const* __restrict__ chunk) {
  constexpr uint32_t kWarps = kScanChunk / 32;
  __shared__ uint64_t part[kWarps][32];
  __shared__ uint32_t warp_tot[S][kWarps];
  uint32_t const tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // lane l of every warp: digit l % S of chunks (l / S) + (32 / S) * (wid + kWarps * i)
  uint64_t sum = 0;
  for (uint32_t c = wid * (32 / S) + lane / S; c < blockIdx.x; c += kWarps * (32 / S))
    sum += chunk[uint64_t(c) * S + lane % S];
  part[wid][lane] = sum;
  uint64_t const i = uint64_t(blockIdx.x) * kScanChunk + tid;
  uint32_t x[S], inc[S];
#pragma unroll
  for (uint32_t k = 0; k < S / 2; ++k) {
    uint4 const a = i < count ? reinterpret_cast<uint4 const*>(sb + i * S)[k]
                              : make_uint4(0, 0, 0, 0);
    x[2 * k] = a.x;
    x[2 * k + 1] = a.z;
  }
#pragma unroll
  for (uint32_t d = 0; d < S; ++d) {
    inc[d] = warp_inclusive(x[d]);
    if (lane == 31) warp_tot[d][wid] = inc[d];
  }
  __syncthreads();
  uint64_t carry = 0;  // digit lane % S before the chunk
  if (wid == 0) {
    for (uint32_t w = 0; w < kWarps; ++w) carry += part[w][lane];
    for (uint32_t o = S; o < 32; o <<= 1) carry += __shfl_xor_sync(0xffffffffu, carry, o);
  }
  __syncthreads();
  if (wid == 0) part[0][lane] = carry;
  __syncthreads();
  if (i >= count) return;
#pragma unroll
  for (uint32_t d = 0; d < S; ++d) {
    uint32_t before = inc[d] - x[d];
    for (uint32_t w = 0; w < wid; ++w) before += warp_tot[d][w];
    sb[i * S + d] = part[0][d] + before;
  }
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

// The same, two counts to a word.
template <int W>
__device__ __forceinline__ void packed_counts(uint32_t const* s, uint32_t n, uint32_t* c) {
  uint32_t x[1 << W];
  digit_counts<W>(s, n, x);
#pragma unroll
  for (uint32_t k = 0; k < (1u << W) / 2; ++k) c[k] = x[2 * k] | x[2 * k + 1] << 16;
}

// Pass 1: digit counts of every superblock (a warp each; whole words).  The
// planes hold zeros past position n.  Bound by reading the planes once.
template <int W>
__global__ void __launch_bounds__(256)
group_counts_kernel(GroupPlanes g, uint64_t n, uint64_t nsb, uint64_t* __restrict__ sb,
                    unsigned long long* __restrict__ chunk) {
  constexpr uint32_t S = 1u << W, K = S - 1;
  constexpr uint32_t kWords = GroupShape<W>::kDigits * GroupShape<W>::kSbBlocks / 32;
  uint64_t const s = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5;
  uint32_t const lane = threadIdx.x & 31;
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
  uint32_t c[S], own = 0;
  digit_counts<W>(acc, total, c);
#pragma unroll
  for (uint32_t d = 0; d < S; ++d)
    if (lane == d) own = c[d];
  __shared__ uint32_t sum[8][S];  // the CTA's eight superblocks are of one chunk
  uint32_t const wid = threadIdx.x >> 5;
  if (lane < S) {
    if (s <= nsb) sb[s * S + lane] = own;  // entry nsb: zeros
    sum[wid][lane] = own;
  }
  __syncthreads();
  if (threadIdx.x < S) {
    uint32_t tot = 0;
    for (uint32_t w = 0; w < 8; ++w) tot += sum[w][threadIdx.x];
    if (tot) atomicAdd(chunk + s / kScanChunk * S + threadIdx.x, tot);
  }
}

// A build samples at the default rate R (group_samples_kernel writes others
// later): a superblock's counts and twice R stay within 16 bits.
constexpr uint32_t kBuildRate = 1u << ecl::detail::kDefaultSelShift;
static_assert(ecl::detail::kDefaultSelShift > 0 && kQuadSbDigits + 2 * kBuildRate <= 65536 &&
              kOctSbDigits + 2 * kBuildRate <= 65536);

// Pass 3: a CTA of 256 threads per superblock, thread t its blocks 2t and
// 2t + 1: their bits of every plane, digit counts by popcounts, the headers
// from one CTA scan (two 16-bit counts per word: a superblock holds fewer than
// 2^16 digits), and the dense samples, two digits at a time, from the
// superblock's own first entry and remainder.  A block goes out in one store
// of 32 bytes.  Bound by instructions (a quarter of them for the samples).
// All group levels of 2^30 symbols of 256 (counts, scans, blocks, samples):
// 1.02 ms; 1.06 with the samples digit by digit, 1.17 with two stores of 16
// bytes as well, 1.56 with a thread per block, three scan launches and a loop
// of 64-bit sample ranks.
template <int W>
__global__ void __launch_bounds__(256, 5)
group_level_kernel(GroupPlanes g, uint64_t n, GroupLevel ql, uint4* __restrict__ blocks,
                   uint64_t const* __restrict__ sb, uint64_t nsb,
                   uint32_t* __restrict__ ds, uint32_t* __restrict__ err) {
  constexpr uint32_t S = 1u << W, kD = GroupShape<W>::kDigits, kSb = GroupShape<W>::kSbBlocks;
  constexpr uint32_t kWarps = 8, kP = S / 2;  // packed count words
  static_assert(kSb == 512, "two blocks per thread");
  __shared__ uint32_t warp_tot[kWarps][4];
  __shared__ uint32_t* entry[S];  // the sample of the superblock's next multiple of R
  __shared__ uint32_t rem[kP];   // R - 1 + the occurrences since the one before it
  uint64_t const sbi = blockIdx.x;
  uint32_t const t = threadIdx.x, lane = t & 31, wid = t >> 5;
  uint64_t const blk = sbi * kSb + 2 * t, p = blk * kD;
  uint64_t const* sbe = sb + sbi * S;
  uint32_t const sh = ql.sel_shift, rm = (1u << sh) - 1u, rm2 = rm * 0x10001u;
  if (ds && t < S) entry[t] = ds + ql.ds_off[t] + (sbe[t] >> sh);
  if (ds && t < kP)
    rem[t] = ((static_cast<uint32_t>(sbe[2 * t]) & rm) |
              (static_cast<uint32_t>(sbe[2 * t + 1]) & rm) << 16) + rm2;
  uint32_t valid[2];
  valid[0] = p < n ? static_cast<uint32_t>(min(uint64_t(kD), n - p)) : 0u;
  valid[1] = p + kD < n ? static_cast<uint32_t>(min(uint64_t(kD), n - p - kD)) : 0u;
  uint32_t c[2][kP];
  uint64_t H[2], M[2], B[2];     // octal: 42 bits of each plane
  uint32_t h[2][3], b[2][3];     // quad: three words of each
  if constexpr (W == 3) {
    uint64_t const i = p >> 5;
    uint32_t const s = static_cast<uint32_t>(p) & 31u, s2 = s + kD;
    auto bits = [&](uint32_t const* __restrict__ w, uint64_t& x, uint64_t& y) {
      uint32_t a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = valid[0] ? __ldg(w + i + u) : 0u;
      x = (uint64_t(__funnelshift_r(a[1], a[2], s)) << 32) | __funnelshift_r(a[0], a[1], s);
      uint32_t const b0 = s2 < 64 ? a[1] : a[2], b1 = s2 < 64 ? a[2] : a[3],
                     b2 = s2 < 64 ? a[3] : 0u;
      y = (uint64_t(__funnelshift_r(b1, b2, s2)) << 32) | __funnelshift_r(b0, b1, s2);
      x &= (1ull << valid[0]) - 1;
      y &= (1ull << valid[1]) - 1;
    };
    bits(g.p[0], H[0], H[1]);
    bits(g.p[1], M[0], M[1]);
    bits(g.p[2], B[0], B[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint64_t const hm = H[u] & M[u];
      uint32_t const s7[7] = {uint32_t(__popcll(H[u])),        uint32_t(__popcll(M[u])),
                              uint32_t(__popcll(B[u])),        uint32_t(__popcll(hm)),
                              uint32_t(__popcll(H[u] & B[u])), uint32_t(__popcll(M[u] & B[u])),
                              uint32_t(__popcll(hm & B[u]))};
      packed_counts<3>(s7, valid[u], c[u]);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t s3[3] = {0, 0, 0};
#pragma unroll
      for (uint32_t k = 0; k < 3; ++k) {
        uint32_t const v = valid[u] > 32 * k ? min(32u, valid[u] - 32 * k) : 0u;
        uint32_t const vm = v == 32 ? ~0u : (1u << v) - 1u;
        h[u][k] = v ? __ldg(g.p[0] + (blk + u) * 3 + k) & vm : 0u;
        b[u][k] = v ? __ldg(g.p[1] + (blk + u) * 3 + k) & vm : 0u;
        s3[0] += __popc(h[u][k]);
        s3[1] += __popc(b[u][k]);
        s3[2] += __popc(h[u][k] & b[u][k]);
      }
      packed_counts<2>(s3, valid[u], c[u]);
    }
  }
  uint32_t e[kP];  // packed counts before block 2t
  {
    uint32_t x[kP];
#pragma unroll
    for (uint32_t k = 0; k < kP; ++k) {
      x[k] = c[0][k] + c[1][k];
      e[k] = warp_inclusive(x[k]);
      if (lane == 31) warp_tot[wid][k] = e[k];
    }
    __syncthreads();
    uint32_t tot[kP];
#pragma unroll
    for (uint32_t k = 0; k < kP; ++k) {
      tot[k] = 0;
      e[k] -= x[k];
    }
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w)
#pragma unroll
      for (uint32_t k = 0; k < kP; ++k) {
        uint32_t const y = warp_tot[w][k];
        if (w < wid) e[k] += y;
        tot[k] += y;
      }
    if (t == 0) {  // pass 1's counts must agree, and the level's totals
      bool ok = true, all = true;
#pragma unroll
      for (uint32_t d = 0; d < S; ++d) {
        uint32_t const own = (tot[d >> 1] >> (16 * (d & 1))) & 0xFFFFu;
        ok = ok && sbe[S + d] - sbe[d] == own;
        if (sbi == 0) all = all && sb[nsb * S + d] == ql.total[d];
      }
      if (!ok) atomicOr(err, 2u);
      if (!all) atomicOr(err, 4u);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (blk + u >= ql.num_blocks) return;
    if (u)
#pragma unroll
      for (uint32_t k = 0; k < kP; ++k) e[k] += c[0][k];
    uint4* out = blocks + (blk + u) * 2;
    if constexpr (W == 3) {
      // planes H, M, B in words 1..3, counts of digits 4..6 above them
      uint64_t const w1 = H[u] | (uint64_t(e[2] & 0xFFFFu) << 42);
      uint64_t const w2 = M[u] | (uint64_t(e[2] >> 16) << 42);
      uint64_t const w3 = B[u] | (uint64_t(e[3] & 0xFFFFu) << 42);
      store_block(out,
                  make_uint4(e[0], e[1], static_cast<uint32_t>(w1),
                             static_cast<uint32_t>(w1 >> 32)),
                  make_uint4(static_cast<uint32_t>(w2), static_cast<uint32_t>(w2 >> 32),
                             static_cast<uint32_t>(w3), static_cast<uint32_t>(w3 >> 32)));
    } else {
      uint32_t dw[6];
#pragma unroll
      for (uint32_t k = 0; k < 3; ++k) {
        dw[2 * k] = spread16(b[u][k]) | (spread16(h[u][k]) << 1);
        dw[2 * k + 1] = spread16(b[u][k] >> 16) | (spread16(h[u][k] >> 16) << 1);
      }
      store_block(out, make_uint4(e[0], e[1] & 0xFFFFu, dw[0], dw[1]),
                  make_uint4(dw[2], dw[3], dw[4], dw[5]));
    }
    if (ds) {
      // entry k of a digit names the block holding its (k R + 1)-th
      // occurrence: the entries below the block's end, less those below its
      // start, are the block's own
      uint32_t more = 0;
#pragma unroll
      for (uint32_t k = 0; k < kP; ++k) {
        uint32_t const z = e[k] + rem[k], hit = (z ^ (z + c[u][k])) & ~rm2;
        if (hit & 0xFFFFu) entry[2 * k][(z & 0xFFFFu) >> sh] = static_cast<uint32_t>(blk + u);
        if (hit >> 16) entry[2 * k + 1][z >> 16 >> sh] = static_cast<uint32_t>(blk + u);
        more |= c[u][k] + 0x7FFF7FFFu - rm2 - 0x10001u;
      }
      if (rm + 1 < kD && (more & 0x80008000u))  // a digit more than R times
#pragma unroll
        for (uint32_t d = 0; d < S; ++d) {
          uint32_t const z = ((e[d >> 1] + rem[d >> 1]) >> (16 * (d & 1))) & 0xFFFFu;
          uint32_t const end = z + ((c[u][d >> 1] >> (16 * (d & 1))) & 0xFFFFu);
          for (uint32_t k = (z >> sh) + 1; k < end >> sh; ++k)
            entry[d][k] = static_cast<uint32_t>(blk + u);
        }
    }
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
  uint64_t const codes = C.size() - 1;  // 2^L
  std::vector<uint64_t> h(C);
  h.resize(C.size() + ceil_div(codes + t.sigma, 4), 0);
  uint16_t* const symbol = reinterpret_cast<uint16_t*>(h.data() + C.size());
  for (uint64_t i = 0; i < t.sigma; ++i) {
    uint64_t const c = padded_code(t, i);
    symbol[c] = static_cast<uint16_t>(i);
    symbol[codes + i] = static_cast<uint16_t>(c);
  }
  GroupStore& qs = t.groups;
  qs.counts.alloc(h.size() * 8);
  EWT_CUDA(cudaMemcpyAsync(qs.counts.get(), h.data(), h.size() * 8, cudaMemcpyHostToDevice, st));
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
  constexpr uint32_t S = 1u << W;
  uint32_t const chunks = static_cast<uint32_t>(ceil_div(nsb + 1, kScanChunk));
  EWT_CUDA(cudaMemsetAsync(chunk.get(), 0, uint64_t(chunks) * S * 8, st));
  group_counts_kernel<W><<<static_cast<uint32_t>(ceil_div(nsb + 1, 8)), 256, 0, st>>>(
      g, n, nsb, sb, chunk.as<unsigned long long>());
  EWT_LAUNCHED();
  group_scan_kernel<S><<<chunks, kScanChunk, 0, st>>>(sb, nsb + 1, chunk.as<uint64_t>());
  EWT_LAUNCHED();
  group_level_kernel<W><<<static_cast<uint32_t>(nsb), 256, 0, st>>>(
      g, n, ql, qs.blocks.as<uint4>() + ql.blk_off * 2, sb, nsb,
      qs.ds.as<uint32_t>(), err);
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
  nr.reserve(uint64_t(2) << std::min<uint32_t>(L, 16));
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
