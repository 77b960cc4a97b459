// Wavelet-tree construction on the GPU.
//
// Pipeline (one GPU, one stream, no host round trip between levels):
//   1. alphabet: given, or detected (presence bitmap kernel for 1/2-byte
//      symbols, a set of the distinct ones on the device, sorted there up to
//      65,536 of them, for wider ones) — wavelet_tree.cuh:590-614;
//   2. shape on the host: minimal codes for non-power-of-two alphabets
//      (:2100-2159), node starts (:2501-2532), nodes per level (:703-724);
//   3. alphabets of up to 2^16 symbols: all levels by bit-plane passes
//      (planes.cuh) over the symbols' codes.  Bytes and 16-bit symbols are
//      mapped to codes as the passes read them, wider ones by remap_kernel
//      (:170-227).  A short code of a non-power-of-two alphabet is padded
//      with zero bits: codes are increasing, so the symbols whose code has
//      ended are the end of every later order, their padding writes zeros
//      there, and level l is the first part of that order (its size follows
//      from the passes' symbol counts, :776-790).  Then the RankSelect counts
//      of all levels and the node-start ranks (precomputeRanksKernel,
//      :332-352) in one launch each;
//   4. larger alphabets: level 0 bits are packed from the text; then for
//      every level l: RankSelect counts of level l; the node kernel computes
//      rank0 at every node start of level l and from it the count table C at
//      each node's split point (zeros of a node = rank0(end) - rank0(start));
//      the split kernel stably partitions every node of level l by its bit
//      (the level l+1 order; the reference re-sorts the text on the top l+1
//      code bits, :806-818) and writes the bits of level l+1 directly;
//   5. select samples of all levels.
// The split kernel has a fast path for tiles that lie inside one node of a
// power-of-two alphabet: warp ballots rank the tile's zeros and ones, both
// go to two contiguous runs, and the next level's bits of each run are
// compacted with warp OR-reductions into shared memory and stored as whole
// words (only a run's two edge words use atomicOr).  Other tiles take a
// general path that stages (destination, symbol) pairs in shared memory.
// No kernel waits on another CTA.
#include <algorithm>
#include <cstring>
#include <string>

#include "internal.cuh"

namespace ewt {

using ecl::detail::prev_pow2_u64;

namespace {

inline bool h_is_pow2(uint64_t n) { return (n & (n - 1)) == 0; }
inline uint64_t h_prev_pow2(uint64_t n) {
  if (n == 0) return 0;
  if (h_is_pow2(n)) return n >> 1;
  return uint64_t(1) << (63 - __builtin_clzll(n));
}
inline uint32_t h_ceil_log2(uint64_t n) {
  uint32_t const hi = 63 - __builtin_clzll(n);
  return h_is_pow2(n) ? hi : hi + 1;
}

// Shortened codes of the last symbols when sigma is not a power of two;
// same construction as createMinimalCodes (wavelet_tree.cuh:2100-2159).
std::vector<CodeH> make_codes(uint64_t sigma) {
  if (h_is_pow2(sigma)) return {};
  uint32_t const bits = h_ceil_log2(sigma);
  std::vector<CodeH> c(sigma);
  for (uint64_t i = 0; i < sigma; ++i) c[i] = {bits, i};
  uint32_t start_bit = 0, code_len = bits;
  uint64_t start_i = 0, left = sigma, kept = 0;
  do {
    for (uint32_t i = code_len - 1; i > 0; --i) {
      uint64_t const p = uint64_t(1) << i;
      if (left <= p) break;
      left -= p;
      start_i += p;
      ++start_bit;
    }
    if (code_len == bits) kept = left;
    if (left == 1) {
      code_len = 1;
      c[sigma - 1] = {start_bit, ((uint64_t(1) << start_bit) - 1)
                                     << (bits - start_bit)};
    } else {
      code_len = h_ceil_log2(left);
      uint64_t const high_mask = ~((uint64_t(1) << (bits - start_bit)) - 1);
      for (uint64_t i = sigma - left; i < sigma; ++i) {
        uint64_t code = (i - start_i) << (bits - start_bit - code_len);
        code += high_mask & c[i].code;
        c[i] = {start_bit + code_len, code};
      }
    }
  } while (code_len > 1);
  return std::vector<CodeH>(c.end() - kept, c.end());
}

// Every node with at least two symbols, level by level, in symbol order:
// [start, end) splits at start + prevPow2(end - start), the descent of
// deviceAccess (wavelet_tree.cuh:1854-1868).
struct LevelNode {
  uint64_t cs, split, end;
};

std::vector<std::vector<LevelNode>> make_level_nodes(uint64_t sigma,
                                                     uint32_t L) {
  std::vector<std::vector<LevelNode>> lv(L);
  std::vector<std::pair<uint64_t, uint64_t>> cur{{0, sigma}}, nxt;
  for (uint32_t l = 0; l < L; ++l) {
    nxt.clear();
    for (auto [a, e] : cur) {
      if (e - a < 2) continue;
      uint64_t const s = a + h_prev_pow2(e - a);
      lv[l].push_back({a, s, e});
      nxt.push_back({a, s});
      nxt.push_back({s, e});
    }
    cur.swap(nxt);
  }
  return lv;
}

// Node starts per level (getNodeInfos, wavelet_tree.cuh:2501-2532): every node
// of at least two symbols but each level's first.  (A symbol begins a node of
// level l where its code's bit l is 0 and its neighbour's 1; the neighbour is
// then the last symbol of a node of at least two, since a node's left child is
// the deeper one, so codes end on a level from the right.)
std::vector<NodeInfoH> make_nodes(uint64_t sigma, uint32_t L) {
  std::vector<NodeInfoH> out;
  out.reserve(sigma);
  if (h_is_pow2(sigma)) {
    for (uint32_t l = 1; l < L; ++l)
      for (uint64_t g = 1; g < uint64_t(1) << l; ++g) out.push_back({g << (L - l), l});
    return out;
  }
  auto const lv = make_level_nodes(sigma, L);
  for (uint32_t l = 1; l < L; ++l)
    for (LevelNode const& nd : lv[l])
      if (nd.cs) out.push_back({nd.cs, l});
  return out;
}

// --------------------------------------------------------------------------
// Alphabet detection for 1- and 2-byte symbols: presence bitmap.
template <class T>
__global__ void presence_kernel(T const* __restrict__ text, uint64_t n,
                                uint32_t* __restrict__ bitmap) {
  constexpr uint32_t kWords = (sizeof(T) == 1 ? 256u : 65536u) / 32u;
  __shared__ uint32_t sm[kWords];
  for (uint32_t i = threadIdx.x; i < kWords; i += blockDim.x) sm[i] = 0;
  __syncthreads();
  uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    uint32_t const c = text[i];
    uint32_t const bit = 1u << (c & 31);
    if (!(sm[c >> 5] & bit)) atomicOr(&sm[c >> 5], bit);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kWords; i += blockDim.x)
    if (sm[i]) atomicOr(&bitmap[i], sm[i]);
}

// Alphabet detection for 4- and 8-byte symbols: a device hash set of the
// distinct symbols (open addressing, linear probing, 64-bit slots).  An
// empty slot holds kEmptySlot; for 8-byte texts the one symbol equal to it is
// recorded in a flag instead.  Each CTA remembers the symbols it has looked up
// in a direct-mapped table in shared memory, so a symbol that repeats goes no
// further (20 M symbols of 10,000: 300 us without).  Others are looked up with
// a plain load first and inserted with atomicCAS only when missing.  A table
// that is more than half full is too small: the host retries with a larger one,
// and every thread ends early, asking for that where it inserts and every
// kAskProbes probes (chains of a table that is large enough are shorter;
// without, each of the text's symbols ran around the full table: 20 M symbols
// of a million 21.4 s, 104 ms so).
constexpr uint64_t kEmptySlot = ~uint64_t(0);
constexpr uint32_t kSeenSlots = 8192;
constexpr uint64_t kAskProbes = 16;

__device__ __forceinline__ uint64_t slot_hash(uint64_t x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  return x;
}

template <class T>
__global__ void __launch_bounds__(1024)
distinct_kernel(T const* __restrict__ text, uint64_t n,
                unsigned long long* __restrict__ table, uint64_t cap_mask,
                unsigned long long* __restrict__ count,
                uint32_t* flags) {  // [0] overflow, [1] max symbol seen
  extern __shared__ __align__(8) uint64_t seen[];
  for (uint32_t i = threadIdx.x; i < kSeenSlots; i += blockDim.x) seen[i] = kEmptySlot;
  __syncthreads();
  uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    uint64_t const key = static_cast<uint64_t>(text[i]);
    if (key == kEmptySlot) {
      flags[1] = 1;
      continue;
    }
    uint64_t const hash = slot_hash(key);
    // (a slot is read and written whole, so racing threads see one key or another)
    uint64_t volatile* const mine = seen + (hash & (kSeenSlots - 1));
    if (*mine == key) continue;
    uint64_t h = hash & cap_mask;
    for (uint64_t probe = 1;; ++probe) {
      if (probe % kAskProbes == 0) {
        if (probe > cap_mask) flags[0] = 1;
        if (*static_cast<uint32_t volatile*>(flags)) return;
      }
      uint64_t const cur = *const_cast<unsigned long long volatile*>(table + h);
      if (cur == key) break;
      if (cur == kEmptySlot) {
        unsigned long long const prev =
            atomicCAS(&table[h], static_cast<unsigned long long>(kEmptySlot),
                      static_cast<unsigned long long>(key));
        if (prev == kEmptySlot) {
          if ((atomicAdd(count, 1ull) + 1) * 2 > cap_mask + 1) flags[0] = 1;
          if (*static_cast<uint32_t volatile*>(flags)) return;
          break;
        }
        if (prev == key) break;
      }
      h = (h + 1) & cap_mask;
    }
    *mine = key;
  }
}

// The table's symbols side by side (order as it comes).
__global__ void __launch_bounds__(256)
compact_kernel(unsigned long long const* __restrict__ table, uint64_t cap,
               uint64_t* __restrict__ out, uint64_t count, uint32_t* __restrict__ next) {
  uint64_t const i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= cap || table[i] == kEmptySlot) return;
  uint32_t const at = atomicAdd(next, 1u);
  if (at < count) out[at] = table[i];
}

// Sorted by counting: symbol i goes to the number of smaller ones (all are
// distinct).  count^2 comparisons, but on every SM and without a pass over
// memory: 10,000 symbols 12 us, 65,536 about 130 us; the host's sort of 10,000
// took 0.5 ms.
constexpr uint64_t kRankSortMax = 65536;

__global__ void __launch_bounds__(256)
rank_sort_kernel(uint64_t const* __restrict__ in, uint32_t count, uint64_t* __restrict__ out) {
  __shared__ uint64_t tile[1024];
  uint32_t const i = blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t const x = i < count ? in[i] : 0;
  uint32_t rank = 0;
  for (uint32_t base = 0; base < count; base += 1024) {
    uint32_t const len = min(1024u, count - base);
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) tile[j] = in[base + j];
    __syncthreads();
#pragma unroll 8
    for (uint32_t j = 0; j < len; ++j) rank += tile[j] < x;
  }
  if (i < count) out[rank] = x;
}

// Sorted distinct symbols of a device-resident 4- or 8-byte text.
template <class T>
std::vector<uint64_t> detect_alphabet_wide(T const* d_text, uint64_t n,
                                           cudaStream_t st) {
  uint64_t cap = 1ull << 16;
  uint32_t const blocks = static_cast<uint32_t>(
      std::min<uint64_t>(ceil_div(n, 1024), uint64_t(sm_count()) * 2));
  set_smem_limit(distinct_kernel<T>, kSeenSlots * 8);
  for (;;) {
    DevBuf table(cap * 8), cnt(8), flags(8);
    EWT_CUDA(cudaMemsetAsync(table.get(), 0xFF, cap * 8, st));
    EWT_CUDA(cudaMemsetAsync(cnt.get(), 0, 8, st));
    EWT_CUDA(cudaMemsetAsync(flags.get(), 0, 8, st));
    distinct_kernel<T><<<blocks, 1024, kSeenSlots * 8, st>>>(
        d_text, n, table.as<unsigned long long>(), cap - 1,
        cnt.as<unsigned long long>(), flags.as<uint32_t>());
    EWT_LAUNCHED();
    uint64_t count = 0;
    uint32_t fl[2] = {0, 0};
    EWT_CUDA(cudaMemcpyAsync(&count, cnt.get(), 8, cudaMemcpyDeviceToHost, st));
    EWT_CUDA(cudaMemcpyAsync(fl, flags.get(), 8, cudaMemcpyDeviceToHost, st));
    EWT_CUDA(cudaStreamSynchronize(st));
    if (!fl[0] && count * 2 <= cap && count <= kRankSortMax) {
      DevBuf list(std::max<uint64_t>(count, 1) * 16), next(4);
      EWT_CUDA(cudaMemsetAsync(next.get(), 0, 4, st));
      uint64_t* const sorted = list.as<uint64_t>() + count;
      compact_kernel<<<static_cast<uint32_t>(ceil_div(cap, 256)), 256, 0, st>>>(
          table.as<unsigned long long>(), cap, list.as<uint64_t>(), count, next.as<uint32_t>());
      EWT_LAUNCHED();
      if (count) {
        rank_sort_kernel<<<static_cast<uint32_t>(ceil_div(count, 256)), 256, 0, st>>>(
            list.as<uint64_t>(), static_cast<uint32_t>(count), sorted);
        EWT_LAUNCHED();
      }
      std::vector<uint64_t> out(count);
      EWT_CUDA(cudaMemcpyAsync(out.data(), sorted, count * 8, cudaMemcpyDeviceToHost, st));
      EWT_CUDA(cudaStreamSynchronize(st));
      if (fl[1]) out.push_back(kEmptySlot);
      return out;
    }
    if (!fl[0] && count * 2 <= cap) {
      std::vector<uint64_t> h(cap);
      EWT_CUDA(cudaMemcpyAsync(h.data(), table.get(), cap * 8,
                               cudaMemcpyDeviceToHost, st));
      EWT_CUDA(cudaStreamSynchronize(st));
      std::vector<uint64_t> out;
      out.reserve(count + 1);
      for (uint64_t v : h)
        if (v != kEmptySlot) out.push_back(v);
      if (fl[1]) out.push_back(kEmptySlot);
      std::sort(out.begin(), out.end());
      return out;
    }
    // table too small: at least four times the symbols seen so far
    uint64_t want = std::max(cap * 2, count * 4);
    cap = 1;
    while (cap < want) cap <<= 1;
  }
}

// Text -> minimal symbols (lower_bound in the sorted alphabet), or with
// `codes` the code of each.  Smem: the alphabet is searched in shared memory.
// A symbol's place in the alphabet's range (kRemapBuckets equal parts) gives
// the two entries to search between: 10,000 symbols spread evenly take two
// steps instead of fourteen (20 M symbols 120 us without).
constexpr uint32_t kRemapBuckets = 4096;

template <class T, class U, bool Smem>
__global__ void __launch_bounds__(1024)
remap_kernel(T const* __restrict__ text, uint64_t n,
             T const* __restrict__ alphabet, uint32_t sigma,
             uint16_t const* __restrict__ codes, U* __restrict__ cur,
             uint32_t* __restrict__ err) {
  extern __shared__ __align__(16) unsigned char remap_smem[];
  __shared__ uint32_t first[kRemapBuckets + 1];  // lower_bound of each bucket's start
  T* const sa = reinterpret_cast<T*>(remap_smem);
  if constexpr (Smem) {
    for (uint32_t i = threadIdx.x; i < sigma; i += blockDim.x) sa[i] = alphabet[i];
    __syncthreads();
  }
  T const* const al = Smem ? sa : alphabet;
  auto search = [&](T x, uint32_t lo, uint32_t hi) {
    while (lo < hi) {
      uint32_t const mid = (lo + hi) >> 1;
      if (al[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
  };
  T const low = al[0], top = al[sigma - 1];
  uint32_t shift = 0;  // bucket of x: (x - low) >> shift < kRemapBuckets
  while ((uint64_t(top) - uint64_t(low)) >> shift >= kRemapBuckets) ++shift;
  for (uint32_t b = threadIdx.x; b <= kRemapBuckets; b += blockDim.x) {
    uint64_t const d = uint64_t(b) << shift;  // past the range: all of the alphabet
    first[b] = (d >> shift) != b || d > uint64_t(top) - uint64_t(low)
                   ? sigma
                   : search(static_cast<T>(uint64_t(low) + d), 0, sigma);
  }
  __syncthreads();
  uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
  uint32_t bad = 0;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    T const x = text[i];
    uint32_t lo = 0;
    if (x > top) {
      bad = 1;
    } else if (x > low) {
      uint32_t const b = static_cast<uint32_t>((uint64_t(x) - uint64_t(low)) >> shift);
      lo = search(x, first[b], first[b + 1]);
    }
    cur[i] = static_cast<U>(codes ? codes[lo] : lo);
  }
  if (bad) atomicOr(err, 1u);
}

// Searching in shared memory keeps two CTAs of 1024 threads on an SM up to
// 80 KB of alphabet; above that the alphabet stays in the caches.
template <class T, class U>
void launch_remap(T const* text, uint64_t n, T const* alphabet, uint64_t sigma,
                  uint16_t const* codes, U* out, uint32_t* err, cudaStream_t st) {
  EWT_REQUIRE(sigma < UINT32_MAX, EWT_ERR_UNSUPPORTED, "alphabet too large");
  uint32_t const grid = static_cast<uint32_t>(
      std::min<uint64_t>(ceil_div(n, 1024), uint64_t(sm_count()) * 2));
  constexpr size_t kMax = 80 * 1024;
  if (sigma * sizeof(T) <= kMax) {
    auto k = remap_kernel<T, U, true>;
    set_smem_limit(k, kMax);
    k<<<grid, 1024, sigma * sizeof(T), st>>>(text, n, alphabet, static_cast<uint32_t>(sigma),
                                             codes, out, err);
  } else {
    remap_kernel<T, U, false><<<grid, 1024, 0, st>>>(
        text, n, alphabet, static_cast<uint32_t>(sigma), codes, out, err);
  }
  EWT_LAUNCHED();
}

// Histogram of minimal symbols (non-power-of-two alphabets of more than
// 2^16 symbols).
template <class T>
__global__ void __launch_bounds__(256)
hist_kernel(T const* __restrict__ text, uint64_t n, uint64_t sigma,
            unsigned long long* __restrict__ occ) {
  uint64_t const stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    uint64_t const c = text[i];
    if (c < sigma) atomicAdd(&occ[c], 1ull);
  }
}

// --------------------------------------------------------------------------
// Node of minimal symbol c on level l: [cs, ce] and its split point.
struct NodeRange {
  uint64_t cs, ce, split;
};

template <bool Pow2>
__device__ __forceinline__ NodeRange node_of(uint64_t c, uint32_t l,
                                             uint32_t L, uint64_t sigma) {
  NodeRange r;
  if (Pow2) {
    uint32_t const w = L - l;  // node width is 2^w symbols
    uint64_t const mask = (w >= 64) ? ~uint64_t(0) : ((uint64_t(1) << w) - 1);
    r.cs = c & ~mask;
    r.ce = r.cs + mask;
    r.split = r.cs + (uint64_t(1) << (w - 1));
  } else {
    uint64_t cs = 0, ce = sigma - 1;
    for (uint32_t k = 0; k < l; ++k) {
      uint64_t const s = cs + prev_pow2_u64(ce - cs + 1);
      if (c < s) ce = s - 1; else cs = s;
    }
    r.cs = cs;
    r.ce = ce;
    r.split = cs + prev_pow2_u64(ce - cs + 1);
  }
  return r;
}

template <bool Pow2>
__device__ __forceinline__ bool level_bit(uint64_t c, uint32_t l, uint32_t L,
                                          uint64_t sigma) {
  if (Pow2) return (c >> (L - 1 - l)) & 1;
  return c >= node_of<false>(c, l, L, sigma).split;
}

// Level 0 bits of an alphabet of more than 2^16 symbols: a thread per output
// word.  Check = validate symbols of a minimal alphabet (c < sigma).
template <class T, bool Pow2, bool Check>
__global__ void __launch_bounds__(256)
fill0_kernel(T const* __restrict__ src, uint64_t size0, uint32_t L,
             uint64_t sigma, uint32_t* __restrict__ out,
             uint32_t* __restrict__ err) {
  uint64_t const w = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, p0 = w * 32;
  if (p0 >= size0) return;
  bool bad = false;
  uint32_t word = 0;
  if (p0 + 32 <= size0) {  // all loads before their first use
    constexpr int kVec = 32 * sizeof(T) / 16;
    uint4 buf[kVec];
#pragma unroll
    for (int q = 0; q < kVec; ++q) buf[q] = __ldg(reinterpret_cast<uint4 const*>(src + p0) + q);
    T const* e = reinterpret_cast<T const*>(buf);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      uint64_t const c = e[i];
      if (Check) bad |= c >= sigma;
      word |= uint32_t(level_bit<Pow2>(c, 0, L, sigma)) << i;
    }
  } else {
    for (uint32_t i = 0; p0 + i < size0; ++i) {
      uint64_t const c = src[p0 + i];
      if (Check) bad |= c >= sigma;
      word |= uint32_t(level_bit<Pow2>(c, 0, L, sigma)) << i;
    }
  }
  out[w] = word;
  if (Check && bad) atomicOr(err, 1u);
}

// For every node of level l with >= 2 symbols: rank0 at its start (stored
// as the node-start rank of the reference) and the count table at its
// split point, C[split] = C[start] + rank0(C[end]) - rank0(C[start]).
__global__ void __launch_bounds__(128)
level_nodes_kernel(TreeView t, LevelNode const* __restrict__ nodes,
                   uint64_t count, uint32_t l, uint64_t* __restrict__ counts,
                   uint64_t* __restrict__ ranks, uint32_t* __restrict__ err) {
  uint64_t const i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  LevelNode const nd = nodes[i];
  ArrayMeta const m = t.rs.meta[l];
  uint64_t const ps = counts[nd.cs];
  uint64_t const pe = counts[nd.end];
  uint64_t const r_start =
      nd.cs ? ps - ecl::detail::rs_rank1<false>(t.rs, m, ps, nullptr) : 0;
  uint64_t const r_end = pe - ecl::detail::rs_rank1<false>(t.rs, m, pe, nullptr);
  counts[nd.split] = ps + (r_end - r_start);
  if (nd.cs) {
    uint64_t const ni = ecl::detail::node_index(t, t.node_base, nd.cs, l);
    if (ni < t.num_ranks) ranks[ni] = r_start;
    else atomicOr(err, 2u);
  }
}

}  // namespace
}  // namespace ewt

#include "planes.cuh"
#include "split.cuh"

namespace ewt {
namespace {

// rank0 at every node start (node i: first symbol and level, in the order the
// ranks are stored in; null: a power-of-two tree's); the count table is
// complete.
__global__ void __launch_bounds__(128)
node_ranks_kernel(TreeView t, NodeInfoH const* __restrict__ nodes, uint64_t count,
                  uint64_t* __restrict__ ranks) {
  uint64_t const i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  NodeInfoH nd;
  if (nodes) {
    nd = nodes[i];
  } else {  // power of two: level l's nodes 1 .. 2^l - 1 follow 2^l - 1 - l others
    uint32_t l = 1;
    while (i >= (uint64_t(2) << l) - 2 - l) ++l;
    nd.level = l;
    nd.start = (i - ((uint64_t(1) << l) - 1 - l) + 1) << (t.levels - l);
  }
  uint64_t const p = t.counts[nd.start];
  ranks[i] = p - ecl::detail::rs_rank1<false>(t.rs, t.rs.meta[nd.level], p, nullptr);
}

// Planes l+1 .. l+count of a level order held as symbols (bits L-2-l ..),
// 32 positions per warp and step.
template <class T>
__global__ void __launch_bounds__(256)
order_planes_kernel(T const* __restrict__ x, uint64_t n, uint32_t L, uint32_t l,
                    uint32_t count, uint32_t* __restrict__ out, uint64_t stride) {
  uint32_t const lane = threadIdx.x & 31;
  uint64_t const words = (n + 31) / 32, step = uint64_t(gridDim.x) * (blockDim.x / 32);
  for (uint64_t w = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) / 32; w < words;
       w += step) {
    uint64_t const at = w * 32 + lane;
    uint64_t const c = at < n ? uint64_t(x[at]) : 0;
    for (uint32_t j = 0; j < count; ++j) {
      uint32_t const v = __ballot_sync(0xffffffffu, (c >> (L - 2 - l - j)) & 1);
      if (lane == 0) out[j * stride + w] = v;
    }
  }
}

// Wide symbols whose codes would take more than kSplitOrderBytes get them in
// parts of so many, each read before the next is made.
constexpr uint64_t kCodePart = uint64_t(1) << 31;

// Words of one level in the passes' store.
uint64_t level_stride(uint64_t n) { return ceil_div(ceil_div(n, 32), 32) * 32; }

// Levels 0 .. L-1 of codes of up to 16 bits by bit-plane passes (planes.cuh),
// level l at words + l * level_stride(n); returns the deeper planes that the
// group levels read.
template <class U>
std::vector<OrderPlanes> run_passes(ewt_tree& t, PlaneText<U> const& x, uint32_t* words,
                                    uint64_t* starts, bool groups, uint32_t* err,
                                    cudaStream_t st) {
  uint64_t const stride = level_stride(x.n);
  std::vector<uint32_t*> out(x.L);
  std::vector<uint64_t> count(x.L, stride);
  for (uint32_t l = 0; l < x.L; ++l) out[l] = words + l * stride;
  // level 0 is written whole but for its padding
  uint64_t const w0 = ceil_div(x.n, 32);
  if (stride > w0) EWT_CUDA(cudaMemsetAsync(words + w0, 0, (stride - w0) * 4, st));
  return run_plane_passes<U>(x, out.data(), count.data(), starts,
                             groups ? group_planes(x.L)
                                    : std::vector<std::pair<uint32_t, uint32_t>>{},
                             err, st);
}

thread_local bool t_texts_synced = false;
thread_local bool t_batch_member = false;
thread_local bool t_within_footprint = false;

// Whether a host text goes straight to the ingest kernel, which is then its
// only reader (kernels read the host text: a Grace host's pageable memory, or
// pinned memory): 1- and 2-byte symbols, a given alphabet (one to be found is
// another read), a 16-byte aligned text.
template <class T>
bool host_ingest(const void* data, uint64_t n, uint64_t sigma) {
  if constexpr (sizeof(T) > 2) {
    return false;
  } else {
    if (sigma < 2 || n == 0 || reinterpret_cast<uintptr_t>(data) % 16) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    int pageable = 0;
    cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, dev);
    cudaPointerAttributes pa{};
    bool const pinned = cudaPointerGetAttributes(&pa, data) == cudaSuccess &&
                        pa.type == cudaMemoryTypeHost;
    (void)cudaGetLastError();
    return pageable || pinned;
  }
}

template <class T>
void build_typed(ewt_tree& t, const void* data, uint64_t n,
                 const void* alphabet, uint64_t sigma, cudaStream_t st) {
  // Host tables that copies to the device read: they outlive the copies (also
  // when the build throws: the guard below them waits first).
  std::vector<T> alphabet_h;
  std::vector<uint16_t> codes, lut;  // padded codes by minimal symbol, by symbol
  std::vector<uint64_t> tables, c_h;
  std::vector<LevelNode> flat;
  DrainOnError drain(st);
  // ---- text on the device
  DevBuf text_owned;
  T const* d_text;
  bool host_text = false;  // the ingest kernel reads the text in host memory
  bool const on_device = is_device_pointer(data);
  // The text may still be in flight on the caller's streams; the build runs
  // on its own stream, so order it after all prior device work (once per
  // batch when a batch of builds already did).
  if (on_device && !texts_synchronized()) EWT_CUDA(cudaDeviceSynchronize());
  if (on_device && reinterpret_cast<uintptr_t>(data) % 16 == 0) {
    d_text = static_cast<T const*>(data);
  } else if (on_device) {
    // The kernels read the text with 16-byte vector loads.
    text_owned.alloc(n * sizeof(T));
    EWT_CUDA(cudaMemcpyAsync(text_owned.get(), data, n * sizeof(T),
                             cudaMemcpyDeviceToDevice, st));
    d_text = text_owned.as<T>();
  } else if (host_ingest<T>(data, n, sigma)) {
    d_text = static_cast<T const*>(data);
    host_text = true;
  } else {
    text_owned.alloc(n * sizeof(T));
    PhaseTimer pt(EWT_PHASE_H2D, st);
    EWT_CUDA(cudaMemcpyAsync(text_owned.get(), data, n * sizeof(T),
                             cudaMemcpyHostToDevice, st));
    d_text = text_owned.as<T>();
  }
  // ---- alphabet
  t.alphabet.clear();
  if (sigma == 0) {
    if (sizeof(T) <= 2) {
      constexpr uint32_t kWords = (sizeof(T) == 1 ? 256u : 65536u) / 32u;
      DevBuf bm(kWords * 4);
      EWT_CUDA(cudaMemsetAsync(bm.get(), 0, kWords * 4, st));
      uint32_t const blocks =
          static_cast<uint32_t>(std::min<uint64_t>(ceil_div(n, 256),
                                                   uint64_t(sm_count()) * 8));
      presence_kernel<T><<<blocks, 256, 0, st>>>(d_text, n, bm.as<uint32_t>());
      EWT_LAUNCHED();
      std::vector<uint32_t> h(kWords);
      EWT_CUDA(cudaMemcpyAsync(h.data(), bm.get(), kWords * 4,
                               cudaMemcpyDeviceToHost, st));
      EWT_CUDA(cudaStreamSynchronize(st));
      for (uint64_t v = 0; v < kWords * 32ull; ++v)
        if ((h[v >> 5] >> (v & 31)) & 1) t.alphabet.push_back(v);
    } else {
      t.alphabet = detect_alphabet_wide<T>(d_text, n, st);
    }
  } else {
    T const* a = static_cast<T const*>(alphabet);
    EWT_REQUIRE(a != nullptr, EWT_ERR_INVALID_ARGUMENT, "alphabet is null");
    t.alphabet.assign(a, a + sigma);
    for (uint64_t i = 1; i < sigma; ++i)
      EWT_REQUIRE(t.alphabet[i] > t.alphabet[i - 1], EWT_ERR_ALPHABET,
                  "alphabet must be sorted and free of duplicates");
  }
  t.sigma = t.alphabet.size();
  EWT_REQUIRE(t.sigma >= 2, EWT_ERR_ALPHABET,
              "alphabet must hold at least two symbols");
  sigma = t.sigma;
  t.L = h_ceil_log2(sigma);
  t.pow2 = h_is_pow2(sigma);
  t.is_min = true;
  for (uint64_t i = 0; i < sigma; ++i)
    if (t.alphabet[i] != i) { t.is_min = false; break; }
  // ---- shape
  set_tree_shape(t);
  uint32_t const L = t.L;

  // ---- device tables
  t.err_d.alloc(kTreeErrBytes);
  EWT_CUDA(cudaMemsetAsync(t.err_d.get(), 0, kTreeErrBytes, st));
  uint32_t* err_build = t.err_d.as<uint32_t>() + 1;
  uint32_t const grid_stream =
      static_cast<uint32_t>(std::min<uint64_t>(ceil_div(n, 256),
                                               uint64_t(sm_count()) * 8));
  bool const by_planes = sizeof(T) <= 2 || L <= kMaxPlanes;
  auto const level_nodes = by_planes ? std::vector<std::vector<LevelNode>>{}
                                     : make_level_nodes(sigma, L);
  DevBuf cur_buf;  // minimal symbols (or codes) of a text the build cannot read as it is
  DevBuf lut_d;
  T const* sym = d_text;
  // A copy that was read for the last time makes room for what is built next
  // where memory is short: a large one (as the planes of large orders do,
  // planes.cuh), and any in a build that was admitted by its footprint.  Elsewhere
  // it stays until the end: the pool hands its pieces out in other pieces, and
  // 150 M bytes of 96 symbols take 2.92 instead of 2.58 ms.
  auto release = [](DevBuf& b) {
    if (t_within_footprint || b.bytes() > kSplitOrderBytes) b.reset();
  };
  if (!t.is_min || (by_planes && sizeof(T) > 2)) {
    alphabet_h.assign(t.alphabet.begin(), t.alphabet.end());
    t.alphabet_d.alloc(sigma * sizeof(T));
    EWT_CUDA(cudaMemcpyAsync(t.alphabet_d.get(), alphabet_h.data(), sigma * sizeof(T),
                             cudaMemcpyHostToDevice, st));
  }
  if (by_planes && (!t.pow2 || !t.is_min)) {
    codes.resize(sigma);
    for (uint64_t i = 0; i < sigma; ++i)
      codes[i] = static_cast<uint16_t>(padded_code(t, i));
    if (sizeof(T) <= 2) {  // by symbol: that of the first alphabet symbol at or above it
      lut.assign(sizeof(T) == 1 ? 256 : 65536, 0);
      uint64_t v = 0;
      for (uint64_t i = 0; i < sigma; ++i)
        for (; v <= t.alphabet[i] && v < lut.size(); ++v) lut[v] = codes[i];
      lut_d.alloc(lut.size() * 2);
      EWT_CUDA(cudaMemcpyAsync(lut_d.get(), lut.data(), lut.size() * 2,
                               cudaMemcpyHostToDevice, st));
    } else if (!t.pow2) {
      lut_d.alloc(sigma * 2);
      EWT_CUDA(cudaMemcpyAsync(lut_d.get(), codes.data(), sigma * 2,
                               cudaMemcpyHostToDevice, st));
    }
  }
  bool in_parts = false;  // codes are made and read part by part
  if constexpr (sizeof(T) > 2) {
    if (by_planes) {
      in_parts = n * 2 > kSplitOrderBytes;
      cur_buf.alloc(in_parts ? kCodePart * 2 : n * 2);
      if (!in_parts) {
        PhaseTimer pt(EWT_PHASE_HIST, st);
        launch_remap<T, uint16_t>(d_text, n, t.alphabet_d.as<T>(), sigma, lut_d.as<uint16_t>(),
                                  cur_buf.as<uint16_t>(), err_build, st);
        release(text_owned);
      }
    } else if (!t.is_min) {
      cur_buf.alloc(n * sizeof(T));
      PhaseTimer pt(EWT_PHASE_HIST, st);
      launch_remap<T, T>(d_text, n, t.alphabet_d.as<T>(), sigma, nullptr, cur_buf.as<T>(),
                         err_build, st);
      sym = cur_buf.as<T>();
    }
  }
  // Group query levels -- except for the short texts of a batch build: the
  // group build's launch latency would be most of their build time; they get
  // rank blocks on every level instead.
  t.n = n;
  bool const want_groups =
      groups_eligible(t) && !(t_batch_member && n < kBatchGroupMinSymbols);
  std::vector<OrderPlanes> kept;  // deeper planes of the group levels' orders
  // The passes, given where level 0 and the class starts (2^L + 1) go.
  auto passes = [&](uint32_t* words, uint64_t* starts) {
    auto run = [&](auto x) {
      x.n = n;
      x.L = L;
      kept = run_passes(t, x, words, starts, want_groups, err_build, st);
      release(text_owned);
      release(cur_buf);
    };
    if constexpr (sizeof(T) <= 2) {
      PlaneText<T> x;
      x.sym = d_text;
      if (!codes.empty()) {
        x.lut = lut_d.as<uint16_t>();
        x.max_symbol = static_cast<uint32_t>(t.alphabet.back());
      }
      if (host_text) x.ingest_phase = EWT_PHASE_H2D;
      run(x);
    } else {
      PlaneText<uint16_t> x;
      if (in_parts) {
        x.part_symbols = kCodePart;
        x.part = [&](uint64_t begin, uint64_t len) {
          launch_remap<T, uint16_t>(d_text + begin, len, t.alphabet_d.as<T>(), sigma,
                                    lut_d.as<uint16_t>(), cur_buf.as<uint16_t>(), err_build, st);
          return cur_buf.as<uint16_t const>();
        };
      } else {
        x.sym = cur_buf.as<uint16_t>();
      }
      run(x);
    }
  };
  // Count table: for power-of-two alphabets the passes' class starts (or, of
  // the split, C[0] = 0 and C[sigma] = n, the rest derived level by level);
  // other alphabets need the symbol counts first, for their level sizes.
  t.counts_d.alloc((sigma + 1) * 8);
  t.level_bits.assign(L, n);
  DevBuf words_early;  // the levels of passes that ran before the layout
  std::vector<uint64_t> code_starts;  // symbols of a smaller code (no power of two)
  if (!t.pow2) {
    t.occ.assign(sigma, 0);
    if (by_planes) {
      uint64_t const slots = uint64_t(1) << L;
      DevBuf starts((slots + 1) * 8);
      words_early.alloc(L * level_stride(n) * 4 + 64);
      passes(words_early.as<uint32_t>(), starts.as<uint64_t>());
      std::vector<uint64_t>& h = code_starts;
      h.resize(slots + 1);
      EWT_CUDA(cudaMemcpyAsync(h.data(), starts.get(), (slots + 1) * 8,
                               cudaMemcpyDeviceToHost, st));
      EWT_CUDA(cudaStreamSynchronize(st));
      for (uint64_t i = 0; i < sigma; ++i) t.occ[i] = h[codes[i] + 1] - h[codes[i]];
    } else if constexpr (sizeof(T) > 2) {
      DevBuf occ_d(sigma * 8);
      EWT_CUDA(cudaMemsetAsync(occ_d.get(), 0, sigma * 8, st));
      {
        PhaseTimer pt(EWT_PHASE_HIST, st);
        hist_kernel<T><<<grid_stream, 256, 0, st>>>(
            sym, n, sigma, occ_d.as<unsigned long long>());
        EWT_LAUNCHED();
      }
      EWT_CUDA(cudaMemcpyAsync(t.occ.data(), occ_d.get(), sigma * 8,
                               cudaMemcpyDeviceToHost, st));
      EWT_CUDA(cudaStreamSynchronize(st));
    }
    // Level sizes (wavelet_tree.cuh:776-790): drop symbols whose code ended.
    for (size_t j = 0; j < t.codes.size(); ++j)
      for (uint32_t l = static_cast<uint32_t>(t.codes[j].len); l < L; ++l)
        t.level_bits[l] -= t.occ[t.codes_start + j];
    c_h.assign(sigma + 1, 0);
    for (uint64_t i = 1; i <= sigma; ++i) c_h[i] = c_h[i - 1] + t.occ[i - 1];
    EWT_CUDA(cudaMemcpyAsync(t.counts_d.get(), c_h.data(), (sigma + 1) * 8,
                             cudaMemcpyHostToDevice, st));
  } else if (!by_planes) {
    uint64_t const ends[2] = {0, n};
    EWT_CUDA(cudaMemcpyAsync(t.counts_d.get(), &ends[0], 8,
                             cudaMemcpyHostToDevice, st));
    EWT_CUDA(cudaMemcpyAsync(t.counts_d.as<uint64_t>() + sigma, &ends[1], 8,
                             cudaMemcpyHostToDevice, st));
    EWT_CUDA(cudaStreamSynchronize(st));  // `ends` leaves scope
  }
  for (uint32_t l = 0; l < L; ++l)
    EWT_REQUIRE(t.level_bits[l] > 0, EWT_ERR_UNSUPPORTED,
                "empty level: every symbol with a code this long is absent");

  // binary levels that group levels cover get no rank blocks
  t.rs.skip_blocks.assign(L, 0);
  if (want_groups) {
    uint32_t covered = 0;
    for (uint32_t w : group_widths(L)) covered += w;
    for (uint32_t l = 0; l < covered; ++l) t.rs.skip_blocks[l] = 1;
  }
  if (words_early.get()) {
    t.rs.layout(t.level_bits, level_stride(n), &words_early);
  } else {
    t.rs.layout(t.level_bits);
  }
  t.ranks_d.alloc(std::max<size_t>(t.nodes.size(), 1) * 8);
  // node bases, nodes per level, short codes: one block, one copy
  size_t const nc = std::max<size_t>(t.codes.size(), 1);
  tables.assign(t.node_base.begin(), t.node_base.end());
  tables.insert(tables.end(), t.nodes_at_level.begin(), t.nodes_at_level.end());
  size_t const at_len = tables.size(), at_code = at_len + nc;
  tables.resize(at_code + nc, 0);
  for (size_t i = 0; i < t.codes.size(); ++i) {
    tables[at_len + i] = t.codes[i].len;
    tables[at_code + i] = t.codes[i].code;
  }
  t.tables_d.alloc(tables.size() * 8);
  EWT_CUDA(cudaMemcpyAsync(t.tables_d.get(), tables.data(), tables.size() * 8,
                           cudaMemcpyHostToDevice, st));
  uint64_t* const tab = t.tables_d.as<uint64_t>();
  t.node_base_d.view(tab, (L + 1) * 8);
  t.nodes_at_level_d.view(tab + L + 1, L * 8);
  t.code_len_d.view(tab + at_len, nc * 8);
  t.code_bits_d.view(tab + at_code, nc * 8);
  std::vector<uint64_t> lv_off(L + 1, 0);
  for (uint32_t l = 0; l < L && !by_planes; ++l) {
    flat.insert(flat.end(), level_nodes[l].begin(), level_nodes[l].end());
    lv_off[l + 1] = flat.size();
  }
  DevBuf nodes_d;  // node starts (passes; of a power of two they follow from the index)
  if (by_planes && !t.pow2 && !t.nodes.empty()) {
    nodes_d.alloc(t.nodes.size() * sizeof(NodeInfoH));
    EWT_CUDA(cudaMemcpyAsync(nodes_d.get(), t.nodes.data(), t.nodes.size() * sizeof(NodeInfoH),
                             cudaMemcpyHostToDevice, st));
  }
  DevBuf lnodes_d;
  if (!flat.empty()) {
    lnodes_d.alloc(flat.size() * sizeof(LevelNode));
    EWT_CUDA(cudaMemcpyAsync(lnodes_d.get(), flat.data(), flat.size() * sizeof(LevelNode),
                             cudaMemcpyHostToDevice, st));
  }

  fill_tree_view(t);
  TreeView& v = t.view;

  uint32_t* const words = t.rs.words.as<uint32_t>();
  if (by_planes) {
    if (t.pow2) passes(words, t.counts_d.as<uint64_t>());
    if (t.is_min) t.alphabet_d.reset();  // only remap_kernel needed it
    build_rs_counts(t.rs, 0, L, st);
    if (!t.nodes.empty()) {
      PhaseTimer pt(EWT_PHASE_NODE_RANKS, st);
      node_ranks_kernel<<<static_cast<uint32_t>(ceil_div(t.nodes.size(), 128)), 128, 0, st>>>(
          v, nodes_d.as<NodeInfoH>(), t.nodes.size(), t.ranks_d.as<uint64_t>());
      EWT_LAUNCHED();
    }
  } else if constexpr (sizeof(T) > 2) {
    {  // level 0 bits
      PhaseTimer pt(EWT_PHASE_FILL, st);
      uint64_t const w0 = ceil_div(t.level_bits[0], 32);
      uint32_t const blocks =
          static_cast<uint32_t>(ceil_div(w0, 256));
      auto k = t.pow2 ? (t.is_min ? fill0_kernel<T, true, true>
                                  : fill0_kernel<T, true, false>)
                      : (t.is_min ? fill0_kernel<T, false, true>
                                  : fill0_kernel<T, false, false>);
      k<<<blocks, 256, 0, st>>>(sym, t.level_bits[0], L, sigma,
                                words + t.rs.meta[0].word_off, err_build);
      EWT_LAUNCHED();
    }
    std::vector<std::pair<uint32_t, uint32_t>> const wanted =
        want_groups ? group_planes(L) : std::vector<std::pair<uint32_t, uint32_t>>{};
    DevBuf ping, pong;
    if (L > 2) ping.alloc(n * sizeof(T));
    if (L > 3) pong.alloc(n * sizeof(T));
    T* bufs[2] = {ping.as<T>(), pong.as<T>()};
    // tiles the fast split leaves to the general one, and their count
    DevBuf slow_tiles((ceil_div(n, kSplitTile) + 1) * 4);
    T const* src = sym;
    for (uint32_t l = 0; l < L; ++l) {
      for (auto const& w : wanted)
        if (w.first == l) {  // a group level starts here
          OrderPlanes o;
          o.level = l;
          o.first = l + 1;
          o.count = o.front = w.second;
          o.stride = ceil_div(ceil_div(n, 32), 32) * 32 + 32;
          o.mem.alloc(o.count * o.stride * 4);
          EWT_CUDA(cudaMemsetAsync(o.mem.get(), 0, o.count * o.stride * 4, st));
          order_planes_kernel<T><<<grid_stream, 256, 0, st>>>(
              src, n, L, l, o.count, o.mem.as<uint32_t>(), o.stride);
          EWT_LAUNCHED();
          kept.push_back(std::move(o));
        }
      build_rs_counts(t.rs, l, l + 1, st);
      uint64_t const ncount = lv_off[l + 1] - lv_off[l];
      if (ncount > 0) {
        PhaseTimer pt(EWT_PHASE_NODE_RANKS, st);
        level_nodes_kernel<<<static_cast<uint32_t>(ceil_div(ncount, 128)), 128,
                             0, st>>>(v, lnodes_d.as<LevelNode>() + lv_off[l],
                                      ncount, l, t.counts_d.as<uint64_t>(),
                                      t.ranks_d.as<uint64_t>(), err_build);
        EWT_LAUNCHED();
      }
      if (l + 1 < L) {
        ArrayMeta const& mn = t.rs.meta[l + 1];
        EWT_CUDA(cudaMemsetAsync(words + mn.word_off, 0,
                                 ceil_div(mn.bits, 32) * 4, st));
        bool const write_order = l + 2 < L;
        T* dst = write_order ? bufs[l & 1] : nullptr;
        PhaseTimer pt(EWT_PHASE_SPLIT, st);
        if (t.pow2)
          launch_split<T, true>(write_order, src, dst, n, t.level_bits[l],
                                mn.bits, l, v, words + mn.word_off,
                                slow_tiles.as<uint32_t>(), err_build, st);
        else
          launch_split<T, false>(write_order, src, dst, n, t.level_bits[l],
                                 mn.bits, l, v, words + mn.word_off,
                                 slow_tiles.as<uint32_t>(), err_build, st);
        src = dst;
      }
    }
  }
  build_rs_samples(t.rs, st);
  if (want_groups && std::count(t.rs.skip_blocks.begin(), t.rs.skip_blocks.end(), 0) == 0) {
    // no rank blocks: only the totals of ones come over (below)
    t.rs.rb.alloc(0);
    t.rs.ds.alloc(0);
    EWT_CUDA(cudaMemcpyAsync(t.rs.meta.data(), t.rs.meta_d.get(), L * sizeof(ArrayMeta),
                             cudaMemcpyDeviceToHost, st));
  } else {
    build_rank_blocks(t.rs, st);
  }
  uint32_t build_err = 0;
  EWT_CUDA(cudaMemcpyAsync(&build_err, err_build, 4, cudaMemcpyDeviceToHost,
                           st));
  std::vector<uint64_t> c(sigma + 1);
  EWT_CUDA(cudaMemcpyAsync(c.data(), t.counts_d.get(), (sigma + 1) * 8,
                           cudaMemcpyDeviceToHost, st));
  EWT_CUDA(cudaStreamSynchronize(st));
  EWT_REQUIRE(!(build_err & 1), EWT_ERR_ALPHABET,
              "the text holds a symbol above the alphabet's last symbol");
  EWT_REQUIRE(build_err == 0, EWT_ERR_CUDA,
              "internal consistency check failed while building levels (kind " +
                  std::to_string(build_err) + ")");
  t.counts.assign(c.begin(), c.begin() + sigma);
  t.occ.resize(sigma);
  for (uint64_t i = 0; i < sigma; ++i) t.occ[i] = c[i + 1] - c[i];
  if (want_groups) {
    std::vector<std::vector<uint32_t const*>> planes;
    for (auto const& w : group_planes(L)) {
      std::vector<uint32_t const*> p{words + t.rs.meta[w.first].word_off};
      for (OrderPlanes const& o : kept)
        if (o.level == w.first)
          for (uint32_t j = 1; j <= w.second; ++j) p.push_back(o.plane(w.first + j));
      planes.push_back(std::move(p));
    }
    build_groups(t, t.pow2 ? c : code_starts, planes, st);
    kept.clear();
  }
  if (by_planes && !t.pow2) {
    // levels that short codes left mostly empty are packed (when the planes are
    // gone: the build's peak is the group levels')
    uint64_t bits = 0;
    for (uint64_t b : t.level_bits) bits += b;
    if (bits * 8 < L * n * 7) t.rs.pack(st);
  }
  v.rs = t.rs.view();
  v.groups = t.groups.view();
  drain.dismiss();  // the stream was waited for above
}

}  // namespace

void set_texts_synchronized(bool v) { t_texts_synced = v; }
bool texts_synchronized() { return t_texts_synced; }
void set_batch_member(bool v) { t_batch_member = v; }
void set_within_footprint(bool v) { t_within_footprint = v; }

void fill_tree_view(ewt_tree& t) {
  TreeView& v = t.view;
  v.rs = t.rs.view();
  v.counts = t.counts_d.as<uint64_t>();
  v.node_ranks = t.ranks_d.as<uint64_t>();
  v.node_base = t.node_base_d.as<uint64_t>();
  v.nodes_at_level = t.nodes_at_level_d.as<uint64_t>();
  v.code_len = t.code_len_d.as<uint64_t>();
  v.code_bits = t.code_bits_d.as<uint64_t>();
  v.alphabet = t.is_min ? nullptr : t.alphabet_d.get();
  v.n = t.n;
  v.sigma = t.sigma;
  v.codes_start = t.codes_start;
  v.num_ranks = t.nodes.size();
  v.num_nodes_until_last_level = t.nodes_until_last;
  v.levels = t.L;
  v.elem_size = t.elem_size;
  v.is_pow2 = t.pow2;
  v.is_min = t.is_min;
  v.groups = t.groups.view();
}

void build_tree(ewt_tree& t, const void* data, uint64_t n, int elem_size,
                const void* alphabet, uint64_t sigma, cudaStream_t stream) {
  EWT_REQUIRE(data != nullptr && n > 0, EWT_ERR_INVALID_ARGUMENT,
              "text must be non-empty");
  t.elem_size = static_cast<uint32_t>(elem_size);
  switch (elem_size) {
    case 1: build_typed<uint8_t>(t, data, n, alphabet, sigma, stream); break;
    case 2: build_typed<uint16_t>(t, data, n, alphabet, sigma, stream); break;
    case 4: build_typed<uint32_t>(t, data, n, alphabet, sigma, stream); break;
    case 8: build_typed<uint64_t>(t, data, n, alphabet, sigma, stream); break;
    default:
      throw Error(EWT_ERR_INVALID_ARGUMENT, "elem_size must be 1, 2, 4 or 8");
  }
}

void minimal_codes(uint64_t sigma, std::vector<uint64_t>& lens,
                   std::vector<uint64_t>& codes) {
  lens.clear();
  codes.clear();
  for (CodeH const& c : make_codes(sigma)) {
    lens.push_back(c.len);
    codes.push_back(c.code);
  }
}

uint64_t build_bytes_bound(uint64_t n, uint32_t elem_size, uint64_t sigma) {
  uint64_t const L = sigma < 2 ? 1 : h_ceil_log2(sigma);
  uint64_t const text = n * elem_size;
  // resident: level bits, L1/L2/samples, and the query side (group levels
  // or rank blocks, and dense select samples: below 2.5 times the level
  // bits -- octal blocks add 61 % and their samples 33 %)
  uint64_t const level_bits = L * (ceil_div(n, 32) + 64) * 4;
  uint64_t const support = L * (n / 8192 + n / 256 + n / 256 + 256);
  uint64_t const query = 5 * level_bits / 2;
  // count table, node ranks and node bases (per symbol and level)
  uint64_t const shape = (sigma + 1) * 8 * 4 + L * 64;
  // transient: a copy of a host text, and twice the symbols' width: the codes of
  // wide symbols with the bit planes that the passes hand on and keep for the
  // group levels (16 levels: 4.1 bytes per symbol), or two level orders of more
  // than 2^16 symbols; chunk tables and scratch.  (Closest for 16-bit symbols of
  // 2^15: 12.4 of 12.8 bytes per symbol.)
  uint64_t const order = n * std::max<uint32_t>(elem_size, L > 16 ? 4 : (L > 8 ? 2 : 1));
  uint64_t const transient = text + 2 * order + n / 64 + (64ull << 20);
  return level_bits + support + query + shape + transient;
}

void set_tree_shape(ewt_tree& t) {
  uint64_t const sigma = t.sigma;
  t.codes = make_codes(sigma);
  t.codes_start = sigma - t.codes.size();
  uint32_t const L = t.L;
  t.nodes = make_nodes(sigma, L);
  t.nodes_at_level.assign(L, 0);
  if (t.pow2) {
    for (uint32_t l = 0; l < L; ++l) t.nodes_at_level[l] = (uint64_t(1) << l) - 1;
  } else {
    // Counted as wavelet_tree.cuh:703-724 does (entry l-1 receives the
    // count of the level that just ended); the last level is counted too.
    uint64_t counter = 0;
    for (size_t i = 0; i < t.nodes.size(); ++i) {
      if (i > 0 && t.nodes[i].level > t.nodes[i - 1].level) {
        t.nodes_at_level[t.nodes[i].level - 1] = counter;
        counter = 0;
      }
      counter++;
    }
    if (!t.nodes.empty() && t.nodes.back().level == L - 1)
      t.nodes_at_level[L - 1] = counter;
  }
  t.node_base.assign(L + 1, 0);
  for (uint32_t l = 1; l <= L; ++l)
    t.node_base[l] = t.node_base[l - 1] + t.nodes_at_level[l - 1];
  EWT_REQUIRE(t.node_base[L] == t.nodes.size(), EWT_ERR_UNSUPPORTED,
              "inconsistent node bookkeeping for this alphabet size");
  t.nodes_until_last = L >= 1 ? t.node_base[L - 1] : 0;
}

}  // namespace ewt
