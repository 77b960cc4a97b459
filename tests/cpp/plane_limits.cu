// The forms of the bit-plane passes for the largest texts, at small sizes: 64-bit
// word indices, orders in two allocations, and texts read in parts must write the
// levels, class starts and kept planes of the usual form.  plane_limits <seed>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../../ecl_wavelet_gb300/csrc/planes.cuh"

using namespace ewt;

struct Result {
  std::vector<uint32_t> levels, planes;
  std::vector<uint64_t> starts;
};

template <class T>
Result run(std::vector<T> const& text, uint32_t L, PlaneLimits const& limits, bool in_parts,
           cudaStream_t st) {
  uint64_t const n = text.size(), stride = ceil_div(ceil_div(n, 32), 32) * 32;
  DevBuf x(n * sizeof(T) + 64), words(L * stride * 4 + 64), starts(((uint64_t(1) << L) + 1) * 8), err(4);
  EWT_CUDA(cudaMemcpyAsync(x.get(), text.data(), n * sizeof(T), cudaMemcpyHostToDevice, st));
  EWT_CUDA(cudaMemsetAsync(words.get(), 0, words.bytes(), st));
  EWT_CUDA(cudaMemsetAsync(err.get(), 0, 4, st));
  std::vector<uint32_t*> out(L);
  for (uint32_t l = 0; l < L; ++l) out[l] = words.as<uint32_t>() + l * stride;
  std::vector<std::pair<uint32_t, uint32_t>> wanted;  // as the group levels of three ask for
  for (uint32_t l = 0; l + 3 <= L; l += 3) wanted.push_back({l, 2});
  PlaneText<T> t;
  DevBuf part(40'000 * sizeof(T));
  if (in_parts) {  // one or two tiles at a time, through one buffer
    t.part_symbols = 40'000;
    t.part = [&](uint64_t begin, uint64_t len) {
      EWT_REQUIRE(len <= 40'000, EWT_ERR_CUDA, "part too long");
      EWT_CUDA(cudaMemcpyAsync(part.get(), x.as<T>() + begin, len * sizeof(T),
                               cudaMemcpyDeviceToDevice, st));
      return part.as<T const>();
    };
  } else {
    t.sym = x.as<T>();
  }
  t.n = n;
  t.L = L;
  auto const kept = run_plane_passes<T>(t, out.data(), std::vector<uint64_t>(L, stride).data(),
                                        starts.as<uint64_t>(), wanted, err.as<uint32_t>(), st, limits);
  Result r;
  r.levels.resize(L * stride);
  r.starts.resize((uint64_t(1) << L) + 1);
  EWT_CUDA(cudaMemcpyAsync(r.levels.data(), words.get(), r.levels.size() * 4, cudaMemcpyDeviceToHost, st));
  EWT_CUDA(cudaMemcpyAsync(r.starts.data(), starts.get(), r.starts.size() * 8, cudaMemcpyDeviceToHost, st));
  for (auto const& w : wanted)
    for (OrderPlanes const& o : kept)
      if (o.level == w.first)
        for (uint32_t j = 1; j <= w.second; ++j) {
          std::vector<uint32_t> p(ceil_div(n, 32));
          EWT_CUDA(cudaMemcpyAsync(p.data(), o.plane(w.first + j), p.size() * 4, cudaMemcpyDeviceToHost, st));
          EWT_CUDA(cudaStreamSynchronize(st));
          r.planes.insert(r.planes.end(), p.begin(), p.end());
        }
  EWT_CUDA(cudaStreamSynchronize(st));
  return r;
}

template <class T>
int check(uint32_t L, uint64_t n, bool skewed, std::mt19937_64& rng, cudaStream_t st) {
  std::vector<T> text(n);
  uint64_t const sigma = uint64_t(1) << L;
  for (auto& c : text) c = T(skewed && rng() % 8 ? sigma / 2 : rng() % sigma);
  Result const usual = run(text, L, {}, false, st);
  int bad = 0;
  for (int form = 1; form < 8; ++form) {
    PlaneLimits limits;
    if (form & 1) limits.wide_words = 0;
    if (form & 2) limits.split_bytes = 0;
    Result const r = run(text, L, limits, form & 4, st);
    bad += r.levels != usual.levels || r.starts != usual.starts || r.planes != usual.planes;
  }
  // the levels hold the text: level 0 is its highest bit
  for (uint64_t i = 0; i < n; ++i)
    if (((usual.levels[i / 32] >> (i % 32)) & 1) != (uint64_t(text[i]) >> (L - 1))) {
      ++bad;
      break;
    }
  std::printf("L %u n %llu %s: %d differences\n", L, (unsigned long long)n, skewed ? "skewed" : "even", bad);
  return bad;
}

int main(int argc, char** argv) {
  std::mt19937_64 rng(argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1);
  cudaStream_t st;
  EWT_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  int bad = 0;
  {
    AllocStream as(st);
    for (uint64_t n : {1ull, 1000ull, 13'825ull, 100'003ull})
      for (bool skewed : {false, true}) {
        for (uint32_t L : {1u, 2u, 5u, 8u}) bad += check<uint8_t>(L, n, skewed, rng, st);
        for (uint32_t L : {9u, 12u, 16u}) bad += check<uint16_t>(L, n, skewed, rng, st);
      }
  }
  EWT_CUDA(cudaStreamSynchronize(st));
  EWT_CUDA(cudaStreamDestroy(st));
  return bad != 0;
}
