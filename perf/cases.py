"""Performance cases of the wavelet-tree library: what its users have it do.

Four kinds of work, each through the package's public entry points:

  build    a text becomes an index, which answers a first batch of mixed
           queries (WaveletTree(...), mixed / mixed_device, getters);
  queries  a batch over an index that the program keeps: access, rank,
           select or mixed, from device buffers or from host arrays;
  texts    many short texts become indexes in one call (build_batch), and
           one batch is answered over all of them (mixed_multi);
  bits     a packed bit array gets rank/select support (RankSelect) and
           answers rank and select batches.

Texts are iid over their alphabet, uniform or Zipf-distributed, as in the
benchmark and the tests; scattered alphabets have their symbols spread over
the type's whole range and are detected from the text when not given.  Every
symbol of the alphabet occurs.  Query batches hold 40 % access, 40 % rank and
20 % select; a few of the selects ask past the symbol's last occurrence.
"""
import math

import numpy as np
import torch

import ecl_wavelet_gb300 as E

DEV = "cuda"
ELEM = {"u8": 1, "u16": 2, "u32": 4, "u64": 8}
SIGNED = {"u8": torch.uint8, "u16": torch.int16, "u32": torch.int32, "u64": torch.int64}
UNSIGNED = {"u8": torch.uint8, "u16": torch.uint16, "u32": torch.uint32,
            "u64": torch.uint64}
NUMPY = {"u8": np.uint8, "u16": np.uint16, "u32": np.uint32, "u64": np.uint64}


def build(n, sigma, dtype="u8", scattered=False, given=True, zipf=False, host=False, m=0):
    return {"kind": "build", "n": n, "sigma": sigma, "dtype": dtype, "scattered": scattered,
            "given": given, "zipf": zipf, "host": host, "m": m}


def queries(n, sigma, m, op="mixed", dtype="u8", scattered=False, zipf=False, host=False):
    return {"kind": "queries", "n": n, "sigma": sigma, "dtype": dtype, "scattered": scattered,
            "given": True, "zipf": zipf, "host": host, "m": m, "op": op}


def texts(count, longest, m, dtype="u8"):
    return {"kind": "texts", "count": count, "longest": longest, "dtype": dtype, "m": m}


def bits(n, percent, m):
    return {"kind": "bits", "n": n, "percent": percent, "m": m}


def listed():
    return [
        # the benchmark's construction: the largest text, resident on the device
        dict(build(6 << 30, 256, m=1 << 25), name="build u8 s256 6Gi"),
        # the tests' configuration 1: a DNA-like text of medium size
        dict(build(1 << 24, 4, m=1 << 20), name="build u8 s4 16Mi"),
        # an ordinary byte text read from a file: host memory, odd length, an
        # alphabet of 96 printable symbols that the library has to find
        dict(build(150_000_001, 96, scattered=True, given=False, host=True, m=750_000),
             name="build u8 s96 host 150M"),
        # large alphabet, skewed: 16-bit tokens
        dict(build(1 << 28, 65536, "u16", zipf=True, m=3_000_000), name="build u16 s65536 zipf 256Mi"),
        # word identifiers: wide symbols, a sparse alphabet to be found
        dict(build(20_000_003, 10_000, "u32", scattered=True, given=False, m=1 << 18),
             name="build u32 s10000 20M"),
        # a short text from host memory: launches and latency
        dict(build(65_537, 256, host=True, m=1000), name="build u8 s256 host 64Ki"),
        # a collection of documents in one call
        dict(texts(64, 1 << 22, 1 << 20), name="texts 64"),
        # the benchmark's query batch over a large index, on the device
        dict(queries(1 << 30, 256, 1 << 24), name="queries s256 1Gi 16Mi"),
        # queries over an ordinary byte text's index (no power of two)
        dict(queries(1 << 27, 96, 1 << 22, scattered=True), name="queries s96 128Mi 4Mi"),
        # an interactive request: a small host batch, where latency counts
        dict(queries(1 << 24, 256, 1024, host=True), name="queries s256 host 1Ki"),
        # a large host batch of one type: copies against kernels
        dict(queries(1 << 28, 64, 3_000_001, op="rank", host=True), name="queries s64 host rank 3M"),
        # the standalone bit vector
        dict(bits((1 << 28) + 17, 50, 1 << 20), name="bits 256Mi"),
    ]


def log_int(rng, lo, hi):
    """Whole number spread over the logarithm of [lo, hi]; half of them odd."""
    return int(min(hi, max(lo, math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "queries", "queries", "texts", "bits"])
    if kind == "texts":
        return texts(log_int(rng, 8, 128), log_int(rng, 1 << 17, 1 << 22),
                     log_int(rng, 1 << 12, 1 << 20), rng.choice(["u8", "u8", "u16"]))
    if kind == "bits":
        return bits(log_int(rng, 1 << 16, 1 << 30), rng.choice([2, 20, 50, 90]),
                    log_int(rng, 1 << 8, 1 << 21))
    dtype = rng.choice(["u8", "u8", "u8", "u16", "u32", "u64"])
    if dtype == "u8":
        sigma = rng.choice([4, 5, 16, 26, 64, 75, 96, 128, 200, 256])
        hi = 1 << 30
    elif dtype == "u16":
        sigma = rng.choice([1024, 4096, 65536, log_int(rng, 300, 60_000)])
        hi = 1 << 28
    else:
        sigma = rng.choice([4096, log_int(rng, 300, 50_000), log_int(rng, 300, 50_000)])
        hi = 1 << 25
    zipf = rng.random() < 0.3
    scattered = dtype in ("u32", "u64") or (rng.random() < 0.4 and sigma <= 96)
    host = rng.random() < 0.4
    if host or scattered or sigma & (sigma - 1):
        hi >>= 2  # within the time that the largest listed case takes
    n = log_int(rng, max(1 << 14, 2 * sigma), hi)
    if kind == "build":
        return build(n, sigma, dtype, scattered, not scattered or rng.random() < 0.5, zipf, host,
                     log_int(rng, 1000, max(1000, min(1 << 22, n // 16))))
    return queries(n, sigma, log_int(rng, 16, 1 << 22), rng.choice(["mixed", "mixed", "access", "rank", "select"]),
                   dtype, scattered, zipf, host)


class State:
    pass


def make_alphabet(case, gen):
    """Sorted symbols (int64; 8-byte symbols stay below 2^63)."""
    sigma = case["sigma"]
    if not case["scattered"]:
        return torch.arange(sigma, device=DEV)
    top = {"u8": 1 << 8, "u16": 1 << 16, "u32": 1 << 32, "u64": 1 << 62}[case["dtype"]]
    if top <= 1 << 16:
        return torch.randperm(top, device=DEV, generator=gen)[:sigma].sort().values
    step = top // sigma  # one symbol in each of sigma equal ranges
    return torch.arange(sigma, device=DEV) * step + \
        torch.randint(0, step, (sigma,), device=DEV, generator=gen)


def make_text(n, alphabet, dtype, zipf, gen):
    """Text of n symbols, every symbol of the alphabet at least once."""
    sigma = alphabet.numel()
    out = torch.empty(n, dtype=SIGNED[dtype], device=DEV)
    symbols = alphabet.to(SIGNED[dtype])
    minimal = bool((alphabet == torch.arange(sigma, device=DEV)).all())
    cdf = None
    if zipf:
        w = 1.0 / torch.arange(1, sigma + 1, device=DEV, dtype=torch.float64) ** 1.1
        cdf = torch.cumsum(w, 0) / w.sum()
    step = 1 << 27
    for a in range(0, n, step):
        b = min(n, a + step)
        if cdf is None and minimal and dtype == "u8":
            out[a:b] = torch.randint(0, sigma, (b - a,), device=DEV, generator=gen,
                                     dtype=torch.uint8)
            continue
        if cdf is None:
            ids = torch.randint(0, sigma, (b - a,), device=DEV, generator=gen)
        else:
            u = torch.rand(b - a, device=DEV, dtype=torch.float64, generator=gen)
            ids = torch.searchsorted(cdf, u).clamp_(max=sigma - 1)
        out[a:b] = symbols[ids]
    at = torch.randperm(n, device=DEV, generator=gen)[:sigma] if n < 1 << 24 else \
        torch.arange(sigma, device=DEV) * (n // sigma)
    out[at] = symbols
    return out


def widened(t, dtype):
    """Symbols as non-negative int64."""
    w = t.to(torch.int64)
    return w if dtype in ("u8", "u64") else w & ((1 << 8 * ELEM[dtype]) - 1)


def make_queries(text, alphabet, dtype, m, gen, op="mixed"):
    """(types, records): uint8 types and [m, 2] int64 records {index, symbol}."""
    n, sigma = text.numel(), alphabet.numel()
    rnd = torch.rand(m, device=DEV, dtype=torch.float64, generator=gen)
    kinds = {"access": 0, "rank": 1, "select": 2}
    types = torch.where(rnd < 0.4, 0, torch.where(rnd < 0.8, 1, 2)) if op == "mixed" else \
        torch.full((m,), kinds[op], device=DEV)
    ids = torch.randint(0, sigma, (m,), device=DEV, generator=gen)
    # selects: symbols as the text holds them, up to about their count
    sample = widened(text[torch.randint(0, n, (1 << 18,), device=DEV, generator=gen)], dtype)
    freq = torch.bincount(torch.searchsorted(alphabet, sample), minlength=sigma).double() / sample.numel()
    sel = torch.searchsorted(alphabet, sample)[torch.randint(0, sample.numel(), (m,), device=DEV, generator=gen)]
    ids = torch.where(types == 2, sel, ids)
    u = torch.rand(m, device=DEV, dtype=torch.float64, generator=gen)
    k = 1 + (u * freq[ids] * n).to(torch.int64)
    index = torch.where(types == 2, k, (u * n).to(torch.int64).clamp_(max=n - 1))
    return types.to(torch.uint8), torch.stack([index, alphabet[ids]], 1).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    s = State()
    s.case = case
    if case["kind"] == "bits":
        prepare_bits(s, gen)
    elif case["kind"] == "texts":
        prepare_texts(s, gen, seed)
    else:
        prepare_text(s, gen)
    torch.cuda.synchronize()
    return s


def prepare_text(s, gen):
    case, dtype = s.case, s.case["dtype"]
    alphabet = make_alphabet(case, gen)
    text = make_text(case["n"], alphabet, dtype, case["zipf"], gen)
    types, records = make_queries(text, alphabet, dtype, case["m"], gen, case.get("op", "mixed"))
    s.alphabet = alphabet.cpu().numpy().astype(NUMPY[dtype]) if case["given"] else None
    s.text = text.view(UNSIGNED[dtype])
    if case["kind"] == "queries":
        torch.cuda.synchronize()
        s.tree = E.WaveletTree(s.text, s.alphabet)
        del s.text
    elif case["host"]:
        s.text = s.text.cpu().numpy()
    access = case.get("op") == "access"
    if case["host"]:
        s.types = types.cpu().numpy()
        s.q = records.cpu().numpy().view(np.uint64).view(E.query_dtype(NUMPY[dtype])).reshape(-1)
        if access:
            s.q = np.ascontiguousarray(s.q["index"])
    else:
        s.types = types
        s.q = records[:, 0].contiguous() if access else records
        s.out = torch.zeros(case["m"], dtype=torch.int64 if not access else SIGNED[dtype], device=DEV)


def prepare_texts(s, gen, seed):
    case, dtype = s.case, s.case["dtype"]
    rng = np.random.default_rng(seed)
    shortest, count = 1 << 16, case["count"]
    # lengths spread over the logarithm of their range (the same for every
    # seed but for their order), alphabets of 4 to 256 symbols in turn
    u = (np.arange(count) + 0.5) / count
    lengths = np.exp(math.log(shortest) + u * math.log(case["longest"] / shortest)).astype(np.int64)
    sigmas = np.array([4, 16, 64, 256])[np.arange(count) % 4]
    order = rng.permutation(count)
    s.texts, s.alphabets, types, records, tree_of = [], [], [], [], []
    for j, i in enumerate(order):
        a = torch.arange(int(sigmas[i]), device=DEV)
        t = make_text(int(lengths[i]), a, dtype, False, gen)
        mi = case["m"] // count + (j < case["m"] % count)
        ty, rec = make_queries(t, a, dtype, mi, gen)
        s.texts.append(t.view(UNSIGNED[dtype]))
        s.alphabets.append(a.cpu().numpy().astype(NUMPY[dtype]))
        types.append(ty)
        records.append(rec)
        tree_of.append(torch.full((mi,), j, device=DEV, dtype=torch.int32))
    mix = torch.randperm(case["m"], device=DEV, generator=gen)
    s.types = torch.cat(types)[mix].cpu().numpy()
    s.q = torch.cat(records)[mix].cpu().numpy().view(np.uint64).view(E.query_dtype(NUMPY[dtype])).reshape(-1)
    s.tree_of = torch.cat(tree_of)[mix].cpu().numpy().view(np.uint32)


def prepare_bits(s, gen):
    n, m = s.case["n"], s.case["m"]
    words = -(-n // 32)
    out = torch.empty(words, dtype=torch.int32, device=DEV)
    weight = 1 << torch.arange(32, device=DEV)
    ones = 0
    step = 1 << 21
    for a in range(0, words, step):
        b = min(words, a + step)
        bit = torch.rand((b - a, 32), device=DEV, generator=gen) < s.case["percent"] / 100
        if b == words and n % 32:
            bit[-1, n % 32:] = False
        ones += int(bit.sum())
        out[a:b] = (bit * weight).sum(1).to(torch.int32)
    s.words = out.cpu().numpy().view(np.uint32)
    s.pos = torch.randint(0, n + 1, (m,), device=DEV, generator=gen).cpu().numpy().astype(np.uint64)
    s.k = torch.randint(1, max(2, ones + 1), (m,), device=DEV, generator=gen).cpu().numpy().astype(np.uint64)


def checked(status):
    if status != E.EWT_OK:
        raise RuntimeError("the batch was refused: %d" % status)


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "build":
        tree = E.WaveletTree(s.text, s.alphabet)
        if case["host"]:
            answers = tree.mixed(s.types, s.q)
        else:
            stream = torch.cuda.current_stream().cuda_stream
            tree.mixed_device(s.types.data_ptr(), s.q.data_ptr(), case["m"], s.out.data_ptr(), stream)
            checked(tree.query_status(stream))
            answers = s.out
        got = {"answers": answers, "counts": tree.export("COUNTS").view(np.int64),
               "alphabet": tree.export("ALPHABET").view(np.int64), "levels": tree.getNumLevels()}
        tree.close()
        return got
    if kind == "queries":
        op = case["op"]
        if case["host"]:
            return s.tree.mixed(s.types, s.q) if op == "mixed" else getattr(s.tree, op)(s.q)
        stream = torch.cuda.current_stream().cuda_stream
        if op == "mixed":
            s.tree.mixed_device(s.types.data_ptr(), s.q.data_ptr(), case["m"], s.out.data_ptr(), stream)
        else:
            getattr(s.tree, op + "_device")(s.q.data_ptr(), case["m"], s.out.data_ptr(), stream)
        return s.out
    if kind == "texts":
        trees = E.build_batch(s.texts, s.alphabets)
        answers = E.mixed_multi(trees, s.tree_of, s.types, s.q)
        counts = np.concatenate([t.export("COUNTS") for t in trees])
        for t in trees:
            t.close()
        return {"answers": answers, "counts": counts.view(np.int64)}
    rs = E.RankSelect([s.words], [case["n"]])
    got = {"rank": rs.rank(0, 1, s.pos), "select": rs.select(0, 1, s.k),
           "ones": rs.export("TOTAL_ONES").view(np.int64)}
    rs.close()
    return got


def work(case):
    """Inputs read once; the index (level bits with the reference's counts
    and samples, 1/16 of them) and the answers written once; 32 bytes of the
    index for each query that is answered on it."""
    m = case["m"]
    if case["kind"] == "bits":
        return {"bytes": case["n"] / 8 * (2 + 1 / 16) + 2 * m * (16 + 32), "flops": 0}
    if case["kind"] == "texts":
        shortest, count, longest = 1 << 16, case["count"], case["longest"]
        n = count * (longest - shortest) / math.log(longest / shortest)
        return {"bytes": n * (ELEM[case["dtype"]] + 5 / 8 * (1 + 1 / 16)) + m * (4 + 25 + 32), "flops": 0}
    per_query = (17 if case.get("op", "mixed") == "mixed" else 16) + 8 + 32
    if case.get("op") == "access":
        per_query = 8 + ELEM[case["dtype"]] + 32
    total = m * per_query
    if case["kind"] == "build":
        levels = max(1, math.ceil(math.log2(case["sigma"])))
        total += case["n"] * (ELEM[case["dtype"]] + levels / 8 * (1 + 1 / 16))
    return {"bytes": total, "flops": 0}


def plain_answers(text, alphabet, dtype, types, records):
    """Answers by sorting the text's positions by symbol: the k-th occurrence
    of a symbol is an entry of its stretch, a rank the number of its entries
    below the position."""
    n, sigma = text.numel(), alphabet.numel()
    ids = torch.searchsorted(alphabet, widened(text, dtype))
    order = torch.sort(ids.to(torch.int32), stable=True).indices
    count = torch.bincount(ids, minlength=sigma)
    start = torch.cumsum(count, 0) - count
    key = ids[order] * (n + 1) + order  # ascending
    out = torch.zeros(types.numel(), dtype=torch.int64, device=DEV)
    index, sym = records[:, 0], records[:, 1]
    c = torch.searchsorted(alphabet, sym)
    acc, rank, sel = types == 0, types == 1, types == 2
    out[acc] = widened(text[index[acc]], dtype)
    out[rank] = torch.searchsorted(key, c[rank] * (n + 1) + index[rank]) - start[c[rank]]
    k = index[sel]
    found = k <= count[c[sel]]
    at = (start[c[sel]] + k - 1).clamp(max=n - 1)
    out[sel] = torch.where(found, order[at], torch.full_like(k, n))
    return out, start


def exact(case, seed):
    """The answers by plain scans in torch; None for texts above 2^28 symbols."""
    if case.get("n", 0) > 1 << 28 or case["kind"] == "texts":
        return None
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    n, m = case["n"], case["m"]
    if case["kind"] == "bits":
        s = State()
        s.case = case
        prepare_bits(s, gen)
        bit = np.unpackbits(s.words.view(np.uint8), bitorder="little")[:n]
        at = np.flatnonzero(bit)
        return {"rank": np.searchsorted(at, s.pos.astype(np.int64)).astype(np.uint64),
                "select": at[np.minimum(s.k.astype(np.int64), at.size) - 1].astype(np.uint64),
                "ones": np.array([at.size], dtype=np.int64)}
    alphabet = make_alphabet(case, gen)
    dtype = case["dtype"]
    text = make_text(n, alphabet, dtype, case["zipf"], gen)
    types, records = make_queries(text, alphabet, dtype, m, gen, case.get("op", "mixed"))
    answers, start = plain_answers(text, alphabet, dtype, types, records)
    if case.get("op") == "access":
        answers = answers.to(SIGNED[dtype])
        return answers.cpu().numpy().view(NUMPY[dtype]) if case["host"] else answers
    if case["host"]:
        answers = answers.cpu().numpy().view(np.uint64)
    if case["kind"] == "queries":
        return answers
    return {"answers": answers, "counts": start.cpu().numpy(), "alphabet": alphabet.cpu().numpy(),
            "levels": max(1, math.ceil(math.log2(case["sigma"])))}
