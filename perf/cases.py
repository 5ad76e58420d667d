"""The calls that programs built on this library spend their time in, as measurable cases.

Every case goes through the public entry points (the Engine and Server classes and, where a
program keeps its data on the GPU, the device calls of the C ABI) on one engine that the
process keeps, as a search program does.  `kind` names the call:

    range      Engine.sieve_range: pi, twins, widest gap, 6-tuples of [lo, lo + len), with
               per-block results and per-segment bitmap hashes where the options ask for them
    gaps       Engine.gap_stats: gap histogram, increasing runs and chains of a range
    wieferich  Engine.wieferich_range: base-2 Fermat quotients of every prime of a range
    fermat     Engine.fermat_quotient: quotients of a host array of primes
    bpsw       Engine.bpsw: verdicts of a host array of candidates
    lists      mp_bpsw_lists_dev: verdicts of candidate lists that are on the device
    tuples     Engine.tuple_count: prime sextuplets of a range
    chains     Engine.chain_sieve: chains of consecutive primes with gaps 2, 4, 6, ...
    served     Server: range and primality requests of mixed sizes, submitted together
"""
import ctypes
import math

import numpy as np
import torch

import mathpub_b200 as mp

SEXTUPLET = (0, 4, 6, 10, 12, 16)
CHAIN_ROWS = 1 << 13                     # far above the chains any of the ranges below holds

_engine = None
_server = None
_height = 0


def _eng(top):
    """The process's engine, with its sieving primes resident up to sqrt(top)."""
    global _engine, _height
    if _engine is None:
        _engine = mp.Engine(0)
    if top > _height:
        _engine.sieve_range(top - 100000, top)
        _height = top
    return _engine


def _srv():
    """The process's server, on an engine of its own, for ranges up to 1e18."""
    global _server
    if _server is None:
        _server = mp.Server(mp.Engine(0))
    return _server


def listed():
    return [
        # one small window looked at by itself (a gap record's surroundings, a served request
        # of the shortest kind): latency of a call
        {"name": "range_short", "kind": "range", "lo": 10**12, "len": 2**20, "block_log2": 0, "hash_log2": 0},
        # a plain segmented sieve of 1e8 integers with a hash for each 32 KiB segment
        {"name": "range_segments", "kind": "range", "lo": 10**9, "len": 10**8, "block_log2": 0, "hash_log2": 19},
        # a chunk of a long scan at a large offset with every output
        {"name": "range_scan", "kind": "range", "lo": 10**15, "len": 2**34, "block_log2": 24, "hash_log2": 20},
        # the same at the top heights, where most sieving primes hit a chunk a few times only
        {"name": "range_high", "kind": "range", "lo": 9 * 10**17, "len": 2**32, "block_log2": 0, "hash_log2": 0},
        # gap statistics of a chunk (A158939, A252768)
        {"name": "gaps", "kind": "gaps", "lo": 10**13, "len": 2**32},
        # a chunk of a Wieferich scan: sieve, quotients and the chunk log's checksum
        {"name": "wieferich", "kind": "wieferich", "lo": 10**12, "len": 10**9},
        # quotients of a host array of primes at today's search heights (128-bit moduli)
        {"name": "fermat_high", "kind": "fermat", "lo": 10**16, "count": 2**20},
        # a handful of candidates from a search program: latency of a call
        {"name": "bpsw_few", "kind": "bpsw", "count": 100},
        # many lists of uneven length, resident on the device, one launch
        {"name": "bpsw_lists", "kind": "lists", "count": 2**24, "lists": 1024},
        # prime sextuplets over a window (A350826)
        {"name": "tuples", "kind": "tuples", "lo": 10**15, "len": 2 * 10**12},
        # a stretch of a chain search at the record heights (A016045), long enough to hold chains
        {"name": "chains", "kind": "chains", "lo": 1397 * 10**15, "len": 10**15, "k": 11},
        # a mixed stream of requests, continuously batched
        {"name": "served", "kind": "served", "requests": 192},
    ]


def _logu(rng, a, b):
    return int(math.exp(rng.uniform(math.log(a), math.log(b))))


def draw(rng):
    kind = rng.choice(["range", "range", "range", "gaps", "wieferich", "fermat", "bpsw", "lists", "tuples", "chains",
                       "served"])
    if kind == "range":
        c = {"kind": kind, "lo": _logu(rng, 10**9, 9 * 10**17), "len": _logu(rng, 2**16, 2**33),
             "block_log2": 0, "hash_log2": 0}
        if c["len"] >= 2**24 and rng.random() < 0.5:
            c["block_log2"] = rng.choice([22, 24, 26])
        if rng.random() < 0.5:
            c["hash_log2"] = rng.choice([19, 20, 22])
        return c
    if kind == "gaps":
        return {"kind": kind, "lo": _logu(rng, 10**9, 10**15), "len": _logu(rng, 2**22, 2**33)}
    if kind == "wieferich":
        return {"kind": kind, "lo": _logu(rng, 10**9, 10**15), "len": _logu(rng, 10**6, 2 * 10**9)}
    if kind == "fermat":
        return {"kind": kind, "lo": _logu(rng, 10**9, 10**17), "count": _logu(rng, 2**8, 2**21)}
    if kind == "bpsw":
        return {"kind": kind, "count": _logu(rng, 100, 2**20)}
    if kind == "lists":
        return {"kind": kind, "count": _logu(rng, 2**16, 2**24), "lists": _logu(rng, 1, 256)}
    if kind == "tuples":
        return {"kind": kind, "lo": _logu(rng, 10**13, 10**18), "len": _logu(rng, 10**11, 10**13)}
    if kind == "chains":
        return {"kind": kind, "lo": _logu(rng, 10**17, 10**19), "len": _logu(rng, 2 * 10**14, 10**15),
                "k": rng.choice([10, 11])}
    return {"kind": kind, "requests": _logu(rng, 24, 192)}


def _window(case, seed):
    """[lo, hi) of the case for this seed: the start moves by up to a thousandth of the height."""
    r = np.random.default_rng(seed)
    lo = case["lo"] + int(r.integers(0, max(2, case["lo"] // 1000)))
    return lo, lo + case.get("len", 0)


def _top(case):
    return case["lo"] + case["lo"] // 1000 + case.get("len", 0) + 100000


def _fermat_primes(case, seed):
    lo, _ = _window(case, seed)
    e = _eng(_top(case) + 50 * case["count"])
    span = int(case["count"] * math.log(lo) * 1.05) + 20000
    return e.primes_range(lo, lo + span)[: case["count"]]


def _requests(case, seed):
    """70% ranges, 30% primality batches; the kinds and sizes are the stream's, the windows and
    candidates the seed's."""
    r, size = np.random.default_rng(seed), np.random.default_rng(case["requests"])
    cand, _ = mp.bpsw_workload(seed, 1 << 20, 1)
    reqs = []
    for i in range(case["requests"]):
        if i * 7 % 10 < 7:
            lo = int(math.exp(r.uniform(math.log(1e9), math.log(9e17))))
            reqs.append((lo, lo + int(2 ** size.uniform(16, 32))))
        else:
            m = int(size.integers(1, 65537))
            at = int(r.integers(0, len(cand) - m + 1))
            reqs.append(cand[at: at + m].copy())
    return reqs


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("range", "gaps", "wieferich"):
        s["lo"], s["hi"] = _window(case, seed)
        s["e"] = _eng(_top(case))
    elif kind in ("tuples", "chains"):
        s["lo"], s["hi"] = _window(case, seed)
        s["e"] = _eng(0)
    elif kind == "fermat":
        s["p"] = _fermat_primes(case, seed)
        s["e"] = _eng(0)
    elif kind == "bpsw":
        n, _ = mp.bpsw_workload(seed, max(case["count"], 64), 1)
        s["n"] = n[: case["count"]].copy()
        s["e"] = _eng(0)
    elif kind == "lists":
        n, _ = mp.bpsw_workload(seed, case["count"], 1)
        _, lens = mp.bpsw_workload(case["lists"], case["count"], case["lists"])
        offs = np.zeros(len(lens) + 1, dtype=np.uint64)
        offs[1:] = np.cumsum((lens.astype(np.uint64) + np.uint64(31)) & ~np.uint64(31))
        flat = np.zeros(int(offs[-1]), dtype=np.uint64)
        at = 0
        for i, m in enumerate(lens):
            flat[int(offs[i]): int(offs[i]) + int(m)] = n[at: at + int(m)]
            at += int(m)
        s["n"] = torch.from_numpy(flat.view(np.int64)).cuda()
        s["bits"] = torch.zeros(len(flat) // 32, dtype=torch.int32, device="cuda")
        s["offs"], s["lens"] = offs, np.ascontiguousarray(lens)
        s["e"] = _eng(0)
    elif kind == "served":
        s["server"] = _srv()
        s["reqs"] = _requests(case, seed)
    else:
        raise ValueError(kind)
    return s


def _stats(r):
    """The range results, as one array of whole numbers."""
    return np.array([r[f] for f in mp.STATS_FIELDS], dtype=np.uint64)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr() if torch.is_tensor(t) else t.ctypes.data)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "range":
        r = s["e"].sieve_range(s["lo"], s["hi"], block_log2=case["block_log2"], hash_log2=case["hash_log2"])
        out = {"stats": _stats(r)}
        if "blocks" in r:
            out["blocks"] = r["blocks"].view(np.uint64).reshape(len(r["blocks"]), -1)
        if "hashes" in r:
            out["hashes"] = r["hashes"]
        return out
    if kind == "gaps":
        return s["e"].gap_stats(s["lo"], s["hi"])
    if kind == "wieferich":
        r = s["e"].wieferich_range(s["lo"], s["hi"])
        return np.array([r[f] for f in mp.WIEF_FIELDS] + r["hits"], dtype=np.uint64)
    if kind == "fermat":
        return s["e"].fermat_quotient(s["p"])
    if kind == "bpsw":
        return s["e"].bpsw(s["n"])
    if kind == "lists":
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = mp.lib().mp_bpsw_lists_dev(s["e"].handle, _ptr(s["n"]), _ptr(s["offs"]), _ptr(s["lens"]), len(s["lens"]),
                                        _ptr(s["bits"]), mp.MODE_BATCHED, st)
        if rc != mp.MP_OK:
            raise mp.MathpubError(rc, "mp_bpsw_lists_dev")
        return s["bits"]
    if kind == "tuples":
        return np.array(s["e"].tuple_count(s["lo"], s["hi"], SEXTUPLET), dtype=np.uint64)
    if kind == "chains":
        heads, lens = s["e"].chain_sieve(s["lo"], s["hi"], case["k"])
        table = np.zeros((CHAIN_ROWS, 2), dtype=np.uint64)     # every chain, in rows of one table
        table[: len(heads), 0], table[: len(heads), 1] = heads, lens
        return {"count": len(heads), "chains": table}
    v = s["server"]
    ids = [v.submit_range(*q) if isinstance(q, tuple) else v.submit_bpsw(q) for q in s["reqs"]]
    ranges, verdicts = [], []
    for i in ids:
        r = v.poll(i, 1000)
        while r is None:
            r = v.poll(i, 1000)
        if r["status"] != mp.MP_OK:
            raise mp.MathpubError(r["status"], "served request")
        if r["kind"] == 1:
            ranges.append([r["pi"], r["max_gap"], r["gap_start"], r["twins"]])
        else:
            verdicts.append(r["verdicts"])
    return {"ranges": np.array(ranges, dtype=np.uint64).reshape(-1, 4),
            "verdicts": np.concatenate(verdicts) if verdicts else np.zeros(1, dtype=bool)}


def _marks(lo, hi):
    """Multiples k q, k coprime to 30, of the sieving primes 97 <= q <= sqrt(hi) in [lo, hi)
    (Mertens): what a sieve of the range has to strike."""
    top = max(math.sqrt(hi), 98.0)
    return (hi - lo) * (8 / 30) * math.log(math.log(top) / math.log(97.0))


def _nprimes(x):
    return x / max(1.0, math.log(x) - 1)


def work(case):
    kind = case["kind"]
    if kind in ("range", "gaps", "wieferich"):
        lo, hi = case["lo"], case["lo"] + case["len"]
        b = 4 * _nprimes(math.sqrt(hi))                       # the sieving primes
        f = _marks(lo, hi)                                    # one OR for each
        if kind == "range":
            if case["block_log2"]:
                b += 64 * (case["len"] >> case["block_log2"])
            if case["hash_log2"]:
                b += 8 * (case["len"] >> case["hash_log2"])
                f += 2 * case["len"] / 16                     # an XOR and a product for each byte
        elif kind == "gaps":
            f += 4 * case["len"] / math.log(lo)
            b += 9000
        else:
            n = case["len"] / math.log(lo)
            f += n * math.log2(lo) * 2 * 39                   # one three-limb product for each bit
            b += 200
        return {"bytes": b + 64, "flops": f}
    if kind == "fermat":
        k = 39 if case["lo"] < 2**46 else 68
        return {"bytes": 16 * case["count"], "flops": case["count"] * math.log2(case["lo"]) * 2 * k}
    if kind in ("bpsw", "lists"):
        # about a third of the candidates of the workload survive trial division; a product of
        # 19 multiply-adds for each of 62 bits
        return {"bytes": 8.125 * case["count"], "flops": case["count"] * 0.45 * 62 * 2 * 19}
    if kind == "tuples":
        # 5005 classes of a wheel of 9699690; one AND for each 32 integers of a class and prime
        return {"bytes": 24e6, "flops": case["len"] * 5005 / 9699690 / 32 * 46}
    if kind == "chains":
        return {"bytes": 24e6, "flops": case["len"] * 12960 / 9699690 / 32 * 80}
    n = case["requests"]
    f = 0.7 * n * 3.9e8 * 0.27 + 0.3 * n * 32768 * 0.45 * 62 * 2 * 19
    return {"bytes": 0.3 * n * 32768 * 8 + 64 * n, "flops": f}


def _is_prime(n):
    if n < 2:
        return False
    for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        if n % p == 0:
            return n == p
    d, t = n - 1, 0
    while d % 2 == 0:
        d, t = d // 2, t + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(t - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _mix64(z):
    m = (1 << 64) - 1
    z = (z + 0x9E3779B97F4A7C15) & m
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9 & m
    z = (z ^ (z >> 27)) * 0x94D049BB133111EB & m
    return z ^ (z >> 31)


def _exact_range(lo, hi):
    """The range results by a plain numpy sieve (lo > 16)."""
    top = hi + 4096
    root = math.isqrt(top) + 1
    small = np.ones(root + 1, dtype=bool)
    small[:2] = False
    for q in range(2, math.isqrt(root) + 1):
        if small[q]:
            small[q * q:: q] = False
    f = np.ones(top - lo, dtype=bool)
    for q in np.flatnonzero(small).tolist():
        f[max(q * q, -(-lo // q) * q) - lo:: q] = False
    p = np.flatnonzero(f).astype(np.int64)
    n = int(np.searchsorted(p, hi - lo))
    gaps = np.diff(p)[:n]
    g = int(np.argmax(gaps))
    six = p[:n][np.all([f[p[:n] + o] for o in SEXTUPLET], axis=0)]
    cks = sum(_mix64(lo + int(x)) for x in six) & ((1 << 64) - 1)
    return np.array([n, int(f[p[:n] + 2].sum()), int(gaps[g]), lo + int(p[g]), len(six), cks, lo + int(p[0]),
                     lo + int(p[n - 1])], dtype=np.uint64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "range" and case["len"] <= 2**22 and case["lo"] <= 10**13:
        out = {"stats": _exact_range(*_window(case, seed))}
        if case["hash_log2"]:
            out["hashes"] = None
        return out
    if kind == "bpsw" and case["count"] <= 20000:
        n, _ = mp.bpsw_workload(seed, max(case["count"], 64), 1)
        return np.array([_is_prime(int(x)) for x in n[: case["count"]]])
    if kind == "fermat" and case["count"] <= 200000:
        return np.array([(pow(2, p - 1, p * p) - 1) // p for p in _fermat_primes(case, seed).tolist()],
                        dtype=np.uint64)
    return None
