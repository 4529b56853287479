"""The work that a program has this library do, as cases to be timed.

A case is a dict of plain values; its "kind" says which public call it goes
through:

* build     DeviceStructure.build of a resident text: wavelet matrix and/or
            levelwise tree, with or without rank/select and a follow-on batch
            of access, rank and select queries
* huffman   DeviceStructure.huffman of a resident text: code table, levels,
            rank/select, then queries
* batch     Batch.build of many independent texts, some results fetched
* query     access, rank and select batches against a resident structure
* serve     requests (build + query batch) through the server, all in flight
* compute   the drop-in wx_ps().compute: host text in, host structure out
* reduce    reduce_alphabet of a resident text

Sizes and distributions are those of the library's configured workloads and
tests, from the smallest served text to the largest benchmark text.
"""
import ctypes
import math

import numpy as np
import torch

import pwm_gb300 as pg

OPS = (("access", pg.Q_ACCESS), ("rank", pg.Q_RANK), ("select", pg.Q_SELECT))
NP = {1: np.uint8, 2: np.uint16, 4: np.uint32}
TORCH = {1: torch.uint8, 2: torch.int16, 4: torch.int32}
BATCH_STRIDE = 512  # a batch's program fetches one text in so many


def listed():
    return [
        # the smallest served texts: launches and host latency
        {"name": "build_u8_4k", "kind": "build", "n": 4099, "width": 1, "levels": 8, "dist": "zipf", "matrix": True,
         "tree": True, "rank_select": True, "queries": 1000},
        # an ordinary byte text, odd length, queried once built
        {"name": "build_u8_1m", "kind": "build", "n": 1000003, "width": 1, "levels": 8, "dist": "zipf", "matrix": True,
         "tree": True, "rank_select": True, "queries": 10000},
        # DNA-like bytes, the few-symbol alphabet
        {"name": "build_dna_2p26", "kind": "build", "n": 1 << 26, "width": 1, "levels": 2, "dist": "dna",
         "matrix": True, "tree": True, "rank_select": False, "queries": 0},
        # the headline: a 1 GiB byte text, both structures, rank/select
        {"name": "build_u8_1gib", "kind": "build", "n": 1 << 30, "width": 1, "levels": 8, "dist": "zipf",
         "matrix": True, "tree": True, "rank_select": True, "queries": 10000},
        # wide alphabet, 16 levels, both structures
        {"name": "build_u16_2p28", "kind": "build", "n": 1 << 28, "width": 2, "levels": 16, "dist": "mix",
         "matrix": True, "tree": True, "rank_select": False, "queries": 0},
        # 32-bit symbols over 2^20 values: a matrix alone, with rank/select
        {"name": "build_u32_2p26", "kind": "build", "n": 1 << 26, "width": 4, "levels": 20, "dist": "uniform",
         "matrix": True, "tree": False, "rank_select": True, "queries": 10000},
        # Huffman-shaped matrix of the wide text, code table included
        {"name": "huffman_u16_2p28", "kind": "huffman", "n": 1 << 28, "width": 2, "dist": "mix", "tree": False,
         "queries": 10000},
        # 4096 texts of uneven length and mixed alphabets in one batch
        {"name": "batch_4096", "kind": "batch", "texts": 4096},
        # large query batches against a resident 16-level matrix
        {"name": "query_u16_2p28", "kind": "query", "n": 1 << 28, "width": 2, "levels": 16, "dist": "mix",
         "tree": False, "queries": 1 << 22},
        # a burst of mixed requests on an eight-slot server
        {"name": "serve_64", "kind": "serve", "requests": 64, "queries": 10000},
        # the drop-in call from a program that knows nothing of the GPU
        {"name": "compute_u8_20m", "kind": "compute", "n": 20000003, "width": 1, "levels": 8, "dist": "zipf",
         "tree": True},
        # alphabet reduction, the step before a build of a raw text
        {"name": "reduce_u16_2p28", "kind": "reduce", "n": 1 << 28, "width": 2, "dist": "mix"},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _alphabet(rng):
    """Width, levels and distribution of a text, and its largest size here."""
    pick = rng.random()
    if pick < 0.15:
        return 1, 2, "dna", 1 << 26
    if pick < 0.45:
        return 1, 8, "zipf", 1 << 30
    if pick < 0.65:
        return 1, rng.randint(1, 8), "uniform", 1 << 30
    if pick < 0.85:
        return 2, 16, "mix", 1 << 28
    return 4, rng.randint(17, 20), "uniform", 1 << 26


def draw(rng):
    kind = rng.choice(["build", "build", "build", "build", "huffman", "huffman", "batch", "query", "query", "serve",
                       "compute", "reduce"])
    if kind == "batch":
        return {"kind": kind, "texts": _log_uniform(rng, 16, 4096)}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randint(8, 64), "queries": _log_uniform(rng, 100, 10000)}
    if kind == "huffman":
        width, dist, most = rng.choice([(1, "zipf", 1 << 28), (2, "mix", 1 << 28)])
        return {"kind": kind, "n": _log_uniform(rng, 1 << 12, most), "width": width, "dist": dist,
                "tree": rng.random() < 0.5, "queries": _log_uniform(rng, 100, 10000)}
    if kind == "reduce":
        width, dist, most = rng.choice([(1, "zipf", 1 << 29), (2, "mix", 1 << 28), (4, "uniform", 1 << 26)])
        return {"kind": kind, "n": _log_uniform(rng, 1 << 12, most), "width": width, "dist": dist}
    width, levels, dist, most = _alphabet(rng)
    if kind == "compute":
        return {"kind": kind, "n": _log_uniform(rng, 1 << 10, min(most, 1 << 26)), "width": width, "levels": levels,
                "dist": dist, "tree": rng.random() < 0.5}
    if kind == "query":
        return {"kind": kind, "n": _log_uniform(rng, 1 << 16, min(most, 1 << 28)), "width": width, "levels": levels,
                "dist": dist, "tree": rng.random() < 0.5, "queries": _log_uniform(rng, 1 << 10, 1 << 22)}
    shape = rng.choice([(True, False), (False, True), (True, True), (True, True)])
    rank_select = rng.random() < 0.6
    return {"kind": kind, "n": _log_uniform(rng, 1 << 10, most), "width": width, "levels": levels, "dist": dist,
            "matrix": shape[0], "tree": shape[1], "rank_select": rank_select,
            "queries": _log_uniform(rng, 100, 10000) if rank_select else 0}


def _device_text(case, seed):
    """The seeded text of a case, generated on the device."""
    n, width = case["n"], case["width"]
    t = torch.empty(n, dtype=TORCH[width], device="cuda")
    dist = {"zipf": pg.GEN_ZIPF256, "dna": pg.GEN_DNA4, "mix": pg.GEN_MIX16, "uniform": pg.GEN_UNIFORM}[case["dist"]]
    torch.cuda.synchronize()  # the library's stream is not torch's
    pg.generate(dist, seed, n, width, param=1 << case.get("levels", 20), device_ptr=t.data_ptr())
    pg.default_context().sync()
    return t


def _symbols(t):
    """The text's symbols as non-negative 64-bit numbers."""
    return t.to(torch.int64) & ((1 << (8 * t.element_size())) - 1)


def _operands(text, queries, seed):
    """Uniform positions, symbols taken from the text, occurrences uniform
    within each symbol's count; device arrays."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = text.numel()
    counts = torch.zeros(1, dtype=torch.int64, device="cuda")
    for i in range(0, n, 1 << 26):
        c = torch.bincount(_symbols(text[i:i + (1 << 26)]))
        if c.numel() > counts.numel():
            c[:counts.numel()] += counts
            counts = c
        else:
            counts[:c.numel()] += c
    pos = torch.randint(0, n, (queries,), device="cuda", generator=g)
    sym = _symbols(text[torch.randint(0, n, (queries,), device="cuda", generator=g)])
    share = torch.rand(queries, dtype=torch.float64, device="cuda", generator=g)
    occ = 1 + torch.minimum((share * counts[sym]).floor().to(torch.int64), counts[sym] - 1)
    out = [torch.empty(queries, dtype=torch.int64, device="cuda") for _ in OPS]
    return {"pos": pos, "sym": sym, "occ": occ, "out": out, "count": queries}


class _Words:
    """A structure's level array in device memory, for torch.as_tensor: the
    tensor keeps this object, and so the structure, alive."""

    def __init__(self, ds, which):
        v = ds.view(which)
        self.ds = ds
        self.__cuda_array_interface__ = {"shape": (int(v.total_words),), "typestr": "<i8",
                                         "data": (int(v.words), False), "version": 2}


def _words(ds, which):
    return torch.as_tensor(_Words(ds, which), device="cuda")


def _query(ds, which, q):
    n = q["count"]
    ds.query(which, pg.Q_ACCESS, q["pos"].data_ptr(), None, n, q["out"][0].data_ptr())
    ds.query(which, pg.Q_RANK, q["sym"].data_ptr(), q["pos"].data_ptr(), n, q["out"][1].data_ptr())
    ds.query(which, pg.Q_SELECT, q["sym"].data_ptr(), q["occ"].data_ptr(), n, q["out"][2].data_ptr())
    return q["out"]


def _batch_texts(count, seed):
    """Log-normal lengths (median 2^16, sigma 1.5, 2^10 to 2^24); 15% Zipf
    bytes with 8 levels, 85% DNA-like over {0..4} with 3 levels, symbol 4 in
    geometric runs of mean 50."""
    rng = np.random.default_rng(count)  # the lengths are the corpus's, the symbols the seed's
    lengths = np.clip(np.exp(rng.normal(math.log(65536.0), 1.5, count)), 1 << 10, 1 << 24).astype(np.int64)
    levels = np.where(rng.random(count) < 0.15, 8, 3).astype(np.uint32)
    offsets = np.zeros(count + 1, dtype=np.uint64)
    offsets[1:] = np.cumsum(lengths)
    total = int(offsets[-1])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    zipf = torch.cumsum(1.0 / torch.arange(1, 257, dtype=torch.float64, device="cuda"), 0)
    zipf = (zipf / zipf[-1]).to(torch.float32)
    perm = torch.randperm(256, device="cuda", generator=g).to(torch.uint8)
    dna = torch.tensor([0.29, 0.49, 0.69, 0.98], device="cuda") / 0.98
    start = 0.02 / (50.0 * 0.98 + 0.02)
    text = torch.empty(total, dtype=torch.uint8, device="cuda")
    ends = torch.from_numpy(offsets[1:].astype(np.int64)).cuda()
    byte_text = torch.from_numpy(levels == 8).cuda()
    for i in range(0, total, 1 << 26):
        m = min(1 << 26, total - i)
        u = torch.rand(m, device="cuda", generator=g)
        at = torch.arange(i, i + m, device="cuda")
        is_byte = byte_text[torch.searchsorted(ends, at, right=True)]
        z = perm[torch.searchsorted(zipf, u).clamp_(max=255)]
        d = torch.searchsorted(dna, u).clamp_(max=3).to(torch.uint8)
        v = torch.rand(m, device="cuda", generator=g)
        run = 1 + (torch.log(torch.rand(m, device="cuda", generator=g) + 1e-12) / math.log(0.98)).to(torch.int64)
        four = torch.cummax(torch.where(v < start, at + run, 0), 0).values > at
        text[i:i + m] = torch.where(is_byte, z, torch.where(four, 4, d).to(torch.uint8))
        del u, at, is_byte, z, d, v, run, four
    return text, offsets, levels


def _serve_requests(case, seed):
    """Host texts of the batch's law, every twentieth a 32-bit one over 2^20
    values, each with a mixed query batch on its matrix or its tree."""
    rng = np.random.default_rng(seed)
    zipf = np.cumsum(1.0 / np.arange(1, 257))
    zipf /= zipf[-1]
    perm = rng.permutation(256).astype(np.uint8)
    dna = np.cumsum([0.29, 0.2, 0.2, 0.29, 0.02])
    reqs = []
    for i in range(case["requests"]):
        n = int(np.clip(np.exp(rng.normal(math.log(65536.0), 1.5)), 1 << 10, 1 << 24))
        if i % 20 == 7:
            t, levels = rng.integers(0, 1 << 20, n).astype(np.uint32), 20
        elif rng.random() < 0.15:
            t, levels = perm[np.searchsorted(zipf, rng.random(n)).clip(max=255)], 8
        else:
            t, levels = np.searchsorted(dna, rng.random(n)).clip(max=4).astype(np.uint8), 3
        nq = case["queries"]
        ops = rng.integers(0, 3, nq).astype(np.uint8)
        sym = t[rng.integers(0, n, nq)].astype(np.int64)
        counts = np.bincount(t, minlength=1 << levels)[sym]
        occ = 1 + np.minimum(np.floor(rng.random(nq) * counts).astype(np.int64), counts - 1)
        a = np.where(ops == 0, rng.integers(0, n, nq), sym).astype(np.uint64)
        b = np.where(ops == 1, rng.integers(0, n + 1, nq), occ).astype(np.uint64)
        reqs.append((t, levels, ops, a, b, i % 2))
    return reqs


_server = None


def _the_server():
    """One server for the process, as a serving program has."""
    global _server
    if _server is None:
        _server = pg.Server(150 * 10 ** 9, slots=8)
    return _server


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "build":
        s["text"] = _device_text(case, seed)
        s["ds"] = pg.DeviceStructure(case["n"], case["width"], case["levels"], matrix=case["matrix"],
                                     tree=case["tree"], rank_select=case["rank_select"])
        s["which"] = [w for w in (0, 1) if case["tree" if w else "matrix"]]
        s["words"] = [_words(s["ds"], w) for w in s["which"]]
        if case["queries"]:
            s["q"] = _operands(s["text"], case["queries"], seed)
    elif kind == "huffman":
        s["text"] = _device_text(case, seed)
        # the program's own buffer for the levels: mean code lengths stay below 7 bits of a byte and 14 of a wide
        # symbol, and 64 levels end in at most 16 words of padding
        s["levels"] = torch.zeros(case["n"] * (7 if case["width"] == 1 else 14) // 64 + 1024, dtype=torch.int64,
                                  device="cuda")
        s["q"] = _operands(s["text"], case["queries"], seed)
    elif kind == "batch":
        s["text"], offsets, levels = _batch_texts(case["texts"], seed)
        s["batch"] = pg.Batch(offsets, levels, word_width=1, tree=True)
    elif kind == "query":
        text = _device_text(case, seed)
        s["ds"] = pg.DeviceStructure(case["n"], case["width"], case["levels"], matrix=not case["tree"],
                                     tree=case["tree"], rank_select=True)
        s["ds"].build(text.data_ptr())
        s["ds"].check()
        s["q"] = _operands(text, case["queries"], seed)
    elif kind == "serve":
        s["server"] = _the_server()
        s["requests"] = _serve_requests(case, seed)
    elif kind == "compute":
        s["text"] = _device_text(case, seed).cpu().numpy().view(NP[case["width"]])
        s["wx"] = pg.wx_ps(NP[case["width"]], case["tree"])
    else:
        s["text"] = _device_text(case, seed)
        s["out"] = torch.empty_like(s["text"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "build":
        s["ds"].build(s["text"].data_ptr())
        out = list(s["words"])
        if case["queries"]:
            out += _query(s["ds"], s["which"][-1], s["q"])
        return out
    if kind == "huffman":
        ds = pg.DeviceStructure.huffman(s["text"].data_ptr(), case["n"], case["width"], tree=case["tree"])
        which = 1 if case["tree"] else 0
        ds.check()  # torch's stream is not the library's
        words = _words(ds, which)
        s["levels"][:words.numel()].copy_(words)
        return [s["levels"], *_query(ds, which, s["q"])]
    if kind == "batch":
        s["batch"].build(s["text"].data_ptr())
        s["batch"].check()
        out = []
        for i in range(0, case["texts"], BATCH_STRIDE):
            for which in (0, 1):
                ws = s["batch"].download(i, which)
                out.append(ws.bvs().data.view(np.int64))
                if not which:
                    out.append(np.array(ws.zeros(), dtype=np.int64))
        return out
    if kind == "query":
        return _query(s["ds"], 1 if case["tree"] else 0, s["q"])
    if kind == "serve":
        srv = s["server"]
        sent = [srv.submit(t, levels, matrix=True, tree=True, which=which, ops=ops, a=a, b=b)
                for t, levels, ops, a, b, which in s["requests"]]
        out = []
        for rid, answers in sent:
            srv.wait(rid)
            srv.release(rid)
            out.append(answers)
        return np.concatenate(out).view(np.int64)
    if kind == "compute":
        ws = s["wx"].compute(s["text"], case["n"], case["levels"])
        return [ws.bvs().data.view(np.int64), np.array(ws.zeros(), dtype=np.int64)]
    most = pg.reduce_alphabet(s["text"].data_ptr(), case["n"], case["width"], s["out"].data_ptr())
    return [s["out"], most]


def exact(case, seed):
    """Every output is a bit vector, a count, a position or a symbol: whole
    numbers, equal or wrong, with no rounding to measure."""
    return None


def _level_bytes(n, levels, structures, rank_select):
    """Bytes of level bits and of their rank/select blocks and samples."""
    per = 8 * ((n + 63) // 64)
    if rank_select:
        per += 8 * (n // 2048 + 1) + 4 * (n // 8192 + 2)
    return structures * levels * per


def _query_bytes(queries, levels):
    """Operands in, answers out, and a 32-byte sector of a level for each
    position looked at: one a level for access, two for rank, one for select."""
    return queries * (8 + 8 + 16 + 8 + 16 + 8 + levels * 4 * 32)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # the law's mean length; 15% of the texts have 8 levels, the others 3
        n = case["texts"] * 65536.0 * math.exp(1.5 ** 2 / 2) * 0.93
        return {"bytes": n + n * 2 * (0.15 * 8 + 0.85 * 3) / 8, "flops": 0}
    if kind == "serve":
        n = case["requests"] * 65536.0 * math.exp(1.5 ** 2 / 2) * 0.93
        text = n * (0.05 * 4 + 0.95)
        bits = n * 2 * (0.05 * 20 + 0.95 * (0.15 * 8 + 0.85 * 3)) / 8
        return {"bytes": text + bits + case["requests"] * case["queries"] * (25 + 4 * 32), "flops": 0}
    n, width = case["n"], case["width"]
    if kind == "query":
        return {"bytes": _query_bytes(case["queries"], case["levels"]), "flops": 0}
    if kind == "compute":
        return {"bytes": n * width + _level_bytes(n, case["levels"], 1, False), "flops": 0}
    if kind == "reduce":
        return {"bytes": 2 * n * width, "flops": 0}
    if kind == "huffman":
        # mean code length of the two distributions
        bits = 6.1 if case["dist"] == "zipf" else 13.0
        return {"bytes": n * width + n * bits / 8 * (1 + 1.0 / 32) + _query_bytes(case["queries"], bits), "flops": 0}
    structures = int(case["matrix"]) + int(case["tree"])
    queries = _query_bytes(case["queries"], case["levels"]) if case["queries"] else 0
    return {"bytes": n * width + _level_bytes(n, case["levels"], structures, case["rank_select"]) + queries,
            "flops": 0}
