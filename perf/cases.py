"""Performance cases of the framework: what its users have it do, through the public Python API.

Three things are done with this framework: opening a transaction database (from a file's bytes
or from a CSR in host memory), mining it (maximal frequent itemsets, or every frequent itemset
level by level), and counting waves of prefix item lists against the vertical bitmap for a
search that lives elsewhere.  The sizes are those of the repository's five configurations
(tensorfim_b200/synth.py), of the level-wise shape (tensorfim_b200/levelwise.py) and of its
tests: 1 to thousands of prefixes per wave, 10,000 to 8.4 million transactions, tens to
thousands of items, dense categorical data and sparse long-tail data.

A case names a data source.  For databases the seed gives the item ids and the order of the
transactions (the mined sets are other sets, of the same number and lengths); for waves it
draws the bitmap and the lists.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tensorfim_b200 as tf

CUDA = "cuda"


def listed() -> list[dict]:
    return [
        # One search node counted by a caller's own search: the reference's per-node call on its
        # small dense configuration (10,000 transactions, 69 counted items).  Latency.
        {"name": "wave_node", "kind": "wave", "data": "dense", "nodes": 1, "items": 69, "tx": 10_000, "max_len": 4,
         "device": False},
        # A ragged wave over the base rows of the replicated configuration (271 counted items), from
        # host lists: the ordinary call of a caller that batches a few dozen nodes.
        {"name": "wave_ragged", "kind": "wave", "data": "dense", "nodes": 37, "items": 271, "tx": 49_001, "max_len": 6,
         "device": False},
        # A dense wave with every buffer on the device (the counting microbenchmark's shape).
        {"name": "wave_dense", "kind": "wave", "data": "dense", "nodes": 512, "items": 1024, "tx": 1 << 18, "max_len": 3,
         "device": True},
        # A wave over a long-tail bitmap: thousands of items of low support, prefixes of one or two
        # items drawn by their supports.
        {"name": "wave_longtail", "kind": "wave", "data": "longtail", "nodes": 300, "items": 6162, "tx": 1_000_000,
         "max_len": 2, "device": True},
        # The largest wave: a level of 2,048 prefixes at the level-wise prototype's size.
        {"name": "wave_level", "kind": "wave", "data": "dense", "nodes": 2048, "items": 512, "tx": 1 << 23, "max_len": 4,
         "device": True},
        # Small dense categorical mine with the default options: launches and latency.
        {"name": "mine_dense_10k", "kind": "mine", "data": "dirichlet", "rows": 10_000, "replicas": 1, "minsup": 0.10,
         "lookahead": "filtered", "graphs": False},
        # Two million dense rows at a high threshold (the learned proposal's evaluation database).
        {"name": "mine_dense_2m", "kind": "mine", "data": "dominant", "rows": 2_000_000, "replicas": 1, "minsup": 0.70,
         "lookahead": "learned", "graphs": False},
        # The dense replicated configuration at half its rows, minsup 6%: tens of thousands of MFIs,
        # the benchmark's workload.
        {"name": "mine_replicated", "kind": "mine", "data": "zipf", "rows": 49_000, "replicas": 128, "minsup": 0.06,
         "lookahead": "learned", "graphs": False},
        # The sparse long-tail configuration: a million rows over 40,000 items.
        {"name": "mine_longtail", "kind": "mine", "data": "longtail", "rows": 1_000_000, "replicas": 1, "minsup": 0.0005,
         "lookahead": "learned", "graphs": False},
        # Every frequent itemset of the level-wise prototype's database.
        {"name": "mine_all", "kind": "mine_all", "tx": 1 << 23, "items": 512, "patterns": 80, "minsup": 0.0015},
        # A whole session from a transaction file's bytes, as the command line runs it: parse,
        # ingest, mine, results, close.
        {"name": "session_text", "kind": "session", "data": "longtail", "rows": 300_007, "replicas": 1, "minsup": 0.001,
         "lookahead": "learned"},
        # A dense database opened from a CSR in pinned memory, its item tables read, closed.
        {"name": "open_csr", "kind": "open", "data": "zipf", "rows": 49_000, "replicas": 16, "minsup": 0.06},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["wave", "wave", "wave", "mine", "mine", "mine", "mine_all", "session", "open"])
    if kind == "wave":
        while True:
            data = rng.choice(["dense", "dense", "longtail"])
            tx = _log(rng, 5_000, 1 << 23)
            nodes = _log(rng, 1, 2048)
            items = _log(rng, 16, 1024) if data == "dense" else _log(rng, 512, 6162)
            if nodes * items * tx <= 2048 * 512 << 23 and items * tx <= 6162 * 1_000_000 and nodes * tx <= 2048 << 23:
                break
        return {"kind": "wave", "data": data, "nodes": nodes, "items": items, "tx": tx, "max_len": rng.randint(1, 6),
                "device": nodes * items > 1 << 14 or rng.random() < 0.5}
    if kind == "mine_all":
        return {"kind": "mine_all", "tx": _log(rng, 100_000, 1 << 23), "items": rng.randint(64, 512),
                "patterns": rng.randint(16, 80), "minsup": round(rng.uniform(0.0015, 0.004), 5)}
    data = rng.choice(["dirichlet", "majority", "dominant", "zipf", "longtail"])
    rows, lo, hi, digits = {"dirichlet": (_log(rng, 5_000, 100_000), 0.09, 0.15, 3),
                            "majority": (_log(rng, 7_000, 700_000), 0.80, 0.92, 3),
                            "dominant": (_log(rng, 20_000, 2_000_000), 0.66, 0.80, 3),
                            "zipf": (49_000, 0.06, 0.12, 3),
                            "longtail": (_log(rng, 100_000, 1_000_000), 0.0005, 0.002, 5)}[data]
    reps = _log(rng, 1, 128) if data == "zipf" and kind == "mine" else _log(rng, 1, 16) if data == "zipf" else 1
    if kind != "mine":
        rows = min(rows, 300_007)
    case = {"kind": kind, "data": data, "rows": rows, "replicas": reps, "minsup": round(rng.uniform(lo, hi), digits)}
    if data == "longtail":
        case["minsup"] = max(case["minsup"], round(200 / rows, 5))
    if kind != "open":
        case["lookahead"] = rng.choice(["learned", "filtered"])
    if kind == "mine":
        case["graphs"] = rng.random() < 0.25
    return case


# ------------------------------------------------------------------------------ populations
def _rng(seed) -> np.random.Generator:
    return np.random.Generator(np.random.PCG64(seed))


def _groups(data: str) -> list[np.ndarray]:
    """The attribute groups' value probabilities of a categorical population."""
    if data == "dirichlet":       # 23 groups x 5 values
        rng = _rng(0)
        return [rng.dirichlet(np.full(5, 0.5)) for _ in range(23)]
    if data == "zipf":            # 74 groups of 2-60 values, Zipf(1.3) within each
        rng = _rng(2)
        sizes = rng.integers(2, 61, size=74)
        while abs(int(sizes.sum()) - 2100) > 40:
            sizes = rng.integers(2, 61, size=74)
        out = []
        for k in sizes:
            w = np.arange(1, int(k) + 1, dtype=np.float64) ** -1.3
            out.append(w[rng.permutation(int(k))] / w.sum())
        return out
    # one dominant value per group, the rest split evenly
    rng = _rng(1 if data == "majority" else 4)
    lo, hi = (0.65, 0.95) if data == "majority" else (0.55, 0.90)
    sizes = np.full(43, 3) if data == "majority" else rng.integers(2, 16, size=60)
    out = []
    for k in sizes:
        dom = rng.uniform(lo, hi)
        p = np.full(int(k), (1.0 - dom) / (int(k) - 1))
        p[int(rng.integers(int(k)))] = dom
        out.append(p)
    return out


def _source() -> torch.Generator:
    return torch.Generator(CUDA).manual_seed(11)


def _shuffled(n: int, gen: torch.Generator) -> torch.Tensor:
    return torch.randperm(n, device=CUDA, generator=gen)


def _categorical(case: dict, seed: torch.Generator) -> tuple[torch.Tensor, torch.Tensor]:
    """Rows with one value per group; `replicas` exact copies.  (offsets, items) on the GPU."""
    gen = _source()
    groups = _groups(case["data"])
    n, reps, g = case["rows"], case["replicas"], len(groups)
    cols = torch.empty(n, g, dtype=torch.int32, device=CUDA)
    first = 0
    for k, p in enumerate(groups):
        cdf = torch.tensor(np.cumsum(p)[:-1], device=CUDA)
        u = torch.rand(n, dtype=torch.float64, device=CUDA, generator=gen)
        cols[:, k] = torch.searchsorted(cdf, u, right=True).to(torch.int32) + first
        first += len(p)
    ids = _shuffled(first, seed).to(torch.int32) + 1
    cols = ids[cols[_shuffled(n, seed)].long()].sort(1).values
    items = cols.reshape(-1).repeat(reps)
    return torch.arange(0, (n * reps + 1) * g, g, dtype=torch.int64, device=CUDA), items


def _longtail(case: dict, seed: torch.Generator) -> tuple[torch.Tensor, torch.Tensor]:
    """Poisson(10) + 1 items per row over 40,000: 70% from 2,000 patterns whose items are each
    dropped half of the time, the rest Zipf(1.1).  (offsets, items) on the GPU."""
    rng, gen = _rng(3), _source()
    n, n_items, n_pat = case["rows"], 40_000, 2_000
    lens = rng.poisson(6, n_pat) + 2
    pats = np.zeros((n_pat, int(lens.max())), dtype=np.int64)
    for k, m in enumerate(lens):
        pats[k, :m] = rng.choice(n_items, int(m), replace=False) + 1
    pat_cdf = torch.tensor(np.cumsum(rng.exponential(1.0, n_pat)), device=CUDA)
    zipf = np.arange(1, n_items + 1, dtype=np.float64) ** -1.1
    zipf_cdf = torch.tensor(np.cumsum(zipf) / zipf.sum(), device=CUDA)
    ranked = torch.tensor(rng.permutation(n_items) + 1, device=CUDA)
    pats = torch.tensor(pats, device=CUDA)

    length = torch.poisson(torch.full((n,), 10.0, device=CUDA), generator=gen).long() + 1
    quota = torch.round(0.7 * length).long()
    u = torch.rand(n, 3, dtype=torch.float64, device=CUDA, generator=gen) * pat_cdf[-1]
    drawn = pats[torch.searchsorted(pat_cdf, u, right=True).clamp_(max=n_pat - 1)].reshape(n, -1)
    keep = (drawn > 0) & (torch.rand(drawn.shape, device=CUDA, generator=gen) < 0.5)
    keep &= keep.cumsum(1) <= quota[:, None]
    row = torch.arange(n, device=CUDA)
    rest = (length - keep.sum(1)).clamp_(min=0)
    rest_rows = torch.repeat_interleave(row, rest)
    v = torch.rand(rest_rows.numel(), dtype=torch.float64, device=CUDA, generator=gen)
    rest_items = ranked[torch.searchsorted(zipf_cdf, v, right=True).clamp_(max=n_items - 1)]
    ids, row = _shuffled(n_items, seed) + 1, _shuffled(n, seed)
    key = torch.cat([(row[:, None] * 65536 + ids[drawn - 1])[keep], row[rest_rows] * 65536 + ids[rest_items - 1]]).unique()
    offsets = torch.zeros(n + 1, dtype=torch.int64, device=CUDA)
    offsets[1:] = torch.bincount(key >> 16, minlength=n).cumsum(0)
    return offsets, (key & 65535).to(torch.int32)


def _csr(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    gen = torch.Generator(CUDA).manual_seed(seed)
    # the rows come from the case alone; `gen` gives them their order and ids
    return _longtail(case, gen) if case["data"] == "longtail" else _categorical(case, gen)


def _pinned(t: torch.Tensor) -> np.ndarray:
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def _text(offsets: torch.Tensor, items: torch.Tensor) -> np.ndarray:
    """The transaction file's bytes: ids separated by a space, one row per line."""
    v = items.long()
    digits = torch.ones_like(v)
    for k in range(1, 7):
        digits += v >= 10 ** k
    end = (digits + 1).cumsum(0)
    out = torch.full((int(end[-1]),), 32, dtype=torch.uint8, device=CUDA)
    for k in range(int(digits.max())):
        m = digits > k
        out[end[m] - 2 - k] = (48 + v[m] // 10 ** k % 10).to(torch.uint8)
    out[end[offsets[1:] - 1] - 1] = 10
    return out.cpu().numpy()


def _bit_rows(on: torch.Tensor) -> torch.Tensor:
    """(rows, tx) booleans -> (rows, words) int32, bit t % 32 of word t // 32 = transaction t."""
    pad = torch.nn.functional.pad(on, (0, -on.shape[1] % 32)).view(on.shape[0], -1, 32)
    return (pad.long() << torch.arange(32, device=CUDA)).sum(2).to(torch.int32)


def _planted(case: dict, seed: int) -> torch.Tensor:
    """Patterns of 2-6 items that fire in 0.2-1.5% of the transactions, noise of 0.02% per item."""
    rng, gen = _rng(0), _source()
    n, d = case["tx"], case["items"]
    rows = torch.zeros(d, (n + 31) // 32, dtype=torch.int32, device=CUDA)
    for _ in range(case["patterns"]):
        its = rng.choice(d, size=int(rng.integers(2, 7)), replace=False)
        fire = torch.rand(1, n, device=CUDA, generator=gen) < (0.2 + 1.3 * rng.random()) / 100
        rows[torch.tensor(its, device=CUDA)] |= _bit_rows(fire)
    for e in range(d):
        rows[e] |= _bit_rows(torch.rand(1, n, device=CUDA, generator=gen) < 0.0002)[0]
    return rows[_shuffled(d, torch.Generator(CUDA).manual_seed(seed))]


def _longtail_supports(d: int) -> np.ndarray:
    return np.maximum(0.1 * np.arange(1, d + 1, dtype=np.float64) ** -0.9, 0.0005)


def _wave_bitmap(case: dict, seed: int) -> torch.Tensor:
    """Items x transactions as bits.  dense: supports of 1/16 to 15/16; longtail: Zipf supports
    from a tenth of the transactions down to 0.05%."""
    n, d = case["tx"], case["items"]
    gen = torch.Generator(CUDA).manual_seed(seed)
    words = (n + 31) // 32
    if case["data"] == "dense":
        p16 = torch.tensor(_rng(5).integers(1, 16, size=(d, 1)), device=CUDA)
        rows = torch.zeros(d, words, dtype=torch.int32, device=CUDA)
        for bit in range(4):      # binary expansion of p16 / 16, one random word per digit
            r = torch.randint(-2 ** 31, 2 ** 31, (d, words), dtype=torch.int32, device=CUDA, generator=gen)
            rows = torch.where((p16 >> bit & 1).bool(), rows | r, rows & r)
        if n % 32:
            rows[:, -1] &= (1 << n % 32) - 1
        return rows
    per = torch.tensor(np.maximum(1, _longtail_supports(d) * n).astype(np.int64), device=CUDA)
    item = torch.repeat_interleave(torch.arange(d, device=CUDA), per)
    t = torch.randint(0, n, (item.numel(),), device=CUDA, generator=gen)
    key = (item * (words * 32) + t).unique()
    flat = torch.zeros(d * words, dtype=torch.int64, device=CUDA)
    flat.index_add_(0, key >> 5, torch.ones_like(key) << (key & 31))
    return flat.view(d, words).to(torch.int32)


def _wave_lists(case: dict, seed: int) -> list[list[int]]:
    rng = _rng([seed, 1])
    d = case["items"]
    w = _longtail_supports(d) if case["data"] == "longtail" else np.ones(d)
    w /= w.sum()
    return [sorted(int(x) for x in rng.choice(d, size=min(d, int(rng.integers(1, case["max_len"] + 1))), replace=False, p=w))
            for _ in range(case["nodes"])]


def _min_count(case: dict) -> int:
    return max(1, case["tx"] // (50 if case["data"] == "dense" else 2000))


# ------------------------------------------------------------------------------ the interface
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "wave":
        rows = _wave_bitmap(case, seed).cpu().numpy().view(np.uint32)
        st["db"] = tf.Database.from_bitmap(rows, case["tx"], case["items"])
        st["lists"] = _wave_lists(case, seed)
        st["min_count"] = _min_count(case)
        if case["device"]:
            off = np.concatenate([[0], np.cumsum([len(x) for x in st["lists"]])])
            st["d_off"] = torch.tensor(off, dtype=torch.int64, device=CUDA)
            st["d_items"] = torch.tensor([x for l in st["lists"] for x in l], dtype=torch.int32, device=CUDA)
            st["counts"] = torch.zeros(case["nodes"], case["items"], dtype=torch.int32, device=CUDA)
            st["nfreq"] = torch.zeros(case["nodes"], dtype=torch.int32, device=CUDA)
            torch.cuda.synchronize()
    elif kind == "mine_all":
        rows = _planted(case, seed).cpu().numpy().view(np.uint32)
        st["db"] = tf.Database.from_bitmap(rows, case["tx"], case["items"])
    else:
        offsets, items = _csr(case, seed)
        if kind == "session":
            st["text"] = _text(offsets, items)
        else:
            st["offsets"], st["items"] = _pinned(offsets), _pinned(items)
        if kind == "mine":
            st["db"] = tf.Database.from_csr(st.pop("offsets"), st.pop("items"), case["minsup"])
    return st


def _mfis(r) -> dict:
    return {"items": r.items, "offsets": r.offsets, "supports": r.supports}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "wave":
        db = state["db"]
        if not case["device"]:
            return db.count_wave(state["lists"], state["min_count"])
        db.count_wave_device(state["d_items"].data_ptr(), state["d_off"].data_ptr(), case["nodes"], case["max_len"],
                             state["min_count"], state["counts"].data_ptr(), state["nfreq"].data_ptr())
        return state["counts"], state["nfreq"]
    if kind == "mine":
        return _mfis(state["db"].mine(lookahead=case["lookahead"], graphs=case["graphs"]))
    if kind == "mine_all":
        return _mfis(state["db"].mine_all(min_count=max(1, int(case["tx"] * case["minsup"]))))
    if kind == "session":
        with tf.Database.from_text(state["text"], case["minsup"]) as db:
            return _mfis(db.mine(lookahead=case["lookahead"]))
    with tf.Database.from_csr(state["offsets"], state["items"], case["minsup"]) as db:
        return {"ids": db.dense_to_orig(), "freq": db.dense_freq(), "rows": db.info["trans_num_reduced"],
                "roots": db.info["dimension_reduced"], "min_count": db.info["min_count"]}


def work(case: dict) -> dict:
    """One pass's least bytes and operations (a support over N transactions: N multiply-adds)."""
    if case["kind"] in ("wave", "mine_all"):
        d, row = case["items"], case["tx"] / 8
        if case["kind"] == "mine_all":
            return {"bytes": d * row, "flops": 0.0}
        b = case["nodes"]
        return {"bytes": d * row + 4.0 * b * d, "flops": 2.0 * b * d * case["tx"]}
    n = case["rows"] * case["replicas"]
    if case["data"] == "longtail":
        held = 4.0 * 11 * n                                   # the transactions' items
        text = 5.7 * 11 * n
    else:
        groups = _groups(case["data"])
        frequent = sum(int((p >= case["minsup"]).sum()) for p in groups)
        held = frequent * n / 8 if case["kind"] == "mine" else 4.0 * len(groups) * n   # bitmap rows, or the CSR
        text = 4.5 * len(groups) * n
    return {"bytes": text if case["kind"] == "session" else held, "flops": 0.0}


# ------------------------------------------------------------------------------ exact values
def _count_exact(rows: torch.Tensor, lists: list[list[int]], n: int) -> torch.Tensor:
    d = rows.shape[0]
    member = torch.zeros(len(lists), d, dtype=torch.float64, device=CUDA)
    for i, l in enumerate(lists):
        member[i, l] = 1.0
    need = member.sum(1, keepdim=True)
    counts = torch.zeros(len(lists), d, dtype=torch.float64, device=CUDA)
    step = max(1, (1 << 26) // max(d, len(lists)) // 32)
    for w in range(0, rows.shape[1], step):
        bits = (rows[:, w:w + step, None] >> torch.arange(32, device=CUDA, dtype=torch.int32) & 1).reshape(d, -1).double()
        counts += (member @ bits == need).double() @ bits.T
    return counts.long()


def _maximal_exact(offsets: np.ndarray, items: np.ndarray, minsup: float) -> dict:
    """The maximal frequent itemsets of a small database, by depth-first search over Python
    integers as bit rows: descending support, then descending item lists."""
    n = len(offsets) - 1
    row_of = np.repeat(np.arange(n), np.diff(offsets))
    bits = {}
    for e in np.unique(items):
        on = np.zeros(n, dtype=np.uint8)
        on[row_of[items == e]] = 1
        if on.sum() >= n * minsup:
            bits[int(e)] = int.from_bytes(np.packbits(on).tobytes(), "big")
    need = n * minsup
    found = []

    def grow(head, mask, tail):
        for k, e in enumerate(tail):
            m = mask & bits[e]
            rest = [x for x in tail[k + 1:] if (m & bits[x]).bit_count() >= need]
            if rest:
                grow(head + [e], m, rest)
            elif all(x in head or x == e or (m & bits[x]).bit_count() < need for x in bits):
                found.append((m.bit_count(), tuple(sorted(head + [e], reverse=True))))

    grow([], (1 << (-(-n // 8) * 8)) - 1, sorted(bits))
    found.sort(key=lambda f: (f[0], f[1]), reverse=True)
    lens = [len(f[1]) for f in found]
    return {"items": np.array([x for f in found for x in f[1]], dtype=np.int32),
            "offsets": np.concatenate([[0], np.cumsum(lens)]).astype(np.int64),
            "supports": np.array([f[0] for f in found], dtype=np.int32)}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "wave":
        counts = _count_exact(_wave_bitmap(case, seed), _wave_lists(case, seed), case["tx"])
        return counts, (counts >= _min_count(case)).sum(1)
    if kind == "mine" and case["data"] == "dirichlet" and case["rows"] <= 20_000:
        offsets, items = _csr(case, seed)
        return _maximal_exact(offsets.cpu().numpy(), items.cpu().numpy(), case["minsup"])
    if kind == "open":
        offsets, items = _csr(case, seed)
        n = offsets.numel() - 1
        f = torch.bincount(items.long()).cpu().numpy()
        ids = np.flatnonzero(f >= n * case["minsup"])
        held = torch.tensor(f >= n * case["minsup"], device=CUDA)[items.long()]
        rows = torch.zeros(n, dtype=torch.int64, device=CUDA)
        rows.index_add_(0, torch.repeat_interleave(torch.arange(n, device=CUDA), offsets.diff()), held.long())
        return {"ids": ids.astype(np.int32), "freq": f[ids].astype(np.int32), "rows": int((rows > 0).sum()),
                "roots": int((f / n > case["minsup"]).sum()), "min_count": math.ceil(n * case["minsup"])}
    return None
