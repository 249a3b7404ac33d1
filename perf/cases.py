"""
Performance cases of the executor: whole queries and tasks as a GPU service
runs them through the public entry points (pg-strom_b200/xpu_b200.py, the
binding of include/xpu_b200.h).

A pass of a query opens its session, runs the outer chunks, takes the final
groups and closes the session, because a session serves one query; what
outlives the query in a service (resident chunks, response buffers, cached
dimension tables) is made by prepare().  Tables have the shapes and value
distributions of the benchmark configurations
(pg-strom_b200/producer/xb_configs.py) and are made on the GPU from the seed:
heap pages and Arrow buffers are written there byte for byte as the chunk
producers write them.

Families (a case's "family") and what they stand for:

  scan        heap scan + filter + GROUP BY g: count, sum(int), sum(numeric),
              avg(float8 with NULLs)
  nogroup     the same scan under an aggregate without GROUP BY
  wide        the same scan under every partial-state form of kds_final
  text        GROUP BY a text column of the scanned table, varlenas and
              numerics in every on-disk form
  join        two-way hash join + GROUP BY a dimension's text column
  arrow       Arrow columns, GROUP BY a high-cardinality int8 key, the groups
              handed on as hash parts in device memory (multi-GPU exchange)
  topn        the same with NULLs in the columns, ORDER BY sum DESC LIMIT n
  projection  scan whose rows go into a device kds_dst
  served      many small scan queries at once through Submit / Poll
"""
import ctypes
import math
import os
import struct
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _sub in ("pg-strom_b200", os.path.join("pg-strom_b200", "producer")):
    _p = os.path.join(ROOT, _sub)
    if _p not in sys.path:
        sys.path.insert(0, _p)

import xb_configs as C  # noqa: E402
import xpu_b200  # noqa: E402
from xb_producer import (BLCKSZ, Agg, BoolOp, Column, Const, Func, SessionBuilder, Table, Var,  # noqa: E402
                         encode_text_from_dict, kern_multirels, maxalign, numeric_typmod)

PAGE_ROOM = BLCKSZ - 24             # a heap page without its header
CHUNK_PAGES = 8190                  # pages of a 64 MB chunk
ARROW_CHUNK_ROWS = 2_500_000        # rows of an Arrow chunk (record batch)
SCAN_ROW = 68                       # heap bytes of a scan row: tuple and line pointer
JOIN_ROW = 52                       # heap bytes of a fact row
TEXT_WORDS = 150
DAY0, DAY_LO, DAY_HI = 16436, 17532, 18262      # Unix days: 2015-01-01, 2018-01-01, 2020-01-01


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one 64 KB chunk, the smallest chunk command: launches and host calls count
        {"name": "scan_64kb", "family": "scan", "rows": 913, "groups": 64, "limit": 300, "parts": 0},
        # the plain scan configuration, five resident 64 MB chunks
        {"name": "scan_4m", "family": "scan", "rows": 4_000_000, "groups": 64, "limit": 300, "parts": 0},
        # an aggregate over a whole table, without GROUP BY
        {"name": "nogroup_20m", "family": "nogroup", "rows": 20_000_003, "limit": 700},
        # a report query: statistics of every kind, 3000 groups
        {"name": "wide_2m", "family": "wide", "rows": 2_000_000, "groups": 3000, "limit": 600},
        # text keys and numerics read from the scanned rows
        {"name": "text_1m", "family": "text", "rows": 1_000_001, "limit": 700},
        # the drop-in path: one 64 MB chunk and the dimension tables come from pinned host memory
        {"name": "join_host_64mb", "family": "join", "rows": 1_250_000, "dim1": 200_000, "dim2": 10_000,
         "stride": 1, "copies": 1, "miss": 0.0, "host": True, "cached": False},
        # sparse keys, two dimension rows per key, facts without a match: the hashed probe
        {"name": "join_sparse_10m", "family": "join", "rows": 10_000_000, "dim1": 100_000, "dim2": 5_000,
         "stride": 37, "copies": 2, "miss": 0.2, "host": False, "cached": False},
        # the headline: 100M resident fact rows, dimension tables cached across queries
        {"name": "join_100m", "family": "join", "rows": 100_000_000, "dim1": 200_000, "dim2": 10_000,
         "stride": 1, "copies": 1, "miss": 0.0, "host": False, "cached": True},
        # the 1000 largest of some millions of groups, NULLs in the columns
        {"name": "topn_20m", "family": "topn", "rows": 20_000_000, "keys": 2_000_000, "nulls": 0.1, "limit": 1000},
        # the high-cardinality configuration, its groups split for eight GPUs
        {"name": "arrow_500m", "family": "arrow", "rows": 500_000_000, "keys": 10_000_000, "parts": 8},
        # rows of a filtered scan returned to the executor
        {"name": "projection_4m", "family": "projection", "rows": 4_000_000, "limit": 300},
        # small queries of many clients: chunk sizes, selectivities and group counts of the mixed batch
        {"name": "served_24", "family": "served", "commands": 24, "rows_lo": 960, "rows_hi": 980_000,
         "groups_hi": 16_000, "mix": 1},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fam = rng.choice(["scan", "scan", "nogroup", "wide", "text", "join", "join", "arrow", "topn", "projection",
                      "served"])
    if fam == "scan":
        groups = _log_uniform(rng, 1, 1_000_000)
        return {"family": fam, "rows": _log_uniform(rng, 900, 20_000_000), "groups": groups,
                "limit": rng.randint(1, 900), "parts": 0 if groups <= 16_000 else rng.choice([1, 2, 4, 8])}
    if fam == "nogroup":
        return {"family": fam, "rows": _log_uniform(rng, 900, 40_000_000), "limit": rng.randint(1, 1000)}
    if fam == "wide":
        return {"family": fam, "rows": _log_uniform(rng, 900, 8_000_000), "groups": _log_uniform(rng, 1, 12_000),
                "limit": rng.randint(1, 1000)}
    if fam == "text":
        return {"family": fam, "rows": _log_uniform(rng, 900, 2_000_000), "limit": rng.randint(1, 1000)}
    if fam == "join":
        host = rng.random() < 0.25
        return {"family": fam, "rows": _log_uniform(rng, 10_000, 1_250_000 if host else 100_000_000),
                "dim1": _log_uniform(rng, 1_000, 400_000), "dim2": _log_uniform(rng, 100, 20_000),
                "stride": rng.choice([1, 1, 37]), "copies": rng.choice([1, 1, 2]),
                "miss": rng.choice([0.0, 0.0, 0.2]), "host": host, "cached": rng.random() < 0.5}
    if fam == "arrow":
        rows = _log_uniform(rng, 1_000_000, 400_000_000)
        return {"family": fam, "rows": rows, "keys": _log_uniform(rng, 20_000, min(rows, 10_000_000)),
                "parts": rng.choice([1, 2, 4, 8])}
    if fam == "topn":
        rows = _log_uniform(rng, 100_000, 60_000_000)
        return {"family": fam, "rows": rows, "keys": _log_uniform(rng, 10_000, min(rows, 4_000_000)),
                "nulls": rng.choice([0.0, 0.1, 0.3]), "limit": rng.choice([10, 100, 1000])}
    if fam == "projection":
        return {"family": fam, "rows": _log_uniform(rng, 900, 8_000_000), "limit": rng.randint(1, 600)}
    return {"family": fam, "commands": rng.randint(2, 32), "rows_lo": 960, "rows_hi": _log_uniform(rng, 50_000, 980_000),
            "groups_hi": _log_uniform(rng, 64, 16_000), "mix": rng.randint(2, 1 << 20)}


def _topn_keep(case):
    return min(case["limit"], case["keys"])


def _served_commands(case):
    """(rows, selectivity limit, groups) of each served query: log-uniform
    sizes and group counts, uniform selectivity."""
    r = np.random.default_rng(case["mix"])
    return [(int(np.exp(r.uniform(math.log(case["rows_lo"]), math.log(case["rows_hi"])))), int(r.integers(1, 901)),
             int(np.exp(r.uniform(0.0, math.log(case["groups_hi"])))))
            for _ in range(case["commands"])]


def work(case):
    """The chunk bytes and the result bytes of one pass."""
    fam = case["family"]
    if fam == "scan":
        nbytes = case["rows"] * SCAN_ROW + min(case["groups"], case["rows"]) * 128
    elif fam == "nogroup":
        nbytes = case["rows"] * SCAN_ROW + 256
    elif fam == "wide":
        nbytes = case["rows"] * SCAN_ROW + min(case["groups"], case["rows"]) * 320
    elif fam == "text":
        nbytes = case["rows"] * 228 + TEXT_WORDS * 300
    elif fam == "join":
        nbytes = case["rows"] * JOIN_ROW + (0 if case["cached"] else
                                            case["dim1"] * case["copies"] * 80 + case["dim2"] * 64) + 25 * 100
    elif fam == "arrow":
        nbytes = case["rows"] * 24 + case["keys"] * 160
    elif fam == "topn":
        nbytes = case["rows"] * (24.375 if case["nulls"] else 24) + case["keys"] * 112 + _topn_keep(case) * 160
    elif fam == "projection":
        nbytes = case["rows"] * SCAN_ROW + case["rows"] * case["limit"] / 1000 * 72
    else:
        nbytes = sum(n * SCAN_ROW + min(g, n) * 128 for n, _, g in _served_commands(case))
    return {"bytes": float(nbytes), "flops": 0.0}


# ---------------------------------------------------------------------------
# columns from the seed
# ---------------------------------------------------------------------------
class _Rand:
    """Seeded draws on the device; one generator per state."""

    def __init__(self, seed, device):
        self.d = device
        self.g = torch.Generator(device=device)
        self.g.manual_seed(0x5EED0000 + int(seed))

    def ints(self, lo, hi, n, dtype):
        """lo .. hi - 1"""
        return torch.randint(lo, hi, (n,), generator=self.g, device=self.d, dtype=dtype)

    def uniform(self, n):
        return torch.rand(n, generator=self.g, device=self.d, dtype=torch.float64)

    def normal(self, n):
        return torch.randn(n, generator=self.g, device=self.d, dtype=torch.float64)


def _scan_columns(r, n, groups):
    return {"a": r.ints(0, 1000, n, torch.int32), "b": r.normal(n), "bnull": r.uniform(n) < 0.05,
            "c": r.ints(0, 1_000_000, n, torch.int64), "g": r.ints(0, groups, n, torch.int32)}


def _text_columns(r, n):
    return {"t": r.ints(0, TEXT_WORDS, n, torch.int64), "n": r.ints(-10 ** 12, 10 ** 12, n, torch.int64),
            "nnull": r.uniform(n) < 0.03, "form": r.ints(0, 3, n, torch.int64), "v": r.ints(0, 1000, n, torch.int32)}


def _text_words():
    return [w.encode() for w in C.long_strings(TEXT_WORDS, seed=C.SEED_BASE + 6)]


def _join_dims(case, seed):
    """The dimension tables (host arrays): keys, region codes and flags."""
    r = np.random.default_rng([int(seed), 77])
    pk1 = np.tile(np.arange(1, case["dim1"] + 1, dtype=np.int64) * case["stride"], case["copies"]).astype(np.int32)
    pk2 = (np.arange(1, case["dim2"] + 1, dtype=np.int64) * case["stride"]).astype(np.int32)
    return {"pk1": pk1, "region": r.integers(0, len(C.REGIONS), len(pk1)), "pk2": pk2,
            "flag": r.integers(0, 5, case["dim2"]).astype(np.int16)}


def _fact_columns(r, case):
    n, n1, n2 = case["rows"], case["dim1"], case["dim2"]
    i1 = r.ints(0, n1, n, torch.int32)
    w = 1.0 / torch.arange(1, n2 + 1, device=r.d, dtype=torch.float64) ** 1.1       # bounded Zipf
    cdf = torch.cumsum(w, 0)
    i2 = torch.searchsorted(cdf / cdf[-1], r.uniform(n), right=True, out_int32=True).clamp_(max=n2 - 1)
    qty = r.ints(1, 51, n, torch.int32)
    price = r.ints(100, 1_000_001, n, torch.int64)
    miss = r.uniform(n) < case["miss"] if case["miss"] else None
    return {"i1": i1, "i2": i2, "qty": qty, "price": price, "miss": miss}


def _arrow_columns(r, n, keys, nulls):
    """One chunk's columns; with nulls, validity masks of v1, v2 and d."""
    c = {"k": r.ints(0, keys, n, torch.int64), "v1": r.ints(-1_000_000, 1_000_001, n, torch.int32),
         "v2": torch.exp(r.normal(n)), "d": r.ints(DAY0, DAY0 + 3652, n, torch.int32)}
    for col in ("v1", "v2", "d"):
        c[col + "_ok"] = r.uniform(n) >= nulls if nulls else None
    return c


def _arrow_chunk_sizes(rows):
    return [min(ARROW_CHUNK_ROWS, rows - at) for at in range(0, rows, ARROW_CHUNK_ROWS)]


# ---------------------------------------------------------------------------
# heap pages on the device
# ---------------------------------------------------------------------------
def _bytes_of(x):
    """[n, width] bytes of a fixed-width column"""
    return x.contiguous().view(torch.uint8).view(x.numel(), x.element_size())


def _numeric_varlena(unscaled, scale, form=None):
    """(bytes [n, w], length [n]) of numerics with |value| < 10^8: the short
    format, or where form is given 0 = short, 1 = long, 2 = long under a
    4-byte varlena header (encode_numeric, xb_producer.py)."""
    dev, n = unscaled.device, unscaled.numel()
    a = unscaled.abs() * 10 ** (4 - scale)
    groups = torch.stack([a // 100_000_000, a // 10_000 % 10_000, a % 10_000], 1)
    nz = groups != 0
    some = nz.any(1)
    first = torch.where(some, nz.int().argmax(1), 0)
    last = torch.where(some, 2 - nz.flip(1).int().argmax(1), -1)
    ndig = torch.where(some, last - first + 1, 0)
    weight = torch.where(some, 1 - first, 0)
    neg = (unscaled < 0) & some
    zeros = torch.zeros(n, 2, dtype=torch.int64, device=dev)
    digits = torch.gather(torch.cat([groups, zeros], 1), 1, first[:, None] + torch.arange(3, device=dev))
    digits = torch.where(torch.arange(3, device=dev) < ndig[:, None], digits, 0).to(torch.int16)
    short = (0x8000 | (neg.long() << 13) | (scale << 7) | (weight & 0x7F))
    width = 9 if form is None else 14
    out = torch.zeros(n, width, dtype=torch.uint8, device=dev)
    dig = _bytes_of(digits.view(-1)).view(n, 6)

    def lay(rows, at, head_words):
        for j, w in enumerate(head_words):
            out[rows, at + 2 * j] = (w[rows] & 0xFF).to(torch.uint8)
            out[rows, at + 2 * j + 1] = (w[rows] >> 8 & 0xFF).to(torch.uint8)
        out[rows, at + 2 * len(head_words):at + 2 * len(head_words) + 6] = dig[rows]

    if form is None:
        length = 3 + 2 * ndig
        out[:, 0] = (length << 1 | 1).to(torch.uint8)
        lay(slice(None), 1, [short])
        return out, length
    long_head = (neg.long() << 14) | scale
    length = torch.where(form == 0, 3, torch.where(form == 1, 5, 8)) + 2 * ndig
    for f in range(3):
        rows = (form == f).nonzero().view(-1)
        if f < 2:
            out[rows, 0] = (length[rows] << 1 | 1).to(torch.uint8)
        else:
            out[rows, 0] = (length[rows] << 2 & 0xFF).to(torch.uint8)   # a 4-byte header, below 64 bytes
        lay(rows, 4 if f == 2 else 1, [short] if f == 0 else [long_head, weight & 0xFFFF])
    return out, length


def _word_varlena(codes, words, device):
    """(bytes [n, w], length [n]) of dictionary strings, 1- or 4-byte header"""
    imgs = [bytes([(len(w) + 1) << 1 | 1]) + w if len(w) <= 126 else struct.pack("<I", (len(w) + 4) << 2) + w
            for w in words]
    tab = np.zeros((len(imgs), max(map(len, imgs))), dtype=np.uint8)
    for i, x in enumerate(imgs):
        tab[i, :len(x)] = np.frombuffer(x, dtype=np.uint8)
    lens = torch.tensor([len(x) for x in imgs], device=device)
    return torch.from_numpy(tab).to(device)[codes], lens[codes]


def _tuples(cols, n, blk0, per_page):
    """Heap tuples of n rows as ([n, w] bytes, [n] lengths).  A column is
    (bytes [n, w], lengths or None, alignment, NULL mask or None); rows lie
    per_page to a page, the first page being block blk0."""
    dev = cols[0][0].device
    ncols = len(cols)
    width = maxalign(24 + sum(b.shape[1] + a - 1 for b, _, a, _ in cols))
    rows = torch.arange(n, device=dev)
    uniform = all(ln is None and nm is None for _, ln, _, nm in cols)
    img = torch.zeros(n if uniform else n + 1, width, dtype=torch.uint8, device=dev)
    hasnull = torch.zeros(n, dtype=torch.bool, device=dev)
    bitmap = torch.zeros(n, dtype=torch.int64, device=dev)
    off = 24 if uniform else torch.full((n,), 24, dtype=torch.int64, device=dev)
    for j, (b, ln, al, nm) in enumerate(cols):
        if uniform:
            off = (off + al - 1) // al * al
            img[:, off:off + b.shape[1]] = b
            off += b.shape[1]
            continue
        up = (off + al - 1) // al * al
        at = up if ln is None else torch.where(b[:, 0] & 1 == 1, off, up)
        size = b.shape[1] if ln is None else ln
        base = rows * width + at
        if nm is not None:
            hasnull |= nm
            base = torch.where(nm, n * width, base)         # a NULL's bytes go to a spare row
            bitmap |= (~nm).long() << j
            off = torch.where(nm, off, at + size)
        else:
            bitmap |= 1 << j
            off = at + size
        img.view(-1)[(base[:, None] + torch.arange(b.shape[1], device=dev)).view(-1)] = b.reshape(-1)
    length = torch.full((n,), off, dtype=torch.int64, device=dev) if uniform else off
    img = img[:n]
    blk = rows // per_page + blk0
    mask = 0x0B00 | (0 if uniform else 0x0002)
    head = torch.zeros(n, 12, dtype=torch.int16, device=dev)
    head[:, 0] = 2                                          # xmin
    head[:, 6] = (blk >> 16).to(torch.int16)
    head[:, 7] = (blk & 0xFFFF).to(torch.int16)
    head[:, 8] = (rows % per_page + 1).to(torch.int16)
    head[:, 9] = ncols
    head[:, 10] = (mask | hasnull.long()).to(torch.int16)
    head[:, 11] = (24 | torch.where(hasnull, bitmap, 0) << 8).to(torch.int16)
    img[:, :24] = head.view(torch.uint8)
    return img, length, uniform


def _fill_pages(pages, img, length, uniform, per_page):
    """Tuples into pages ([p, 8192] bytes, zeroed): line pointers upwards
    from the header, tuples downwards from the end."""
    dev, np_, n = img.device, pages.shape[0], img.shape[0]
    full = np_ * per_page
    if full > n:
        img = torch.cat([img, img.new_zeros(full - n, img.shape[1])])
        length = torch.cat([length, length.new_zeros(full - n)])
    size = (length + 7 & ~7).view(np_, per_page)
    off = BLCKSZ - torch.cumsum(size, 1)
    if uniform:
        w = int((int(length[0]) + 7) // 8 * 8)
        pages[:, BLCKSZ - per_page * w:] = img[:, :w].reshape(np_, per_page, w).flip(1).reshape(np_, -1)
    else:
        words = img.shape[1] // 8
        k = torch.arange(words, device=dev)
        at = torch.arange(np_, device=dev)[:, None] * (BLCKSZ // 8) + off // 8
        live = (k < (size.view(-1, 1) // 8)).view(-1)
        dst = (at.view(-1, 1) + k).view(-1)[live]
        pages.view(-1).view(torch.int64)[dst] = img.contiguous().view(torch.int64).view(-1)[live]
    used = (length > 0).view(np_, per_page)
    lp = torch.where(used, off | 1 << 15 | length.view(np_, per_page) << 17, 0)
    pages[:, 24:24 + 4 * per_page] = lp.to(torch.int32).view(torch.uint8).view(np_, -1)
    head = torch.zeros(np_, 12, dtype=torch.int16, device=dev)
    head[:, 5] = 4                                          # PD_ALL_VISIBLE
    head[:, 6] = (24 + 4 * used.sum(1)).to(torch.int16)
    head[:, 7] = torch.where(used, off, BLCKSZ).min(1).values.to(torch.int16)
    head[:, 8] = BLCKSZ
    head[:, 9] = BLCKSZ | 4
    pages[:, :24] = head.view(torch.uint8)


class _Chunks:
    """KDS chunks of one table, resident on the device: their addresses
    (heap pages 16-byte aligned) and the memory that holds them."""

    def __init__(self):
        self.mem, self.addr, self.nbytes = [], [], []

    def add(self, length, pages_at, device):
        shift = -pages_at % 16
        t = torch.zeros(length + shift + 64, dtype=torch.uint8, device=device)
        t = t[shift:shift + length]
        self.mem.append(t)
        self.addr.append(t.data_ptr())
        self.nbytes.append(length)
        return t


def _heap_chunks(table, make_cols, n, per_page, device):
    """KDS_FORMAT_BLOCK chunks of a table of n rows; make_cols(lo, hi) gives
    the columns of its rows lo..hi-1."""
    head = table.kds_header("b")
    out = _Chunks()
    blk = 0
    for lo in range(0, n, per_page * CHUNK_PAGES):
        hi = min(n, lo + per_page * CHUNK_PAGES)
        np_ = -(-(hi - lo) // per_page)
        at = len(head) + maxalign(4 * np_)
        buf = out.add(at + BLCKSZ * np_, at, device)
        h = bytearray(head)
        struct.pack_into("<Q", h, 0, len(buf))
        struct.pack_into("<I", h, 16, np_)
        struct.pack_into("<II", h, 44, at, 0)
        buf[:len(h)] = torch.frombuffer(h, dtype=torch.uint8).to(device)
        buf[len(h):len(h) + 4 * np_] = torch.arange(blk, blk + np_, device=device, dtype=torch.int32).view(torch.uint8)
        img, length, uniform = _tuples(make_cols(lo, hi), hi - lo, blk, per_page)
        pages = torch.zeros(np_, BLCKSZ, dtype=torch.uint8, device=device)
        _fill_pages(pages, img, length, uniform, per_page)
        buf[at:] = pages.view(-1)
        blk += np_
    return out


def _rows_per_page(sizes):
    """The most rows a page can be given so that the rows, in order, fit
    every page; sizes are the rows' MAXALIGNed tuple sizes."""
    per = max(1, int(PAGE_ROOM / (4 + float(sizes.double().mean()))))
    while per > 1:
        pad = torch.cat([sizes, sizes.new_zeros(-sizes.numel() % per)]).view(-1, per)
        if int(pad.sum(1).max()) + 4 * per <= PAGE_ROOM:
            break
        per -= 1
    return per


def _scan_chunks(c, n, device):
    table = Table("t0", [Column("id", "int8"), Column("a", "int4"), Column("b", "float8"),
                         Column("c", "numeric", numeric_typmod(12, 2)), Column("g", "int4")], n)

    def cols(lo, hi):
        s = slice(lo, hi)
        num, ln = _numeric_varlena(c["c"][s], 2)
        return [(_bytes_of(torch.arange(lo, hi, device=device)), None, 8, None), (_bytes_of(c["a"][s]), None, 4, None),
                (_bytes_of(c["b"][s]), None, 8, c["bnull"][s]), (num, ln, 4, None), (_bytes_of(c["g"][s]), None, 4, None)]
    return _heap_chunks(table, cols, n, PAGE_ROOM // SCAN_ROW, device)


def _text_chunks(c, n, device):
    table = Table("t6", [Column("id", "int8"), Column("t", "text"), Column("n", "numeric", numeric_typmod(18, 4)),
                         Column("v", "int4")], n)
    words = _text_words()

    def cols(lo, hi):
        s = slice(lo, hi)
        txt, tl = _word_varlena(c["t"][s], words, device)
        num, nl = _numeric_varlena(c["n"][s], 4, c["form"][s])
        return [(_bytes_of(torch.arange(lo, hi, device=device)), None, 8, None), (txt, tl, 4, None),
                (num, nl, 4, c["nnull"][s]), (_bytes_of(c["v"][s]), None, 4, None)]
    sizes = torch.cat([_tuples(cols(lo, min(n, lo + 200_000)), min(n, lo + 200_000) - lo, 0, 1)[1] + 7 & ~7
                       for lo in range(0, n, 200_000)])
    return _heap_chunks(table, cols, n, _rows_per_page(sizes), device)


def _fact_chunks(c, case, device):
    table = Table("fact", [Column("fk1", "int4"), Column("fk2", "int4"), Column("qty", "int4"),
                           Column("price", "int8")], case["rows"])
    stride, n1 = case["stride"], case["dim1"]

    def cols(lo, hi):
        s = slice(lo, hi)
        k1 = c["i1"][s] + 1
        if c["miss"] is not None:
            k1 = torch.where(c["miss"][s], k1 + n1, k1)     # beyond every dimension key
        return [(_bytes_of((k * stride).to(torch.int32)), None, 4, None) for k in (k1, c["i2"][s] + 1)] + \
               [(_bytes_of(c["qty"][s]), None, 4, None), (_bytes_of(c["price"][s]), None, 8, None)]
    return _heap_chunks(table, cols, case["rows"], PAGE_ROOM // JOIN_ROW, device)


_ARROW_TYPES = [("k", "int8"), ("v1", "int4"), ("v2", "float8"), ("d", "date")]
_arrow_heads = {}


def _arrow_head(n, nulls):
    """(header bytes, length, {column: (validity, values) offsets}) of an
    Arrow chunk of n rows, laid out by the chunk producer."""
    if (n, nulls) not in _arrow_heads:
        ok = np.zeros((n + 7) // 8, dtype=np.uint8) if nulls else None
        cols = {"k": {"tag": 2, "bitwidth": 64, "values": np.zeros(n, np.int64)},
                "v1": {"tag": 2, "bitwidth": 32, "values": np.zeros(n, np.int32), "validity": ok},
                "v2": {"tag": 3, "precision": 2, "values": np.zeros(n), "validity": ok},
                "d": {"tag": 8, "unit": 0, "values": np.zeros(n, np.int32), "validity": ok}}
        table = Table("t2", [Column(nm, ty) for nm, ty in _ARROW_TYPES], n)
        buf = table.arrow_kds(cols)
        at = {nm: struct.unpack_from("<Q8xQ", buf, 72 + 168 * j + 120) for j, (nm, _) in enumerate(_ARROW_TYPES)}
        _arrow_heads[(n, nulls)] = (bytes(buf[:len(table.kds_header("a", n))]), len(buf), at)
    return _arrow_heads[(n, nulls)]


def _pack_bits(ok):
    n = ok.numel()
    x = torch.cat([ok, ok.new_zeros(-n % 8)]).view(-1, 8).to(torch.uint8)
    return (x << torch.arange(8, device=x.device, dtype=torch.uint8)).sum(1, dtype=torch.uint8)


def _arrow_chunks(r, case, device):
    nulls = case.get("nulls", 0.0)
    out = _Chunks()
    for n in _arrow_chunk_sizes(case["rows"]):
        head, length, at = _arrow_head(n, bool(nulls))
        c = _arrow_columns(r, n, case["keys"], nulls)
        buf = out.add(length, 0, device)
        buf[:len(head)] = torch.frombuffer(bytearray(head), dtype=torch.uint8).to(device)
        for nm, _ in _ARROW_TYPES:
            v = c[nm].view(torch.uint8)
            buf[at[nm][1]:at[nm][1] + v.numel()] = v
            if nm != "k" and nulls:
                bits = _pack_bits(c[nm + "_ok"])
                buf[at[nm][0]:at[nm][0] + bits.numel()] = bits
    return out


# ---------------------------------------------------------------------------
# sessions and their result columns
# ---------------------------------------------------------------------------
# words of a partial state in a kds_final tuple: h = varlena header and
# flags, i = integer, f = float8
_FIELDS = {"NROWS_ANY": "i", "NROWS_COND": "i", "PMIN_INT32": "hi", "PMAX_INT64": "hi", "PMIN_FP64": "hf",
           "PMAX_FP64": "hf", "PSUM_INT": "hii", "PSUM_INT64": "hiii", "PSUM_FP": "hif", "PAVG_FP": "hif",
           "PSUM_NUMERIC": "hiii", "PAVG_NUMERIC": "hiii", "STDDEV": "hiff", "COVAR": "hifffff"}
_AGGS = {"scan": [("nrows", "NROWS_ANY"), ("sum_a", "PSUM_INT"), ("sum_c", "PSUM_NUMERIC"), ("avg_b", "PAVG_FP")],
         "nogroup": [("nrows", "NROWS_ANY"), ("nb", "NROWS_COND"), ("sum_a", "PSUM_INT"), ("sum_c", "PSUM_NUMERIC"),
                     ("avg_b", "PAVG_FP"), ("min_b", "PMIN_FP64"), ("max_b", "PMAX_FP64")],
         "wide": [("nrows", "NROWS_ANY"), ("nb", "NROWS_COND"), ("min_a", "PMIN_INT32"), ("max_a", "PMAX_INT64"),
                  ("min_b", "PMIN_FP64"), ("max_b", "PMAX_FP64"), ("sum_b", "PSUM_FP"), ("avg_c", "PAVG_NUMERIC"),
                  ("sd_b", "STDDEV"), ("cov", "COVAR")],
         "text": [("nrows", "NROWS_ANY"), ("nn", "NROWS_COND"), ("sum_n", "PSUM_NUMERIC"), ("avg_n", "PAVG_NUMERIC"),
                  ("sum_v", "PSUM_INT")],
         "join": [("amount", "PSUM_INT64"), ("nrows", "NROWS_ANY")],
         "arrow": [("nrows", "NROWS_ANY"), ("sum_v1", "PSUM_INT"), ("min_v2", "PMIN_FP64"), ("max_v2", "PMAX_FP64"),
                   ("sum_v2", "PSUM_FP")]}
_AGGS["topn"] = _AGGS["arrow"]
_AGGS["served"] = _AGGS["scan"]


def _topn_session(case):
    """The Arrow query ORDER BY sum(v2) DESC, k LIMIT n."""
    vk, vv1, vv2, vd = Var(0, 1, "int8"), Var(0, 2, "int4"), Var(0, 3, "float8"), Var(0, 4, "date")
    lo, hi = DAY_LO - C.UNIX_TO_PG_DAYS, DAY_HI - C.UNIX_TO_PG_DAYS
    return SessionBuilder(0, C.DEVTASK_PREAGG | C.DEVKIND_GPU).build(
        scan_quals=BoolOp("And", [Func("date_ge", [vd, Const("date", lo)], "bool"),
                                  Func("date_lt", [vd, Const("date", hi)], "bool")]),
        groupby_keys=[vk],
        aggs=[Agg("NROWS_ANY"), Agg("PSUM_INT", Func("int4_to_int8", [vv1], "int8")),
              Agg("PMIN_FP64", vv2), Agg("PMAX_FP64", vv2), Agg("PSUM_FP", vv2)],
        ngroups_estimate=float(case["keys"]),
        sort_keys=[("PSUM_FP64", 5, False, False), ("VREF", 6, True, False)], sort_limit=case["limit"])


def _projection_session(limit):
    typmod = numeric_typmod(12, 2)
    vid, va, vb, vc, vg = (Var(0, 1, "int8"), Var(0, 2, "int4"), Var(0, 3, "float8"), Var(0, 4, "numeric", typmod),
                           Var(0, 5, "int4"))
    return SessionBuilder(0, C.DEVTASK_SCAN | C.DEVKIND_GPU).build(
        scan_quals=Func("int4lt", [va, Const("int4", limit)], "bool"),
        projection=[vid, va, vb, vc, Func("int4pl", [Func("int4mul", [va, Const("int4", 2)], "int4"), vg], "int4")])


def _state_words(aggs):
    """(name, kind, word of the tuple) of every field, and the key's word."""
    at = maxalign(15 + (len(aggs) + 1 + 7) // 8) // 8
    out = []
    for name, action in aggs:
        for j, kind in enumerate(_FIELDS[action]):
            out.append(("%s.%d" % (name, j), kind, at))
            at += 1
    return out, at


class _Final:
    """A kds_final (int64 words, numpy or torch) as an executor reads it."""

    def __init__(self, words, head):
        length, _, nitems, _ = struct.unpack_from("<QQII", head, 0)
        nslots, = struct.unpack_from("<I", head, 40)
        ncolmeta, = struct.unpack_from("<I", head, 68)
        row0 = maxalign(72 + 168 * ncolmeta) // 8 + nslots
        self.w, self.n = words, nitems
        self.t = (length - words[row0:row0 + nitems]) >> 3

    def field(self, kind, at):
        v = self.w[self.t + at]
        return v if kind != "f" else v.view(torch.float64 if isinstance(v, torch.Tensor) else np.float64)


def _np_empty(kind, n):
    return np.zeros(n, dtype=np.float64 if kind == "f" else np.int64)


def _by_key(final, aggs, ngroups, key_of=None):
    """Every field as an array over the dense domain of an int4 key, or of
    the codes that key_of reads."""
    fields, key_at = _state_words(aggs)
    if final is None:
        return {name: _np_empty(kind, ngroups) for name, kind, _ in fields}
    k = key_of(final, key_at) if key_of else final.w[final.t + key_at] & 0xFFFFFFFF
    out = {}
    for name, kind, at in fields:
        out[name] = _np_empty(kind, ngroups)
        out[name][k] = final.field(kind, at)
    return out


def _word_key(index):
    """key -> code reader of a text key column (4-byte varlena header)."""
    def read(final, key_at):
        b = final.w.view(np.uint8)
        codes = np.empty(final.n, dtype=np.int64)
        for i, t in enumerate((final.t + key_at) * 8):
            ln = (int(b[t]) | int(b[t + 1]) << 8) >> 2
            codes[i] = index[bytes(b[t + 4:t + ln])]
        return codes
    return read


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
_dev = None


def _device():
    """The GPU's one executor, as a service holds it."""
    global _dev
    if _dev is None:
        _dev = xpu_b200.Device(0)
    return _dev


def _pinned(nbytes):
    return torch.empty((nbytes + 7) // 8, dtype=torch.int64, pin_memory=True).numpy().view(np.uint8)


def _final_bytes(ngroups, tuple_bytes):
    return (1 << 20) + ngroups * (3 * 8 + 16 + tuple_bytes)


def tables(case, seed, device):
    """The outer chunks and the session(s) of a case."""
    fam = case["family"]
    r = _Rand(seed, device)
    if fam in ("scan", "nogroup", "wide", "projection"):
        c = _scan_columns(r, case["rows"], case.get("groups", 64))
        session = {"scan": lambda: C.scan_groupby_session(case["limit"], case["groups"]),
                   "nogroup": lambda: C.scan_nogroup_session(case["limit"]),
                   "wide": lambda: C.wide_groupby_session(case["limit"], case["groups"]),
                   "projection": lambda: _projection_session(case["limit"])}[fam]()
        return {"chunks": _scan_chunks(c, case["rows"], device), "session": session}
    if fam == "text":
        return {"chunks": _text_chunks(_text_columns(r, case["rows"]), case["rows"], device),
                "session": C.long_varlena_session(case["limit"], TEXT_WORDS)}
    if fam == "join":
        d = _join_dims(case, seed)
        dim1 = Table("dim1", [Column("pk", "int4", values=d["pk1"]),
                              Column("region", "text", values=encode_text_from_dict(d["region"], C.REGIONS))],
                     len(d["pk1"]))
        dim2 = Table("dim2", [Column("pk", "int4", values=d["pk2"]), Column("flag", "int2", values=d["flag"])],
                     len(d["pk2"]))
        km = kern_multirels([dim1.hash_kds(C.host_join_hash_int4(d["pk1"])),
                             dim2.hash_kds(C.host_join_hash_int4(d["pk2"]))])
        # one handle names one set of dimension tables
        handle = 0
        if case["cached"]:
            handle = (int(seed) * 2654435761 ^ case["dim1"] * 40503 ^ case["dim2"] * 9176 ^ case["stride"] << 8 ^
                      case["copies"]) & 0x7FFFFFFF | 1
        return {"chunks": _fact_chunks(_fact_columns(r, case), case, device),
                "session": C.join_groupby_session(3, inner_handle=handle), "kmrels": km}
    if fam == "arrow":
        return {"chunks": _arrow_chunks(r, case, device),
                "session": C.arrow_groupby_session(DAY_LO, DAY_HI, float(case["keys"]))}
    if fam == "topn":
        return {"chunks": _arrow_chunks(r, case, device), "session": _topn_session(case)}
    queries = []
    for n, limit, groups in _served_commands(case):
        queries.append({"chunks": _scan_chunks(_scan_columns(r, n, groups), n, device),
                        "session": C.scan_groupby_session(limit, groups), "groups": groups})
    return {"queries": queries}


def prepare(case, seed):
    fam = case["family"]
    st = tables(case, seed, torch.device("cuda", 0))
    st["case"], st["dev"], st["nrels"] = case, _device(), 2 if fam == "join" else 0
    if fam == "join":
        km = _pinned(st["kmrels"].nbytes)[:st["kmrels"].nbytes]
        km[:] = st["kmrels"]
        st["kmrels"] = km
        st["key_of"] = _word_key({w.encode(): i for i, w in enumerate(C.REGIONS)})
        if case["host"]:
            host = [_pinned(t.numel())[:t.numel()] for t in st["chunks"].mem]
            for h, t in zip(host, st["chunks"].mem):
                h[:] = t.cpu().numpy()
            st["host"], st["chunks"] = host, None
        st["out"] = _pinned(_final_bytes(len(C.REGIONS), 200))
    elif fam == "text":
        st["key_of"] = _word_key({w: i for i, w in enumerate(_text_words())})
        st["out"] = _pinned(_final_bytes(TEXT_WORDS, 500))
    elif fam == "projection":
        st["dst_bytes"] = (1 << 16) + 96 * case["rows"]
        st["dst"] = torch.empty((st["dst_bytes"] + 128) // 8, dtype=torch.int64, device="cuda")
        st["masks"] = torch.tensor([(1 << 8 * i) - 1 if i < 8 else -1 for i in range(9)], device="cuda")
    elif fam == "served":
        for q in st["queries"]:
            q["out"] = _pinned(_final_bytes(q["groups"], 128))
    elif case.get("parts"):
        groups = case["keys"] if fam == "arrow" else case["groups"]
        st["part_bytes"] = case["parts"] * _final_bytes(0, 0) + _final_bytes(min(groups, case["rows"]), 144)
        st["part_buf"] = torch.empty(st["part_bytes"] // 8 + 1, dtype=torch.int64, device="cuda")
    else:
        groups = {"nogroup": 1, "topn": case.get("limit", 0)}.get(fam, case.get("groups"))
        st["out"] = _pinned(_final_bytes(groups, 320))
    st["done"] = torch.cuda.Event()
    st["done"].record()
    torch.cuda.synchronize()
    return st


def _execute(st, s):
    """The query's chunks through its session: one task, or a batch."""
    if st.get("host"):
        for h in st["host"]:
            s.exec(h)
    elif len(st["chunks"].addr) == 1:
        s.exec(st["chunks"].addr[0], on_device=True)
    else:
        b = s.batch(st["chunks"].addr)
        try:
            b.exec()
        finally:
            b.close()


def _host_final(s, out):
    buf, _ = s.final(out=out)
    return None if buf is None else _Final(buf[:len(buf) // 8 * 8].view(np.int64), bytes(buf[:72]))


def _parts_by_key(st, offs):
    """The device-resident parts, read there into arrays over the keys."""
    case = st["case"]
    arrow = case["family"] == "arrow"
    ngroups = case["keys"] if arrow else case["groups"]
    fields, key_at = _state_words(_AGGS[case["family"]])
    words = st["part_buf"]
    heads = torch.stack([words[o // 8:o // 8 + 9] for o in offs[:-1]]).cpu().numpy()
    out = {name: torch.zeros(ngroups, dtype=torch.float64 if kind == "f" else torch.int64, device="cuda")
           for name, kind, _ in fields}
    for o, head in zip(offs, heads):
        f = _Final(words[o // 8:], head.tobytes())
        k = f.w[f.t + key_at]
        if not arrow:
            k = k & 0xFFFFFFFF
        for name, kind, at in fields:
            out[name][k] = f.field(kind, at)
    return out


def _run_projection(st):
    """The projected rows as 64-byte tuple images (the row id, which depends
    on the order in which rows found their place, cut off) by id."""
    st["done"].synchronize()
    dst, nbytes = st["dst"], st["dst_bytes"]
    s = xpu_b200.Session(st["dev"], st["session"])
    out = torch.zeros(st["case"]["rows"], 8, dtype=torch.int64, device="cuda")
    step = nbytes // len(st["chunks"].addr) & ~7
    try:
        for i, addr in enumerate(st["chunks"].addr):
            res, req, e = xpu_b200.results_buffer(0), ctypes.c_uint64(), xpu_b200.KernErrorbuf()
            rc = xpu_b200.lib().xpuB200ExecTaskDst(s.h, ctypes.c_void_p(addr), 1,
                                                   ctypes.c_void_p(dst.data_ptr() + i * step), step, 1,
                                                   ctypes.byref(req), ctypes.c_void_p(res.ctypes.data),
                                                   ctypes.byref(e))
            if rc:
                raise xpu_b200.XpuB200Error(rc, e)
            n = xpu_b200.parse_results(res)["nitems_out"]
            w = dst[i * step // 8:]
            row0 = maxalign(72 + 168 * 5) // 8
            t = (step - w[row0:row0 + n]) >> 3
            img = w[t[:, None] + torch.arange(8, device="cuda")]
            nb = (img[:, :1] & 0xFFFFFFFF) - 4
            img &= st["masks"][(nb - 8 * torch.arange(8, device="cuda")).clamp_(0, 8)]
            out[img[:, 2]] = img
    finally:
        s.close()
    st["done"].record()
    return {"rows": out}


def _run_served(st):
    """All clients' queries in flight together: every chunk submitted, then
    each query finished as its ticket is done."""
    dev = st["dev"]
    open_, got = [], []
    try:
        for q in st["queries"]:
            s = xpu_b200.Session(dev, q["session"])
            open_.append(s)
            q["tickets"] = [dev.submit(s, a, on_device=True) for a in q["chunks"].addr]
        for q, s in zip(st["queries"], open_):
            for t in q["tickets"]:
                dev.poll(t)
            got.append(_by_key(_host_final(s, q["out"]), _AGGS["served"], q["groups"]))
    finally:
        for s in open_:
            s.close()
    return {name: np.concatenate([g[name] for g in got]) for name in got[0]}


def run(state):
    case = state["case"]
    fam = case["family"]
    if fam == "projection":
        return _run_projection(state)
    if fam == "served":
        return _run_served(state)
    s = xpu_b200.Session(state["dev"], state["session"], state.get("kmrels"), state["nrels"])
    try:
        if case.get("parts"):
            state["done"].synchronize()         # the last pass's groups have been read
            _execute(state, s)
            out = _parts_by_key(state, s.final_parts(case["parts"], state["part_buf"].data_ptr(), state["part_bytes"]))
            state["done"].record()
            return out
        _execute(state, s)
        final = _host_final(s, state["out"])
    finally:
        s.close()
    aggs = _AGGS[fam]
    if fam == "nogroup":
        return {name: _np_empty(kind, 1) if final is None or final.n == 0 else final.field(kind, at)
                for name, kind, at in _state_words(aggs)[0]}
    if fam == "topn":
        fields, key_at = _state_words(aggs)
        out = {name: final.field(kind, at) for name, kind, at in fields}
        out["key"] = final.field("i", key_at)
        return out
    ngroups = {"join": len(C.REGIONS), "text": TEXT_WORDS}.get(fam, case.get("groups"))
    return _by_key(final, aggs, ngroups, state.get("key_of"))


# ---------------------------------------------------------------------------
# the results from the columns, in 64 bits
# ---------------------------------------------------------------------------
def _sum(ngroups, g, x):
    return torch.zeros(ngroups, dtype=x.dtype, device=x.device).index_add_(0, g, x)


def _extreme(ngroups, g, x, how):
    init = {"amin": float("inf"), "amax": float("-inf")}[how]
    return torch.full((ngroups,), init, dtype=x.dtype, device=x.device).scatter_reduce_(0, g, x, how)


_DBL_MAX = 1.7976931348623157e308


def _minmax_fp(out, name, ngroups, g, x, nrows):
    """min and max of float8: groups without a value hold DBL_MAX (min) or
    -DBL_MAX (max), absent groups 0."""
    for nm, how, empty in (("min_" + name, "amin", _DBL_MAX), ("max_" + name, "amax", -_DBL_MAX)):
        m = _extreme(ngroups, g, x, how)
        m = torch.where(torch.isinf(m), torch.full_like(m, empty), m)
        out[nm + ".0"] = None
        out[nm + ".1"] = torch.where(nrows > 0, m, torch.zeros_like(m))


def _sums128(out, name, n, s):
    out[name + ".0"], out[name + ".1"], out[name + ".2"], out[name + ".3"] = None, n, s, s >> 63


def _scan_exact(c, limit, ngroups, fam):
    dev = c["a"].device
    m = (c["a"] < limit).nonzero().view(-1)
    g = c["g"][m].long() if fam != "nogroup" else torch.zeros(m.numel(), dtype=torch.int64, device=dev)
    a, b, cc, notnull = c["a"][m].long(), c["b"][m], c["c"][m], ~c["bnull"][m]
    gb, b, ab = g[notnull], b[notnull], a[notnull].double()
    nrows = _sum(ngroups, g, torch.ones_like(g))
    nb = _sum(ngroups, gb, torch.ones_like(gb))
    sb = _sum(ngroups, gb, b)
    out = {"nrows.0": nrows}
    if fam != "scan":
        out["nb.0"] = nb
    if fam == "wide":
        lo = torch.full((ngroups,), 1 << 40, device=dev).scatter_reduce_(0, g, a, "amin")
        hi = torch.full((ngroups,), -1, device=dev).scatter_reduce_(0, g, a, "amax")
        for nm, v in (("min_a", lo), ("max_a", hi)):
            out[nm + ".0"], out[nm + ".1"] = None, torch.where(nrows > 0, v, 0)
        _minmax_fp(out, "b", ngroups, gb, b, nrows)
        out["sum_b.0"], out["sum_b.1"], out["sum_b.2"] = None, nb, sb
        _sums128(out, "avg_c", nrows, _sum(ngroups, g, cc))
        sxx = _sum(ngroups, gb, b * b)
        out.update({"sd_b.0": None, "sd_b.1": nb, "sd_b.2": sb, "sd_b.3": sxx})
        out.update({"cov.0": None, "cov.1": nb, "cov.2": sb, "cov.3": sxx, "cov.4": _sum(ngroups, gb, ab),
                    "cov.5": _sum(ngroups, gb, ab * ab), "cov.6": _sum(ngroups, gb, b * ab)})
        return out
    out["sum_a.0"], out["sum_a.1"], out["sum_a.2"] = None, nrows, _sum(ngroups, g, a)
    _sums128(out, "sum_c", nrows, _sum(ngroups, g, cc))
    out["avg_b.0"], out["avg_b.1"], out["avg_b.2"] = None, nb, sb
    if fam == "nogroup":
        _minmax_fp(out, "b", ngroups, gb, b, nrows)
    return out


def _text_exact(c, limit):
    m = (c["v"] < limit).nonzero().view(-1)
    g, v, n, notnull = c["t"][m], c["v"][m].long(), c["n"][m], ~c["nnull"][m]
    nrows = _sum(TEXT_WORDS, g, torch.ones_like(g))
    nn = _sum(TEXT_WORDS, g[notnull], torch.ones_like(g[notnull]))
    sn = _sum(TEXT_WORDS, g[notnull], n[notnull])
    out = {"nrows.0": nrows, "nn.0": nn}
    _sums128(out, "sum_n", nn, sn)
    _sums128(out, "avg_n", nn, sn)
    out["sum_v.0"], out["sum_v.1"], out["sum_v.2"] = None, nrows, _sum(TEXT_WORDS, g, v)
    return out


def _join_exact(case, seed, c):
    d = _join_dims(case, seed)
    dev, n1 = c["i1"].device, case["dim1"]
    ok = torch.from_numpy(d["flag"]).to(dev)[c["i2"].long()] < 3
    if c["miss"] is not None:
        ok &= ~c["miss"]
    m = ok.nonzero().view(-1)
    amount, i1 = c["qty"][m].long() * c["price"][m], c["i1"][m].long()
    region = torch.from_numpy(d["region"]).to(dev)
    n, s = 0, 0
    for k in range(case["copies"]):
        g = region[k * n1:(k + 1) * n1][i1]
        n, s = n + _sum(len(C.REGIONS), g, torch.ones_like(g)), s + _sum(len(C.REGIONS), g, amount)
    out = {}
    _sums128(out, "amount", n, s)
    out["nrows.0"] = n
    return out


def _arrow_exact(case, r):
    keys, dev = case["keys"], r.d
    acc = {"nrows.0": torch.zeros(keys, dtype=torch.int64, device=dev)}
    for nm in ("n1", "s1", "n2"):
        acc[nm] = torch.zeros_like(acc["nrows.0"])
    s2 = torch.zeros(keys, dtype=torch.float64, device=dev)
    lo, hi = torch.full_like(s2, float("inf")), torch.full_like(s2, float("-inf"))
    for n in _arrow_chunk_sizes(case["rows"]):
        c = _arrow_columns(r, n, keys, case.get("nulls", 0.0))
        m = (c["d"] >= DAY_LO) & (c["d"] < DAY_HI)
        if c["d_ok"] is not None:
            m &= c["d_ok"]
        acc["nrows.0"].index_add_(0, c["k"][m], torch.ones_like(c["k"][m]))
        m1 = m if c["v1_ok"] is None else m & c["v1_ok"]
        acc["n1"].index_add_(0, c["k"][m1], torch.ones_like(c["k"][m1]))
        acc["s1"].index_add_(0, c["k"][m1], c["v1"][m1].long())
        m2 = m if c["v2_ok"] is None else m & c["v2_ok"]
        k2, v2 = c["k"][m2], c["v2"][m2]
        acc["n2"].index_add_(0, k2, torch.ones_like(k2))
        s2.index_add_(0, k2, v2)
        lo.scatter_reduce_(0, k2, v2, "amin")
        hi.scatter_reduce_(0, k2, v2, "amax")
    there = acc["nrows.0"] > 0
    lo = torch.where(there, torch.where(torch.isinf(lo), torch.full_like(lo, _DBL_MAX), lo), torch.zeros_like(lo))
    hi = torch.where(there, torch.where(torch.isinf(hi), torch.full_like(hi, -_DBL_MAX), hi), torch.zeros_like(hi))
    return {"nrows.0": acc["nrows.0"], "sum_v1.0": None, "sum_v1.1": acc["n1"], "sum_v1.2": acc["s1"],
            "min_v2.0": None, "min_v2.1": lo, "max_v2.0": None, "max_v2.1": hi,
            "sum_v2.0": None, "sum_v2.1": acc["n2"], "sum_v2.2": s2}


def _topn_exact(case, r):
    every = _arrow_exact(case, r)
    # the keys ascending, then stably by descending sum, groups without one last
    have = (every["nrows.0"] > 0).nonzero().view(-1)
    s = torch.where(every["sum_v2.1"][have] > 0, every["sum_v2.2"][have], float("-inf"))
    top = have[torch.sort(s, descending=True, stable=True).indices][:case["limit"]]
    out = {nm: None if v is None else v[top] for nm, v in every.items()}
    out["key"] = top
    return out


def exact(case, seed, device=None):
    fam = case["family"]
    device = device or torch.device("cuda", 0)
    r = _Rand(seed, device)
    if fam == "projection":
        return None                     # rows come back as bytes
    if fam in ("scan", "nogroup", "wide"):
        ngroups = case.get("groups", 1)
        return _scan_exact(_scan_columns(r, case["rows"], case.get("groups", 64)), case["limit"], ngroups, fam)
    if fam == "text":
        return _text_exact(_text_columns(r, case["rows"]), case["limit"])
    if fam == "join":
        return _join_exact(case, seed, _fact_columns(r, case))
    if fam == "arrow":
        return _arrow_exact(case, r)
    if fam == "topn":
        return _topn_exact(case, r)
    got = [_scan_exact(_scan_columns(r, n, groups), limit, groups, "scan")
           for n, limit, groups in _served_commands(case)]
    return {nm: None if got[0][nm] is None else torch.cat([g[nm] for g in got]) for nm in got[0]}
