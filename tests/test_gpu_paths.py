"""The branches that the group tables, the final stage and the launches take
by size: each at the sizes around its border, against the generators' arrays
or the oracle (integers, numerics and keys exact, float sums within 1e-12 of
the sum of the terms' magnitudes)."""
import struct

import numpy as np
import pytest

import xb_configs as C
import xb_exchange as X
import xb_final as F
import xb_oracle as O
import xpu_b200
from xb_producer import Agg, Column, Const, Func, SessionBuilder, Table, Var, numeric_typmod

pytestmark = pytest.mark.gpu


def _truth(expect):
    return {k: [v["nrows"], v["sum_a"], v["sum_c"], v["avg_b"]] for k, v in expect.items()}


def _run(device, sess, chunks, km=None, nrels=0):
    s = xpu_b200.Session(device, sess, km, nrels)
    try:
        for ch in chunks:
            s.exec(ch)
        final, res = s.final()
        return (F.decode_kds_final(final, sess) if final is not None else {}), res
    finally:
        s.close()


def _oracle(sess, chunks):
    o = O.Oracle(sess)
    for ch in chunks:
        o.exec(ch)
    out = F.decode_kds_final(o.final(), sess)
    o.close()
    return out


# ---- shared group tables: the capacity follows the estimate, the groups
# may be more or fewer (est entries of 112 + 8 bytes: 256 entries at most)
@pytest.mark.parametrize("est,groups", [(1, 1), (1, 700), (3, 3), (60, 64), (64, 900), (200, 200), (224, 230),
                                        (225, 225), (400, 390), (410, 3000), (300, 1), (2048, 3), (2049, 3), (1000, 90),
                                        (1000, 127), (1000, 129), (2000, 256)])
def test_shared_table_estimates(device, est, groups):
    tbl, _, _, expect, meta = C.scan_groupby(nrows=40_000, seed_config=60 + est % 7, a_limit=600, ngroups=groups)
    got, res = _run(device, C.scan_groupby_session(600, est), tbl.block_chunks(pages_per_chunk=300))
    assert res["nitems_in"] == meta["nitems_in"]
    assert F.compare_groups(got, _truth(expect)) == []


@pytest.mark.parametrize("est,groups", [(1, 2), (3, 3), (100, 112), (113, 150), (500, 3), (2000, 70)])
def test_shared_table_of_large_entries(device, est, groups):
    tbl, _, _, expect, _ = C.wide_groupby(nrows=30_000, seed_config=70, ngroups=groups)
    got, _ = _run(device, C.wide_groupby_session(ngroups=est), tbl.block_chunks(pages_per_chunk=300))
    assert F.compare_groups(got, expect) == []


def test_estimate_far_above_the_groups(device, monkeypatch):
    # a few groups take about as long under a high estimate as under the right
    # one, on both kernels (20 times as long in the global table)
    tbl, _, _, expect, _ = C.scan_groupby(nrows=1_000_000, seed_config=71, a_limit=600, ngroups=3)
    ups = [device.upload(c) for c in tbl.block_chunks(pages_per_chunk=4000)]
    try:
        for jit in ("1", "0"):
            monkeypatch.setenv("XPU_B200_JIT", jit)
            ms = {}
            for est in (3, 1000):
                s = xpu_b200.Session(device, C.scan_groupby_session(600, est))
                b = s.batch([p for _, p in ups])
                b.exec()
                got = F.decode_kds_final(s.final()[0], C.scan_groupby_session(600, est))
                assert F.compare_groups(got, _truth(expect)) == []
                ms[est] = min(b.time(3) for _ in range(5))
                b.close()
                s.close()
            assert ms[1000] < 3 * ms[3], (jit, ms)
    finally:
        for base, _ in ups:
            device.free(base)


# ---- no GROUP BY: every state form from the lanes' registers
@pytest.mark.parametrize("nrows,limit", [(50_000, 1000), (50_000, 3), (33, 1000), (1, 1000), (31, 500), (2_000, 0)])
def test_no_group_by_state_forms(device, nrows, limit):
    r = np.random.default_rng(nrows + limit)
    w = r.integers(-2 ** 62, 2 ** 62, nrows, dtype=np.int64)
    tbl, a, b, bnull, c, g = C._scan_table(nrows, 61, 0.1, 64)
    tbl.columns[0].values = w                                   # id: sums beyond 64 bits
    typmod = numeric_typmod(12, 2)
    vi, va, vb, vc = Var(0, 1, "int8"), Var(0, 2, "int4"), Var(0, 3, "float8"), Var(0, 4, "numeric", typmod)
    sess = SessionBuilder(0, C.DEVTASK_PREAGG | C.DEVKIND_GPU).build(
        scan_quals=Func("int4lt", [va, Const("int4", limit)], "bool"), groupby_keys=[],
        aggs=[Agg("NROWS_ANY"), Agg("NROWS_COND", vb), Agg("PMIN_INT32", va),
              Agg("PMAX_INT64", vi), Agg("PMIN_FP64", vb), Agg("PMAX_FP64", vb), Agg("PSUM_INT64", vi),
              Agg("PSUM_FP", vb), Agg("PSUM_NUMERIC", vc, typmod), Agg("PAVG_NUMERIC", vc, typmod),
              Agg("STDDEV", vb), Agg("COVAR", vb, arg1=Func("int4_to_float8", [va], "float8"))],
        ngroups_estimate=1.0)
    chunks = tbl.block_chunks(pages_per_chunk=100)
    got, _ = _run(device, sess, chunks)
    m = a < limit
    n, mb = int(m.sum()), m & ~bnull
    if n == 0:
        assert got == {}
        return
    nb, x, y = int(mb.sum()), b[mb], a[mb].astype(np.float64)
    ap = lambda v: F.Approx(float(v.sum()), float(np.abs(v).sum()))  # noqa: E731
    sc = int(c[m].sum())
    valid = 1 if nb else 0
    want = [n, nb, (1, int(a[m].min())), (1, int(w[m].max())),
            (valid, float(x.min()) if nb else None), (valid, float(x.max()) if nb else None),
            (n, sum(w[m].tolist())), (nb, ap(x)), (n, sc, 2), (n, sc, 2), (nb, ap(x), ap(x * x)),
            (nb, ap(x), ap(x * x), ap(y), ap(y * y), ap(x * y))]
    assert F.compare_groups(got, {(): want}) == []


def test_no_group_by_over_a_join(device):
    # joined rows counted and summed in the lanes' registers
    fact, _, km, _, meta = C.join_groupby(nfact=30_000, ndim1=100, ndim2=10, seed_config=66)
    k1, k2 = Var(0, 1, "int4"), Var(0, 2, "int4")
    sess = SessionBuilder(2, C.DEVTASK_PREAGG | C.DEVKIND_GPU).build(
        joins=[([k1], [Func("int4eq", [k1, Var(1, 1, "int4")], "bool")], []),
               ([k2], [Func("int4eq", [k2, Var(2, 1, "int4")], "bool")], [])],
        aggs=[Agg("NROWS_ANY"), Agg("PSUM_INT", Func("int4_to_int8", [k1], "int8")),
              Agg("PMAX_INT32", Var(1, 1, "int4")), Agg("PMIN_INT32", k2)],
        ngroups_estimate=1.0)
    chunks = fact.block_chunks(pages_per_chunk=100)
    o = O.Oracle(sess, km)
    for ch in chunks:
        o.exec(ch)
    want = F.decode_kds_final(o.final(), sess)
    o.close()
    got, _ = _run(device, sess, chunks, km, 2)
    assert want and F.compare_groups(got, want) == []


# ---- infinities, NaN and the ends of int8 in every form of the updates: the
# groups' states start at INT64_MAX / INT64_MIN, which values may equal
def _extreme_table(nrows):
    r = np.random.default_rng(67)
    g = (np.arange(nrows) % 8).astype(np.int32)
    b = r.integers(-1000, 1000, nrows).astype(np.float64)       # finite sums are exact
    pick = (np.arange(nrows) // 8) % 5
    b[(g == 1) & (pick == 2)] = np.inf
    b[(g == 2) & (pick == 3)] = -np.inf
    b[(g == 3) & (pick == 1)] = np.inf
    b[(g == 3) & (pick == 4)] = -np.inf
    b[(g == 4) & (pick == 0)] = np.nan
    b[g == 6] = np.inf
    b[g == 7] = -np.inf
    top, low = np.iinfo(np.int64).max, np.iinfo(np.int64).min
    w = r.integers(-5, 6, nrows, dtype=np.int64)
    w[g == 0], w[g == 1] = top, low
    w[(g == 2) & (pick == 1)], w[(g == 2) & (pick == 2)] = top, low
    return Table("t", [Column("w", "int8", values=w), Column("b", "float8", values=b, nulls=(g == 5)),
                       Column("g", "int4", values=g)], nrows)


def _plain(groups):
    """decoded groups with floats as comparable texts, undefined values left out"""
    one = lambda v: repr(float(v)) if isinstance(v, (float, np.floating)) else v        # noqa: E731
    return {k: [tuple(one(x) for x in (s[:1] if s[0] == 0 else s)) if isinstance(s, tuple) else one(s) for s in v]
            for k, v in groups.items()}


@pytest.mark.parametrize("path", ["vm", "shared", "global", "slices", "none"])
def test_extreme_values(device, monkeypatch, path):
    monkeypatch.setenv("XPU_B200_JIT", "0" if path == "vm" else "1")
    monkeypatch.setenv("XPU_B200_PARTITION", "1" if path == "slices" else "0")
    vw, vb, vg = Var(0, 1, "int8"), Var(0, 2, "float8"), Var(0, 3, "int4")
    aggs = [Agg("NROWS_ANY"), Agg("PMIN_INT64", vw), Agg("PMAX_INT64", vw), Agg("PMIN_FP64", vb), Agg("PMAX_FP64", vb),
            Agg("PSUM_FP", vb), Agg("PAVG_INT64", vw), Agg("STDDEV", vb), Agg("COVAR", vb, arg1=vb)]
    chunks = _extreme_table(6_000).block_chunks(pages_per_chunk=20)
    flags = C.DEVTASK_PREAGG | C.DEVKIND_GPU
    if path == "none":
        sessions = [SessionBuilder(0, flags).build(scan_quals=Func("int4eq", [vg, Const("int4", i)], "bool"), aggs=aggs,
                                                   ngroups_estimate=1.0) for i in range(8)]
    else:
        est = {"global": 20_000.0, "slices": 1_000_000.0}.get(path, 8.0)
        sessions = [SessionBuilder(0, flags).build(groupby_keys=[vg], aggs=aggs, ngroups_estimate=est)]
    for sess in sessions:
        want = _plain(_oracle(sess, chunks))
        s = xpu_b200.Session(device, sess)
        try:
            for ch in chunks:
                s.exec(ch)
            got = _plain(F.decode_kds_final(s.final()[0], sess))
            info = s.info()
        finally:
            s.close()
        assert info["kernels"] == {"b": "vm" if path == "vm" else "jit"}, info
        assert info["partition_used"] == (path == "slices"), info
        assert got == want


# ---- filters that none, few and all rows of a page pass
@pytest.mark.parametrize("limit", [0, 1, 500, 1000])
@pytest.mark.parametrize("nrows", [1, 31, 130, 20_000])
def test_filter_selectivities(device, nrows, limit):
    tbl, sess, _, expect, meta = C.scan_groupby(nrows=nrows, seed_config=62, a_limit=limit, ngroups=2_000)
    got, res = _run(device, sess, tbl.block_chunks(pages_per_chunk=7))
    assert (res["nitems_raw"], res["nitems_in"]) == (meta["nitems_raw"], meta["nitems_in"])
    assert F.compare_groups(got, _truth(expect)) == []


@pytest.mark.parametrize("nrows,batch", [(1, 1), (33, 10), (5_000, 1_025), (40_000, 3_001)])
def test_compaction_arrow_units(device, nrows, batch):
    chunks, sess, expect, meta = C.arrow_nulls(nrows=nrows, nkeys=500, rows_per_chunk=batch, short_rows=0)
    got, res = _run(device, sess, chunks)
    assert res["nitems_in"] == meta["nitems_in"]
    assert F.compare_groups(got, expect) == []


# ---- Arrow rows compacted between the quals and the rest: none, few and all
# of a unit's rows wait in the queue
@pytest.mark.parametrize("lo,hi", [(30_000, 30_001), (16_436, 16_437), (17_532, 18_262), (0, 30_000)])
@pytest.mark.parametrize("nrows,batch", [(1, 1), (33, 33), (1_024, 1_024), (20_000, 3_001)])
def test_compaction_arrow_selectivities(device, nrows, batch, lo, hi):
    chunks, _, _, _ = C.arrow_groupby(nrows=nrows, nkeys=300, rows_per_chunk=batch, seed_config=69, with_expect=False)
    sess = C.arrow_groupby_session(lo, hi, ngroups_estimate=300.0)
    want = _oracle(sess, chunks)
    got, res = _run(device, sess, chunks)
    assert res["nitems_raw"] == nrows
    assert res["nitems_in"] == sum(v[0] for v in want.values())
    if lo == 30_000 or hi == 30_000:
        assert res["nitems_in"] == (nrows if hi == 30_000 else 0)
    assert F.compare_groups(got, want) == []


def test_value_saved_by_the_quals(device):
    # a SaveExpr in the scan quals whose slot an aggregate reads
    chunks, _, _, _ = C.arrow_groupby(nrows=20_000, nkeys=500, rows_per_chunk=3_001, seed_config=65, with_expect=False)
    for saved in (False, True):
        sess = C.arrow_saved_qual_session(saved)
        want = _oracle(sess, chunks)
        assert len(want) == 500
        got, _ = _run(device, sess, chunks)
        assert F.compare_groups(got, want) == []


# ---- chunk headers: more chunks than one fetch takes, a header larger than
# its slot (30 columns)
def test_many_chunks_in_a_batch(device):
    tbl, sess, _, expect, meta = C.scan_groupby(nrows=36_000, seed_config=63)
    chunks = tbl.block_chunks(pages_per_chunk=1)
    assert len(chunks) > 2 * 128
    ups = [device.upload(c) for c in chunks]
    s = xpu_b200.Session(device, sess)
    try:
        b = s.batch([p for _, p in ups])
        assert b.exec()["nitems_in"] == meta["nitems_in"]
        b.close()
        final, _ = s.final()
    finally:
        s.close()
        for base, _ in ups:
            device.free(base)
    assert F.compare_groups(F.decode_kds_final(final, sess), _truth(expect)) == []


def test_batch_closed_after_its_session(device):
    tbl, sess, _, expect, meta = C.scan_groupby(nrows=5_000, seed_config=68)
    ups = [device.upload(c) for c in tbl.block_chunks(pages_per_chunk=20)]
    try:
        for _ in range(3):
            s = xpu_b200.Session(device, sess)
            b = s.batch([p for _, p in ups])
            assert b.exec()["nitems_in"] == meta["nitems_in"]
            got = F.decode_kds_final(s.final()[0], sess)
            s.close()
            other = xpu_b200.Session(device, sess)      # takes the pooled stream
            b.close()
            other.close()
            assert F.compare_groups(got, _truth(expect)) == []
    finally:
        for base, _ in ups:
            device.free(base)


def test_chunk_header_of_many_columns(device):
    n, r = 3_000, np.random.default_rng(64)
    k, v = r.integers(0, 50, n, dtype=np.int32), r.integers(-1000, 1000, n, dtype=np.int32)
    cols = [Column("c%d" % i, "int4", values=np.full(n, i, dtype=np.int32)) for i in range(28)]
    tbl = Table("t", cols + [Column("k", "int4", values=k), Column("v", "int4", values=v)], n)
    vk, vv = Var(0, 29, "int4"), Var(0, 30, "int4")
    sess = SessionBuilder(0, C.DEVTASK_PREAGG | C.DEVKIND_GPU).build(
        groupby_keys=[vk], aggs=[Agg("NROWS_ANY"), Agg("PSUM_INT", Func("int4_to_int8", [vv], "int8"))],
        ngroups_estimate=50.0)
    chunk, = tbl.block_chunks()
    base, p = device.upload(chunk)
    s = xpu_b200.Session(device, sess)
    try:
        s.exec(p, on_device=True)
        got = F.decode_kds_final(s.final()[0], sess)
    finally:
        s.close()
        device.free(base)
    want = {(i,): [int((k == i).sum()), (int((k == i).sum()), int(v[k == i].sum()))] for i in np.unique(k).tolist()}
    assert F.compare_groups(got, want) == []


# ---- kds_final by tiles: NULL and present keys side by side (tuples of two
# layouts), text keys, few and many hash parts
def _parts(device, sess, chunks, nparts):
    s = xpu_b200.Session(device, sess)
    try:
        for ch in chunks:
            s.exec(ch)
        whole = s.final()[0]
        base, offs = X.final_parts(device, s, nparts)
        raw = device.download(base, offs[-1])
        device.free(base)
    finally:
        s.close()
    out, sizes = {}, []
    for p in range(nparts):
        part = raw[offs[p]:offs[p + 1]]
        length, usage, n = struct.unpack_from("<QQI", part, 0)
        part = part[:length]
        ncol, = struct.unpack_from("<I", part, 68)
        nslots, = struct.unpack_from("<I", part, 40)
        idx = np.frombuffer(part[(72 + 168 * ncol + 7) & ~7:].tobytes(), dtype=np.uint64, offset=8 * nslots, count=n)
        for o in idx.tolist():
            h, = struct.unpack_from("<I", part, length - o + 4)
            assert h % nparts == p
        got = F.decode_kds_final(part, sess)
        assert len(got) == n and not set(got) & set(out)
        out.update(got)
        sizes.append(n)
    return F.decode_kds_final(whole, sess), out, sizes


@pytest.mark.parametrize("nparts", [1, 2, 8, 1_100])
def test_final_parts(device, nparts):
    chunks, sess, expect, _ = C.arrow_nulls(nrows=20_000, nkeys=3_000, short_rows=0)
    whole, parts, sizes = _parts(device, sess, chunks, nparts)
    assert F.compare_groups(whole, expect) == []
    assert F.compare_groups(parts, expect) == []
    assert sum(sizes) == len(expect)


@pytest.mark.parametrize("nparts", [1, 5])
def test_final_parts_text_keys(device, nparts):
    tbl, sess, _, expect, _ = C.long_varlena_groupby(nrows=6_000, ngroups=140)
    whole, parts, _ = _parts(device, sess, tbl.block_chunks(), nparts)
    assert F.compare_groups(whole, expect) == []
    assert F.compare_groups(parts, expect) == []


# ---- LIMIT: the groups sorted by one CTA (4096 at most), picked first by
# the leading digits of the first key, or sorted whole
@pytest.mark.parametrize("ngroups,limit,keys", [
    (4_000, 10, [("PSUM_FP64", 7, False, False)]),
    (9_000, 1, [("PSUM_FP64", 7, True, False)]),
    (9_000, 1_000, [("PSUM_FP64", 7, False, True), ("VREF", 11, True, False)]),
    (9_000, 4_096, [("VREF", 11, False, False)]),
    (9_000, 5_000, [("VREF", 11, True, False)]),
    (9_000, 100, [("VREF", 1, False, False), ("VREF", 11, True, False)]),      # counts: thousands of ties
    (9_000, 20_000, [("PMINMAX_INT64", 3, True, False), ("VREF", 11, False, False)]),
])
def test_limit(device, ngroups, limit, keys):
    tbl, _, _, expect, _ = C.wide_groupby(nrows=60_000, seed_config=65, ngroups=ngroups)
    sess = C.wide_groupby_session(ngroups=ngroups, sort={"keys": keys, "limit": limit})
    chunks = tbl.block_chunks(pages_per_chunk=300)
    got, res = _run(device, sess, chunks)
    want = F.order_groups(list(_oracle(sess, chunks).items()), sess, keys, None, limit)
    assert res["final_nitems"] == len(want) == len(got)
    vals = [F.sort_key_values(x, sess, keys) for x in got.items()]
    for p in range(1, len(vals)):
        assert F._cmp_values(vals[p - 1], vals[p], keys) <= 0, p
    if keys[-1][0] == "VREF" and keys[-1][1] == 11:             # a total order: the very groups
        assert list(got) == [x[0] for _, x in want]
    assert F.compare_groups(got, {k: expect[k] for k in got}) == []


# ---- replay on slices of the table: probes that leave a slice (256 slots of
# 288 bytes, half full), chunks replayed on an empty and on a filled table
@pytest.mark.parametrize("est,groups", [(64_000, 40), (64_000, 20_000), (64_000, 120_000)])
def test_replay_slices(device, monkeypatch, est, groups):
    monkeypatch.setenv("XPU_B200_PARTITION", "1")
    tbl, _, _, expect, _ = C.wide_groupby(nrows=200_000, seed_config=66, ngroups=groups)
    sess = C.wide_groupby_session(ngroups=est)
    chunks = tbl.block_chunks(pages_per_chunk=700)
    assert len(chunks) >= 3
    s = xpu_b200.Session(device, sess)
    try:
        for ch in chunks:
            s.exec(ch)
        assert s.info()["partition_used"], s.info()
        got = F.decode_kds_final(s.final()[0], sess)
    finally:
        s.close()
    assert F.compare_groups(got, expect) == []


# ---- kds_final counted by one CTA (16384 slots at most) or by tiles
@pytest.mark.parametrize("est,slots", [(1, 2048), (3_840, 16_384), (3_841, 32_768)])
@pytest.mark.parametrize("groups", [1, 33, 3_000])
def test_final_of_small_tables(device, est, slots, groups):
    tbl, _, _, expect, _ = C.scan_groupby(nrows=12_000, seed_config=67, a_limit=700, ngroups=groups)
    sess = C.scan_groupby_session(700, est)
    s = xpu_b200.Session(device, sess)
    try:
        assert s.info()["gtable_cap"] == slots
        for ch in tbl.block_chunks(pages_per_chunk=300):
            s.exec(ch)
        got = F.decode_kds_final(s.final()[0], sess)
    finally:
        s.close()
    assert F.compare_groups(got, _truth(expect)) == []


# ---- sessions of one plan shape share a kernel: a session with a small shared
# table opened after one with a large table must not take its shared memory
def test_shared_kernel_of_two_table_sizes(device):
    tbl, _, _, expect, _ = C.scan_groupby(nrows=20_000, seed_config=68, a_limit=600, ngroups=200)
    chunks = tbl.block_chunks(pages_per_chunk=100)
    large, small = C.scan_groupby_session(600, 200), C.scan_groupby_session(600, 1)
    a, b = xpu_b200.Session(device, large), xpu_b200.Session(device, small)
    try:
        for ch in chunks:
            a.exec(ch)
            b.exec(ch)
        assert a.info()["smem_bytes"] > b.info()["smem_bytes"]
        for s, sess in ((a, large), (b, small)):
            assert F.compare_groups(F.decode_kds_final(s.final()[0], sess), _truth(expect)) == []
    finally:
        a.close()
        b.close()
