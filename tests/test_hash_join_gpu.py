"""Hash join (join_algo HASH) and partitioned hash join (join_algo PARTITION)
against the CPU oracle's pair multiset: primary-key / foreign-key joins,
duplicate keys on both sides, a hot build key that overflows one
partition's shared-memory table (taken in chunks), float keys where -0.0
equals +0.0, sizes that need two radix passes, wide payloads and empty
sides.  Pairs are compared after sorting by (left row, right row)."""
import ctypes as C

import numpy as np
import pytest

import eiger_b200 as gx
import oracle as O
from tests.helpers import to_dev

pytestmark = pytest.mark.gpu

ALGOS = [gx.JOIN_HASH, gx.JOIN_PARTITION]


def mem_stats():
    cur, peak = C.c_int64(), C.c_int64()
    gx.check(gx.lib.gx_mem_stats(C.byref(cur), C.byref(peak)))
    return cur.value, peak.value


def rowid_pairs(lk, rk, algo, **kw):
    t = gx.inner_eq_join_rowids(to_dev(lk), to_dev(rk), gx.make_join_hint(algo, gx.MAT_GFUR, **kw))
    l, r = t.numpy_columns()
    o = np.lexsort((r, l))
    return l[o], r[o]


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("kdt", [np.int32, np.int64, np.uint32, np.uint64])
def test_pkfk_rowids(algo, kdt):
    npk, nfk = 1 << 15, 1 << 18
    pk = O.gen_perm(npk, kdt, seed=42)
    fk = O.gen_keys(nfk, kdt, groups=npk, seed=98, miss_frac=0.1)
    l, r = rowid_pairs(pk, fk, algo)
    el, er = O.join_pairs(pk, fk)
    assert np.array_equal(l, el) and np.array_equal(r, er)


@pytest.mark.parametrize("algo", ALGOS)
def test_left_larger_than_right(algo):
    # The smaller side builds; output columns stay in left / right order.
    lk = O.gen_keys(100_000, np.int32, groups=5000, seed=1)
    rk = O.gen_keys(7000, np.int32, groups=6000, seed=2)
    l, r = rowid_pairs(lk, rk, algo)
    el, er = O.join_pairs(lk, rk)
    assert np.array_equal(l, el) and np.array_equal(r, er)


@pytest.mark.parametrize("algo", ALGOS)
def test_hot_build_key_and_duplicates(algo):
    # 6000 build rows share one key (more than a 2048-row shared-table chunk),
    # the rest are random duplicates; every probe row of the hot key matches
    # all 6000.
    rng = np.random.default_rng(3)
    bk = rng.integers(0, 3000, size=20_000).astype(np.int64)
    bk[rng.choice(20_000, 6000, replace=False)] = 77
    pk = rng.integers(0, 4000, size=5_000).astype(np.int64)
    pk[:40] = 77
    l, r = rowid_pairs(bk, pk, algo)
    el, er = O.join_pairs(bk, pk)
    assert np.array_equal(l, el) and np.array_equal(r, er)
    assert len(l) > 40 * 6000


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("kdt", [np.float32, np.float64])
def test_float_keys_signed_zero(algo, kdt):
    rng = np.random.default_rng(4)
    lk = rng.integers(-50, 50, size=4000).astype(kdt)
    rk = rng.integers(-50, 50, size=9000).astype(kdt)
    lk[:10] = -0.0
    rk[:10] = 0.0
    l, r = rowid_pairs(lk, rk, algo)
    el, er = O.join_pairs(lk, rk)
    assert np.array_equal(l, el) and np.array_equal(r, er)


@pytest.mark.parametrize("algo", ALGOS)
def test_two_pass_partition_sizes(algo):
    # 2^21 build keys: the partitioned plan uses 11 radix bits (two passes).
    nb, npr = 1 << 21, 1 << 22
    bk = O.gen_perm(nb, np.int32, seed=5) * 3
    pk = O.gen_keys(npr, np.int32, groups=nb, seed=6, miss_frac=0.2) * 3
    m = O.join_probe_unique(bk, pk)
    l, r = rowid_pairs(bk, pk, algo)
    o = np.argsort(r, kind="stable")
    hit = np.nonzero(m >= 0)[0]
    assert np.array_equal(r[o], hit) and np.array_equal(l[o], m[hit])


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("mat", [gx.MAT_GFUR, gx.MAT_GFTR])
def test_wide_payloads(algo, mat):
    a = O.gen_keys(3000, np.int64, groups=500, seed=3)
    b = O.gen_keys(2000, np.int64, groups=700, seed=4)
    ap1 = O.gen_values(3000, np.int32, lo=0, hi=1 << 30, seed=5)
    ap2 = O.gen_values(3000, np.float64, seed=6)
    bp1 = O.gen_values(2000, np.int16, lo=-1000, hi=1000, seed=7)
    t = gx.inner_eq_join([to_dev(a), to_dev(ap1), to_dev(ap2)], [to_dev(b), to_dev(bp1)],
                         gx.make_join_hint(algo, mat))
    key, c1, c2, c3 = t.numpy_columns()
    el, er = O.join_pairs(a, b)
    exp = np.stack([a[el], ap1[el].astype(np.int64), ap2[el].view(np.int64), bp1[er].astype(np.int64)])
    got = np.stack([key, c1.astype(np.int64), c2.view(np.int64), c3.astype(np.int64)])
    assert np.array_equal(got[:, np.lexsort(got[::-1])], exp[:, np.lexsort(exp[::-1])])


@pytest.mark.parametrize("algo", ALGOS)
def test_empty_and_disjoint_sides(algo):
    e = np.zeros(0, dtype=np.int32)
    x = np.array([1, 2, 3], dtype=np.int32)
    for lk, rk in ((e, x), (x, e), (x, np.array([4, 5], np.int32))):
        t = gx.inner_eq_join_rowids(to_dev(lk), to_dev(rk), gx.make_join_hint(algo, gx.MAT_GFUR))
        assert t.num_rows == 0 and t.num_columns == 2


@pytest.mark.parametrize("algo", ALGOS)
def test_max_out_is_enforced(algo):
    x = np.arange(100, dtype=np.int32)
    with pytest.raises(gx.GxError):
        gx.inner_eq_join([to_dev(x), to_dev(x)], [to_dev(x), to_dev(x)], gx.make_join_hint(algo, gx.MAT_GFUR, max_out=50))


@pytest.mark.parametrize("algo", [gx.JOIN_SORT, gx.JOIN_HASH])
@pytest.mark.parametrize("kdt", [np.int32, np.uint32, np.int64, np.uint64])
@pytest.mark.parametrize("nb,npr", [(1, 1), (3, 2049), (5000, 2048 * 3), (20_000, 70_001)])
def test_unique_sparse_keys_one_pass(algo, kdt, nb, npr):
    # Unique build keys too sparse for direct placement: slots with the row id
    # or the single payload (4 or 8 bytes), few and many matches (buffers given
    # back when under half is used), keys at the type's limits and equal to the
    # empty slots' markers, and one duplicated key (another plan then).
    rng = np.random.default_rng(nb)
    lim = np.iinfo(kdt)
    special = np.array([lim.max, lim.min, 0, lim.max - 1], kdt)
    special = np.concatenate([special, np.array([-1], np.int64).astype(kdt),
                              np.array([-2**63], np.int64).astype(kdt) if np.dtype(kdt).itemsize == 8 else special[:1]])
    pool = np.unique(np.concatenate([special, rng.integers(lim.min, lim.max, 2 * nb, dtype=kdt)]))
    for with_special in (False, True):
        body = np.setdiff1d(pool, special)
        bk = rng.permutation(body)[:nb]
        if with_special and nb > 6:
            bk[: len(np.unique(special))] = np.unique(special)
        for dup in (False, True):
            if dup and nb > 1:
                bk = bk.copy()
                bk[-1] = bk[0]
            for share in (0.95, 0.05):
                pk = np.where(rng.random(npr) < share, bk[rng.integers(0, nb, npr)],
                              rng.integers(lim.min, lim.max, npr, dtype=kdt))
                pk[: min(npr, 6)] = special[: min(npr, 6)]
                el, er = O.join_pairs(bk, pk)
                l, r = rowid_pairs(bk, pk, algo)
                assert np.array_equal(l, el) and np.array_equal(r, er)
                for pdt in (np.int64, np.float32, np.int16):
                    bp, pp = np.arange(nb).astype(pdt), np.arange(npr).astype(np.int64)
                    t = gx.inner_eq_join([to_dev(bk), to_dev(bp)], [to_dev(pk), to_dev(pp)],
                                         gx.make_join_hint(algo, gx.MAT_GFUR))
                    key, b, p = t.numpy_columns()
                    o = np.lexsort((b, p))
                    e = np.lexsort((bp[el], er))
                    swap = nb > npr
                    assert not swap and np.array_equal(p[o], er[e]) and np.array_equal(b[o], bp[el][e])
                    assert np.array_equal(key[o], pk[er[e]])


@pytest.mark.parametrize("kdt", [np.int32, np.int64])
@pytest.mark.parametrize("nb", [1 << 17, 1 << 19])
def test_partition_join_whose_copies_give_up(monkeypatch, kdt, nb):
    # No wait for the copies of full tiles: the first pass (7 bits) or the first
    # of two (9 bits) moves nothing and the join reports it; the next is whole.
    bk = O.gen_perm(nb, kdt, seed=5) * kdt(3)
    pk = O.gen_keys(2 * nb, kdt, groups=nb, seed=6, miss_frac=0.2) * kdt(3)
    monkeypatch.setenv("GX_PART_COPY_POLLS", "0")
    with pytest.raises(gx.GxError, match="did not complete"):
        rowid_pairs(bk, pk, gx.JOIN_PARTITION)
    monkeypatch.delenv("GX_PART_COPY_POLLS")
    l, r = rowid_pairs(bk, pk, gx.JOIN_PARTITION)
    m = O.join_probe_unique(bk, pk)
    o = np.argsort(r, kind="stable")
    hit = np.nonzero(m >= 0)[0]
    assert np.array_equal(r[o], hit) and np.array_equal(l[o], m[hit])


@pytest.mark.parametrize("algo", [gx.JOIN_SORT, gx.JOIN_HASH])
@pytest.mark.parametrize("form", ["rowids", "table"])
@pytest.mark.parametrize("npr,share", [(1 << 20, 0.05), (1 << 24, 0.05), (1 << 24, 0.45)])
def test_selective_join_is_written_when_it_returns(algo, form, npr, share):
    # Few matches of sparse unique keys, on a stream that the NULL stream does
    # not wait for: nothing may be left in flight when the call returns (the
    # result is read through the NULL stream).
    import torch
    nb, step, n_pay = 100_003, 1_000_003, 6
    g = torch.Generator(device="cuda")
    g.manual_seed(npr)
    ids = torch.randperm(nb, device="cuda", generator=g)
    pid = torch.randint(0, nb, (npr,), device="cuda", generator=g)
    miss = torch.rand(npr, device="cuda", generator=g) >= share
    bk, pk = ids * step, (pid + miss * nb) * step
    row_of = torch.empty_like(ids)
    row_of[ids] = torch.arange(nb, device="cuda")
    want_p = torch.nonzero(~miss).squeeze(1)
    want_b = row_of[pid[want_p]]
    pays = [pk * (c + 2) for c in range(n_pay)]
    hint = gx.make_join_hint(algo, gx.MAT_GFUR)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        if form == "rowids":
            t = gx.inner_eq_join_rowids(bk, pk, hint, stream=s)
            assert s.query()
            b, p = t.numpy_columns()
            assert np.array_equal(b, want_b.cpu().numpy()) and np.array_equal(p, want_p.cpu().numpy())
        else:
            t = gx.inner_eq_join([bk, ids], [pk, *pays], hint, stream=s)
            assert s.query()
            cols = t.numpy_columns()
            assert np.array_equal(cols[0], pk[want_p].cpu().numpy()) and np.array_equal(cols[1], pid[want_p].cpu().numpy())
            for c in range(n_pay):
                assert np.array_equal(cols[2 + c], pays[c][want_p].cpu().numpy())
        del t


@pytest.mark.parametrize("kdt", [np.int32, np.uint32, np.int64, np.uint64])
@pytest.mark.parametrize("nb,npr", [(2, 7), (900, 2049), (40_000, 50_001), (4_000, (1 << 20) + 5)])
@pytest.mark.parametrize("marker", [False, True])
def test_duplicate_build_keys_in_the_key_table(kdt, nb, npr, marker):
    # Duplicated integer keys are probed in the table that was built to find
    # out whether they are unique, below and above the size at which a probe is
    # queued before that is known: row ids, one payload (held in the slots) of 4
    # and 8 bytes, a narrow one, and two.  Keys at the type's limits, and with
    # `marker` the 8-byte key that marks empty slots (another table then).
    rng = np.random.default_rng(nb)
    lim = np.iinfo(kdt)
    edge = np.array([lim.max, lim.min, lim.max - 1, 0], kdt)
    if np.dtype(kdt).itemsize == 8 and not marker:
        edge = edge[edge.view(np.uint64) != np.uint64(2**63)]
    elif marker:
        edge = np.append(edge, np.array([-2**63 if np.dtype(kdt).itemsize == 8 else -2**31], np.int64).astype(kdt))
    pool = np.concatenate([edge, rng.integers(1, lim.max - 1, nb, dtype=kdt)])
    bk = rng.choice(pool[: max(2, nb // 2)], nb)
    bk[-1] = bk[0]
    pk = rng.choice(np.concatenate([pool, rng.integers(1, lim.max - 1, nb, dtype=kdt)]), npr)
    el, er = O.join_pairs(bk, pk)
    l, r = rowid_pairs(bk, pk, gx.JOIN_HASH)
    assert np.array_equal(l, el) and np.array_equal(r, er)
    pp = np.arange(npr)
    for pdts in ((np.int64,), (np.float32,), (np.int16,), (np.int64, np.int32)):
        bps = [(np.arange(nb) * (c + 1)).astype(d) for c, d in enumerate(pdts)]
        t = gx.inner_eq_join([to_dev(bk), *map(to_dev, bps)], [to_dev(pk), to_dev(pp)],
                             gx.make_join_hint(gx.JOIN_HASH, gx.MAT_GFUR))
        cols = t.numpy_columns()
        key, b, p = cols[0], cols[1:-1], cols[-1]
        assert np.array_equal(key, pk[p])
        o, e = np.lexsort((*b, p)), np.lexsort((*[x[el] for x in bps], er))
        assert np.array_equal(p[o], er[e])
        for got, x in zip(b, bps):
            assert np.array_equal(got[o], x[el][e])


@pytest.mark.parametrize("kdt", [np.int32, np.int64])
@pytest.mark.parametrize("share", [0.0, 0.01, 0.5, 1.0])
def test_hash_join_outputs_follow_the_matches(kdt, share):
    # A long probe's outputs have room for the matches that a sample predicts,
    # not for every probe row.
    import torch
    nb, npr, step, n_pay = 50_021, (1 << 22) + 1, 10_007, 5
    t = torch.int32 if kdt == np.int32 else torch.int64
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    ids = torch.randperm(nb, device="cuda", generator=g)
    pid = torch.randint(0, nb, (npr,), device="cuda", generator=g)
    miss = torch.rand(npr, device="cuda", generator=g) >= share
    bk, pk = (ids * step).to(t), (pid * step + miss.long()).to(t)
    pays = [pid * (c + 1) for c in range(n_pay)]
    torch.cuda.synchronize()
    current, _ = mem_stats()
    gx.check(gx.lib.gx_mem_reset_peak())
    out = gx.inner_eq_join([bk, ids], [pk, *pays], gx.make_join_hint(gx.JOIN_HASH, gx.MAT_GFUR))
    _, peak = mem_stats()
    width = np.dtype(kdt).itemsize + 8 * (n_pay + 1)
    # A table of 2^17 slots of 16 bytes, tile states, and 1.2% of the rows to
    # spare in each column.
    assert peak - current <= (share + 0.012) * npr * width + (4 << 20)
    want = torch.nonzero(~miss).squeeze(1)
    assert out.num_rows == want.numel()
    cols = out.numpy_columns()
    assert np.array_equal(cols[0], pk[want].cpu().numpy()) and np.array_equal(cols[1], pid[want].cpu().numpy())
    for c in range(n_pay):
        assert np.array_equal(cols[2 + c], pays[c][want].cpu().numpy())


@pytest.mark.parametrize("kdt", [np.int32, np.int64])
@pytest.mark.parametrize("pay", [False, True])
def test_matches_that_the_sample_misses(kdt, pay):
    # Every row matches but the ones that the size of the outputs is sampled
    # from: the probe runs again with room for all.
    nb, npr, step = 4099, (1 << 22) + 77, 10_007
    rng = np.random.default_rng(9)
    ids = rng.permutation(nb)
    pid = rng.integers(0, nb, npr)
    i = np.arange(1 << 15, dtype=np.uint64)
    every = npr // (1 << 15)
    miss = np.zeros(npr, bool)
    miss[(i * every + (i * 2654435761 % 2**32) % every).astype(np.int64)] = True
    bk, pk = (ids * step).astype(kdt), (pid * step + miss).astype(kdt)
    want = np.nonzero(~miss)[0]
    row_of = np.empty(nb, np.int64)
    row_of[ids] = np.arange(nb)
    hint = gx.make_join_hint(gx.JOIN_HASH, gx.MAT_GFUR)
    if pay:
        out = gx.inner_eq_join([to_dev(bk), to_dev(ids)], [to_dev(pk), to_dev(pid)], hint)
        key, b, p = out.numpy_columns()
        assert np.array_equal(key, pk[want]) and np.array_equal(b, pid[want]) and np.array_equal(p, pid[want])
    else:
        b, p = gx.inner_eq_join_rowids(to_dev(bk), to_dev(pk), hint).numpy_columns()
        assert np.array_equal(b, row_of[pid[want]]) and np.array_equal(p, want)
