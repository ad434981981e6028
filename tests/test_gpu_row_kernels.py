"""Row kernels of the fused pass at the sizes where they can go wrong: every
product count around a bin's capacity, columns spread evenly or crowded into a
few neighbours, and column spans around the limits of the packed sort keys.
Structure is compared exactly and values within the stated bounds of
helpers.py, against the FP64 oracle."""
import numpy as np
import pytest

import spgemm_b200 as sg
from spgemm_b200 import workloads as W
from helpers import assert_structure_equal, assert_values_close, compensated_tolerance, plain_tolerance
from test_gpu_batch import DeviceBatch, check_all
from test_gpu_parity import ref_product

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 204, 205, 255, 256, 257, 511, 512,
          513, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096]


def rows_of(counts, n, lengths, crowd, seed, empty=0):
    """A and B such that row i of A*B has counts[i] products, from rows of B of
    the given lengths in turn (the last one cut to fit) and `empty` empty rows
    of B spread among them. Columns: distinct in a row of B, uniform in [0, n),
    or (crowd) within 64 neighbours but for one far column in each row."""
    rng = np.random.default_rng(seed)
    ar, ac, br, bc, k = [], [], [], [], 0
    for i, count in enumerate(counts):
        left, turn, used = count, 0, []
        while left > 0:
            size = min(lengths[turn % len(lengths)], left, 60 if crowd else n)
            if crowd:
                cols = np.concatenate([n // 3 + rng.choice(64, size - 1, replace=False), [n - 1 - i]])
            else:
                cols = rng.choice(n, size, replace=False) if n < 10000 else np.unique(rng.integers(0, n, 4 * size))
                cols = rng.permutation(cols)[:size]
            br += [k] * size
            bc += sorted(cols.tolist())
            used.append(k)
            k += 1
            left -= size
            turn += 1
        used += list(range(k, k + empty))
        k += empty
        ar += [i] * len(used)
        ac += used
    vals = lambda size: rng.uniform(-1, 1, size).astype(np.float32)
    A = W.from_coo(len(counts), k, np.array(ar), np.array(ac), vals(len(ar)))
    B = W.from_coo(k, n, np.array(br), np.array(bc), vals(len(br)))
    return A, B


def check_rows(A, B, precision, tuning):
    ref = ref_product(A, B)
    with sg.Handle(precision) as h:
        h.set_tuning(**tuning)
        C = h.multiply_host(A, B)
        stats = h.stats()
    assert_structure_equal(C.rowptr, C.col, ref["rowptr"], ref["col"])
    tol = plain_tolerance(ref) if precision == sg.PLAIN else compensated_tolerance(ref)
    assert_values_close(C.val, ref, tol)
    return stats


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("n", [5003, (1 << 20) + 77, 1 << 25])
@pytest.mark.parametrize("lengths,crowd", [((1,), False), ((13, 40, 3), False), ((60, 5), True)])
def test_sorted_rows_around_their_capacities(precision, n, lengths, crowd):
    A, B = rows_of(COUNTS, n, lengths, crowd, seed=len(lengths))
    stats = check_rows(A, B, precision, dict(warp_cap_max=0))
    assert sum(stats["rows_per_symbolic_bin"][10:13]) == len(COUNTS), stats


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("n", [4096, 4128, 40999, (1 << 27) + 5])
@pytest.mark.parametrize("lengths,crowd,empty", [((1,), False, 0), ((2, 1), False, 40), ((11, 3, 60), False, 3),
                                                 ((33, 200), False, 0), ((60, 5), True, 0)])
def test_warp_rows_around_their_capacities(precision, n, lengths, crowd, empty):
    """Default tuning: rows of at most 32 products in registers (with empty
    rows of B among their entries), rows of at most 4096 columns in a warp's
    bitmap, wider ones hashed; rows of more outputs than those hold are redone."""
    A, B = rows_of([c for c in COUNTS if c <= 2048], n, lengths, crowd, seed=n % 1000, empty=empty)
    stats = check_rows(A, B, precision, {})
    assert sum(stats["rows_per_symbolic_bin"][:5]) == A.rows, stats


@pytest.mark.parametrize("csc", [False, True])
@pytest.mark.parametrize("m", [1, 63, 64, 65, 4095, 4096, 4097, 20011])
def test_row_analysis_and_scans_by_size(m, csc):
    """Row counts around a scan tile and a block of row analysis, A rows of a
    few entries with some above what a group of lanes walks (1024), most
    columns of A empty, and B rows that are often empty."""
    rng = np.random.default_rng(m)
    k, n = 30011, 700
    lens = rng.integers(0, 4, m)
    for size, i in zip((1024, 1025, 1300, 4000), rng.choice(m, min(m, 4), replace=False)):
        lens[i] = size
    used = np.sort(rng.choice(k, 5000, replace=False))
    r = np.repeat(np.arange(m), lens)
    c = np.concatenate([used[np.sort(rng.choice(5000, x, replace=False))] for x in lens]) if lens.sum() else r
    A = W.from_coo(m, k, r, c, rng.uniform(-1, 1, len(r)).astype(np.float32))
    blens = rng.integers(0, 3, k)
    br = np.repeat(np.arange(k), blens)
    bc = np.concatenate([np.sort(rng.choice(n, x, replace=False)) for x in blens])
    B = W.from_coo(k, n, br, bc, rng.uniform(-1, 1, len(br)).astype(np.float32))
    ref = ref_product(A, B)
    with sg.Handle() as h:
        C = h.multiply_host(A.to_csc() if csc else A, B)
        assert h.stats()["intermediate_products"] == ref["products"]
    assert_structure_equal(C.rowptr, C.col, ref["rowptr"], ref["col"])
    assert_values_close(C.val, ref, plain_tolerance(ref))


@pytest.mark.parametrize("seed", range(12))
def test_unsorted_rows_are_refused(seed):
    """Rows of B must rise strictly: a repeat or a swap inside a row is
    refused wherever it lies, equal or falling columns across a row boundary
    (also over empty rows) are not."""
    rng = np.random.default_rng(seed)
    k, n = 700, 40
    lens = rng.integers(0, 6, k)
    col = np.concatenate([np.sort(rng.choice(n, x, replace=False)) for x in lens]).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    B = W.Csr(k, n, ptr, col, np.ones(len(col), np.float32))
    A = W.er(300, 4.0, seed, cols=k)
    with sg.Handle() as h:
        assert len(h.multiply_host(A, B).col) == len(ref_product(A, B)["col"])
        row = int(rng.choice(np.nonzero(lens >= 2)[0]))
        at = int(ptr[row] + rng.integers(0, lens[row] - 1))
        if seed % 2:
            B.col[at], B.col[at + 1] = col[at + 1], col[at]
        else:
            B.col[at + 1] = col[at]
        with pytest.raises(sg.SpgemmError) as e:
            h.multiply_host(A, B)
        assert e.value.status == 1


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("table", [64, 256, 1024])
@pytest.mark.parametrize("stride", [1, 3, 700])
def test_hashed_rows_reuse_and_overflow(precision, table, stride):
    """Rows of a 27-point operator (their pattern stays in a warp's table from
    row to row) with random rows among them, which switch the reuse off or
    overflow; columns next to each other, or apart so that every slot holds
    one column. Runs twice, with the same bits: A is in CSR."""
    rng = np.random.default_rng(table + stride)
    S = W.stencil27(33, seed=stride)
    n, keep = S.rows, 9000
    lens = np.diff(S.rowptr)[:keep].astype(np.int64)
    r, c = np.repeat(np.arange(keep), lens), S.col[:lens.sum()].astype(np.int64)
    odd = rng.choice(keep, 400, replace=False)
    own = ~np.isin(r, odd)
    extra = [np.sort(rng.choice(n, rng.integers(2, 60), replace=False)) for _ in odd]
    r = np.concatenate([r[own], np.repeat(odd, [len(x) for x in extra])])
    c = np.concatenate([c[own], *extra])
    A = W.from_coo(keep, n, r, c, rng.uniform(-1, 1, len(r)).astype(np.float32))
    B = W.Csr(n, n * stride, S.rowptr, (S.col.astype(np.int64) * stride).astype(np.int32), S.val)
    ref = ref_product(A, B)
    out = []
    for _ in range(2):
        with sg.Handle(precision) as h:
            h.set_tuning(warp_table_max=table)
            out.append(h.multiply_host(A, B))
    assert_structure_equal(out[0].rowptr, out[0].col, ref["rowptr"], ref["col"])
    tol = plain_tolerance(ref) if precision == sg.PLAIN else compensated_tolerance(ref)
    assert_values_close(out[0].val, ref, tol)
    assert np.array_equal(out[0].col, out[1].col)
    assert np.array_equal(out[0].val.view(np.uint32), out[1].val.view(np.uint32))


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("lengths", [(4096,), (1500, 700, 1), (513, 90), (260,), (130, 7)])
def test_sorted_rows_of_few_long_entries(precision, lengths):
    """Rows of 1025 to 4096 products from one to some thirty entries: several
    warps of the team walk an entry together."""
    counts = [1025, 1500, 1537, 2047, 2048, 2049, 3000, 3073, 4095, 4096]
    A, B = rows_of(counts, 300_000, lengths, False, seed=lengths[0], empty=1)
    check_rows(A, B, precision, dict(warp_cap_max=0))


@pytest.mark.parametrize("m,k", [(1, 5), (37, 1), (300, 4000), (19000, 3)])
def test_copy_by_rows_per_warp(m, k):
    """C of few or many rows, short and long, so that a warp of the copy takes
    from 1 to 32 of them, with empty rows between."""
    rng = np.random.default_rng(m + k)
    rows = np.repeat(np.arange(m), rng.integers(0, min(k, 4) + 1, m))
    cols = np.concatenate([np.sort(rng.choice(k, n, replace=False)) for n in np.bincount(rows, minlength=m)]) \
        if len(rows) else rows
    A = W.from_coo(m, k, rows, cols, rng.uniform(-1, 1, len(rows)).astype(np.float32))
    B = W.er(k, 30.0, m, cols=900)
    check_rows(A, B, sg.PLAIN, {})


def grouped_rows(m, seed, n=60_000):
    """Rows of A with nine entries, three on each of three rows of B that share
    all their columns: how often neighbouring entries meet the same columns
    lies at the limit between hashed and sorted rows and depends on the order
    in which A's entries are taken."""
    rng = np.random.default_rng(seed)
    cols = np.sort(np.stack([rng.choice(n, 6, replace=False) for _ in range(3 * m)]), axis=1)
    B = W.from_coo(9 * m, n, np.repeat(np.arange(9 * m), 6), np.repeat(cols, 3, axis=0).ravel(),
                   rng.uniform(-1, 1, 54 * m).astype(np.float32))
    A = W.from_coo(m, 9 * m, np.repeat(np.arange(m), 9), np.arange(9 * m),
                   rng.uniform(-1, 1, 9 * m).astype(np.float32))
    perm = rng.permutation(9 * m)  # A's columns in any order: groups mixed
    order = np.argsort(perm, kind="stable")
    A = W.from_coo(m, 9 * m, np.repeat(np.arange(m), 9), perm, A.val)
    B = W.from_coo(9 * m, n, np.repeat(np.arange(9 * m), 6), B.col.reshape(-1, 6)[order].ravel(),
                   B.val.reshape(-1, 6)[order].ravel())
    return A, B


@pytest.mark.parametrize("a_format", ["csc", "csr"])
@pytest.mark.parametrize("m", [5, 40, 700])
def test_replayed_rows_keep_their_kernels(m, a_format):
    """The transpose of a CSC A leaves the entries of a row in any order, so a
    replay must not decide anew between hashing and sorting: its launches are
    sized for the planned run's lists."""
    db = DeviceBatch([grouped_rows(m, seed) for seed in (m, m + 1)], a_format)
    with sg.Handle() as h:
        h.batch_plan(db.A, db.B)
        refs = check_all(h, db.pairs)
        for graph in (True, True, True, False, False):
            h.batch_execute(graph=graph)
            check_all(h, db.pairs, refs=refs)


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("n", [40_000, (1 << 22) + 3])
@pytest.mark.parametrize("windows,width", [(1, 40), (2, 60), (4, 30), (16, 9), (5, 400), (3, 1)])
def test_sorted_rows_of_crowded_columns(precision, n, windows, width):
    """Rows of up to 4096 products whose columns lie in a few narrow windows
    far apart, each met many times (in most products, when a window is one
    column wide), with a few columns elsewhere: crowded buckets, cut finer or
    sorted as a whole."""
    rng = np.random.default_rng(windows * 1000 + width)
    counts = [c for c in COUNTS if c > 30] + [300, 700, 1500, 3001, 3999]
    starts = np.sort(rng.choice(n // 500 - 1, windows, replace=False)) * 500
    near = (starts[:, None] + np.arange(width)).ravel()
    ar, br, bc, k = [], [], [], 0
    for i, count in enumerate(counts):
        left = count
        while left > 0:
            cols = np.unique(np.concatenate([rng.choice(near, min(len(near), 45), replace=False),
                                             rng.integers(0, n, rng.integers(0, 3))]))[:left]
            br.append(np.full(len(cols), k))
            bc.append(cols)
            ar.append(i)
            k += 1
            left -= len(cols)
    br, bc = np.concatenate(br), np.concatenate(bc)
    vals = lambda x: rng.uniform(-1, 1, len(x)).astype(np.float32)
    A = W.from_coo(len(counts), k, np.array(ar), np.arange(k), vals(ar))
    B = W.from_coo(k, n, br, bc, vals(br))
    stats = check_rows(A, B, precision, dict(warp_cap_max=0))
    assert sum(stats["rows_per_symbolic_bin"][10:13]) == len(counts), stats
