"""Which kernel merges a row: the names the profile reports, so that a change
of the rules cannot leave a kernel, or a table's overflow, untested. Structure
exactly, values within the bounds of helpers.py, against the FP64 oracle."""
import numpy as np
import pytest

import spgemm_b200 as sg
from spgemm_b200 import workloads as W
from helpers import assert_structure_equal, assert_values_close, compensated_tolerance, plain_tolerance
from test_gpu_batch import DeviceBatch, check_all, ref_product

pytestmark = pytest.mark.gpu


def product(A, B, precision=sg.PLAIN, csc=False, **tuning):
    """The checked product; returns the launched first-pass kernels and the
    rows that overflowed their table or bitmap."""
    ref = ref_product(A, B)
    with sg.Handle(precision) as h:
        h.set_tuning(**tuning)
        h.set_profiling(True)
        C = h.multiply_host(A.to_csc() if csc else A, B)
        names = {n for n in h.kernel_times() if n.startswith("k_fused_")}
        for n in [n for n in names if n.startswith("k_fused_warp+cols")]:  # one launch of both tables
            names |= {n.replace("+cols", ""), n.replace("warp+", "")}
        overflow = h.stats()["warp_overflow_rows"]
    assert_structure_equal(C.rowptr, C.col, ref["rowptr"], ref["col"])
    tol = plain_tolerance(ref) if precision == sg.PLAIN else compensated_tolerance(ref)
    assert_values_close(C.val, ref, tol)
    return names, overflow


def renumbered(M, seed):
    """M with its rows and columns numbered at random."""
    perm = np.random.default_rng(seed).permutation(M.rows)
    r = perm[np.repeat(np.arange(M.rows), np.diff(M.rowptr))]
    return W.from_coo(M.rows, M.cols, r, perm[M.col], M.val)


def rows_sharing(outputs, sharing, run, n, seed=0):
    """A and B such that row i of A*B has outputs[i] columns, `sharing`
    products each: A's entries are that many B rows of one pattern, whose
    columns come in runs of `run`, the runs apart, spread over [0, n)."""
    rng = np.random.default_rng(seed)
    br, bc, k = [], [], 0
    for o in outputs:
        starts = np.sort(rng.choice(n // (3 * run) - 1, -(-o // run), replace=False)) * (3 * run)
        cols = (starts[:, None] + np.arange(run)).ravel()[:o]
        for _ in range(sharing):
            br.append(np.full(o, k))
            bc.append(cols)
            k += 1
    m = len(outputs)
    br, bc = np.concatenate(br), np.concatenate(bc)
    A = W.from_coo(m, k, np.repeat(np.arange(m), sharing), np.arange(k), rng.uniform(-1, 1, k).astype(np.float32))
    return A, W.from_coo(k, n, br, bc, rng.uniform(-1, 1, len(br)).astype(np.float32))


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("csc", [False, True])
def test_grids_are_grouped_and_numbered_at_random_are_not(precision, csc):
    S = W.stencil27(36, seed=1)
    names, overflow = product(S, S, precision, csc)
    assert "k_fused_warp<2>" in names and "k_fused_cols<2>" not in names, names
    assert overflow == 0
    R = renumbered(S, 2)
    names, overflow = product(R, R, precision, csc)
    assert "k_fused_cols<2>" in names, names
    assert overflow == 0


@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
@pytest.mark.parametrize("table,bin_", [(256, 2), (512, 3), (1024, 4)])
@pytest.mark.parametrize("run", [1, 4])
def test_outputs_around_a_tables_limit(precision, table, bin_, run):
    """Rows of up to 4/5 of the slots stay, one more and they are redone."""
    slots = table if run == 1 else table // 2
    per_slot = 1 if run == 1 else (4 if precision == sg.PLAIN or bin_ == 2 else 2)
    limit = slots * 4 // 5
    fits = [limit * per_slot - d for d in (0, 1, 2, 3)] + [table // 2, 30, limit // 2]
    fits = [o for o in fits if 2 * o <= 2048]
    beyond = [o for o in (limit * per_slot + d for d in (1, 2, 40)) if 2 * o <= 2048]
    outputs = (fits + beyond) * 5
    A, B = rows_sharing(outputs, 2, run, 90_000, seed=table + run)
    names, overflow = product(A, B, precision, warp_table_max=table)
    assert ("k_fused_cols<%d>" if run == 1 else "k_fused_warp<%d>") % bin_ in names, names
    assert overflow == 5 * len(beyond), (names, overflow)


@pytest.mark.parametrize("table,bin_", [(256, 2), (512, 3), (1024, 4)])
@pytest.mark.parametrize("over", [-70, -1, 0, 1, 70])
@pytest.mark.parametrize("run", [1, 4])
def test_spans_around_the_packed_order(table, bin_, over, run):
    """The table's order packs a column (or group) offset above a slot index;
    rows whose span leaves no room take another kernel."""
    limit = 1 << ((26 - bin_) if run == 1 else (28 - bin_))
    n = limit + over
    A, B = rows_sharing([300, 101, 150, 203], 3, run, 50_000, seed=bin_)
    stretched = B.col.astype(np.int64)
    stretched[stretched >= 25_000] += n - 50_000  # spans up to n
    last = np.isin(np.arange(len(B.col)), B.rowptr[1:] - 1)
    stretched[last] = n - 1
    first = np.isin(np.arange(len(B.col)), B.rowptr[:-1])
    stretched[first] = 0
    B = W.Csr(B.rows, n, B.rowptr, stretched.astype(np.int32), B.val)
    assert (np.diff(stretched)[np.diff(np.repeat(np.arange(B.rows), np.diff(B.rowptr))) == 0] > 0).all()
    product(A, B, sg.PLAIN, warp_table_max=table)
    product(A, B, sg.COMPENSATED, warp_table_max=table)


def one_of_each(rng):
    """One product with rows for each kernel of the default tuning and (with
    sorting off) for the block kernels."""
    n = 50_000
    parts = [rows_sharing([3] * 40, 2, 1, n), rows_sharing([7] * 40, 2, 1, n), rows_sharing([12] * 40, 2, 1, n),
             rows_sharing([100] * 64, 3, 1, 4000), rows_sharing([20] * 64, 2, 1, n), rows_sharing([60] * 64, 3, 1, n),
             rows_sharing([120] * 64, 3, 4, n), rows_sharing([150] * 64, 3, 1, n),
             rows_sharing([200] * 64, 1, 1, n), rows_sharing([400] * 64, 1, 1, n), rows_sharing([900] * 64, 1, 1, n),
             rows_sharing([1900] * 64, 1, 1, n), rows_sharing([4000] * 64, 1, 1, n)]
    m = k = 0
    ar, ac, br, bc = [], [], [], []
    for A, B in parts:
        m0 = -(-m // 64) * 64  # a block of row analysis each
        ar.append(np.repeat(np.arange(A.rows), np.diff(A.rowptr)) + m0)
        ac.append(A.col + k)
        br.append(np.repeat(np.arange(B.rows), np.diff(B.rowptr)) + k)
        bc.append(B.col)
        m, k = m0 + A.rows, k + B.rows
    ar, ac, br, bc = (np.concatenate(x) for x in (ar, ac, br, bc))
    val = lambda x: rng.uniform(-1, 1, len(x)).astype(np.float32)
    A, B = W.from_coo(m, k, ar, ac, val(ar)), W.from_coo(k, n, br, bc, val(br))
    return A, B


@pytest.mark.parametrize("esc", [True, False])
def test_every_first_pass_kernel_runs(esc):
    A, B = one_of_each(np.random.default_rng(1))
    names, overflow = product(A, B, **({} if esc else dict(esc_p_min=4096)))
    want = {"k_fused_tiny", "k_fused_bits", "k_fused_warp<0>", "k_fused_warp<2>", "k_fused_cols<2>"}
    want |= {f"k_fused_esc<{t}>" for t in (32, 64, 128, 256, 512)} if esc else {"k_fused_mid"}
    assert want <= names, want - names
    if not esc:
        names, _ = product(A, B, esc_p_min=4096, mid_cols=0, warp_p_max=100)
        assert {"k_fused_block<11>", "k_fused_block<12>", "k_fused_block<13>"} <= names, names


@pytest.mark.parametrize("a_format", ["csc", "csr"])
def test_replays_of_both_tables(a_format):
    S = W.stencil27(14, seed=3)
    db = DeviceBatch([(S, S), (renumbered(S, 4),) * 2, (renumbered(S, 5),) * 2], a_format)
    with sg.Handle() as h:
        h.batch_plan(db.A, db.B)
        refs = check_all(h, db.pairs)
        for graph in (True, True, False):
            h.batch_execute(graph=graph)
            check_all(h, db.pairs, refs=refs)


@pytest.mark.parametrize("esc", [True, False])
@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
def test_rows_of_many_entries_and_few_products(precision, esc):
    """Rows of A with thousands of entries of which few meet a product (most
    rows of B are empty), from one product to 4096: a block walks them."""
    rng = np.random.default_rng(4)
    k, n = 60_000, 30_000
    blens = np.where(rng.random(k) < 0.1, rng.integers(1, 9, k), 0)
    br = np.repeat(np.arange(k), blens)
    bc = np.concatenate([np.sort(rng.choice(n, x, replace=False)) for x in blens])
    empty, full = np.nonzero(blens == 0)[0], np.nonzero(blens)[0]
    lists = []
    for entries in (1024, 1025, 3000, 9000):  # at most 512 rows of 1025 fit A
        for used in (0, 1, 4, 20, 60, 200, 500, 800):
            lists.append(np.sort(np.concatenate([rng.choice(empty, entries - used, replace=False),
                                                 rng.choice(full, used, replace=False)])))
    val = lambda x: rng.uniform(-1, 1, len(x)).astype(np.float32)
    ar, ac = np.repeat(np.arange(len(lists)), [len(x) for x in lists]), np.concatenate(lists)
    A, B = W.from_coo(len(lists), k, ar, ac, val(ar)), W.from_coo(k, n, br, bc, val(br))
    names, _ = product(A, B, precision, **({} if esc else dict(esc_p_min=4096)))
    assert ("k_fused_esc<512>" in names) == esc, names


def expanded(A, B):
    """Every product of A*B in order: (row, column, 64-bit value)."""
    lens = np.diff(B.rowptr).astype(np.int64)[A.col]
    own = np.repeat(np.arange(len(A.col)), lens)
    pos = np.repeat(B.rowptr[A.col].astype(np.int64) - (np.cumsum(lens) - lens), lens) + np.arange(lens.sum())
    row = np.repeat(np.arange(A.rows), np.diff(A.rowptr))[own]
    return row, B.col[pos], A.val.astype(np.float64)[own] * B.val.astype(np.float64)[pos]


@pytest.mark.parametrize("esc", [True, False])
@pytest.mark.parametrize("precision", [sg.PLAIN, sg.COMPENSATED])
def test_infinities_and_nans(precision, esc):
    """Operands with infinities and NaNs, the all-ones pattern (the hash's mark
    of an absent value) among them, in every kernel: the structure is kept; a
    sum with a NaN, or infinities of both signs, is NaN; one with infinities of
    one sign is that infinity (the compensated forms may make it NaN); all
    other sums stay within the bounds."""
    rng = np.random.default_rng(2)
    A, B = one_of_each(rng)
    for M, share in ((A, 0.02), (B, 0.003)):
        bad = rng.random(len(M.val)) < share
        kinds = np.array([np.inf, -np.inf, np.nan, 0.0], np.float32)
        kinds[3:] = np.array([0xffffffff], np.uint32).view(np.float32)
        bits = M.val.view(np.uint32)
        bits[bad] = kinds.view(np.uint32)[rng.integers(0, 4, bad.sum())]
    row, col, val = expanded(A, B)
    key = row.astype(np.int64) * B.cols + col
    order = np.argsort(key, kind="stable")
    start = np.nonzero(np.diff(key[order], prepend=-1))[0]
    with np.errstate(all="ignore"):
        total = np.add.reduceat(val[order], start)
        absum = np.add.reduceat(np.abs(val[order]), start)
    ref = {"val": total, "absum": absum, "nterms": np.diff(np.append(start, len(key)))}
    with sg.Handle(precision) as h:
        h.set_tuning(**({} if esc else dict(esc_p_min=4096)))
        C = h.multiply_host(A, B)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(row[order][start], minlength=A.rows))])
    assert_structure_equal(C.rowptr, C.col, ptr, col[order][start])
    finite = np.isfinite(total)
    assert 0.05 < finite.mean() < 1.0
    one_sign = np.isinf(total)
    assert np.isnan(C.val[np.isnan(total)]).all()
    if precision == sg.PLAIN:
        assert np.array_equal(C.val[one_sign], total[one_sign].astype(np.float32))
    else:
        assert not np.isfinite(C.val[one_sign]).any()
    part = {k: v[finite] for k, v in ref.items()}
    tol = plain_tolerance(part) if precision == sg.PLAIN else compensated_tolerance(part)
    assert_values_close(C.val[finite], part, tol)


@pytest.mark.parametrize("csc", [False, True])
def test_more_rows_than_the_scan_sums_by_itself(csc):
    """33.6 million rows: above 8192 tiles of row counts the tile sums are
    scanned in a launch of their own. Every third row is empty, the others have
    one entry of A, and every row of B has two."""
    import torch
    m, k = 33_600_001, 1000
    i = torch.arange(m, device="cuda")
    has = i % 3 != 0
    rows = i[has]
    kk = (rows * 7919) % k
    ptr = torch.zeros(m + 1, dtype=torch.int32, device="cuda")
    ptr[1:] = torch.cumsum(has, 0).int()
    val = (rows % 13 + 1).float()
    bptr = (2 * torch.arange(k + 1, device="cuda")).int()
    bcol = torch.stack([torch.arange(k, device="cuda") % 50, 60 + torch.arange(k, device="cuda") % 40], 1).int().reshape(-1)
    bval = (torch.arange(2 * k, device="cuda") % 11 - 5).float()
    if csc:
        order = torch.argsort(kk, stable=True)
        cptr = torch.zeros(k + 1, dtype=torch.int32, device="cuda")
        cptr[1:] = torch.cumsum(torch.bincount(kk, minlength=k), 0).int()
        arrays = (cptr, rows[order].int(), val[order])
    else:
        arrays = (ptr, kk.int(), val)
    a = sg.device_cm(*(t.data_ptr() for t in arrays), len(rows), m, k, sg.COL_MAJOR if csc else sg.ROW_MAJOR)
    b = sg.device_cm(bptr.data_ptr(), bcol.data_ptr(), bval.data_ptr(), 2 * k, k, 100, sg.ROW_MAJOR)
    with sg.Handle() as h:
        nnz = h.symbolic(a, b)
        assert nnz == 2 * len(rows)
        out = (torch.empty(m + 1, dtype=torch.int32, device="cuda"), torch.empty(nnz, dtype=torch.int32, device="cuda"),
               torch.empty(nnz, device="cuda"))
        h.numeric(*(t.data_ptr() for t in out))
    assert torch.equal(out[0], 2 * ptr)
    assert torch.equal(out[1].view(-1, 2), bcol.view(-1, 2)[kk])
    assert torch.equal(out[2].view(-1, 2), val[:, None] * bval.view(-1, 2)[kk])
