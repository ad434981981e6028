"""Calls repeated on one handle within a product: what one call leaves behind
must not reach the next one's result."""
import ctypes as C

import numpy as np
import pytest

import spgemm_b200 as sg
from spgemm_b200 import workloads as W
from helpers import assert_structure_equal, assert_values_close, compensated_tolerance, plain_tolerance
from test_gpu_batch import DeviceBatch, ref_product
from test_gpu_legacy import _coo_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a_format", ["csr", "csc"])
@pytest.mark.parametrize("precision,long_rows", [(sg.PLAIN, 0), (sg.PLAIN, 1), (sg.PLAIN, 2), (sg.PLAIN, 3),
                                                 (sg.COMPENSATED, 2)])
def test_numeric_again_after_one_symbolic(precision, long_rows, a_format):
    """spgemm_numeric may be called again after one spgemm_symbolic: each call
    fills its own buffers whole, long rows included."""
    import torch
    A = W.rmat(13, 16, 5)
    ref = ref_product(A, A)
    tol = plain_tolerance(ref) if precision == sg.PLAIN else compensated_tolerance(ref)
    d = DeviceBatch([(A, A)], a_format)
    with sg.Handle(precision) as h:
        h.set_tuning(long_rows=long_rows)
        nnz = h.symbolic(d.A[0], d.B[0])
        assert nnz == len(ref["col"])
        assert h.stats()["rows_per_symbolic_bin"][9] > 0
        for _ in range(3):
            ptr = torch.full((A.rows + 1,), -1, dtype=torch.int32, device="cuda")
            col = torch.full((nnz,), -1, dtype=torch.int32, device="cuda")
            val = torch.full((nnz,), float("nan"), device="cuda")
            h.numeric(ptr.data_ptr(), col.data_ptr(), val.data_ptr())
            assert_structure_equal(ptr.cpu().numpy(), col.cpu().numpy(), ref["rowptr"], ref["col"])
            assert_values_close(val.cpu().numpy(), ref, tol)


def test_host_call_with_empty_row_ranges():
    """C copied back in pieces, some of them without rows (one row holds most
    of C), then in one piece: long rows are computed in the piece they are in."""
    rng = np.random.default_rng(3)
    A = W.rmat(12, 16, 6)
    rows = np.repeat(np.arange(A.rows), np.diff(A.rowptr))
    extra = np.sort(rng.choice(A.cols, A.cols // 2, replace=False))
    r = np.concatenate([rows[rows != 7], np.full(len(extra), 7)])
    c = np.concatenate([A.col[rows != 7], extra])
    A = W.from_coo(A.rows, A.cols, r, c, rng.uniform(-1, 1, len(r)).astype(np.float32))
    ref = ref_product(A, A)
    with sg.Handle() as h:
        for chunk in (4096, 0, 1 << 16):
            h.set_copy_chunk(chunk)
            C = h.multiply_host(A, A)
            assert_structure_equal(C.rowptr, C.col, ref["rowptr"], ref["col"])
            assert_values_close(C.val, ref, plain_tolerance(ref))


def overflowing(m=600, n=40_000, seed=8):
    """Rows of about 400 distinct columns, each product's column met about
    three times (so the rows are hashed, and overflow the table), with some
    long rows."""
    rng = np.random.default_rng(seed)
    groups = [np.sort(rng.choice(n, 20, replace=False)) for _ in range(200)]
    B = W.from_coo(600, n, np.repeat(np.arange(600), 20), np.concatenate([groups[k // 3] for k in range(600)]),
                   rng.uniform(-1, 1, 12000).astype(np.float32))
    r, c = [], []
    for i in range(m):
        g = np.arange(200) if i % 50 == 0 else np.sort(rng.choice(200, 20, replace=False))
        r += [i] * (3 * len(g))
        c += np.sort(np.concatenate([3 * g, 3 * g + 1, 3 * g + 2])).tolist()
    return W.from_coo(m, 600, np.array(r), np.array(c), rng.uniform(-1, 1, len(r)).astype(np.float32)), B


@pytest.mark.parametrize("operands", ["overflowing", "rmat"])
def test_symbolic_pass_again_after_one_analysis(operands):
    """mm.h: cudaBinGEMM (or cudaSimpleGEMM) again after one cudaInitGEMM, and
    cudaMergeGEMM again, leave the same C as one call of each."""
    L = sg.lib()
    L.spgemm_set_verbose(0)
    L.spgemm_set_exit_on_error(0)
    try:
        A, B = overflowing() if operands == "overflowing" else (W.rmat(12, 12, 8, values="sym"),) * 2
        ref = ref_product(A, B)
        if operands == "overflowing":
            with sg.Handle() as h:
                h.multiply_host(A, B)
                assert h.stats()["warp_overflow_rows"] > 400
        ta, tb = _coo_of(A, True), _coo_of(B, False)
        Ah = L.cudaCOO2CM(sg.COO(C.cast(ta, C.POINTER(sg.Triplet)), A.nnz, A.cols, A.rows, sg.COL_MAJOR))
        Bh = L.cudaCOO2CM(sg.COO(C.cast(tb, C.POINTER(sg.Triplet)), B.nnz, B.cols, B.rows, sg.ROW_MAJOR))
        Cm = L.cudaInitGEMM(Ah, Bh)
        for again in range(4):
            (L.cudaSimpleGEMM if again == 2 else L.cudaBinGEMM)(Ah, Bh, Cm)
            assert L.spgemm_legacy_status() == 0
            for _ in range(1 + again % 2):
                L.cudaMergeGEMM(Cm)
                assert L.spgemm_legacy_status() == 0
                R = sg.CM()
                assert L.spgemm_get_result(C.byref(R)) == 0
                got = [np.ctypeslib.as_array(p, (k,)).copy()
                       for p, k in ((R.ptr, R.num_rows + 1), (R.idx, R.nnz), (R.val, R.nnz))]
                L.cmFree(C.byref(R))
                assert_structure_equal(got[0], got[1], ref["rowptr"], ref["col"])
                assert_values_close(got[2], ref, plain_tolerance(ref))
        for M in (Ah, Bh):
            L.cmFree(C.byref(M))
    finally:
        L.spgemm_set_verbose(1)
        L.spgemm_set_exit_on_error(1)


def test_workspace_without_long_rows():
    """A product without long rows allocates nothing for them: 4 M rows of one
    entry take at most 130 bytes a row beside operands and output."""
    import torch
    m = 1 << 22
    ptr = torch.arange(m + 1, dtype=torch.int32, device="cuda")
    idx = torch.randint(0, m, (m,), dtype=torch.int32, device="cuda")
    val = torch.ones(m, device="cuda")
    a = sg.device_cm(ptr.data_ptr(), idx.data_ptr(), val.data_ptr(), m, m, m, sg.ROW_MAJOR)
    with sg.Handle() as warm:  # kernels loaded, contexts made
        assert warm.symbolic(a, a) == m
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with sg.Handle() as h:
        assert h.symbolic(a, a) == m
        used = free - torch.cuda.mem_get_info()[0]
    assert used <= 130 * m + (8 << 20), used / m


def test_products_of_changing_shapes_on_one_handle():
    """The workspace's arrays move when a product of another shape comes:
    larger and smaller rows, columns and entries, both formats of A, with and
    without long rows."""
    rng = np.random.default_rng(9)
    shapes = [(50, 4000, 3000, 40.0), (30_000, 60, 500, 2.0), (700, 700, 700, 9.0), (1, 50_000, 2000, 3000.0),
              (9000, 9000, 9000, 6.0), (64, 64, 64, 60.0), (20_000, 20_000, 40_000, 3.0)]
    pairs = [(W.er(m, d, i, cols=k), W.er(k, 8.0, 50 + i, cols=n)) for i, (m, k, n, d) in enumerate(shapes)]
    pairs.append((W.rmat(11, 16, 3),) * 2)
    refs = [ref_product(A, B) for A, B in pairs]
    with sg.Handle() as h:
        for i in rng.permutation(np.repeat(np.arange(len(pairs)), 3)):
            A, B = pairs[i]
            C = h.multiply_host(A.to_csc() if rng.random() < 0.5 else A, B)
            assert_structure_equal(C.rowptr, C.col, refs[i]["rowptr"], refs[i]["col"])
            assert_values_close(C.val, refs[i], plain_tolerance(refs[i]))
