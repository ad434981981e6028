"""Calls repeated on one handle within a product: what one call leaves behind
must not reach the next one's result."""
import numpy as np
import pytest

import spgemm_b200 as sg
from spgemm_b200 import workloads as W
from helpers import assert_structure_equal, assert_values_close, compensated_tolerance, plain_tolerance
from test_gpu_batch import DeviceBatch, ref_product

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
