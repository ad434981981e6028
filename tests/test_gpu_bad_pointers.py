"""Row and column pointers that no kernel may follow: each is refused as an
invalid argument, in either format of A, for B and in a batch, and the handle
stays usable."""
import numpy as np
import pytest

import spgemm_b200 as sg
from spgemm_b200 import workloads as W
from helpers import assert_structure_equal
from test_gpu_batch import DeviceBatch, ref_product

pytestmark = pytest.mark.gpu

BAD = [-2 ** 31, -1000, -1, 10 ** 6, 2 ** 31 - 1]


def broken(ptr, at, value):
    p = ptr.copy()
    p[at] = value
    return p


@pytest.mark.parametrize("deg", [3.0, 12.0, 40.0])
@pytest.mark.parametrize("operand", ["A csr", "A csc", "B"])
def test_bad_pointers_are_refused(operand, deg):
    A = W.er(700, deg, 1)
    ref = ref_product(A, A)
    csc = A.to_csc()
    ptr = csc.colptr if operand == "A csc" else A.rowptr
    with sg.Handle() as h:
        for at in (0, 1, 350, 699, 700):
            for value in BAD + [int(ptr[max(at - 1, 0)]) - 1]:
                a, b = A, A
                if operand == "A csr":
                    a = W.Csr(700, 700, broken(A.rowptr, at, value), A.col, A.val)
                elif operand == "A csc":
                    a = W.Csc(700, 700, broken(csc.colptr, at, value), csc.rowidx, csc.val)
                else:
                    b = W.Csr(700, 700, broken(A.rowptr, at, value), A.col, A.val)
                with pytest.raises(sg.SpgemmError) as e:
                    h.multiply_host(a, b)
                assert e.value.status == 1, (at, value)
        C = h.multiply_host(A, A)
        assert_structure_equal(C.rowptr, C.col, ref["rowptr"], ref["col"])


@pytest.mark.parametrize("a_format", ["csr", "csc"])
def test_bad_pointers_in_a_batch(a_format):
    A = W.er(300, 5.0, 2)
    good = DeviceBatch([(A, A), (A, A)], a_format)
    for value in BAD:
        d = DeviceBatch([(A, A), (A, A)], a_format)
        d.keep[0][0][150] = value  # the first A's pointers
        with sg.Handle() as h:
            with pytest.raises(sg.SpgemmError) as e:
                h.batch_plan(d.A, d.B)
            assert e.value.status == 1, value
            h.batch_plan(good.A, good.B)
