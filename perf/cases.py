"""Performance cases: the products and conversions that programs run through
the library's public entry points, with their inputs, passes and exact values.

A case is a dict of plain values; `family` says which path it takes:

* ``er``        C = A*B, entries spread uniformly (Poisson row lengths)
* ``rmat``      C = A*A of an R-MAT graph: power-law rows, up to tens of
                thousands of entries
* ``stencil``   C = A*A of a 27-point stencil on an s^3 grid, magnitudes
                log-uniform over eight decades with random signs
* ``galerkin``  two chained products P^T (A P), the coarse operator of a
                multigrid level, P aggregating 2x2x2 points
* ``batch``     many independent products of uneven size, planned once and
                replayed as one CUDA graph
* ``host``      the host-array call: operands in pinned host memory, C back in
                pinned host memory
* ``coo``       device triplets in any order to CSR or CSC

The first four go through the handle's two-phase call on device arrays
(symbolic, then numeric into arrays of the size it reports), in plain or
compensated FP32, with A as CSC (the layout the call protocol of the reference
engine uses) or CSR. Inputs are drawn on the device, from the seed alone.
"""
import math

import numpy as np
import torch

import spgemm_b200 as sg

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
RMAT = (0.57, 0.19, 0.19)   # quadrant probabilities a, b, c of the R-MAT sampler
MARGINAL_BIT = 0.24         # chance of a 1 in each bit of an R-MAT column (b + d)
CHUNK = 150_000_000         # products expanded at once by the 64-bit product


def listed():
    return [
        # The smallest calls: a coarse-level or per-element operator, where
        # launches and host round trips are all there is.
        {"name": "er_500", "family": "er", "m": 500, "k": 500, "n": 500, "deg_a": 4.0, "deg_b": 4.0,
         "same": True, "csc": False, "compensated": False},
        # The plain configuration: 4096 x 4096, 8 entries a row, A*A.
        {"name": "er_4096", "family": "er", "m": 4096, "k": 4096, "n": 4096, "deg_a": 8.0, "deg_b": 8.0,
         "same": True, "csc": True, "compensated": False},
        # One rectangular product of the size the batch draws from, called by
        # itself: rows of a few hundred products with hardly a repeated column.
        {"name": "er_rect_100003", "family": "er", "m": 100003, "k": 60013, "n": 80021, "deg_a": 16.0,
         "deg_b": 13.0, "same": False, "csc": False, "compensated": False},
        # Road-network degree: a million very short rows, where the passes over
        # rows and pointers weigh as much as the products.
        {"name": "er_1000003_deg3", "family": "er", "m": 1000003, "k": 1000003, "n": 1000003, "deg_a": 3.0,
         "deg_b": 3.0, "same": True, "csc": False, "compensated": False},
        # A mid-size power-law graph whose order is no power of two, in the
        # compensated form: long rows accumulate in FP64.
        {"name": "rmat_30011_comp", "family": "rmat", "n": 30011, "ef": 12.0, "csc": True, "compensated": True},
        # The headline: R-MAT 2^18, average degree 16, 2.9e9 products.
        {"name": "rmat_262144", "family": "rmat", "n": 262144, "ef": 16.0, "csc": True, "compensated": False},
        # Structured: 27-point stencil on 96^3, plain ...
        {"name": "stencil_96", "family": "stencil", "s": 96, "csc": True, "compensated": False},
        # ... and an odd, smaller grid in the compensated form that cancelling
        # operators are run with.
        {"name": "stencil_61_comp", "family": "stencil", "s": 61, "csc": False, "compensated": True},
        # Multigrid set-up: the Galerkin product of a 64^3 level.
        {"name": "galerkin_64_comp", "family": "galerkin", "s": 64, "compensated": True},
        # A serving loop's batch: products of uneven size in one graph replay.
        {"name": "batch_48", "family": "batch", "count": 48, "n_lo": 1000, "n_hi": 40000, "deg_lo": 4.0,
         "deg_hi": 32.0, "sizes_seed": 7, "compensated": False},
        # A host program's call: pinned operands up, the product, C back.
        {"name": "host_er_20011", "family": "host", "n": 20011, "deg": 16.0, "csc": True, "compensated": False},
        # Assembly: a graph's edge list in arrival order to CSR.
        {"name": "coo_rmat_262144", "family": "coo", "n": 262144, "ef": 16.0, "col_major": False},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same families and ranges."""
    family = rng.choice(["er", "er", "er", "rmat", "rmat", "stencil", "stencil", "galerkin", "batch",
                         "host", "coo"])
    comp = rng.random() < 0.35
    csc = rng.random() < 0.5
    if family == "er":
        deg_a = round(_log_uniform(rng, 2, 32), 2)
        deg_b = round(_log_uniform(rng, 2, 32), 2)
        top = min(1.0e6, 2.0e8 / (deg_a * deg_b))   # at most 2e8 products
        m = int(_log_uniform(rng, 300, top))
        same = rng.random() < 0.4
        k = m if same else max(100, int(m * _log_uniform(rng, 0.4, 2.5)))
        n = m if same else max(100, int(m * _log_uniform(rng, 0.4, 2.5)))
        return {"family": "er", "m": m, "k": k, "n": n, "deg_a": deg_a, "deg_b": deg_a if same else deg_b,
                "same": same, "csc": csc, "compensated": comp}
    if family == "rmat":
        return {"family": "rmat", "n": int(_log_uniform(rng, 1000, 200000)),
                "ef": round(rng.uniform(4, 16), 2), "csc": csc, "compensated": comp}
    if family == "stencil":
        return {"family": "stencil", "s": int(_log_uniform(rng, 9, 92)), "csc": csc, "compensated": comp}
    if family == "galerkin":
        return {"family": "galerkin", "s": 2 * int(_log_uniform(rng, 5, 36)), "compensated": comp}
    if family == "batch":
        return {"family": "batch", "count": rng.randint(8, 48), "n_lo": 1000, "n_hi": rng.randint(5000, 40000),
                "deg_lo": 4.0, "deg_hi": round(rng.uniform(12, 32), 2), "sizes_seed": rng.randint(0, 10 ** 6),
                "compensated": comp}
    if family == "host":
        return {"family": "host", "n": int(_log_uniform(rng, 500, 40000)), "deg": round(rng.uniform(4, 16), 2),
                "csc": csc, "compensated": comp}
    return {"family": "coo", "n": int(_log_uniform(rng, 2000, 262144)), "ef": round(rng.uniform(4, 16), 2),
            "col_major": csc}


# ---------------------------------------------------------------------------
# Operands, on the device
# ---------------------------------------------------------------------------

class Csr:
    """rowptr / col int32, val float32 tensors; columns ascending in a row."""

    def __init__(self, rows, cols, rowptr, col, val):
        self.rows, self.cols, self.rowptr, self.col, self.val = rows, cols, rowptr, col, val

    @property
    def nnz(self):
        return self.col.numel()

    def row_of(self):
        return torch.repeat_interleave(torch.arange(self.rows, device=DEV),
                                       (self.rowptr[1:] - self.rowptr[:-1]).long())

    def csc(self):
        """(colptr, rowidx, val): rows ascending in a column."""
        order = torch.argsort(self.col, stable=True)
        return _pointers(self.col.long(), self.cols), self.row_of()[order].int(), self.val[order]


def _pointers(major, n_major):
    ptr = torch.zeros(n_major + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(major, minlength=n_major)[:n_major], 0)
    return ptr.int()


def _from_keys(keys, rows, cols, val):
    r = torch.div(keys, cols, rounding_mode="floor")
    return Csr(rows, cols, _pointers(r, rows), (keys - r * cols).int(), val)


def _rng(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + salt)


def _uniform(g, n, low, high):
    return torch.rand(n, generator=g, device=DEV) * (high - low) + low


def _skewed_columns(g, count, n):
    """Columns of the R-MAT column marginal, folded into [0, n)."""
    c = torch.zeros(count, dtype=torch.int64, device=DEV)
    for _ in range(max(1, math.ceil(math.log2(n)))):
        c = 2 * c + (torch.rand(count, generator=g, device=DEV) < MARGINAL_BIT)
    return torch.where(c < n, c, c // 2)


# A random pattern belongs to the case, so that every seed's C has as many
# entries; the seed relabels its rows and columns (the inner dimension of a
# product alike in both factors) and draws the values.

def _poisson_pattern(rows, cols, deg, salt, skewed=False):
    """Poisson(deg) entries a row, columns uniform (or skewed), repeats dropped."""
    g = _rng(0, salt)
    lens = torch.poisson(torch.full((rows,), float(deg), device=DEV), generator=g).long()
    r = torch.repeat_interleave(torch.arange(rows, device=DEV), lens)
    c = (_skewed_columns(g, r.numel(), cols) if skewed
         else torch.randint(0, cols, (r.numel(),), generator=g, device=DEV))
    keys = torch.unique(r * cols + c)
    return torch.div(keys, cols, rounding_mode="floor"), keys % cols


def _rmat_edges(n, ef, g):
    """About ef * n edges of an R-MAT graph on n vertices, in arrival order."""
    a, b, c = RMAT
    scale = max(1, math.ceil(math.log2(n)))
    want = int(ef * n * 4 ** scale / float(n) ** 2) if n < 1 << scale else int(ef * n)
    r = torch.zeros(want, dtype=torch.int64, device=DEV)
    q = torch.zeros(want, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        u = torch.rand(want, generator=g, device=DEV)
        r = 2 * r + (u >= a + b)
        q = 2 * q + (((u >= a) & (u < a + b)) | (u >= a + b + c))
    keep = (r < n) & (q < n)
    return r[keep][: int(ef * n)], q[keep][: int(ef * n)]


def _labels(n, g, rotate=False):
    """New labels of n indices: any order, or a rotation, which keeps the
    neighbourhoods of popular indices."""
    if rotate:
        return (torch.arange(n, device=DEV) + torch.randint(0, n, (1,), generator=g, device=DEV)) % n
    return torch.randperm(n, generator=g, device=DEV)


def _relabelled(pattern, row_labels, col_labels, g, low=-1.0, high=1.0):
    r, c = pattern
    rows, cols = row_labels.numel(), col_labels.numel()
    keys = torch.sort(row_labels[r] * cols + col_labels[c]).values
    return _from_keys(keys, rows, cols, _uniform(g, keys.numel(), low, high))


def _rmat(n, ef, g):
    r, q = _rmat_edges(n, ef, _rng(0, 1))
    keys = torch.unique(r * n + q)
    labels = _labels(n, g, rotate=True)
    return _relabelled((torch.div(keys, n, rounding_mode="floor"), keys % n), labels, labels, g, 1.0, 0.0)


def _er_pair(m, k, n, deg_a, deg_b, same, g, salt=0, skewed=False):
    """Independent A (m x k) and B (k x n), or one square matrix twice."""
    A = _poisson_pattern(m, k, deg_a, salt, skewed)
    rows = _labels(m, g, skewed)
    if same:
        M = _relabelled(A, rows, rows, g)
        return M, M
    B = _poisson_pattern(k, n, deg_b, salt + 1, skewed)
    inner, cols = _labels(k, g, skewed), _labels(n, g, skewed)
    return _relabelled(A, rows, inner, g), _relabelled(B, inner, cols, g)


def _stencil(s, g, diffusion=False):
    """27-point stencil: signs random and magnitudes log-uniform in
    [1e-4, 1e4], or a diffusion operator with varying coefficients."""
    n = s ** 3
    i = torch.arange(n, device=DEV)
    x, y, z = i % s, (i // s) % s, i // (s * s)
    keys = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                ok = ((x + dx >= 0) & (x + dx < s) & (y + dy >= 0) & (y + dy < s) & (z + dz >= 0) & (z + dz < s))
                keys.append((i * n + i + dx + s * (dy + s * dz))[ok])
    keys = torch.sort(torch.cat(keys)).values
    if diffusion:
        on_diagonal = torch.div(keys, n, rounding_mode="floor") == keys % n
        v = torch.where(on_diagonal, 26.0, -1.0) * _uniform(g, keys.numel(), 0.5, 1.5)
    else:
        sign = torch.where(torch.rand(keys.numel(), generator=g, device=DEV) < 0.5, -1.0, 1.0)
        v = sign * torch.pow(10.0, _uniform(g, keys.numel(), -4.0, 4.0))
    return _from_keys(keys, n, n, v.float())


def _prolongator(s):
    h = s // 2
    i = torch.arange(s ** 3, device=DEV)
    x, y, z = i % s, (i // s) % s, i // (s * s)
    agg = x // 2 + h * (y // 2 + h * (z // 2))
    return Csr(s ** 3, h ** 3, torch.arange(s ** 3 + 1, device=DEV).int(), agg.int(),
               torch.ones(s ** 3, device=DEV))


def _transpose(M):
    ptr, idx, val = M.csc()
    return Csr(M.cols, M.rows, ptr, idx, val)


def _batch_sizes(case):
    """n and degree of each product: part of the case, not of the seed."""
    rng = np.random.default_rng(case["sizes_seed"])
    ns = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]), case["count"])).astype(int)
    return [(int(n), float(d)) for n, d in zip(ns, rng.uniform(case["deg_lo"], case["deg_hi"], case["count"]))]


def _products(case, seed):
    """The case's products as (A, B) pairs; a chained product as its factors."""
    f, g = case["family"], _rng(seed, 1)
    if f == "er":
        return [_er_pair(case["m"], case["k"], case["n"], case["deg_a"], case["deg_b"], case["same"], g)]
    if f == "rmat":
        A = _rmat(case["n"], case["ef"], g)
        return [(A, A)]
    if f == "stencil":
        A = _stencil(case["s"], g)
        return [(A, A)]
    if f == "host":
        return [_er_pair(case["n"], case["n"], case["n"], case["deg"], case["deg"], True, g)]
    if f == "galerkin":
        return [(_stencil(case["s"], g, diffusion=True), _prolongator(case["s"]))]
    if f == "batch":
        return [_er_pair(n, n, n, d, d, False, g, salt=2 * i, skewed=i % 2 == 1)
                for i, (n, d) in enumerate(_batch_sizes(case))]
    raise ValueError(f)


# ---------------------------------------------------------------------------
# What a program holds before the call, and one pass
# ---------------------------------------------------------------------------

def _device_cm(arrays, rows, cols, kind):
    ptr, idx, val = arrays
    return sg.device_cm(ptr.data_ptr(), idx.data_ptr(), val.data_ptr(), idx.numel(), rows, cols, kind)


def _row_major(M):
    arrays = (M.rowptr, M.col, M.val)
    return _device_cm(arrays, M.rows, M.cols, sg.ROW_MAJOR), arrays


def _col_major(M):
    arrays = M.csc()
    return _device_cm(arrays, M.rows, M.cols, sg.COL_MAJOR), arrays


class _Array:
    """A device array of the library's, for torch to look at in place. Tensors
    over it hold the handle that owns the memory, so they may outlive the state."""

    def __init__(self, handle, pointer, count, kind):
        self.handle = handle
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (pointer, False), "version": 3}


def _address(p):
    return sg.C.cast(p, sg.C.c_void_p).value


def _pinned(t):
    return t.cpu().pin_memory().numpy()


def prepare(case, seed):
    f = case["family"]
    if f == "coo":
        g = _rng(seed, 1)
        r, c = _rmat_edges(case["n"], case["ef"], g)
        v = torch.rand(r.numel(), generator=g, device=DEV)
        triplets = torch.stack([r.int(), c.int(), v.view(torch.int32)], 1).contiguous()
        return {"family": f, "case": case, "handle": sg.Handle(), "triplets": triplets}
    handle = sg.Handle(sg.COMPENSATED if case["compensated"] else sg.PLAIN)
    pairs = _products(case, seed)
    if f == "batch":
        A = [_row_major(a) for a, _ in pairs]
        B = [_row_major(b) for _, b in pairs]
        total = handle.batch_plan([a for a, _ in A], [b for b, _ in B])
        row_off, _ = handle.batch_offsets()
        first = handle.batch_result(0)
        out = [torch.as_tensor(_Array(handle, _address(first.ptr), int(row_off[-1]) + len(pairs), "<i4"), device=DEV),
               torch.as_tensor(_Array(handle, _address(first.idx), total, "<i4"), device=DEV),
               torch.as_tensor(_Array(handle, _address(first.val), total, "<f4"), device=DEV)]
        return {"family": f, "handle": handle, "keep": (A, B), "out": out}
    (M, B), = pairs
    if f == "galerkin":
        A_cm, A_keep = _col_major(M)
        P_cm, P_keep = _row_major(B)
        # P's CSR arrays read as CSC are P^T
        PT_cm = _device_cm(P_keep, B.cols, B.rows, sg.COL_MAJOR)
        return {"family": f, "handle": handle, "keep": (A_keep, P_keep), "A": A_cm, "P": P_cm, "PT": PT_cm}
    if f == "host":
        Bh = sg.Csr(B.rows, B.cols, _pinned(B.rowptr), _pinned(B.col), _pinned(B.val))
        if case["csc"]:
            Ah = sg.Csc(M.rows, M.cols, *[_pinned(t) for t in M.csc()])
        else:
            Ah = Bh
        # room for every product: an upper bound a caller knows before the call
        room = int((B.rowptr[1:] - B.rowptr[:-1]).long()[M.col.long()].sum())
        out = [torch.empty(M.rows + 1, dtype=torch.int32, pin_memory=True),
               torch.empty(room, dtype=torch.int32, pin_memory=True),
               torch.empty(room, dtype=torch.float32, pin_memory=True)]
        return {"family": f, "handle": handle, "A": Ah, "B": Bh, "out": out}
    A_cm, A_keep = _col_major(M) if case["csc"] else _row_major(M)
    B_cm, B_keep = _row_major(B)
    return {"family": f, "handle": handle, "keep": (A_keep, B_keep), "A": A_cm, "B": B_cm}


def _multiply(handle, A, B):
    nnz = handle.symbolic(A, B)
    rowptr = torch.empty(A.num_rows + 1, dtype=torch.int32, device=DEV)
    col = torch.empty(nnz, dtype=torch.int32, device=DEV)
    val = torch.empty(nnz, dtype=torch.float32, device=DEV)
    handle.numeric(rowptr.data_ptr(), col.data_ptr(), val.data_ptr())
    return rowptr, col, val


def run(state):
    f, h = state["family"], state["handle"]
    if f == "batch":
        h.batch_execute()
        return state["out"]
    if f == "host":
        rowptr, col, val = state["out"]
        nnz = h.multiply_host_to(state["A"], state["B"], rowptr.numpy(), col.numpy(), val.numpy())
        return [rowptr, col[:nnz], val[:nnz]]
    if f == "coo":
        case, t = state["case"], state["triplets"]
        kind = sg.COL_MAJOR if case["col_major"] else sg.ROW_MAJOR
        ptr = torch.empty(case["n"] + 1, dtype=torch.int32, device=DEV)
        idx = torch.empty(t.shape[0], dtype=torch.int32, device=DEV)
        val = torch.empty(t.shape[0], dtype=torch.float32, device=DEV)
        h.coo_to_cm(t.data_ptr(), t.shape[0], case["n"], case["n"], kind, ptr.data_ptr(), idx.data_ptr(),
                    val.data_ptr())
        return [ptr, idx, val]
    if f == "galerkin":
        ap = _multiply(h, state["A"], state["P"])
        AP = _device_cm(ap, state["A"].num_rows, state["P"].num_cols, sg.ROW_MAJOR)
        return list(_multiply(h, state["PT"], AP))
    return list(_multiply(h, state["A"], state["B"]))


# ---------------------------------------------------------------------------
# Exact values and the work of one pass
# ---------------------------------------------------------------------------

def _expand(A, B, j0, j1):
    """Products of A's entries [j0, j1): (row, column, 64-bit value)."""
    k = A.col[j0:j1].long()
    lens = (B.rowptr[1:] - B.rowptr[:-1]).long()[k]
    own = torch.repeat_interleave(torch.arange(j1 - j0, device=DEV), lens)
    first = torch.cumsum(lens, 0) - lens
    pos = B.rowptr[k].long()[own] + torch.arange(own.numel(), device=DEV) - first[own]
    val = A.val[j0:j1].double()[own] * B.val[pos].double()
    return own, B.col[pos].long(), val


def _row_products(A, B):
    """Products before each row of A (rows + 1 values)."""
    ends = torch.zeros(A.nnz + 1, dtype=torch.int64, device=DEV)
    ends[1:] = torch.cumsum((B.rowptr[1:] - B.rowptr[:-1]).long()[A.col.long()], 0)
    return ends[A.rowptr.long()]


def _product64(A, B):
    """A * B with 64-bit values: expand, sort by (row, column), sum."""
    before = _row_products(A, B).cpu().numpy()
    rowptr = A.rowptr.cpu().numpy()
    cols, vals, counts = [], [], []
    r0 = 0
    while r0 < A.rows:
        r1 = max(r0 + 1, int(np.searchsorted(before, before[r0] + CHUNK, side="right")) - 1)
        j0, j1 = int(rowptr[r0]), int(rowptr[r1])
        own, col, val = _expand(A, B, j0, j1)
        row = torch.repeat_interleave(torch.arange(r1 - r0, device=DEV),
                                      (A.rowptr[r0 + 1: r1 + 1] - A.rowptr[r0:r1]).long())
        keys, order = torch.sort(row[own] * B.cols + col)
        new = torch.ones(keys.numel(), dtype=torch.bool, device=DEV)
        new[1:] = keys[1:] != keys[:-1]
        distinct = keys[new]
        vals.append(torch.zeros(distinct.numel(), dtype=torch.float64, device=DEV).index_add_(
            0, torch.cumsum(new, 0) - 1, val[order]))
        cols.append((distinct % B.cols).int())
        counts.append(torch.bincount(torch.div(distinct, B.cols, rounding_mode="floor"), minlength=r1 - r0))
        r0 = r1
    ptr = torch.zeros(A.rows + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.cat(counts), 0)
    return Csr(A.rows, B.cols, ptr.int(), torch.cat(cols), torch.cat(vals))


def exact(case, seed):
    f = case["family"]
    if f == "coo":
        g = _rng(seed, 1)
        r, c = _rmat_edges(case["n"], case["ef"], g)
        v = torch.rand(r.numel(), generator=g, device=DEV).double()
        major, minor = (c, r) if case["col_major"] else (r, c)
        order = torch.argsort(major * case["n"] + minor, stable=True)
        return [_pointers(major, case["n"]), minor[order].int(), v[order]]
    pairs = _products(case, seed)
    if f == "galerkin":
        (A, P), = pairs
        C = _product64(_transpose(P), _product64(A, P))
        return [C.rowptr, C.col, C.val]
    out = [_product64(A, B) for A, B in pairs]
    return [torch.cat([C.rowptr for C in out]), torch.cat([C.col for C in out]), torch.cat([C.val for C in out])]


def _bytes(M):
    return 4 * (M.rows + 1) + 8 * M.nnz


def _outputs(A, B, products):
    """nnz of A*B, from evenly spaced rows when the product is large."""
    step = max(1, products // 20_000_000)
    if step > 1:
        pick = torch.arange(0, A.rows, step, device=DEV)
        lens = (A.rowptr[1:] - A.rowptr[:-1]).long()[pick]
        ptr = torch.zeros(pick.numel() + 1, dtype=torch.int64, device=DEV)
        ptr[1:] = torch.cumsum(lens, 0)
        src = torch.repeat_interleave(A.rowptr[pick].long() - ptr[:-1], lens) + torch.arange(int(ptr[-1]), device=DEV)
        A = Csr(pick.numel(), A.cols, ptr.int(), A.col[src], A.val[src])
    own, col, _ = _expand(A, B, 0, A.nnz)
    return step * torch.unique(A.row_of()[own] * B.cols + col).numel()


def work(case):
    """Each operand read once and C written once; two operations a product."""
    if case["family"] == "coo":
        nnz = int(case["ef"] * case["n"])
        return {"bytes": 20 * nnz + 4 * (case["n"] + 1), "flops": 0}
    pairs = _products(case, 0)
    if case["family"] == "galerkin":
        (A, P), = pairs
        pairs = [(A, P), (_transpose(P), _product64(A, P))]
    bytes_, flops = 0, 0
    for A, B in pairs:
        products = int(_row_products(A, B)[-1])
        bytes_ += _bytes(A) + _bytes(B) + 4 * (A.rows + 1) + 8 * _outputs(A, B, products)
        flops += 2 * products
    return {"bytes": bytes_, "flops": flops}
