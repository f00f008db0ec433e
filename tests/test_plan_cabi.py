"""``fne_create``'s check of a COO pattern against the element graph (CPU: a refused pattern never reaches a device)."""

import ctypes

import numpy as np
import pytest

from fenics_nonlinear_energies_b200 import _lib


def _create(rows, cols, variant):
    """Return code of ``fne_create`` for two Neo-Hookean tets (five free nodes) with this pattern."""
    elems = (3 * np.array([[0, 1, 2, 3], [1, 2, 3, 4]])[:, :, None] + np.arange(3)).reshape(2, 12)
    d = _lib.Desc()
    keep = []

    def put(name, a, conv):
        arr, ptr = conv(a)
        keep.append(arr)
        setattr(d, name, ptr)

    put("elems", elems, _lib.i64)
    put("total_to_free_reord", np.arange(15), _lib.i64)
    put("owned_rows", rows, _lib.i64)
    put("owned_cols", cols, _lib.i64)
    put("energy_weights", np.ones(2), _lib.f64)
    put("dirichlet", np.zeros(15), _lib.f64)
    for k, n in (("e0", 8), ("e1", 8), ("e2", 8), ("e3", 2)):
        put(k, np.ones(n), _lib.f64)
    d.family, d.precision, d.npe, d.block_size, d.kernel_variant = _lib.FNE_NEOHOOKEAN, 0, 4, 3, variant
    d.n_elem, d.n_total, d.n_free, d.lo, d.hi, d.nnz = 2, 15, 15, 0, 15, int(np.size(rows))
    d.s[0] = d.s[1] = 1.0
    h = ctypes.c_void_p()
    code = _lib.lib.fne_create(ctypes.byref(d), ctypes.byref(h))
    if code == _lib.FNE_OK:
        _lib.lib.fne_destroy(h)
    return code


def _pattern(node_columns):
    """Rows of every node with the columns that ``node_columns`` makes of its neighbours' (node, component) list."""
    near = [[0, 1, 2, 3], [0, 1, 2, 3, 4], [0, 1, 2, 3, 4], [0, 1, 2, 3, 4], [1, 2, 3, 4]]
    rows, cols = [], []
    for a, nodes in enumerate(near):
        c = node_columns([3 * b + k for b in nodes for k in range(3)])
        for k in range(3):
            rows += [3 * a + k] * len(c)
            cols += c
    return np.array(rows), np.array(cols)


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("case", ["missing", "apart"])
def test_tet_pattern_without_whole_column_nodes_is_refused(case, variant):
    """A component missing from a coupled node's columns, or a node's columns in two places: the values have no
    place, by the tiles of row nodes (variant 0) as by the row-gather kernel (1)."""
    change = {"missing": lambda c: [x for x in c if x != 8], "apart": lambda c: [x for x in c if x != 8] + [8]}[case]
    assert _create(*_pattern(change), variant) == _lib.FNE_ELAYOUT
    assert _create(*_pattern(lambda c: c), variant) != _lib.FNE_ELAYOUT
