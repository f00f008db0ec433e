"""Device CG (``fne_cg_*``) against the scalar CG oracle (``oracle/krylov.py``).

Same iteration count and stop reason, the same iterate to 1e-9 relative
(FP64 arithmetic, different summation order), on shuffled COO patterns with
FP64 and FP32 value storage; the stopping rules at the edges (first-iteration
negative curvature, later negative curvature, iteration limits that are not
a multiple of the graph length, zero right-hand side, missing and zero
diagonals); bitwise reproducibility and independence of the graph length;
and the Hessians the assemblers produce.
"""

import numpy as np
import pytest
import torch

from oracle import krylov
from oracle.assembler import OracleAssembler
from fenics_nonlinear_energies_b200 import meshes

pytestmark = pytest.mark.gpu


def _laplacian_coo(m, shift, seed, drop_diag=()):
    """Symmetric 5-point pattern on an m x m grid, random symmetric values, shuffled COO order."""
    rng = np.random.default_rng(seed)
    idx = np.arange(m * m).reshape(m, m)
    rows, cols = [idx.ravel()], [idx.ravel()]
    for a, b in ((idx[:, :-1], idx[:, 1:]), (idx[:-1, :], idx[1:, :])):
        rows += [a.ravel(), b.ravel()]
        cols += [b.ravel(), a.ravel()]
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    off = rows != cols
    w = np.zeros(rows.size)
    key = np.minimum(rows, cols) * (m * m) + np.maximum(rows, cols)
    _, inv = np.unique(key, return_inverse=True)
    w_sym = -(0.5 + rng.random(inv.max() + 1))
    w[off] = w_sym[inv[off]]
    diag = np.zeros(m * m)
    np.add.at(diag, rows[off], -w[off])
    w[~off] = diag[rows[~off]] + shift[rows[~off]] if np.ndim(shift) else diag[rows[~off]] + shift
    keep = ~np.isin(np.where(~off, rows, -1), np.asarray(drop_diag, dtype=np.int64))
    rows, cols, w = rows[keep], cols[keep], w[keep]
    order = rng.permutation(rows.size)
    return m * m, rows[order], cols[order], w[order]


def _dense(n, rows, cols, vals):
    A = np.zeros((n, n))
    np.add.at(A, (rows, cols), vals)
    return A


def _solve_both(n, rows, cols, vals, b, rtol, maxit, fp32=False, chunk=16):
    from fenics_nonlinear_energies_b200.newton import DeviceCG

    v = vals.astype(np.float32).astype(np.float64) if fp32 else vals
    A = _dense(n, rows, cols, v)
    diag = np.full(n, np.nan)
    on = rows == cols
    diag[rows[on]] = v[on]
    x_ref, it_ref, why_ref = krylov.pcg(A, krylov.jacobi_scaling(diag), b, rtol, maxit)
    cg = DeviceCG(n, rows, cols, fp32=fp32, chunk=chunk)
    cg.update(torch.as_tensor(vals, dtype=torch.float32 if fp32 else torch.float64, device="cuda"))
    x, it = cg.solve(torch.as_tensor(b, device="cuda"), rtol=rtol, maxit=maxit)
    why = cg.REASONS.index(cg.reason)
    cg.close()
    return x.cpu().numpy(), it, why, x_ref, it_ref, why_ref


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("m", [3, 40, 130])
def test_cg_spd_matches_oracle(m, fp32):
    n, rows, cols, vals = _laplacian_coo(m, 0.05, seed=m)
    b = np.random.default_rng(m + 1).standard_normal(n)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-8, 2000, fp32=fp32)
    assert (it, why) == (it_ref, why_ref) == (it_ref, krylov.CONVERGED)
    np.testing.assert_allclose(x, x_ref, rtol=0, atol=1e-9 * np.abs(x_ref).max())


def test_cg_negative_curvature_first_and_later():
    n, rows, cols, vals = _laplacian_coo(30, -1e6, seed=3)   # negative definite
    b = np.random.default_rng(4).standard_normal(n)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-10, 500)
    assert (it, why) == (it_ref, why_ref) == (1, krylov.NEGATIVE_CURVATURE)
    assert np.array_equal(x, b)
    shift = np.full(n, 0.02)
    shift[:5] = -3.0                                          # a few negative modes
    n, rows, cols, vals = _laplacian_coo(30, shift, seed=5)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-12, 500)
    assert (it, why) == (it_ref, why_ref) and why == krylov.NEGATIVE_CURVATURE and it > 1
    np.testing.assert_allclose(x, x_ref, rtol=0, atol=1e-9 * np.abs(x_ref).max())


@pytest.mark.parametrize("maxit,chunk", [(0, 16), (1, 16), (7, 16), (37, 16), (37, 3), (16, 16), (17, 1)])
def test_cg_iteration_limit(maxit, chunk):
    n, rows, cols, vals = _laplacian_coo(50, 1e-3, seed=6)
    b = np.random.default_rng(7).standard_normal(n)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-14, maxit, chunk=chunk)
    assert (it, why) == (it_ref, why_ref) == (maxit, krylov.ITERATION_LIMIT)
    np.testing.assert_allclose(x, x_ref, rtol=0, atol=1e-9 * max(1.0, np.abs(x_ref).max()))


def test_cg_zero_rhs_and_diagonal_edge_cases():
    n, rows, cols, vals = _laplacian_coo(20, 0.1, seed=8)
    x, it, why, *_ = _solve_both(n, rows, cols, vals, np.zeros(n), 1e-8, 100)
    assert (it, why) == (0, krylov.ZERO_RHS) and not x.any()
    # a missing diagonal entry and a zero one: Jacobi scale 1 there
    n, rows, cols, vals = _laplacian_coo(20, 0.1, seed=9, drop_diag=[3])
    vals = vals.copy()
    vals[(rows == 7) & (cols == 7)] = 0.0
    b = np.random.default_rng(10).standard_normal(n)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-8, 1000)
    assert (it, why) == (it_ref, why_ref)
    np.testing.assert_allclose(x, x_ref, rtol=0, atol=1e-8 * np.abs(x_ref).max())


def test_cg_reproducible_and_chunk_independent():
    from fenics_nonlinear_energies_b200.newton import DeviceCG

    n, rows, cols, vals = _laplacian_coo(90, 0.01, seed=11)
    b = torch.as_tensor(np.random.default_rng(12).standard_normal(n), device="cuda")
    v = torch.as_tensor(vals, device="cuda")
    outs = []
    for chunk in (16, 16, 5, 1):
        cg = DeviceCG(n, rows, cols, chunk=chunk)
        cg.update(v)
        outs.append(cg.solve(b, rtol=1e-9, maxit=3000))
        # the same handle again, with another right-hand side in between
        cg.solve(2.0 * b, rtol=1e-3, maxit=3000)
        outs.append(cg.solve(b, rtol=1e-9, maxit=3000))
        cg.close()
    for x, it in outs[1:]:
        assert it == outs[0][1] and torch.equal(x, outs[0][0])


@pytest.mark.parametrize("family", ["gl", "he"])
def test_cg_on_assembled_hessian(family):
    from fenics_nonlinear_energies_b200 import _lib
    from fenics_nonlinear_energies_b200.assembler import GLCudaAssembler, HECudaAssembler
    from fenics_nonlinear_energies_b200.newton import DeviceCG

    if family == "gl":
        params, u = meshes.gl_problem(n=48, seed=1)
        asm, ref = GLCudaAssembler(params), OracleAssembler("gl", params)
    else:
        params, u = meshes.he_beam_problem(nx=12, ny=3, nz=3)
        u = u + 1e-3 * np.random.default_rng(2).standard_normal(u.size)
        asm = HECudaAssembler(params)
        ref = OracleAssembler("he", params, block_size=3, coordinate_key="nodes2coord", dirichlet_key="u_0_ref")
    ud = torch.as_tensor(u, device="cuda")
    _, g, _ = asm.eval(ud, _lib.FNE_GRAD | _lib.FNE_HESS)
    lay = asm.layout
    rows = np.asarray(lay.owned_rows) - lay.lo
    cols = np.asarray(lay.owned_cols)
    hv = asm.owned_values.double().cpu().numpy()
    A = _dense(asm.n_owned, rows, cols, hv)
    x_ref, it_ref, why_ref = krylov.pcg(A, krylov.jacobi_scaling(np.diag(A)), -g.cpu().numpy(), 1e-6, 1000)
    cg = DeviceCG.for_assembler(asm)
    cg.update(asm.owned_values)
    x, it = cg.solve(-g, rtol=1e-6, maxit=1000)
    assert it == it_ref and cg.REASONS.index(cg.reason) == why_ref
    np.testing.assert_allclose(x.cpu().numpy(), x_ref, rtol=0, atol=1e-8 * np.abs(x_ref).max())
    cg.close()
    asm.cleanup()
    del ref


def _band_coo(n, m, seed, dense=0):
    """SPD matrix of 2 m + 1 diagonals (ends cut), and a first row and column of ``dense`` entries; shuffled COO order."""
    rng = np.random.default_rng(seed)
    offs = np.sort(rng.choice(np.arange(1, 4 * m + 2), m, replace=False))
    rows = np.concatenate([np.arange(n - d) for d in offs] + ([np.zeros(dense, dtype=np.int64)] if dense else []))
    cols = np.concatenate([np.arange(d, n) for d in offs] + ([n - 1 - np.arange(dense)] if dense else []))
    w = -(0.5 + rng.random(rows.size))
    diag = np.full(n, 0.3)
    np.add.at(diag, rows, -w)
    np.add.at(diag, cols, -w)
    r, c, v = np.r_[rows, cols, np.arange(n)], np.r_[cols, rows, np.arange(n)], np.r_[w, w, diag]
    order = rng.permutation(r.size)
    return n, r[order], c[order], v[order]


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("m,dense", [(3, 0), (4, 0), (5, 0), (7, 0), (2, 40), (4, 40), (9, 40), (9, 0), (20, 0)])
def test_cg_row_lengths_match_oracle(m, dense, fp32):
    """Every form of the product: rows of 7, 9, 11 and 15 entries stored column-major, and rows on CSR with 4, 8, 16
    and 32 lanes (one row of 40 and more, or rows of 19 and 41), with a last batch of rows that is not full.  FP64
    arithmetic in another order: the oracle's iteration count, and its iterate to 1e-9."""
    n, rows, cols, vals = _band_coo(1003, m, 10 * m + dense, dense)
    b = np.random.default_rng(m).standard_normal(n)
    x, it, why, x_ref, it_ref, why_ref = _solve_both(n, rows, cols, vals, b, 1e-8, 500, fp32=fp32)
    assert (it, why) == (it_ref, why_ref) == (it_ref, krylov.CONVERGED)
    np.testing.assert_allclose(x, x_ref, rtol=0, atol=1e-9 * np.abs(x_ref).max())


@pytest.mark.parametrize("m", [3, 9])
def test_cg_one_handle_on_two_streams(m):
    """Matrices and solves of one handle in turn on two streams, nothing waited for in between: a later call finds the
    earlier solve finished, so every result is that of the same call on its own."""
    from fenics_nonlinear_energies_b200.newton import DeviceCG

    n, rows, cols, vals = _band_coo(200_003, m, 77)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal(n), device="cuda")
    mats = [torch.as_tensor(vals * (1.0 + k * (rows == cols)), device="cuda") for k in range(4)]
    alone = []
    for v in mats:
        cg = DeviceCG(n, rows, cols)
        cg.update(v)
        alone.append(cg.solve(b, rtol=1e-8, maxit=300))
        torch.cuda.synchronize()
        cg.close()
    cg = DeviceCG(n, rows, cols)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for k, v in enumerate(mats):
        with torch.cuda.stream(streams[k % 2]):
            cg.update(v)
            outs.append(cg.solve(b, rtol=1e-8, maxit=300))
    torch.cuda.synchronize()
    cg.close()
    for (x, it), (x1, it1) in zip(outs, alone):
        assert it == it1 and torch.equal(x, x1)


def test_cg_solve_is_refused_under_capture_and_runs_after_it():
    from fenics_nonlinear_energies_b200 import _lib
    from fenics_nonlinear_energies_b200.newton import DeviceCG

    n, rows, cols, vals = _band_coo(1003, 3, 30)
    b = torch.as_tensor(np.random.default_rng(3).standard_normal(n), device="cuda")
    cg = DeviceCG(n, rows, cols)
    cg.update(torch.as_tensor(vals, device="cuda"))
    x, it = cg.solve(b, rtol=1e-8)
    out = torch.empty_like(b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out.add_(1.0)
        with pytest.raises(_lib.FneError):
            cg.solve(b, rtol=1e-8, out=torch.empty_like(b))
    side = torch.cuda.Stream()
    for stream in (torch.cuda.current_stream(), side):
        with torch.cuda.stream(stream):
            x1, it1 = cg.solve(b, rtol=1e-8)
        torch.cuda.synchronize()
        assert it1 == it and torch.equal(x1, x)
    cg.close()
