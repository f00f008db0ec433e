"""Device Newton driver and the warm-start MLP kernels.

* BF16 tensor-core GEMM vs float64 products of the same BF16 inputs
  (tolerance 1e-5 relative: FP32 accumulation);
* MLP forward / backward vs the CPU oracle (oracle/mlp.py) with BF16
  rounding at the same points (tolerance 2e-3 relative);
* Newton + golden-section line search reaches the 1e-6 relative gradient
  tolerance on p-Laplace and Ginzburg-Landau, with the energy matching the
  CPU oracle's energy at the returned point.
"""

import numpy as np
import pytest
import torch

from oracle import mlp as omlp
from oracle.assembler import OracleAssembler
from fenics_nonlinear_energies_b200 import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(64, 64, 32), (200, 96, 40), (1, 7, 300), (513, 257, 129), (8192, 256, 256),
                                   (300, 3, 256), (5, 33, 12), (130, 32, 0)])
@pytest.mark.parametrize("transA", [False, True])
@pytest.mark.parametrize("transB", [False, True])
def test_gemm_bf16(M, N, K, transA, transB):
    from fenics_nonlinear_energies_b200.warmstart import gemm

    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    B = torch.randn(K, N, generator=g).to(torch.bfloat16)
    ref = A.double() @ B.double()
    Ad = (A.t().contiguous() if transA else A).cuda()
    Bd = (B.t().contiguous() if transB else B).cuda()
    sam, sak = (1, M) if transA else (K, 1)
    sbk, sbn = (1, K) if transB else (N, 1)
    C = torch.full((M, N), 3.0, dtype=torch.float32, device="cuda")
    gemm(Ad, sam, sak, Bd, sbk, sbn, M, N, K, C, beta=0.5)
    got = C.double().cpu() - 1.5
    assert (got - ref).abs().max() <= 1e-5 * ref.abs().max() + 1e-5


def test_gemm_wait_timeout_is_reported():
    """The tensor-core GEMM's MMA-completion wait, set to give up at once:
    fne_gemm_check_status reports FNE_ETIMEOUT (then cleared), and with the
    default bound restored the next product is exact again."""
    from fenics_nonlinear_energies_b200 import _lib
    from fenics_nonlinear_energies_b200.warmstart import gemm

    A = torch.randn(256, 64).to(torch.bfloat16)
    B = torch.randn(64, 128).to(torch.bfloat16)
    C = torch.zeros(256, 128, dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib.fne_gemm_set_wait_limit(0))
    try:
        gemm(A.cuda(), 64, 1, B.cuda(), 128, 1, 256, 128, 64, C)
        torch.cuda.synchronize()
        assert _lib.lib.fne_gemm_check_status() == _lib.FNE_ETIMEOUT
        assert _lib.lib.fne_gemm_check_status() == _lib.FNE_OK
    finally:
        _lib.check(_lib.lib.fne_gemm_set_wait_limit(-1))
    gemm(A.cuda(), 64, 1, B.cuda(), 128, 1, 256, 128, 64, C)
    torch.cuda.synchronize()
    assert _lib.lib.fne_gemm_check_status() == _lib.FNE_OK
    ref = A.double() @ B.double()
    assert (C.double().cpu() - ref).abs().max() <= 1e-5 * ref.abs().max()


def test_mlp_forward_backward_match_oracle():
    from fenics_nonlinear_energies_b200.warmstart import BF16, NodalMLP

    mlp = NodalMLP((12, 64, 64, 64, 3), seed=3)
    rng = np.random.default_rng(0)
    X = rng.standard_normal((333, 12)).astype(np.float32)
    T = rng.standard_normal((333, 3)).astype(np.float32)
    Y = mlp.forward(torch.as_tensor(X, device="cuda").to(BF16), keep=True)
    W = [w.cpu().numpy() for w in mlp.W]
    b = [v.cpu().numpy() for v in mlp.b]
    Y_ref, saved = omlp.forward(W, b, X)
    assert np.abs(Y.cpu().numpy() - Y_ref).max() <= 2e-3 * np.abs(Y_ref).max()
    dY = (2.0 / Y.numel()) * (Y - torch.as_tensor(T, device="cuda"))
    gW, gb = mlp.backward(dY)
    dY_ref = (2.0 / Y_ref.size) * (Y_ref - T)
    gW_ref, gb_ref = omlp.backward(W, saved, dY_ref)
    for l in range(4):
        assert np.abs(gW[l].cpu().numpy() - gW_ref[l]).max() <= 2e-2 * np.abs(gW_ref[l]).max()
        assert np.abs(gb[l].cpu().numpy() - gb_ref[l]).max() <= 2e-2 * np.abs(gb_ref[l]).max()


def test_mlp_training_reduces_loss():
    from fenics_nonlinear_energies_b200.warmstart import train_mlp

    rng = np.random.default_rng(1)
    F = rng.uniform(-1, 1, (4096, 12)).astype(np.float32)
    T = np.stack([np.sin(2 * F[:, 0]) * F[:, 3], F[:, 1] * F[:, 2], np.cos(F[:, 4])], 1).astype(np.float32)
    mlp, hist = train_mlp(F, T, width=128, epochs=60, batch=1024, lr=2e-3)
    assert hist[-1] < 0.05 * hist[0]


@pytest.mark.parametrize("family", ["plaplace", "gl"])
def test_newton_converges(family):
    from fenics_nonlinear_energies_b200.assembler import GLCudaAssembler, PLaplaceCudaAssembler
    from fenics_nonlinear_energies_b200.newton import newton

    if family == "plaplace":
        params, u0 = meshes.plaplace_problem(n=32, seed=0)
        asm = PLaplaceCudaAssembler(params)
        ref = OracleAssembler("plaplace", params)
    else:
        params, u0 = meshes.gl_problem(n=32, seed=0)
        asm = GLCudaAssembler(params)
        ref = OracleAssembler("gl", params)
    x, info = newton(asm, torch.as_tensor(u0, device="cuda"), tolg_rel=1e-6)
    assert info["converged"], info["message"]
    xs = x.cpu().numpy()
    assert abs(info["energy"] - ref.energy_fn(xs)) <= 1e-10 * max(1.0, abs(info["energy"]))
    assert np.linalg.norm(ref.gradient_fn(xs)) <= 1.01e-6 * info["grad_norm0"]
    assert info["energy"] < ref.energy_fn(u0)


def test_learned_warm_start_cuts_newton_iterations():
    """Train on solver-generated load-path solutions of a small twisted beam and
    compare, on a held-out path, the Newton iterations from the MLP prediction
    with those from the plain previous-step start (same 1e-6 gradient tolerance
    and energy; a rejected prediction is charged both solves)."""
    from fenics_nonlinear_energies_b200 import warmstart_experiment as wx

    res = wx.run(nx=32, ny=3, nz=3, train_paths=6, test_paths=1, steps=12, epochs=60, seed=3, log=lambda *_: None)
    t = res["test"]
    assert t["accepted_steps"] >= t["steps"] - 1
    assert t["learned_newton_its"] <= 0.85 * t["plain_newton_its"], t


@pytest.mark.parametrize("rows", [1, 127, 129, 1300])
@pytest.mark.parametrize("din,dout", [(12, 64), (64, 3), (40, 33), (72, 200)])
def test_fused_layer_edges(rows, din, dout):
    """One layer's fused forward, input gradient and weight gradient at the edges of
    their tiles (rows 128, columns 32 / 64, depth 64 / 128; 1300 rows take the long
    product) and with unaligned row pitches, against float64 products of the same
    BF16 operands: FP32 accumulation (1e-5 of the largest entry, as for the plain
    product) and one BF16 rounding (2^-8 relative)."""
    from fenics_nonlinear_energies_b200 import _lib

    L, vp = _lib.lib, lambda t: t.data_ptr()  # noqa: E731
    f32 = {"dtype": torch.float32}  # the oracle sets float64 as torch's default
    g = torch.Generator().manual_seed(rows * 1000 + din + dout)
    X = torch.randn(rows, din, generator=g).to(torch.bfloat16).cuda()
    W = (torch.randn(dout, din, generator=g) / din ** 0.5).to(torch.bfloat16).cuda()
    b = torch.randn(dout, generator=g, **f32).cuda()
    Z = torch.empty(rows, dout, device="cuda", **f32)
    H = torch.empty(rows, dout, dtype=torch.bfloat16, device="cuda")
    _lib.check(L.fne_mlp_linear_fwd(rows, din, dout, vp(X), vp(W), vp(b), 1, vp(Z), None, vp(H), None))
    ref = X.double() @ W.double().T + b.double()
    assert (Z.double() - ref).abs().max() <= 1e-5 * ref.abs().max() + 1e-5
    silu = torch.nn.functional.silu(Z.double())
    assert ((H.double() - silu).abs() <= 2.0 ** -8 * silu.abs() + 1e-6).all()

    dZ = torch.randn(rows, dout, generator=g).to(torch.bfloat16).cuda()
    Zin = torch.randn(rows, din, generator=g, **f32).cuda()
    dIn = torch.empty(rows, din, dtype=torch.bfloat16, device="cuda")
    part = torch.empty(-(-rows // 128), din, dtype=torch.float64, device="cuda")
    _lib.check(L.fne_mlp_linear_bwd_data(rows, din, dout, vp(dZ), dout, vp(W), vp(Zin), 1, vp(dIn),
                                         vp(part), None))
    s = torch.sigmoid(Zin.double())
    ref = (dZ.double() @ W.double()) * (s * (1 + Zin.double() * (1 - s)))
    assert ((dIn.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max() + 1e-5).all()
    assert (part.sum(0) - ref.sum(0)).abs().max() <= 1e-5 * ref.abs().sum(0).max()

    gW = torch.empty(din, dout, device="cuda", **f32)  # gradient of a layer dout -> din whose dZ is dIn
    gb = torch.empty(din, device="cuda", **f32)
    _lib.check(L.fne_mlp_linear_bwd_weight(rows, dout, din, vp(dIn), din, vp(dZ), dout, vp(gW), vp(part),
                                           vp(gb), None))
    ref = dIn.double().T @ dZ.double()
    assert (gW.double() - ref).abs().max() <= 1e-5 * ref.abs().max() + 1e-5
    assert (gb.double() - part.sum(0)).abs().max() <= 1e-6 * part.sum(0).abs().max() + 1e-6
    # the same from rows padded to a multiple of eight values: the same sums in the same order
    ldx, ldz = -(-dout // 8) * 8, -(-din // 8) * 8
    Xp, Zp = (torch.full((rows, ld), 9.0, dtype=torch.bfloat16, device="cuda") for ld in (ldx, ldz))
    _lib.check(L.fne_mlp_pad_rows(rows, dout, vp(dZ), 0, ldx, vp(Xp), None))
    dIn32 = dIn.float()
    _lib.check(L.fne_mlp_pad_rows(rows, din, vp(dIn32), 1, ldz, vp(Zp), None))
    assert (Xp[:, :dout] == dZ).all() and (Xp[:, dout:] == 0).all() and (Zp[:, :din] == dIn).all()
    gP = torch.empty_like(gW)
    _lib.check(L.fne_mlp_linear_bwd_weight(rows, dout, din, vp(Zp), ldz, vp(Xp), ldx, vp(gP), None, None, None))
    assert torch.equal(gP, gW)
    _lib.check(L.fne_gemm_check_status())


@pytest.mark.parametrize("rows", [1, 129, 1300])
@pytest.mark.parametrize("din,dout", [(12, 64), (64, 3), (40, 33), (72, 200), (1100, 40)])
def test_fused_layers_equal_their_separate_calls(rows, din, dout):
    """The fused forward and input gradient give the bits of the product followed by the elementwise call, and the
    optimiser over a set of tensors those of one call per tensor."""
    from fenics_nonlinear_energies_b200 import _lib
    from fenics_nonlinear_energies_b200.warmstart import gemm

    L, vp = _lib.lib, lambda t: t.data_ptr()  # noqa: E731
    g = torch.Generator().manual_seed(rows + din + dout)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float32).cuda()  # noqa: E731
    new = lambda *s, dtype=torch.float32: torch.full(s, 7.0, dtype=dtype, device="cuda")  # noqa: E731
    X, W, b = rand(rows, din).bfloat16(), (rand(dout, din) / din ** 0.5).bfloat16(), rand(dout)
    for act in (0, 1):
        Z, H, H16 = new(rows, dout), new(rows, dout), new(rows, dout, dtype=torch.bfloat16)
        Z1, H1, H161 = new(rows, dout), new(rows, dout), new(rows, dout, dtype=torch.bfloat16)
        _lib.check(L.fne_mlp_linear_fwd(rows, din, dout, vp(X), vp(W), vp(b), act, vp(Z), vp(H), vp(H16), None))
        gemm(X, din, 1, W, 1, din, rows, dout, din, Z1)
        _lib.check(L.fne_mlp_bias_act(rows, dout, vp(Z1), vp(b), act, vp(H1), vp(H161), None))
        assert torch.equal(Z, Z1) and torch.equal(H, H1) and torch.equal(H16, H161)
        dZ, Zin = rand(rows, dout).bfloat16(), rand(rows, din)
        d16, part = new(rows, din, dtype=torch.bfloat16), new(-(-rows // 128), din, dtype=torch.float64)
        C, d161 = new(rows, din), new(rows, din, dtype=torch.bfloat16)
        _lib.check(L.fne_mlp_linear_bwd_data(rows, din, dout, vp(dZ), dout, vp(W), vp(Zin), act, vp(d16), vp(part), None))
        gemm(dZ, dout, 1, W, din, 1, rows, din, dout, C)
        _lib.check(L.fne_mlp_act_bwd(rows * din, vp(Zin), vp(C), act, vp(C), vp(d161), None))
        assert torch.equal(d16, d161)
        # C holds the FP32 gradients; the sums of a tile are FP64 sums of 128 of them in some order
        sums = torch.stack([C[k:k + 128].double().sum(0) for k in range(0, rows, 128)])
        assert (part - sums).abs().max() <= 128 * 2.0 ** -53 * C.double().abs().max() * 128
    sizes = (dout * din, dout, 1)
    sets = [[[rand(n), rand(n), rand(n).abs(), rand(n).abs()] for n in sizes]]  # p, g, m, v
    sets.append([[t.clone() for t in s] for s in sets[0]])
    p16 = [[new(n, dtype=torch.bfloat16) for n in sizes[:2]] + [None] for _ in range(2)]
    args = (1e-3, 0.9, 0.999, 1e-8, 3)
    import ctypes

    ptrs = [(ctypes.c_void_p * 3)(*(vp(s[k]) for s in sets[0])) for k in range(4)]
    h16 = (ctypes.c_void_p * 3)(*(vp(t) if t is not None else None for t in p16[0]))
    _lib.check(L.fne_mlp_adam_set(3, (ctypes.c_int64 * 3)(*sizes), *ptrs, h16, *args, None))
    for s, t in zip(sets[1], p16[1]):
        _lib.check(L.fne_mlp_adam(s[0].numel(), *(vp(x) for x in s), *args, vp(t) if t is not None else None, None))
    for s, s1 in zip(*sets):
        assert all(torch.equal(x, y) for x, y in zip(s, s1))
    assert all(torch.equal(x, y) for x, y in zip(p16[0][:2], p16[1][:2]))
    _lib.check(L.fne_gemm_check_status())
