"""A GMRES column after its product (csrc/sdd_krylov.cu): one cluster launch for vectors up to 12288 (FP64 basis)
or 16384 (FP32) entries, with the basis slices in shared memory while they fit, separate launches above."""
import numpy as np
import pytest

from oracle import sdd_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N_fm,N_r", [(8, 4), (16, 8), (64, 20), (96, 42), (128, 42)])
def test_one_cycle_is_the_least_squares_solution(cuda, N_fm, N_r, precision):
    """n = 72 (most ranks' slices empty), 336, 3648, 11808 (FP64: slices past shared memory from column 26 on) and
    15744 (FP64: separate launches, FP32: past shared memory from column 41 on): after one cycle of 44 columns the basis is orthonormal to sqrt(n) k roundings
    and the solution is the minimiser of |F - J x| over the basis, found here by dense least squares on the
    products of the same vectors (relative 1e-6: y is a backward-stable solution of the small system, whose
    residual is flat around the minimum; with FP32 products and basis 1e-2 and their rounding of |F|).  A shell
    alone gives the bits that it gives in a batch."""
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    torch = cuda
    nr, k = N_r - 1, 44
    f32 = precision == "mixed"
    p = Plan(N_fm, N_r, 2.0, 1.0, 1.0, 1.0, precision=precision)
    p.set_chain_layout(1)                                # (the automatic launch forms depend on the batch)
    p.set_fx_split(1)
    X0 = torch.from_numpy(np.stack([0.1 * O.seeded_state(N_fm, nr, s) for s in (3, 4)])).cuda()
    opts = dict(tol=1e-30, restart=k, gmres_rtol=1e-30, max_newton=1, max_restarts=1, mixed_matvec=3 if f32 else 0)
    X1 = X0.clone()
    p.newton(X1, 8000.0, 500.0, **opts)
    for b in range(2):
        V = p.krylov_basis(b, 64)
        n = V.shape[1]
        u = 2.0 ** -24 if f32 else 2.0 ** -53
        err = float((V @ V.T - torch.eye(V.shape[0], dtype=torch.float64, device="cuda")).abs().max())
        assert err <= np.sqrt(n) * k * u, err
        q = Plan(N_fm, N_r, 2.0, 1.0, 1.0, 1.0)
        F = q.pfx(X0[b:b + 1], 8000.0, 500.0)[0]
        W = q.pdfx(V.contiguous(), X0[b:b + 1].repeat(V.shape[0], 1), 8000.0, 500.0)
        q.close()
        Q, _ = torch.linalg.qr(W.T)
        best = float((F - Q @ (Q.T @ F)).norm())
        got = float((F - p.pdfx((X0 - X1)[b:b + 1].contiguous(), X0[b:b + 1], 8000.0, 500.0)[0]).norm())
        f = float(F.norm())
        assert got <= (1.01 * best + 1e-5 * f if f32 else (1 + 1e-6) * best + 1e-11 * f), (b, got, best, f)
    alone = X0[1:2].clone()
    p.newton(alone, 8000.0, 500.0, **opts)
    assert torch.equal(alone[0], X1[1])
