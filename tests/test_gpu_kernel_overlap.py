"""The step's kernels start beside the end of the kernel before them (csrc/sdd_internal.cuh): what they read ahead of
their wait are the plan's tables alone, so a run of overlapping steps gives the bits of single steps with the device
idle in between.  Other chunk lengths change roundings: 1e-11 over a few steps, mixed plans (whose FP32 terms may
round the other way) 2^-24."""
import numpy as np
import pytest

from oracle import sdd_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N_fm,N_r,batch,sym,layout,split", [
    (16, 8, 1, False, 1, 1), (64, 20, 1, False, 3, 2), (64, 20, 3, True, 3, 2), (90, 23, 2, True, 2, 2),
    (256, 30, 1, False, 0, 0), (96, 34, 5, False, 3, 2), (96, 34, 40, False, 2, 1), (128, 65, 1, True, 0, 0),
    (64, 24, 70, False, 0, 0)])
def test_overlapping_steps_equal_separate_ones(cuda, N_fm, N_r, batch, sym, layout, split, precision):
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    p = Plan(N_fm, N_r, 2.0, 5e-4, 1.0, 0.01, symmetric=sym, precision=precision)
    p.set_chain_layout(layout)
    p.set_fx_split(split)
    X = cuda.from_numpy(np.stack([0.1 * O.seeded_state(N_fm, N_r - 1, k, sym) for k in range(batch)])).cuda()
    tol = 1e-11 if precision == "fp64" else 2.0 ** -24
    y = p.step(X, 8000.0, 500.0, nsteps=6)
    z = X
    for _ in range(6):
        z = p.step(z, 8000.0, 500.0)
        cuda.cuda.synchronize()
    assert cuda.equal(y, z)
    p.set_chunk_length(1, min(5, N_fm // 2))             # tables made anew between two runs
    p.set_chunk_length(0, min(6, N_fm // 2))
    a = p.step(X, 8000.0, 500.0, nsteps=6)
    b = p.step(X, 8000.0, 500.0, nsteps=6)
    assert cuda.equal(a, b) and float((a - y).norm() / y.norm()) <= tol
    d, rec = p.step_diag(X, 8000.0, 500.0, nsteps=4)
    w = p.step(X, 8000.0, 500.0, nsteps=4)
    assert float((d - w).norm() / w.norm()) <= tol
    assert np.allclose(rec[-1, :, 0].cpu().numpy(),
                       w.norm(dim=1).cpu().numpy(), rtol=tol)
