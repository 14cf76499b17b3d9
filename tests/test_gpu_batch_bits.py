"""A shell's steps give the same bits alone (row kernel of 512 threads, or seven CTAs a row) and in a batch (several CTAs
an SM of fewer threads): the rows' fixed-point scales must not depend on how the row is shared out.  (With sums formed
per warp, two of 400,000 random rows of 384 got another scale with 512, 256 or 160 threads.)"""
import numpy as np
import pytest

from oracle import sdd_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N_fm,N_r,batch,nsteps", [(256, 30, 64, 100), (90, 23, 100, 60)])
def test_rows_do_not_depend_on_the_threads(cuda, N_fm, N_r, batch, nsteps):
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    p = Plan(N_fm, N_r, 2.0, 5e-4, 1.0, 0.01)
    p.set_chain_layout(1)
    p.set_fx_split(1)
    X = cuda.from_numpy(np.stack([0.1 * O.seeded_state(N_fm, N_r - 1, k) for k in range(batch)])).cuda()
    y = p.step(X, 8000.0, 500.0, nsteps=nsteps)
    for k in range(batch):
        p.set_fx_split(1 + k % 2)
        z = p.step(X[k:k + 1].contiguous(), 8000.0, 500.0, nsteps=nsteps)
        assert cuda.equal(z[0], y[k]), k
