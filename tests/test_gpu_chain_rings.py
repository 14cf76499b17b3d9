"""Chains of blocks of 48 rows (nr 33 to 48) take a ring of two slots once a launch has more CTAs than SMs, four
otherwise (csrc/sdd_chain.cu): the same arithmetic, so each shell of a large batch has the bits that it has alone."""
import numpy as np
import pytest

from oracle import sdd_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [1, 2, 3])
@pytest.mark.parametrize("N_fm,N_r,sym,precision", [(6, 34, False, "fp64"), (24, 34, True, "fp64"), (32, 41, False, "mixed"),
                                                    (48, 49, False, "fp64")])
def test_large_batches_equal_shells_alone(cuda, N_fm, N_r, sym, precision, layout):
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    p = Plan(N_fm, N_r, 2.0, 5e-4, 1.0, 0.01, symmetric=sym, precision=precision)
    p.set_chain_layout(layout)
    p.set_fx_split(1)
    B = cuda.cuda.get_device_properties(0).multi_processor_count // 4 + 3      # 4 CTAs a shell at least
    X = cuda.from_numpy(np.stack([0.1 * O.seeded_state(N_fm, N_r - 1, k, sym) for k in range(B)])).cuda()
    for linear in (False, True):
        y = p.step(X, 8000.0, 500.0, nsteps=3, linear=linear)
        F = p.pfx(X, 8000.0, 500.0)
        for b in (0, 1, B - 1):
            one = X[b:b + 1].contiguous()
            assert cuda.equal(p.step(one, 8000.0, 500.0, nsteps=3, linear=linear)[0], y[b])
            assert cuda.equal(p.pfx(one, 8000.0, 500.0)[0], F[b])
