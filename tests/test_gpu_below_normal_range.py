"""Numbers below FP64's normal range keep their bits in the fixed-point transforms and matvecs, as in FP64: whole
numbers in units of 2^-1074 (and the same ones far inside the range, whose results are rounded to those units here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNIT = 2.0 ** -1074


def _units(x):
    return np.rint(np.asarray(x) * 2.0 ** 40).astype(np.float64)        # at most 2^53: exact in both scales


@pytest.mark.parametrize("L", [2, 45, 96, 384])
def test_transforms(cuda, L):
    """Rows below the range, rows that straddle its edge, and beside them a row inside it.  One rounding to units of the
    inverse transforms, another one of the forward ones' scale, and the rounding of the rows themselves
    (16 sqrt(L) 2^-58 of their 1-norm)."""
    from spectraldoublediffusiveconvection_gb300 import Transforms as T
    rng = np.random.default_rng(L)
    x = _units(rng.uniform(-1, 1, (6, L)) * np.array([1.0, 2.0 ** -30, 2.0 ** 13, 1.0, 1.0, 1.0])[:, None])
    x[4, 1:] = 0.0
    for kind in ("DCT", "DST", "IDCT", "IDST"):
        f = getattr(T, kind)
        want = np.asarray(f(x * 2.0 ** -40, n=L)) * 2.0 ** 40
        y = np.asarray(f(x * UNIT, n=L))
        tol = 2.5 + 16 * np.sqrt(L) * 2.0 ** -58 * np.abs(x).sum(axis=1, keepdims=True) + 2.0 ** -52 * np.abs(want)
        assert np.all(np.abs(np.ldexp(y, 1074) - want) <= tol), kind
        assert np.any(y[0] != 0)


@pytest.mark.parametrize("N_r", [8, 20, 33, 50])
def test_solves(cuda, N_r):
    """The top mode of each parity: one product, one rounding to units (and the other one's to a double)."""
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, nr = 6, N_r - 1
    p = Plan(M, N_r, 2.0, 1e-3, 1.0, 0.01)
    G = np.zeros((M, nr))
    G[M - 2:] = _units(np.random.default_rng(N_r).uniform(-1, 1, (2, nr)))
    for field in range(3):
        run = lambda g: (p.a4_bsub(g) if field == 0 else p.nab2_bsub(field, g)).cpu().numpy().reshape(M, nr)[M - 2:]
        want = run(cuda.from_numpy(G.ravel()).cuda())
        y = run(cuda.from_numpy(G.ravel() * UNIT).cuda())
        assert np.any(y != 0)
        assert np.all(np.abs(np.ldexp(y, 1074) - want) <= 1.0 + 2.0 ** -52 * np.abs(want))


@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("layout", [1, 2, 3])
def test_linear_steps(cuda, layout, split):
    """A linear step of a state of amplitude 2^-1040: every field in units carries up to a few hundred of them (M chain
    steps of a few roundings each, of operators of norm about 1), 2^-24 of the state: 1e-6 of the norm.  A nonlinear step
    of it is the linear one (its products underflow)."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, N_r = 32, 20
    p = Plan(M, N_r, 2.0, 1e-3, 1.0, 0.01)
    p.set_chain_layout(layout)
    p.set_fx_split(split)
    X = O.seeded_state(M, N_r - 1, 1)
    X /= np.abs(X).max()
    one = lambda x, lin: p.step(cuda.from_numpy(x.reshape(1, -1)).cuda(), 8000.0, 500.0, linear=lin).cpu().numpy().ravel()
    want = one(X, True)
    for lin in (True, False):
        y = np.ldexp(one(np.ldexp(X, -1040), lin), 1040)
        assert np.linalg.norm(y - want) <= 1e-6 * np.linalg.norm(want)
