"""The block matvecs keep 59 bits of an operator's row and 61 of an operand (csrc/sdd_fixed.cuh): Dr's products are no
less exact than FP64's at any supported size, and every row of a solve's block keeps to the stated bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _profiles(nr, n, seed):
    s = 0.5 * (1 - np.cos(np.pi * np.arange(1, nr + 1) / (nr + 1)))
    c = np.random.default_rng(seed).standard_normal((n, 4)) * np.exp(-np.arange(4) / 1.5)
    return c @ np.sin(np.pi * np.arange(1, 5)[:, None] * s)


@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("N_r", [8, 20, 30, 33, 34, 40, 48, 50, 56, 65])
def test_radial_derivatives_are_no_less_exact_than_fp64(cuda, N_r, split):
    """u . grad T with psi of one mode, equal at all radii, and T the same at all theta is J_theta(psi) times Dr T, row by
    row: the error of Dr T and a few roundings of the row (Dr T's transform of one mode, J_theta, the product, the
    transform back and its scale: 2 roundings in the root mean square are more than they give).  40 profiles: no more
    than FP64's (numpy, the same products summed in order) and those 2."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, nr, n = 8, N_r - 1, 40
    p = Plan(M, N_r, 2.0, 1e-3, 1.0, 0.01)
    p.set_fx_split(split)
    D = O.Operators(M, N_r, 2.0, 1e-3, 1.0, 0.01).Dr
    t = _profiles(nr, n, N_r)
    X = np.zeros((n, 3, M, nr))
    X[:, 0, 0] = 1.0                                     # psi = sin(theta): J_theta(psi) = 2 cos(theta)
    X[:, 1, 0] = t
    y = p.nlin_fx(cuda.from_numpy(X.reshape(n, -1)).cuda()).cpu().numpy().reshape(n, 3, M, nr)[:, 1]
    ref = t.astype(LD) @ D.astype(LD).T
    seq = np.zeros_like(t)
    for k in range(nr):
        seq = seq + D[:, k] * t[:, k:k + 1]
    norm = np.linalg.norm(ref.astype(float), axis=1)
    rms = lambda e: float(np.sqrt(np.mean((np.linalg.norm(e.astype(float), axis=1) / norm) ** 2)))
    assert rms(y[:, 1] / 2 - ref) <= rms(seq - ref) + 2 * 2.0 ** -53


@pytest.mark.parametrize("nr", [1, 7, 8, 9, 16, 24, 25, 31, 32, 33, 48, 49, 64])
def test_rows_of_the_solves_keep_to_their_bound(cuda, nr):
    """The top mode of each parity is its block's product alone.  Rows 2^-58 (nr + 2) times the scaled row's 1-norm
    times the scaled operand's largest entry (the two operands' rounding, the dropped digit product, the sum's last
    bit), and one rounding to a double; smooth operands, random ones and a thin layer at either wall."""
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M = 6
    p = Plan(M, nr + 1, 2.0, 5e-4, 1.0, 0.01)
    rng = np.random.default_rng(nr)
    s = 0.5 * (1 - np.cos(np.pi * np.arange(1, nr + 1) / (nr + 1)))
    for x in (_profiles(nr, 2, 3), rng.standard_normal((2, nr)), np.stack([s * np.exp(-60 * s), (1 - s) * np.exp(-200 * (1 - s))]),
              rng.standard_normal((2, nr)) * 10.0 ** rng.uniform(-15, 0, (2, nr))):
        G = np.zeros((M, nr))
        G[M - 2:] = x                                    # jj = 1 and 0
        g = cuda.from_numpy(G.ravel()).cuda()
        for field, blocks in ((0, "Linv_A4"), (1, "Linv_T"), (2, "Linv_S")):
            y = (p.a4_bsub(g) if field == 0 else p.nab2_bsub(field, g)).cpu().numpy().reshape(M, nr)
            for jj in (0, 1):
                A, v = p.arrays[blocks][jj], G[M - 1 - jj]
                cx = np.frexp(np.abs(A).max(axis=0))[1]
                bound = 2.0 ** -58 * (nr + 2) * np.ldexp(np.abs(A), -cx).sum(axis=1) * np.abs(np.ldexp(v, cx)).max()
                ref = A.astype(LD) @ v.astype(LD)
                assert np.all(np.abs((y[M - 1 - jj] - ref).astype(float)) <= bound + 2.0 ** -53 * np.abs(ref.astype(float)))


def test_zeros_of_a_tiny_column_do_not_set_a_rows_scale(cuda):
    """A column of numbers near 2^-1010 with zeros in it, and a row whose other entries lie 2^-40 below their columns'
    largest: the row keeps to its own bound (test_rows_of_the_solves_keep_to_their_bound)."""
    from spectraldoublediffusiveconvection_gb300.operators import plan_arrays
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, N_r = 4, 12
    nr = N_r - 1
    arrays = plan_arrays(M, N_r, 2.0, 1e-3, 1.0, 0.01)
    A = np.random.default_rng(5).standard_normal((nr, nr))
    A[1] *= 2.0 ** -40
    A[:, 0] = 0.0
    A[0, 0] = 2.0 ** -1010
    arrays["Linv_T"] = np.repeat(A[None], M, axis=0)
    p = Plan(M, N_r, 2.0, 1e-3, 1.0, 0.01, arrays=arrays)
    G = np.zeros((M, nr))
    G[M - 1] = np.random.default_rng(6).standard_normal(nr)
    y = p.nab2_bsub(1, cuda.from_numpy(G.ravel()).cuda()).cpu().numpy().reshape(M, nr)[M - 1]
    v = G[M - 1]
    cx = np.frexp(np.abs(A).max(axis=0))[1]
    bound = 2.0 ** -58 * (nr + 2) * np.ldexp(np.abs(A), -cx).sum(axis=1) * np.abs(np.ldexp(v, cx)).max()
    ref = A.astype(LD) @ v.astype(LD)
    assert np.all(np.abs((y - ref).astype(float)) <= bound + 2.0 ** -53 * np.abs(ref.astype(float)))
