"""The FP64 transforms run in 64-bit fixed point on the integer pipe (csrc/sdd_fixed.cuh): every radix and odd
length against dense sums in extended precision, rows of very different magnitude sharing one complex
transform, the ends of the exponent range, and rows with an infinity or a NaN.

Tolerance.  A row is rounded to 60 bits below a power of two E with sum|x| <= E <= 4 sum|x| (the bound is a
power of two above a sum formed with a relative slack below 1/16).  Rounding the inputs (variance 1/12 ulp^2
each) and the operations of up to 8 stages (below 1/2 ulp^2 each, carried on by the remaining stages) leaves
an error of about sqrt(2 P) ulp; 16 sqrt(P) 2^-60 E <= 16 sqrt(P) 2^-58 sum|x| is more than ten times that, plus
one rounding of the result to a double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _dense(kind, x, n):
    """The library's transforms as sums (Transforms.py:73-129), extended precision; x (rows, n_in)."""
    n_in = x.shape[1]
    L = n if kind.startswith("I") else n_in
    i = np.arange(L).astype(LD)
    pi = LD("3.14159265358979323846264338327950288")
    th = pi * (2 * i + 1) / (2 * LD(L))
    k = np.arange(n_in if kind.startswith("I") else n)
    c = np.cos(np.outer(k, th)) if kind.endswith("CT") else np.sin(np.outer(k, th))
    x = x.astype(LD)
    if kind == "IDST":
        c[0] = 0
        c[n_in:] = 0
    if kind.startswith("I"):
        return x @ c
    y = (x @ c.T) * (LD(2) / L)
    if kind == "DCT":
        y[:, 0] /= 2
    return y


@pytest.mark.parametrize("L", [2, 3, 4, 5, 6, 7, 12, 15, 21, 35, 45, 64, 96, 135, 225, 384, 405, 486, 735, 810])
def test_transforms_to_the_fixed_point_bound(cuda, L):
    from spectraldoublediffusiveconvection_gb300 import Transforms as T
    rng = np.random.default_rng(L)
    x = rng.standard_normal((7, L))
    x[1] *= np.exp(-np.arange(L) / 5.0)
    x[2] *= 1e-9                       # next to row 3 in one complex transform
    x[3] *= 1e9
    x[4] *= 1e-290
    x[5] *= 1e290
    x[6] = 0.0
    x[6, L // 2] = 1.0
    for kind in ("DCT", "DST", "IDCT", "IDST"):
        y = np.asarray(getattr(T, kind)(x.copy(), n=L))
        ref = _dense(kind, x, L)
        l1 = np.abs(x).sum(axis=1, keepdims=True)
        scale = 1.0 if kind.startswith("I") else 2.0 / L
        tol = 16 * np.sqrt(L) * 2.0 ** -58 * l1 * scale + 2.0 ** -52 * np.abs(ref).astype(float)
        assert np.all(np.abs((y - ref).astype(float)) <= tol), kind


def test_non_finite_rows_stay_in_their_pair(cuda):
    from spectraldoublediffusiveconvection_gb300 import Transforms as T
    x = np.random.default_rng(3).standard_normal((8, 48))
    good = np.asarray(T.IDCT(x.copy(), n=48))
    x[2, 5] = np.nan
    x[5, 7] = np.inf
    y = np.asarray(T.IDCT(x.copy(), n=48))
    assert np.isnan(y[2]).all() and np.isnan(y[5]).all()
    for r in (0, 1, 6, 7):
        assert np.array_equal(y[r], good[r])


# ---- block matvecs of the implicit solves ----------------------------------------------------------


def _solve_ld(ops, G, field, sym):
    """The oracle's chains (Matrix_Operators.py:1033-1194) in extended precision on the same FP64 blocks."""
    M, nr, h = ops.N_fm, ops.nr, LD(ops.Pr * ops.dt if field == 0 else (ops.dt if field == 1 else ops.Tau * ops.dt))
    F = np.zeros((M, nr), LD)
    G = G.reshape(M, nr).astype(LD)
    L = (ops.Linv_A4, ops.Linv_T, ops.Linv_S)[field].astype(LD)
    D2, i4, i2 = ops.D2_A4.astype(LD), ops.IR4_A4.astype(LD), ops.IR2_A4.astype(LD)
    for p in ((0 if field == 0 else 1,) if sym else (0, 1)):
        fe, bf = np.zeros(nr, LD), np.zeros(nr, LD)
        for jj in range(p, M, 2):
            row = M - 1 - jj
            if field == 0:
                j = M - jj
                bj, bt, g = -j * (j + 1), -2 * j, G[row]
                if jj > p:
                    fe = fe + F[row + 2]
                    g = g + h * bt * (D2 @ fe + bj * i4 * fe + i4 * bf) - bt * i2 * fe
                F[row] = L[jj] @ g
                bf = bf + bj * F[row] + (bt * fe if jj > p else 0)
            else:
                if jj > p:
                    fe = fe + 2 * h * (row + 2) * F[row + 2]
                F[row] = L[jj] @ (G[row] - (LD(1) / 2 if row == 0 else 1) * fe)
    return F.ravel()


def _run(p, G, field, torch):
    t = torch.from_numpy(np.ascontiguousarray(G)).cuda()
    return (p.a4_bsub(t) if field == 0 else p.nab2_bsub(field, t)).cpu().numpy()


@pytest.mark.parametrize("nr", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64])
def test_chains_are_no_less_exact_than_fp64(cuda, nr):
    """Whole and chunked chains at the edges of the padded block sizes (8, 16, 24, 32, 48, 64) and of one and two
    warps a group, against extended precision: at most twice the error of the same chains in FP64 (numpy; two
    samples of rounding noise) plus four roundings of the result.  Scaling the right-hand side by a power of
    two scales every bit of the result: operands have no range of their own."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, dt = 24, 1e-3
    ops = O.Operators(M, nr + 1, 2.0, dt, 1.0, 0.01)
    p = Plan(M, nr + 1, 2.0, dt, 1.0, 0.01)
    rng = np.random.default_rng(nr)
    s = np.sin(np.pi * np.arange(1, nr + 1) / (nr + 1)) ** 2
    G = (rng.standard_normal((M, nr)) * s * np.exp(-np.arange(M) / 6.0)[:, None]).ravel()
    for field in range(3):
        ref = _solve_ld(ops, G, field, False)
        n = float(np.linalg.norm(ref.astype(float)))
        if field == 0:
            o = O.A4_BSub_TSTEP_V2(G, ops.Linv_A4, ops.D2_A4, ops.IR4_A4, ops.IR2_A4, M, nr, dt, False)
        else:
            o = O.NAB2_BSub_TSTEP_V2(G, ops.Linv_T if field == 1 else ops.Linv_S, M, nr, dt if field == 1 else 0.01 * dt,
                                     False)
        e64 = float(np.linalg.norm((o - ref).astype(float))) / n
        for layout in (1, 2, 3):
            p.set_chain_layout(layout)
            y = _run(p, G, field, cuda)
            assert float(np.linalg.norm((y - ref).astype(float))) / n <= 2 * e64 + 4 * 2.0 ** -53, (field, layout)
            for k in (-300, 200):
                assert np.array_equal(_run(p, np.ldexp(G, k), field, cuda), np.ldexp(y, k))


@pytest.mark.parametrize("N_r", [20, 48])
@pytest.mark.parametrize("layout", [1, 2, 3])
def test_non_finite_operands_follow_fp64(cuda, N_r, layout):
    """An infinity or a NaN in the right-hand side reaches the modes it reaches in FP64 (the modes below it of
    its parity), with whole chains the same infinities; the others are untouched."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, nr, dt = 32, N_r - 1, 1e-3
    ops = O.Operators(M, N_r, 2.0, dt, 1.0, 0.01)
    p = Plan(M, N_r, 2.0, dt, 1.0, 0.01)
    p.set_chain_layout(layout)
    G = np.random.default_rng(1).standard_normal((M, nr))
    for field in range(3):
        clean = _run(p, G.ravel(), field, cuda).reshape(M, nr)
        for bad in (np.nan, np.inf, -np.inf):
            H = G.copy()
            H[20, 5] = bad
            with np.errstate(all="ignore"):
                if field == 0:
                    ref = O.A4_BSub_TSTEP_V2(H.ravel(), ops.Linv_A4, ops.D2_A4, ops.IR4_A4, ops.IR2_A4, M, nr, dt, False)
                else:
                    ref = O.NAB2_BSub_TSTEP_V2(H.ravel(), ops.Linv_T if field == 1 else ops.Linv_S, M, nr,
                                               dt if field == 1 else 0.01 * dt, False)
            ref = ref.reshape(M, nr)
            y = _run(p, H.ravel(), field, cuda).reshape(M, nr)
            touched = np.zeros(M, bool)
            touched[20::-2] = True
            assert np.array_equal(y[~touched], clean[~touched])
            assert not np.isfinite(y[touched]).any()
            if layout == 1:
                assert np.array_equal(y[20], ref[20], equal_nan=True)


# ---- radial contractions and the whole step --------------------------------------------------------


def _oracle_ld():
    """The oracle's functions in extended precision: its source with every array of type float one of long
    doubles."""
    import types
    from oracle import sdd_oracle as O
    with open(O.__file__) as f:
        src = f.read()
    m = types.ModuleType("sdd_oracle_ld")
    m.__dict__["__file__"] = O.__file__
    exec(compile(src.replace("dtype=float", "dtype=np.longdouble"), O.__file__, "exec"), m.__dict__)
    m.Vecs_to_X = lambda psi, t, c, M, nr, sym: np.concatenate([a.T.ravel() for a in (psi, t, c)])   # (sym off)
    return m


@pytest.mark.parametrize("nr", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32, 33, 48, 49, 64])
def test_steps_are_no_less_exact_than_fp64(cuda, nr):
    """The nonlinear term and whole steps (radial derivatives, linear terms, chains) at the edges of the padded
    block sizes, on a smooth state and on one that is not smooth at the walls, against the oracle in extended
    precision: each field at most twice the error of the FP64 oracle (two samples of rounding noise) plus four
    roundings of the result; in the two launch forms of the nonlinear term."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    M, dt, N = 24, 1e-3, 24 * nr
    Q = _oracle_ld()
    ops, opl = O.Operators(M, nr + 1, 2.0, dt, 1.0, 0.01), O.Operators(M, nr + 1, 2.0, dt, 1.0, 0.01)
    for k in ("D", "R", "Dr", "rsq", "gr", "DT0", "Linv_A4", "Linv_T", "Linv_S", "D2_A4", "IR2_A4", "IR4_A4"):
        setattr(opl, k, getattr(ops, k).astype(LD))
    p = Plan(M, nr + 1, 2.0, dt, 1.0, 0.01)
    s = np.sin(np.pi * np.arange(1, nr + 1) / (nr + 1)) ** 4
    X = O.seeded_state(M, nr, nr)
    for X in (X, (X.reshape(3, M, nr) * s).ravel()):
        Xd = cuda.from_numpy(X).cuda().reshape(1, -1)
        XL = X.astype(LD)
        want = ((p.nlin_fx, Q.NLIN_FX(XL, opl.D, opl.R, M, nr, False), O.NLIN_FX(X, ops.D, ops.R, M, nr, False)),
                (lambda x: p.step(x, 8000.0, 500.0), Q.step(opl, XL, 8000.0, 500.0, False),
                 O.step(ops, X, 8000.0, 500.0, False)))
        for split in (1, 2):
            p.set_fx_split(split)
            for fn, ref, o in want:
                y = fn(Xd).cpu().numpy().ravel()
                for f in range(3):
                    r = ref[f * N:(f + 1) * N]
                    n = float(np.linalg.norm(r.astype(float)))
                    e = [float(np.linalg.norm((v[f * N:(f + 1) * N] - r).astype(float))) for v in (y, o)]
                    assert e[0] <= 2 * e[1] + 4 * 2.0 ** -53 * n, (split, f, e, n)


@pytest.mark.parametrize("N_fm,N_r,batch,layouts", [(16, 8, 1, (4,)), (40, 20, 40, (10,)), (64, 24, 8, (3, 11)),
                                                    (64, 24, 32, (10,)), (64, 40, 12, (10,)), (64, 40, 13, (4,)),
                                                    (24, 20, 24, (4,))])
def test_batches_take_the_faster_chains(cuda, N_fm, N_r, batch, layouts):
    """The automatic layout on both sides of its lines (on 152 SMs), and the same steps as whole chains: the
    layouts differ in the order of FP64 sums of a few terms per mode, far below the 1e-12 that any layout keeps to
    the oracle."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    if cuda.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lines are in units of SMs")
    p = Plan(N_fm, N_r, 2.0, 5e-4, 1.0, 0.01)
    X = cuda.from_numpy(np.stack([O.seeded_state(N_fm, N_r - 1, k) for k in range(batch)])).cuda()
    assert p.chain_choice(batch)[0] in layouts
    y = p.step(X, 8000.0, 500.0, nsteps=3)
    p.set_chain_layout(1)
    z = p.step(X, 8000.0, 500.0, nsteps=3)
    for k in range(batch):
        assert float((y[k] - z[k]).norm() / z[k].norm()) <= 1e-12


@pytest.mark.parametrize("N_fm,N_r,sym", [(2, 3, False), (6, 34, True), (30, 8, False), (90, 23, True), (128, 65, False)])
def test_diagnostics_of_a_batch(cuda, N_fm, N_r, sym):
    """The per-shell sums over the CTAs of the radii (the last one adds them), at ragged sizes and twice in a row
    (the counters start again), against the oracle: the norm and the kinetic energy are sums of non-negative
    terms, (3 N_fm nr + 8) roundings at most; the Nusselt numbers N_fm nr roundings of their largest term's sum."""
    from oracle import sdd_oracle as O
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    nr = N_r - 1
    p = Plan(N_fm, N_r, 2.0, 1e-3, 1.0, 0.01, symmetric=sym)
    ops = O.Operators(N_fm, N_r, 2.0, 1e-3, 1.0, 0.01)
    X = np.stack([O.seeded_state(N_fm, nr, k, sym) for k in range(3)])
    Xd = cuda.from_numpy(X).cuda()
    N, u = N_fm * nr, 2.0 ** -53
    for _ in range(2):
        y = p.diagnostics(Xd).cpu().numpy()
        for b in range(3):
            assert abs(y[b, 0] - np.linalg.norm(X[b])) <= (3 * N + 8) * u * y[b, 0]
            ke = O.Kinetic_Energy(X[b], ops.R, ops.D, N_fm, nr, sym)
            # (its terms: squares of transforms of N_fm products of nr)
            assert abs(y[b, 1] - ke) <= 4 * (3 * N + 8) * u * ke + 1e-300
            for f in (1, 2):
                T = X[b, f * N:(f + 1) * N]
                nu = O.Nusselt(T, 2.0, ops.R, ops.D, N_fm, nr)
                w = sum(np.abs(ops.D[0, 1:-1]) @ np.abs(T[k * nr:(k + 1) * nr]) for k in range(0, N_fm, 2))
                assert abs(y[b, 1 + f] - nu) <= 4 * (N + 8) * u * (1 + w * ops.R[0] ** 2 / abs(O.base_state_AT(2.0)))
