"""ShellBatch's starting choice of the chains on both sides of its lines (on 152 SMs), and the same steps as whole
chains: layouts differ in the order of FP64 sums, far below the 1e-12 that any layout keeps to the oracle (mixed plans,
whose FP32 terms may round the other way: 2^-24)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [10, 11, 38, 39, 50, 51])
def test_chains_by_the_batch(cuda, n, precision):
    from spectraldoublediffusiveconvection_gb300.batch import ShellBatch
    if cuda.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lines are in units of SMs")
    shells = [dict(N_r=8 + k % 2, N_theta=(64, 128, 256)[k % 3], Ra=8000.0) for k in range(n)]
    got = []
    for whole in (False, True):
        b = ShellBatch(shells, precision=precision)
        for g in b.groups:
            if whole:
                g.plan.set_chain_layout(1)
                continue
            M = g.plan.N_fm
            if n <= 10:
                want = 0
            elif n <= 38:
                want = 10 if M >= 128 else 8
            else:
                want = 10 if precision == "mixed" and n <= 50 and M >= 256 else 8
            assert g.plan.chain_layout == want, (n, M)
        b.capture(2)
        b.replay(2)
        got.append(b.states())
    tol = 1e-12 if precision == "fp64" else 2.0 ** -24
    for y, z in zip(*got):
        assert float(((y - z) ** 2).sum() ** 0.5) <= tol * float((z ** 2).sum() ** 0.5)
