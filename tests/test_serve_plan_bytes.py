"""The operators' share of the server's memory admission against what the library allocates."""
import pytest

SHAPES = [(64, 20), (256, 26), (256, 34), (512, 48), (540, 65), (16, 10)]


@pytest.mark.parametrize("M,N_r", SHAPES)
@pytest.mark.parametrize("mixed", [False, True])
def test_counts_the_padded_blocks(M, N_r, mixed):
    """Every mode has 13 blocks of its own, padded to ld x ld words and a row of exponents."""
    pytest.importorskip("torch")
    from spectraldoublediffusiveconvection_gb300 import serve
    nr = N_r - 1
    ld = 8 * -(-nr // 8) if nr <= 32 else 16 * -(-nr // 16)
    srv = serve.Server(device="cpu", memory_budget=1, int_precision="mixed" if mixed else "fp64", con_mixed=2 * mixed)
    for kind in ("integrate", "continue"):
        b = srv.plan_bytes(serve.Request(kind, N_r, M, 8000.0))
        assert b >= 8 * 13 * M * ld * (ld + 1) + (12 * M * nr * ld if mixed else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N_r", SHAPES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_matches_the_devices_memory(cuda, M, N_r, precision):
    """Four plans' share of the free memory: within the page of 2 MB that a plan's small tables fill in part, and 4% for
    what the driver keeps beside them."""
    from spectraldoublediffusiveconvection_gb300.operators import plan_arrays
    from spectraldoublediffusiveconvection_gb300.plan import Plan
    from spectraldoublediffusiveconvection_gb300.serve import table_bytes
    A = plan_arrays(M, N_r, 2.0, 1e-3, 1.0, 0.01)
    make = lambda: Plan(M, N_r, 2.0, 1e-3, 1.0, 0.01, precision=precision, arrays=A)
    make().close()                                       # (the transforms' tables, shared by all plans of a size)
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    plans = [make() for _ in range(4)]
    used = (free - cuda.cuda.mem_get_info()[0]) / 4
    for p in plans:
        p.close()
    want = table_bytes(M, N_r - 1, precision == "mixed")
    assert abs(used - want) <= 2.5 * 2 ** 20 + 0.04 * want, (used, want)
