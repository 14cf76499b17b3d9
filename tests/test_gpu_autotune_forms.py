"""The batch autotuner times every distinct form of a group's chains once: layouts 1 and 4 to 9 run whole chains, 2 and
10 chunks with a sequential carry, 3 and 11 with a parallel one (csrc/sdd_chain.cu)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", [0, 1, 8, 10])
def test_each_form_is_timed_once(cuda, start, monkeypatch):
    from spectraldoublediffusiveconvection_gb300.batch import ShellBatch
    b = ShellBatch([dict(N_r=12, N_theta=16, Ra=7000.0), dict(N_r=20, N_theta=64, Ra=8000.0)], precision="mixed")
    for g in b.groups:
        g.plan.set_chain_layout(start)
    seen = []
    monkeypatch.setattr(b, "_time_graph", lambda reps: seen.append(
        tuple(g.plan.chain_choice(len(g.idx))[0] for g in b.groups)) or 1.0)
    monkeypatch.setattr(b, "capture", lambda steps: None)
    b.autotune(steps_per_launch=2, reps=1, fx_modes=(), chunk_scales=())
    form = lambda lay: {2: 0, 10: 0, 3: 1, 11: 1}.get(lay, 2)
    got = [tuple(map(form, s)) for s in seen]
    # the start, the two other forms of the first group, then of the second, and the tuned batch again
    assert len(got) == 6 and got[0] == got[-1]
    assert {s[0] for s in got[:3]} == {0, 1, 2} and {s[1] for s in (got[0], *got[3:5])} == {0, 1, 2}
    assert all(g.plan.chain_layout == start for g in b.groups)      # nothing gained: the choices stay
