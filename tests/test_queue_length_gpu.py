"""How many two-level iterations a solve queues at first comes from the last solve of
the same deck, never from another's: after another deck is loaded the next run
launches as many kernels as the same run in a fresh context."""
import pytest

pytestmark = pytest.mark.gpu


def _launches(s):
    n = s.launch_count()
    st = s.run(1)
    return s.launch_count() - n, st.cg_iters


@pytest.mark.parametrize("mixed", [0, 1])
def test_first_solve_queues_as_in_a_fresh_context(mixed, tmp_path):
    import cfdfs
    from cfdfs import meshgen
    deck = {n: meshgen.write_cavity(str(tmp_path / f"c{n}.inp"), meshgen.CavitySpec(
        n, re=200, dt=0.002, steps=5, grading=g)) for n, g in ((6, 0.0), (24, 1.5))}
    new = lambda: cfdfs.Solver(device=0, deterministic=1, precision=mixed, precond=cfdfs.PC_TWOLEVEL)  # noqa: E731
    fresh = {}
    for n in deck:
        s = new()
        s.load(deck[n])
        s.step0()
        fresh[n] = _launches(s)
        s.close()
    s = new()
    for n in (24, 6, 24):
        s.load(deck[n])
        s.step0()
        assert _launches(s) == fresh[n], n
    s.close()
