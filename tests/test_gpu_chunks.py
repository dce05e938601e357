"""z-chunks of the sweeps: every chunk length gives the same bits.  Lengths at the edges of the
rule's range (1 and 16 planes, and one that does not divide the grid), on a grid with CPML and a
gain slab whose planes fall on chunk borders, against the default the rule picks."""
import numpy as np
import pytest

CASE = "step_g1_gain.params"


def _run(pkg, golden_dir, precision):
    sol = pkg.Solver(pkg.Setup.from_file(golden_dir / "cases" / CASE), precision=precision)
    rng = np.random.default_rng(3)
    for c in ("Ex", "Ey", "Ez"):
        sol.set_field(c, rng.normal(0, 1e-2, sol.shape))
    sol.run(25)
    out = [sol.field(c) for c in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")] + [sol.tls_state("Nu"), sol.probe_series()]
    sol.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 3])
def test_chunk_lengths_give_identical_bits(pkg, monkeypatch, precision):
    from conftest import GOLDEN
    ref = _run(pkg, GOLDEN, precision)
    for planes in ("1", "5", "16"):
        monkeypatch.setenv("FDTD_B200_KCHUNK", planes)
        for a, b in zip(ref, _run(pkg, GOLDEN, precision)):
            assert np.array_equal(a, b), planes
