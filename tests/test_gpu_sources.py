"""Sources that meet in one vector: two plane-wave sheets that cross, two point sources in one cell of
the crossing line, one in the cell next to it and one of another component, against the oracle, for
the two sweeps and the fused step."""
import numpy as np
import pytest

from conftest import GOLDEN
from test_gpu_parity import FIELDS, field_rel_l2, fields

DIPOLES = [(2, 0), (2, 0), (2, 1), (0, 0)]  # (component, cells in +x from the crossing line)


@pytest.mark.gpu
@pytest.mark.parametrize("normal", ["x", "z"])
@pytest.mark.parametrize("precision,tol", [(1, 1e-12), (0, 1e-5)])
def test_crossing_sources_match_oracle(pkg, oracle, monkeypatch, normal, precision, tol):
    text = (GOLDEN / "cases" / "step_g0_sphere.params").read_text()
    for a, n, m, old, size in (("X", 10, 37, "250e-9", "925e-9"), ("Y", 9, 25, "225e-9", "625e-9"), ("Z", 8, 21, "200e-9", "525e-9")):
        text = text.replace(f"N{a} = {n}", f"N{a} = {m}").replace(f"DOMAIN_{a}_MAX = {old}", f"DOMAIN_{a}_MAX = {size}")
    lines = [ln for ln in text.splitlines() if not ln.startswith("DIPOLE_SOURCES")]
    # sheets into one component: normal to x or z, and to y
    wave = "PLANE_WAVE_SOURCES += true, {}, {}, 193.4e12, 0, 2e-15, 0, 1.0, 1, {}, {}, 0, 0, 0, 0, 0, 0"
    comp = 2 if normal == "x" else 0
    lines += [wave.format("412e-9", 1.0, 0, 2) if normal == "x" else wave.format("262e-9", 1.0, 4, 0), wave.format("312e-9", 0.7, 2, comp)]
    for q, (c, dx) in enumerate(DIPOLES):
        lines.append(f"DIPOLE_SOURCES += true, {412e-9 + dx * 25e-9}, 312e-9, 262e-9, {(q + 1) * 1e-7}, 193.4e12, 0, 2e-15, 0, 1.0, 1, {c if normal == 'x' else 2 - c}")
    s = pkg.Setup.from_text("\n".join(lines) + "\n")
    v = s.view
    assert v.n_sheets == 2 and v.n_dipoles == len(DIPOLES)
    assert {v.sheets[q].comp for q in range(2)} == {comp}
    d = [v.dipoles[q] for q in range(len(DIPOLES))]
    assert v.sheets[0].plane == (d[0].i if normal == "x" else d[0].k) and v.sheets[1].plane == d[0].j
    assert (d[0].i, d[0].j, d[0].k) == (d[1].i, d[1].j, d[1].k) and d[2].i == d[0].i + 1
    o = oracle.OracleSolve(s, 0)
    o.run(70)
    ref = {c: o.field(c) for c in FIELDS}
    for fused in "01":
        monkeypatch.setenv("FDTD_B200_FUSED", fused)
        sol = pkg.Solver(s, precision=precision)
        sol.run(70)
        mine = fields(sol)
        assert field_rel_l2(mine, ref, "E") <= tol and field_rel_l2(mine, ref, "H") <= tol, fused
        sol.close()
