"""Which solves step with one launch: by the grid's size, how full its tiles are, CPML and sheets."""
import pytest

from test_gpu_fused import DS, _params

SHEET = {"x": (0, 2), "z": (4, 0)}  # direction, polarization
CASES = [
    # (cells, npml, sheets, precision, one launch)
    ((180, 180, 92), 0, "", 0, False), ((180, 180, 94), 0, "", 0, True), ((176, 180, 100), 0, "", 0, False),
    ((104, 110, 110), 0, "z", 1, True), ((104, 104, 104), 0, "z", 1, False), ((104, 110, 120), 0, "xz", 1, False),
    ((116, 110, 110), 0, "xz", 1, True),
    ((216, 215, 216), 8, "", 1, True), ((208, 208, 208), 8, "", 1, False), ((158, 262, 222), 8, "", 1, True), ((216, 215, 216), 8, "z", 1, False),
    ((226, 226, 226), 8, "z", 1, True), ((230, 300, 360), 8, "", 0, False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("n,npml,sheets,precision,one", CASES)
def test_size_rule(pkg, n, npml, sheets, precision, one):
    extra = [f"PLANE_WAVE_SOURCES += true, {9 * DS}, 1.0, 193.4e12, 0, 2e-15, 0, 1.0, 1, {SHEET[a][0]}, {SHEET[a][1]}, 0, 0, 0, 0, 0, 0"
             for a in sheets]
    s = pkg.Setup.from_text(_params(n, npml, extra, boundary=1 if npml else 0))
    assert s.shape == n and s.view.n_sheets == len(sheets)
    sol = pkg.Solver(s, precision=precision)
    assert (sol.fused_planes > 0) == one
    sol.close()
