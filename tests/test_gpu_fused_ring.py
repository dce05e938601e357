"""The fused step in chunks long enough that its ring of four stages is refilled: against the two
sweeps, bit for bit, with seeded fields everywhere.  3 planes are the first length with a refill, 4
and 5 wrap the ring, 9 wraps it twice, 64 (the whole height) up to eighteen times, on grids whose
last chunk is a remainder.  fused_planes says that the length asked for is the one launched."""
import numpy as np
import pytest

from test_gpu_fused import DS, FIELDS, WAVES, _gain, _params, _run, _spheres

CASES = [
    # (cells, npml, what)
    ((61, 21, 75), 5, "many"), ((124, 29, 33), 10, "gain"), ((121, 22, 38), 6, "waves"), ((66, 15, 34), 0, "waves"),
]


def _text(n, npml, what):
    extra = []
    if what == "gain":
        extra += _gain(n, npml)
    if what == "waves":
        extra += WAVES
    if what == "many":
        extra += _spheres(20, [(m - 2 * npml) * DS for m in n])
    return _params(n, npml, extra, boundary=1 if npml else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,npml,what", CASES)
def test_refilled_ring_matches_sweeps(pkg, monkeypatch, n, npml, what, precision):
    text = _text(n, npml, what)
    runs = (1, 6)
    monkeypatch.setenv("FDTD_B200_FUSED", "0")
    ref, _, rows = _run(pkg, text, precision, runs)
    assert rows > 128 if what == "many" else rows <= 64
    monkeypatch.setenv("FDTD_B200_FUSED", "1")
    for planes in (3, 4, 5, 9, 64):
        monkeypatch.setenv("FDTD_B200_FUSED_KCHUNK", str(planes))
        sol = pkg.Solver(pkg.Setup.from_text(text), precision=precision)
        assert sol.fused_planes == min(planes, sol.shape[2], 64)
        sol.close()
        got, _, _ = _run(pkg, text, precision, runs)
        for k in ref:
            assert np.array_equal(ref[k], got[k]), (k, planes)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_refilled_ring_stops_where_the_sweeps_stop(pkg, monkeypatch, precision):
    n, npml = (64, 20, 42), 5
    text = _params(n, npml, _gain(n, npml)) + "STABILITY_MAX_E = 1e-300\nSTABILITY_MONITOR_INTERVAL = 2\n"
    res = []
    for fused, planes in (("0", "5"), ("1", "5"), ("1", "64")):
        monkeypatch.setenv("FDTD_B200_FUSED", fused)
        monkeypatch.setenv("FDTD_B200_FUSED_KCHUNK", planes)
        sol = pkg.Solver(pkg.Setup.from_text(text), precision=precision)
        assert (sol.fused_planes != 0) == (fused == "1")
        rng = np.random.default_rng(1)
        for c in FIELDS:
            sol.set_field(c, rng.normal(0, 1 if c[0] == "E" else 1e-3, sol.shape))
        with pytest.raises(pkg.FdtdError) as e:
            sol.run(60)
        assert e.value.code == pkg.FDTD_ERR_UNSTABLE
        res.append([sol.steps_done] + [sol.field(c) for c in FIELDS] + [sol.tls_state("Pz"), sol.probe_series(), sol.dft(0)])
        sol.close()
    for r in res[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(res[0], r))
