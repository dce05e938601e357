"""Probes that read only E ride along with the next step's H sweep on small grids; with per-kernel timing
they keep launches of their own.  Both record the same samples and DFT sums: over runs split anywhere,
and up to and including the step at which the stability monitor stops a run."""
import numpy as np
import pytest

from test_gpu_fused import FIELDS, _params


def _solver(pkg, extra, timing, precision):
    lines = _params((40, 24, 22), 5).replace("SAVE_EVERY = 2", "SAVE_EVERY = 1").splitlines()
    lines = [ln for ln in lines if not ln.startswith("POINT_FIELD_DETECTORS")]
    lines += [f"POINT_FIELD_DETECTORS += true, p{c}, 2e-7, 1e-7, 1e-7, {c}" for c in (0, 1, 2, 6)] + list(extra)
    sol = pkg.Solver(pkg.Setup.from_text("\n".join(lines) + "\n"), precision=precision)
    assert sol.n_probes == 4 and sol.fused_planes == 0
    rng = np.random.default_rng(3)
    for c in FIELDS:
        sol.set_field(c, rng.normal(0, 1e-2 if c[0] == "E" else 1e-5, sol.shape))
    sol.set_timing(timing)
    return sol


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 3])
def test_ride_records_what_own_launches_record(pkg, precision):
    out, launches = [], []
    for timing, runs in ((2, (12,)), (0, (12,)), (0, (1, 4, 7))):
        sol = _solver(pkg, (), timing, precision)
        l0 = sol.kernel_launches
        for n in runs:
            sol.run(n)
        launches.append(sol.kernel_launches - l0)
        out.append((sol.probe_series(), [sol.dft(p) for p in range(4)]))
        sol.close()
    assert launches[1] == launches[0] - 11 and launches[2] == launches[0] - 9  # the last step of a run has its own
    for a in out[1:]:
        assert np.array_equal(out[0][0], a[0]) and np.array_equal(out[0][1], a[1])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1, 3])
@pytest.mark.parametrize("interval", [1, 3])
def test_ride_keeps_the_sample_of_the_failed_step(pkg, precision, interval):
    out = []
    for timing in (2, 0):
        sol = _solver(pkg, ("STABILITY_MAX_E = 1e-300", f"STABILITY_MONITOR_INTERVAL = {interval}"), timing, precision)
        with pytest.raises(pkg.FdtdError) as e:
            sol.run(80)
        assert e.value.code == pkg.FDTD_ERR_UNSTABLE
        with pytest.raises(pkg.FdtdError):
            sol.run(4)
        out.append((sol.steps_done, sol.probe_series(), [sol.dft(p) for p in range(4)]))
        sol.close()
    (na, sa, da), (nb, sb, db) = out
    assert na == nb < 80 and len(sa) == na
    assert np.array_equal(sa, sb) and np.array_equal(da, db)
