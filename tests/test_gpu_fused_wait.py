"""The fused step's waits are bounded.  With the row-ready barriers held (FDTD_B200_FUSED_HOLD: they
never complete) and a 20 us bound, every block gives up after its copies have arrived: fdtd_run
returns FDTD_ERR_TIMEOUT, the handle stays stopped, it is destroyed cleanly and a new handle steps
as the sweeps do.  No GPU fault is involved: the kernel flags the status word and returns."""
import numpy as np
import pytest

from conftest import GOLDEN

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("planes", ["2", "12"])
def test_fused_wait_expires_with_timeout_status(pkg, monkeypatch, precision, planes):
    s = pkg.Setup.from_file(GOLDEN / "cases" / "step_g0_sphere.params")
    out = []
    for fused in "01":
        monkeypatch.setenv("FDTD_B200_FUSED", fused)
        monkeypatch.setenv("FDTD_B200_FUSED_KCHUNK", planes)
        if fused == "1":
            monkeypatch.setenv("FDTD_B200_FUSED_HOLD", "1")
            monkeypatch.setenv("FDTD_B200_WAIT_NS", "20000")
            held = pkg.Solver(s, precision=precision)
            for n in (3, 1):
                with pytest.raises(pkg.FdtdError) as e:
                    held.run(n)
                assert e.value.code == pkg.FDTD_ERR_TIMEOUT and "wait" in str(e.value)
            held.close()
            monkeypatch.delenv("FDTD_B200_FUSED_HOLD")
            monkeypatch.delenv("FDTD_B200_WAIT_NS")
        sol = pkg.Solver(s, precision=precision)
        sol.run(20)
        out.append([sol.field(c) for c in FIELDS])
        sol.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
