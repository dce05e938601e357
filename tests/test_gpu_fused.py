"""The one-launch step (fused.cu) against the two sweeps, bit for bit: it evaluates the same rounded
operations, so every field, the gain state, the probe series and the DFT are equal (the sweeps
themselves are held to the reference and the oracle elsewhere).  Sizes sit at the edges of its
tiles: 30 vectors in x (4 cells in FP32, 2 in FP64), 7 rows in y, chunk borders in z; CPML widths
that are and are not whole vectors, no CPML (metal box), more material rows than fit in shared
memory, plane-wave sheets, gain."""
import numpy as np
import pytest

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
DS = 20e-9


def _params(n, npml, extra=(), boundary=1):
    core = [m - 2 * npml for m in n]
    size = [m * DS for m in core]
    mid = [0.5 * s for s in size]
    lines = ["MESH_MODE = 0", *(f"N{a} = {m}" for a, m in zip("XYZ", core)),
             *(f"D{a}_UNIFORM = {DS}" for a in "XYZ"), *(f"DOMAIN_{a}_MIN = 0" for a in "XYZ"),
             *(f"DOMAIN_{a}_MAX = {s}" for a, s in zip("XYZ", size)), "LAMBDA0 = 1550e-9", "CFL_FACTOR = 0.99",
             "N_STEPS = 50", "SAVE_EVERY = 2", f"BOUNDARY_TYPE = {boundary}", f"CPML_NPML = {npml}", "CPML_M = 3.0",
             "CPML_RERR = 1e-6", "CPML_ALPHA0 = 0.05", "CPML_KAPPA_MAX = 5.0", "CPML_ALPHA_LINEAR = true",
             "BACKGROUND_N = 1.0", "MESH_OVERRIDE_ENABLED = false", "DFT_FREQS = 168e12, 218e12, 3",
             "STRUCTURES += box, 2.0, " + ", ".join(f"{(m // 2 + q) * DS}" for m in core for q in (-2, 2)) + ', ""',
             f"DIPOLE_SOURCES += true, {mid[0]}, {mid[1]}, {mid[2]}, 1e-7, 193.4e12, 0, 2e-15, 0, 1.0, 1, 2",
             f"POINT_FIELD_DETECTORS += true, p, {0.7 * size[0]}, {mid[1]}, {mid[2]}, 2, 4", *extra]
    return "\n".join(lines) + "\n"


def _gain(n, npml):
    size = [(m - 2 * npml) * DS for m in n]
    box = ", ".join(f"{f * s}" for s in size for f in (0.25, 0.8))
    return ("TLS_ENABLED = true", "TLS_MATERIALS += g, 1550e-9, 3.1e13, 1e-12, 1e24, 0.3", "PUMP_RATE = 1e11",
            f'STRUCTURES += box, 3.4, {box}, g')


WAVES = (f"PLANE_WAVE_SOURCES += true, {4 * DS}, 1.0, 193.4e12, 0, 2e-15, 0, 1.0, 1, 4, 0, 0, 0, 0, 0, 0, 0",
         f"PLANE_WAVE_SOURCES += true, {6 * DS}, 0.5, 0, 1300e-9, 0, 20e12, 1.5, 0, 3, 2, {2 * DS}, {8 * DS}, 0, 0, {2 * DS}, {9 * DS}")


def _spheres(count, size):
    rng = np.random.default_rng(2)
    return tuple("STRUCTURES += sphere, {:.3f}, {}, {}, {}, {}, 0, 0, \"\"".format(
        rng.uniform(1.2, 3.5), *(rng.uniform(0.1, 0.9) * s for s in size), rng.uniform(1.5, 4) * DS) for _ in range(count))


def _run(pkg, text, precision, runs, seed=5):
    sol = pkg.Solver(pkg.Setup.from_text(text), precision=precision)
    rng = np.random.default_rng(seed)
    for c in FIELDS:  # every plane and face holds something, the ones that are never updated too
        sol.set_field(c, rng.normal(0, 1e-2 if c[0] == "E" else 1e-5, sol.shape))
    l0 = sol.kernel_launches
    for n in runs:
        sol.run(n)
    out = {c: sol.field(c) for c in FIELDS}
    out["series"], out["dft"] = sol.probe_series(), sol.dft(1)
    out.update({w: sol.tls_state(w) for w in ("Pz", "Pz_prev", "Nu", "Ng")})
    launches = sol.kernel_launches - l0
    rows = sol.material_rows
    sol.close()
    return out, launches, rows


CASES = [
    # (cells, npml, what)
    ((40, 17, 20), 4, ()), ((119, 15, 19), 7, ()), ((120, 28, 24), 8, ("gain",)), ((121, 22, 18), 6, ("waves",)),
    ((124, 29, 33), 10, ("gain",)), ((241, 23, 25), 9, ("gain", "waves")), ((61, 21, 75), 5, ("many",)),
    ((131, 15, 13), 0, ()), ((60, 28, 14), 0, ("waves",)),
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,npml,what", CASES)
def test_fused_step_matches_sweeps(pkg, monkeypatch, n, npml, what, precision):
    extra = []
    if "gain" in what:
        extra += _gain(n, npml)
    if "waves" in what:
        extra += WAVES
    if "many" in what:
        extra += _spheres(20, [(m - 2 * npml) * DS for m in n])
    text = _params(n, npml, extra, boundary=1 if npml else 0)
    runs = (1, 4, 6, 7)  # odd and even: the state ends in either copy
    monkeypatch.setenv("FDTD_B200_FUSED", "0")
    ref, launches2, rows = _run(pkg, text, precision, runs)
    assert rows > 128 if "many" in what else rows <= 64
    monkeypatch.setenv("FDTD_B200_FUSED", "1")
    for planes in (None, "1", "5", "64"):
        if planes:
            monkeypatch.setenv("FDTD_B200_FUSED_KCHUNK", planes)
        got, launches1, _ = _run(pkg, text, precision, runs)
        assert launches1 == launches2 - sum(runs)  # one launch a step instead of two
        for k in ref:
            assert np.array_equal(ref[k], got[k]), (k, planes)


@pytest.mark.gpu
def test_fused_step_stops_where_the_sweeps_stop(pkg, monkeypatch):
    """A run that the stability monitor stops leaves the failed step's state, in whichever copy it is."""
    n, npml = (64, 20, 22), 5
    text = _params(n, npml, _gain(n, npml)) + "STABILITY_MAX_E = 1e-300\nSTABILITY_MONITOR_INTERVAL = {}\n"
    for interval in (1, 2, 3):
        res = []
        for fused in "01":
            monkeypatch.setenv("FDTD_B200_FUSED", fused)
            sol = pkg.Solver(pkg.Setup.from_text(text.format(interval)), precision=0)
            sol.set_field("Ez", np.random.default_rng(1).normal(0, 1, sol.shape))
            with pytest.raises(pkg.FdtdError) as e:
                sol.run(60)
            assert e.value.code == pkg.FDTD_ERR_UNSTABLE
            with pytest.raises(pkg.FdtdError):
                sol.run(3)
            res.append((sol.steps_done, [sol.field(c) for c in FIELDS], sol.tls_state("Pz"), sol.probe_series()))
            sol.close()
        a, b = res
        assert a[0] == b[0]
        assert all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))
        assert np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])


@pytest.mark.gpu
def test_fused_and_two_sweep_steps_mix(pkg, monkeypatch):
    """Per-kernel timing steps with the two sweeps; runs of either kind may follow each other."""
    n, npml = (90, 24, 26), 6
    text = _params(n, npml, _gain(n, npml))
    out = []
    for fused in "01":
        monkeypatch.setenv("FDTD_B200_FUSED", fused)
        sol = pkg.Solver(pkg.Setup.from_text(text), precision=0)
        sol.set_field("Ez", np.random.default_rng(4).normal(0, 1e-2, sol.shape))
        for mode, steps in ((0, 5), (2, 4), (0, 3), (2, 1), (1, 6)):
            sol.set_timing(mode)
            sol.run(steps)
        out.append([sol.field(c) for c in FIELDS] + [sol.tls_state("Nu"), sol.dft(0)])
        sol.close()
    assert all(np.array_equal(x, y) for x, y in zip(*out))
