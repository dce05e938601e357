"""The second copy of the fields that the fused step writes to: handed between handles of one size from
run to run (an odd run leaves a handle's state in the copy it was handed), taken by several threads
at once, returned to the memory pool with the last handle, and allocated only once enough steps pay
for it, behind steps that are under way.  The bits are those of the two sweeps."""
import ctypes as ct
import threading

import numpy as np
import pytest

from test_gpu_fused import FIELDS, _gain, _params


def _solver(pkg, text, seed, precision=0):
    sol = pkg.Solver(pkg.Setup.from_text(text), precision=precision)
    rng = np.random.default_rng(seed)
    for c in FIELDS:
        sol.set_field(c, rng.normal(0, 1e-2 if c[0] == "E" else 1e-5, sol.shape))
    return sol


def _state(sol):
    return [sol.field(c) for c in FIELDS] + [sol.tls_state("Nu"), sol.probe_series()]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("threads", [False, True])
def test_handles_share_copies(pkg, monkeypatch, precision, threads):
    sizes = [(64, 20, 22), (64, 20, 22), (64, 20, 22), (60, 24, 22)]
    texts = [_params(n, 5, _gain(n, 5)) for n in sizes]
    runs = (1, 2, 3, 1, 4)
    out = []
    for fused in "01":
        monkeypatch.setenv("FDTD_B200_FUSED", fused)
        sols = [_solver(pkg, t, seed, precision) for seed, t in enumerate(texts)]
        if threads:
            work = [threading.Thread(target=lambda s=s: [s.run(n) for n in runs]) for s in sols]
            for t in work:
                t.start()
            for t in work:
                t.join()
        else:
            for n in runs:
                for s in sols:
                    s.run(n)
            sols[1].close()  # its copies serve the others
            for s in (sols[0], sols[2], sols[3]):
                s.run(3)
        out.append([_state(s) for q, s in enumerate(sols) if threads or q != 1])
        for q, s in enumerate(sols):
            if threads or q != 1:
                s.close()
    for a, b in zip(*out):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))


def _pool_used():
    """Bytes in use of the device's default memory pool."""
    import torch
    torch.cuda.init()
    rt = ct.CDLL("libcudart.so.12")  # loaded with torch
    pool, used = ct.c_void_p(), ct.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ct.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ct.byref(used)) == 0  # cudaMemPoolAttrUsedMemCurrent
    return used.value


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [2, 3])
def test_idle_copies_are_bounded_and_returned(pkg, monkeypatch, steps):
    monkeypatch.setenv("FDTD_B200_FUSED", "1")
    base = _pool_used()
    sizes = [(120 + 4 * q, 56, 50) for q in range(7)]
    bytes_of = [6 * 8 * -(-n[0] // 16) * 16 * n[1] * n[2] for n in sizes]  # rows padded to 128 bytes
    sols = [_solver(pkg, _params(n, 0, boundary=0), 1, precision=1) for n in sizes]
    own = _pool_used() - base
    for s in sols:
        s.run(steps)
    held = _pool_used() - base - own
    assert 0 < held < 5 * max(bytes_of) * 1.1  # four copies at most
    for s in sols:
        s.close()
    assert _pool_used() <= base


@pytest.mark.gpu
def test_copy_is_taken_when_steps_pay(pkg, monkeypatch):
    n = (116, 100, 110)
    text = _params(n, 0, boundary=0)
    pay = 16 + int(350e6 / (n[0] * n[1] * n[2]))
    got, per_step = [], []
    for runs in ((10, pay - 11, 1, 10), (pay + 5, 10)):  # short runs that come to `pay` steps; one long run
        sol = _solver(pkg, text, 2, precision=1)
        assert sol.fused_planes > 0
        for k in runs:
            l0 = sol.kernel_launches
            sol.run(k)
            per_step.append((sol.kernel_launches - l0) / k)
        got.append(_state(sol))
        sol.close()  # the last handle: the next one finds no idle copy
    two, one = per_step[0], per_step[3]
    assert two > one + 0.5 and per_step[1] > one + 0.5
    assert one < per_step[4] < one + 0.5 * (two - one) and per_step[5] == one
    monkeypatch.setenv("FDTD_B200_FUSED", "0")
    for runs, g in zip(((10, pay - 11, 1, 10), (pay + 5, 10)), got):
        ref = _solver(pkg, text, 2, precision=1)
        ref.run(sum(runs))
        assert all(np.array_equal(x, y) for x, y in zip(g, _state(ref)))
        ref.close()


@pytest.mark.gpu
def test_probes_ride_up_to_the_first_fused_step(pkg, monkeypatch):
    """E-only probes ride with the next H sweep; the step before the first fused one has no such sweep."""
    n = (116, 100, 110)
    text = _params(n, 0, boundary=0).replace(", 2, 4\n", ", 2\n").replace("SAVE_EVERY = 2", "SAVE_EVERY = 1")
    out = []
    for fused in (None, "0"):
        if fused:
            monkeypatch.setenv("FDTD_B200_FUSED", fused)
        sol = _solver(pkg, text, 4, precision=1)
        assert sol.n_probes == 1 and (sol.fused_planes > 0) == (fused is None)
        sol.run(320)
        sol.run(3)
        out.append(_state(sol) + [sol.dft(0)])
        sol.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
