"""Field reads of every length class (plain, through the pinned chunk, several chunks) give the same
values wherever they land: fresh, touched, misaligned, pinned, and from several threads at once."""
import ctypes as ct
import threading

import numpy as np
import pytest

from test_gpu_fused import _params

PTR = ct.POINTER(ct.c_double)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(40, 41, 70), (64, 64, 33), (129, 127, 63), (170, 161, 153), (180, 181, 193)])
def test_reads_into_any_memory(pkg, n):
    import torch
    lib = pkg.load_library()
    rng = np.random.default_rng(7)
    sols, ref = [], []
    for _ in range(3):
        sol = pkg.Solver(pkg.Setup.from_text(_params(n, 6)), precision=1)
        ref.append(rng.normal(size=n))
        sol.set_field("Ey", ref[-1])
        sols.append(sol)
    cells = int(np.prod(n))

    def read(q, out):
        assert lib.fdtd_get_field(sols[q]._h, 1, out.ctypes.data_as(PTR)) == 0
        return out.reshape(n)

    for shift in (0, 1, 511):
        buf = np.full(cells + shift + 1, np.nan)
        assert np.array_equal(read(0, buf[shift:shift + cells]), ref[0])
        assert np.isnan(buf[:shift]).all() and np.isnan(buf[shift + cells:]).all()
    assert np.array_equal(sols[0].field("Ey"), ref[0])
    pinned = torch.empty(cells, dtype=torch.float64, pin_memory=True).numpy()
    assert np.array_equal(read(0, pinned), ref[0])
    bad = []

    def reader(q):
        out = np.empty(cells)
        for _ in range(6):
            out[:] = 0
            if not np.array_equal(read(q, out), ref[q]) or not np.array_equal(sols[q].field("Ey"), ref[q]):
                bad.append(q)

    work = [threading.Thread(target=reader, args=(q,)) for q in range(3)]
    for t in work:
        t.start()
    for t in work:
        t.join()
    assert not bad
    for s in sols:
        s.close()
