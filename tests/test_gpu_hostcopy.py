"""Fields and populations read back through pinned memory, in one copy, plainly or in chunks by several
threads, are the device's values whatever the size, with arrays left out, and from several threads at once."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(itlbm, nx, ny):
    return itlbm.Case(itlbm.desc(nx, ny, itlbm.make_op(3, 0.5), tau=0.8, A_fact=0.1, radius=0.2 * min(nx, ny), v0=0.05))


def moments(fR, fB):
    """rho_R and rho_B of read_pops, summed in index order as the fields' kernel does."""
    out = []
    for f in (fR, fB):
        a = f.reshape(-1, 19)
        s = np.zeros(a.shape[0])
        for i in range(19):
            s = s + a[:, i]
        out.append(s)
    return out


# in one copy up to 1 MB, plainly up to 16 MB, in chunks of 512 kB up to 64 MB and of 2 MB beyond
@pytest.mark.parametrize("nx,ny", [(8, 8), (160, 163), (160, 165), (313, 335), (640, 655), (656, 655), (1031, 517), (1290, 1310)])
def test_fields_of_every_size(gpu, nx, ny):
    with make(gpu, nx, ny) as c:
        c.step(2, keep_aux=True)
        post = c.read_pops(1)
        f = c.read_fields()
        rR, rB = moments(*post)
        assert np.array_equal(f["rho_R"], rR) and np.array_equal(f["rho_B"], rB)
        # some of the arrays only
        part = {k: np.full(c.n, -1.0) for k in ("rho_B", "uy")}
        p = lambda k: part[k].ctypes.data_as(C.POINTER(C.c_double)) if k in part else None  # noqa: E731
        gpu.check(gpu.lib().itlbm_case_read_fields(c.handle, *[p(k) for k in ("rho_R", "rho_B", "ux", "uy", "uz")], None),
                  "read_fields")
        assert all(np.array_equal(part[k], f[k]) for k in part)


def test_several_threads_read_at_once(gpu):
    cases = [make(gpu, 700, 640), make(gpu, 300, 200), make(gpu, 650, 660)]
    for c in cases:
        c.step(2, keep_aux=True)
    want = [c.read_fields() for c in cases]
    bad = []

    def work(i):
        for _ in range(5):
            got = cases[i].read_fields()
            if not all(np.array_equal(got[k], want[i][k]) for k in got):
                bad.append(i)

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for c in cases:
        c.close()
    assert not bad
