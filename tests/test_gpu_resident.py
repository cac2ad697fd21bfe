"""The resident multi-step kernel (a call of many steps on a box whose tiles fit the device at once) gives
the bits of the same steps taken one launch at a time: a node's update is the same code in both, so
the comparison is exact."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OPS = [("P1", 1), ("P3", 3), ("F1", 11), ("F2", 12), ("F3", 13)]
N = 14  # steps of one call, above the number from which a call takes the resident kernel


def make(itlbm, nx, ny, tipo, prec, geometry=0, v0=0.03, radius=None):
    op = itlbm.make_op(tipo, 0.5)
    d = itlbm.desc(nx, ny, op, tau=0.83, A_fact=0.2 if tipo < 11 else 0.08, precision=prec, geometry=geometry, p=2, q=1,
                   radius=0.23 * min(nx, ny) if radius is None else radius, v0=0.0 if geometry else v0)
    return itlbm.Case(d)


def results(c, strip=False):
    a, b = c.read_pops(0), c.read_pops(1)
    f = c.read_profile() if strip else c.read_fields(force=True)
    return [*a, *b, *[f[k] for k in sorted(f)]]


def same(x, y):
    return all(np.array_equal(p, q, equal_nan=True) for p, q in zip(x, y))


def both_ways(itlbm, nx, ny, tipo, prec, n=N, geometry=0, setup=None):
    got = []
    for many in (True, False):
        with make(itlbm, nx, ny, tipo, prec, geometry) as c:
            if setup:
                setup(c)
            if many:
                c.step(n, keep_aux=True)
            else:
                for _ in range(n - 1):
                    c.step(1)
                c.step(1, keep_aux=True)
            got.append(results(c, geometry == 1))
    return got


# the smallest sides, odd and thin boxes, one tile across, and a box of each tile configuration and one
# that no longer fits
BOXES = {0: [(8, 8), (9, 33), (33, 9), (40, 40), (61, 130), (190, 200), (215, 210), (235, 230), (250, 256), (270, 275), (300, 300)],
         1: [(8, 8), (9, 33), (33, 9), (40, 40), (61, 130), (270, 280), (330, 340), (380, 380), (388, 380), (400, 400)],
         2: [(8, 8), (9, 33), (33, 9), (40, 40), (61, 130), (270, 280), (380, 390), (460, 470), (540, 550), (570, 560)]}


@pytest.mark.parametrize("prec,nx,ny", [(p, *b) for p in BOXES for b in BOXES[p]])
@pytest.mark.parametrize("name,tipo", OPS, ids=[o[0] for o in OPS])
def test_many_steps_equal_single_steps(gpu, prec, nx, ny, name, tipo):
    a, b = both_ways(gpu, nx, ny, tipo, prec)
    assert same(a, b)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("name,tipo", [OPS[1], OPS[2]], ids=["P3", "F1"])
def test_strips_and_odd_counts(gpu, prec, name, tipo):
    for n in (6, 7):
        a, b = both_ways(gpu, 50, 50, tipo, prec, n=n, geometry=1)
        assert same(a, b)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("n", [6, 7])
def test_empty_sites_are_streamed_unchanged(gpu, prec, n):
    """Sites with rho <= 1e-30 (in FP32 an exact -rho0 deviation is not reached by the rounding of a zero
    population, so they may collide there; NaN sites never do) are streamed unchanged by both kernels."""
    def setup(c):
        fR, fB = c.read_pops(0)
        rng = np.random.default_rng(3)
        for k, v in ((0, 0.0), (1, np.nan)):
            at = rng.choice(c.n, 5, replace=False)
            fR.reshape(-1, 19)[at] = v
            fB.reshape(-1, 19)[at] = v
        c.write_pops(fR, fB)

    a, b = both_ways(gpu, 30, 41, 3, prec, n=n, setup=setup)
    assert same(a, b)


def test_more_steps_than_one_launch(gpu):
    with make(gpu, 16, 16, 3, 0) as c, make(gpu, 16, 16, 3, 0) as d:
        c.step(5001)
        for _ in range(10):
            d.step(500)
        d.step(1)
        assert same(c.read_pops(0), d.read_pops(0))


def test_captured_steps_replay(gpu):
    """A call under stream capture records launches that can be replayed."""
    import torch
    with make(gpu, 40, 40, 3, 1) as c, make(gpu, 40, 40, 3, 1) as d:
        s = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(s):
            g.capture_begin()
            c.step(8, stream=ctypes.c_void_p(s.cuda_stream))
            g.capture_end()
            g.replay()
            g.replay()
        s.synchronize()
        d.step(16)
        assert same(c.read_pops(0), d.read_pops(0))


def test_threads_and_streams(gpu):
    """Cases stepped by several threads on streams of their own, at once."""
    import torch
    boxes = [(100, 100, 3, 0), (200, 200, 12, 1), (120, 90, 13, 2), (64, 64, 11, 0)]
    want, got, wrong = [], [None] * len(boxes), []
    for nx, ny, t, prec in boxes:
        with make(gpu, nx, ny, t, prec) as c:
            for _ in range(200):
                c.step(1)
            want.append(c.read_pops(0))

    def work(i):
        try:
            nx, ny, t, prec = boxes[i]
            s = torch.cuda.Stream()
            with make(gpu, nx, ny, t, prec) as c:
                for _ in range(20):
                    c.step(10, stream=ctypes.c_void_p(s.cuda_stream))
                got[i] = c.read_pops(0)
        except Exception as e:  # reported by the main thread
            wrong.append(e)

    th = [threading.Thread(target=work, args=(i,)) for i in range(len(boxes))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not wrong, wrong
    for a, b in zip(want, got):
        assert same(a, b)


def test_batch_of_large_boxes(gpu):
    """FP64 boxes on both sides of the size from which a batch takes them one at a time, in each configuration."""
    boxes = [(194, 194, 12), (195, 196, 3), (230, 229, 11), (256, 250, 13), (60, 50, 1)]

    def desc(nx, ny, t):
        return gpu.desc(nx, ny, gpu.make_op(t, 0.5), tau=0.83, A_fact=0.2 if t < 11 else 0.08, radius=0.23 * min(nx, ny))

    with gpu.Batch() as b:
        b.hold_finished(True)
        for tag, box in enumerate(boxes):
            b.submit(desc(*box), 44, tag)
        while b.stats().finished < len(boxes):
            b.advance()
            b.poll()
        for tag, (nx, ny, t) in enumerate(boxes):
            got = b.read_fields(tag, nx * ny, gpu.FIELDS_VTK)
            with gpu.Case(desc(nx, ny, t)) as c:
                for _ in range(43):
                    c.step(1)
                c.step(1, keep_aux=True)
                want = c.read_fields()
            assert all(np.array_equal(got[k], want[k]) for k in want), tag
            b.release(tag)


@pytest.mark.parametrize("steps", [24, 25, 26, 40, 41, 42])
def test_short_replays(gpu, steps):
    """A batch of all storage forms at the replay lengths from which each takes the resident kernel (the replay after
    the first step has steps - 1 sub-steps)."""
    boxes = [(50, 40, 12, 0), (61, 70, 3, 1), (90, 40, 11, 2)]

    def desc(nx, ny, t, prec):
        return gpu.desc(nx, ny, gpu.make_op(t, 0.5), tau=0.83, A_fact=0.2 if t < 11 else 0.08, radius=0.23 * min(nx, ny),
                        precision=prec)

    with gpu.Batch() as b:
        b.hold_finished(True)
        for tag, box in enumerate(boxes):
            b.submit(desc(*box), steps, tag)
        while b.stats().finished < len(boxes):
            b.advance()
            b.poll()
        for tag, box in enumerate(boxes):
            got = b.read_fields(tag, box[0] * box[1], gpu.FIELDS_VTK)
            with gpu.Case(desc(*box)) as c:
                for _ in range(steps - 1):
                    c.step(1)
                c.step(1, keep_aux=True)
                want = c.read_fields()
            assert all(np.array_equal(got[k], want[k]) for k in want), tag
            b.release(tag)
