"""Which kernel steps which box: the comparisons of test_gpu_resident.py are of two kernels only where the
library reports a plan, so the plans are asserted here over the same boxes."""
import ctypes as C
import subprocess
import sys
from pathlib import Path

import pytest

from test_gpu_resident import BOXES, OPS, both_ways, make, same

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parent.parent

# (threads, nodes, CTAs per SM) of every configuration compiled for a storage form
CONFIGS = {0: {(64, 64), (128, 128), (160, 160), (192, 192), (224, 224), (256, 256)},
           1: {(64, 64), (128, 128), (256, 256), (256, 512)},
           2: {(64, 64), (128, 128), (256, 256), (256, 512), (256, 1024)}}
# of BOXES, those that no tiling fits; and boxes for the configurations that BOXES leaves out
BEYOND = {0: [(270, 275), (300, 300)], 1: [(400, 400)], 2: [(540, 550), (570, 560)]}
MORE = {0: [(270, 272)], 1: [(11, 6163)], 2: [(11, 6163), (540, 540)]}


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_boxes_take_every_configuration(gpu, prec):
    seen = {}
    for nx, ny in BOXES[prec] + MORE[prec]:
        for _, tipo in OPS:
            with make(gpu, nx, ny, tipo, prec) as c:
                p = c.plan()
                assert (p.bx == 0) == ((nx, ny) in BEYOND[prec]), (nx, ny, tipo)
                if p.bx:
                    w, h = -(-nx // p.bx), -(-ny // p.by)
                    assert w * h <= p.nodes and p.bx * p.by <= p.per_sm * 148
                    seen.setdefault((p.threads, p.nodes), set()).add(p.per_sm)
    assert set(seen) == CONFIGS[prec], seen
    if prec == 1:  # 256 threads of one node each: three CTAs per SM, and four with fewer registers
        assert seen[(256, 256)] == {3, 4}


@pytest.mark.parametrize("prec,nx,ny", [(p, *b) for p in MORE for b in MORE[p]])
@pytest.mark.parametrize("name,tipo", OPS, ids=[o[0] for o in OPS])
def test_many_steps_equal_single_steps(gpu, prec, nx, ny, name, tipo):
    a, b = both_ways(gpu, nx, ny, tipo, prec)
    assert same(a, b)


def test_sides_below_the_smallest_are_not_resident(gpu):
    with make(gpu, 7, 40, 3, 0) as c:
        assert c.plan().bx == 0


@pytest.mark.parametrize("prec,longest", [(0, 24), (1, 24), (2, 40)])
def test_batch_replays_take_it_from_their_length_on(gpu, prec, longest):
    for chunk in (longest - 1, longest):
        with gpu.Batch(chunk=chunk) as b:
            b.submit(gpu.desc(61, 70, gpu.make_op(3, 0.5), tau=0.83, radius=14, precision=prec), 1000, 1)
            b.submit(gpu.desc(640, 600, gpu.make_op(3, 0.5), tau=0.83, radius=80, precision=prec), 1000, 2)
            b.advance()
            assert b.plan(1).bx == 0  # step 0 alone
            b.advance()
            assert b.plan(2).bx == 0
        with gpu.Batch(chunk=chunk) as b:
            b.submit(gpu.desc(61, 70, gpu.make_op(3, 0.5), tau=0.83, radius=14, precision=prec), 1000, 1)
            b.advance()
            b.advance()
            assert (b.plan(1).bx > 0) == (chunk == longest)


class GreenContext:
    """Sixteen of the device's SMs as a green context, by the driver API."""

    def __init__(self):
        self.L = L = C.CDLL("libcuda.so.1")
        resource = C.c_char * 144
        every, part, rest = resource(), resource(), resource()
        n, self.desc, self.ctx, self.stream = C.c_uint(1), C.c_void_p(), C.c_void_p(), C.c_void_p()
        for code in (L.cuDeviceGetDevResource(0, every, 1), L.cuDevSmResourceSplitByCount(part, C.byref(n), every, rest, 0, 16),
                     L.cuDevResourceGenerateDesc(C.byref(self.desc), part, 1),
                     L.cuGreenCtxCreate(C.byref(self.ctx), self.desc, 0, 1),
                     L.cuGreenCtxStreamCreate(C.byref(self.stream), self.ctx, 1, 0)):
            if code:
                pytest.skip(f"no green context ({code})")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.L.cuStreamDestroy_v2(self.stream)
        self.L.cuGreenCtxDestroy(self.ctx)


@pytest.mark.parametrize("prec,nx,ny", [(0, 100, 100), (1, 300, 310), (2, 40, 40)])
def test_a_stream_with_fewer_sms(gpu, prec, nx, ny):
    """What a stream of a green context cannot hold at once is stepped launch by launch, in the same bits."""
    with make(gpu, nx, ny, 12, prec) as c, make(gpu, nx, ny, 12, prec) as d, GreenContext() as g:
        assert c.plan().bx
        c.step(9, stream=g.stream)
        c.step(7, keep_aux=True, stream=g.stream)
        c.sync()
        d.step(16, keep_aux=True)
        assert all((x == y).all() for x, y in zip(c.read_pops(0), d.read_pops(0)))
        f, h = c.read_fields(force=True), d.read_fields(force=True)
        assert all((f[k] == h[k]).all() for k in f)


def test_a_batch_with_fewer_sms(gpu):
    desc = gpu.desc(100, 100, gpu.make_op(3, 0.5), tau=0.83, radius=23)
    with gpu.Case(desc) as d, GreenContext() as g:
        old, ctx = C.c_void_p(), C.c_void_p()
        assert g.L.cuCtxGetCurrent(C.byref(old)) == 0 and g.L.cuCtxFromGreenCtx(C.byref(ctx), g.ctx) == 0
        assert g.L.cuCtxSetCurrent(ctx) == 0
        try:
            b = gpu.Batch()
        finally:
            assert g.L.cuCtxSetCurrent(old) == 0
        with b:
            b.hold_finished(True)
            b.submit(desc, 101, 1)
            while b.stats().finished < 1:
                b.advance()
            assert b.plan(1).bx == 0
            got = b.read_fields(1, 100 * 100)
        d.step(101, keep_aux=True)
        want = d.read_fields()
        assert all((got[k] == want[k]).all() for k in got)


def test_room_for_the_state_alone(gpu):
    """On a device with too little memory for a case's exchange between tiles, but enough for its state, the case is
    created and stepped launch by launch."""
    import torch
    for spare_mb in range(38, 70, 2):  # the state takes 40 MB, the exchange 9
        free, _ = torch.cuda.mem_get_info()
        try:
            hog = torch.empty(free - (spare_mb << 20), dtype=torch.uint8, device="cuda")
        except torch.OutOfMemoryError:
            torch.cuda.empty_cache()
            continue
        try:
            c = make(gpu, 250, 250, 3, 0)
        except gpu.ItlbmError as e:
            assert e.code == -2
            c = None
        del hog
        torch.cuda.empty_cache()
        if c:
            break
    with c, make(gpu, 250, 250, 3, 0) as d:
        assert c.plan().bx == 0 and d.plan().bx
        c.step(8)
        d.step(8)
        assert all((x == y).all() for x, y in zip(c.read_pops(0), d.read_pops(0)))


@pytest.mark.parametrize("nx,prec,most", [(40, 0, 1), (200, 0, 3), (40, 1, 1), (300, 2, 3)])
def test_a_case_loads_only_what_its_plan_looks_at(gpu, nx, prec, most):
    """The first case of a process does not load the kernels of every storage form and configuration."""
    code = (f"import sys; sys.path.insert(0, 'oracle'); import oracle; m = oracle.load_package()\n"
            f"c = m.Case(m.desc({nx}, {nx}, m.make_op(3, 0.5), radius=9, precision={prec}))\n"
            f"assert c.plan().bx and 1 <= m.lib().itlbm_internal_configurations() <= {most}")
    subprocess.run([sys.executable, "-c", code], cwd=REPO, check=True)


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_captured_steps_have_full_dependencies(gpu, prec):
    """Steps in a graph follow one another by plain edges: an early begin makes a graph of small steps slower."""
    L = C.CDLL("libcuda.so.1")
    s, g, n = C.c_void_p(), C.c_void_p(), C.c_size_t(64)
    with make(gpu, 40, 50, 3, prec) as c:
        c.step(2)
        c.sync()
        assert L.cuStreamCreate(C.byref(s), 1) == 0 and L.cuStreamBeginCapture_v2(s, 1) == 0
        c.step(5, stream=s)
        assert L.cuStreamEndCapture(s, C.byref(g)) == 0
        src, dst, data = (C.c_void_p * 64)(), (C.c_void_p * 64)(), ((C.c_ubyte * 8) * 64)()
        assert L.cuGraphGetEdges_v2(g, src, dst, data, C.byref(n)) == 0
        assert n.value == 4 and all(data[i][2] == 0 for i in range(4))  # CU_GRAPH_DEPENDENCY_TYPE_DEFAULT
        assert L.cuGraphDestroy(g) == 0 and L.cuStreamDestroy_v2(s) == 0


@pytest.mark.parametrize("prec,small,large", [(1, 128, 160), (2, 128, 256)])
def test_steps_one_by_one_do_not_crowd(gpu, prec, small, large):
    """The CTAs of both boxes find an SM each, so single steps of the larger take about as long (1.6 times where those
    of several steps waited side by side)."""
    import torch
    us = []
    for n in (small, large):
        with make(gpu, n, n, 12, prec) as c:
            times = []
            for _ in range(7):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(torch.cuda.default_stream())
                for _ in range(200):
                    c.step(1)
                e1.record(torch.cuda.default_stream())
                torch.cuda.synchronize()
                times.append(e0.elapsed_time(e1))
            us.append(min(times))
    assert us[1] < 1.3 * us[0], us


@pytest.mark.parametrize("prec,few,many", [(0, 4, 16), (1, 4, 16), (2, 4, 60)])
def test_few_small_cases_go_with_the_tables(gpu, prec, few, many):
    """Beside a box that the device does not hold, small cases are resident only where they are enough to fill it;
    which way they go changes no bit.  When that box is gone, and when there is none, they always are."""
    def desc(n, t, p):
        return gpu.desc(n, n, gpu.make_op(t, 0.5), tau=0.83, A_fact=0.2 if t < 11 else 0.08, radius=0.23 * n, precision=p)

    fields = []
    for boxes, steps in (([(640, 3, 1)] + [(100, 3, prec)] * few, 121), ([(640, 3, 1)] + [(100, 3, prec)] * many, 121),
                         ([(100, 3, prec)] * few, 121)):
        with gpu.Batch(chunk=60, diag_every=60) as b:
            b.hold_finished(True)
            for tag, box in enumerate(boxes):
                b.submit(desc(*box), steps if box[0] == 100 else 61, tag)
            b.advance()
            b.advance()
            large = boxes[0][0] == 640
            assert (b.plan(len(boxes) - 1).bx > 0) == (not large or len(boxes) > 1 + few)
            if large:
                assert b.plan(0).bx == 0 and b.stats().finished == 1
            b.advance()
            assert b.plan(len(boxes) - 1).bx > 0 and b.stats().finished == len(boxes)
            fields.append(b.read_fields(len(boxes) - 1, 100 * 100))
    for f in fields[1:]:
        assert all((f[k] == fields[0][k]).all() for k in f)


def test_boxes_without_a_partial_column_do_not_choose_narrow_tiles(gpu):
    """Their tilings are the same, and the choice holds for every case that the batch gets later."""
    for _ in range(8):
        with gpu.Batch(chunk=40) as b:
            b.submit(gpu.desc(512, 512, gpu.make_op(3, 0.5), tau=0.83, radius=100, precision=1), 1000, 1)
            for _ in range(3):
                b.advance()
            assert b.stats().narrow_edges == 0


def test_tables_that_grow_are_timed_again(gpu):
    """The windows of a second timing, on tables that have doubled, are steps like any others."""
    def desc(n, t, p):
        return gpu.desc(n, n, gpu.make_op(t, 0.5), tau=0.83, A_fact=0.2 if t < 11 else 0.08, radius=0.23 * n, precision=p)

    boxes = [(430, 3, 1), (301, 12, 0), (433, 11, 1), (590, 13, 2), (420, 1, 1)]
    with gpu.Batch(chunk=40, diag_every=40) as b:
        b.hold_finished(True)
        b.submit(desc(*boxes[0]), 161, 0)
        b.advance()
        b.advance()
        for tag, box in enumerate(boxes[1:], 1):
            b.submit(desc(*box), 81, tag)
        while b.stats().finished < len(boxes):
            b.advance()
        for tag, (n, t, p) in enumerate(boxes):
            got = b.read_fields(tag, n * n)
            with gpu.Case(desc(n, t, p)) as c:
                for _ in range(160 if tag == 0 else 80):
                    c.step(1)
                c.step(1, keep_aux=True)
                want = c.read_fields()
            assert all((got[k] == want[k]).all() for k in want), tag
