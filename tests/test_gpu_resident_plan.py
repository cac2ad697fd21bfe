"""Which kernel steps which box: the comparisons of test_gpu_resident.py are of two kernels only where the
library reports a plan, so the plans are asserted here over the same boxes."""
import pytest

from test_gpu_resident import BOXES, OPS, both_ways, make, same

pytestmark = pytest.mark.gpu

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
