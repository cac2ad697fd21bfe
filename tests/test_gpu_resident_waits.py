"""The waits of the resident kernel: bounded, but not shorter than what a neighbour legitimately still has to do."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def desc(itlbm, nx, ny, tipo=3, prec=0):
    return itlbm.desc(nx, ny, itlbm.make_op(tipo, 0.5), tau=0.83, A_fact=0.2 if tipo < 11 else 0.08,
                      radius=0.23 * min(nx, ny), precision=prec)


def polls(itlbm, b, n):
    """Sets the limit of a batch's waits for a CTA."""
    f = itlbm.lib().itlbm_internal_batch_polls
    f.argtypes = [C.c_void_p, C.c_int]
    f(b._h, n)


def test_a_case_waits_for_its_neighbours_earlier_cases(gpu, tmp_path):
    """37 boxes of 8 tiles fill the device.  One in 37 has 200 steps to run and the others their first one, so the
    eight CTAs that take those are 40 cases behind when the last two boxes come, one of which lies half on them and
    half on CTAs that have been waiting since.  A wait of 16000 polls (5 ms or more) is several times what a tile
    takes, and far less than those 40."""
    rounds, chunk = 40, 200
    for name, box in (("long", (64, 32)), ("last", (48, 32))):
        with gpu.Case(desc(gpu, *box)) as c:
            c.step(1)
            c.save(tmp_path / name)
    with gpu.Batch(chunk=chunk) as b:
        polls(gpu, b, 16000)
        tag = 0
        for _ in range(rounds):
            b.submit_saved(tmp_path / "long", 10 ** 6, tag)
            for k in range(36):
                b.submit(desc(gpu, 64, 32), 10 ** 6, tag + 1 + k)
            tag += 37
        last = [tag, tag + 1]
        for t in last:
            b.submit_saved(tmp_path / "last", chunk + 1, t)
        b.hold_finished(True)
        b.advance()
        p = b.plan(0)
        assert p.bx * p.by == 8 and p.per_sm * 148 == 8 * 37
        assert b.plan(last[0]).bx * b.plan(last[0]).by == 6
        assert b.stats().finished == 2
        with gpu.Case(desc(gpu, 48, 32)) as c:
            for _ in range(chunk):
                c.step(1)
            c.step(1, keep_aux=True)
            want = c.read_fields()
        for t in last:
            got = b.read_fields(t, 48 * 32, gpu.FIELDS_VTK)
            assert all(np.array_equal(got[k], want[k]) for k in want)
