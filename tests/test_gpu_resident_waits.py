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


def expired(itlbm, call):
    with pytest.raises(itlbm.ItlbmError) as e:
        call()
    assert e.value.code == -7  # ITLBM_E_TIMEOUT


def test_a_case_whose_wait_ran_out(gpu, tmp_path):
    """Every call that steps it or reads it says so, until it is given a new state; then it goes on as any other."""
    with gpu.Case(desc(gpu, 40, 50)) as c, gpu.Case(desc(gpu, 40, 50)) as d:
        c.step(10)
        pops = c.read_pops(0)
        c.step(10, keep_aux=True)
        c.sync()
        f = gpu.lib().itlbm_internal_case_expire
        f.argtypes = [C.c_void_p]
        assert f(c.handle) == 0
        done = c.steps_done
        for call in (lambda: c.step(10), lambda: c.step(1), c.sync, lambda: c.read_pops(0), c.read_fields, lambda: c.diag_drop(19),
                     lambda: c.save(tmp_path / "s")):
            expired(gpu, call)
        assert c.steps_done == done
        c.write_pops(*pops)
        c.step(30)
        d.step(40)
        assert all(np.array_equal(x, y) for x, y in zip(c.read_pops(0), d.read_pops(0)))


def test_a_batch_whose_wait_ran_out(gpu, tmp_path):
    """The cases of test_a_case_waits_for_its_neighbours_earlier_cases, in fewer rounds of longer tiles, with a limit
    below the time of one: the launch ends by itself, the advance says so, and so does every one after it."""
    with gpu.Case(desc(gpu, 64, 32)) as c:
        c.step(1)
        c.save(tmp_path / "long")
    with gpu.Case(desc(gpu, 48, 32)) as c:
        c.step(1)
        c.save(tmp_path / "last")
    with gpu.Batch() as b:
        polls(gpu, b, 200)
        for k in range(0, 37 * 8, 37):
            b.submit_saved(tmp_path / "long", 10 ** 6, k)
            for j in range(36):
                b.submit(desc(gpu, 64, 32), 10 ** 6, k + 1 + j)
        for t in (1000, 1001):
            b.submit_saved(tmp_path / "last", 10 ** 6, t)
        for call in (b.advance, b.advance, lambda: b.save(1000, tmp_path / "s")):
            expired(gpu, call)
    with gpu.Batch() as b:  # the device is none the worse
        b.submit(desc(gpu, 64, 32), 30, 1)
        while b.stats().finished < 1:
            b.advance()


MIXED = [(100, 100, 3, 0), (61, 70, 11, 0), (40, 90, 12, 0), (120, 110, 3, 1), (64, 64, 11, 1), (90, 95, 13, 2), (50, 60, 12, 2)]


def check_against_single_steps(itlbm, b, steps, boxes):
    for tag, box in enumerate(boxes):
        got = b.read_fields(tag, box[0] * box[1], itlbm.FIELDS_VTK)
        with itlbm.Case(desc(itlbm, *box)) as c:
            for _ in range(steps - 1):
                c.step(1)
            c.step(1, keep_aux=True)
            want = c.read_fields()
        assert all(np.array_equal(got[k], want[k]) for k in want), box


@pytest.mark.parametrize("room", [0, 1, 60 * 3 + 1, 60 * 7 + 10])
def test_tags_start_again(gpu, room):
    """A batch comes to the end of its tags before, in and after the replay that would use the last `room` of them."""
    L = gpu.lib()
    L.itlbm_internal_batch_tag.argtypes = [C.c_void_p, C.c_uint]
    L.itlbm_internal_batch_tag_of.argtypes = [C.c_void_p]
    L.itlbm_internal_batch_tag_of.restype = C.c_uint
    with gpu.Batch(chunk=60, diag_every=60) as b:
        b.hold_finished(True)
        for tag, box in enumerate(MIXED):
            b.submit(desc(gpu, *box), 361, tag)
        b.advance()
        b.advance()
        assert all(b.plan(tag).bx > 0 for tag in range(len(MIXED)))
        assert L.itlbm_internal_batch_tag(b._h, 2 ** 31 - 1 - room) == 3
        tags = []
        while b.stats().finished < len(MIXED):
            b.advance()
            b.poll()
            tags.append(L.itlbm_internal_batch_tag_of(b._h))
        assert min(tags[:-1]) < 2000 and max(tags) < 2 ** 31
        check_against_single_steps(gpu, b, 361, MIXED)


def test_a_replay_longer_than_a_launch(gpu):
    boxes = [(16, 16, 12, 0), (20, 17, 3, 1), (33, 9, 11, 2), (24, 24, 3, 0)]
    with gpu.Batch(chunk=5000, diag_every=5000) as b:
        b.hold_finished(True)
        for tag, box in enumerate(boxes):
            b.submit(desc(gpu, *box), 4801, tag)
        b.advance()
        b.advance()
        assert b.stats().finished == len(boxes) and all(b.plan(tag).bx > 0 for tag in range(len(boxes)))
        check_against_single_steps(gpu, b, 4801, boxes)
