"""The FP64 collision's shared-divisor quotients round as the language's division does: against the
oracle's plain divisions, bit for bit, for gradients and forces from the subnormal range to overflow, zero
components and empty colours, on both sides of the range that takes the shared reciprocal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tipo,chi", [(1, 0.5), (3, 2.0), (12, 0.5)], ids=["P1", "P3", "F2"])
def test_quotients_round_as_divisions(gpu, oracle, tipo, chi):
    rng = np.random.default_rng(11)
    n = 4000
    W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
    cR = rng.uniform(0, 1, size=n) ** rng.integers(1, 60, size=n)
    cR[::17] = 0.0
    fR = W[None, :] * cR[:, None] * (1 + 0.01 * rng.normal(size=(n, 19)))
    fB = W[None, :] * (1 - cR)[:, None] * (1 + 0.01 * rng.normal(size=(n, 19)))
    gm = rng.normal(size=(n, 3))
    gm *= 2.0 ** rng.integers(-30, 4, size=(n, 1))
    gm[::3] *= 10.0 ** rng.integers(-170, 155, size=(len(gm[::3]), 1))        # whole vectors
    gm[1::3] *= 10.0 ** rng.integers(-90, 60, size=(len(gm[1::3]), 3))        # components apart
    gm[rng.uniform(size=(n, 3)) < 0.15] = 0.0
    gm[5] = 0.0
    gm[7] = [2.0 ** -200, 0.0, -2.0 ** -200]  # the edges of the range
    gm[8] = [2.0 ** 200, 2.0 ** -200, 0.0]
    gm[10] = [2.0 - 2.0 ** -52, 0.0, 0.0]     # |g| with a mantissa of ones
    F = rng.normal(size=(n, 3)) * 10.0 ** rng.integers(-250, -2, size=(n, 3))
    F[rng.uniform(size=(n, 3)) < 0.2] = 0.0
    op = gpu.make_op(tipo, chi)
    with np.errstate(all="ignore"):
        aR, aB = gpu.dev_colisao_comum(op, 0.8, 0.1, 0.8, fR, fB, gm, F if tipo >= 11 else None)
        for k in range(n):
            bR, bB = fR[k].copy(), fB[k].copy()
            oracle.orc().orc_colisao_comum(tipo, chi, 0.8, 0.1, 0.8, oracle._ptr(bR), oracle._ptr(bB),
                                           oracle._ptr(np.ascontiguousarray(gm[k])),
                                           oracle._ptr(np.ascontiguousarray(F[k])))
            assert np.array_equal(aR[k], bR, equal_nan=True) and np.array_equal(aB[k], bB, equal_nan=True), k
    if tipo < 11:
        f = W[None, :] * (1 + 0.01 * rng.normal(size=(n, 19)))
        got = gpu.dev_perturbacao(op, 0.1, gm, f)
        for k in range(n):
            want = f[k].copy()
            oracle.orc().orc_perturbacao(tipo, chi, 0.1, oracle._ptr(np.ascontiguousarray(gm[k])), oracle._ptr(want))
            assert np.array_equal(got[k], want, equal_nan=True), k
