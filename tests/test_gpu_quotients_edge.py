"""The shared-divisor quotients at the divisors and dividends where their final rounding has the least room: mantissas
of k ulps below 2, and quotients next to the middle of two doubles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def near_midpoints(k, most=64):
    """Dividends A 2^-52 in [1, 2) of the divisor B 2^-52, B = 2^53 - k, whose quotient A / B lies r / (B 2^54) off the
    middle of two doubles, |r| <= most: A 2^54 = B M + r with M odd."""
    B, out = 2 ** 53 - k, []
    for r in range(-most, most + 1):
        if r == 0 or k % 2 == 0:
            continue
        A = r * pow(pow(2, 54, B), -1, B) % B
        M = (A * 2 ** 54 - r) // B
        if 2 ** 52 <= A < B and M % 2 == 1:
            assert abs(2 * M * B - A * 2 ** 55) == 2 * abs(r)
            out.append(A)
    return out


@pytest.mark.parametrize("tipo", [11, 13], ids=["F1", "F3"])
def test_quotients_next_to_a_midpoint(gpu, oracle, tipo):
    """rho_R / rho, which scales every population, with rho_R = A and rho_B = B - A in the rest population alone (both
    exact, and so is their sum)."""
    cases = [(A, 2 ** 53 - k) for k in range(1, 80, 2) for A in near_midpoints(k)]
    assert len(cases) > 800 and {2 ** 53 - B for _, B in cases} >= set(range(1, 80, 2))
    n = len(cases)
    fR, fB = np.zeros((n, 19)), np.zeros((n, 19))
    fR[:, 0] = [A * 2.0 ** -52 for A, _ in cases]
    fB[:, 0] = [(B - A) * 2.0 ** -52 for A, B in cases]
    assert all(int((x + y) * 2 ** 52) == B for (x, y, (_, B)) in zip(fR[:, 0], fB[:, 0], cases))
    rng = np.random.default_rng(5)
    gm = 0.01 * rng.normal(size=(n, 3))
    F = 1e-3 * rng.normal(size=(n, 3))
    op = gpu.make_op(tipo, 0.5)
    aR, aB = gpu.dev_colisao_comum(op, 0.8, 0.1, 0.8, fR, fB, gm, F)
    for i in range(n):
        bR, bB = fR[i].copy(), fB[i].copy()
        oracle.orc().orc_colisao_comum(tipo, 0.5, 0.8, 0.1, 0.8, oracle._ptr(bR), oracle._ptr(bB),
                                       oracle._ptr(np.ascontiguousarray(gm[i])), oracle._ptr(np.ascontiguousarray(F[i])))
        assert np.array_equal(aR[i], bR) and np.array_equal(aB[i], bB), cases[i]
