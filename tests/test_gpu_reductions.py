"""Read-out reductions against numpy in FP64, at the sizes where their blocks,
rows and vectors begin and end."""
import numpy as np
import pytest

from cast_simulator_b200.cuda import CudaPrecision, CudaStatevector
from cast_simulator_b200.simulator import Stream, inner_product, marginal_probabilities, qubit_populations

pytestmark = pytest.mark.gpu


def _state(n, prec, seed):
    rng = np.random.default_rng(seed)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi *= 0.7 / np.linalg.norm(psi)  # not normalised: sums carry the norm
    if prec == CudaPrecision.F32:
        psi = psi.astype(np.complex64).astype(np.complex128)
    sv = CudaStatevector(n, prec)
    sv.upload(psi)
    return sv, psi


@pytest.mark.parametrize("prec", [CudaPrecision.F64, CudaPrecision.F32])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 9, 10, 11, 12, 13, 17, 21])
def test_reductions(n, prec):
    (sv, psi), (other, phi) = _state(n, prec, n), _state(n, prec, 50 + n)
    st = Stream()
    p = np.abs(psi) ** 2
    idx = np.arange(1 << n)
    # FP64 sums of 2^n nonnegative terms: every order is within 2^n roundings of
    # the exact sum, and pairwise block sums within far fewer
    eps = 2.3e-16 * (n + 64)
    p1, norm = qubit_populations(sv, st)
    assert abs(norm - p.sum()) <= eps * p.sum()
    assert abs(sv.norm_squared() - p.sum()) <= eps * p.sum()
    for q in range(n):
        assert abs(p1[q] - p[(idx >> q) & 1 == 1].sum()) <= eps * p.sum()
    assert abs(inner_product(sv, other, st) - np.vdot(psi, phi)) <= eps * 0.49
    assert inner_product(sv, sv, st).imag == pytest.approx(0.0, abs=eps)
    picks = [[0], [n - 1], list(range(min(n, 12))), list(range(max(0, n - 12), n)),
             list(range(n - 1, -1, -2))[:12], [0, 0], [n - 1, 0, n // 2]]
    for measured in picks:
        # extended precision: numpy adds a bin's terms one after the other
        want = np.zeros(1 << len(measured), dtype=np.longdouble)
        key = np.zeros(1 << n, dtype=np.int64)
        for j, q in enumerate(measured):
            key |= ((idx >> q) & 1) << j
        np.add.at(want, key, p.astype(np.longdouble))
        got = marginal_probabilities(sv, measured, st)
        assert np.abs(got - want).max() <= eps * p.sum(), measured
