"""The QR's reflectors at the edges of their plain path (squared norms between 1e-280
and 1e280): an update scaled by powers of two that put its columns' squares on either
side of them has the ranks of the unscaled one and its product, scaled back, to 1e-11."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-480, -466, -464, -440, 430, 452])
def test_scaled_updates(hc, e):
    rng = np.random.default_rng(12)
    M, a, b, c = 200, 12, 9, 15
    (AU, AV), (BU, BV), (CU, CV) = (O.graded_lowrank(rng, M, r, 4.0) for r in (a, b, c))
    out = []
    for s in (0, e):
        f = 2.0 ** s
        r, U, V, _ = hc.hcore_dgemm(M, -1.0, np.asfortranarray(AU * f), AV, a, BU, BV, b, 1.0,
                                    np.asfortranarray(CU * f), CV, c, maxrk=a + c, acc=1e-3 * f)
        out.append((r, (U @ V.T) * 2.0 ** -s))
    assert out[0][0] == out[1][0]
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 1e-11 * np.linalg.norm(out[0][1])
