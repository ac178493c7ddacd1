"""GPU test of the zeros of P^R at zero energy offset: with purely imaginary G
that is symmetric in (i, j), as physical G is, its two products cancel exactly
where k - q = k, in the reference's order of operations, and the other k-points
leave the rounding of that order.  The oracle's zeros are the library's."""
import numpy as np
import pytest

from test_gpu_gw_tiles import DE, _run, rgf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("nky,nkz,ndiag,nm,nen", [(1, 1, 2, 5, 40), (1, 2, 3, 4, 70), (2, 2, 1, 6, 533)])
def test_cancelling_retarded_polarization(rgf, nky, nkz, ndiag, nm, nen, imag):  # noqa: F811
    from oracle import oracle as O
    rng = np.random.default_rng(nen)
    nk, nx = nky * nkz, 3

    def symmetric():
        a = rng.normal(size=(nk, nen, nx, nm, nm))
        return 1j * (a + np.swapaxes(a, -1, -2))
    G = [symmetric() for _ in range(3)]
    W = [symmetric() for _ in range(3)]
    P, _ = _run(rgf, G, W, [np.zeros_like(G[0]) for _ in range(3)], dict(nky=nky, nkz=nkz, ndiag=ndiag), imag)
    R = O.gw_polarization(*G, nky, nkz, ndiag, DE, 2.0, imag_only=imag)
    zero = R[2] == 0
    # every element of the band at zero offset, for one q at least
    assert np.any(zero[:, nen // 2 - 1, :, 0, 1])
    assert np.array_equal(P[2] == 0, zero)
    for g, r in zip(P, R):
        assert np.max(np.abs(g - r)) <= 1e-12 * np.max(np.abs(r))
