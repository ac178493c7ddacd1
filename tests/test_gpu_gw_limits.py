"""GPU tests of the direct GW convolutions at the limits of what a call may
hold: factors that are not finite."""
import numpy as np
import pytest

from test_gpu_gw_tiles import ALPHA, _arrays, rgf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imag", [True, False])
def test_a_nan_factor_reaches_every_banded_element(rgf, imag):  # noqa: F811
    """The first energy too, whose sum is empty."""
    rng = np.random.default_rng(8)
    nm, nx, nen = 3, 5, 30
    G, W, S = (_arrays(rng, 3, 1, nen, nx, nm) for _ in range(3))
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_self_energy(*G, *W, SL=S[0], SG=S[1], SR=S[2], dE=np.nan, alpha_mix=ALPHA, nky=1, nkz=1, ndiag=1,
                           imag_only=imag)
    i = np.arange(nm)
    band = np.abs(i[:, None] - i) <= 1
    for s in S:
        assert np.array_equal(np.isnan(s), np.broadcast_to(band, s.shape))
