"""GPU tests of the direct GW convolutions at the limits of what a call may
hold: factors that are not finite, and the longest energy axes."""
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


def test_more_energies_than_a_grid_has_tiles(rgf):  # noqa: F811
    """65535 x 32 energies and one tile more; unit pulses, whose sums are
    single products at known offsets."""
    import torch
    nen, nx, h = 65535 * 32 + 30, 3, (65535 * 32 + 30) // 2 - 1
    a, b = 5, nen - 3
    shift = 700_001
    z = lambda: torch.zeros(1, nen, nx, 1, 1, dtype=torch.complex128, device="cuda")
    GL, GG, GR = z(), z(), z()
    GL[0, a], GG[0, b], GG[0, a + shift] = 2j, 3j, 5j
    P = [z() for _ in range(3)]
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_polarization(GL, GG, GR, PL=P[0], PG=P[1], PR=P[2], dE=1.0, spindeg=1.0, nky=1, nkz=1, ndiag=0,
                            imag_only=True)
        f = 1.0 / (2 * 3.14159265359)
        # P^<(n) = G^<(e) G^>(e - n): n = -shift; P^>: n = +shift (b - a lies outside the window)
        want = [{h - shift: 1j * 10 * f}, {h + shift: 1j * 10 * f}, {}]
        for p, w in zip(P, want):
            p = p[0, :, :, 0, 0].cpu().numpy()
            assert sorted(set(np.nonzero(p)[0])) == sorted(w)
            for k, v in w.items():
                assert np.all(np.abs(p[k] - v) < 1e-14)
        # S^<(e) = G^<(e - n) W^<(n) at e = a + n
        W, S = [z() for _ in range(3)], [z() for _ in range(3)]
        W[0][0, h + shift] = 7.0
        ctx.gw_self_energy(GL, GG, GR, *W, SL=S[0], SG=S[1], SR=S[2], dE=1.0, alpha_mix=1.0, nky=1, nkz=1, ndiag=0,
                           imag_only=True)
        s = S[0][0, :, :, 0, 0].cpu().numpy()
        assert list(set(np.nonzero(s)[0])) == [a + shift]
        assert np.all(np.abs(s[a + shift] + 14 * f) < 1e-14)
