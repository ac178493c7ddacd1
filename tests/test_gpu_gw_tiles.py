"""GPU tests of the tiled GW convolutions at the sizes where their tiles end:
windows of one output, of a whole tile of 512 and of one more, ragged blocks
and energy counts, short chains whose edge copies cover every block, and
lines with infinities and NaNs.  Against the CPU oracle; both sides sum at
most nk * nen products of three FP64 roundings each in different orders, so
they agree to nk * nen * 2^-52 of the largest output's terms: 1e-12 covers
the largest case (2 * 1044 terms, sum of magnitudes below 40 of an output)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

DE, ALPHA = 0.01, 0.3


@pytest.fixture(scope="module")
def rgf():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from liteqt_b200 import build, rgf as R
    build.build()
    R.load()
    return R


def _arrays(rng, n, nk, nen, nx, nm):
    return [rng.normal(size=(nk, nen, nx, nm, nm)) + 1j * rng.normal(size=(nk, nen, nx, nm, nm)) for _ in range(n)]


def _run(rgf, G, W, S0, grid, imag):
    P = [np.full_like(G[0], 7.0) for _ in range(3)]
    S = [s.copy() for s in S0]
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_polarization(*G, PL=P[0], PG=P[1], PR=P[2], dE=DE, spindeg=2.0, imag_only=imag, **grid)
        ctx.gw_self_energy(*G, *W, SL=S[0], SG=S[1], SR=S[2], dE=DE, alpha_mix=ALPHA, imag_only=imag, **grid)
    return P, S


def _oracle(G, W, S0, grid, imag):
    from oracle import oracle as O
    a = (grid["nky"], grid["nkz"], grid["ndiag"], DE)
    P = O.gw_polarization(*G, *a, 2.0, imag_only=imag)
    S = [s.copy() for s in S0]
    O.gw_self_energy(*G, *W, *S, *a, ALPHA, imag_only=imag)
    return P, S


@pytest.mark.parametrize("imag", [True, False])
@pytest.mark.parametrize("nky,nkz,ndiag,nm,nx,nen", [
    (1, 1, 0, 1, 3, 20),      # window of one offset, every block an edge copy
    (1, 1, 1, 3, 4, 19),      # empty window
    (2, 1, 9, 3, 5, 65),      # band wider than the block, odd energy count
    (1, 1, 1, 9, 6, 532),     # 513 offsets: one more than a tile
    (1, 2, 0, 2, 7, 1044),    # two tiles and a remainder of energies
])
def test_gw_tiles_match_oracle(rgf, nky, nkz, ndiag, nm, nx, nen, imag):
    rng = np.random.default_rng(nen + nm)
    nk = nky * nkz
    G, W, S0 = (_arrays(rng, 3, nk, nen, nx, nm) for _ in range(3))
    grid = dict(nky=nky, nkz=nkz, ndiag=ndiag)
    P, S = _run(rgf, G, W, S0, grid, imag)
    Pr, Sr = _oracle(G, W, S0, grid, imag)
    for g, r in zip(P + S, list(Pr) + Sr):
        if np.any(r):
            assert rel_err(g, r) < 1e-12
        assert np.array_equal(g == 0, r == 0)


@pytest.mark.parametrize("imag", [True, False])
def test_gw_non_finite_values_reach_the_same_outputs(rgf, imag):
    nky, nkz, nm, nx, nen = 1, 2, 4, 6, 50
    rng = np.random.default_rng(3)
    G, W, S0 = (_arrays(rng, 3, 2, nen, nx, nm) for _ in range(3))
    G[0][1, 7, 2, 1, 2] = complex(np.inf, 1.0)
    G[2][0, 30, 3, 0, 0] = complex(0.0, np.nan)
    G[1][0, 3, 3, 3, 1] = complex(1.0, -np.inf)       # outside the band
    W[0][1, 20, 3, 2, 2] = complex(1.0, np.inf)
    W[2][0, 25, 2, 1, 1] = complex(np.nan, 0.0)
    grid = dict(nky=nky, nkz=nkz, ndiag=1)
    P, S = _run(rgf, G, W, S0, grid, imag)
    Pr, Sr = _oracle(G, W, S0, grid, imag)
    hit = 0
    for g, r in zip(P + S, list(Pr) + Sr):
        fine = np.isfinite(r)
        hit += np.count_nonzero(~fine)
        assert np.count_nonzero(fine)
        assert np.array_equal(fine, np.isfinite(g))
        assert rel_err(np.where(fine, g, 0), np.where(fine, r, 0)) < 1e-12
    assert hit
