"""GPU tests of the FFT convolutions at every transform length of the
library's own kernels (N = 64 .. 8192: a power of two of energies, the next
even count, which takes the next length, and ragged counts), at k-grids with
and without a register form, and at one energy count beyond them.  Both sides
are FFT evaluations: their errors are a few times log2(N) 2^-53 of an output's
largest magnitude, so 1e-12 bounds them with room."""
import numpy as np
import pytest

from oracle import gw_fft as F

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module")
def rgf():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from liteqt_b200 import build, rgf as R
    build.build()
    R.load()
    return R


@pytest.mark.parametrize("nky,nkz,nen", [(1, 1, n) for n in (2, 32, 34, 64, 66, 128, 130, 256, 258, 512, 514, 1024,
                                                             1026, 2048, 2050, 4096, 4098)] +
                         [(2, 1, 70), (1, 2, 100), (2, 2, 334), (4, 1, 50), (1, 4, 1000), (2, 4, 36), (4, 2, 36),
                          (4, 4, 514), (3, 1, 66), (5, 3, 46)])
def test_fft_lengths_and_k_grids(rgf, monkeypatch, nky, nkz, nen):
    import torch
    monkeypatch.setenv("RGF_GW_FFT_CHUNK", "7")
    nm, ndiag, nij, first_ij, nx, nk = 3, 1, 7, 2, 2, nky * nkz
    rng = np.random.default_rng(nen + nk)
    A = [rng.normal(size=(nij, nx, nk, nen)) + 1j * rng.normal(size=(nij, nx, nk, nen)) for _ in range(8)]
    D = [torch.from_numpy(a).cuda() for a in A]
    out = [torch.full((nij, nx, nk, nen), complex(7.0, 7.0), dtype=torch.complex128, device="cuda") for _ in range(6)]
    grid = dict(nky=nky, nkz=nkz, nm=nm, ndiag=ndiag, first_ij=first_ij, dEn=0.013)
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_polarization_fft(*D[:5], PL=out[0], PG=out[1], PR=out[2], spindeg=2.0, **grid)
        ctx.gw_self_energy_fft(*D[:3], *D[5:], SL=out[3], SG=out[4], SR=out[5], **grid)
    want = list(F.gw_polarization_fft(*A[:5], nky, nkz, nm, ndiag, first_ij, 0.013, 2.0))
    want += list(F.gw_self_energy_fft(*A[:3], *A[5:], nky, nkz, nm, ndiag, first_ij, 0.013))
    for g, w in zip(out, want):
        g = g.cpu().numpy()
        scale = np.max(np.abs(w))
        assert scale > 0
        assert np.max(np.abs(g - w)) <= TOL * scale
        for i in range(nij):
            if not F.in_band(i, first_ij, nm, ndiag):
                assert not np.any(g[i])


@pytest.mark.parametrize("nen", [40, 4098])
def test_fft_odd_line_count(rgf, nen):
    """One banded element of one block: an odd number of series."""
    import torch
    rng = np.random.default_rng(nen)
    A = [rng.normal(size=(1, 1, 2, nen)) + 1j * rng.normal(size=(1, 1, 2, nen)) for _ in range(5)]
    D = [torch.from_numpy(a).cuda() for a in A]
    out = [torch.zeros_like(D[0]) for _ in range(3)]
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_polarization_fft(*D, PL=out[0], PG=out[1], PR=out[2], nky=1, nkz=2, nm=1, ndiag=0, first_ij=1,
                                dEn=0.01, spindeg=1.0)
    for g, w in zip(out, F.gw_polarization_fft(*A, 1, 2, 1, 0, 1, 0.01, 1.0)):
        assert np.max(np.abs(g.cpu().numpy() - w)) <= TOL * np.max(np.abs(w))
