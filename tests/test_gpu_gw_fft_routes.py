"""GPU tests of the FFT convolutions on both sides of each limit between the
library's own transforms and cuFFT's (counts of k-points and of energies),
against the oracle; tolerance of test_gpu_gw_fft_sizes (FFT rounding on both
sides)."""
import numpy as np
import pytest

from oracle import gw_fft as F
from test_gpu_gw_fft_sizes import TOL, rgf  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nky,nkz,nen", [(1, 8, 256), (1, 8, 258), (9, 1, 64), (1, 3, 256), (5, 5, 60), (5, 6, 60),
                                         (3, 3, 512), (3, 3, 514), (3, 3, 992), (3, 3, 994), (2, 3, 1024), (1, 40, 34)])
def test_fft_grids_on_both_routes(rgf, nky, nkz, nen):  # noqa: F811
    import torch
    nx, nk = 2, nky * nkz
    rng = np.random.default_rng(nen + nk)
    A = [rng.normal(size=(1, nx, nk, nen)) + 1j * rng.normal(size=(1, nx, nk, nen)) for _ in range(8)]
    D = [torch.from_numpy(a).cuda() for a in A]
    out = [torch.zeros_like(D[0]) for _ in range(6)]
    grid = dict(nky=nky, nkz=nkz, nm=1, ndiag=0, first_ij=1, dEn=0.013)
    with rgf.Context(rgf.Options()) as ctx:
        ctx.gw_polarization_fft(*D[:5], PL=out[0], PG=out[1], PR=out[2], spindeg=2.0, **grid)
        ctx.gw_self_energy_fft(*D[:3], *D[5:], SL=out[3], SG=out[4], SR=out[5], **grid)
    want = list(F.gw_polarization_fft(*A[:5], nky, nkz, 1, 0, 1, 0.013, 2.0))
    want += list(F.gw_self_energy_fft(*A[:3], *A[5:], nky, nkz, 1, 0, 1, 0.013))
    for g, w in zip(out, want):
        assert np.max(np.abs(g.cpu().numpy() - w)) <= TOL * np.max(np.abs(w))


def test_slice_outside_the_band_can_be_captured(rgf):  # noqa: F811
    """A slice without a banded element is zeroed in stream order and nothing
    else, so the call can be part of a captured graph."""
    import torch
    A = [torch.ones(3, 2, 1, 8, dtype=torch.complex128, device="cuda") for _ in range(8)]
    out = [torch.full_like(A[0], 7.0) for _ in range(6)]
    grid = dict(nky=1, nkz=1, nm=4, ndiag=0, first_ij=2, dEn=0.01)
    s = torch.cuda.Stream()
    with rgf.Context(rgf.Options()) as ctx:
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=s):
            ctx.gw_polarization_fft(*A[:5], PL=out[0], PG=out[1], PR=out[2], spindeg=2.0, stream=s.cuda_stream, **grid)
            ctx.gw_self_energy_fft(*A[:3], *A[5:], SL=out[3], SG=out[4], SR=out[5], stream=s.cuda_stream, **grid)
        torch.cuda.synchronize()
        assert all(torch.all(o == 7.0) for o in out)
        g.replay()
        torch.cuda.synchronize()
        assert not any(torch.any(o != 0) for o in out)
        out[0].fill_(7.0)
        ctx.gw_polarization_fft(*A[:5], PL=out[0], PG=out[1], PR=out[2], spindeg=2.0, **grid)
        torch.cuda.synchronize()
        assert not torch.any(out[0] != 0)


def test_short_call_close_to_the_memory_limit(rgf):  # noqa: F811
    """Four series of 64 energies with 24 MB left on the device."""
    import torch
    rng = np.random.default_rng(1)
    A = [rng.normal(size=(1, 2, 2, 64)) + 1j * rng.normal(size=(1, 2, 2, 64)) for _ in range(5)]
    D = [torch.from_numpy(a).cuda() for a in A]
    out = [torch.zeros_like(D[0]) for _ in range(3)]

    def run():
        with rgf.Context(rgf.Options()) as ctx:
            ctx.gw_polarization_fft(*D, PL=out[0], PG=out[1], PR=out[2], nky=1, nkz=2, nm=1, ndiag=0, first_ij=1,
                                    dEn=0.01, spindeg=1.0)
    run()       # loads the kernels
    for o in out:
        o.zero_()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    for unit in (1 << 30, 16 << 20, 2 << 20):
        while torch.cuda.mem_get_info()[0] > (24 << 20) + unit:
            held.append(torch.cuda.caching_allocator_alloc(unit))
    try:
        run()
    finally:
        for p in held:
            torch.cuda.caching_allocator_delete(p)
        torch.cuda.empty_cache()
    for g, w in zip(out, F.gw_polarization_fft(*A, 1, 2, 1, 0, 1, 0.01, 1.0)):
        assert np.max(np.abs(g.cpu().numpy() - w)) <= TOL * np.max(np.abs(w))
