"""GPU tests of the direct GW convolutions at the limits of what a call may
hold: factors that are not finite, the longest energy axes, several chunks of
scratch, and no memory for it."""
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


def _device_arrays(n, nen, nx, nm, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(1, nen, nx, nm, nm, dtype=torch.complex128, device="cuda", generator=g) for _ in range(n)]


GRID = dict(nky=1, nkz=1, ndiag=63, imag_only=True)


def _p(ctx, G):
    import torch
    P = [torch.full_like(G[0], 7.0) for _ in range(3)]
    ctx.gw_polarization(*G, PL=P[0], PG=P[1], PR=P[2], dE=0.01, spindeg=2.0, **GRID)
    return P


def _s(ctx, G, W, S0):
    S = [s.clone() for s in S0]
    ctx.gw_self_energy(*G, *W, SL=S[0], SG=S[1], SR=S[2], dE=0.01, alpha_mix=ALPHA, **GRID)
    return S


def test_blocks_in_several_chunks(rgf):  # noqa: F811
    """Twelve blocks whose series take several chunks of the context's scratch,
    against calls of one chunk each, bit for bit, with one context."""
    import torch
    nm, nx, nen = 64, 12, 96
    G, W, S0 = (_device_arrays(3, nen, nx, nm, s) for s in (1, 2, 3))
    with rgf.Context(rgf.Options()) as ctx:
        P, S = _p(ctx, G), _s(ctx, G, W, S0)
        for b in range(0, nx, 3):
            for g, w in zip(P, _p(ctx, [x[:, :, b:b + 3].contiguous() for x in G])):
                assert torch.equal(g[:, :, b:b + 3], w)
        for b in range(2, nx - 2):   # a chain of three blocks ends as its third one
            one = [[x[:, :, [b] * 3].contiguous() for x in A] for A in (G, W, S0)]
            for g, w in zip(S, _s(ctx, *one)):
                for at in {2: (0, 1, 2), nx - 3: (nx - 3, nx - 2, nx - 1)}.get(b, (b,)):
                    assert torch.equal(g[:, :, at], w[:, :, 2])


@pytest.mark.parametrize("left_mb", [100, 40])
def test_calls_close_to_the_memory_limit(rgf, left_mb):  # noqa: F811
    """The series of all blocks do not fit, then not those of one block (56 and
    94 MB): the calls still run.  Both sums have at most 96 products of an
    output, so 1e-12 of the largest output bounds the two orders' rounding."""
    import torch
    nm, nx, nen = 64, 4, 96
    G, W, S0 = (_device_arrays(3, nen, nx, nm, s) for s in (4, 5, 6))
    with rgf.Context(rgf.Options()) as ctx:
        want = _p(ctx, G) + _s(ctx, G, W, S0)
    P, S = [torch.full_like(G[0], 7.0) for _ in range(3)], [s.clone() for s in S0]
    # the kernels are loaded: nothing but the calls' own memory is allocated below
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    for unit in (1 << 30, 16 << 20, 2 << 20):
        while torch.cuda.mem_get_info()[0] > (left_mb << 20) + unit:
            held.append(torch.cuda.caching_allocator_alloc(unit))
    try:
        with rgf.Context(rgf.Options()) as ctx:
            ctx.gw_polarization(*G, PL=P[0], PG=P[1], PR=P[2], dE=0.01, spindeg=2.0, **GRID)
            ctx.gw_self_energy(*G, *W, SL=S[0], SG=S[1], SR=S[2], dE=0.01, alpha_mix=ALPHA, **GRID)
    finally:
        for p in held:
            torch.cuda.caching_allocator_delete(p)
        torch.cuda.empty_cache()
    for g, w in zip(P + S, want):
        assert torch.max(torch.abs(g - w)) <= 1e-12 * torch.max(torch.abs(w))
        assert torch.equal(g == 0, w == 0)


def test_a_context_gives_large_scratch_back(rgf):  # noqa: F811
    """A block whose series exceed what a context keeps (256 MB)."""
    import torch
    G = _device_arrays(3, 600, 3, 64, 7)
    P = [torch.empty_like(g) for g in G]
    free = []
    with rgf.Context(rgf.Options()) as ctx:
        for _ in range(2):     # the first call loads the kernels
            ctx.gw_polarization(*G, PL=P[0], PG=P[1], PR=P[2], dE=0.01, spindeg=2.0, **GRID)
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])
    free.append(torch.cuda.mem_get_info()[0])
    assert free[2] - free[1] <= 257 << 20
    assert free[0] == free[1]
