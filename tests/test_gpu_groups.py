"""GPU tests of the run-time-sized block operations and of tasks shared by a
cluster of CTAs: parity with the oracle at block sizes around the limits of
the tiles (64) and of the elimination's row counts (128, 256), for task counts
that select clusters of 8, 4 and 2 and single CTAs, and bit-identical results
whatever the number of CTAs.  Tolerances: conftest.compare_spread (1e-10 of the
oracle, or 8x the spread of the FP64 problem under one rounding of its input)."""
import numpy as np
import pytest

from conftest import compare_spread, perturbed_inputs
from test_gpu_parity import gpu_solve, oracle_solve, random_sigma, rgf  # noqa: F401
from liteqt_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm,nx,nen,scattering", [
    (80, 3, 2, False),      # smallest run-time-sized block, two panels
    (88, 4, 2, True),       # odd number of 8-row subtiles
    (120, 3, 3, False),     # last size of 128 elimination rows
    (136, 3, 2, True),      # first size of 256 elimination rows, ragged tile of 8
    (248, 2, 1, False),     # largest odd size
    (64, 4, 20, True),      # clusters of 4
    (128, 3, 40, False),    # clusters of 2
])
def test_shared_and_tiled_tasks_match_oracle(rgf, nm, nx, nen, scattering):  # noqa: F811
    from oracle import oracle as O
    d = S.make_device(nm, nx, seed=900 + nm)
    E = S.energy_grid(nen, -1.9, 2.1)
    sl, sr = random_sigma(nm, nx, nen, seed=nm) if scattering else (None, None)
    opts, oopts = rgf.Options(eta_dev=1e-4, eta_lead=1e-3), O.Opts(eta_dev=1e-4, eta_lead=1e-3)
    g = gpu_solve(rgf, d.Hii, d.H1i, E, opts, sl, sr)
    r = oracle_solve(d.Hii, d.H1i, E, oopts, sl, sr)
    floors = [oracle_solve(*perturbed_inputs(d.Hii, d.H1i, seed), E, oopts, sl, sr) for seed in range(2)]
    assert g["rc"] == 0 and np.all(g["info"]["status"] == 0)
    compare_spread(g, r, floors, nm, d.H1i)
    assert np.array_equal(g["info"]["sancho_iters_left"], r["stats"]["sancho_iters_left"])


@pytest.mark.parametrize("nm", [64, 104, 128, 200, 256])
def test_results_do_not_depend_on_the_cluster(rgf, nm):  # noqa: F811
    """The same energies alone (clusters of 8), among 30 (4), 60 (2) and 160
    (single CTAs): the same bits."""
    import torch
    nx = 3
    d = S.make_device(nm, nx, seed=nm)
    H, H1 = torch.from_numpy(d.Hii).cuda(), torch.from_numpy(d.H1i).cuda()
    E = S.energy_grid(160, -2.0, 2.0)
    res = []
    with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
        for nen in (2, 30, 60, 160):
            out = {k: torch.zeros(nen, nx, nm, nm, dtype=torch.complex128, device="cuda")
                   for k in ("ldos", "ndens", "pdens", "GRi1")}
            out.update({k: torch.zeros(nen, dtype=torch.float64, device="cuda") for k in ("T", "tr", "tre")})
            ctx.solve_energies(H, H1, E[:nen], (0.1, -0.1), (300.0, 300.0), **out)
            res.append({k: v[:2].cpu().numpy() for k, v in out.items()})
    for o in res[1:]:
        for k in o:
            assert np.array_equal(o[k], res[0][k]), k


@pytest.mark.parametrize("nm", [32, 96, 128])
def test_singular_block_in_a_shared_task(rgf, nm):  # noqa: F811
    """A zero pivot zeroes the block and sets the status on every path: a
    decoupled row of zeros at E = 0 without broadening, in one of two blocks'
    interior, alone and among single-CTA tasks."""
    nx = 3
    d = S.make_device(nm, nx, seed=5)
    Hii, H1i = d.Hii.copy(), d.H1i.copy()
    Hii[1, 5, :] = Hii[1, :, 5] = 0.0
    H1i[1:, 5, :] = 0.0
    H1i[1:, :, 5] = 0.0
    for nen in (1, 160):
        E = np.concatenate([[0.0], np.linspace(0.5, 1.0, nen - 1)])
        g = gpu_solve(rgf, Hii, H1i, E, rgf.Options())
        assert g["info"]["status"][0] & rgf.RGF_ST_SINGULAR
        assert np.all(np.isfinite(g["ldos"]))
        assert not np.any(g["info"]["status"][1:] & rgf.RGF_ST_SINGULAR)
