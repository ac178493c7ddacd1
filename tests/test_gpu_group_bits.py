"""GPU tests that a task's results do not depend on the CTAs that share it: the
same energies in clusters of 8, 4 and 2 CTAs and by single CTAs (the count of
energies in a call decides), for every output of every solve, bit for bit."""
import numpy as np
import pytest

from conftest import random_sigma
from test_gpu_cms import OUTS, _gpu, rgf  # noqa: F401
from liteqt_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k][:len(a[k])]), k


@pytest.mark.parametrize("nm", [64, 128, 256])
def test_ballistic_cluster_repeats(rgf, nm):  # noqa: F811
    """Every CTA of a cluster factorises the same left broadening, part of
    which the others update: twenty runs, and a run by single CTAs."""
    d = S.make_device(nm, 2, seed=nm)
    E = S.energy_grid(150, -2.0, 2.0)
    ref = _gpu(rgf, d, None, E, rgf.Options(eta_dev=1e-4))
    for _ in range(20):
        _same(_gpu(rgf, d, None, E[:3], rgf.Options(eta_dev=1e-4)), ref)


# energies: by single CTAs, then in clusters of 2, 4 and 8
COUNTS = (160, 60, 30, 2)


@pytest.mark.parametrize("nm,overlap,scatter", [(64, False, True), (64, True, False), (104, False, True),
                                                (104, True, True), (128, True, True), (128, False, True)])
def test_every_output_of_a_solve(rgf, nm, overlap, scatter):  # noqa: F811
    d = S.make_device(nm, 3, seed=nm)
    Sii = S.make_overlap(nm, 3, seed=nm) if overlap else None
    E = S.energy_grid(COUNTS[0], -2.0, 2.0)
    sl, sr = (random_sigma(nm, 3, 60, seed=nm) if scatter else (None, None))
    if scatter:   # the first 60 energies' are compared, the others only fill the launch
        sl, sr = (np.concatenate([a, np.broadcast_to(a[:1], (COUNTS[0] - 60,) + a.shape[1:])]) for a in (sl, sr))
    opts = rgf.Options(eta_dev=1e-4)
    ref = _gpu(rgf, d, Sii, E, opts, sl, sr)
    for n in COUNTS[1:]:
        _same(_gpu(rgf, d, Sii, E[:n], opts, *((sl[:n], sr[:n]) if scatter else ())), ref)


@pytest.mark.parametrize("nm", [64, 88, 128])
def test_w_solves(rgf, nm):  # noqa: F811
    from test_gpu_w import _gpu_w
    Vii, V1i = S.make_coulomb(nm, 3, seed=nm)
    P = S.make_polarization(nm, 3, COUNTS[0], seed=3)
    ref, _ = _gpu_w(rgf, Vii, V1i, *P)
    for n in COUNTS[1:]:
        _same(_gpu_w(rgf, Vii, V1i, *(p[:n] for p in P))[0], ref)


@pytest.mark.parametrize("plan", [False, True])
def test_few_tasks_of_different_sizes(rgf, plan):  # noqa: F811
    """One launch of few tasks, nb = 32 among larger ones (where alone it takes
    no cluster), against launches of single CTAs."""
    import torch
    devices, tasks, keep, want = [], [], [], []
    for k, nm in enumerate((32, 64, 96, 128, 256)):
        d = S.make_device(nm, 3, seed=nm)
        H, H1 = torch.from_numpy(d.Hii).cuda(), torch.from_numpy(d.H1i).cuda()
        cd = rgf.c_device()
        cd.nm, cd.nx, cd.Hii, cd.H1i = nm, 3, H.data_ptr(), H1.data_ptr()
        cd.mu[0], cd.mu[1], cd.temp[0], cd.temp[1] = 0.1, -0.1, 300.0, 300.0
        devices.append(cd)
        out = {n: torch.zeros(2, 3, nm, nm, dtype=torch.complex128, device="cuda")
               for n in ("ldos", "ndens", "pdens", "GRi1")}
        out["T"] = torch.zeros(2, dtype=torch.float64, device="cuda")
        for e in range(2):
            t = rgf.c_task()
            t.device, t.E = k, (-1.3, 0.6)[e]
            for n, v in out.items():
                setattr(t, n, v[e:].data_ptr())
            tasks.append(t)
        keep.append((H, H1, out))
        E = np.concatenate([[-1.3, 0.6], np.linspace(-2.0, 2.0, 158 if nm < 256 else 148)])
        full = {n: torch.zeros((len(E),) + v.shape[1:], dtype=v.dtype, device="cuda") for n, v in out.items()}
        with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
            ctx.solve_energies(H, H1, E, (0.1, -0.1), (300.0, 300.0), **full)
        want.append({n: v[:2] for n, v in full.items()})
    with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
        if plan:
            with ctx.plan(devices, tasks) as p:
                p.execute(info=np.zeros(len(tasks), rgf.INFO_DTYPE))
        else:
            ctx.solve_batch(devices, tasks)
    torch.cuda.synchronize()
    for (_, _, out), w in zip(keep, want):
        for n in out:
            assert torch.equal(out[n], w[n]), n
