"""GPU test of several host threads at work at the same time, each with its own
context: calls of 1, 12 and 200 energies, block sizes with different shared
memory, and convolutions on k-grids with different shared memory.  Every call
returns RGF_OK with the bits of a call made alone: nothing one call sets
(limits of a kernel, which belong to the device) may disturb another."""
import threading

import numpy as np
import pytest

from test_gpu_cms import rgf  # noqa: F401
from liteqt_b200 import synthetic as S

pytestmark = pytest.mark.gpu

MU, TEMP = (0.1, -0.1), (300.0, 300.0)


def _together(jobs):
    """Runs the jobs at the same time, a thread each; the first error, if any."""
    errors = []
    gate = threading.Barrier(len(jobs))

    def guard(job):
        try:
            job(gate)
        except Exception as e:   # noqa: BLE001
            errors.append(e)
            gate.abort()
    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


@pytest.mark.parametrize("sizes", [(64,), (128,), (8, 64, 104, 128)])
def test_concurrent_solves(rgf, sizes):  # noqa: F811
    import torch
    nx, reps = 2, 40
    dev = {nm: S.make_device(nm, nx, seed=nm) for nm in sizes}
    H = {nm: (torch.from_numpy(d.Hii).cuda(), torch.from_numpy(d.H1i).cuda()) for nm, d in dev.items()}
    E = S.energy_grid(200, -2.0, 2.0)

    def outputs(nm, nen):
        o = {k: torch.zeros(nen, nx, nm, nm, dtype=torch.complex128, device="cuda") for k in ("ldos", "ndens")}
        o["T"] = torch.zeros(nen, dtype=torch.float64, device="cuda")
        return o
    want = {}
    for nm in sizes:
        with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
            want[nm] = outputs(nm, 200)
            assert ctx.solve_energies(*H[nm], E, MU, TEMP, **want[nm]) == 0
    torch.cuda.synchronize()

    def job(nm, nen):
        def run(gate):
            out = outputs(nm, nen)
            torch.cuda.synchronize()
            with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
                gate.wait()
                for _ in range(reps):
                    assert ctx.solve_energies(*H[nm], E[:nen], MU, TEMP, **out) == 0
            for k, v in out.items():
                assert torch.equal(v, want[nm][k][:nen]), (nm, nen, k)
        return run
    _together([job(sizes[i % len(sizes)], (1, 12, 1, 200)[(i // len(sizes)) % 4]) for i in range(16)])


def test_concurrent_convolutions_on_different_grids(rgf):  # noqa: F811
    import torch
    nen, reps = 64, 40

    def job(nkz):
        def run(gate):
            g = torch.Generator(device="cuda").manual_seed(nkz)
            A = [torch.randn(4, 2, nkz, nen, dtype=torch.complex128, device="cuda", generator=g) for _ in range(5)]
            out = [torch.zeros_like(A[0]) for _ in range(3)]
            first = None
            with rgf.Context(rgf.Options()) as ctx:
                torch.cuda.synchronize()
                gate.wait()
                for _ in range(reps):
                    ctx.gw_polarization_fft(*A, PL=out[0], PG=out[1], PR=out[2], nky=1, nkz=nkz, nm=2, ndiag=1,
                                            first_ij=1, dEn=0.01, spindeg=2.0)
                    if first is None:
                        first = [o.clone() for o in out]
                        torch.cuda.synchronize()
            for a, b in zip(out, first):
                assert torch.equal(a, b)
        return run
    _together([job(n) for n in (100, 3, 90, 5, 60, 7, 33, 9)])


def test_plan_of_few_tasks_after_calls_with_other_limits(rgf):  # noqa: F811
    """A plan made for clusters, replayed after calls whose kernels take less
    shared memory."""
    import torch
    nm, nx = 128, 2
    d, small = S.make_device(nm, nx, seed=1), S.make_device(8, nx, seed=2)
    H, H1 = torch.from_numpy(d.Hii).cuda(), torch.from_numpy(d.H1i).cuda()
    ldos = torch.zeros(3, nx, nm, nm, dtype=torch.complex128, device="cuda")
    T = torch.zeros(3, dtype=torch.float64, device="cuda")
    cd = rgf.c_device()
    cd.nm, cd.nx, cd.Hii, cd.H1i = nm, nx, H.data_ptr(), H1.data_ptr()
    cd.mu[0], cd.mu[1], cd.temp[0], cd.temp[1] = *MU, *TEMP
    tasks = []
    for e in range(3):
        t = rgf.c_task()
        t.E, t.ldos, t.T = 0.3 * e, ldos[e].data_ptr(), T[e:].data_ptr()
        tasks.append(t)
    info = np.zeros(3, rgf.INFO_DTYPE)
    with rgf.Context(rgf.Options(eta_dev=1e-4)) as ctx:
        with ctx.plan([cd], tasks) as plan:
            assert plan.execute(info=info) == 0
            want = ldos.clone()
            for _ in range(3):
                o = np.zeros((1, nx, 8, 8), complex)
                assert ctx.solve_energies(small.Hii, small.H1i, np.array([0.1]), MU, TEMP, ldos=o) == 0
                ldos.zero_()
                torch.cuda.synchronize()
                assert plan.execute(info=info) == 0
                assert torch.equal(ldos, want)
