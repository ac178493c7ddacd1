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
