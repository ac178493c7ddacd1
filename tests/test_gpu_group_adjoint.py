"""GPU tests of the adjoint RGF where a cluster of CTAs shares an energy: the
analytic adjoint of the oracle, and the same bits as from single CTAs.  Chains
of up to 17 blocks run the reverse sweep in one segment, whose first product
overwrites an operand of the trace before it.  Tolerance: test_gpu_adjoint's
(1e-10 for T, 1e-9 of the largest derivative), or 8x the spread of the FP64
problem under one rounding of its input."""
import numpy as np
import pytest

from conftest import perturbed_inputs
from test_gpu_adjoint import gpu_adjoint, rgf  # noqa: F401
from liteqt_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nm,nx", [(64, 2), (64, 5), (64, 17), (128, 5), (128, 18), (96, 3)])
def test_adjoint_in_a_cluster(rgf, nm, nx):  # noqa: F811
    from oracle import oracle as O
    d = S.make_device(nm, nx, seed=600 + nm + nx)
    E = np.concatenate([[-1.7, 0.4], np.linspace(-2.0, 2.0, 158)])
    few = gpu_adjoint(rgf, d, E[:2], rgf.Options())
    many = gpu_adjoint(rgf, d, E, rgf.Options())
    assert np.all(few[5]["status"] == 0)
    for a, b in zip(few[:3], many[:3]):
        assert np.array_equal(a, b[:2])
    for _ in range(5):
        again = gpu_adjoint(rgf, d, E[:2], rgf.Options())
        assert all(np.array_equal(a, b) for a, b in zip(few[:3], again[:3]))
    T, dTdV, dTds = few[:3]
    for ie, e in enumerate(E[:2]):
        Tr, dVr, dsr = O.adjoint_numpy(O.to_blocks(d.Hii), O.to_blocks(d.H1i), e, O.Opts())
        fT = fV = fs = 0.0
        for seed in range(2):
            P, Q = perturbed_inputs(d.Hii, d.H1i, seed)
            a, b, c = O.adjoint_numpy(O.to_blocks(P), O.to_blocks(Q), e, O.Opts())
            fT, fV, fs = max(fT, abs(a - Tr)), max(fV, np.max(np.abs(b - dVr))), max(fs, abs(c - dsr))
        assert abs(T[ie] - Tr) <= max(1e-10 * max(1.0, abs(Tr)), 8 * fT)
        assert np.max(np.abs(dTdV[ie] - dVr)) <= max(1e-9 * np.max(np.abs(dVr)), 8 * fV)
        assert abs(dTds[ie] - dsr) <= max(1e-9 * max(abs(dsr), 1.0), 8 * fs)
