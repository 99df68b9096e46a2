"""GPU: Sutherland's viscosity of the FP64 viscous fluxes at temperatures outside the usual range, against the
oracle: zero, negative, very small and very large ones, with and without Sutherland's constant."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t_s", [0.0, 1.0, 110.4])
@pytest.mark.parametrize("T", [0.0, -0.5, -1.0, 1e-160, 1e-100, 0.7, 1e90, 1e120, 1e200, np.inf, np.nan])
def test_viscosity(gpu_lib, t_s, T):
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    n = (6, 5, 4)
    P = abi.make_params(*n, viscous=1, rg=1.0, c_s=1e-2, t_s=t_s, bc=[dict(kind=abi.BC_PERIODIC)] * 6)
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(2)
    q = np.zeros((6, *shape))
    q[0] = 1.0
    q[1:4] = r.uniform(-0.7, 0.7, (3, *shape))
    q[4] = 1.0
    q[5] = T  # uniform: no heat flux where it is finite
    m = [np.ascontiguousarray(e + 0.1 * r.uniform(-1, 1, shape)) for e in (1., 0., 0., 0., 1., 0., 0., 0., 1.)]
    J = np.ones(shape)
    with np.errstate(all="ignore"):
        want = orc.viscous(P, q, m, J)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = Flame3D(P)
    s.set_metrics([dev(a) for a in m], dev(J))
    F = [s.viscous_field() for _ in range(3)]
    s.viscousFlux(*F, dev(q))
    s.close()
    for a, b in zip(F, want):
        g = a.cpu().numpy()
        assert (np.isfinite(g) == np.isfinite(b)).all()
        ok = np.isfinite(b)
        # ~40 roundings of sums whose terms are a few times the largest flux
        if ok.any():
            assert np.abs(g[ok] - b[ok]).max() <= 200 * 2.0 ** -53 * np.abs(b[ok]).max()
