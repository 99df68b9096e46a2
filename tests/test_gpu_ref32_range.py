"""GPU: WENO7 of the Float32 form where a smoothness indicator leaves Float32's range: its weight is zero, as
the quotient of the reference gives it (schemes.jl:178-185), and the value is that of the others."""
import numpy as np
import pytest

from flame3d_mhd_gb300.abi import BC_PERIODIC, PREC_REF32, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("character", [0, 1])
@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("towards", [1, -1])
def test_indicators_beyond_float32(gpu_lib, character, d, towards):
    """Cells of density and pressure 1e19 in a supersonic stream of order one: their squares overflow. Upwind
    of them one, two or three of a stencil's indicators do, and the right-hand side stays finite wherever
    the oracle's is."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    n = [12, 12, 12]
    n[d] = 40
    P = make_params(*n, viscous=0, character=character, phi1=0.0, phi2=5.0, phi3=6.0, precision=PREC_REF32,
                    bc=[dict(kind=BC_PERIODIC)] * 6)
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(8)
    Q = np.zeros((6, *shape), dtype=np.float32)
    Q[0] = r.uniform(0.9, 1.1, shape)
    Q[1 + d] = 3.0 * towards
    Q[4] = r.uniform(0.9, 1.1, shape) / 1.4
    at = [9, 9, 9]
    for p in (14, 30):
        at[2 - d] = p
        Q[0][tuple(at)] *= 1e19
        Q[4][tuple(at)] *= 1e19
    Q[5] = Q[4] / (Q[0] * np.float32(287.0))
    m = [np.full(shape, e, dtype=np.float32) for e in (1, 0, 0, 0, 1, 0, 0, 0, 1)]
    J = np.ones(shape, dtype=np.float32)
    want = orc.rhs32(P, Q, m, J)[:, 4:-4, 4:-4, 4:-4]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = Flame3D(P)
    s.set_metrics([dev(a) for a in m], dev(J))
    got = s.rhs(dev(Q)).cpu().numpy()[:, 4:-4, 4:-4, 4:-4]
    s.close()
    ok = np.isfinite(want)
    # cells whose faces read a large value at an outer position only
    line = np.moveaxis(want, 3 - d, -1)[:, 5, 5]
    for p in (14, 30):
        near = np.array([p - 4 - 3 * towards, p - 4 - 2 * towards])
        assert np.isfinite(line[:, near]).all()
    assert not ok.all() and np.isfinite(got[ok]).all()
    # indicators of order one, from Float32 terms of up to 2e4 of them: weights within ~3e-3, candidates that
    # differ by ~0.3
    small = ok & (np.abs(want) < 100.0)
    assert np.abs(got[small] - want[small]).max() <= 1e-2
