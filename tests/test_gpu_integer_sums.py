"""GPU: the viscous gradients as integer differences and the finite-volume linear states as integer
strips (f3d_fixed.cuh) against the oracle. Sizes around strips and blocks; velocities that jump by up
to 1e12 between neighbouring blocks, values outside the integer range (below 2^-823) and
non-finite ones, which take the FP64 forms."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
PER = [dict(kind=abi.BC_PERIODIC)] * 6


def _blocks(shape, r, lo, hi):
    b = 10.0 ** r.uniform(lo, hi, [-(-n // 7) for n in shape])
    return b.repeat(7, 0).repeat(7, 1).repeat(7, 2)[:shape[0], :shape[1], :shape[2]]


@pytest.mark.parametrize("n", [(4, 5, 6), (31, 9, 8), (33, 6, 12)])
@pytest.mark.parametrize("kind", ["smooth", "wide", "tiny", "nonfinite"])
def test_viscous_gradients(gpu_lib, n, kind):
    import torch
    from scipy.ndimage import maximum_filter

    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    P = abi.make_params(*n, viscous=1, rg=1.0, c_s=1e-2, t_s=1.0, bc=PER)
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(17)
    scale = {"smooth": 1.0, "wide": _blocks(shape, r, -6, 6), "tiny": 1e-260, "nonfinite": 1.0}[kind]
    q = np.empty((6, *shape))
    q[0] = r.uniform(0.8, 1.2, shape)
    q[1:4] = scale * r.uniform(-0.7, 0.7, (3, *shape))
    q[5] = r.uniform(0.6, 0.8, shape)
    q[4] = q[0] * q[5]
    if kind == "nonfinite":
        q[1, 6, 6, 6], q[2, 7, 5, 5] = np.nan, np.inf
    m = [np.ascontiguousarray(e + 0.1 * r.uniform(-1, 1, shape)) for e in (1., 0, 0, 0, 1, 0, 0, 0, 1)]
    J = np.ones(shape)
    s = Flame3D(P)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s.set_metrics([dev(a) for a in m], dev(J))
    F = [s.viscous_field() for _ in range(3)]
    s.viscousFlux(*F, dev(q))
    want = orc.viscous(P, q, m, J)
    cut = (slice(2, -2),) * 3
    vel = maximum_filter(np.abs(q[1:4]).max(0), size=5)[cut]
    tem = maximum_filter(q[5], size=5)[cut]
    here = np.abs(q[1:4]).max(0)[cut]
    # a gradient is three differences (sum of weights 1.5) times metrics below 1.1, a stress at most
    # 4/3 + 2 * 2/3 of them, a flux three stresses times metrics: below 20 mu W with ~20 roundings on
    # each side; mu <= 0.01, conductivity <= 0.05 at these temperatures
    vel, here = (np.where(np.isfinite(v), v, 1.0) for v in (vel, here))
    stress, heat = 1000 * EPS * 0.01 * vel, 1000 * EPS * 0.05 * tem
    for a, b in zip(F, want):
        g = a.cpu().numpy()
        assert (np.isfinite(g) == np.isfinite(b)).all()
        ok = np.isfinite(b)
        err = np.where(ok, np.abs(np.where(ok, g, 0) - np.where(ok, b, 0)), 0)
        assert ok.all() == (kind != "nonfinite")
        assert (err[:3] <= stress).all()
        assert (err[3] <= 3 * stress * here + heat).all()
    s.close()


@pytest.mark.parametrize("n", [(8, 9, 10), (31, 17, 16), (33, 15, 14)])
@pytest.mark.parametrize("phi", [0.0, 0.5, 0.1234567, 1.0])
@pytest.mark.parametrize("scheme", [abi.SCHEME_FVM_EIGEN, abi.SCHEME_FVM_CONS])
def test_finite_volume_linear_states(gpu_lib, n, phi, scheme):
    """Every face linear: within 1e-12 of the oracle's fluxes, the bound of the finite-volume faces."""
    import torch

    from conftest import rel_linf
    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    from test_oracle_fvm import _coords, _state
    P = abi.make_params(*n, viscous=0, phi1=5.0, phi2=6.0, phi3=7.0, linear_phi=phi, scheme=scheme, bc=PER)
    x, y, z = _coords(P, 0.02)
    m, J, Q, U = orc.prepare(P, _state(P, 21, spikes=0, noise=0.03), x, y, z)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = Flame3D(P)
    s.set_metrics([dev(a) for a in m], dev(J))
    s.set_coordinates(dev(x), dev(y), dev(z))
    sensor, Uq = orc.sensor(P, Q), orc.prim2c(P, Q)
    for d in range(3):
        S = orc.metric_norm(P, m[3 * d], m[3 * d + 1], m[3 * d + 2])
        want = orc.fvm_face_flux(P, d, scheme == abi.SCHEME_FVM_EIGEN, sensor, S, Q, Uq, x, y, z)
        F = torch.zeros((5, *orc.face_shape(P, d)), dtype=torch.float64, device="cuda")
        s.advect(d, F, dev(sensor), dev(Q))
        assert rel_linf(F.cpu().numpy(), want) <= 1e-12
    s.close()
