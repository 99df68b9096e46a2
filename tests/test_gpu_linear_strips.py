"""GPU: the linear (UP7 / CD6 blend) face fluxes of the FP64 sweeps, summed as integers in strips
of five faces (f3d_fixed.cuh), against sums in extended precision of the library's own split
fluxes. Sizes around the edges of strips and tiles; a density that jumps by up to 1e12 between
neighbouring blocks, so that strips with a wide spread of magnitudes (summed in FP64) sit beside
integer ones; blends with and without a small common denominator."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu

UP7 = np.array([-3, 25, -101, 319, 214, -38, 4], dtype=np.longdouble) / 420
CD6 = np.array([0, 1, -8, 37, 37, -8, 1], dtype=np.longdouble) / 60
EPS = 2.0 ** -53


def state(shape, wide, seed):
    r = np.random.default_rng(seed)
    q = np.empty((6, *shape))
    blocks = 10.0 ** r.uniform(-6.0, 6.0, size=[-(-n // 9) for n in shape]) if wide else np.ones([-(-n // 9) for n in shape])
    scale = blocks.repeat(9, 0).repeat(9, 1).repeat(9, 2)[:shape[0], :shape[1], :shape[2]]
    q[0] = scale * r.uniform(0.8, 1.2, shape)
    q[1:4] = r.uniform(-0.7, 0.7, (3, *shape))
    q[4] = q[0] * r.uniform(0.6, 0.8, shape)
    q[5] = q[4] / (q[0] * 287.0)
    return q


@pytest.mark.parametrize("n", [(4, 5, 6), (9, 63, 64), (65, 66, 7), (64, 8, 69), (130, 17, 9)])
@pytest.mark.parametrize("phi,wide", [(1.0, False), (1.0, True), (0.0, True), (0.5, True), (0.9, True), (0.1234567, True)])
def test_linear_faces(gpu_lib, n, phi, wide):
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    nx, ny, nz = n
    per = dict(kind=abi.BC_PERIODIC)
    # phi1 above any sensor value: every face is linear
    P = abi.make_params(nx, ny, nz, phi1=5.0, phi2=6.0, phi3=7.0, linear_phi=phi, viscous=0, bc=[per] * 6)
    s = Flame3D(P)
    shape = (nz + 8, ny + 8, nx + 8)
    r = np.random.default_rng(5)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    eye = [1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0]
    s.set_metrics([dev(e + 0.1 * r.uniform(-1, 1, shape)) for e in eye], dev(np.ones(shape)))
    Q = dev(state(shape, wide, 7))
    lin = UP7 * np.longdouble(phi) + CD6 * (1 - np.longdouble(phi))
    for d in range(3):
        Fp, Fm, F = s.field(5), s.field(5), s.face_field(d)
        s.fluxSplit(d, Q, Fp, Fm)
        s.advect(d, F, None, Q)
        ax = 3 - d  # numpy axis of direction d
        cut = [slice(None)] + [slice(4, -4)] * 3
        cut[ax] = slice(None)
        p, m = (np.moveaxis(a.cpu().numpy()[tuple(cut)], ax, -1) for a in (Fp, Fm))
        nf = p.shape[-1] - 7
        want = sum(lin[k] * (p[..., k:k + nf].astype(np.longdouble) + m[..., 7 - k:7 - k + nf].astype(np.longdouble))
                   for k in range(7))
        got = np.moveaxis(F.cpu().numpy(), ax, -1)
        # any FP64 sum of the 14 products is within 15 eps sum |lin| |F|; the split of the sweep may
        # round differently from the one read here by a few eps of its terms, which are of the
        # size of the largest component (velocities, sound speed and metrics of order one)
        big = np.maximum(np.abs(p), np.abs(m)).max(0)
        win = np.max([big[..., k:k + nf] for k in range(8)], axis=0)
        tol = 64 * EPS * float(2 * np.abs(lin).sum()) * win
        assert np.isfinite(got).all()
        assert (np.abs(got - want).max(0) <= tol).all(), float((np.abs(got - want).max(0) / tol).max())
    s.close()


def test_nonfinite_values_reach_the_faces(gpu_lib):
    """A NaN and an infinity in the state make exactly the faces non-finite whose stencils read
    them, as sums in FP64 do."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    per = dict(kind=abi.BC_PERIODIC)
    P = abi.make_params(40, 8, 8, phi1=5.0, phi2=6.0, phi3=7.0, viscous=0, bc=[per] * 6)
    s = Flame3D(P)
    shape = (16, 16, 48)
    one, zero = torch.ones(shape, dtype=torch.float64).cuda(), torch.zeros(shape, dtype=torch.float64).cuda()
    s.set_metrics([one, zero, zero, zero, one, zero, zero, zero, one], one)
    q = state(shape, False, 3)
    q[1, 6, 6, 20] = np.nan   # u
    q[0, 9, 9, 31] = np.inf   # rho
    Q = torch.from_numpy(q).cuda()
    Fp, Fm, F = s.field(5), s.field(5), s.face_field(0)
    s.fluxSplit(0, Q, Fp, Fm)
    s.advect(0, F, None, Q)
    # the split puts such a cell's flux on one side: face t reads Fp at t .. t+6, Fm at t+1 .. t+7
    p, m = (~np.isfinite(a.cpu().numpy()[:, 4:-4, 4:-4]) for a in (Fp, Fm))
    assert p.any() or m.any()
    want = np.any([p[..., k:k + 41] | m[..., 7 - k:48 - k] for k in range(7)], axis=0)
    assert (~np.isfinite(F.cpu().numpy()) == want).all()
    s.close()


def test_zero_components_stay_zero(gpu_lib):
    """A component without momentum or pressure term has a flux of exactly zero."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    per = dict(kind=abi.BC_PERIODIC)
    P = abi.make_params(40, 8, 8, phi1=5.0, phi2=6.0, phi3=7.0, viscous=0, bc=[per] * 6)
    s = Flame3D(P)
    shape = (16, 16, 48)
    one, zero = torch.ones(shape, dtype=torch.float64).cuda(), torch.zeros(shape, dtype=torch.float64).cuda()
    s.set_metrics([one, zero, zero, zero, one, zero, zero, zero, one], one)
    q = state(shape, False, 3)
    q[3] = 0.0
    F = s.face_field(0)
    s.advect(0, F, None, torch.from_numpy(q).cuda())
    f = F.cpu().numpy()
    assert (f[3] == 0.0).all() and (f[[0, 1, 2, 4]] != 0.0).all()
    s.close()
