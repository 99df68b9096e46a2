"""GPU: WENO faces of a component that is many orders of magnitude smaller than the others, against the
oracle, each component relative to its own size."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu
FAR = 5.0


@pytest.mark.parametrize("size", [1e-3, 1e-30, 1e-60, 1e-75, 1e-90, 1e-150])
@pytest.mark.parametrize("phi", [(0.0, FAR, FAR + 1), (0.0, 0.0, FAR)], ids=["weno7", "weno5"])
@pytest.mark.parametrize("d", [0, 1, 2])
def test_small_transverse_momentum(gpu_lib, size, phi, d):
    """A velocity component of `size` beside others of order one: its momentum flux has smoothness
    indicators far below the weights' floor, so its faces are the scheme's linear ones."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    n = [10, 10, 10]
    n[d] = 40
    P = abi.make_params(*n, viscous=0, character=0, phi1=phi[0], phi2=phi[1], phi3=phi[2],
                        bc=[dict(kind=abi.BC_PERIODIC)] * 6)
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(6)
    other = (d + 1) % 3
    q = np.empty((6, *shape))
    q[0] = r.uniform(0.9, 1.1, shape)
    q[1:4] = r.uniform(0.2, 0.3, (3, *shape))
    q[1 + other] = size * r.uniform(0.5, 1.0, shape)
    q[4] = r.uniform(0.9, 1.1, shape) / 1.4
    q[5] = q[4] / (q[0] * 287.0)
    m = [np.full(shape, e) for e in (1., 0., 0., 0., 1., 0., 0., 0., 1.)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = Flame3D(P)
    s.set_metrics([dev(a) for a in m], dev(np.ones(shape)))
    Fp, Fm, F = s.field(5), s.field(5), s.face_field(d)
    s.fluxSplit(d, dev(q), Fp, Fm)
    s.advect(d, F, None, dev(q))
    s.close()
    k = 1 + other
    ax, cut = 2 - d, [slice(4, -4)] * 3
    cut[ax] = slice(None)
    p, q_ = (np.moveaxis(a.cpu().numpy()[k][tuple(cut)], ax, -1) for a in (Fp, Fm))
    got = np.moveaxis(F.cpu().numpy()[k], ax, -1)
    nf = got.shape[-1]
    P_ = lambda i: p[..., i:i + nf]  # noqa: E731
    M_ = lambda i: q_[..., i:i + nf]  # noqa: E731
    # the reference's weights at vanishing indicators: (1, 12, 18, 4) / 35 and (1, 6, 3) / 10
    if phi[1] == FAR:
        c = np.array([[-3, 13, -23, 25, 0, 0, 0], [0, 1, -5, 13, 3, 0, 0], [0, 0, -1, 7, 7, -1, 0], [0, 0, 0, 3, 13, -5, 1]])
        c, first, last = (np.array([1, 12, 18, 4]) @ c) / (35 * 12), 0, 7
    else:
        c = np.array([[2, -7, 11, 0, 0], [0, -1, 5, 2, 0], [0, 0, 2, 5, -1]])
        c, first, last = (np.array([1, 6, 3]) @ c) / (10 * 6), 1, 6
    terms = [c[i] * P_(first + i) for i in range(len(c))] + [c[i] * M_(last - i) for i in range(len(c))]
    if size < 1e-20:  # indicators below 1e-36, their floor 1e-20 (1e-16)
        assert (np.abs(got - sum(terms)) <= 1e-13 * sum(np.abs(t) for t in terms)).all()
    host = lambda t: np.ascontiguousarray(t.cpu().numpy())  # noqa: E731
    want = orc.face_flux(P, d, np.zeros(shape), np.ones(shape), host(Fp), host(Fm), q, *m[3 * d:3 * d + 3])[k]
    want = np.moveaxis(want, ax, -1)
    # weights of indicators that the two sides form in other orders, from the same split fluxes
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
