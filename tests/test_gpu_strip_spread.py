"""GPU: sums of the integer strips (f3d_fixed.cuh) whose own window holds none of the strip's large
values keep the accuracy of FP64 sums of their own terms. Steps and impulses of many orders of
magnitude at every offset from the strips' starts, in both directions along the line; each value
is held to a tolerance relative to what it reads."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
PER = [dict(kind=abi.BC_PERIODIC)] * 6
LINEAR = dict(phi1=5.0, phi2=6.0, phi3=7.0)  # above any sensor value: every face is linear


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _box(d, n, m=6):
    """Interior size (nx, ny, nz): n along direction d, m across."""
    return tuple(n if e == d else m for e in range(3))


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("step", [1e-6, 1e-12, 1e-20])
@pytest.mark.parametrize("offset", range(5))
def test_finite_volume_states_beside_a_step(gpu_lib, d, step, offset):
    """CD6 states (their outermost coefficients are zero) of a gas whose density and pressure fall by
    `step` and rise again: faces that read the small state alone have its flux."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    from oracle import oracle as orc
    n = _box(d, 72)
    P = abi.make_params(*n, viscous=0, linear_phi=0.0, scheme=abi.SCHEME_FVM_CONS, bc=PER, **LINEAR)
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    z, y, x = np.meshgrid(*[(np.arange(k) - 3.5) for k in shape], indexing="ij")
    i = np.broadcast_to(np.arange(shape[2 - d]).reshape([-1 if a == 2 - d else 1 for a in range(3)]), shape)
    small = ((i >= 12 + offset) & (i < 31 + offset)) | ((i >= 44 + offset) & (i < 57 + offset))
    r = np.random.default_rng(4)
    rho = np.where(small, step, 1.0) * r.uniform(0.99, 1.01, shape)
    Q = np.empty((6, *shape))
    Q[0], Q[1:4] = rho, np.array([0.3, -0.2, 0.4]).reshape(3, 1, 1, 1)
    Q[4] = 0.7 * rho
    Q[5] = Q[4] / (rho * P.rg)
    m, J = [np.full(shape, e) for e in (1., 0., 0., 0., 1., 0., 0., 0., 1.)], np.ones(shape)
    s = Flame3D(P)
    s.set_metrics([_dev(a) for a in m], _dev(J))
    s.set_coordinates(_dev(x), _dev(y), _dev(z))
    phi, U = np.zeros(shape), orc.prim2c(P, Q)
    want = orc.fvm_face_flux(P, d, False, phi, np.ones(shape), Q, U, x, y, z)
    F = torch.zeros((5, *orc.face_shape(P, d)), dtype=torch.float64, device="cuda")
    s.advect(d, F, _dev(phi), _dev(Q))
    s.close()
    got = np.moveaxis(F.cpu().numpy(), 3 - d, -1)
    want = np.moveaxis(want, 3 - d, -1)
    line = np.moveaxis(small, 2 - d, -1)[0, 0]
    faces = [t for t in range(want.shape[-1]) if line[t + 1:t + 7].all()]  # CD6 reads positions t+1 .. t+6
    assert len(faces) >= 18
    # an HLLC flux of states with relative error ~4 eps is within ~100 eps of its largest component
    scale = np.abs(want).max(0)
    for t in faces:
        assert (np.abs(got[..., t] - want[..., t]).max(0) <= 1e-13 * scale[..., t]).all(), t


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("towards", [1, -1])
@pytest.mark.parametrize("step", [1e-9, 1e-12, 1e-19])
def test_reverse_of_localised_cotangents(gpu_lib, d, towards, step):
    """Cotangents of a masked objective: they fall by `step` and rise again along one direction, at
    every offset from a strip's start. The gas is supersonic, so a cell hears from one side. UP7
    (integer strips) against a blend 2^-40 away from it, which has no small denominator and is summed in
    FP64: the two linear operators differ by 2^-40 of their coefficients."""
    from flame3d_mhd_gb300.solver import Flame3D
    for offset in range(5):
        n = _box(d, 72)
        shape = (n[2] + 8, n[1] + 8, n[0] + 8)
        r = np.random.default_rng(6)
        q = np.empty((6, *shape))
        q[0] = r.uniform(0.8, 1.2, shape)
        q[1:4] = r.uniform(-0.2, 0.2, (3, *shape))
        q[1 + d] += 3.0 * towards
        q[4] = q[0] * r.uniform(0.6, 0.8, shape)
        q[5] = q[4] / (q[0] * 287.0)
        i = np.arange(n[d])
        small = ((i >= 8 + offset) & (i < 27 + offset)) | ((i >= 40 + offset) & (i < 53 + offset))
        mag = np.where(small, step, 1.0).reshape([-1 if a == 2 - d else 1 for a in range(3)])
        Lbar = np.zeros((5, *shape))
        inner = (5, n[2], n[1], n[0])
        Lbar[:, 4:-4, 4:-4, 4:-4] = mag * r.uniform(0.5, 1.0, inner) * r.choice([-1.0, 1.0], inner)
        out = []
        for phi in (1.0, 1.0 - 2.0 ** -40):
            s = Flame3D(abi.make_params(*n, viscous=0, linear_phi=phi, bc=PER, **LINEAR))
            one, zero = np.ones(shape), np.zeros(shape)
            s.set_metrics([_dev(a) for a in (one, zero, zero, zero, one, zero, zero, zero, one)], _dev(one))
            U = s.field(5)
            Q = _dev(q)
            s.prim2c(U, Q)
            s.fillGhost(Q, U)
            out.append(s.rhs_vjp(U, _dev(Lbar)).cpu().numpy()[:, 4:-4, 4:-4, 4:-4])
            s.close()
        a, b = out
        # Fp of cell c enters the right-hand sides of c - 3 .. c + 4, Fm those of c - 4 .. c + 3
        hears = np.arange(-3, 5) if towards > 0 else np.arange(-4, 4)
        reach = np.array([mag.ravel()[(c + hears) % n[d]].max() for c in range(n[d])]).reshape(mag.shape)
        assert (reach == step).sum() >= 15
        scale = np.abs(b).max()
        # coefficients differ by 60/420 2^-40, the Jacobian's entries are below `scale` per unit of cotangent
        off = np.abs(a - b) / (scale * reach)
        assert off.max() <= 8 * 2.0 ** -40, (offset, float(off.max()))


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("towards", [1, -1])
@pytest.mark.parametrize("phi", [1.0, 0.5])
def test_linear_faces_beside_large_values(gpu_lib, d, towards, phi):
    """Face fluxes against sums in extended precision of the library's own split fluxes. A supersonic
    gas (one of Fp, Fm is zero) with, at every offset from a strip's start, four cells of density ~1, one
    2^-5 below and the rest ~2^-20: a face that reads the middle cell under its smallest coefficient
    has nothing else of that size."""
    from flame3d_mhd_gb300.solver import Flame3D
    n = _box(d, 64, 12)
    s = Flame3D(abi.make_params(*n, viscous=0, linear_phi=phi, bc=PER, **LINEAR))
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(9)
    rho = 2.0 ** -20 * r.uniform(1.0, 2.0, shape)
    line = np.moveaxis(rho, 2 - d, -1)  # a view: lines along the direction
    big = r.uniform(1.0, 1.9, line.shape)
    for a in range(line.shape[0]):
        for b in range(line.shape[1]):
            for c in range((3 * a + b) % 20, 72 - 8, 20):
                at = range(c, c + 5) if towards > 0 else range(c + 4, c - 1, -1)
                for k, p in enumerate(at):
                    line[a, b, p] = big[a, b, p] * (1.0 if k < 4 else 2.0 ** -5)
    q = np.zeros((6, *shape))
    q[0] = rho
    q[1 + d] = 3.0 * towards
    q[4] = rho / 1.4
    q[5] = q[4] / (rho * 287.0)
    one, zero = np.ones(shape), np.zeros(shape)
    s.set_metrics([_dev(a) for a in (one, zero, zero, zero, one, zero, zero, zero, one)], _dev(one))
    Fp, Fm, F = s.field(5), s.field(5), s.face_field(d)
    s.fluxSplit(d, _dev(q), Fp, Fm)
    s.advect(d, F, None, _dev(q))
    s.close()
    ax, cut = 3 - d, [slice(None)] + [slice(4, -4)] * 3
    cut[ax] = slice(None)
    p, m = (np.moveaxis(a.cpu().numpy()[tuple(cut)], ax, -1).astype(np.longdouble) for a in (Fp, Fm))
    nf = p.shape[-1] - 7
    lin = [(u * phi + c * (1 - phi)) / np.longdouble(420) for u, c in zip((-3, 25, -101, 319, 214, -38, 4), (0, 7, -56, 259, 259, -56, 7))]
    terms = [lin[k] * (p[..., k:k + nf] + m[..., 7 - k:7 - k + nf]) for k in range(7)]
    got = np.moveaxis(F.cpu().numpy(), ax, -1)
    # one of the pair is zero, so a sum has seven rounded products and coefficients: 7 + 7 + 2 roundings
    # of at most the sum of the terms' magnitudes
    off = np.abs(got - sum(terms)) / (EPS * sum(np.abs(t) for t in terms) + 1e-300)
    assert off.max() <= 16.0, float(off.max())


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("small", [1e-4, 1e-6, 1e-9, 1e-15, 1e-300])
@pytest.mark.parametrize("inner", [True, False])
def test_viscous_differences_of_values_that_cancel(gpu_lib, d, small, inner):
    """f[-2] = f[2] of size one (or f[-1] = f[1]) beside values of size `small`: the large ones cancel in the
    fourth-order difference, which keeps the accuracy of the small ones."""
    from flame3d_mhd_gb300.solver import Flame3D
    n = _box(d, 40, 5)
    c_s, t_s, T = 1e-2, 1.0, 0.7
    s = Flame3D(abi.make_params(*n, viscous=1, rg=1.0, c_s=c_s, t_s=t_s, bc=PER))
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(12)
    f = small * r.uniform(0.5, 1.0, 48) * r.choice([-1.0, 1.0], 48)
    centres = np.arange(6, 44, 5)
    for c in centres:
        k = 1 if inner else 2
        f[c - k] = f[c + k] = r.uniform(0.5, 1.0)
    q = np.zeros((6, *shape))
    q[0], q[5], q[4] = 1.0, T, T
    q[1 + d] = f.reshape([-1 if a == 2 - d else 1 for a in range(3)])
    one, zero = np.ones(shape), np.zeros(shape)
    s.set_metrics([_dev(a) for a in (one, zero, zero, zero, one, zero, zero, zero, one)], _dev(one))
    F = [s.viscous_field() for _ in range(3)]
    s.viscousFlux(*F, _dev(q))
    s.close()
    # only the normal gradient is there: the normal stress is 4/3 mu times it
    got = np.moveaxis(F[d].cpu().numpy()[d], 2 - d, -1)[..., centres - 2]
    v = f.astype(np.longdouble)
    diff = (v[centres - 2] - v[centres + 2]) - 8 * (v[centres - 1] - v[centres + 1])
    mu = np.longdouble(c_s) * np.longdouble(T) ** np.longdouble(1.5) / (np.longdouble(T) + t_s)
    want = mu * diff / 12 * np.longdouble(4) / 3
    # roundings: the difference 3, viscosity 5, stress and its factors 6
    assert (np.abs(got - want) <= 16 * EPS * np.abs(want)).all(), float((np.abs(got - want) / np.abs(want)).max() / EPS)


@pytest.mark.parametrize("d", [0, 1, 2])
@pytest.mark.parametrize("parity", [0, 1])
@pytest.mark.parametrize("phi", [0.5 + 1.6e-14, 0.9 - 1.6e-14, 1.0 - 1.6e-14, 1.6e-14, 0.3, 0.1 + 0.2])
def test_linear_faces_of_a_blend_near_a_small_denominator(gpu_lib, d, parity, phi):
    """A blend 1.6e-14 away from a quotient of small numbers is not that quotient: a supersonic gas whose
    density alternates from cell to cell, in which the two schemes' difference is largest."""
    from flame3d_mhd_gb300.solver import Flame3D
    n = _box(d, 64)
    s = Flame3D(abi.make_params(*n, viscous=0, linear_phi=phi, bc=PER, **LINEAR))
    shape = (n[2] + 8, n[1] + 8, n[0] + 8)
    r = np.random.default_rng(10)
    odd = (np.arange(shape[2 - d]) % 2 == parity).reshape([-1 if a == 2 - d else 1 for a in range(3)])
    q = np.zeros((6, *shape))
    q[0] = np.where(odd, 1.0, 2.0 ** -20) * r.uniform(1.0, 1.01, shape)
    q[1 + d] = 3.0
    q[4] = q[0] / 1.4
    q[5] = q[4] / (q[0] * 287.0)
    one, zero = np.ones(shape), np.zeros(shape)
    s.set_metrics([_dev(a) for a in (one, zero, zero, zero, one, zero, zero, zero, one)], _dev(one))
    Fp, Fm, F = s.field(5), s.field(5), s.face_field(d)
    s.fluxSplit(d, _dev(q), Fp, Fm)
    s.advect(d, F, None, _dev(q))
    s.close()
    ax, cut = 3 - d, [slice(None)] + [slice(4, -4)] * 3
    cut[ax] = slice(None)
    p, m = (np.moveaxis(a.cpu().numpy()[tuple(cut)], ax, -1).astype(np.longdouble) for a in (Fp, Fm))
    nf = p.shape[-1] - 7
    e = np.longdouble(phi)
    lin = [(u * e + c * (1 - e)) / np.longdouble(420) for u, c in zip((-3, 25, -101, 319, 214, -38, 4), (0, 7, -56, 259, 259, -56, 7))]
    terms = [lin[k] * (p[..., k:k + nf] + m[..., 7 - k:7 - k + nf]) for k in range(7)]
    got = np.moveaxis(F.cpu().numpy(), ax, -1)
    # as beside large values: 16 roundings of the terms
    off = np.abs(got - sum(terms)) / (EPS * sum(np.abs(t) for t in terms) + 1e-300)
    assert off.max() <= 16.0, float(off.max())
