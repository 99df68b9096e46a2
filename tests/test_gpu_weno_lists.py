"""GPU: the FP64 right-hand side, whose WENO faces are listed and computed apart from the tiles
(k_weno.cu), against the differences of the face fluxes that f3d_debug_face_flux computes within
the tiles. Sizes around the 32-face chunks and the tiles; thresholds that give every branch, only
WENO7 faces (the list filled from its front to its end), only WENO5 faces (from its back), or none."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53
TINY, FAR = 1e-300, 5.0
THRESHOLDS = {"all": (0.05, 0.3, 0.6), "weno7": (TINY, 4.5, FAR), "weno5": (TINY, 2 * TINY, FAR), "none": (FAR - 1, FAR, FAR)}


@pytest.mark.parametrize("n", [(4, 4, 4), (33, 5, 9), (64, 65, 6), (70, 9, 31)])
@pytest.mark.parametrize("which", sorted(THRESHOLDS))
@pytest.mark.parametrize("character,split", [(1, "SW"), (0, "AUSM")])
def test_rhs_equals_differences_of_tile_faces(gpu_lib, n, which, character, split):
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    nx, ny, nz = n
    per = dict(kind=abi.BC_PERIODIC)
    p1, p2, p3 = THRESHOLDS[which]
    s = Flame3D(abi.make_params(nx, ny, nz, phi1=p1, phi2=p2, phi3=p3, viscous=0, character=character, split=split,
                                bc=[per] * 6))
    shape = (nz + 8, ny + 8, nx + 8)
    r = np.random.default_rng(11)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    eye = [1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0]
    s.set_metrics([dev(e + 0.1 * r.uniform(-1, 1, shape)) for e in eye], dev(np.ones(shape)))
    q = np.empty((6, *shape))
    q[0] = r.uniform(0.7, 1.3, shape)
    q[1:4] = r.uniform(-0.6, 0.6, (3, *shape))
    q[4] = r.uniform(0.3, 1.5, shape) ** 2
    q[5] = q[4] / (q[0] * 287.0)
    Q, phi = dev(q), s.field(1)
    s.shockSensor(phi, Q)
    want, scale = 0.0, 0.0
    for d in range(3):
        F = s.face_field(d)
        s.advect(d, F, phi, Q)
        f = np.moveaxis(F.cpu().numpy(), 3 - d, -1)
        want = want + np.moveaxis(f[..., :-1] - f[..., 1:], -1, 3 - d)
        scale = scale + np.moveaxis(np.abs(f[..., :-1]) + np.abs(f[..., 1:]), -1, 3 - d)
    I = (slice(None), *(slice(4, -4),) * 3)
    for _ in range(2):  # the second pass starts from the counts the first one cleared
        got = s.rhs(Q).cpu().numpy()[I]
        # the two paths form the same face fluxes in another order of rounding: an FP64 WENO flux of
        # this state is within ~1e3 eps of its exact value relative to the largest component
        tol = 2048 * EPS * scale.max(0)
        assert (np.abs(got - want).max(0) <= tol).all(), float((np.abs(got - want).max(0) / tol).max())
    s.close()


@pytest.mark.parametrize("n", [(4, 4, 4), (33, 5, 9), (70, 9, 31), (520, 130, 120)])
@pytest.mark.parametrize("which", ["all", "weno7", "weno5", "none"])
@pytest.mark.parametrize("character,split", [(1, "SW"), (0, "LF")])
def test_reverse_equals_the_tiles_reverse(gpu_lib, n, which, character, split):
    """The RHS VJP, whose WENO faces are reversed from their lists (k_weno_vjp.cu), against the same
    call with metric cotangents requested, which reverses them within the tiles. The largest grid is
    above the size up to which the three directions are taken at once."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    nx, ny, nz = n
    if nx > 500 and (which != "all" or not character):
        pytest.skip("one case of the largest grid is enough")
    per = dict(kind=abi.BC_PERIODIC)
    p1, p2, p3 = THRESHOLDS[which]
    s = Flame3D(abi.make_params(nx, ny, nz, phi1=p1, phi2=p2, phi3=p3, viscous=0, character=character, split=split,
                                bc=[per] * 6))
    shape = (nz + 8, ny + 8, nx + 8)
    g = torch.Generator(device="cuda").manual_seed(3)
    uni = lambda *sh: torch.rand(sh, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    eye = [1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0]
    # periodic inputs: the metrics are smooth functions of the cell indices
    z, y, x = torch.meshgrid(*[torch.arange(m, dtype=torch.float64, device="cuda") - 4 for m in shape], indexing="ij")
    w = [torch.sin(2 * np.pi * (x / nx + k * y / ny + z / nz)) for k in range(1, 10)]
    s.set_metrics([e + 0.1 * v for e, v in zip(eye, w)], torch.ones(shape, dtype=torch.float64, device="cuda"))
    Q = torch.empty((6, *shape), dtype=torch.float64, device="cuda")
    Q[0] = 0.7 + 0.6 * uni(*shape)
    Q[1:4] = 1.2 * uni(3, *shape) - 0.6
    Q[4] = (0.3 + 1.2 * uni(*shape)) ** 2
    Q[5] = Q[4] / (Q[0] * 287.0)
    U = s.field(5)
    s.prim2c(U, Q)
    s.fillGhost(Q, U)
    Lbar = s.field(5)
    Lbar[:, 4:-4, 4:-4, 4:-4] = 2.0 * uni(5, nz, ny, nx) - 1.0
    runs = [s.rhs_vjp(U, Lbar).clone() for _ in range(2)]  # the second finds the planes cleared
    bars = [s.field(1) for _ in range(10)]
    s.set_metrics_cotangent(bars[:9], bars[9])
    want = s.rhs_vjp(U, Lbar)
    # both are sums of the same ~1e4 rounded products in another order: the derivative of a WENO face
    # is formed with relative error ~1e3 eps of its largest terms, which are O(1/(1 - w)) of the result
    scale = want.abs().max()
    for got in runs:
        assert torch.isfinite(got).all()
        assert (got - want).abs().max() <= 1e-11 * scale, float((got - want).abs().max() / scale)
    s.close()


@pytest.mark.parametrize("n", [(4, 4, 4), (33, 5, 9), (65, 9, 63)])
@pytest.mark.parametrize("fixed,hybrid", [((5.0, 6.0, 7.0), (3.5, 6.0, 7.0)), ((0.0, 0.0, 0.0), (1e-30, 1e-30, 1e-30))])
@pytest.mark.parametrize("split", ["SW", "LF", "VL", "AUSM"])
def test_reverse_of_a_fixed_branch(gpu_lib, n, fixed, hybrid, split):
    """Every face linear or every face NND2, reversed by the tiles without WENO code (which split cells
    for NND2 faces alone), against the same faces under the hybrid switch with metric cotangents
    requested, whose tiles hold all branches and split every cell."""
    import torch

    from flame3d_mhd_gb300.solver import Flame3D
    nx, ny, nz = n
    per = dict(kind=abi.BC_PERIODIC)
    out = []
    for p in (fixed, hybrid):
        s = Flame3D(abi.make_params(nx, ny, nz, phi1=p[0], phi2=p[1], phi3=p[2], viscous=0, character=0, split=split,
                                    bc=[per] * 6))
        shape = (nz + 8, ny + 8, nx + 8)
        g = torch.Generator(device="cuda").manual_seed(3)
        uni = lambda *sh: torch.rand(sh, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
        eye = [1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0]
        # periodic inputs: the metrics are smooth functions of the cell indices
        z, y, x = torch.meshgrid(*[torch.arange(m, dtype=torch.float64, device="cuda") - 4 for m in shape], indexing="ij")
        w = [torch.sin(2 * np.pi * (x / nx + k * y / ny + z / nz)) for k in range(1, 10)]
        s.set_metrics([e + 0.1 * v for e, v in zip(eye, w)], torch.ones(shape, dtype=torch.float64, device="cuda"))
        Q = torch.empty((6, *shape), dtype=torch.float64, device="cuda")
        Q[0] = 0.7 + 0.6 * uni(*shape)
        Q[1:4] = 1.2 * uni(3, *shape) - 0.6
        Q[4] = (0.3 + 1.2 * uni(*shape)) ** 2
        Q[5] = Q[4] / (Q[0] * 287.0)
        U = s.field(5)
        s.prim2c(U, Q)
        s.fillGhost(Q, U)
        Lbar = s.field(5)
        Lbar[:, 4:-4, 4:-4, 4:-4] = 2.0 * uni(5, nz, ny, nx) - 1.0
        if p is hybrid:
            bars = [s.field(1) for _ in range(10)]
            s.set_metrics_cotangent(bars[:9], bars[9])
        out.append(s.rhs_vjp(U, Lbar).clone())
        s.close()
    # sums of the same ~100 rounded products a cell in another order
    assert torch.isfinite(out[0]).all()
    assert (out[0] - out[1]).abs().max() <= 1e-13 * out[1].abs().max()
