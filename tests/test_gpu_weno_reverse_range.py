"""GPU: the reverse of listed WENO faces (k_weno_vjp.cu) at the ends of what it takes, against the reverse
within the tiles (the same call with metric cotangents requested)."""
import numpy as np
import pytest

from flame3d_mhd_gb300 import abi

pytestmark = pytest.mark.gpu
FAR, TINY = 5.0, 1e-300
THRESHOLDS = {"weno7": (TINY, 4.5, FAR), "weno5": (TINY, 2 * TINY, FAR)}


def _solver(n, which, character, split="SW"):
    from flame3d_mhd_gb300.solver import Flame3D
    p1, p2, p3 = THRESHOLDS[which]
    return Flame3D(abi.make_params(*n, phi1=p1, phi2=p2, phi3=p3, viscous=0, character=character, split=split,
                                   bc=[dict(kind=abi.BC_PERIODIC)] * 6))


def _both(s, U, Lbar):
    """Ubar from the lists and from the tiles"""
    listed = s.rhs_vjp(U, Lbar).clone()
    bars = [s.field(1) for _ in range(10)]
    s.set_metrics_cotangent(bars[:9], bars[9])
    tiles = s.rhs_vjp(U, Lbar).clone()
    s.set_metrics_cotangent(None)
    return listed, tiles


def _case(s, n, size):
    import torch
    nx, ny, nz = n
    shape = (nz + 8, ny + 8, nx + 8)
    g = torch.Generator(device="cuda").manual_seed(3)
    uni = lambda *sh: torch.rand(sh, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    one, zero = torch.ones(shape, dtype=torch.float64, device="cuda"), torch.zeros(shape, dtype=torch.float64, device="cuda")
    s.set_metrics([one, zero, zero, zero, one, zero, zero, zero, one], one)
    Q = torch.empty((6, *shape), dtype=torch.float64, device="cuda")
    Q[0] = size * (0.7 + 0.6 * uni(*shape))
    Q[1:4] = 1.2 * uni(3, *shape) - 0.6
    Q[4] = size * (0.3 + 1.2 * uni(*shape)) ** 2
    Q[5] = Q[4] / (Q[0] * 287.0)
    U = s.field(5)
    s.prim2c(U, Q)
    s.fillGhost(Q, U)
    Lbar = s.field(5)
    Lbar[:, 4:-4, 4:-4, 4:-4] = 2.0 * uni(5, nz, ny, nx) - 1.0
    return U, Lbar


@pytest.mark.parametrize("which", sorted(THRESHOLDS))
@pytest.mark.parametrize("character", [0, 1])
@pytest.mark.parametrize("size", [1e-12, 1e20, 1e27])
def test_reverse_of_large_and_small_fluxes(gpu_lib, which, character, size):
    """Densities and pressures of 1e20 and 1e27: the squares of the weights' bases reach 1e84 and
    1e112, their products leave the FP64 range."""
    import torch
    s = _solver((33, 9, 6), which, character)
    U, Lbar = _case(s, (33, 9, 6), size)
    listed, tiles = _both(s, U, Lbar)
    s.close()
    assert torch.isfinite(tiles).all() and torch.isfinite(listed).all()
    # as for sizes of order one: both are sums of the same rounded products in another order
    for a, b in zip(listed, tiles):
        assert (a - b).abs().max() <= 1e-11 * b.abs().max()


@pytest.mark.parametrize("which", sorted(THRESHOLDS))
@pytest.mark.parametrize("component", [None, 1])
def test_no_cotangent_beside_non_finite_values(gpu_lib, which, component):
    """Component-wise faces whose cotangent is zero pass nothing on, also where the state is not finite."""
    import torch
    n = (40, 9, 6)
    s = _solver(n, which, 0)
    U, Lbar = _case(s, n, 1.0)
    U[1, 8, 8, 12] = U[2, 8, 9, 30] = 1e200  # pressures at their floor, so the faces stay WENO; fluxes overflow
    if component is None:
        Lbar[..., 4:28] = 0.0  # a masked objective: only the right part of the grid counts
    else:
        keep = Lbar[component].clone()
        Lbar.zero_()
        Lbar[component, ..., 28:44] = keep[..., 28:44]
    listed, tiles = _both(s, U, Lbar)
    s.close()
    fin = torch.isfinite(tiles)
    assert not fin.all() and fin[:, 4:-4, 4:-4, 4:-4].any()
    # (the lists' quotients hold where the tiles' products overflow: more of their values may be finite)
    assert torch.isfinite(listed[fin]).all()
    assert (listed[fin] - tiles[fin]).abs().max() <= 1e-11 * tiles[fin].abs().max()
