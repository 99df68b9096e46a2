"""GPU: a context's first calls on a stream of PyTorch's pool, which does not wait for the legacy
stream, give what they give on the default stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(32, 16, 16), (96, 64, 48)])
def test_first_reverse_call_on_a_side_stream(gpu_lib, n):
    import torch

    from flame3d_mhd_gb300 import cases
    from flame3d_mhd_gb300.solver import Flame3D, side_stream
    c = cases.sod(*n)
    xyz = [torch.from_numpy(np.ascontiguousarray(c[k])).cuda() for k in "xyz"]
    Q0 = torch.from_numpy(np.ascontiguousarray(c["Q"])).cuda()
    first = Flame3D(c["params"])
    m, J = first.compute_metrics(*xyz)
    U = first.field(5)
    first.prim2c(U, Q0)
    first.fillGhost(Q0, U)
    g = torch.Generator(device="cuda").manual_seed(2)
    bar = first.field(5)
    bar[:, 4:-4, 4:-4, 4:-4] = 2.0 * torch.rand((5, n[2], n[1], n[0]), generator=g, dtype=torch.float64, device="cuda") - 1.0
    first.set_metrics(m, J)
    want = first.rk3_step_vjp(c["dt"], U, bar)
    L = first.rhs(Q0)
    first.close()
    s = Flame3D(c["params"])
    with side_stream():
        s.set_metrics(m, J)
        got_L = s.rhs(Q0)
        got = s.rk3_step_vjp(c["dt"], U, bar)
    torch.cuda.synchronize()
    s.close()
    assert torch.equal(got_L, L)
    # the same sums, with additions across tiles in another order (tests of the lists: 1e-11)
    assert (got - want).abs().max() <= 1e-11 * want.abs().max()
