"""GPU: right-hand sides, stages and reverse steps captured into a CUDA graph by the caller give on replay
what direct calls give, on grids below and above the size up to which launches overlap."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(16, 12, 8), (48, 40, 40)])
@pytest.mark.parametrize("viscous,character", [(0, 1), (1, 0)])
def test_calls_captured_by_the_caller(gpu_lib, n, viscous, character):
    import torch

    from flame3d_mhd_gb300 import cases
    from flame3d_mhd_gb300.cases import params_copy
    from flame3d_mhd_gb300.solver import Flame3D
    c = cases.sod(*n)
    P = params_copy(c["params"], viscous=viscous, character=character)
    s = Flame3D(P)
    m, J = s.compute_metrics(*[torch.from_numpy(np.ascontiguousarray(c[k])).cuda() for k in "xyz"])
    s.set_metrics(m, J)
    Q0 = torch.from_numpy(np.ascontiguousarray(c["Q"])).cuda()
    U0 = s.field(5)
    s.prim2c(U0, Q0)
    s.fillGhost(Q0, U0)
    g = torch.Generator(device="cuda").manual_seed(1)
    bar = s.field(5)
    bar[:, 4:-4, 4:-4, 4:-4] = 2.0 * torch.rand((5, n[2], n[1], n[0]), generator=g, dtype=torch.float64, device="cuda") - 1.0
    U, Un, Q, L, back = U0.clone(), torch.zeros_like(U0), Q0.clone(), s.field(5), s.field(5)

    def calls():
        U.copy_(U0)
        Q.copy_(Q0)
        s.rhs(Q, L)
        for stage in (1, 2, 3):
            s.rk3_stage(stage, c["dt"], U, Un, Q)
        s.rk3_step_vjp(c["dt"], U0, bar, back)

    calls()  # the first reverse call allocates
    torch.cuda.synchronize()
    want = [t.clone() for t in (L, U, Q, back)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for t in (L, U, Q, back):
        t.zero_()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip((L, U, Q), want):
        assert torch.equal(a, b)
    assert (back - want[3]).abs().max() <= 1e-11 * want[3].abs().max()  # additions across tiles in another order
    s.close()
