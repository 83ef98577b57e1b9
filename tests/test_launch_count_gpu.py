"""ugks_launch_count against the launches that the profiler sees."""
import numpy as np
import pytest

from test_tensor_tables import rectangle
from ugks2d_high_order_b200.case import reference_case


def launches(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return sum("ugks" in n or n.startswith("k_") for n in names)


# 5 and 6 rows: every cell is next to a wall; 7 and more: the inner cells have a kernel of their own; above 16 columns the
# first layer's transpose has another form
@pytest.mark.gpu
@pytest.mark.parametrize("tensor", [True, False])
@pytest.mark.parametrize("nx,ny", [(5, 5), (5, 6), (5, 7), (8, 12), (18, 7)])
def test_adjoint_launches(nx, ny, tensor):
    from ugks2d_high_order_b200.solver import Solver
    t = rectangle(12, 12)
    if not tensor:
        p = np.random.default_rng(1).permutation(len(t[0]))
        t = tuple(np.ascontiguousarray(a[p]) for a in t)
    s = Solver(reference_case("S2CN2").with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny), *t)
    try:
        s.init_freestream()
        seed = np.ones(4)
        s.s2cn2_step_vjp(seed=seed)
        n = s.launch_count
        seen = launches(lambda: s.s2cn2_step_vjp(seed=seed))
        assert seen > 0 and s.launch_count - n == seen
        s.s2cn2_forward_checkpointed(3, 2)
        n = s.launch_count
        seen = launches(lambda: s.s2cn2_backward(seed))
        assert s.launch_count - n == seen
    finally:
        s.close()
