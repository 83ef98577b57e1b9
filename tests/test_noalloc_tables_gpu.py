"""ugks_step_explicit_noalloc and a context take the same kernels for a velocity table, whatever the table."""
import ctypes

import numpy as np
import pytest

from test_tensor_tables import cases, rectangle
from ugks2d_high_order_b200.case import reference_case

pytestmark = pytest.mark.gpu


def both(t, nx=3, ny=4, nsteps=2):
    """(h, b, W, dt) after nsteps by a context and by the allocation-free entry point."""
    import torch
    from ugks2d_high_order_b200 import capi
    from ugks2d_high_order_b200.solver import Solver
    u, v, w = (np.ascontiguousarray(a) for a in t)
    c = reference_case("Explicit").with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny, wall_ux=(-0.5, 0.7))
    rng = np.random.default_rng(3)
    h = (1 + 0.05 * rng.uniform(-1, 1, (ny, nx, 1))) / (2 * np.pi) * np.exp(-(u ** 2 + v ** 2) / 2) * (1 + 0.05 * rng.uniform(-1, 1, (ny, nx, len(u))))
    W = np.stack([h @ w, h @ (w * u), h @ (w * v), 0.5 * (h @ (w * (u * u + v * v)) + h @ w)], -1)
    s = Solver(c, u, v, w)
    try:
        s.upload(h, h, W)
        dt, _ = s.step_explicit(nsteps)
        want = s.download() + (dt,)
        g = [torch.from_numpy(a.copy()).cuda() for a in (u, v, w, h, h, W)]
        d = np.zeros(1)
        rc = capi.load().ugks_step_explicit_noalloc(ctypes.byref(s._params), *(ctypes.c_void_p(a.data_ptr()) for a in g), nsteps,
                                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                                    d.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), None)
        assert rc == capi.UGKS_OK
        return tuple(a.cpu().numpy() for a in g[3:]) + (d[0],), want
    finally:
        s.close()


def same(t):
    """The same kernels on the same numbers: the same bits."""
    return all(np.array_equal(np.asarray(a).reshape(-1), np.asarray(b).reshape(-1)) for a, b in zip(*both(t)))


# (those whose weights are no quadrature weights are for the rule alone)
@pytest.mark.parametrize("name,table", [(n, t) for n, t, _ in cases() if n not in ("one weight zero", "one weight negative", "one weight nan",
                                                                                   "one row", "one column")])
def test_tables(name, table):
    """Tensor products, square, rectangular and above 1024 velocities, and tables that miss the rule by one of its conditions."""
    assert same(table)


def test_tables_at_the_limit_of_the_rule():
    """One weight moved by five units in the last place, the rule's limit with the factors' own rounding."""
    u, v, w = rectangle(16, 16)
    for seed in range(40):
        rng = np.random.default_rng(seed)
        x, y = rng.uniform(0.8, 1.25, (2, 16))
        z = w * np.tile(x, 16) * np.repeat(y, 16)
        z = np.tile(z[:16], 16) * np.repeat(z[::16] / z[0], 16)
        k = rng.integers(len(z))
        for _ in range(5):
            z[k] = np.nextafter(z[k], 9e9)
        assert same((u, v, z)), seed
