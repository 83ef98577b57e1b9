"""The S2 closures' gates on a tensor-product velocity table: what the general kernels refuse is refused there."""
import numpy as np
import pytest

from test_tensor_tables import rectangle
from ugks2d_high_order_b200.case import reference_case


# The Shakhov directions' moments have to vanish to 2e-12 as they stand.  Their energy carries the rounding of half the mean's
# square times the direction: 1e-15 at rest, 1e-10 and more at 3000.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 16), (28, 34), (50, 50)])
@pytest.mark.parametrize("mean,refused", [(0.0, [0, 0]), (3000.0, [444, 444]), (10000.0, [444, 444])])
def test_moments_of_the_directions(shape, mean, refused):
    """The targets and the evolution of a gas at a mean velocity far above its thermal width, on a table moved with it and
    on the same table in another order, which takes the general kernels."""
    from test_explicit_tensor_range import codes
    from ugks2d_high_order_b200.solver import Solver
    (u, v, w), (nx, ny) = rectangle(*shape), (4, 9)
    t = (u + mean, v, w)
    c = reference_case("S2CN2").with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny, wall_ux=(mean, mean), wall_tnative=(2.0, 2.0))
    h = np.broadcast_to(np.exp(-(u ** 2 + v ** 2) / 2) / (2 * np.pi), (ny, nx, len(u))).copy()
    W = np.stack([h @ w, h @ (w * t[0]), h @ (w * v), 0.5 * (h @ (w * (t[0] ** 2 + v ** 2)) + h @ w)], -1)
    for p in (np.random.default_rng(1).permutation(len(u)), np.arange(len(u))):
        s = Solver(c, *(np.ascontiguousarray(a[p]) for a in t))
        try:
            s.upload(h[..., p], h[..., p], W)
            assert codes(s, lambda s: s.s2cn2_init(), lambda s: s.evolution_s2(True)) == refused
        finally:
            s.close()
