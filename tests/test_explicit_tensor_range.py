"""Explicit steps on a tensor-product velocity table against the same table in another order, which takes the general kernels,
outside the reference's units: dense and cold states, where the projections' weight floors pass 1e-16, densities at which
the product of the slopes' four denominators overflows, and states that the projections' gates refuse."""
import numpy as np
import pytest

from test_tensor_tables import EXPLICIT_TOL, rectangle
from ugks2d_high_order_b200.case import reference_case


def state(t, nx, ny, rho, T, seed=7, noise=0.05):
    """A state of density rho and temperature T with a twentieth of variation from cell to cell and velocity to velocity."""
    rng = np.random.default_rng(seed)
    r, U, V = 1 + noise * rng.uniform(-1, 1, (ny, nx, 1)), *(0.1 * np.sqrt(T) * rng.uniform(-1, 1, (2, ny, nx, 1)))
    tc = T * (1 + noise * rng.uniform(-1, 1, (ny, nx, 1)))
    h = rho * r / (np.pi * tc) * np.exp(-((t[0] - U) ** 2 + (t[1] - V) ** 2) / tc)
    h = h * (1 + noise * rng.uniform(-1, 1, h.shape))
    b = 0.5 * tc * h
    return h, b, np.stack([h @ t[2], h @ (t[2] * t[0]), h @ (t[2] * t[1]), 0.5 * (h @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + b @ t[2])], -1)


def case(nx, ny, rho=1.0, T=2.0):
    """Walls at the state's temperature; the viscosity grows with the density, so that the relaxation time keeps its size."""
    c = reference_case("Explicit")
    return c.with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny, mu_ref=c.mu_ref * rho, wall_ux=(-0.5, 0.7), wall_tnative=(0.9 * T, 1.05 * T))


def both(c, t, run, h, b, W):
    """run(solver) on the table (tensor kernels) and on the table in another order (general kernels), the arrays of the
    distribution in the first order."""
    from ugks2d_high_order_b200.solver import Solver
    p = np.random.default_rng(1).permutation(len(t[0]))
    out = []
    for q in (np.arange(len(p)), p):
        s = Solver(c, *(np.ascontiguousarray(a[q]) for a in t))
        try:
            s.upload(h[..., q], b[..., q], W)
            got = run(s)
        finally:
            s.close()
        back = np.argsort(q)
        out.append([a[..., back] if isinstance(a, np.ndarray) and a.shape[-1:] == (len(q),) else a for a in got])
    return out


def close(a, b, tol=EXPLICIT_TOL):
    for x, y in zip(a, b):
        x, y = np.asarray(x).reshape(-1), np.asarray(y).reshape(-1)
        assert np.isfinite(y).all() and np.abs(x - y).max() <= tol * np.abs(y).max()


# Tolerance: EXPLICIT_TOL, whose reasons hold in any units: relative roundings of the largest value, 3 steps.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 16), (20, 28), (50, 50)])
@pytest.mark.parametrize("rho,T", [(10.0, 0.5), (1e4, 2.0)])
def test_dense_states(shape, rho, T):
    """max |h| above 1: the equilibria's and the stream's floors are eps times the maximum."""
    from oracle.oracle import Oracle
    t, (nx, ny) = rectangle(*shape, scale=2.0 * np.sqrt(T / 2)), (4, 5)
    c, s0 = case(nx, ny, rho, T), state(t, nx, ny, rho, T)
    assert s0[0].max() > 1

    def run(s):
        s.step_explicit(3)
        return s.download() + (s.wall_aero(),)

    got, want = both(c, t, run, *s0)
    close(got, want)
    o = Oracle(c, *t)
    o.set_state(*s0)
    for _ in range(3):
        o.explicit_step()
    close(got, o.get_state())


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(32, 32), (50, 50)])
def test_stream_floor(shape):
    """The stream projection's weights.  At the velocities far from the mean of an almost uniform gas the fluxes cancel and the
    residual is the projection's: the floor, eps max(1, max |h|), times a polynomial whose coefficients are the rounding
    errors of the moments.  So the two paths' residuals there agree in size, not in value: over all inner cells the medians
    agree to a factor of 30 (they have one origin), where a floor of eps alone is 9e5 smaller."""
    rho, (nx, ny), t = 6e6, (6, 8), rectangle(*shape)
    # no wall forcing, and few collisions: the face equilibria have floors of their own
    c = case(nx, ny, rho).with_(wall_ux=(0.0, 0.0), wall_tnative=(2.0, 2.0), mu_ref=rho * 100)
    h = np.repeat(np.repeat(rho / (2 * np.pi) * np.exp(-(t[0] ** 2 + t[1] ** 2) / 2)[None, None], ny, 0), nx, 1)
    mid = np.argsort(h[0, 0])[-8:]
    h[..., mid] *= 1 + 1e-8 * np.random.default_rng(3).uniform(-1, 1, (ny, nx, 8))
    b = h.copy()
    W = np.stack([h @ t[2], h @ (t[2] * t[0]), h @ (t[2] * t[1]), 0.5 * (h @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + b @ t[2])], -1)

    def run(s):
        s.time_step(), s.evolution(), s.compute_residual()
        return (s.array("res_h", (ny, nx, len(t[0]))),)

    got, want = both(c, t, run, h, b, W)
    far = h[0, 0] < 1e-33 * h.max()
    assert h.max() > 5e5 and far.sum() > 8
    g, w = (np.median(np.abs(a[0][2:-2, :, far])) for a in (got, want))
    assert w > 0 and 1 / 30 < g / w < 30


# Tolerance: EXPLICIT_TOL, relative roundings of the largest value as in any units.  One step: its slopes are the ones at stake.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 4), (16, 16), (50, 50)])
@pytest.mark.parametrize("rho", [1e76, 1e80, 1e140])
def test_slopes_of_large_values(shape, rho):
    t, (nx, ny) = rectangle(*shape), (4, 5)

    def run(s):
        s.step_explicit(1)
        return s.download() + (s.wall_aero(),)

    close(*both(case(nx, ny, rho), t, run, *state(t, nx, ny, rho, 2.0)))


def codes(s, *steps):
    """The reference's abort code of each operator, 0 for none."""
    from ugks2d_high_order_b200.capi import UgksError
    out = []
    for f in steps:
        try:
            f(s)
            out.append(0)
        except UgksError as e:
            out.append(e.reference_code)
    return out


OPERATORS = [lambda s: s.time_step(), lambda s: s.evolution(), lambda s: s.compute_residual(), lambda s: s.apply_explicit_update()]


# The smallest pivot of the equilibrium's Gram matrix falls as the mean's fourth power: 1e-11 of its largest entry at 100
# and 1e-17 at 1000, on either side of the rule's 2.2e-13.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 16), (50, 50)])
@pytest.mark.parametrize("mean,refused", [(100.0, [0, 0, 0, 0]), (1000.0, [0, 446, 444, 444])])
def test_pivots_of_a_fast_mean(shape, mean, refused):
    """A gas whose mean velocity is far above its thermal width, on a table moved with it."""
    (u, v, w), (nx, ny) = rectangle(*shape), (3, 4)
    t = (u + mean, v, w)
    c = case(nx, ny).with_(wall_ux=(mean, mean), wall_tnative=(2.0, 2.0))
    h = np.broadcast_to(np.exp(-(u ** 2 + v ** 2) / 2) / (2 * np.pi), (ny, nx, len(u))).copy()
    W = np.stack([h @ w, h @ (w * t[0]), h @ (w * v), 0.5 * (h @ (w * (t[0] ** 2 + v ** 2)) + h @ w)], -1)
    got, want = both(c, t, lambda s: codes(s, *OPERATORS), h, h, W)
    assert want == refused and got == refused


# A distribution whose density, momentum and energy are the state's and whose heat flux is A: its Shakhov equilibria are of
# size 0.02 A, and their moments, which the projection's gate takes from W to 1e-10, carry rounding errors of 1e-16 of that and
# more: far below the gate at A = 1, above it at 1e10.
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 16), (50, 50)])
@pytest.mark.parametrize("A,refused", [(1.0, [0]), (1e10, [444])])
def test_moments_of_the_projected_equilibria(shape, A, refused):
    t, (nx, ny) = rectangle(*shape), (3, 4)
    M = np.exp(-(t[0] ** 2 + t[1] ** 2) / 2) / (2 * np.pi)
    psi = np.stack([np.ones_like(t[0]), t[0], t[1], 0.5 * (t[0] ** 2 + t[1] ** 2)])
    g = t[0] * (t[0] ** 2 + t[1] ** 2 - 4)
    g = g - psi.T @ np.linalg.solve((psi * (t[2] * M)) @ psi.T, psi @ (t[2] * M * g))
    full = lambda a: np.broadcast_to(a, (ny, nx, len(M))).copy()
    W = np.broadcast_to([M @ t[2], 0.0, 0.0, 0.5 * (M @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + M @ t[2])], (ny, nx, 4)).copy()
    c = case(nx, ny).with_(wall_ux=(0.0, 0.0), wall_tnative=(2.0, 2.0))

    from ugks2d_high_order_b200.solver import Solver
    order = np.random.default_rng(1).permutation(len(M))
    for q in (np.arange(len(M)), order):
        s = Solver(c, *(np.ascontiguousarray(a[q]) for a in t))
        try:
            s.upload(full(M[q]), full(M[q]), W)
            assert codes(s, *OPERATORS[:3]) == [0, 0, 0]   # the Maxwellian: no residual
            s.upload(full((M * (1 + A * g))[q]), full(M[q]), W)
            assert codes(s, OPERATORS[3]) == refused
        finally:
            s.close()
