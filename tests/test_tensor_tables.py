"""tensor_table (csrc/ugks_lo.cuh): which velocity tables take the 1-D sums of the S2 closures."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from ugks2d_high_order_b200.build import CSRC, NVCC, ROOT
from ugks2d_high_order_b200.case import velocity_table
from ugks2d_high_order_b200.velocity import raw_rule

MAIN = r"""
#include <cstdio>
#include <vector>
#include "ugks_lo.cuh"
int main() {
    int n;
    while (std::scanf("%d", &n) == 1) {
        std::vector<double> t(3 * (size_t)n);
        for (double& x : t) if (std::scanf("%la", &x) != 1) return 1;
        double tab[ugks::kTensorTab];
        int nu = 0, nv = 0;
        const bool ok = ugks::tensor_table(n, t.data(), t.data() + n, t.data() + 2 * n, &nu, &nv, tab);
        std::printf("%d %d %d", ok, nu, nv);
        for (int a = 0; ok && a < ugks::kTensorTab; ++a) std::printf(" %a", tab[a]);
        std::printf("\n");
    }
}
"""


def rectangle(nu, nv, scale=2.0):
    """The tensor product of two half-range rules of nu and nv abscissae, as fill_velocity maps them."""
    (x, a), (y, b) = (raw_rule(n // 2) for n in (nu, nv))
    ax, ay = (scale * np.sqrt(2.0) * np.exp(q * q) * c for q, c in ((x, a), (y, b)))
    s = scale * np.sqrt(2.0)
    return np.tile(s * x, nv), np.repeat(s * y, nu), np.tile(ax, nv) * np.repeat(ay, nu)


def cases():
    for n in (16, 24, 32, 48, 50):
        yield f"{n}^2", velocity_table(n), (n, n)
    yield "20x28", rectangle(20, 28), (20, 28)
    yield "64x36", rectangle(64, 36), (64, 36)
    u, v, w = rectangle(8, 12)
    yield "second axis fastest", (v, u, w), None
    p = np.random.default_rng(1).permutation(len(u))
    yield "shuffled", (u[p], v[p], w[p]), None
    for name, f in (("one weight off", 1 + 1e-14), ("one weight zero", 0.0), ("one weight negative", -1.0), ("one weight nan", np.nan)):
        z = w.copy()
        z[37] *= f
        yield name, (u, v, z), None
    z = u.copy()
    z[41] = np.nextafter(z[41], 9)
    yield "one abscissa off", (z, v, w), None
    yield "eight digits", (u, v, np.round(w, 8)), None
    yield "one row", (u[:8], v[:8], w[:8]), None
    yield "one column", (u[::8], v[::8], w[::8]), None
    yield "not a multiple", (u[:-1], v[:-1], w[:-1]), None
    yield "66 abscissae", rectangle(66, 4), None


def test_tensor_table(tmp_path):
    if shutil.which(NVCC) is None:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(MAIN)
    subprocess.run([NVCC, "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"), "-o", str(exe), str(src)], check=True)
    every = list(cases())
    text = "".join(f"{len(t[0])}\n" + " ".join(float(x).hex() for a in t for x in a) + "\n" for _, t, _ in every)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    for (name, (u, v, w), shape), line in zip(every, out):
        f = line.split()
        assert (f[0] == "1") == (shape is not None), name
        if shape is None:
            continue
        nu, nv = shape
        assert (int(f[1]), int(f[2])) == shape, name
        tab = np.array([float.fromhex(x) for x in f[3:]]).reshape(8, 64)
        assert np.array_equal(np.tile(tab[0, :nu], nv), u) and np.array_equal(np.repeat(tab[2, :nv], nu), v), name
        wk = np.tile(tab[1, :nu], nv) * np.repeat(tab[3, :nv], nu)
        assert np.abs(wk / w - 1).max() <= 4 * np.finfo(float).eps, name
        assert not tab[1, nu:].any() and not tab[3, nv:].any(), name


# Tolerance: both paths accept a closure at a scaled moment residual of 5e-13; its Jacobian is of order one in
# the units of these states, so their Maxwellians may differ by about that, once per node state and step: 3 steps
# with at most 2 uses each give 3e-12 of the largest value, 1e-11 with a margin of three.
TOL = 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 16), (24, 24), (20, 28), (28, 34), (64, 36), (50, 50)])
def test_tensor_path_matches_oracle_and_general_path(shape):
    """S2CN2 on a tensor table against the oracle, and against the same table in another order, which takes the
    general kernels."""
    from oracle.oracle import Oracle
    from ugks2d_high_order_b200.case import reference_case
    from ugks2d_high_order_b200.solver import Solver
    t = rectangle(*shape)
    c = reference_case("S2CN2").with_(nx=5, ny=9, dx=0.2, dy=1 / 9, wall_ux=(-2.0, 3.0), wall_tnative=(1.8, 2.1))
    rng = np.random.default_rng(5)
    W = np.empty((9, 5, 4))
    W[..., 0] = 1 + 0.05 * rng.uniform(-1, 1, (9, 5))
    W[..., 1:3] = W[..., :1] * 0.2 * rng.uniform(-1, 1, (9, 5, 2))
    W[..., 3] = W[..., 0] * 1.5 + 0.5 * (W[..., 1] ** 2 + W[..., 2] ** 2) / W[..., 0]
    U, V = W[..., 1] / W[..., 0], W[..., 2] / W[..., 0]
    h = (W[..., 0] / (2 * np.pi))[..., None] * np.exp(-((t[0] - U[..., None]) ** 2 + (t[1] - V[..., None]) ** 2) / 2)
    b = h.copy()
    m = [h @ t[2], h @ (t[2] * t[0]), h @ (t[2] * t[1]), 0.5 * (h @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + b @ t[2])]
    W = np.stack(m, -1)

    def gpu(table, hb):
        s = Solver(c, *table)
        try:
            s.upload(hb[0], hb[1], W)
            s.s2cn2_init()
            assert s.step_s2cn2(3)[0] == 3
            return s.download()
        finally:
            s.close()

    def close(a, b, tol=TOL):
        for x, y in zip(a, b):
            assert np.abs(np.asarray(x).reshape(-1) - np.asarray(y).reshape(-1)).max() <= tol * np.abs(y).max()

    got = gpu(t, (h, b))
    o = Oracle(c, *t)
    o.set_state(h, b, W)
    o.s2cn2_init()
    for _ in range(3):
        o.s2cn2_step()
    close(got, o.get_state())
    p = rng.permutation(len(t[0]))
    ph, pb, pW = gpu(tuple(a[p] for a in t), (h[..., p], b[..., p]))
    close((got[0][..., p], got[1][..., p], got[2]), (ph, pb, pW))


# Tolerance: the two paths sum the same terms in other orders and leave out projection weights below 1e-16 of the
# equilibrium: a few roundings of the largest value a step, 1e-12 over three steps with a wide margin for the walls'
# density, a quotient of two sums.
EXPLICIT_TOL = 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("shape,grid", [((8, 4), (4, 3)), ((16, 16), (1, 5)), ((24, 24), (7, 9)), ((20, 28), (3, 4)),
                                        ((32, 32), (2, 11)), ((64, 36), (5, 7)), ((50, 50), (4, 6))])
def test_explicit_tensor_path_matches_oracle_and_general_path(shape, grid):
    """Explicit steps on a tensor table, fused and operator by operator, against the oracle and against the same
    table in another order, which takes the general kernels."""
    from oracle.oracle import Oracle
    from ugks2d_high_order_b200.case import reference_case
    from ugks2d_high_order_b200.solver import Solver
    t, (nx, ny) = rectangle(*shape), grid
    c = reference_case("Explicit").with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny, omega=0.81, wall_ux=(-2.0, 3.0), wall_tnative=(1.8, 2.1))
    rng = np.random.default_rng(7)
    rho, U, V, T = 1 + 0.05 * rng.uniform(-1, 1, (ny, nx)), *(0.2 * rng.uniform(-1, 1, (2, ny, nx))), 2 + 0.1 * rng.uniform(-1, 1, (ny, nx))
    h = (rho / (np.pi * T))[..., None] * np.exp(-((t[0] - U[..., None]) ** 2 + (t[1] - V[..., None]) ** 2) / T[..., None])
    h *= 1 + 0.05 * rng.uniform(-1, 1, h.shape)
    b = 0.5 * T[..., None] * h
    W = np.stack([h @ t[2], h @ (t[2] * t[0]), h @ (t[2] * t[1]), 0.5 * (h @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + b @ t[2])], -1)

    def gpu(table, hb, operators=False):
        s = Solver(c, *table)
        try:
            s.upload(hb[0], hb[1], W)
            for _ in range(3):
                if operators:
                    s.time_step(), s.evolution(), s.compute_residual(), s.apply_explicit_update()
                else:
                    s.step_explicit(1)
            return s.download() + (s.wall_aero(),)
        finally:
            s.close()

    def close(a, b):
        for x, y in zip(a, b):
            assert np.abs(np.asarray(x).reshape(-1) - np.asarray(y).reshape(-1)).max() <= EXPLICIT_TOL * np.abs(y).max()

    got = gpu(t, (h, b))
    o = Oracle(c, *t)
    o.set_state(h, b, W)
    for _ in range(3):
        o.explicit_step()
    close(got, o.get_state())
    close(gpu(t, (h, b), operators=True), got)
    p = rng.permutation(len(t[0]))
    ph, pb, pW, aero = gpu(tuple(a[p] for a in t), (h[..., p], b[..., p]))
    close((got[0][..., p], got[1][..., p], got[2], got[3]), (ph, pb, pW, aero))


# Tolerance: the two paths' closures meet their moments to 5e-13 each, and the closure systems they enter amplify that by
# their condition, of order 1e2 in these units: 1e-10 of the largest cotangent.
VJP_TOL = 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("shape,grid", [((14, 14), (5, 9)), ((12, 20), (8, 12)), ((24, 10), (3, 9)), ((32, 32), (4, 9)),
                                        ((34, 28), (18, 10)), ((64, 36), (3, 11))])
def test_adjoint_tensor_path_matches_general_path(shape, grid):
    """One S2CN2 step's vector-Jacobian product on a tensor table against the same table in another order."""
    from ugks2d_high_order_b200.case import reference_case
    from ugks2d_high_order_b200.solver import Solver
    t, (nx, ny) = rectangle(*shape), grid
    c = reference_case("S2CN2").with_(nx=nx, ny=ny, dx=1 / nx, dy=1 / ny, wall_ux=(-2.0, 3.0), wall_tnative=(1.8, 2.1))
    rng = np.random.default_rng(7)
    rho, U, V, T = (a + s * rng.uniform(-1, 1, (ny, nx, 1)) for a, s in ((1, 0.05), (0.1, 0.2), (0, 0.2), (2, 0.1)))
    h = rho / (np.pi * T) * np.exp(-((t[0] - U) ** 2 + (t[1] - V) ** 2) / T) * (1 + 0.02 * np.tanh(t[0] * t[1]))
    b = 0.5 * c.ck * T * h
    W = np.stack([h @ t[2], h @ (t[2] * t[0]), h @ (t[2] * t[1]), 0.5 * (h @ (t[2] * (t[0] ** 2 + t[1] ** 2)) + b @ t[2])], -1)
    gh, gb, gW, seed = rng.normal(size=h.shape), rng.normal(size=h.shape), rng.normal(size=W.shape), rng.normal(size=4)

    def vjp(p):
        s = Solver(c, *(np.ascontiguousarray(a[p]) for a in t))
        try:
            s.upload(h[..., p], b[..., p], W)
            s.s2cn2_init()
            return s.s2cn2_step_vjp(gh[..., p], gb[..., p], gW, seed)
        finally:
            s.close()

    p = rng.permutation(len(t[0]))
    got, want = vjp(np.arange(len(p))), vjp(p)
    for x, y in zip((got[0][..., p], got[1][..., p], got[2], got[3]), want):
        assert np.isfinite(y).all() and np.abs(x - y).max() <= VJP_TOL * np.abs(y).max()
