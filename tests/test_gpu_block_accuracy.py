"""Backward error of the FP64 block solves on blocks whose 32 x 32 diagonal squares are ill-conditioned.

A solve by substitution has a normwise backward error |A x - b| / (|A| |x|) (infinity norms) of a few
rounding errors whatever the condition of the triangles; the bound is the one of the well-conditioned
blocks, 8 m eps.  Blocks: unit triangles of -a (their inverses grow like (1 + a)^31), the same
upper ones times a random unit lower factor, Kahan's triangle, rows scaled over 1e-8..1e8, triangles whose
inverse is out of the FP64 range, and whole blocks near the ends of that range.  Cells: blocks
linearised at a rough state (random density, velocity and pressure per node), solved forward and
transposed; their squares reach max|U| max|U^-1| of 1e6 to 1e12.
"""
import numpy as np
import pytest

EPS = 2.0**-53


def backward_error(a, x, b):
    x = x.astype(np.longdouble)
    a = a.astype(np.longdouble)
    n = lambda v: np.max(np.abs(v))
    return float(n(a @ x - b) / (np.max(np.sum(np.abs(a), axis=1)) * n(x)))


def blocks(kind, m, rng):
    upper = lambda a: np.triu(-a * np.ones((m, m)), 1) + np.eye(m)
    lower = np.tril(rng.uniform(-1, 1, size=(m, m)), -1) + np.eye(m)
    if kind == "ones":
        return upper(1.0)
    if kind == "dense":
        return lower @ upper(1.0)
    if kind == "half":
        return lower @ upper(0.5)
    if kind == "lower":
        return upper(1.0).T
    if kind == "kahan":
        return np.diag(np.sin(0.9) ** np.arange(m)) @ upper(np.cos(0.9))
    if kind == "graded":
        return np.diag(10.0 ** rng.uniform(-8, 8, m)) @ rng.uniform(-1, 1, size=(m, m))
    if kind == "range":  # an inverse entry of 1e400
        a = 1e-200 * np.eye(m)
        a[range(0, m, 2), range(1, m, 2)] = 1.0
        return a
    return rng.uniform(-1, 1, size=(m, m)) * {"tiny": 1e-290, "huge": 1e290}[kind]


KINDS = ["ones", "lower", "dense", "half", "kahan", "graded", "range", "tiny", "huge"]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("width,variants", [(12, (0, 1, 2)), (32, (0, 1, 2)), (36, (0, 1, 2)), (100, (0, 1)), (324, (0,))])
def test_ill_conditioned_blocks(kind, width, variants):
    from dg_hdg_euler_cpp_b200.solver import BlockJacobi

    count = 3
    rng = np.random.default_rng(width)
    a = np.stack([blocks(kind, width, rng) for _ in range(count)])
    x0 = rng.uniform(0.5, 1, size=(count, width))
    for b in (np.einsum("bij,bj->bi", a, x0), np.max(np.abs(a)) * 2.0 ** rng.uniform(-1, 1, size=(count, width))):
        if kind == "range" and b[0, 1] > 1e-100:
            continue  # its solution would be out of range
        for variant in variants:
            bj = BlockJacobi(width, count, "fp64", variant)
            bj.factor(a)
            x = bj.apply(b.reshape(-1)).reshape(count, width)
            bj.close()
            for i in range(count):
                assert backward_error(a[i], x[i], b[i]) <= 8 * width * EPS, (variant, i)


def rough_state(cells, k, seed):
    """Random admissible nodal values ([cell][variable][node]): rho, p in [1/e, e], velocities N(0, 3), gamma = 3."""
    rng = np.random.default_rng(seed)
    shape = (cells, (k + 1) ** 2)
    rho, p = np.exp(rng.uniform(-1, 1, shape)), np.exp(rng.uniform(-1, 1, shape))
    vx, vy = 3 * rng.standard_normal(shape), 3 * rng.standard_normal(shape)
    return np.stack([rho, rho * vx, rho * vy, p / 2 + rho * (vx * vx + vy * vy) / 2], axis=1).reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 3, 4, 6, 8])
def test_cell_blocks_of_a_rough_linearisation(k):
    from dg_hdg_euler_cpp_b200.solver import Solver

    s = Solver(nx=5, ny=3, k=k, cfl=2.0, integrator="be", steps=1, method="dg", precision="fp64")
    u = s.initial()
    s.freeze(u)
    s.set_stage(u, 1e3)
    s.dg_refresh(s.tensor(rough_state(s.cells, k, k)))
    s.precond_refresh("dg")
    m = s.block
    b = np.random.default_rng(k).uniform(-1, 1, size=s.size)
    for op in ("dg", "dg_t"):
        x = s.precond_apply(op, s.tensor(b)).cpu().numpy()
        for cell in range(s.cells):
            a = s.dg_block(cell, cell)
            sl = slice(cell * m, (cell + 1) * m)
            assert backward_error(a.T if op == "dg_t" else a, x[sl], b[sl]) <= 8 * m * EPS, (op, cell)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("width", [4, 12, 28, 32])
def test_fp32_factors_in_the_subnormal_range(width):
    """FP32 factors of blocks around 1e-40, in steps of 2^-149: 2^-16 of the largest entry, so that a solve by
    quotients keeps a backward error of 8 m 2^-16; a reciprocal of such a pivot is out of range."""
    from dg_hdg_euler_cpp_b200.solver import BlockJacobi

    count = 6
    rng = np.random.default_rng(width)
    a = 1e-40 * rng.uniform(-1, 1, size=(count, width, width))
    b = 1e-40 * rng.uniform(-1, 1, size=(count, width))
    bj = BlockJacobi(width, count, "mixed", 0)
    bj.factor(a)
    x = bj.apply(b.reshape(-1)).reshape(count, width)
    bj.close()
    for i in range(count):
        assert backward_error(a[i], x[i], b[i]) <= 8 * width * 2.0**-16, i
