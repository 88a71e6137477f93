"""Block solves and fused factorisations with more blocks than resident warps and CTAs: every warp's ring of
factor chunks runs on from block to block, a buffer or slot is used again, and the last round is ragged.

Every block of a solve is checked by its backward error |A x - b| / (|A| |x|) (infinity norms) against
8 m eps (eps: 2^-53, 2^-24 for FP32 factors, 2^-11 for FP16 factors with a growth factor of 8: 2^-8),
as for single blocks.  The blocks repeat a few distinct ones, in an order that no power of two divides.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"fp64": 2.0**-53, "mixed": 2.0**-24}


def backward_errors(a, x, b):
    n = lambda v: np.max(np.abs(v), axis=-1)
    return n(np.einsum("bij,bj->bi", a, x) - b) / (np.max(np.sum(np.abs(a), axis=2), axis=1) * n(x))


def check_blocks(width, precision, count, seed=0):
    from dg_hdg_euler_cpp_b200.solver import BlockJacobi

    rng = np.random.default_rng(width + seed)
    distinct = rng.uniform(-1, 1, size=(min(37, count), width, width))
    a = distinct[np.arange(count) % len(distinct)]
    b = rng.uniform(-1, 1, size=(count, width))
    bj = BlockJacobi(width, count, precision, 0)
    bj.factor(a)
    x = bj.apply(b.reshape(-1)).reshape(count, width)
    bj.close()
    for first in range(0, count, 512):
        s = slice(first, first + 512)
        assert np.max(backward_errors(a[s], x[s], b[s])) <= 8 * width * EPS[precision], first


@pytest.mark.parametrize("width", [64, 100, 124, 128, 132, 144, 160, 256])
def test_fp32_rings(width):
    """FP32 factors, held whole up to 64 wide, streamed above; from 128 on only a square's triangle is
    fetched.  Twice the resident warps (20 an SM) and a ragged rest."""
    check_blocks(width, "mixed", 2 * 20 * 148 + 5 if width < 160 else 20 * 148 + 5)


@pytest.mark.parametrize("width", [36, 68, 100, 132])
def test_fp64_rings(width):
    """FP64 factors, held whole up to 44 wide, streamed above, with inverted squares."""
    check_blocks(width, "fp64", 20 * 148 + 7)


def linearised(nx, ny, k, **kw):
    from dg_hdg_euler_cpp_b200.solver import Solver

    s = Solver(nx=nx, ny=ny, k=k, cfl=2.0, integrator="be", steps=1, method=kw.pop("method", "dg"), **kw)
    u = s.initial()
    s.freeze(u)
    s.set_stage(u, .004)
    i = np.arange(s.size)
    return s, u + 1e-3 * s.tensor(.2 * np.sin(.31 * i) + .1 * np.cos(.79 * i))


@pytest.mark.parametrize("precision,op,k", [("mixed16", "dg", 4), ("mixed16", "dg", 5), ("fp64", "dg_t", 4), ("mixed", "dg_t", 4),
                                            ("fp64", "dg", 2)])
def test_cells_in_many_rounds(precision, op, k):
    """Cells of a mesh with more cells than resident warps (24 an SM at most) and fused CTAs: the first and
    the last of each round and some between."""
    s, u = linearised(67, 59, k, method="dg", precision=precision)
    s.dg_refresh(u)
    s.precond_refresh("dg")
    m = s.block
    b = np.random.default_rng(k).uniform(-1, 1, size=s.size)
    x = s.precond_apply(op, s.tensor(b)).cpu().numpy()
    bound = 2.0**-8 if precision == "mixed16" else 8 * m * EPS[precision]
    edges = [w * 148 * r + d for w in (12, 16, 20, 24) for r in (1, 2) for d in (-1, 0)]
    for cell in sorted({0, 1, 295, 296, 591, 592, 1184, s.cells // 2, s.cells - 2, s.cells - 1, *edges}):
        if cell >= s.cells:
            continue
        a = s.dg_block(cell, cell)
        a = a.T if op == "dg_t" else a
        sl = slice(cell * m, (cell + 1) * m)
        assert backward_errors(a[None], x[None, sl], b[None, sl])[0] <= bound, cell
    s.close()


@pytest.mark.parametrize("nx,k", [(20, 8), (49, 2)])
def test_fused_fp64_residency_bitwise_equal(nx, k):
    """FP64 cells through one CTA per SM and through all resident ones, more cells than slots."""
    out = []
    for ctas in (1, 2):
        s, u = linearised(nx, nx, k, method="dg", precision="fp64")
        s.dg_refresh(u)
        s.fused_ctas(ctas)
        s.precond_refresh("dg")
        out.append(s.precond_apply("dg", s.tensor(np.random.default_rng(k).uniform(-1, 1, size=s.size))).cpu().numpy())
        s.close()
    assert np.array_equal(*out)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed16"])
def test_degree_zero_cells(precision):
    """4 x 4 cell blocks: one warp's LU, a slab of four rows."""
    s, u = linearised(5, 3, 0, method="dg", precision=precision)
    s.dg_refresh(u)
    s.precond_refresh("dg")
    b = np.random.default_rng(0).uniform(-1, 1, size=s.size)
    for op in ("dg",) if precision == "mixed16" else ("dg", "dg_t"):
        x = s.precond_apply(op, s.tensor(b)).cpu().numpy()
        for cell in range(s.cells):
            a = s.dg_block(cell, cell)
            sl = slice(4 * cell, 4 * cell + 4)
            bound = 2.0**-8 if precision == "mixed16" else 8 * 4 * EPS[precision]
            assert backward_errors((a.T if op == "dg_t" else a)[None], x[None, sl], b[None, sl])[0] <= bound, (op, cell)
    s.close()


def test_degree_zero_schur_apply():
    """The FP32 Schur apply of 4-row faces against FP64 condensation, to 2e-5 (FP32 factors and blocks)."""
    out = []
    for kw in (dict(precision="fp64"), dict(precision="mixed", condense32=1)):
        s, u = linearised(5, 3, 0, method="hdg", **kw)
        s.hdg_refresh_projected(u, s.residual(u))
        v = np.random.default_rng(0).uniform(-1, 1, size=s.trace_size)
        out.append([t.cpu().numpy() for t in (s.hdg_apply(s.tensor(v)), s.hdg_rhs(), s.hdg_recover(s.tensor(v)))])
        s.close()
    for exact, got in zip(*out):
        assert np.max(np.abs(got - exact)) <= 2e-5 * np.max(np.abs(exact))
