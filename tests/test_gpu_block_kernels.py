"""The batched LU, the block solves and the FP32 Schur apply at the edges of their tiles.

Blocks: widths around the panel (32), the halves of a panel (16), the warps' row counts and the last
slab's row sharing (4, 8, 16), up to the widest (512); the pivots equal a numpy restatement of
first-largest partial pivoting, and a solve's normwise backward error |A x - b| / (|A| |x|) (infinity
norms) stays below 8 m eps, the usual bound of partial pivoting with a growth factor of 8 (eps: 2^-53,
or 2^-24 for FP32 factors).  Degrees: the cell blocks of one odd mesh per degree, assembled and
factored by the solver itself, solved forward and transposed under the same bound; FP16 factors carry
2^-11 relative rounding of L and U (and of the row scales), whose product's growth over |A| is
allowed a factor of 8: 2^-8.  The FP32 Schur apply is linear in a matrix rounded to FP32 after an FP32-accurate
condensation, and matches the FP64 operator to 2e-5, the accuracy of the FP32 condensation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"fp64": 2.0**-53, "mixed": 2.0**-24}


def ref_pivots(a):
    a = a.copy()
    n = a.shape[0]
    perm = np.arange(n)
    for k in range(n):
        p = k + int(np.argmax(np.abs(a[k:, k])))
        if p != k:
            a[[k, p]] = a[[p, k]]
            perm[[k, p]] = perm[[p, k]]
        a[k + 1:, k] /= a[k, k]
        a[k + 1:, k + 1:] -= np.outer(a[k + 1:, k], a[k, k + 1:])
    return perm


def backward_error(a, x, b):
    n = lambda v: np.max(np.abs(v))
    return n(a @ x - b) / (np.max(np.sum(np.abs(a), axis=1)) * n(x))


@pytest.mark.parametrize("width", [4, 8, 12, 16, 20, 28, 32, 36, 40, 48, 64, 68, 96, 100, 128, 132, 144, 160, 196, 224,
                                   256, 260, 324, 384, 404, 512])
def test_blocks_at_tile_edges(width):
    from dg_hdg_euler_cpp_b200.solver import BlockJacobi

    count = 5
    rng = np.random.default_rng(width)
    a = rng.uniform(-1, 1, size=(count, width, width))
    b = rng.uniform(-1, 1, size=(count, width))
    for precision in ("fp64", "mixed"):
        bj = BlockJacobi(width, count, precision, 0)
        bj.factor(a)
        x = bj.apply(b.reshape(-1)).reshape(count, width)
        perm = bj.perm()
        bj.close()
        for i in range(count):
            assert backward_error(a[i], x[i], b[i]) <= 8 * width * EPS[precision], (precision, i)
            assert (perm[i] == ref_pivots(a[i])).all(), (precision, i)


def frozen(nx, ny, k, **kw):
    from dg_hdg_euler_cpp_b200.solver import Solver

    s = Solver(nx=nx, ny=ny, k=k, cfl=2.0, integrator="be", steps=1, **kw)
    u = s.initial()
    s.freeze(u)
    s.set_stage(u, .004)
    i = np.arange(s.size)
    return s, u + 1e-3 * s.tensor(.2 * np.sin(.31 * i) + .1 * np.cos(.79 * i))


@pytest.mark.parametrize("k", range(1, 9))
def test_cell_blocks_by_degree(k):
    rng = np.random.default_rng(k)
    for precision, tol in (("fp64", None), ("mixed", None), ("mixed16", 2.0**-8)):
        s, u = frozen(5, 3, k, method="dg", precision=precision)
        s.dg_refresh(u)
        s.precond_refresh("dg")
        m = s.block
        b = rng.uniform(-1, 1, size=s.size)
        bound = tol or 8 * m * EPS[precision]
        for op in ("dg",) if precision == "mixed16" else ("dg", "dg_t"):
            x = s.precond_apply(op, s.tensor(b)).cpu().numpy()
            for cell in (0, 7, s.cells - 1):
                a = s.dg_block(cell, cell)
                sl = slice(cell * m, (cell + 1) * m)
                assert backward_error(a.T if op == "dg_t" else a, x[sl], b[sl]) <= bound, (precision, op, cell)
        s.close()


@pytest.mark.parametrize("k", range(1, 9))
def test_fp32_schur_apply_by_degree(k):
    out = []
    for kw in (dict(precision="fp64"), dict(precision="mixed", condense32=1)):
        s, u = frozen(5, 3, k, method="hdg", **kw)
        s.hdg_refresh_projected(u, s.residual(u))
        v = np.random.default_rng(k).uniform(-1, 1, size=s.trace_size)
        out.append([t.cpu().numpy() for t in (s.hdg_apply(s.tensor(v)), s.hdg_rhs(), s.hdg_recover(s.tensor(v)))])
        s.close()
    for exact, got in zip(*out):
        assert np.max(np.abs(got - exact)) <= 2e-5 * np.max(np.abs(exact))


@pytest.mark.parametrize("restart", [4, 16, 31])
@pytest.mark.parametrize("nx,ny,k", [(3, 3, 1), (5, 3, 2), (16, 9, 3)])
def test_gmres_cycles(nx, ny, k, restart):
    """The reductions, the Hessenberg update and the back substitution at full and partial cycles: the
    returned solution's own residual in the 2-norm, 1e-12 in the solver's weighted norm, whose weights
    vary by less than 1e2 over a mesh of equal cells; stepped and replayed cycles alike."""
    found = []
    for graph in (False, True):
        s, u = frozen(nx, ny, k, method="dg", restart=restart)
        s.dg_refresh(u)
        s.precond_refresh("dg")
        s.gmres_graph(graph)
        rhs = s.residual(u)
        x = s.gmres("dg", rhs, 2000, 1e-12)[0]
        r = (s.dg_apply(x) - rhs).cpu().numpy()
        assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(rhs.cpu().numpy())
        found.append(x.cpu().numpy())
        s.close()
    assert (found[0] == found[1]).all()
