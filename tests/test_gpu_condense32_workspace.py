"""The FP32 condensation's workspace: its size, and meshes that it takes in several chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(nx, ny, k, condense32):
    from dg_hdg_euler_cpp_b200.solver import Solver

    return Solver(nx=nx, ny=ny, k=k, cfl=2.0, integrator="be", steps=1, method="hdg", precision="mixed", condense32=condense32)


@pytest.mark.parametrize("nx,ny,k", [(64, 64, 8), (64, 48, 6), (80, 70, 3)])
def test_workspace_size(nx, ny, k):
    """A context holds an augmented matrix in FP32 for every cell, as much as the FP32 LU needs, and no more: against
    FP64 storage of the same mesh it saves half of S and of the workspace and all of X, less its FP32 factors, their
    permutation and a volume vector (to 1 % of the workspace, for the pools' alignment and row padding)."""
    full, slim = context(nx, ny, k, 0), context(nx, ny, k, 1)
    cells, m, t = nx * ny, 4 * (k + 1) ** 2, 16 * (k + 1)
    workspace = cells * m * (m + t + 1) * 4
    saved = cells * (4 * t * t + 8 * m * t - 4 * m * m - 4 * m - 8 * m) + workspace
    got = full.device_bytes() - slim.device_bytes()
    full.close()
    slim.close()
    assert got >= saved - workspace // 100


@pytest.mark.parametrize("nx,ny,k", [(31, 27, 8), (41, 43, 5), (67, 61, 2)])
def test_chunks(nx, ny, k):
    """More cells than the workspace holds in FP64, the last chunk ragged: the Schur apply, the right-hand side and the
    recovery match FP64 condensation to 2e-5, the accuracy of FP32 factors and Schur blocks."""
    out = []
    for condense32 in (0, 1):
        s = context(nx, ny, k, condense32)
        u = s.initial()
        s.freeze(u)
        s.set_stage(u, .004)
        i = np.arange(s.size)
        u = u + 1e-3 * s.tensor(.2 * np.sin(.31 * i) + .1 * np.cos(.79 * i))
        s.hdg_refresh_projected(u, s.residual(u))
        v = np.random.default_rng(k).uniform(-1, 1, size=s.trace_size)
        out.append([x.cpu().numpy() for x in (s.hdg_apply(s.tensor(v)), s.hdg_rhs(), s.hdg_recover(s.tensor(v)))])
        s.close()
    for exact, got in zip(*out):
        assert np.max(np.abs(got - exact)) <= 2e-5 * np.max(np.abs(exact))
