"""What the autotuner's cached choices depend on: contexts of one degree and precision in one process, on
paths that differ by the mesh or by the volume rule, are each timed on their own."""
import pytest

pytestmark = pytest.mark.gpu


def tuned(nx, k, precision, quad=0):
    from dg_hdg_euler_cpp_b200.solver import Solver

    s = Solver(nx=nx, ny=nx, k=k, quad=quad, cfl=2.0, integrator="be", steps=1, method="dg", precision=precision, autotune=1)
    u = s.initial()
    s.freeze(u)
    s.set_stage(u, .003)
    s.dg_refresh(u)
    s.precond_refresh("dg")
    report = s.autotune_report()
    s.close()
    return report


def test_fused_residency_is_timed_per_mesh():
    """A mesh with fewer cells than SMs runs the same grid with either residency: nothing is timed there,
    and no choice is left for a larger mesh, which times its own (mixed16: always the fused path)."""
    small, large, again = tuned(6, 4, "mixed16"), tuned(40, 4, "mixed16"), tuned(40, 4, "mixed16")
    assert small["fused_ms"] == [0.0, 0.0] and small["fused_ctas"] == 2
    assert all(t > 0 for t in large["fused_ms"])
    assert again["fused_ms"] == [0.0, 0.0] and again["fused_ctas"] == large["fused_ctas"]


def test_variant_is_timed_per_volume_rule():
    """FP64 variant 0 is the fused launch under the collocated rule, assembly and LU in the pool under the
    over-integrated one."""
    collocated, over = tuned(8, 3, "fp64"), tuned(8, 3, "fp64", quad=6)
    assert all(t > 0 for t in collocated["tune_ms"]["dg"]) and all(t > 0 for t in over["tune_ms"]["dg"])
