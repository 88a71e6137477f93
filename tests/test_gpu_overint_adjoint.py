"""The adjoint product under over-integrated volume rules of different sizes, in turn on one device: a kernel must
take its rule from its own argument, not from what a former launch left in shared memory (a rule's size read
before the copy of the rule was complete let threads run with another one, out of range with a random one).

<w, J d> = <J^T w, d> to 1e-12 of |w| |J d| + |J^T w| |d| (sums of up to 2e4 products, each rounded to 1e-16), and
the same product comes out bitwise the same whatever ran before it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RULES = [(1, 16), (8, 10), (1, 3), (3, 9), (8, 16), (5, 8), (2, 13), (6, 12), (4, 6)]  # degree, points per direction


def context(k, quad):
    from dg_hdg_euler_cpp_b200.solver import Solver

    s = Solver(nx=17, ny=13, k=k, quad=quad, cfl=2.0, integrator="be", steps=1, method="dg", restart=1)
    u = s.initial()
    s.freeze(u)
    s.set_stage(u, .004)
    s.dg_refresh(u)
    return s


def test_adjoint_products_of_interleaved_rules():
    contexts = [context(k, quad) for k, quad in RULES]
    first = {}
    for turn in range(8):
        for i in np.random.default_rng(turn).permutation(len(contexts)):
            s = contexts[i]
            rng = np.random.default_rng(100 + i)
            w, d = (s.tensor(rng.standard_normal(s.size)) for _ in range(2))
            jt, jd = s.dg_apply_T(w), s.dg_apply(d)
            scale = float(w.norm() * jd.norm() + jt.norm() * d.norm())
            assert abs(float(w @ jd - jt @ d)) <= 1e-12 * scale, RULES[i]
            got = jt.cpu().numpy()
            assert (first.setdefault(i, got) == got).all(), RULES[i]
    for s in contexts:
        s.close()
