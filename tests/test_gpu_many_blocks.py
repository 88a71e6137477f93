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
