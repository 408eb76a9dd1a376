"""GPU kernels at the sizes where their tiling can go wrong, each against the
operation it computes."""
import numpy as np
import pytest

from topopt3d_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import topopt3d_b200 as T
    return T


def make(T, nel, levels, seed=0, rmin=1.5, assemble=True, opts=None):
    t = T.TopOpt(nel, rmin=rmin, mg_levels=levels)
    P.apply_bcs(t, P.cantilever_bcs(nel))
    t.FEInitialize()
    t.MatIntFnc(np.random.default_rng(seed).uniform(0.3, 0.8, int(np.prod(nel))))
    if assemble:
        t.FEAssemble(opts)
    return t


# plane groups and blocks of the coarsest inverse: one block (24 unknowns),
# several planes a block (60, 54), one plane a block (48), two and three
# blocks a plane (38, 54, 49), a partial last group, each dimension longest
@pytest.mark.parametrize("nel", [(1, 1, 1), (2, 1, 1), (29, 1, 1), (1, 22, 1), (2, 2, 13),
                                 (6, 3, 3), (3, 8, 4), (8, 4, 4), (5, 5, 5), (4, 5, 12),
                                 (12, 6, 6), (9, 9, 8)])
def test_coarsest_inverse_is_the_inverse(T, nel):
    """With one level the V-cycle is the coarsest inverse: K (V r) = r.  The
    explicit inverse of a symmetric positive definite matrix leaves
    |K V r - r| <= n u cond(K) |r|, with the condition number of this K (its
    columns come from the operator itself; a slender beam's is 1e8)."""
    t = make(T, nel, 1)
    n = 3 * t.nNode
    r = np.random.default_rng(3).standard_normal(n)
    z, y = np.zeros_like(r), np.zeros_like(r)
    t.vcycle(r, z)
    t.apply(z, y)
    K = np.zeros(n * n)
    t.apply(np.eye(n).reshape(-1), K, nrhs=n)
    w = np.linalg.eigvalsh(K.reshape(n, n))
    assert np.linalg.norm(y - r) <= n * 1.1e-16 * w[-1] / w[0] * np.linalg.norm(r)
