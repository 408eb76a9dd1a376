"""One context over several assemblies: other supports, other numbers of
elements next to fixed dofs, the same design again."""
import numpy as np
import pytest

from topopt3d_b200 import problems as P

pytestmark = pytest.mark.gpu

# level 1 (65 x 33 x 33 nodes) is above the persistent coarse levels: mixed
# solves take it on the tensor cores, with correction rows next to fixed dofs
NEL = (128, 64, 64)
LEVELS = 4


def point(j, k):
    """A support on the node in the middle of level-1 element (j, k) of the
    face x = max: it makes that element, and no other, a general one."""
    return ("support", (float(NEL[0]), 2.0 * j + 1, 2.0 * k + 1), (P.TINY,) * 3, P.OPEN,
            (1.0, 1.0, 1.0))


# eight level-1 elements around one; the ninth's eight nodes are theirs too
RING = [point(j, k) for j in (10, 11, 12) for k in (20, 21, 22) if (j, k) != (11, 21)]
INNER = [point(11, 21)]


def step(T, t, bc, x):
    """Assemble and solve from zero with these supports: U, iterations."""
    o = T.default_opts(precision=T.PREC_MIXED, rtol=1e-8)
    t.set_bc_arrays(np.zeros(t.nNode, np.uint8), np.zeros(3 * t.nNode))
    P.apply_bcs(t, bc)
    t.FEInitialize()
    t.MatIntFnc(x)
    t.FEAssemble(o)
    t.set("U", np.zeros(3 * t.nNode))
    t.FESolve(o)
    return np.array(t.U), t.last_solve["iterations"]


def test_more_general_elements_with_the_same_correction_rows(T):
    """The second supports have one general element more than the first and the
    same 33 x 33 x 2 + 32 level-1 nodes next to fixed dofs: the buffers of the
    correction rows grow while their number stays.  The context must then solve
    as a new one: below the target, in as many
    iterations to within one."""
    x = np.random.default_rng(3).uniform(0.3, 0.8, int(np.prod(NEL)))
    base = P.cantilever_bcs(NEL)
    t = T.TopOpt(NEL, mg_levels=LEVELS)
    step(T, t, base + RING, x)
    U, its = step(T, t, base + RING + INNER, x)
    new = T.TopOpt(NEL, mg_levels=LEVELS)
    V, ref = step(T, new, base + RING + INNER, x)
    F, y = np.array(t.F), np.zeros_like(U)
    for u in (U, V):
        t.apply(u, y)
        assert np.linalg.norm(F - y) <= 1.0001e-8 * np.linalg.norm(F)
    assert abs(its - ref) <= 1


@pytest.mark.parametrize("supports", ["face", "face and ring"])
def test_an_assembly_does_not_depend_on_those_before(T, supports):
    """The smoothers' bounds and the solution of a design are the same, bit for
    bit, whether the context has assembled it before, or other supports, or
    nothing: each correction row is one warp's sum and every reduction has a
    fixed order."""
    x = np.random.default_rng(4).uniform(0.3, 0.8, int(np.prod(NEL)))
    base = P.cantilever_bcs(NEL)
    bc = base + (RING if "ring" in supports else [])
    other = base + ([] if "ring" in supports else RING)
    new = T.TopOpt(NEL, mg_levels=LEVELS)
    ref = step(T, new, bc, x)
    lam = [new.level_lambda(l) for l in range(LEVELS - 1)]
    again = step(T, new, bc, x)
    t = T.TopOpt(NEL, mg_levels=LEVELS)
    step(T, t, other, x)
    after = step(T, t, bc, x)
    for c, got in ((new, again), (t, after)):
        assert [c.level_lambda(l) for l in range(LEVELS - 1)] == lam
        assert got[1] == ref[1] and np.array_equal(got[0], ref[0])
