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


# the eigensolver's Gram and recombination kernels: blocks of 8, 40 / 72
# (Gram tiles) and 8 .. 64 output columns, fewer rows than a chunk of 64 and
# a partial last one (81, 648 and 1,155 dof), odd and even row counts
@pytest.mark.parametrize("nel,levels,nev,block", [((2, 2, 2), 1, 1, 3), ((5, 5, 5), 1, 2, 4),
                                                  ((10, 6, 4), 2, 3, 7), ((10, 6, 4), 2, 3, 10),
                                                  ((10, 6, 4), 2, 6, 13),
                                                  ((10, 6, 4), 2, 4, 20),
                                                  ((10, 6, 4), 2, 8, 32)])
def test_eigensolver_block_sizes(T, nel, levels, nev, block):
    """The lowest lumped-mass frequencies against a dense generalized
    eigensolve of the operator's own columns: a residual of tol leaves a
    relative eigenvalue error of tol^2 cond, below rounding (n u cond)."""
    t = make(T, nel, levels)
    n = 3 * t.nNode
    lam, _ = t.frequency(nev, 1.0, block=block, tol=1e-9, maxit=2000)
    assert t.last_eig["rc"] == 0
    K = np.zeros(n * n)
    t.apply(np.eye(n).reshape(-1), K, nrhs=n)
    K = K.reshape(n, n)
    # DiagMassFnc: element volume x density / 24 at each of its nodes, 1e-8
    # at fixed dofs
    nx, ny, nz = nel
    rho = t.rho.reshape(nz, ny, nx)
    m = np.zeros((nz + 1, ny + 1, nx + 1))
    for c in range(8):
        i, j, k = c & 1, (c >> 1) & 1, c >> 2
        m[k:k + nz, j:j + ny, i:i + nx] += rho / 24.0
    fm, _ = t.get_bc()
    free = np.array([not (fm[d // 3] >> (d % 3)) & 1 for d in range(n)])
    M = np.repeat(m.reshape(-1), 3)[free]
    import scipy.linalg as sl
    ref = sl.eigh(np.diag(M), K[np.ix_(free, free)], eigvals_only=True)[::-1]
    w = np.linalg.eigvalsh(K)
    assert np.allclose(lam, ref[:lam.size], rtol=n * 1.1e-16 * w[-1] / w[0] + 1e-13, atol=0)


# the tiled filter: halos of 1 (also a radius with one tap), 2 and 3 elements
# and the untiled form beyond, below, at and across the 32 x 16 x 4 tiles
@pytest.mark.parametrize("rmin", [0.9, 1.5, 2.0, 2.5, 3.0, 4.0, 4.3])
@pytest.mark.parametrize("nel", [(1, 1, 1), (3, 2, 5), (31, 16, 4), (33, 17, 9), (64, 15, 3)])
def test_filter_matches_its_matrix(T, nel, rmin):
    """P and P^T against the row-normalised cone summed in numpy: at most 305
    terms of one sign pattern, so rounding stays below 305 u of sum |terms|."""
    nx, ny, nz = nel
    t = T.TopOpt(nel, rmin=rmin, mg_levels=1 if max(nel) < 32 else 2)
    rng = np.random.default_rng(5)
    n = int(rmin)

    def cone(v):
        out = np.zeros_like(v)
        for k in range(-n, n + 1):
            for j in range(-n, n + 1):
                for i in range(-n, n + 1):
                    d = np.sqrt(i * i + j * j + k * k)
                    if d >= rmin or abs(i) >= nx or abs(j) >= ny or abs(k) >= nz:
                        continue
                    dst = tuple(slice(max(0, -a), m - max(0, a)) for a, m in
                                ((k, nz), (j, ny), (i, nx)))
                    src = tuple(slice(max(0, a), m - max(0, -a)) for a, m in
                                ((k, nz), (j, ny), (i, nx)))
                    out[dst] += (1.0 - d / rmin) * v[src]
        return out
    rows = cone(np.ones((nz, ny, nx)))
    for transpose in (False, True):
        v = rng.uniform(-1.0, 1.0, (nz, ny, nx))
        ref = cone(v / rows) if transpose else cone(v) / rows
        size = cone(np.abs(v) / rows) if transpose else cone(np.abs(v)) / rows
        got = t.filter(v.reshape(-1), transpose=transpose).reshape(nz, ny, nx)
        assert np.all(np.abs(got - ref) <= 2 * 305 * 1.1e-16 * size)


# the OC bisection keeps its elements in registers on few blocks: part of a
# block, exactly one and one element more, exactly one element a thread on 148
# blocks (151,552), past it, exactly two, past that (the arrays read again)
@pytest.mark.parametrize("nel", [(13, 6, 6), (16, 8, 8), (41, 5, 5), (64, 37, 64), (64, 37, 65),
                                 (128, 37, 64), (64, 75, 65)])
def test_oc_update_over_sizes(T, oracle, nel):
    """The bisection against the oracle's: the same branches, so what differs is
    rounding (1e-16 a term; the last multiplier interval, 1e-9 of the
    multiplier, moves the constraint sum 1e5 times more than its rounding)."""
    n = int(np.prod(nel))
    t = T.TopOpt(nel, mg_levels=2 if n < 2000 else 4)
    rng = np.random.default_rng(n)
    x = rng.uniform(0.2, 0.8, n)
    dfdx = -rng.uniform(0.0, 1.0, n)
    dfdx[::7] = 0.3
    dgdx = rng.uniform(0.5, 1.5, n) / n
    oc = T.OC(n, move=0.2)
    oc.xval = x.copy()
    xg = oc.Update(t, dfdx.copy(), np.array([0.02]), dgdx[:, None])
    xo, cho = oracle.oc_update(x, dfdx, 0.02, dgdx, 0.2)
    assert np.max(np.abs(xg - xo)) < 1e-12 and abs(oc.Change - cho) < 1e-12


# the z chunks of the matrix-free operator, from one plane to all: a block of
# columns cuts z at other planes than one column does
@pytest.mark.parametrize("nel", [(1, 1, 1), (12, 6, 6), (5, 9, 30), (30, 7, 17), (48, 24, 24)])
def test_apply_chunks_give_the_same_values(T, nel):
    """A node's value does not depend on the chunk it is in, bit for bit."""
    t = make(T, nel, 1 if int(np.prod(nel)) < 2000 else 3, assemble=False)
    n, nb = 3 * t.nNode, 40
    u = np.random.default_rng(1).standard_normal(nb * n)
    y, y1 = np.zeros_like(u), np.zeros(n)
    t.apply(u, y, nrhs=nb)
    for j in (0, nb - 1):
        t.apply(u[j * n:(j + 1) * n], y1)
        assert np.array_equal(y1, y[j * n:(j + 1) * n])


# CG's dot products: in the operator's epilogue (degree 2), by a pass of their
# own (other degrees, one level), one column and blocks of 3 and 8, on meshes of
# one CTA and of many
@pytest.mark.parametrize("nel,levels", [((4, 3, 2), 1), ((12, 6, 6), 2), ((31, 14, 9), 3)])
@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("nb", [1, 3, 8])
def test_cg_dot_products(T, nel, levels, degree, nb):
    """Every column ends below its target, and no sooner than CG has to: the
    same iterations as the column alone (a sum in another order moves ||r|| by
    1e-14 of itself, an iteration moves it by tenths)."""
    o = T.default_opts(cheb_degree=degree, rtol=1e-6, precision=T.PREC_FP64)
    t = make(T, nel, levels, opts=o)
    n = 3 * t.nNode
    b = np.random.default_rng(2).standard_normal((nb, n))
    fm, _ = t.get_bc()
    b[:, [d for d in range(n) if (fm[d // 3] >> (d % 3)) & 1]] = 0.0
    U, y = np.zeros_like(b), np.zeros_like(b)
    its = t.solve(b, U, nrhs=nb, opts=o)["iterations"]
    t.apply(U, y, nrhs=nb)
    assert np.all(np.linalg.norm(b - y, axis=1) <= 1.0001e-6 * np.linalg.norm(b, axis=1))
    alone = []
    for j in range(nb):
        Uj = np.zeros(n)
        alone.append(t.solve(b[j].copy(), Uj, opts=o)["iterations"])
        assert np.linalg.norm(Uj - U[j]) <= 1e-5 * np.linalg.norm(Uj)
    assert its == sum(alone)


# the captured CG loop outlives the operator: one column and a block, both
# forms, with other smoother options and other boundary conditions in between
@pytest.mark.parametrize("nb", [1, 3])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("nel", [(12, 6, 6), (32, 16, 16)])
def test_a_new_operator_solves_as_in_a_new_context(T, nel, mixed, nb):
    """After other designs, options and supports the context solves as one that
    has seen the last of them only, bit for bit."""
    prec = T.PREC_MIXED if mixed else T.PREC_FP64
    b = np.random.default_rng(4).standard_normal((nb, 3 * int(np.prod(np.add(nel, 1)))))

    def step(t, bc, seed, degree):
        o = T.default_opts(precision=prec, cheb_degree=degree)
        t.set_bc_arrays(np.zeros(t.nNode, np.uint8), np.zeros(3 * t.nNode))
        P.apply_bcs(t, bc)
        t.FEInitialize()
        t.MatIntFnc(np.random.default_rng(seed).uniform(0.3, 0.8, t.nElem))
        t.FEAssemble(o)
        t.set("U", np.zeros(3 * t.nNode))
        t.FESolve(o)
        U = np.zeros_like(b)
        t.solve(b, U, nrhs=nb, opts=o)
        return np.array(t.U), U
    one, two = P.cantilever_bcs(nel), P.bcs("cfg2", nel)
    t = T.TopOpt(nel, mg_levels=3)
    for bc, seed, degree in ((one, 1, 2), (one, 2, 2), (one, 2, 1), (two, 3, 2), (one, 4, 2)):
        got = step(t, bc, seed, degree)
        ref = step(T.TopOpt(nel, mg_levels=3), bc, seed, degree)
        assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
