"""Accuracy of the coarsest level's explicit inverse.  With one level the
V-cycle applies it by itself; the exact K^-1 r comes from iterative refinement in
extended precision."""
import numpy as np
import pytest

from topopt3d_b200 import problems as P

pytestmark = pytest.mark.gpu


def design(kind, nel):
    nx, ny, nz = nel
    if kind == "uniform":
        return np.full(nx * ny * nz, 0.5)
    if kind == "rough":
        return np.random.default_rng(1).uniform(0.1, 1.0, nx * ny * nz)
    z, y, x = np.meshgrid(np.linspace(0, 1, nz), np.linspace(0, 1, ny), np.linspace(0, 1, nx),
                          indexing="ij")
    return (0.55 + 0.25 * np.sin(7 * x + 3 * y) * np.cos(5 * z)).reshape(-1)


def operator(T, nel, kind):
    """A context with one level, its dense K and the free dofs."""
    t = T.TopOpt(nel, mg_levels=1)
    P.apply_bcs(t, P.cantilever_bcs(nel))
    t.FEInitialize()
    t.MatIntFnc(design(kind, nel))
    t.FEAssemble()
    n = 3 * t.nNode
    K = np.zeros(n * n)
    t.apply(np.eye(n).reshape(-1), K, nrhs=n)
    fm, _ = t.get_bc()
    free = np.array([not (fm[d // 3] >> (d % 3)) & 1 for d in range(n)], float)
    return t, K.reshape(n, n), free


def energy_errors(t, K, free, Kinv, count):
    """Relative errors in the energy norm of the context's K^-1 r and of Kinv r,
    for random r."""
    Kl = K.astype(np.longdouble)
    rng = np.random.default_rng(5)
    got, ref = [], []
    for _ in range(count):
        r = rng.standard_normal(free.size) * free
        x = (Kinv @ r).astype(np.longdouble)
        for _ in range(8):
            x += Kinv @ (r - Kl @ x).astype(float)
        z = np.zeros_like(r)
        t.vcycle(r.copy(), z)
        for v, out in ((z, got), (Kinv @ r, ref)):
            e = v - x
            out.append(float(np.sqrt(abs(e @ (Kl @ e)) / (x @ (Kl @ x)))))
    return np.median(got), np.median(ref)


def test_inverse_is_as_accurate_as_lapack(T):
    """On compact levels the error is that of LAPACK's inverse, in the mean over
    meshes and designs: both round each entry once per pivot block.  (Products
    summed onto the entries round sixteen times as often, and double it.)"""
    ratio = []
    for nel in ((6, 6, 6), (8, 6, 6), (7, 12, 7), (9, 9, 8)):
        for kind in ("uniform", "smooth", "rough"):
            t, K, free = operator(T, nel, kind)
            got, ref = energy_errors(t, K, free, np.linalg.inv(K), 12)
            ratio.append(got / ref)
    assert np.exp(np.mean(np.log(ratio))) < np.sqrt(2.0)


@pytest.mark.parametrize("nel", [(150, 1, 1), (300, 1, 1)])
def test_inverse_of_a_slender_beam(T, nel):
    """A backward stable factorisation leaves an error of some u cond(K) at
    most in the energy norm, also where cond(K) is 1e11; CG with such an inverse
    converges at once."""
    for kind in ("uniform", "smooth", "rough"):
        t, K, free = operator(T, nel, kind)
        w = np.linalg.eigvalsh(K)
        got, _ = energy_errors(t, K, free, np.linalg.inv(K), 4)
        assert got <= 1.1e-16 * w[-1] / w[0]
        t.FESolve(T.default_opts(rtol=1e-8, precision=T.PREC_FP64))
        assert t.last_solve["status"] == 0 and t.last_solve["iterations"] <= 3
