"""One V-cycle of the pressure and diffusion solves against the same cycle from
scipy products: the hierarchy of the library's host phase (aggregates and term
structure, checked by test_amg_symbolic.py), its numeric phase, the Chebyshev
bounds by power iteration, the smoothers, and the coarsest level by a direct
solve. The pressure solve's first iteration (GCR) returns x = (b.q / q.q) z with
z = M^-1 b and q = A z, the diffusion solve's (BiCGStab) a combination of two
cycles, so a solve stopped after one shows the cycle itself, and with it every
form that its kernels take: the fixed-width formats and their streaming loads,
CSR where they are refused, the dense operator in one and two passes over its
columns and its absence, the coarsest inverse in one and four blocks, the power
iteration in a cluster and in kernels of its own.

FP64 differs by rounding alone: some 60 phases of sums of up to 400 terms, and
a coarsest level of condition up to 1e4, stay below 1e-10. The mixed form keeps
matrices, transfers and vectors in FP32 (6e-8); through the same condition that
is at most 6e-4, with the one exception of a hierarchy of one level, whose cycle
is the inverse itself: 2e-3 holds all."""
import numpy as np
import pytest

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

from .test_amg_symbolic import _lists, harness  # noqa: F401
from .test_gpu_node_orders import renumber

COARSEST, CHEB_ROWS = 256, 50000


def power_bound(A, dinv):
    h = (np.arange(A.shape[0], dtype=np.uint64) * 2654435761) & 0xFFFFFFFF
    h ^= h >> 15
    h = (h * 2246822519) & 0xFFFFFFFF
    h ^= h >> 13
    v, norm = h * (2.0 / 4294967296.0) - 1.0, 1.0
    for _ in range(15):
        v = dinv * (A @ v) / norm
        norm = np.linalg.norm(v)
    return 1.1 * norm


def hierarchy(L, A, wp=0.74):
    import scipy.sparse as sp

    levels = []
    while True:
        n = A.shape[0]
        lv = dict(A=A, dinv=1.0 / A.diagonal())
        levels.append(lv)
        if n <= COARSEST:
            return levels
        nc, h = _lists(L, A)
        rows = np.repeat(np.arange(n), np.diff(h["prp"]))
        own = np.zeros(h["pcols"].size)
        own[h["prp"][:-1] + h["pdiag"]] = 1.0
        pv = own - wp * lv["dinv"][rows] * np.add.reduceat(A.data[h["pglist"]], h["pgptr"][:-1])
        lv["P"] = sp.csr_matrix((pv, h["pcols"], h["prp"]), shape=(n, nc))
        tv = np.add.reduceat(A.data[h["tta"]] * pv[h["ttp"]], h["ttptr"][:-1])
        cv = np.add.reduceat(pv[h["ctp"]] * tv[h["ctt"]], h["ctptr"][:-1])
        if len(levels) > 1 and n <= CHEB_ROWS:
            lv["lambda"] = power_bound(A, lv["dinv"])
        A = sp.csr_matrix((cv, h["ccols"], h["crp"]), shape=(nc, nc))


def cycle(levels, b, l=0, degree=3, ratio=30.0, omega=0.8):
    lv = levels[l]
    A, dinv = lv["A"], lv["dinv"]
    if l == len(levels) - 1:
        return np.linalg.solve(A.toarray(), b)

    def smooth(x):
        if "lambda" not in lv:
            return x + omega * dinv * (b - A @ x)
        hi = lv["lambda"]
        theta, delta = 0.5 * (hi + hi / ratio), 0.5 * (hi - hi / ratio)
        r = dinv * (b - A @ x)
        d, rho = r / theta, delta / theta
        x = x + d
        for _ in range(1, degree):
            new = 1.0 / (2.0 * theta / delta - rho)
            r = r - dinv * (A @ d)
            d = new * rho * d + 2.0 * new / delta * r
            x, rho = x + d, new
        return x

    x = smooth(np.zeros_like(b))
    x = x + lv["P"] @ cycle(levels, lv["P"].T @ (b - A @ x), l + 1)
    return smooth(x)


def first_iterate(levels, b, gcr=True):
    A = levels[0]["A"]
    z = cycle(levels, b)
    q = A @ z
    if gcr:
        return (b @ q) / (q @ q) * z
    alpha = (b @ b) / (b @ q)
    s = b - alpha * q
    sz = cycle(levels, s)
    t = A @ sz
    return alpha * z + (t @ s) / (t @ t) * sz


def csr_refused(rp):
    longest, slots = np.diff(rp).max(), 32 * ((rp.size - 1 + 31) // 32)
    width = 7 if longest <= 7 else 15
    return longest > width or slots * width > 2 * rp[-1] + 4096


def pressure(m, prec):
    f = rt.Flow(rt.Mesh(m), rt.default_settings(precision=prec))
    f.set_field("U", np.random.default_rng(5).normal(0, 0.1, 3 * m.nn))
    f.initialize()
    f.assemble_momentum(copy=False)
    f.update_mdot()
    A, b = f.assemble_pcorr()
    return f, A, b, f.solve("pcorr", 1e-30, 1)


def conduction(n, prec):
    m, gamma, src, _ = meshgen.conduction(n)
    d = rt.Diffusion(rt.Mesh(m), rt.default_diffusion_settings(precision=prec))
    d.set_field("gamma", gamma)
    d.set_field("src", src)
    A, b = d.assemble()
    return d, A, b, d.solve(1e-30, 1)


# rows of the levels
CAVITIES = [((5, 5, 6), [252]),                  # four blocks for the inverse, no cycle above it
            ((6, 6, 6), [343, 48]),              # a coarse level too small for the dense operator
            ((12, 12, 12), [2197, 280, 11]),     # dense operator, columns in one pass
            ((16, 16, 16), [4913, 646, 23]),     # in two
            ((20, 20, 20), [9261, 1132, 34]),    # none
            ((61, 53, 47), [160704, 20352, 528, 10]),  # two passes, a Chebyshev level above them
            ((85, 85, 85), None)]                # streaming loads in FP64, power iteration by kernels
STARS = [(3, 5, 4), (5, 5, 4), (5, 8, 6), (5, 10, 12)]  # widths 7 and 15; both others CSR


def check(harness, handle, A, b, solved, prec, rows=None, gcr=True):
    import scipy.sparse as sp

    x, it, _ = solved[:3]
    assert it == 1
    rp, cols = handle.mesh.graph()
    levels = hierarchy(harness, sp.csr_matrix((A, cols, rp), shape=(b.size, b.size)))
    n = [lv["A"].shape[0] for lv in levels]
    assert rows is None or n == rows, n
    want = first_iterate(levels, b, gcr)
    assert np.linalg.norm(x - want) <= (1e-10 if prec == rt.OA_PREC_FP64 else 2e-3) * np.linalg.norm(want)
    return rp


PRECISIONS = pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])


@pytest.mark.gpu
@PRECISIONS
@pytest.mark.parametrize("shape,rows", CAVITIES)
def test_hex_blocks(harness, shape, rows, prec):  # noqa: F811
    f, A, b, solved = pressure(meshgen.cavity(shape, perturb=0.2), prec)
    assert not csr_refused(check(harness, f, A, b, solved, prec, rows))


# 256 rows, one more than a multiple of 32 (225) and of 256 (513)
@pytest.mark.gpu
@PRECISIONS
@pytest.mark.parametrize("shape", [(7, 7, 3), (4, 4, 8), (2, 8, 18)])
def test_group_and_block_edges(harness, shape, prec):  # noqa: F811
    f, A, b, solved = pressure(meshgen.cavity(shape), prec)
    assert not csr_refused(check(harness, f, A, b, solved, prec))


# columns instead of distances in all or some groups; the large ones with
# streaming loads in FP64
@pytest.mark.gpu
@PRECISIONS
@pytest.mark.parametrize("order", ["half", "random"])
@pytest.mark.parametrize("shape", [(20, 20, 20), (85, 85, 85)])
def test_node_orders(harness, shape, order, prec):  # noqa: F811
    f, A, b, solved = pressure(renumber(meshgen.cavity(shape, perturb=0.2), order), prec)
    assert not csr_refused(check(harness, f, A, b, solved, prec))


@pytest.mark.gpu
@PRECISIONS
@pytest.mark.parametrize("star", STARS)
def test_blocks_around_an_axis(harness, star, prec):  # noqa: F811
    f, A, b, solved = pressure(meshgen.star_prism(*star), prec)
    assert csr_refused(check(harness, f, A, b, solved, prec)) == (star in STARS[2:])


@pytest.mark.gpu
@PRECISIONS
@pytest.mark.parametrize("n", [3, 6, 12, 20, 66])
def test_tets(harness, n, prec):  # noqa: F811
    d, A, b, solved = conduction(n, prec)
    assert not csr_refused(check(harness, d, A, b, solved, prec, gcr=False))
