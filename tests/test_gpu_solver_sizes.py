"""The pressure-correction and scalar-diffusion solves at the sizes where their
kernels change form: row counts around 32 and 256 (groups of the fixed-width
storage, blocks of the vector kernels), coarsest levels of 8 to 252 rows
(dense inverse in one block up to 128 rows, in four blocks above), hierarchies
with and without a dense operator, rows of 7 entries (hex block), 15 (Kuhn
tets) and more than the fixed width holds (several blocks around an axis), one
and many disjoint systems.

The solver's own residual is a recurrence (FP64) or an FP64 residual of the
stored matrix (mixed); the residual of its solution on the host may differ by
rounding, ||A|| ||x|| eps / ||b|| <= 1e-11 for these systems (condition below
1e4), so it is held to the tolerance plus 1e-10."""
import numpy as np
import pytest

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def host_residual(gm, A, b, x):
    import scipy.sparse as sp

    rp, cols = gm.graph()
    M = sp.csr_matrix((A, cols, rp), shape=(gm.nn, gm.nn))
    return np.linalg.norm(b - M @ x) / np.linalg.norm(b)


def pressure_residual(m, prec, refs=None, **kw):
    gm = rt.Mesh(m)
    f = rt.Flow(gm, rt.default_settings(precision=prec, **kw))
    if refs is not None:
        f.set_reference_nodes(refs)
    f.set_field("U", np.random.default_rng(5).normal(0, 0.1, 3 * m.nn))
    f.initialize()
    f.assemble_momentum(copy=False)
    f.update_mdot()
    A, b = f.assemble_pcorr()
    x, it, res = f.solve("pcorr", RTOL, 2000)
    assert it > 0 and res <= RTOL
    return host_residual(gm, A, b, x)


# rows: 8, 12, 32, 33 (3 x 11 x 1), 125, 128, 252, 343 (first coarse level),
# 2,197 (coarse levels below the dense operator's limit), 9,261 (above it)
SHAPES = [(1, 1, 1), (2, 1, 1), (3, 3, 1), (10, 2, 1), (4, 4, 4), (3, 3, 7), (5, 5, 6), (6, 6, 6), (12, 12, 12),
          (20, 20, 20)]


@pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])
@pytest.mark.parametrize("shape", SHAPES)
def test_pressure_solve_sizes(shape, prec):
    assert pressure_residual(meshgen.cavity(shape), prec) <= RTOL + 1e-10


@pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])
@pytest.mark.parametrize("blocks", [3, 5])
def test_pressure_solve_without_fixed_width(blocks, prec):
    m = meshgen.star_prism(blocks, 5, 4)
    assert pressure_residual(m, prec) <= RTOL + 1e-10


@pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])
def test_batch_segments_of_uneven_size(prec):
    # segments of 8, 5,832 (two chunks) and 27 rows
    b = meshgen.batch_cavities(sizes=[1, 17, 2], seed=3)
    assert pressure_residual(b.mesh, prec, refs=b.ref_nodes, ref_node=-1) <= RTOL + 1e-10


@pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])
@pytest.mark.parametrize("n", [1, 3, 6, 12])
def test_diffusion_solve_sizes(n, prec):
    m, gamma, src, _ = meshgen.conduction(n)
    gm = rt.Mesh(m)
    d = rt.Diffusion(gm, rt.default_diffusion_settings(precision=prec))
    d.set_field("gamma", gamma)
    d.set_field("src", src)
    A, b = d.assemble()
    x, it, res, _ = d.solve(RTOL, 2000)
    assert it > 0 and res <= RTOL
    assert host_residual(gm, A, b, x) <= RTOL + 1e-10
