"""Green-Gauss gradients from summed edge areas (shifted interpolation on block
meshes) against the oracle's loop over integration points, at node counts around
the kernel's groups of 32 nodes and blocks of 256, on skewed meshes, and the
velocity correction fused with the pressure gradient inside an outer iteration.

Both sides are FP64 sums of the same terms in another order: at most 24 terms
per component, each rounded once, so 1e-12 of the field's norm leaves three
decades."""
import numpy as np
import pytest

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


# nodes: 8, 12, 32, 36, 64, 66, 252, 256, 264, 1,001
SHAPES = [(1, 1, 1), (2, 1, 1), (3, 3, 1), (8, 1, 1), (3, 3, 3), (10, 2, 1), (5, 5, 6), (7, 7, 3), (10, 7, 2),
          (12, 10, 6)]


@pytest.mark.parametrize("shape", SHAPES)
def test_gradients(oracle_mod, shape):
    m = meshgen.cavity(shape, perturb=0.15, seed=4)
    r = np.random.default_rng(8)
    U, p = r.normal(0, 1, 3 * m.nn), r.normal(0, 1, m.nn)
    oc = oracle_mod.FlowCase(m, oracle_mod.default_settings(), U0=U.reshape(-1, 3))
    oc.field("p")[:] = p
    gf = rt.Flow(rt.Mesh(m), rt.default_settings())
    gf.set_field("U", U)
    gf.set_field("p", p)
    for _ in range(2):  # the second from a non-zero old gradient
        oc.update_grad_p(), oc.update_grad_u()
        gf.update_gradient("p"), gf.update_gradient("U")
    assert rel(gf.get_field("gradP"), oc.field("gradP")) < 1e-12
    assert rel(gf.get_field("gradU"), oc.field("gradU")) < 1e-12


@pytest.mark.parametrize("du_mode", [0, 1])
@pytest.mark.parametrize("shape", [(3, 3, 1), (5, 5, 6), (10, 7, 2)])
def test_velocity_correction(oracle_mod, shape, du_mode):
    kw = dict(mom_rtol=1e-13, pc_rtol=1e-13, du_mode=du_mode)
    m = meshgen.cavity(shape, perturb=0.15, seed=4)
    U0 = meshgen.initial_velocity(m, sigma=0.1, seed=4)
    oc = oracle_mod.FlowCase(m, oracle_mod.default_settings(**kw), U0=U0)
    gf = rt.Flow(rt.Mesh(m), rt.default_settings(**kw))
    gf.set_field("U", U0)
    oc.initialize()
    gf.initialize()
    for _ in range(3):
        oc.simple_iteration()
    gf.simple_iterate(3)
    for k in ("U", "gradP", "gradU"):
        assert rel(gf.get_field(k), oc.field(k)) < 1e-10, k


# nodes: 2,940 and 3,000 (the velocity gradient takes the edge form from there),
# 3,072 (whole blocks), 3,150 (78 past a block, 14 past a group), 3,328, 3,375
@pytest.mark.parametrize("shape", [(13, 13, 14), (14, 19, 9), (15, 15, 11), (13, 14, 14), (12, 15, 15), (14, 14, 14)])
def test_gradients_around_the_edge_forms_lowest_size(oracle_mod, shape):
    test_gradients(oracle_mod, shape)
