"""FP64 momentum assembly on both sides of the sizes at which its kernel takes
another register budget (100,000 rows of a block mesh, 312,500 with unshifted
interpolation), against the oracle: each matrix entry is a sum of at most 24
rounded terms, so 1e-12 of the norm leaves three decades."""
import numpy as np
import pytest

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# 99,452, 100,050 and 314,432 rows
@pytest.mark.parametrize("shape,kw", [((45, 45, 46), {}), ((45, 74, 28), {}), ((45, 74, 28), dict(du_mode=1)),
                                      ((45, 74, 28), dict(hr=1)), ((45, 74, 28), dict(u_shifted=0)),
                                      ((67, 67, 67), dict(u_shifted=0)),
                                      ((67, 67, 67), dict(u_shifted=0, du_mode=1))])
def test_momentum_assembly(oracle_mod, shape, kw):
    m = meshgen.cavity(shape, perturb=0.2, seed=4)
    U0 = meshgen.initial_velocity(m, sigma=0.1, seed=4)
    oc = oracle_mod.FlowCase(m, oracle_mod.default_settings(**kw), U0=U0)
    gf = rt.Flow(rt.Mesh(m), rt.default_settings(**kw))
    gf.set_field("U", U0)
    r = np.random.default_rng(5)
    state = {"p": r.normal(0, 1, m.nn), "gradP": r.normal(0, 1, 3 * m.nn), "gradU": r.normal(0, 1, 9 * m.nn),
             "mDot": r.normal(0, 0.01, 12 * m.ne), "div": r.normal(0, 1e-3, m.nn)}
    if "hr" in kw:
        state["betaU"] = r.uniform(0, 1, 3 * m.nn)
    for k, v in state.items():
        oc.field(k)[:] = v
        gf.set_field(k, v)
    A, b = gf.assemble_momentum()
    A_o, b_o = oc.assemble_momentum()
    assert rel(A, A_o) < 1e-12
    assert rel(b, b_o) < 1e-12
