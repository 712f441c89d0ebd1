"""A change of the Chebyshev degree between two solves of one hierarchy: the whole
cycle takes it at once, the levels below the dense operator included. One GCR
iteration on the same system then gives the bits of a flow that had the degree
from the start, and the graph form those of the eager one."""
import numpy as np
import pytest

from openaccel_b200 import meshgen
from openaccel_b200 import runtime as rt

pytestmark = pytest.mark.gpu

TUNING = dict(block_rows=128, block_elements=128, block_assembly=128, gcr_chunk=2, amg_refresh=8)


def flow(prec=rt.OA_PREC_FP64, **kw):
    m = meshgen.cavity(16, perturb=0.2, seed=9)  # 4,913 -> 646 -> 23 rows
    f = rt.Flow(rt.Mesh(m), rt.default_settings(precision=prec, **kw))
    f.set_field("U", meshgen.initial_velocity(m, sigma=0.1, seed=9))
    f.initialize()
    return f


@pytest.mark.parametrize("prec", [rt.OA_PREC_FP64, rt.OA_PREC_MIXED])
@pytest.mark.parametrize("graphs", [0, 1])
def test_degree_changes_for_the_whole_cycle(graphs, prec):
    def one(f):
        f.assemble_momentum(copy=False)
        f.update_mdot()
        f.assemble_pcorr(copy=False)
        return lambda: f.solve("pcorr", 1e-30, 1)[0]

    a, b = flow(prec, use_graphs=graphs), flow(prec, use_graphs=graphs)
    sa, sb = one(a), one(b)
    a.set_tuning(**TUNING, amg_cheb_degree=4)
    x3 = sb()
    b.set_tuning(**TUNING, amg_cheb_degree=4)
    x4 = sa()
    assert np.linalg.norm(x4 - x3) > 1e-6 * np.linalg.norm(x4)
    np.testing.assert_array_equal(sb(), x4)


def test_degree_change_in_the_iteration_graph():
    out = []
    for graphs in (1, 2):
        f = flow(use_graphs=graphs)
        st = f.simple_iterate(3)
        f.set_tuning(**TUNING, amg_cheb_degree=4)
        st += f.simple_iterate(3)
        out.append((f.get_field("p"), [s["pc_iters"] for s in st]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
