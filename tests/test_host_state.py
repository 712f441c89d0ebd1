"""The library's host side on the stand-in for the CUDA runtime (fake_cudart.cpp):
what it captures again and what it launches, without a GPU."""
import os
import subprocess
import sys

from .test_memory_limit import ROOT, fake  # noqa: F401

HEAD = r"""
import ctypes as C
from openaccel_b200 import meshgen, runtime as rt
fake = C.CDLL(None)
"""


def run(fake, code):  # noqa: F811
    r = subprocess.run([sys.executable, "-c", HEAD + code], cwd=ROOT, capture_output=True, text=True,
                       env={**os.environ, "LD_PRELOAD": fake, "PYTHONPATH": ROOT}, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]


def test_new_segments_are_captured(fake):  # noqa: F811
    """Captured solver chunks hold the addresses of the segments' buffers: setting
    the reference nodes again frees those, so the next solve has to capture."""
    run(fake, r"""
b = meshgen.batch_cavities(sizes=[4, 6], seed=7)
f = rt.Flow(rt.Mesh(b.mesh), rt.default_settings(ref_node=-1, use_graphs=1))
f.initialize()
f.assemble_pcorr()
captures = []
for nodes in (None, b.ref_nodes, None, b.ref_nodes):
    if nodes is not None:
        f.set_reference_nodes(nodes)
    f.solve("pcorr", 1e-8, 4)
    captures.append(fake.fake_captures())
assert captures == [1, 2, 2, 3], captures
""")


def test_solve_without_room_for_a_large_cluster(fake):  # noqa: F811
    """The power iteration of small levels takes a cluster of more than the
    portable 8 blocks only where one can be placed."""
    run(fake, r"""
fake.fake_max_cluster(8)
f = rt.Flow(rt.Mesh(meshgen.cavity(12)), rt.default_settings())
f.initialize()
f.assemble_pcorr()
f.solve("pcorr", 1e-8, 4)
""")
