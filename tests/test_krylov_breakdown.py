"""Breakdowns of the Krylov iterations.

A kernel of many blocks in which one block sets the solver's done flag must take
its own test of that flag as one decision per block: the blocks then add up
partials together, and a block in which some warps have left adds up values
that were never written. No run can show that reliably, so the kernels' source
is checked here on the CPU; on the GPU a system that breaks down in its first
iteration has to be reported as such, with the zero iterate, however often it
is solved."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from openaccel_b200 import runtime as rt

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def kernels(path):
    """(name, body) of every __global__ function of a source file."""
    src = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"__global__[^;{]*?\bk_(\w+)\s*\([^;{]*\)\s*\{", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield "k_" + m.group(1), src[m.end():i]


def test_flag_set_inside_a_grid_is_tested_once_per_block():
    found = dict(kernels(os.path.join(ROOT, "openaccel_b200", "csrc", "oa_krylov.cu")))
    assert {"k_s_update", "k_gcr_update", "k_spmv", "k_segments"} <= set(found)
    writers = [n for n, body in found.items() if re.search(r"sc->done\s*=[^=]", body) and "blockIdx.x == 0" in body]
    assert sorted(writers) == ["k_gcr_update", "k_s_update"]
    for n in writers:
        assert not re.search(r"if\s*\(sc->done\)", found[n]), n
        assert re.match(r"\s*if \(block_done\(sc\)\) return;", found[n]), n


@pytest.mark.gpu
@pytest.mark.parametrize("pairs", [1, 16, 129, 65536])
def test_breakdown_is_reported(pairs):
    """Blocks [[1, 1], [-3, 1]] with b = (1, 1): A M^-1 b = (2, -2), so rh.v is
    exactly zero in every summation order (whole numbers)."""
    import torch

    n = 2 * pairs
    dev = lambda a: torch.from_numpy(a).cuda()
    first = np.arange(n, dtype=np.int32) // 2 * 2
    rp = dev(np.arange(0, 2 * n + 1, 2, dtype=np.int32))
    cols = dev(np.stack([first, first + 1], axis=1).ravel())
    diag = dev(np.arange(n, dtype=np.int32) % 2)
    A = dev(np.tile([1.0, 1.0, -3.0, 1.0], pairs))
    b = dev(np.ones(n))
    L = rt.lib()
    for _ in range(20):
        x = torch.full((n,), 7.0, dtype=torch.float64, device="cuda")
        it, res = C.c_int(-1), C.c_double(-1.0)
        st = L.oa_pcorr_solve_static(n, rp.data_ptr(), cols.data_ptr(), diag.data_ptr(), A.data_ptr(), b.data_ptr(),
                                     x.data_ptr(), 1e-10, 100, C.byref(it), C.byref(res),
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 5 and b"breakdown" in L.oa_last_error()
        assert it.value == 0 and res.value == 1.0
        assert not x.any()
