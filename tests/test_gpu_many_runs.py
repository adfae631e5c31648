"""Schedules of many short runs: rows in time order, so that neighbouring rows change their support class.

The runs are bucketed by class in blocks of 4,096; the cases hold fewer than one block, a few more than one, and
several blocks (the row order is the data's, without a baseline sort).  The batched exports and the workspace
entry must give the FP64 oracle's grids: 1e-12 in the 64-bit library, 1e-5 in the 32-bit one.
"""
import ctypes
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth
from bullseye_gb300.imaging import run_imaging
from tests.golden.cases import cpu_conv
from tests.test_gpu_parity import gpu_libs, oracle_libs, rel  # noqa: F401
from tests.test_gpu_uneven import _init_struct

pytestmark = pytest.mark.gpu

TOL = {"double": 1e-12, "single": 1e-5}


def _problem(precision, n_times, n_chan, call_jones):
    p = synth.small_problem("double", nx=96, ny=95, n_ant=11, n_times=n_times, n_chan=n_chan, n_facets=2, jones=call_jones,
                            s=13, os=5, wplanes=24, min_support=13, cell=30.0)
    p.uvw = p.uvw.astype(np.float32).astype(np.float64)  # both libraries choose the same cells
    return p.astype(precision)


def _oracle(oracle_libs, p, call):
    r = p.astype("double")
    return run_imaging(oracle_libs["double"], r.with_conv(cpu_conv(r)), call, keep_raw=True)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("n_times,n_chan", [(3, 2), (30, 24), (60, 24)])
def test_time_ordered_rows(precision, n_times, n_chan, gpu_libs, oracle_libs):
    import torch
    from bullseye_gb300.library import check
    lib = gpu_libs[precision]
    p = _problem(precision, n_times, n_chan, False)
    # device rows as they come: one baseline number for all (unused by this call) leaves their order
    q = replace(p, antenna1=np.zeros_like(p.antenna1), antenna2=np.ones_like(p.antenna2))
    keep = []
    other = [(ctypes.c_int * 64)() for _ in range(4)]
    items, ms = (ctypes.c_int * 64)(), (ctypes.c_float * 64)()
    width = other[0]
    lib.bullseye_set_device_inputs(1)
    lib.bullseye_set_batched_profiling(1)
    try:
        st, _ = _init_struct(q, torch, keep)
        st.baseline_starting_indexes = None
        st.is_final_data_chunk = True
        lib.initLibrary(ctypes.byref(st))
        assert lib.bullseye_grid_batched(ctypes.byref(st), 1, 0) == 0
        lib.gridding_barrier()
        check(lib)
        k = lib.bullseye_batched_profile(*other, items, ms, 64)
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_batched_profiling(0)
        lib.bullseye_set_device_inputs(0)
    grid = keep[0]["grid"]
    runs = sum(items[i] for i in range(k) if width[i] > 0) // 2  # facets
    assert sum(items[i] > 0 for i in range(k)) >= 2  # classes
    assert n_times < 60 or runs > 2 * 4096
    assert rel(grid, _oracle(oracle_libs, p, "facet_4_cor").raw_grid) <= TOL[precision]


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("n_times,n_chan", [(3, 2), (60, 24)])
def test_workspace_entry(precision, n_times, n_chan, gpu_libs, oracle_libs):
    import torch
    from bullseye_gb300 import autograd
    p = _problem(precision, n_times, n_chan, True)
    g = autograd.FacetGeometry.from_problem(p)
    back = torch.as_tensor(np.argsort(g.order), device="cuda")
    for k in ("uvw", "wt", "fl", "fr", "field", "spw", "a1", "a2", "tid"):
        a = g.arrays[k]
        g.arrays[k] = (a.view(torch.int32)[back].view(torch.uint32) if a.dtype == torch.uint32 else a[back]).contiguous()
    g.arrays["starts"] = None  # fixed row segments
    vis = torch.as_tensor(np.ascontiguousarray(p.vis), device="cuda")
    grids, _ = autograd.facet_grid(g, vis, torch.as_tensor(np.ascontiguousarray(p.jones), device="cuda"))
    assert rel(grids.cpu().numpy(), _oracle(oracle_libs, p, "facet_4_cor_corrections").raw_grid) <= TOL[precision]
