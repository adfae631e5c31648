"""The layout of a support class is timed on the first call that has records to time it on.

A call without records (switched off here; a call of little work has none either) runs one fixed layout, so it
decides nothing: the next call with records must time the candidates.  Timing launches count, a graph replay's
launches are those of the call alone, so the difference between two equal calls shows whether there were any.
A full support of 29 is used by no other test.
"""
import ctypes

import pytest

from bullseye_gb300 import synth
from tests.test_gpu_uneven import _init_struct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["double", "single"])
def test_timed_after_a_call_without_records(precision, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", precision)
    p = synth.small_problem(precision, nx=128, n_ant=12, n_times=20, n_chan=8, n_facets=2, s=14, os=5)
    keep = []
    lib.bullseye_set_device_inputs(1)
    try:
        st, _ = _init_struct(p, torch, keep)
        lib.initLibrary(ctypes.byref(st))

        def launches():
            before = lib.bullseye_kernel_launches()
            assert lib.bullseye_grid_batched(ctypes.byref(st), 1, 0) == 0
            lib.gridding_barrier()
            check(lib)
            return lib.bullseye_kernel_launches() - before

        lib.bullseye_set_visibility_records(0)
        launches()
        lib.bullseye_set_visibility_records(1)
        first, second = launches(), launches()
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_device_inputs(0)
    # the first one also runs its schedule once by itself (6 launches); two launches per layout, two layouts at least
    assert first - second >= 6 + 4
