"""A launch that the runtime refuses leaves the caller's grid as it was.

The number of times is set so high that the Jones inversion asks for more blocks than a grid may have: the
runtime answers with an error on the host and nothing of that launch reaches the GPU.  The workspace and
allocation-free entries must report it with the caller's grid unchanged.
"""
import ctypes

import numpy as np
import pytest

from bullseye_gb300 import synth
from tests.test_zz_no_alloc import _device_struct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entry", ["workspace", "noalloc"])
def test_grid_is_unchanged(entry, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", "single")
    p = synth.small_problem("single", nx=64, n_ant=5, n_times=6, n_chan=2, n_facets=2, jones=True, s=4, os=9, wplanes=4,
                            min_support=5)
    keep = []
    st, arrs = _device_struct(p, torch, keep)
    start = torch.randn(arrs["grid"].shape, dtype=torch.complex64, device="cuda")
    arrs["grid"].copy_(start)
    terms = p.n_antennas * p.n_facets * p.channels  # Jones terms per time
    st.no_timestamps_read = 0xC0000000 * 256 // terms  # 3 x 2^30 blocks of 256; a grid has 2^31 - 1 at most
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    nb = int(lib.bullseye_facet_4_cor_corrections_ws_bytes(ctypes.byref(st)))
    ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
    if entry == "workspace":
        at = ctypes.c_void_p((ws.data_ptr() + 255) // 256 * 256)
        rc = lib.bullseye_facet_4_cor_corrections_ws(ctypes.byref(st), at, nb, stream)
    else:
        rc = lib.bullseye_facet_4_cor_corrections_noalloc(ctypes.byref(st), stream)
    lib.bullseye_clear_error()
    assert rc != 0
    torch.cuda.synchronize()
    assert np.array_equal(arrs["grid"].cpu().numpy(), start.cpu().numpy())
    # the same call with the right number of times goes through
    st.no_timestamps_read = p.n_timestamps
    if entry == "workspace":
        assert lib.bullseye_facet_4_cor_corrections_ws(ctypes.byref(st), at, nb, stream) == 0
    else:
        assert lib.bullseye_facet_4_cor_corrections_noalloc(ctypes.byref(st), stream) == 0
    torch.cuda.synchronize()
    check(lib)
    assert not np.array_equal(arrs["grid"].cpu().numpy(), start.cpu().numpy())
