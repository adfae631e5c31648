"""Cells that no visibility touches keep what the caller's grid holds, and an infinity stays one.

The 32-bit library's wide accumulation converts whole grids around a call.  Infinities, NaNs, zeros of either
sign, denormals and the largest values lie in cells that a first call showed to be left alone, and an infinity
in one that is not: for bullseye_grid_batched_facets the untouched words must come back bit for bit (a NaN as a
NaN) with no second word, for the workspace and allocation-free entries and the library's own grids as the
values that they are.
"""
import ctypes

import numpy as np
import pytest

from bullseye_gb300 import synth
from tests.test_gpu_uneven import _init_struct, _problem
from tests.test_gpu_wide_accumulation import _grid
from tests.test_zz_no_alloc import _device_struct

pytestmark = pytest.mark.gpu

SPECIAL = np.array([np.inf, -np.inf, np.nan, -0.0, 0.0, 1e-42, 3.4028234e38, -3.4028234e38, 1.5], np.float32)


def _plant(zero_cells, shape):
    """A complex64 grid with special components in the cells that are left alone."""
    r = np.random.default_rng(3)
    out = np.zeros(shape, np.complex64)
    at = np.flatnonzero(zero_cells.reshape(-1))
    assert at.size > 200
    out.view(np.float32).reshape(-1, 2)[at] = SPECIAL[r.integers(0, SPECIAL.size, (at.size, 2))]
    return out


def _words(x):
    return np.ascontiguousarray(x).reshape(-1).view(np.float32)


def _same(got, want, bits):
    g, w = _words(got), _words(want)
    nan = np.isnan(w)
    assert np.isnan(g[nan]).all()
    if bits:
        assert np.array_equal(g[~nan].view(np.int32), w[~nan].view(np.int32))
    else:
        assert np.array_equal(g[~nan], w[~nan])


@pytest.mark.parametrize("n_times", [10, 60])  # few and many visibilities for the blocks' cells: either form
@pytest.mark.parametrize("wplanes", [1, 4])
def test_caller_blocks(wplanes, n_times, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.abi import BullseyeFacet
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", "single")
    p = synth.small_problem("single", nx=96, n_ant=7, n_times=n_times, n_chan=3, n_facets=3, jones=False, s=4, os=9,
                            wplanes=wplanes, min_support=5 if wplanes > 1 else None, seed=31)
    n = 90
    size = p.cube * 4 * n * n
    table = (BullseyeFacet * 2)()
    for f in range(2):
        ra, dec = p.facet_centres[f]
        table[f] = BullseyeFacet(float(ra), float(dec), p.cell_x, p.cell_y, n, n, f * size)
    keep = []
    lib.bullseye_set_device_inputs(1)
    try:
        st, _ = _init_struct(p, torch, keep)
        lib.initLibrary(ctypes.byref(st))
        check(lib)

        def run(start):
            grids = torch.as_tensor(start, device="cuda")
            lo = torch.zeros(2 * size, dtype=torch.complex64, device="cuda")
            norms = torch.zeros(2 * p.cube * 4, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()  # torch's fills run on its own stream
            _grid(lib, st, table, grids, lo, norms)
            return grids.cpu().numpy(), lo.cpu().numpy()

        first, first_lo = run(np.zeros(2 * size, np.complex64))
        alone = (_words(first).reshape(-1, 2) == 0).all(1) & (_words(first_lo).reshape(-1, 2) == 0).all(1)
        start = _plant(alone, 2 * size)
        hit = np.flatnonzero(~alone)[::7]
        start[hit] = np.inf + 1j
        got, got_lo = run(start)
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_device_inputs(0)
    _same(got[alone], start[alone], bits=True)
    assert not _words(got_lo[alone]).any()
    assert np.isposinf(got[hit].real).all()
    assert not got_lo[hit].real.any()


@pytest.mark.parametrize("entry", ["workspace", "noalloc"])
@pytest.mark.parametrize("wplanes", [1, 4])
def test_caller_grid(entry, wplanes, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", "single")
    p = synth.small_problem("single", nx=96, n_ant=7, n_times=10, n_chan=3, n_facets=3, jones=True, s=4, os=9,
                            wplanes=wplanes, min_support=5 if wplanes > 1 else None)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    keep = []

    def run(start):
        st, arrs = _device_struct(p, torch, keep)
        arrs["grid"].copy_(torch.as_tensor(start))
        if entry == "workspace":
            nb = int(lib.bullseye_facet_4_cor_corrections_ws_bytes(ctypes.byref(st)))
            ws = torch.empty(nb + 256, dtype=torch.uint8, device="cuda")
            at = ctypes.c_void_p((ws.data_ptr() + 255) // 256 * 256)
            assert lib.bullseye_facet_4_cor_corrections_ws(ctypes.byref(st), at, nb, stream) == 0
        else:
            assert lib.bullseye_facet_4_cor_corrections_noalloc(ctypes.byref(st), stream) == 0
        torch.cuda.synchronize()
        check(lib)
        return arrs["grid"].cpu().numpy()

    shape = (p.n_facets, p.cube, 4, p.ny, p.nx)
    first = run(np.zeros(shape, np.complex64))
    alone = (first == 0).reshape(-1)
    start = _plant(alone, shape)
    got = run(start).reshape(-1)
    _same(got[alone], start.reshape(-1)[alone], bits=False)


def test_library_grid(gpu_required, built_libraries):
    """Initial contents of the library's own grids, through a call and its copy-back."""
    import torch
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", "single")
    p = _problem("single", 4)
    keep = []
    lib.bullseye_set_device_inputs(1)
    try:
        def run(start):
            st, _ = _init_struct(p, torch, keep)
            st.is_final_data_chunk = True
            keep[-1]["grid"][...] = start
            lib.initLibrary(ctypes.byref(st))
            assert lib.bullseye_grid_batched(ctypes.byref(st), 1, 0) == 0
            lib.gridding_barrier()
            check(lib)
            lib.releaseLibrary()
            return keep[-1]["grid"].reshape(-1).copy()

        alone = run(0) == 0
        start = _plant(alone, keep[-1]["grid"].shape)
        got = run(start)
    finally:
        lib.bullseye_set_device_inputs(0)
    _same(got[alone], start.reshape(-1)[alone], bits=False)
