"""Work items of several segments in more than one support class.

Tracks change their class along the way, so that an item's segments are separated by rows of other classes; odd
channels are taken last to first; 21 times give segments that may not stay together (their first groups
break), 63 times segments that may.  Records, preparation in place and a record budget that ends inside an item, and
facets that leave rows out (two masks, facets alternating).  The FP64 oracle is the reference: 1e-12 in the 64-bit
library, 1e-5 in the 32-bit one.
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
FACETS = 48
_REF = {}


def _problem(n_times):
    p = synth.small_problem("double", nx=72, ny=71, n_ant=8, n_times=n_times, n_chan=40, n_facets=FACETS, s=13, os=5,
                            wplanes=24, min_support=14, cell=60.0, seed=17)
    return replace(p, uvw=(p.uvw * np.array([0.1, 0.02, 1.0])).astype(np.float32).astype(np.float64))


def _oracle(oracle_libs, p, key):
    if key not in _REF:
        r = p.astype("single").astype("double")
        _REF[key] = run_imaging(oracle_libs["double"], r.with_conv(cpu_conv(r)), "facet_4_cor", keep_raw=True)
    return _REF[key]


def _classes_with_long_items(lib):
    """Classes of the last profiled call whose items take two segments or more: at least sixteen (segment,
    facet) pairs per CTA of a launch that fills the register files."""
    width, nc, J, wide, items = ((ctypes.c_int * 64)() for _ in range(5))
    k = lib.bullseye_batched_profile(width, nc, J, wide, items, (ctypes.c_float * 64)(), 64)
    n = 0
    for i in range(k):
        if width[i] == 0 or nc[i] != 4:
            continue
        W = width[i]
        owners = (W + 31) // 32 * 32 if wide[i] & 1 else W
        threads = max(32, (owners * ((W + J[i] - 1) // J[i]) + 31) // 32 * 32)
        n += items[i] >= 16 * 152 * (65536 // (threads * (wide[i] >> 1)))
    return n


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("form", ["records", "in_place", "partial"])
@pytest.mark.parametrize("n_times", [21, 63])
def test_forms(precision, form, n_times, gpu_libs, oracle_libs):
    from bullseye_gb300.library import check
    lib = gpu_libs[precision]
    p = _problem(n_times).astype("single").astype(precision)
    lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
    lib.bullseye_set_record_budget((1 << 24) if form == "partial" else 0)
    lib.bullseye_set_batched_profiling(1)
    try:
        res = run_imaging(lib, p, "facet_4_cor", keep_raw=True, repack=True, norm_bins=(2 * p.conv_support + 1) ** 2)
        check(lib)
        assert _classes_with_long_items(lib) >= 2
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_record_budget(0)
        lib.bullseye_set_batched_profiling(0)
    ref = _oracle(oracle_libs, _problem(n_times), n_times)
    assert rel(res.raw_grid, ref.raw_grid) <= TOL[precision]
    assert rel(res.normalization, ref.normalization) <= (1e-12 if precision == "double" else 1e-6)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("form", ["records", "in_place"])
def test_row_masks(precision, form, gpu_libs, oracle_libs):
    import torch
    from bullseye_gb300.abi import BullseyeFacet
    from bullseye_gb300.library import check
    lib = gpu_libs[precision]
    p = _problem(21).astype("single").astype(precision)
    r = np.random.default_rng(9)
    # the first facet of a pair misses the ends of most tracks, the second single rows and whole baselines
    ends = (p.timestamp_ids >= 4) & (p.timestamp_ids < 17) | (p.antenna1 == 0)
    masks = [ends, (r.random(p.rows) >= 0.3) & (p.antenna2 != 5)]
    size = 4 * p.ny * p.nx
    facets = (BullseyeFacet * FACETS)()
    for f in range(FACETS):
        ra, dec = p.facet_centres[f]
        facets[f] = BullseyeFacet(float(ra), float(dec), p.cell_x, p.cell_y, p.nx, p.ny, f * size)
    keep = []
    ct = torch.complex64 if precision == "single" else torch.complex128
    lib.bullseye_set_device_inputs(1)
    lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
    try:
        st, order = _init_struct(p, torch, keep)
        lib.initLibrary(ctypes.byref(st))
        check(lib)
        mask = torch.as_tensor(np.stack([masks[f % 2][order] for f in range(FACETS)]).astype(np.uint8), device="cuda")
        grids = torch.zeros(FACETS * size, dtype=ct, device="cuda")
        lo = torch.zeros_like(grids)
        norms = torch.zeros(FACETS * 4, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()  # torch's fills run on its own stream
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        assert lib.bullseye_grid_batched_facets(ctypes.byref(st), ctypes.cast(facets, ctypes.c_void_p), FACETS, ptr(mask),
                                                ptr(grids), ptr(lo) if precision == "single" else ctypes.c_void_p(0),
                                                ptr(norms), 1) == 0
        lib.gridding_barrier()
        check(lib)
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_device_inputs(0)
    got = (grids.to(torch.complex128) + lo.to(torch.complex128)).cpu().numpy().reshape(FACETS, 1, 4, p.ny, p.nx)
    got_norm = norms.cpu().numpy().reshape(FACETS, 1, 4)
    for half in range(2):
        q = _problem(21)
        q = replace(q, flagged_rows=q.flagged_rows | ~masks[half])
        ref = _oracle(oracle_libs, q, ("mask", half))
        assert rel(got[half::2], ref.raw_grid[half::2]) <= TOL[precision]
        assert rel(got_norm[half::2], ref.normalization[half::2]) <= (1e-12 if precision == "double" else 1e-6)
