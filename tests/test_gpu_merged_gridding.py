"""Merged gridding of staged chunks (gridder.cuh find_groups, merge_groups, grid_groups).

Consecutive visibilities that share their footprint corner and one tap row are summed along the other
axis before they touch the grid.  The cases sit where that can go wrong:

* tracks that stand still (groups as long as a chunk, and tracks longer than one), move slowly, move a
  cell or more per sample (groups of one), and run off the grid (invalid records inside a chunk);
* tracks that move mostly along u and mostly along v (the two merge axes);
* supports from 3 to the largest, wider and narrower than a thread's rows, with odd grids;
* one, two and four correlations, records and preparation in place, the per-track kernels.

Everything is compared with the FP64 oracle at the libraries' bars: 1e-12 for the 64-bit library, 1e-5
for the 32-bit one.
"""
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth
from bullseye_gb300.imaging import run_imaging
from tests.golden.cases import cpu_conv
from tests.test_gpu_parity import gpu_libs, oracle_libs, rel  # noqa: F401

pytestmark = pytest.mark.gpu

TOL = {"double": 1e-12, "single": 1e-5}


def _problem(s, wplanes, pace, axis, n_facets, jones, nx=131, n_times=70, n_chan=3):
    """Tracks of 70 samples whose extent along one axis is `pace` of a 1500 m array's and a tenth of that
    along the other (single precision uvw, so that both libraries choose the same cells)."""
    p = synth.small_problem("double", nx=nx, ny=nx - 1, n_ant=6, n_times=n_times, n_chan=n_chan, n_facets=n_facets,
                            jones=jones, s=s, os=9, wplanes=wplanes, min_support=min(5, 2 * s + 1), cell=60.0, seed=17)
    uvw = p.uvw * np.array([pace, 0.1 * pace, 1.0]) if axis == "u" else p.uvw * np.array([0.1 * pace, pace, 1.0])
    return replace(p, uvw=uvw.astype(np.float32).astype(np.float64))


def _check(lib, oracle, p, call, precision):
    from bullseye_gb300.library import check
    q = p.astype(precision)
    r = q.astype("double")
    res = run_imaging(lib, q, call, keep_raw=True, uniform=True, norm_bins=(2 * p.conv_support + 1) ** 2)
    check(lib)
    ref = run_imaging(oracle, r.with_conv(cpu_conv(r)), call, keep_raw=True, uniform=True)
    assert rel(res.raw_grid, ref.raw_grid) <= TOL[precision]
    assert rel(res.normalization, ref.normalization) <= (1e-12 if precision == "double" else 1e-6)
    assert rel(res.sampling, ref.sampling) <= TOL[precision]


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("axis", ["u", "v"])
@pytest.mark.parametrize("pace", [0.0, 0.02, 0.4, 2.5])
@pytest.mark.parametrize("s,wplanes", [(1, 1), (3, 1), (4, 5), (15, 7), (31, 4)])
def test_track_paces(precision, axis, pace, s, wplanes, gpu_libs, oracle_libs):
    p = _problem(s, wplanes, pace, axis, 2, True)
    _check(gpu_libs[precision], oracle_libs["double"], p, "facet_4_cor_corrections", precision)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("call", ["facet_single_pol", "grid_duel_pol", "grid_4_cor"])
@pytest.mark.parametrize("form", ["default", "in_place", "per_track"])
def test_forms_and_correlations(precision, call, form, gpu_libs, oracle_libs):
    lib = gpu_libs[precision]
    lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
    lib.bullseye_set_batched_calls(0 if form == "per_track" else 1)
    try:
        p = _problem(7, 4, 0.1, "v", 2 if call.startswith("facet") else 0, False)
        _check(lib, oracle_libs["double"], p, call, precision)
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_batched_calls(1)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("form", ["records", "in_place", "partial"])
@pytest.mark.parametrize("n_chan,n_facets", [(1, 40), (37, 40)])
def test_work_items_of_several_segments(precision, form, n_chan, n_facets, gpu_libs, oracle_libs):
    """Enough (segment, facet) pairs that a work item takes several segments: tracks that change support
    class, odd channels backwards, rows and channels that are left out, and a record budget that ends
    inside an item."""
    lib = gpu_libs[precision]
    p = _problem(4, 6, 0.05, "u", n_facets, False, nx=65, n_times=41, n_chan=n_chan)
    enabled = np.ones(n_chan, bool)
    enabled[1::5] = False
    p = replace(p, enabled_channels=enabled)
    lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
    lib.bullseye_set_record_budget((1 << 20) if form == "partial" else 0)
    try:
        _check(lib, oracle_libs["double"], p, "facet_4_cor", precision)
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_record_budget(0)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("s", [3, 11, 19])
@pytest.mark.parametrize("n_times", [31, 33, 63, 64, 65, 128, 129])
def test_chunk_edges(precision, s, n_times, gpu_libs, oracle_libs):
    """Segments that end on, one before and one after a staged chunk's end (32 or 64 records), at supports
    whose launches find the next chunk's groups in one warp and at one whose launches do so in every warp."""
    p = _problem(s, 3, 0.05, "u", 2, False, n_times=n_times, n_chan=2)
    _check(gpu_libs[precision], oracle_libs["double"], p, "facet_4_cor", precision)


@pytest.mark.parametrize("call", ["facet_4_cor", "grid_duel_pol"])
def test_compensation_switched_between_calls(call, gpu_libs, oracle_libs):
    """Each call starts from what the one before left, with and without the second word of its cells."""
    lib = gpu_libs["single"]
    p = _problem(5, 4, 0.1, "v", 2 if call.startswith("facet") else 0, False)
    try:
        for on in (1, 0, 1):
            lib.bullseye_set_compensated(on)
            _check(lib, oracle_libs["double"], p, call, "single")
    finally:
        lib.bullseye_set_compensated(1)
