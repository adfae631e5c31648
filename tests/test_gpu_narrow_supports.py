"""Supports that one warp owns with two rows per thread (full supports of 3, 5 and 7) and the next ones past it.

Slow, fast and irregular tracks, prepared in place, from records and through the workspace entry, against the FP64
oracle: 1e-12 in the 64-bit library, 1e-5 in the 32-bit one.
"""
import numpy as np
import pytest

from bullseye_gb300.imaging import run_imaging
from tests.golden.cases import cpu_conv
from tests.test_gpu_merged_gridding import _problem
from tests.test_gpu_parity import gpu_libs, oracle_libs, rel  # noqa: F401

pytestmark = pytest.mark.gpu

TOL = {"double": 1e-12, "single": 1e-5}


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("form", ["records", "in_place", "workspace"])
@pytest.mark.parametrize("pace", [0.02, 2.5])
@pytest.mark.parametrize("s,wplanes", [(1, 1), (2, 1), (3, 1), (3, 4), (4, 1)])
def test_forms(precision, form, pace, s, wplanes, gpu_libs, oracle_libs):
    from bullseye_gb300.library import check
    lib = gpu_libs[precision]
    p = _problem(s, wplanes, pace, "u", 2, True).astype(precision)
    r = p.astype("double")
    ref = run_imaging(oracle_libs["double"], r.with_conv(cpu_conv(r)), "facet_4_cor_corrections", keep_raw=True)
    if form == "workspace":
        import torch
        from bullseye_gb300 import autograd
        g = autograd.FacetGeometry.from_problem(p)
        grids, norm = autograd.facet_grid(g, torch.as_tensor(np.ascontiguousarray(p.vis[g.order]), device="cuda"),
                                          torch.as_tensor(np.ascontiguousarray(p.jones), device="cuda"))
        grid, norm = grids.cpu().numpy(), norm.cpu().numpy()
    else:
        lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
        try:
            res = run_imaging(lib, p, "facet_4_cor_corrections", keep_raw=True, repack=True,
                              norm_bins=(2 * p.conv_support + 1) ** 2)
            check(lib)
        finally:
            lib.bullseye_set_visibility_records(1)
        grid, norm = res.raw_grid, res.normalization
    assert rel(grid, ref.raw_grid) <= TOL[precision]
    assert rel(norm, ref.normalization) <= (1e-12 if precision == "double" else 1e-6)
