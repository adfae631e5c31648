"""Both forms in which bullseye_grid_batched_facets accumulates into the caller's cells (32-bit library).

Calls whose cells are few for their visibilities take the wide form, others the pair form: facets of 48^2 and of
192^2 cells lie on either side (4 and 68 cells per pair of visibility and facet; the line is at 14), 96^2 just
past it.  Blocks start at odd offsets, with gaps or one on top of another, over random initial values.  Each cell must
hold its initial value plus what the FP64 oracle grids for the facets that cover it, within 1e-5 of the largest
value, and cells outside every block their bits.
"""
import ctypes

import numpy as np
import pytest

from bullseye_gb300 import synth
from bullseye_gb300.imaging import run_imaging
from tests.golden.cases import cpu_conv
from tests.test_gpu_parity import gpu_libs, oracle_libs  # noqa: F401
from tests.test_gpu_uneven import _init_struct
from tests.test_gpu_wide_accumulation import _grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["records", "in_place"])
@pytest.mark.parametrize("wplanes", [1, 5])
@pytest.mark.parametrize("layout", ["gaps", "same"])
@pytest.mark.parametrize("n", [48, 96, 192])
def test_forms(n, layout, wplanes, form, gpu_libs, oracle_libs):
    import torch
    from bullseye_gb300.abi import BullseyeFacet
    from bullseye_gb300.library import check
    lib = gpu_libs["single"]
    p = synth.small_problem("single", nx=n, n_ant=10, n_times=12, n_chan=4, n_facets=3, s=8, os=7, wplanes=wplanes,
                            min_support=9 if wplanes > 1 else None, cell=60.0 * 96 / n)
    r = p.astype("double")
    ref = run_imaging(oracle_libs["double"], r.with_conv(cpu_conv(r)), "facet_4_cor", keep_raw=True).raw_grid
    size = 4 * n * n
    offs = [1, 1 + size + 5, 1 + 2 * size + 7] if layout == "gaps" else [3, 3, 3 + size]
    total = offs[-1] + size + 7
    facets = (BullseyeFacet * 3)()
    for f in range(3):
        ra, dec = p.facet_centres[f]
        facets[f] = BullseyeFacet(float(ra), float(dec), p.cell_x, p.cell_y, n, n, offs[f])
    gen = torch.Generator(device="cuda").manual_seed(5)
    start = torch.randn(total, dtype=torch.complex64, device="cuda", generator=gen) * float(np.abs(ref).max())
    grids, lo = start.clone(), torch.zeros_like(start)
    norms = torch.zeros(12, dtype=torch.float64, device="cuda")
    keep = []
    lib.bullseye_set_device_inputs(1)
    lib.bullseye_set_visibility_records(0 if form == "in_place" else 1)
    try:
        st, _ = _init_struct(p, torch, keep)
        lib.initLibrary(ctypes.byref(st))
        check(lib)
        torch.cuda.synchronize()  # torch's fills run on its own stream
        for _ in range(2):  # the second call adds the same once more
            _grid(lib, st, facets, grids, lo, norms)
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_visibility_records(1)
        lib.bullseye_set_device_inputs(0)
    got = (grids.to(torch.complex128) + lo.to(torch.complex128)).cpu().numpy()
    want = start.cpu().numpy().astype(np.complex128)
    outside = np.ones(total, bool)
    for f in range(3):
        want[offs[f]:offs[f] + size] += 2 * ref[f].reshape(-1)
        outside[offs[f]:offs[f] + size] = False
    assert np.abs(ref).max() > 0
    assert np.array_equal(grids.cpu().numpy()[outside], start.cpu().numpy()[outside])
    assert not lo.cpu().numpy()[outside].any()
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    # the second words are corrections (each addition rounds off 6e-8 of a cell)
    assert np.abs(lo.cpu().numpy()).max() <= 1e-4 * np.abs(want).max()
