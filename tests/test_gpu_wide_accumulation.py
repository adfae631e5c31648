"""The 32-bit library's wide accumulation around bullseye_grid_batched_facets: the caller's blocks become
FP64 pairs for the call and FP32 values and corrections after it.

Blocks at odd element offsets (cells pairwise unaligned), with gaps, and facets that share cells (the same
block twice, and overlapping blocks): each cell must hold its initial value plus what the facets that
cover it give on disjoint blocks, within the libraries' bars (1e-12 and 1e-5 of the largest value), and cells
outside every block must keep their bits.
"""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_uneven import TOL, _init_struct, _problem

pytestmark = pytest.mark.gpu


def _grid(lib, st, facets, grids, lo, norms):
    from bullseye_gb300.library import check
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rc = lib.bullseye_grid_batched_facets(ctypes.byref(st), ctypes.cast(facets, ctypes.c_void_p), len(facets),
                                          ctypes.c_void_p(0), p(grids), p(lo), p(norms), 1)
    assert rc == 0
    lib.gridding_barrier()
    check(lib)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("layout", ["odd", "same", "overlap"])
def test_blocks(precision, layout, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.abi import BullseyeFacet
    from bullseye_gb300.library import check, load_library
    torch.cuda.set_device(0)
    lib = load_library("GPU", precision)
    p = _problem(precision, 4)
    n = [63, 48, 63] if layout == "odd" else [64, 64, 64]
    size = [p.cube * 4 * k * k for k in n]
    if layout == "odd":  # gaps of 5 and 2 cells
        offs = [1, 1 + size[0] + 5, 1 + size[0] + 5 + size[1] + 2]
    elif layout == "same":
        offs = [3, 3, 3 + size[0]]
    else:  # the second starts inside the first, the third touches the second's end
        offs = [1, 1 + size[0] // 2 + 3, 1 + size[0] // 2 + 3 + size[1]]
    total = max(o + s for o, s in zip(offs, size)) + 7

    def table(at):
        t = (BullseyeFacet * 3)()
        for f in range(3):
            ra, dec = p.facet_centres[f]
            t[f] = BullseyeFacet(float(ra), float(dec), p.cell_x, p.cell_y, n[f], n[f], at[f])
        return t

    apart = [0, size[0], size[0] + size[1]]
    ct = torch.complex64 if precision == "single" else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(5)
    start = torch.randn(total, dtype=ct, device="cuda", generator=gen)
    keep = []
    lib.bullseye_set_device_inputs(1)
    try:
        st, _ = _init_struct(p, torch, keep)
        lib.initLibrary(ctypes.byref(st))
        check(lib)
        norms = torch.zeros(3 * p.cube * 4, dtype=torch.float64, device="cuda")
        alone, alone_lo = (torch.zeros(sum(size), dtype=ct, device="cuda") for _ in range(2))
        grids, lo = start.clone(), torch.zeros(total, dtype=ct, device="cuda")
        torch.cuda.synchronize()  # torch's fills run on its own stream
        _grid(lib, st, table(apart), alone, alone_lo, norms)
        first = norms.cpu().numpy().copy()
        norms.zero_()
        torch.cuda.synchronize()
        _grid(lib, st, table(offs), grids, lo, norms)
        got = (grids.to(torch.complex128) + lo.to(torch.complex128)).cpu().numpy()
        each = (alone.to(torch.complex128) + alone_lo.to(torch.complex128)).cpu().numpy()
        lib.releaseLibrary()
    finally:
        lib.bullseye_set_device_inputs(0)
    want = start.to(torch.complex128).cpu().numpy()
    outside = np.ones(total, bool)
    for f in range(3):
        want[offs[f]:offs[f] + size[f]] += each[apart[f]:apart[f] + size[f]]
        outside[offs[f]:offs[f] + size[f]] = False
    assert outside.any() and np.abs(each).max() > 0
    assert np.array_equal(grids.cpu().numpy()[outside], start.cpu().numpy()[outside])
    assert not lo.cpu().numpy()[outside].any()
    assert np.abs(got - want).max() <= TOL[precision] * np.abs(want).max()
    assert np.allclose(norms.cpu().numpy(), first, rtol=1e-12)
