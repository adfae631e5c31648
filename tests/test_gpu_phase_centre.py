"""A facet at the phase centre is gridded, degridded and predicted with exactly the identity transform.

Samples with v = 0 and w of both signs lie on a cell boundary of a 1-D kernel: a transform that is off by one
rounding error (1e-17) moves them to the next cell.  The kernel table holds random values, so that the next
cell's taps differ.  The regular export, the workspace and allocation-free entries, the adjoint and the
prediction must all take the oracle's cells (1e-12 in the 64-bit library, 1e-5 in the 32-bit one).
"""
import ctypes
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth
from bullseye_gb300.imaging import run_imaging
from tests.golden.cases import cpu_conv
from tests.test_gpu_parity import gpu_libs, oracle_libs, rel  # noqa: F401
from tests.test_zz_no_alloc import _device_struct

pytestmark = pytest.mark.gpu

TOL = {"double": 1e-12, "single": 1e-5}


def _problem(precision, dec):
    p = synth.small_problem("double", nx=96, ny=95, n_ant=6, n_times=9, n_chan=3, n_facets=1, jones=True, s=4, os=7)
    uvw = p.uvw * np.array([1.0, 0.0, 1.0])
    uvw[::2, 2] *= -1
    assert (uvw[:, 2] > 0).any() and (uvw[:, 2] < 0).any()
    conv = np.random.default_rng(2).uniform(0.2, 1.0, p.conv.shape).astype(np.float32).astype(np.float64)
    centre = (0.0, float(np.float32(dec * 3600.0)))
    p = replace(p, uvw=uvw.astype(np.float32).astype(np.float64), conv=conv, phase_centre=centre,
                facet_centres=np.array([centre]))
    return p.astype(precision)


def _oracle(oracle_libs, p):
    r = p.astype("double")
    return run_imaging(oracle_libs["double"], r.with_conv(cpu_conv(r)), "facet_4_cor_corrections", keep_raw=True)


@pytest.mark.parametrize("dec", [-40.0, -30.0, 12.5, 61.0])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_gridding(precision, dec, gpu_libs, oracle_libs):
    import torch
    from bullseye_gb300 import autograd
    from bullseye_gb300.library import check
    p = _problem(precision, dec)
    ref = _oracle(oracle_libs, p)
    lib = gpu_libs[precision]
    res = run_imaging(lib, p, "facet_4_cor_corrections", repack=True, keep_raw=True, norm_bins=(2 * p.conv_support + 1) ** 2)
    check(lib)
    assert rel(res.raw_grid, ref.raw_grid) <= TOL[precision]
    geom = autograd.FacetGeometry.from_problem(p)
    vis = torch.as_tensor(np.ascontiguousarray(p.vis[geom.order]), device="cuda")
    grids, _ = autograd.facet_grid(geom, vis, torch.as_tensor(np.ascontiguousarray(p.jones), device="cuda"))
    assert rel(grids.cpu().numpy(), ref.raw_grid) <= TOL[precision]
    if precision == "single":
        st, arrs = _device_struct(p, torch, [])
        assert lib.bullseye_facet_4_cor_corrections_noalloc(
            ctypes.byref(st), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        check(lib)
        assert rel(arrs["grid"].cpu().numpy(), ref.raw_grid) <= TOL[precision]


@pytest.mark.parametrize("dec", [-40.0, -30.0, 12.5, 61.0])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_degridding(precision, dec, gpu_libs):
    import torch
    from bullseye_gb300 import autograd
    p = _problem(precision, dec)
    geom = autograd.FacetGeometry.from_problem(p)
    r = np.random.default_rng(8)
    shape = (1, 1, 4, p.ny, p.nx)
    cd = np.complex64 if precision == "single" else np.complex128
    grid = (r.normal(size=shape) + 1j * r.normal(size=shape)).astype(cd)
    got = autograd.predict(geom, torch.as_tensor(grid, device="cuda"), from_grid=True).cpu().numpy()
    back, _ = autograd.grid_adjoint(geom, torch.zeros(geom.order.size, p.channels, 4, dtype=torch.as_tensor(grid).dtype,
                                                      device="cuda"), None, torch.as_tensor(grid, device="cuda"))
    back = back.cpu().numpy()
    s, os, W = p.conv_support, p.conv_oversample, 2 * p.conv_support + 1
    rad = float(np.float32(np.pi / (180.0 * 3600.0)))
    k = p.conv.astype(np.float64)
    want, weight = np.zeros(got.shape, np.complex128), np.zeros(got.shape)
    for i, row in enumerate(geom.order):
        for c in range(p.channels):
            lam = float(p.wavelengths.reshape(-1)[c])
            u = float(p.uvw[row, 0]) / lam * (p.nx * float(p.cell_x) * rad)
            v = float(p.uvw[row, 1]) / lam * -(p.ny * float(p.cell_y) * rad)
            x, y = int(np.floor(u)) + p.nx // 2 - s, int(np.floor(v)) + p.ny // 2 - s
            if x < 0 or y < 0 or x + W + 2 >= p.nx or y + W + 2 >= p.ny:
                continue
            fu, fv = int((1 - u + np.floor(u)) * os), int((1 - v + np.floor(v)) * os)
            tap = k[fv + os * np.arange(W)][:, None] * k[fu + os * np.arange(W)][None, :]
            want[i, c] = (grid[0, 0, :, y:y + W, x:x + W].astype(np.complex128) * tap).sum((1, 2))
            ok = not p.flagged_rows[row]
            weight[i, c] = p.weights[row, c] * (~p.flags[row, c]) * ok
    assert np.abs(want).max() > 0
    assert rel(got, want) <= TOL[precision]
    assert rel(back, want * weight) <= TOL[precision]
