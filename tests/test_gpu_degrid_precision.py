"""The gather's precision in the 32-bit library: gradients with w kernels, and prediction divided by tap sums.

With complex taps a visibility gathered by itself (products of taps rounded to FP32, 32 partial sums over its
cells, a tree over these) is emulated here, and the adjoint's error against FP64 over random gradients may be a
fiftieth larger (the spread of a root mean square over some ten thousand values).

A value divided by its tap sum may be a tenth further off than the value itself: the quotient's own rounding adds
0.4 of 2^-24 in root mean square to the 1.2 to 1.5 of the gathered values.
"""
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth

pytestmark = pytest.mark.gpu


def _problem(wplanes, s, n_times):
    p = synth.small_problem("double", nx=96, n_ant=14, n_times=n_times, n_chan=4, n_facets=1, s=s, os=15, wplanes=wplanes,
                            min_support=2 * s + 1 if wplanes > 1 else None, seed=23)
    return replace(p, facet_centres=np.array([p.phase_centre]), weights=np.ones_like(p.weights),
                   flags=np.zeros_like(p.flags), flagged_rows=np.zeros_like(p.flagged_rows)).astype("single")


def _footprints(p, order):
    W, os = 2 * p.conv_support + 1, p.conv_oversample
    lam, rad = p.wavelengths.reshape(-1).astype(np.float64), float(np.float32(np.pi / (180.0 * 3600.0)))
    u, v, w = (p.uvw[order, k].astype(np.float64)[:, None] / lam for k in range(3))
    u, v = u * (p.nx * float(p.cell_x) * rad), v * -(p.ny * float(p.cell_y) * rad)
    wide = p.wplanes > 1
    flip = (w < 0) & wide
    u, v = np.where(flip, -u, u), np.where(flip, -v, v)
    ru, rv = (np.rint(u), np.rint(v)) if wide else (np.floor(u), np.floor(v))
    x, y = ru.astype(int) + p.nx // 2 - p.conv_support, rv.astype(int) + p.ny // 2 - p.conv_support
    plane = np.rint(np.abs(w) * ((p.wplanes - 1) / p.wmax)).astype(int) if wide else np.zeros_like(x)
    ok = (x >= 0) & (y >= 0) & (x + W + 2 < p.nx) & (y + W + 2 < p.ny) & (plane < p.wplanes)
    fu, fv = ((1 - (u - ru)) * os).astype(int), ((1 - (v - rv)) * os).astype(int)
    r, c = np.nonzero(ok)
    conv = p.conv.reshape(p.wplanes, -1)
    taps = np.arange(W) * os
    ku = conv[plane[r, c][:, None], fu[r, c][:, None] + taps].astype(np.complex128)
    kv = conv[plane[r, c][:, None], fv[r, c][:, None] + taps].astype(np.complex128)
    yy = y[r, c][:, None, None] + np.arange(W)[None, :, None]
    xx = x[r, c][:, None, None] + np.arange(W)[None, None, :]
    return r, c, yy, xx, ku, kv, flip[r, c]


def _f32(a):
    return a.astype(np.float32).astype(np.float64)


def test_gradients_with_w_kernels(gpu_required, built_libraries):
    import torch
    from bullseye_gb300 import autograd
    p = _problem(4, 11, 40)
    geom = autograd.FacetGeometry.from_problem(p)
    rng = np.random.default_rng(4)
    grad = (rng.normal(size=(1, 1, 4, p.ny, p.nx)) + 1j * rng.normal(size=(1, 1, 4, p.ny, p.nx))).astype(np.complex64)
    zero = torch.zeros((geom.order.size, p.channels, 4), dtype=torch.complex64, device="cuda")
    got, _ = autograd.grid_adjoint(geom, zero, None, torch.as_tensor(grad, device="cuda"))
    r, c, yy, xx, ku, kv, flip = _footprints(p, geom.order)
    got = got.cpu().numpy()[r, c].astype(np.complex128)
    got = np.where(flip[:, None], got.conj(), got)
    N, cells = r.size, yy.shape[1] * xx.shape[2]
    assert N > 1500
    a, k = ku[:, None, :], kv[:, :, None]
    tr = _f32(a.real * k.real - _f32(a.imag * k.imag)).reshape(N, cells)
    ti = -_f32(a.real * k.imag + _f32(a.imag * k.real)).reshape(N, cells)
    err = [0.0, 0.0]
    for q in range(4):
        g = grad[0, 0, q].astype(np.complex128)[yy, xx].reshape(N, cells)
        exact = (g * (k * a).conj().reshape(N, cells)).sum(1)
        sums = []
        for part in (g.real * tr - _f32(g.imag * ti), g.real * ti + _f32(g.imag * tr)):
            part = np.pad(_f32(part), ((0, 0), (0, -cells % 32))).reshape(N, -1, 32)
            s = np.zeros((N, 32))
            for j in range(part.shape[1]):
                s = _f32(s + part[:, j])
            for off in (16, 8, 4, 2, 1):
                s = _f32(s + s[:, np.arange(32) ^ off])
            sums.append(s[:, 0])
        err[0] += np.sum(np.abs(got[:, q] - exact) ** 2)
        err[1] += np.sum(np.abs(sums[0] + 1j * sums[1] - exact) ** 2)
    assert 0 < np.sqrt(err[0]) <= 1.02 * np.sqrt(err[1])


@pytest.mark.parametrize("s", [3, 7])
def test_prediction_divided_by_tap_sums(s, gpu_required, built_libraries):
    import torch
    from bullseye_gb300 import autograd
    p = _problem(1, s, 40)
    geom = autograd.FacetGeometry.from_problem(p)
    rng = np.random.default_rng(5)
    grid = (rng.normal(size=(1, 1, 4, p.ny, p.nx)) + 1j * rng.normal(size=(1, 1, 4, p.ny, p.nx))).astype(np.complex64)
    r, c, yy, xx, ku, kv, _ = _footprints(p, geom.order)
    tap = (kv[:, :, None] * ku[:, None, :]).real
    exact = np.stack([(grid[0, 0, q].astype(np.complex128)[yy, xx] * tap).sum((1, 2)) for q in range(4)], 1)
    off = []
    for divide in (False, True):
        got = autograd.predict(geom, torch.as_tensor(grid, device="cuda"), from_grid=True, normalise=divide)
        want = exact / tap.sum((1, 2))[:, None] if divide else exact
        d = got.cpu().numpy()[r, c].astype(np.complex128) - want
        off.append(np.sqrt(np.sum(np.abs(d) ** 2) / np.sum(np.abs(want) ** 2)))
    assert 0 < off[1] <= 1.1 * off[0]
