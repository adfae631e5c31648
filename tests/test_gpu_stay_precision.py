"""Work items of several segments keep the precision of single ones (32-bit library).

A segment gridded by itself adds its visibilities to a cell in FP32 and the sum to the grid without loss.  That
sum is emulated here, visibility by visibility (products of taps, then fused multiply-adds, rounded as FP32), and
its grid's error against FP64 is the bar: the same facet many times over, so that items take several segments,
may be no further off.  Slow and fast tracks, segments shorter and longer than a staged chunk; the facet lies at the
phase centre and the weights are one, so that the visibilities enter as they are.
"""
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth
from bullseye_gb300.imaging import baseline_index, run_imaging
from tests.test_gpu_parity import gpu_libs  # noqa: F401

pytestmark = pytest.mark.gpu

FACETS = 48


def _problem(n_times, pace, wplanes):
    p = synth.small_problem("double", nx=64, n_ant=10, n_times=n_times, n_chan=30, n_facets=1, s=7, os=15,
                            wplanes=wplanes, min_support=9 if wplanes > 1 else None, cell=80.0, seed=17)
    p = replace(p, uvw=p.uvw * np.array([pace, 0.3 * pace, 1.0]), facet_centres=np.array([p.phase_centre] * FACETS),
                weights=np.ones_like(p.weights), flags=np.zeros_like(p.flags), flagged_rows=np.zeros_like(p.flagged_rows))
    return p.astype("single")


def _grids(p):
    """The first correlation's grid in FP64, and from FP32 sums of single segments."""
    W, os, n, C = 2 * p.conv_support + 1, p.conv_oversample, p.nx, p.channels
    b = baseline_index(p.antenna1, p.antenna2, p.n_antennas)
    slots = {int(v): i for i, v in enumerate(np.unique(b))}
    track = np.array([slots[int(v)] for v in b])
    acc = np.zeros((len(slots) * C, n, n, 2), np.float32)
    exact = np.zeros((n, n), np.complex128)
    lam = p.wavelengths.reshape(-1).astype(np.float64)
    rad = float(np.float32(np.pi / (180.0 * 3600.0)))
    conv = p.conv.reshape(p.wplanes, -1)
    taps = np.arange(W) * os
    wide = p.wplanes > 1
    for t in np.unique(p.timestamp_ids):
        rows = np.flatnonzero(p.timestamp_ids == t)
        u, v, w = (p.uvw[rows, k].astype(np.float64)[:, None] / lam for k in range(3))
        u, v = u * (n * float(p.cell_x) * rad), v * -(n * float(p.cell_y) * rad)
        flip = (w < 0) & wide
        u, v = np.where(flip, -u, u), np.where(flip, -v, v)
        ru, rv = (np.rint(u), np.rint(v)) if wide else (np.floor(u), np.floor(v))
        x, y = ru.astype(int) + n // 2 - p.conv_support, rv.astype(int) + n // 2 - p.conv_support
        plane = np.rint(np.abs(w) * ((p.wplanes - 1) / p.wmax)).astype(int) if wide else np.zeros_like(x)
        ok = (x >= 0) & (y >= 0) & (x + W + 2 < n) & (y + W + 2 < n) & (plane < p.wplanes)
        fu, fv = ((1 - (u - ru)) * os).astype(int), ((1 - (v - rv)) * os).astype(int)
        r, c = np.nonzero(ok)
        at = (track[rows][r] * C + c)[:, None, None]
        yy, xx = y[r, c][:, None, None] + np.arange(W)[None, :, None], x[r, c][:, None, None] + np.arange(W)[None, None, :]
        ku = conv[plane[r, c][:, None], fu[r, c][:, None] + taps].astype(np.complex128)
        kv = conv[plane[r, c][:, None], fv[r, c][:, None] + taps].astype(np.complex128)
        vis = p.vis[rows[r], c, 0].astype(np.complex128)
        vis = np.where(flip[r, c], vis.conj(), vis)
        np.add.at(exact, (yy, xx), vis[:, None, None] * kv[:, :, None] * ku[:, None, :])
        f32 = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
        a, k = ku[:, None, :], kv[:, :, None]
        tr = f32(a.real * k.real - f32(a.imag * k.imag))
        ti = f32(a.real * k.imag + f32(a.imag * k.real))
        vr, vi = vis.real[:, None, None], vis.imag[:, None, None]
        old = acc[at, yy, xx].astype(np.float64)
        acc[at, yy, xx, 0] = f32(f32(old[..., 0] + vr * tr) - vi * ti)
        acc[at, yy, xx, 1] = f32(f32(old[..., 1] + vr * ti) + vi * tr)
    s = acc.astype(np.float64).sum(0)
    return exact, s[..., 0] + 1j * s[..., 1]


@pytest.mark.parametrize("n_times,pace,wplanes", [(16, 0.03, 6), (16, 0.5, 1), (30, 1.0, 1), (45, 2.0, 6), (100, 2.0, 6),
                                                  (100, 0.5, 1), (150, 0.5, 6)])
def test_error(n_times, pace, wplanes, gpu_libs):
    from bullseye_gb300.library import check
    lib = gpu_libs["single"]
    p = _problem(n_times, pace, wplanes)
    exact, unmerged = _grids(p)
    # as the library returns it, in FP32; a twentieth for the spread of two root mean squares over some 2,000 cells
    bar = 1.05 * np.sqrt(np.sum(np.abs(unmerged.astype(np.complex64) - exact) ** 2))
    got = run_imaging(lib, p, "facet_4_cor", keep_raw=True, repack=True, norm_bins=(2 * p.conv_support + 1) ** 2).raw_grid
    check(lib)
    err = np.sqrt(np.mean([np.sum(np.abs(g[0, 0] - exact) ** 2) for g in got]))
    assert 0 < err <= bar
