"""Degridding by groups and runs of rows (adjoint.cu degrid_adjoint_kernel).

A warp takes 32 rows of a channel and reads the grid once per stretch of rows that share their
footprint: groups with a common v tap row in the adjoint and in prediction with a 1-D kernel, runs of one
corner and w plane in prediction with w kernels.  The cases: standing and slow tracks (stretches longer
than a warp's rows), a cell or more per sample, tracks that leave the grid; windows narrower and wider
than a warp; kernel rows that are staged and ones that are read from the table; rows in track order and
in no order.  Prediction and the adjoint with unit weights (the same sums) are held to the FP64 oracle at
the libraries' bars, 1e-12 and 1e-5.
"""
from dataclasses import replace

import numpy as np
import pytest

from bullseye_gb300 import synth
from oracle.predict import predict as oracle_predict

pytestmark = pytest.mark.gpu


def _problem(s, wplanes, pace, os_):
    p = synth.small_problem("double", nx=131, ny=130, n_ant=5, n_times=75, n_chan=2, n_facets=2, s=s, os=os_,
                            wplanes=wplanes, min_support=min(5, 2 * s + 1), cell=60.0, seed=23)
    uvw = (p.uvw * np.array([pace, 0.3 * pace, 1.0])).astype(np.float32).astype(np.float64)
    return replace(p, uvw=uvw, jones=None, weights=np.ones_like(p.weights), flags=np.zeros_like(p.flags),
                   flagged_rows=np.zeros_like(p.flagged_rows))


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("order", ["tracks", "none"])
@pytest.mark.parametrize("pace", [0.002, 0.1, 2.5])
@pytest.mark.parametrize("s,wplanes,os_", [(3, 1, 63), (3, 3, 9), (8, 1, 9), (13, 5, 15), (31, 4, 15), (20, 2, 63)])
def test_gather_matches_oracle(precision, order, pace, s, wplanes, os_, gpu_required, built_libraries):
    import torch
    from bullseye_gb300.autograd import FacetGeometry, grid_adjoint, predict
    q = _problem(s, wplanes, pace, os_)
    p = q.astype(precision)
    geom = FacetGeometry.from_problem(p)
    if order == "none":
        perm = np.random.default_rng(3).permutation(p.rows)
        at = torch.as_tensor(perm, device="cuda")
        for k in ("uvw", "wt", "fl", "fr", "tid"):
            geom.arrays[k] = geom.arrays[k][at].contiguous()
        for k in ("field", "spw", "a1", "a2"):
            geom.arrays[k] = geom.arrays[k].view(torch.int32)[at].contiguous().view(torch.uint32)
        geom.order = geom.order[perm]
    ct = torch.complex64 if precision == "single" else torch.complex128
    rng = np.random.default_rng(7)
    G = rng.normal(size=geom.grid_shape) + 1j * rng.normal(size=geom.grid_shape)
    G = torch.as_tensor(G, device="cuda").to(ct).contiguous()
    vis = torch.zeros((p.rows, p.channels, 4), dtype=ct, device="cuda")
    back = np.argsort(geom.order)
    got = predict(geom, G, None, from_grid=True).cpu().numpy()[back]
    adj = grid_adjoint(geom, vis, None, G)[0].cpu().numpy()[back]
    want = oracle_predict(p.astype("double"), G.cpu().numpy().astype(np.complex128), faceting=True, normalise=False)
    if not np.any(want):  # every footprint leaves the grid
        assert not np.any(got) and not np.any(adj)
        return
    tol = 1e-12 if precision == "double" else 1e-5
    assert _rel(got, want) <= tol
    assert _rel(adj, want) <= tol
