"""The work that users of the imaging libraries have them do, as cases that can be timed.

Five kinds of call, each through an entry point that a program calls:

  pipeline  the pipeliner's whole sequence on host arrays (initLibrary, repack_input_data, a gridding
            call, the sampling function, gridding_barrier, weight_uniformly, normalize, finalize,
            releaseLibrary);
  batched   bullseye_grid_batched on device-resident rows, visibilities and sampling function, with the
            copy-back of the final chunk into page-locked host grids;
  facets    bullseye_grid_batched_facets into the caller's device grids: equal or uneven facets;
  step      autograd.facet_grid forward, and its gradients for given output gradients;
  predict   autograd.predict: model images to visibilities.

Observations are an array's Earth-rotation tracks: the EVLA positions for 27 antennas, a disc of
antennas otherwise.  Declination, hour angle, visibilities, weights, flags and gains come from the seed;
the kernel table, the channels and the facet layout are the case's.  `turn` is the Earth's rotation
between two samples in degrees (0.06 is a 14 s integration).  Rows are single precision values in both
precisions of the library.
"""
import ctypes
import math

import numpy as np
import torch

from bullseye_gb300 import autograd, filters, synth
from bullseye_gb300.abi import BullseyeFacet, gridding_parameters_type
from bullseye_gb300.imaging import GRID_CALLS, GriddingProblem, baseline_index
from bullseye_gb300.library import check, load_library

ARCSEC = float(np.float32(math.pi / (180.0 * 3600.0)))  # the libraries' single precision constant
DEC0 = -30.0 * 3600.0  # phase centre, arcsec
FIELD = 3.0 * 3600.0   # facet centres lie within 3 degrees of it
SOURCES = 20
EXACT_CELLS = 4e10     # cell updates that the 64-bit restatement grids in a few seconds


# ----------------------------------------------------------------------------- cases
def _case(kind, **kw):
    c = dict(kind=kind, precision="single", ants=27, times=50, chans=16, facets=1, n=1024, cell=5.0, planes=64,
             half=31, least=15, os=15, turn=0.06, jones=True, call="facet_4_cor_corrections", pinned=True, masked=False)
    c.update(kw)
    return c


def listed():
    return [
        # a quick look at a few minutes of data of a small array: latency of the whole sequence
        _case("pipeline", name="pipeline-small", ants=8, times=12, chans=3, facets=2, n=96, cell=60.0, planes=1, half=3,
              least=7, os=15, turn=5.0, pinned=False),
        # plain imaging, one facet, natural kernel, one channel, as the reference's first example
        _case("pipeline", name="pipeline-plain", ants=64, times=120, chans=1, facets=0, n=1024, cell=2.0, planes=1,
              half=3, least=7, os=63, turn=0.75, jones=False, call="grid_4_cor", pinned=False),
        # one correlation, faceted: continuum imaging of total intensity (the per-track kernels)
        _case("pipeline", name="pipeline-one-corr", times=100, chans=16, facets=4, n=512, cell=10.0, planes=32, half=15,
              least=7, jones=False, call="facet_single_pol"),
        # direction-dependent imaging of one chunk of rows, host to image
        _case("pipeline", name="pipeline-facets", times=100, chans=64, facets=8, n=512, cell=10.0),
        # device-resident chunk of the 16-facet workload, with the sampling function
        _case("batched", name="batched-chunk", times=100, chans=64, facets=16),
        # a long observation of the same
        _case("batched", name="batched-long", times=400, chans=64, facets=16),
        # a short snapshot into small facets: launches and tails
        _case("facets", name="facets-snapshot", times=16, chans=15, facets=8, n=250, cell=10.0, planes=32, half=15,
              least=7, jones=False, call="facet_4_cor"),
        # uneven facets, each with its own rows
        _case("facets", name="facets-uneven", times=200, chans=32, facets=24, n=1024, planes=128, jones=False,
              call="facet_4_cor", masked=True),
        # the 64-bit library
        _case("facets", name="facets-double", precision="double", times=40, chans=16, facets=4, n=1000),
        # calibration: gridding and its gradients, many baselines on one wide facet
        _case("step", name="step-wide", ants=64, times=60, chans=16, facets=1, n=2048, cell=4.0, planes=32, half=15,
              least=7, turn=0.09),
        # prediction of a sky model from 16 facets
        _case("predict", name="predict-facets", times=50, chans=64, facets=16),
        # prediction from one image without gains
        _case("predict", name="predict-plain", ants=64, times=120, chans=1, facets=1, n=1024, cell=2.0, planes=1, half=3,
              least=7, os=63, turn=0.75, jones=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["pipeline", "batched", "facets", "facets", "step", "predict"])
        wide = rng.random() < 0.75  # w-projection
        half = rng.choice([7, 15, 23, 31]) if wide else rng.choice([3, 3, 4, 7])
        c = _case(kind, ants=rng.choice([8, 16, 27, 27, 27, 40, 64]), times=_log(rng, 10, 400), chans=_log(rng, 1, 64),
                  facets=_log(rng, 1, 16), n=_log(rng, 200, 2048), planes=_log(rng, 16, 128) if wide else 1, half=half,
                  least=rng.choice([7, 2 * (half // 2) + 1]) if wide else 2 * half + 1,
                  os=15 if wide else rng.choice([15, 63]), jones=rng.random() < 0.6)
        # the longest baseline reaches a fifth to four fifths of the way to the grid's edge
        c["cell"] = round(rng.uniform(0.2, 0.8) / (2 * ARCSEC * _longest(c) / (synth.C_LIGHT / 1.5e9)), 3)
        c["turn"] = round(min(math.exp(rng.uniform(math.log(0.03), math.log(1.0))), 120.0 / c["times"]), 4)
        c["call"] = "facet_4_cor_corrections" if c["jones"] else "facet_4_cor"
        if kind == "pipeline":
            c["pinned"] = rng.random() < 0.5
            c["n"] = min(c["n"], 1024)
            if not c["jones"]:
                c["call"] = rng.choice(["facet_4_cor", "facet_single_pol", "facet_duel_pol"])
        if kind in ("facets", "predict", "step") and rng.random() < 0.25:
            c["precision"] = "double"
        if kind == "facets" and not c["jones"]:
            c["masked"] = rng.random() < 0.5
        if kind == "step":
            c["jones"], c["call"] = True, "facet_4_cor_corrections"
        if _cost(c) <= most * (0.03 if c["precision"] == "double" else 1.0) and _grid_cells(c) <= 16 << 20:
            return c


def _corrs(c):
    return GRID_CALLS[c["call"]][0]


def _sizes(c):
    """Facet sizes: equal, or spread over a factor of four about n for a masked (uneven) layout."""
    F = max(1, c["facets"])
    if not c["masked"]:
        return [c["n"]] * F
    r = np.random.default_rng(21 + F)
    return [int(c["n"] * 2.0 ** x) // 2 * 2 + 1 * (i % 3 == 1) for i, x in enumerate(r.uniform(-1.5, 0.5, F))]


def _grid_cells(c):
    return sum(n * n for n in _sizes(c))


def _supports(c):
    if c["planes"] == 1:
        return np.array([2 * c["half"] + 1])
    return np.asarray(filters.plane_supports(c["planes"], c["least"], 2 * c["half"] + 1))


def _baselines(c):
    return c["ants"] * (c["ants"] - 1) // 2


def _pairs(c):
    share = 0.35 if c["masked"] else 1.0  # the masks' mean kept share (see _masks)
    return c["times"] * _baselines(c) * c["chans"] * max(1, c["facets"]) * share


def _cells_per_pair(c):
    """Mean squared support over w planes: |w| is near enough uniform over the lower half of its range."""
    s = _supports(c).astype(np.float64)
    return float(np.mean(s[:max(1, (s.size + 1) // 2)] ** 2))


def _cost(c):
    return _pairs(c) * _cells_per_pair(c) * (2 if c["kind"] == "step" else 1)


def work(c):
    """Bytes: rows, gains and grids (or images) read and written once.  Flops: 8 per complex multiply-add
    of a visibility's support and correlation, 6 per correlation for the phase, 128 for the gains."""
    size = 4 if c["precision"] == "single" else 8
    nc = _corrs(c)
    vis = c["times"] * _baselines(c) * c["chans"]
    per_vis = 4 * (2 * size + size + 1)
    gains = c["times"] * c["ants"] * max(1, c["facets"]) * c["chans"] * 8 * size if c["jones"] else 0
    grids = _grid_cells(c) * nc * 2 * size
    bytes_ = vis * per_vis + vis // c["chans"] * (3 * size + 25) + gains + grids
    flops = _pairs(c) * (8 * nc * _cells_per_pair(c) + 6 * nc + (128 if c["jones"] else 0))
    if c["kind"] in ("pipeline", "batched"):
        bytes_ += _grid_cells(c) * 2 * size  # the sampling function
        flops += vis * 8 * _cells_per_pair(c)
    if c["kind"] == "step":
        return {"bytes": 2 * bytes_ + vis * 8 * size + gains, "flops": 2 * flops}
    if c["kind"] == "predict":
        bytes_ = vis * 8 * size + vis // c["chans"] * (3 * size + 25) + gains + grids
    return {"bytes": bytes_, "flops": flops}


# ----------------------------------------------------------------------------- inputs
def _array(c):
    """Antenna positions in the local equatorial frame, metres."""
    if c["ants"] == 27:
        return synth.evla27_equatorial()
    return synth.enu_to_equatorial(synth.disc_layout(c["ants"], 2000.0 if c["planes"] == 1 else 1500.0, 1),
                                   np.deg2rad(-30.0))


def _longest(c):
    xyz = _array(c)
    return float(np.linalg.norm(xyz[:, None] - xyz[None], axis=-1).max())


def _tables(c):
    """What the case fixes: channels, kernel table, facet layout (arcsec)."""
    xyz = _array(c)
    lam = (synth.C_LIGHT / np.linspace(1.0e9, 1.5e9, c["chans"])).astype(np.float32)
    fov = c["n"] * c["cell"] * synth.ARCSEC
    if c["planes"] > 1:
        wmax = float(np.float32(_longest(c) / lam.min() * 1.001))
        conv, _ = filters.wproj_kernels(c["half"], c["os"], c["planes"], wmax, fov, min_support=c["least"])
        conv = conv.astype(np.complex64).astype(np.complex128)
    else:
        wmax = 1.0
        conv = filters.pswf_kernel(c["half"], c["os"]).astype(np.float32).astype(np.float64)
    r = np.random.default_rng(9)
    F = max(1, c["facets"])
    off = r.uniform(-FIELD, FIELD, (64, 2))[:F]
    dec0 = math.radians(DEC0 / 3600.0)
    centres = np.stack([off[:, 0] / math.cos(dec0), DEC0 + off[:, 1]], axis=1).astype(np.float32)
    if c["facets"] == 0:
        centres = np.array([[0.0, DEC0]], np.float32)
    return dict(xyz=xyz, lam=lam, wmax=wmax, conv=conv, centres=centres, sizes=_sizes(c))


def _inputs(c, seed, tab, time_major=False):
    """Rows, visibilities and gains of one observation (numpy rows, torch device data), baseline-major, or
    in Measurement Set order with time_major."""
    r = np.random.default_rng(seed)
    dec = np.deg2rad(-30.0 + r.uniform(-3.0, 3.0))
    xyz, start = tab["xyz"], np.deg2rad(r.uniform(-30.0, 30.0))  # hour angle of the middle of the track
    spin = np.array([[math.cos(start), -math.sin(start), 0], [math.sin(start), math.cos(start), 0], [0, 0, 1]])
    uvw, a1, a2, tid = synth.earth_rotation_rows(xyz @ spin.T, c["times"], dec, np.deg2rad(c["turn"] * (c["times"] - 1)))
    if not time_major:
        order = np.argsort(baseline_index(a1, a2, c["ants"]), kind="stable")
        uvw, a1, a2, tid = uvw[order], a1[order], a2[order], tid[order]
    uvw = uvw.astype(np.float32)
    R, Ch, dev = uvw.shape[0], c["chans"], "cuda"
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    reach = c["n"] * c["cell"] * synth.ARCSEC * 0.4
    l, m = (torch.as_tensor(r.uniform(-reach, reach, SOURCES), dtype=torch.float32, device=dev) for _ in range(2))
    flux = torch.as_tensor(r.uniform(0.1, 2.0, SOURCES), dtype=torch.complex64, device=dev)
    g = torch.as_tensor(uvw, device=dev)
    path = g[:, 0:1] * l + g[:, 1:2] * m + g[:, 2:3] * (torch.sqrt(1 - l * l - m * m) - 1)
    vis = torch.randn((R, Ch, 4), dtype=torch.complex64, device=dev, generator=gen) * 0.01
    for k in range(Ch):
        ph = path * (-2 * math.pi / float(tab["lam"][k]))
        s = torch.polar(torch.ones_like(ph), ph) @ flux
        vis[:, k, 0] += s
        vis[:, k, 3] += s
    weights = torch.rand((R, Ch, 4), device=dev, generator=gen) + 0.5
    flags = (torch.rand((R, Ch, 1), device=dev, generator=gen) < 0.02).expand(R, Ch, 4).contiguous()
    flagged_rows = torch.rand(R, device=dev, generator=gen) < 0.02
    jones = None
    if c["jones"]:
        shape = (c["times"], c["ants"], max(1, c["facets"]), 1, Ch)
        jones = 0.05 * torch.randn(shape + (4,), dtype=torch.complex64, device=dev, generator=gen)
        for k in (0, 3):
            jones[..., k] = torch.polar(0.9 + 0.2 * torch.rand(shape, device=dev, generator=gen),
                                        (2 * torch.rand(shape, device=dev, generator=gen) - 1) * math.pi)
    return dict(uvw=uvw, a1=a1, a2=a2, tid=tid, vis=vis, weights=weights, flags=flags, flagged_rows=flagged_rows,
                jones=jones)


def _masks(c, seed, d):
    """[F][R] bytes: each facet keeps a share of the baselines and a range of times."""
    r = np.random.default_rng(seed + 5)
    b = baseline_index(d["a1"], d["a2"], c["ants"])
    t = d["tid"].astype(np.int64)
    out = np.zeros((max(1, c["facets"]), b.size), np.uint8)
    for f in range(out.shape[0]):
        share = r.uniform(0.2, 1.0, 2)
        keep = r.random(int(b.max()) + 1) < share[0]
        t0, span = int(r.integers(0, c["times"])), max(1, int(share[1] * c["times"]))
        out[f] = keep[b] & (((t - t0) % c["times"]) < span)
    return out


def _grads(c, seed):
    """Output gradients of a step: the residual grids of a fit, complex noise here."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 17)
    g = torch.randn((max(1, c["facets"]), 1, 4, c["n"], c["n"]), dtype=torch.complex64, device="cuda", generator=gen)
    return g.to(_ctype(c))


def _model(c, seed):
    """Model images: point sources in each facet, with polarisation."""
    r = np.random.default_rng(seed + 23)
    n, F = c["n"], max(1, c["facets"])
    img = torch.zeros((F, 1, 4, n, n), dtype=_ctype(c), device="cuda")
    for f in range(F):
        y, x = (torch.as_tensor(r.integers(n // 4, 3 * n // 4, SOURCES), device="cuda") for _ in range(2))
        for k in range(4):
            flux = r.uniform(0.1, 2.0, SOURCES) + 1j * r.uniform(-0.1, 0.1, SOURCES)
            img[f, 0, k, y, x] = torch.as_tensor(flux, device="cuda").to(torch.complex64).to(_ctype(c))
    return img


def _taper(c, tab):
    k = np.real(tab["conv"][0]) if c["planes"] > 1 else tab["conv"]
    return filters.gridding_correction(k, c["half"], c["os"], c["n"])


def _normalised(c):
    """Prediction divides by the tap sum with a natural kernel; a w kernel's tap sum can come near zero."""
    return c["planes"] == 1


def _ctype(c):
    return torch.complex64 if c["precision"] == "single" else torch.complex128


def _rtype(c):
    return torch.float32 if c["precision"] == "single" else torch.float64


def _np_conv(c, tab):
    one = c["precision"] == "single"
    kind = (np.complex64 if one else np.complex128) if c["planes"] > 1 else (np.float32 if one else np.float64)
    return np.ascontiguousarray(tab["conv"].astype(kind))


# ----------------------------------------------------------------------------- the library's own state
class _Live:
    """The library holds one set of tables at a time: the cases that keep it initialised share it."""
    lib, key, keep = None, None, None

    @classmethod
    def release(cls):
        if cls.lib is not None:
            cls.lib.releaseLibrary()
            cls.lib.bullseye_set_device_inputs(0)
            check(cls.lib)
        cls.lib = cls.key = cls.keep = None

    @classmethod
    def attach(cls, key, lib, st, keep):
        if cls.key == key:
            return
        cls.release()
        lib.bullseye_set_device_inputs(1)
        lib.initLibrary(ctypes.byref(st))
        check(lib)
        cls.lib, cls.key, cls.keep = lib, key, keep


def _p(t):
    if t is None:
        return None
    return ctypes.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


def _struct(c, tab, conv, own):
    """gridding_parameters with the tables; `own` keeps what it points at."""
    rd = np.float32 if c["precision"] == "single" else np.float64
    Ch, R = c["chans"], c["times"] * _baselines(c)
    own.update(lam=tab["lam"].astype(rd), conv=conv, on=np.ones(Ch, np.bool_), cgi=np.zeros(Ch, np.uintp),
               centres=tab["centres"].astype(rd))
    st = gridding_parameters_type(c["precision"])()
    st.chunk_max_row_count = st.row_count = R
    st.nx = st.ny = c["n"]
    st.cell_size_x = st.cell_size_y = c["cell"]
    st.conv, st.conv_support, st.conv_oversample = _p(conv), c["half"], c["os"]
    st.phase_centre_ra, st.phase_centre_dec = 0.0, DEC0
    st.should_invert_jones_terms = bool(c["jones"])
    st.channel_grid_indicies, st.cube_channel_dim_size = _p(own["cgi"]), 1
    st.baseline_count = _baselines(c) + c["ants"]
    st.number_of_polarization_terms, st.number_of_polarization_terms_being_gridded = 4, _corrs(c)
    st.polarization_index, st.second_polarization_index = 0, 3
    st.spw_count, st.channel_count, st.antenna_count = 1, Ch, c["ants"]
    st.no_timestamps_read = c["times"]
    st.enabled_channels, st.reference_wavelengths = _p(own["on"]), _p(own["lam"])
    st.num_facet_centres, st.facet_centres = max(1, c["facets"]), _p(own["centres"])
    st.wplanes, st.wmax_est = c["planes"], tab["wmax"]
    return st


def _set_rows(st, rows):
    st.visibilities, st.uvw_coords, st.visibility_weights = _p(rows["vis"]), _p(rows["uvw"]), _p(rows["weights"])
    st.flags, st.flagged_rows, st.field_array = _p(rows["flags"]), _p(rows["flagged_rows"]), _p(rows["zero"])
    st.spw_index_array, st.antenna_1_ids, st.antenna_2_ids = _p(rows["zero"]), _p(rows["a1"]), _p(rows["a2"])
    st.timestamp_ids, st.jones_terms = _p(rows["tid"]), _p(rows["jones"])
    st.baseline_starting_indexes = _p(rows["starts"])


def _rows(c, d, place):
    """The row arrays in the library's types, each placed by `place`."""
    ct, rt = _ctype(c), _rtype(c)
    b = baseline_index(d["a1"], d["a2"], c["ants"])
    starts = np.zeros(_baselines(c) + c["ants"] + 1, np.int64)
    np.add.at(starts, b + 1, 1)
    t = torch.as_tensor
    return dict(
        vis=place(d["vis"].to(ct)), weights=place(d["weights"].to(rt)), uvw=place(t(d["uvw"]).to(rt)),
        flags=place(d["flags"].to(torch.uint8)), flagged_rows=place(d["flagged_rows"].to(torch.uint8)),
        zero=place(torch.zeros(b.size, dtype=torch.int32)), a1=place(t(d["a1"].astype(np.int32))),
        a2=place(t(d["a2"].astype(np.int32))), tid=place(t(d["tid"].astype(np.int64))),
        jones=None if d["jones"] is None else place(d["jones"].to(ct)), starts=place(t(np.cumsum(starts))))


def _host(c):
    def place(x):
        x = x.cpu().contiguous()
        return x.pin_memory() if c["pinned"] else x
    return place


# ----------------------------------------------------------------------------- prepare
def prepare(c, seed):
    tab = _tables(c)
    lib = load_library("GPU", c["precision"])
    d = _inputs(c, seed, tab, time_major=c["kind"] == "pipeline")
    s = dict(case=c, lib=lib, tab=tab)
    if c["kind"] in ("step", "predict"):
        s["geom"] = _geometry(c, tab, d)
        if c["kind"] == "step":
            s["vis"] = d["vis"].to(_ctype(c)).requires_grad_(True)
            s["jones"] = d["jones"].to(_ctype(c)).requires_grad_(True)
            s["grad"] = _grads(c, seed)
        else:
            s["jones"] = None if d["jones"] is None else d["jones"].to(_ctype(c))
            s["model"] = _model(c, seed)
            taper = torch.as_tensor(_taper(c, tab), device="cuda")
            s["taper"] = (taper, taper)
        return s
    own = s["own"] = {}
    conv = _np_conv(c, tab)
    st = s["st"] = _struct(c, tab, conv, own)
    if c["kind"] == "pipeline":
        _Live.release()
        s["rows"] = _rows(c, d, _host(c))
        F, nc, n, ct = max(1, c["facets"]), _corrs(c), c["n"], _ctype(c)
        s["grid"] = torch.zeros((F, 1, nc, n, n), dtype=ct, pin_memory=c["pinned"])
        s["sf"] = torch.zeros((F, 1, 1, n, n), dtype=ct, pin_memory=c["pinned"])
        st.output_buffer, st.sampling_function_buffer = _p(s["grid"]), _p(s["sf"])
        st.should_grid_sampling_function = True
        st.sampling_function_channel_grid_indicies, st.sampling_function_channel_count = _p(own["cgi"]), 1
        st.is_final_data_chunk = True
        _set_rows(st, s["rows"])
        return s
    s["rows"] = _rows(c, d, lambda x: x.cuda())
    _set_rows(st, s["rows"])
    key = repr(sorted((k, v) for k, v in c.items() if k != "name"))
    s["live"] = key
    F, ct = max(1, c["facets"]), _ctype(c)
    if c["kind"] == "batched":
        s["grid"] = torch.zeros((F, 1, 4, c["n"], c["n"]), dtype=ct, pin_memory=True)
        s["sf"] = torch.zeros((F, 1, 1, c["n"], c["n"]), dtype=ct, pin_memory=True)
        st.output_buffer, st.sampling_function_buffer = _p(s["grid"]), _p(s["sf"])
        st.should_grid_sampling_function = True
        st.sampling_function_channel_grid_indicies, st.sampling_function_channel_count = _p(own["cgi"]), 1
        st.is_final_data_chunk = True
    else:
        cells = _grid_cells(c)
        s["grid"] = torch.zeros(4 * cells, dtype=ct, device="cuda")
        s["lo"] = torch.zeros_like(s["grid"]) if c["precision"] == "single" else None
        s["norm"] = torch.zeros((F, 4), dtype=torch.float64, device="cuda")
        s["facets"], at = (BullseyeFacet * F)(), 0
        for f, n in enumerate(tab["sizes"]):
            s["facets"][f] = BullseyeFacet(float(tab["centres"][f, 0]), float(tab["centres"][f, 1]), _cell(c), _cell(c), n, n, at)
            at += 4 * n * n
        s["mask"] = torch.as_tensor(_masks(c, seed, d), device="cuda") if c["masked"] else None
    _attach(s)
    s["init"] = _Live.keep["st"]
    torch.cuda.synchronize()
    return s


def _cell(c):
    """The facets' cell size as the struct of the case's precision holds it."""
    return float(np.float32(c["cell"])) if c["precision"] == "single" else float(c["cell"])


def _attach(s):
    """The library initialised with the case's tables (its own grids: small for caller-owned output)."""
    if _Live.key == s["live"]:
        return
    c, own = s["case"], {}
    st = _struct(c, s["tab"], _np_conv(c, s["tab"]), own)
    if c["kind"] == "batched":
        st.should_grid_sampling_function = True
        st.sampling_function_channel_grid_indicies, st.sampling_function_channel_count = _p(own["cgi"]), 1
    _Live.attach(s["live"], s["lib"], st, dict(st=st, own=own))


def _geometry(c, tab, d):
    one = c["precision"] == "single"
    rd, cd = (np.float32, np.complex64) if one else (np.float64, np.complex128)
    R, Ch = d["uvw"].shape[0], c["chans"]
    p = GriddingProblem(
        precision=c["precision"], vis=np.broadcast_to(np.zeros((1, 1, 1), cd), (R, Ch, 4)), uvw=d["uvw"].astype(rd),
        wavelengths=tab["lam"].astype(rd).reshape(1, -1), weights=d["weights"].cpu().numpy().astype(rd),
        flags=d["flags"].cpu().numpy(), flagged_rows=d["flagged_rows"].cpu().numpy(), field_ids=np.zeros(R, np.uint32),
        spw_ids=np.zeros(R, np.uint32), antenna1=d["a1"], antenna2=d["a2"], timestamp_ids=d["tid"], n_antennas=c["ants"],
        n_timestamps=c["times"], nx=c["n"], ny=c["n"], cell_x=c["cell"], cell_y=c["cell"], conv=_np_conv(c, tab),
        conv_support=c["half"], conv_oversample=c["os"], wplanes=c["planes"], wmax=tab["wmax"], phase_centre=(0.0, DEC0),
        facet_centres=tab["centres"].astype(rd))
    return autograd.FacetGeometry.from_problem(p)


# ----------------------------------------------------------------------------- run
def run(s):
    c, lib = s["case"], s["lib"]
    if c["kind"] == "step":
        grids, norm = autograd.facet_grid(s["geom"], s["vis"], s["jones"])
        gv, gj = torch.autograd.grad(grids, (s["vis"], s["jones"]), s["grad"])
        return {"grids": grids.detach(), "norm": norm, "vis": gv, "jones": gj}
    if c["kind"] == "predict":
        return autograd.predict(s["geom"], s["model"], s["jones"], normalise=_normalised(c), taper=s["taper"])
    st, ref = s["st"], ctypes.byref(s["st"])
    if c["kind"] == "pipeline":
        return _run_pipeline(s, lib, st, ref)
    _attach(s)
    if c["kind"] == "batched":
        lib.bullseye_zero_grids()
        rc = lib.bullseye_grid_batched(ref, 0 if c["jones"] else 1, 1)
        lib.gridding_barrier()
        if rc:
            check(lib)
        bins = (2 * c["half"] + 1) ** 2
        norm = np.ctypeslib.as_array(ctypes.cast(s["init"].normalization_terms, ctypes.POINTER(ctypes.c_double)),
                                     shape=(max(1, c["facets"]), 4, bins))[:, :, 0].copy()
        return {"grids": s["grid"], "sampling": s["sf"], "norm": norm}
    with torch.cuda.stream(torch.cuda.ExternalStream(lib.bullseye_get_stream())):
        s["grid"].zero_()
        s["norm"].zero_()
        if s["lo"] is not None:
            s["lo"].zero_()
        rc = lib.bullseye_grid_batched_facets(ref, ctypes.cast(s["facets"], ctypes.c_void_p), len(s["facets"]),
                                              _p(s["mask"]), _p(s["grid"]), _p(s["lo"]), _p(s["norm"]),
                                              0 if c["jones"] else 1)
        if rc:
            check(lib)
        if s["lo"] is not None:
            s["grid"] += s["lo"]
    return {"grids": s["grid"], "norm": s["norm"]}


def _run_pipeline(s, lib, st, ref):
    c = s["case"]
    call = c["call"]
    s["grid"].zero_()
    s["sf"].zero_()
    lib.initLibrary(ref)
    lib.repack_input_data(ref)
    getattr(lib, call)(ref)
    (lib.facet_sampling_function if GRID_CALLS[call][1] else lib.grid_sampling_function)(ref)
    lib.gridding_barrier()
    lib.weight_uniformly(ref)
    F, nc, n = max(1, c["facets"]), _corrs(c), c["n"]
    bins = (2 * c["half"] + 1) ** 2
    norm = np.ctypeslib.as_array(ctypes.cast(st.normalization_terms, ctypes.POINTER(ctypes.c_double)),
                                 shape=(F, nc, bins))[:, :, 0].copy()
    lib.normalize(ref)
    lib.finalize(ref)
    lib.releaseLibrary()
    check(lib)
    # the packed single precision images lie at the start of every facet's block
    flat = s["grid"].view(torch.float32).reshape(-1)
    step = nc * n * n
    images = torch.stack([flat[f * step:f * step + n * n].view(n, n) for f in range(F)])
    return {"images": images, "sampling": s["sf"], "norm": norm}


# ----------------------------------------------------------------------------- in 64 bits
def _footprints(c, tab, d, facet, size, faceting, sampling):
    """Corner, tap offsets, w plane, conjugation and phase (turns) of every (row, channel) in one facet."""
    g = torch.as_tensor(d["uvw"].astype(np.float64), device="cuda")
    inv = 1.0 / torch.as_tensor(tab["lam"].astype(np.float64), device="cuda")
    u, v, w = ((g[:, k:k + 1] * inv).reshape(-1) for k in range(3))
    turns = None
    if faceting and not sampling:
        ra, dec = (float(x) * ARCSEC for x in tab["centres"][facet])
        dec0 = DEC0 * ARCSEC
        l = math.cos(dec) * math.sin(ra)
        m = math.sin(dec) * math.cos(dec0) - math.cos(dec) * math.sin(dec0) * math.cos(ra)
        nn = math.sin(dec) * math.sin(dec0) + math.cos(dec) * math.cos(dec0) * math.cos(ra)
        turns = u * -l + v * -m + w * (1.0 - math.sqrt(1.0 - l * l - m * m))
        turns = turns - torch.round(turns)
        u, v = u - w * (l / nn), v - w * (m / nn)
    scale = size * _cell(c) * ARCSEC
    u, v = u * scale, v * -scale
    wide = c["planes"] > 1
    flip = (w < 0) & wide
    u, v = torch.where(flip, -u, u), torch.where(flip, -v, v)
    ru, rv = (torch.round(u), torch.round(v)) if wide else (torch.floor(u), torch.floor(v))
    corner = size // 2 - c["half"]
    W = 2 * c["half"] + 1
    x, y = ru.long() + corner, rv.long() + corner
    plane = torch.round(w.abs() * ((c["planes"] - 1) / tab["wmax"])).long() if wide else torch.zeros_like(x)
    ok = (x >= 0) & (y >= 0) & (x + W + 2 < size) & (y + W + 2 < size) & (plane < c["planes"])
    fu, fv = ((1.0 - u + ru) * c["os"]).long(), ((1.0 - v + rv) * c["os"]).long()
    return x, y, fu, fv, plane, flip, turns, ok


def _windows(c, tab, x, y, fu, fv, plane, keep):
    """Per w plane and chunk: the kept samples, their cells [k, rows, columns] (relative) and their taps."""
    conv = torch.as_tensor(tab["conv"], device="cuda").reshape(c["planes"], -1).to(torch.complex128)
    W, os = 2 * c["half"] + 1, c["os"]
    tap = torch.arange(W, device="cuda")
    at = torch.nonzero(keep).reshape(-1)
    at = at[torch.argsort(plane[at], stable=True)]
    counts = torch.bincount(plane[at], minlength=c["planes"]).tolist()
    lo = 0
    for p, k in enumerate(counts):
        used = torch.nonzero(conv[p].abs() > 0).reshape(-1)
        first = max(0, math.ceil((int(used[0]) - 2 * os) / os)) if used.numel() else 0
        last = min(W - 1, int(used[-1]) // os) if used.numel() else 0
        t = tap[first:last + 1]
        part = max(1, (1 << 23) // (t.numel() ** 2))
        for b in range(lo, lo + k, part):
            i = at[b:min(lo + k, b + part)]
            ku = conv[p][fu[i][:, None] + t * os]
            kv = conv[p][fv[i][:, None] + t * os]
            yield i, y[i][:, None, None] + t[None, :, None], x[i][:, None, None] + t[None, None, :], ku, kv
        lo += k


def _apply_gains(vis, jones, rows, facet):
    """J_p^-1 V J_q^-H of [k, 4] visibilities, for rows' (times, antenna 1, antenna 2) and channels."""
    t, a1, a2, ch = rows
    p = torch.linalg.inv(jones[t, a1, facet, 0, ch].reshape(-1, 2, 2))
    q = torch.linalg.inv(jones[t, a2, facet, 0, ch].reshape(-1, 2, 2))
    return (p @ vis.reshape(-1, 2, 2) @ q.mH).reshape(-1, 4)


def exact(c, seed):
    cells = _pairs(c) * _cells_per_pair(c) * (2 if c["kind"] == "step" else 1)
    if cells > EXACT_CELLS:
        return None
    tab = _tables(c)
    d = _inputs(c, seed, tab, time_major=c["kind"] == "pipeline")
    F, Ch, nc = max(1, c["facets"]), c["chans"], _corrs(c)
    R = d["uvw"].shape[0]
    faceting = GRID_CALLS[c["call"]][1]
    pols = {1: [0], 2: [0, 3], 4: [0, 1, 2, 3]}[nc]
    t, a1, a2 = (torch.as_tensor(d[k].astype(np.int64), device="cuda").repeat_interleave(Ch) for k in ("tid", "a1", "a2"))
    rows = (t, a1, a2, torch.arange(Ch, device="cuda").repeat(R))
    row_ok = ~d["flagged_rows"].repeat_interleave(Ch)
    weight = d["weights"].double().reshape(-1, 4) * (~d["flags"].reshape(-1, 4) & row_ok[:, None])
    masks = torch.as_tensor(_masks(c, seed, d), device="cuda").bool() if c["masked"] else None
    jones = None if d["jones"] is None else d["jones"].to(torch.complex128)
    vis = d["vis"].to(torch.complex128).reshape(-1, 4)

    def seen(f, v, j):
        """Weighted, corrected, rotated visibilities of facet f, and its footprints."""
        fp = _footprints(c, tab, d, f, tab["sizes"][f], faceting, False)
        turns, flip, ok = fp[6], fp[5], fp[7]
        if masks is not None:
            ok = ok & masks[f].repeat_interleave(Ch)
        out = v if j is None else _apply_gains(v, j, rows, f)
        out = out[:, pols] * weight[:, pols]
        if turns is not None:
            out = out * torch.polar(torch.ones_like(turns), 2 * math.pi * turns)[:, None]
        return torch.where(flip[:, None], out.conj(), out), fp[:5], ok

    def grid(size, out, fp, ok):
        k = out.shape[1]
        g = torch.zeros((size * size, 2 * k), dtype=torch.float64, device="cuda")
        norm = torch.zeros(R * Ch, dtype=torch.float64, device="cuda")
        for i, yy, xx, ku, kv in _windows(c, tab, *fp, ok):
            taps = kv[:, :, None] * ku[:, None, :]
            val = torch.view_as_real(taps[..., None] * out[i][:, None, None, :]).reshape(-1, 2 * k)
            g.index_add_(0, (yy * size + xx).reshape(-1), val)
            norm[i] = (ku.sum(1) * kv.sum(1)).real
        g = torch.view_as_complex(g.view(size, size, k, 2)).permute(2, 0, 1)
        return g, norm

    if c["kind"] == "predict":
        return _exact_predict(c, seed, tab, d, jones, rows, faceting)
    grids, norms = [], []
    for f in range(F):
        out, fp, ok = seen(f, vis, jones)
        g, norm = grid(tab["sizes"][f], out, fp, ok)
        grids.append(g)
        norms.append((norm[:, None] * weight[:, pols] * ok[:, None]).sum(0))
    norm = torch.stack(norms)
    if c["kind"] == "facets":
        return {"grids": torch.cat([g.reshape(-1) for g in grids]), "norm": norm}
    if c["kind"] == "step":
        gv, gj = _exact_gradients(c, seed, tab, vis, jones, seen)
        return {"grids": torch.stack(grids)[:, None], "norm": norm[:, None], "vis": gv.reshape(R, Ch, 4), "jones": gj}
    fp = _footprints(c, tab, d, 0, c["n"], faceting, True)
    one = row_ok[:, None].to(torch.complex128)
    sf, _ = grid(c["n"], one, fp[:5], fp[7])
    sampling = sf.expand(F, 1, 1, c["n"], c["n"])
    g = torch.stack(grids)[:, None]
    if c["kind"] == "batched":
        return {"grids": g, "sampling": sampling, "norm": norm.cpu().numpy()}
    image = g[:, 0, 0] / (float(np.float32(1e-7)) + sf.real) / norm[:, 0, None, None]
    image = torch.fft.ifftshift(image, dim=(-2, -1))
    # finalize's inverse transform is not scaled by the number of cells
    image = torch.fft.fftshift(torch.fft.ifft2(image) * (c["n"] ** 2), dim=(-2, -1)).real
    return {"images": image, "sampling": sampling, "norm": norm.cpu().numpy()}


def _exact_gradients(c, seed, tab, vis, jones, seen):
    """Gradients of the grids for the given output gradients: the footprints' conjugate sums, taken back
    through the weights, phases and gains by torch."""
    grad = _grads(c, seed).to(torch.complex128)
    v, j = vis.clone().requires_grad_(True), jones.clone().requires_grad_(True)
    for f in range(max(1, c["facets"])):
        out, fp, ok = seen(f, v, j)
        flat = grad[f, 0].permute(1, 2, 0).reshape(-1, 4)
        back = torch.zeros_like(out)
        for i, yy, xx, ku, kv in _windows(c, tab, *fp, ok):
            taps = (kv[:, :, None] * ku[:, None, :]).conj().reshape(i.numel(), 1, -1)
            back[i] = (taps @ flat[(yy * c["n"] + xx).reshape(i.numel(), -1)]).reshape(-1, 4)
        out.backward(back)
    return v.grad, j.grad


def _exact_predict(c, seed, tab, d, jones, rows, faceting):
    n = c["n"]
    taper = torch.as_tensor(_taper(c, tab), device="cuda")
    model = _model(c, seed).to(torch.complex128) / (taper[:, None] * taper[None, :])
    total = torch.zeros((d["uvw"].shape[0] * c["chans"], 4), dtype=torch.complex128, device="cuda")
    t, a1, a2, ch = rows
    for f in range(max(1, c["facets"])):
        uv = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(model[f, 0], dim=(-2, -1))), dim=(-2, -1))
        flat = uv.permute(1, 2, 0).reshape(-1, 4)
        x, y, fu, fv, plane, flip, turns, ok = _footprints(c, tab, d, f, n, faceting, False)
        part = torch.zeros_like(total)
        for i, yy, xx, ku, kv in _windows(c, tab, x, y, fu, fv, plane, ok):
            taps = (kv[:, :, None] * ku[:, None, :]).conj().reshape(i.numel(), 1, -1)
            part[i] = (taps @ flat[(yy * n + xx).reshape(i.numel(), -1)]).reshape(-1, 4)
            if _normalised(c):
                part[i] /= taps.real.sum(-1)
        part = torch.where(flip[:, None], part.conj(), part)
        part = part * torch.polar(torch.ones_like(turns), -2 * math.pi * turns)[:, None]
        if jones is not None:
            p, q = (jones[t, a, f, 0, ch].reshape(-1, 2, 2) for a in (a1, a2))
            part = (p @ part.reshape(-1, 2, 2) @ q.mH).reshape(-1, 4)
        total += torch.where(ok[:, None], part, torch.zeros_like(part))
    return total.reshape(-1, c["chans"], 4)
