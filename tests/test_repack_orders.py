"""repack_input_data (host only) over row orders and row widths: rows in order stay, wide rows move in place
along the permutation's cycles, narrow ones through a copy.  Every array must equal numpy's stable sort by
baseline slot."""
import ctypes

import numpy as np
import pytest

from bullseye_gb300.abi import complex_dtype, gridding_parameters_type, real_dtype
from bullseye_gb300.imaging import baseline_index


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("chans", [1, 3, 16])
@pytest.mark.parametrize("order", ["sorted", "time", "reversed", "random", "one_moved"])
def test_repack_orders(precision, chans, order, built_libraries):
    from bullseye_gb300.library import load_library
    lib = load_library("GPU", precision)
    n, times = 5, 9
    a1, a2 = (np.tile(x, times).astype(np.uint32) for x in np.triu_indices(n))
    b = baseline_index(a1, a2, n)
    rng = np.random.default_rng(2)
    sort = np.argsort(b, kind="stable")
    R = b.size
    perm = {"sorted": sort, "time": np.arange(R), "reversed": sort[::-1], "random": rng.permutation(R),
            "one_moved": np.concatenate([sort[1:], sort[:1]])}[order]
    a1, a2, b = a1[perm].copy(), a2[perm].copy(), b[perm]
    cd, rd = complex_dtype(precision), real_dtype(precision)
    arrays = dict(visibilities=rng.normal(size=(R, chans, 4)).astype(cd), uvw_coords=rng.normal(size=(R, 3)).astype(rd),
                  visibility_weights=rng.normal(size=(R, chans, 4)).astype(rd), flags=rng.random((R, chans, 4)) < 0.5,
                  flagged_rows=rng.random(R) < 0.5, spw_index_array=rng.integers(0, 9, R).astype(np.uint32),
                  antenna_1_ids=a1, antenna_2_ids=a2, field_array=rng.integers(0, 9, R).astype(np.uint32),
                  timestamp_ids=rng.integers(0, 99, R).astype(np.uintp))
    before = {k: v.copy() for k, v in arrays.items()}
    starts = np.zeros(n * (n + 1) // 2 + 1, np.uintp)
    st = gridding_parameters_type(precision)()
    for k, v in arrays.items():
        setattr(st, k, v.ctypes.data_as(ctypes.c_void_p))
    st.baseline_starting_indexes = starts.ctypes.data_as(ctypes.c_void_p)
    st.row_count, st.baseline_count, st.antenna_count = R, starts.size - 1, n
    st.channel_count, st.number_of_polarization_terms, st.should_invert_jones_terms = chans, 4, True
    lib.repack_input_data(ctypes.byref(st))
    want = np.argsort(b, kind="stable")
    for k, v in arrays.items():
        np.testing.assert_array_equal(v, before[k][want], err_msg=k)
    np.testing.assert_array_equal(starts, np.concatenate([[0], np.cumsum(np.bincount(b, minlength=starts.size - 1))]))
