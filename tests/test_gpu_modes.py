"""Groups outside the fast decode mode among groups inside it, on the tcgen05 path: a warp decodes a unit part by part where one of its
columns has such a group, and only there."""
import numpy as np
import pytest

from int4matmul_kernels_b200 import capi
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem
from test_gpu_stream import FORMATS, fmt_id, one_hot_problem

pytestmark = pytest.mark.gpu


# groups of 64: the first one, one in the first unit's last part, one in the middle of a unit, the last one (a unit that is only partly
# there); columns of one warp, of every other warp, of the second tile only
@pytest.mark.parametrize("groups", [(0,), (3,), (41,), (80,), (0, 17, 80)], ids=str)
@pytest.mark.parametrize("columns", [slice(5, 6), slice(0, None, 64), slice(130, 140)], ids=str)
@pytest.mark.parametrize("m", [1, 4, 32, 48, 128, 200])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_some_groups_outside_the_fast_mode(fmt, m, columns, groups):
    bits, sparse = fmt
    n, s = 81 * 64, 448
    p = oracle.make_packed_problem(bits, n, s, m, 64, sparse=sparse, seed=m)
    for i, g in enumerate(groups):
        if i % 2 == 0:
            p["zeros"][g, columns] += np.float16(0.5)                 # no integer
        else:
            p["scales"][g, columns] = -p["scales"][g, columns]        # exponent coding
    got = run_problem(p, path=capi.PATH_TCGEN05)
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], np.arange(s))
    assert_parity(got, want, bound, f"{fmt} m={m} {groups} {columns}")


@pytest.mark.parametrize("rows", [8, 64, 128])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_either_coding_at_the_limits_of_fp16(fmt, rows):
    """Columns of every sign and size of scale beside each other, -0 (linear) and the smallest numbers among them: exact weights."""
    bits, sparse = fmt
    p = one_hot_problem(bits, sparse, 128, 128, 64, 17, "fraction")
    scales = np.array([-0.0, -6e-8, -6.1e-5, -0.01, -1.0, -200.0, 0.0, 6e-8, 0.01, 1000.0], np.float16)
    zeros = np.array([0.0, -0.0, 7.0, 6e-8, -3.5, 2047.0, 0.1], np.float16)
    p["scales"] = np.ascontiguousarray(np.resize(scales, p["scales"].shape))
    p["zeros"] = np.ascontiguousarray(np.resize(zeros, p["zeros"].shape))
    w16 = oracle.dequant_w16(bits, p["q"], p["scales"], p["zeros"], p["group_size"], p["keep"])
    finite = np.isfinite(w16.astype(np.float32)).all(axis=0)
    assert finite.sum() > 100
    eye = p["x"][0]
    for lo in range(0, p["n"], rows):
        got = run_problem(dict(p, x=np.ascontiguousarray(eye[lo:lo + rows])[None], m=rows), path=capi.PATH_TCGEN05, route="mtx")[0]
        want = np.where(w16[lo:lo + rows] == 0, np.float16(0), w16[lo:lo + rows])       # (a sum that is zero has no sign of its weight)
        assert np.array_equal(got[:, finite].view(np.uint16), want[:, finite].view(np.uint16))
