"""Groups outside the fast decode mode among groups inside it, on the tcgen05 path: a warp decodes a unit part by part where one of its
columns has such a group, and only there."""
import numpy as np
import pytest

from int4matmul_kernels_b200 import capi
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem
from test_gpu_stream import FORMATS, fmt_id

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
