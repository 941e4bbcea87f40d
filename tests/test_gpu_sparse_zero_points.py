"""16:32 weights with zero-points around the bounds of the fast decode, which XORs them into the nibbles: exact weights."""
import numpy as np
import pytest

from int4matmul_kernels_b200 import capi
from oracle import reference_oracle as oracle

from helpers import run_problem
from test_gpu_stream import one_hot_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", [capi.PATH_AUTO, capi.PATH_TCGEN05])
@pytest.mark.parametrize("rows", [8, 64, 128])
@pytest.mark.parametrize("zero", [0, 1, 15, 16, 126, 127, 128, 255, 256])
def test_dropped_weights_are_zero_and_kept_ones_exact(path, rows, zero):
    p = one_hot_problem(4, True, 128, 128, 64, 11, "integer")
    p["zeros"][:] = zero
    w16 = oracle.dequant_w16(4, p["q"], p["scales"], p["zeros"], p["group_size"], p["keep"])
    eye = p["x"][0]
    for lo in range(0, p["n"], rows):
        got = run_problem(dict(p, x=np.ascontiguousarray(eye[lo:lo + rows])[None], m=rows), path=path, route="mtx")[0]
        assert np.array_equal(got.view(np.uint16), w16[lo:lo + rows].view(np.uint16))
