"""16:32 weights with zero-points around the bounds of the fast decode, which XORs them into the nibbles: exact weights."""
import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops, packing
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem
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


@pytest.mark.parametrize("m", [1, 40, 64, 100])
@pytest.mark.parametrize("zeros", [(128, 256), (100, 160), (0, 256)])
def test_zero_points_of_both_fast_decodes_beside_each_other(m, zeros):
    """The decode for zero-points up to 255 keeps them in the place of the eighth nibble: mask bytes with none, one, seven and all of eight kept."""
    n, s = 512, 192
    p = oracle.make_packed_problem(4, n, s, m, 64, sparse=True, seed=m)
    rng = np.random.default_rng(m)
    p["zeros"] = rng.integers(*zeros, size=p["zeros"].shape).astype(np.float16)
    bytes_kept = np.array([[0x00, 0xFF, 0x00, 0xFF], [0xFF, 0x01, 0xFE, 0x00], [0x80, 0x7F, 0xFF, 0x00], [0x55, 0xAA, 0x0F, 0xF0]], np.uint8)
    p["mask"] = np.where(rng.random((n // 32, s)) < 0.5, bytes_kept.view(np.int32)[rng.integers(0, 4, (n // 32, s)), 0], p["mask"])
    got = run_problem(p, path=capi.PATH_TCGEN05, route="mtx")
    want, bound = oracle.expected_columns(4, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], np.arange(s))
    assert_parity(got, want, bound, f"m={m} {zeros}")


def test_zero_points_up_to_255_cost_little_more_than_those_up_to_127():
    """48 rows 16384 x 16384: 1.29 times the time; without a fast decode of their own 1.53 (before the masks of that one were made cheaper, 1.67)."""
    w = packing.synthetic_weights(4, 16384, 16384, 64, sparse=True, seed=1)
    x = torch.randn((1, 48, 16384), generator=torch.Generator().manual_seed(1)).half().cuda()
    out = torch.empty((1, 48, 16384), dtype=torch.float16, device="cuda")

    def time_of(zero):
        zeros = torch.full_like(w["zeros"], zero)
        times = []
        for _ in range(12):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(10):
                ops.quant_int4_linear_mult_mtx(out, w["matrix"], x, w["scales"], zeros, 64, w["mask"])
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)
    assert time_of(200) < 1.41 * time_of(100)
