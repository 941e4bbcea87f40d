"""GPU parity tests of the few-row tcgen05 shapes (2..32 rows) where column tiles are shared: the owner of a tile sums its partners'
shares with every warpgroup, some rows each."""
import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem
from test_gpu_stream import FORMATS, fmt_id

pytestmark = pytest.mark.gpu
P = capi.PATH_TCGEN05


# one 256-k unit per CTA and as many partners as units (16384 x 64); a last unit that is only partly there; tiles cut in two or
# three with a CTA in the middle (19 and 75 tiles of 8 units); whole tiles after shared ones (300 tiles); S % 128 = 64
@pytest.mark.parametrize("n,s,g", [(16384, 64, 128), (8256, 320, 192), (2048, 2432, -1), (2048, 9536, 64), (512, 38400, 128)])
@pytest.mark.parametrize("m", [2, 3, 4, 5, 9, 16, 17, 31, 32])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_shared_tiles(fmt, m, n, s, g):
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p, path=P)
    assert capi.load().i4mm_last_launch_shape() == (16 if m <= 16 else 32)
    cols = np.unique(np.concatenate([np.arange(64), s - 1 - np.arange(64), np.random.default_rng(m).integers(0, s, 100)]))
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], g, p["x"], cols)
    assert_parity(got[..., cols], want, bound, f"{fmt} m={m} {n}x{s} g{g}")
    again = run_problem(p, path=P)
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("batch", [2, 7, 16, 32])
def test_matvec_route_adds_into_outs(fmt, batch):
    bits, sparse = fmt
    p = oracle.make_problem(bits, 4096, 192, 1, 128, sparse=sparse, batch=batch, seed=37)
    base = np.random.default_rng(2).standard_normal((batch, 1, 192)).astype(np.float16)
    got = run_problem(p, path=P, outs_in=base)
    want, _, bound = oracle.expected(p, outs_in=base)
    assert_parity(got, want, bound, f"accumulate {fmt}")
