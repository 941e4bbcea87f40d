"""GPU parity tests of the few-row kernel (up to 8 activation rows of a small matrix, the default route), for every format:
the edges of its steps (128 k), tiles (64 columns), K parts, row classes, dequantisation modes and of the rule itself."""
import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem
from test_gpu_stream import FORMATS, fmt_id, one_hot_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("rows", [3, 8])
@pytest.mark.parametrize("kind", ["integer", "fraction", "large", "exponent"])
def test_dequantised_weights_are_bit_exact(fmt, rows, kind):
    """x = rows of the identity: the outputs are rows of the fp16 weight matrix, exactly, in every mode."""
    bits, sparse = fmt
    p = one_hot_problem(bits, sparse, 192, 128, 64, 11, "integer" if kind == "exponent" else kind,
                        exponent_frac=0.5 if kind == "exponent" else 0.0)
    w16 = oracle.dequant_w16(bits, p["q"], p["scales"], p["zeros"], p["group_size"], p["keep"])
    eye = p["x"][0]
    for lo in range(0, p["n"], rows):
        q = dict(p, x=np.ascontiguousarray(eye[lo:lo + rows])[None], m=min(rows, p["n"] - lo))
        got = run_problem(q, route="mtx")[0]
        assert np.array_equal(got.view(np.uint16), w16[lo:lo + rows].view(np.uint16)), (fmt, kind, lo)


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("m", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("n,s,g", [(64, 64, 64), (128, 192, 64), (320, 128, 64), (1024, 320, 128), (1088, 64, 192),
                                   (2048, 1024, -1), (4096, 4096, 128), (4096, 4160, 128), (8256, 5184, 256)])
def test_parity_over_sizes(fmt, m, n, s, g):
    bits, sparse = fmt
    p = oracle.make_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p)
    want, _, bound = oracle.expected(p, outs_in=np.zeros((1, 1, s), np.float16) if m == 1 else None)
    assert_parity(got, want, bound, f"{fmt} m={m} {n}x{s} g{g}")
    again = run_problem(p)
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("batch", [1, 6, 8])
def test_matvec_route_adds_into_outs(fmt, batch):
    bits, sparse = fmt
    p = oracle.make_problem(bits, 2048, 256, 1, 128, sparse=sparse, batch=batch, seed=31)
    base = np.random.default_rng(1).standard_normal((batch, 1, 256)).astype(np.float16)
    got = run_problem(p, outs_in=base)
    want, _, bound = oracle.expected(p, outs_in=base)
    assert_parity(got, want, bound, f"accumulate {fmt}")


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_activations_reach_every_output(value):
    p = oracle.make_problem(4, 512, 128, 2, 128, seed=3)
    p["q"][:] = 15
    p["zeros"][:] = 1
    p["matrix"] = oracle.pack_dense_pow2(4, p["q"])
    p["x"][0, 1, 300] = value
    got = run_problem(p)[0]
    assert np.isfinite(got[0]).all()
    assert (np.isnan(got[1]).all() if np.isnan(value) else (got[1] == np.float16(value)).all())


def test_scratch_is_zero_again_after_shared_tiles():
    from int4matmul_kernels_b200 import ops
    p = oracle.make_problem(4, 16384, 64, 8, 128, seed=9)
    run_problem(p)
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0
    assert capi.load().i4mm_last_launch_shape() == 16
