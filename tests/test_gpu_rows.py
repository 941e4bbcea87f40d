"""GPU parity tests of the few-row kernel (up to 8 activation rows of a small matrix, the default route), for every format:
the edges of its steps (128 k), tiles (64 columns), K parts, row classes, dequantisation modes, and both sides of every
bound of the rule that sends calls to it."""
import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem, to_dev
from test_gpu_stream import FORMATS, fmt_id, one_hot_problem

pytestmark = pytest.mark.gpu

FEW_ROWS = 8                                       # what i4mm_last_launch_shape says after this kernel


def took_few_rows():
    return capi.load().i4mm_last_launch_shape() == FEW_ROWS


def expected_few_rows(bits, rows, n, s, adds):
    """The rule, restated."""
    width, weights = min(n, s), n * s / 2 ** 20
    if rows == 1:
        return weights <= (48 if s <= 18944 else 36) and (adds or bits == 2 or width <= 3072)
    if rows > 8 or weights > 16:
        return False
    return (n <= 131072 and (bits == 2 or width <= 3072)) if rows <= 4 else (n <= 65536 and width <= 2560)


@pytest.mark.parametrize("adds,rows,n,s,few", [
    (True, 1, 4096, 12288, "all"), (True, 1, 4096, 12352, ""),                                 # 48 Mi weights and just over
    (True, 1, 2560, 18944, "all"), (True, 1, 1984, 19008, "all"), (True, 1, 2048, 19008, ""),  # uneven tiles: 36 Mi
    (False, 1, 3072, 16384, "all"), (False, 1, 3136, 3136, "int2"), (False, 1, 3136, 8192, "int2"), (False, 1, 5120, 5120, "int2"),
    (False, 1, 16384, 3072, "all"), (False, 1, 16448, 3072, ""),
    (False, 4, 3072, 5440, "all"), (False, 4, 3072, 5504, ""), (False, 4, 3136, 3136, "int2"), (False, 2, 131072, 64, "all"),
    (False, 3, 131136, 64, ""),
    (False, 8, 2560, 6528, "all"), (False, 5, 2560, 6592, ""), (False, 5, 2624, 2624, ""), (False, 8, 65536, 64, "all"),
    (False, 6, 65600, 64, ""), (False, 8, 1024, 1024, "all"), (False, 9, 1024, 1024, "")])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_which_calls_take_it(fmt, adds, rows, n, s, few):
    bits, sparse = fmt
    dev = dict(dtype=torch.int32, device="cuda")
    matrix = torch.zeros((n // 16 if sparse else n * bits // 32, s), **dev)
    mask = torch.full((n // 32, s), 0xFFFF, **dev) if sparse else None
    x = torch.ones((1, rows, n), dtype=torch.float16, device="cuda")
    scales = torch.full((1, s), 2.0 ** -10, dtype=torch.float16, device="cuda")
    zeros = torch.full((1, s), -1.0, dtype=torch.float16, device="cuda")                       # every weight is 2^-10
    out = torch.zeros((1, rows, s), dtype=torch.float16, device="cuda")
    getattr(ops, f"quant_int{bits}_linear_mult_{'vec' if adds else 'mtx'}")(out, matrix, x, scales, zeros, -1, mask)
    assert took_few_rows() == (few == "all" or few == f"int{bits}") == expected_few_rows(bits, rows, n, s, adds)
    assert (out == torch.tensor((n // 2 if sparse else n) * 2.0 ** -10, dtype=torch.float16)).all()


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("n", [64, 192, 384])
@pytest.mark.parametrize("tiles_per_sm", [4, 8])
def test_ctas_that_walk_several_column_tiles(fmt, m, n, tiles_per_sm):
    """More column tiles than CTAs fit on the GPU, with fewer 128-k steps per tile than a CTA has warps: copies run ahead
    over tile borders and the sums' memory is used again."""
    bits, sparse = fmt
    s = 64 * (tiles_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + tiles_per_sm // 4 * 2 - 1)
    p = oracle.make_packed_problem(bits, n, s, m, 64, sparse=sparse, seed=n + m)
    rng = np.random.default_rng(1)
    cols = np.unique(np.concatenate([np.arange(192), s - 1 - np.arange(192), rng.integers(0, s, 400)]))
    w = {k: to_dev(p[k]) if p[k] is not None else None for k in ("matrix", "mask", "scales", "zeros", "x")}
    outs = []
    for path in (capi.PATH_AUTO, capi.PATH_STATIC_WEIGHTS, capi.PATH_AUTO):
        outs.append(torch.empty((1, m, s), dtype=torch.float16, device="cuda"))
        getattr(ops, f"quant_int{bits}_linear_mult_mtx")(outs[-1], w["matrix"], w["x"], w["scales"], w["zeros"], 64, w["mask"], path=path)
        assert took_few_rows() == expected_few_rows(bits, m, n, s, False)
    torch.cuda.synchronize()
    assert expected_few_rows(bits, m, n, s, False) or (m > 1 and n * s > 2 ** 24)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], cols)
    assert_parity(outs[0].cpu().numpy()[..., cols], want, bound, f"{fmt} m={m} {n}x{s}")


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
        assert took_few_rows()
        assert np.array_equal(got.view(np.uint16), w16[lo:lo + rows].view(np.uint16)), (fmt, kind, lo)


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("m", [1, 2, 4, 5, 8])
@pytest.mark.parametrize("n,s,g", [(64, 64, 64), (128, 192, 64), (320, 128, 64), (1024, 320, 128), (1088, 64, 192),
                                   (2048, 1024, -1), (2560, 4160, 128), (4096, 4096, 128), (4096, 4160, 128), (8256, 5184, 256)])
def test_parity_over_sizes(fmt, m, n, s, g):
    bits, sparse = fmt
    p = oracle.make_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p)
    assert took_few_rows() == expected_few_rows(bits, m, n, s, m == 1)
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
    assert took_few_rows()
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
    assert took_few_rows() and np.isfinite(got[0]).all()
    assert (np.isnan(got[1]).all() if np.isnan(value) else (got[1] == np.float16(value)).all())


def test_scratch_is_zero_again_after_shared_tiles():
    p = oracle.make_problem(4, 16384, 64, 8, 128, seed=9)
    run_problem(p)
    assert took_few_rows()
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0
