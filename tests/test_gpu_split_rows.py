"""GPU parity tests of the few-row tcgen05 shapes (1..128 rows a tile) where column tiles are shared: the owner of a tile sums its partners'
shares, with its epilogue warps alone or with every warpgroup, some rows each (dense int4 with up to 3 rows runs in another k order)."""
import ctypes

import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops
from oracle import reference_oracle as oracle

from helpers import assert_parity, run_problem, to_dev
from test_gpu_stream import FORMATS, fmt_id

pytestmark = pytest.mark.gpu
P = capi.PATH_TCGEN05
# schedules of the weight-streaming shape (up to 148 CTAs a tile)
STREAMED = (capi.STREAM_EQUAL_RANGES, capi.STREAM_WHOLE_TILES, *range(capi.STREAM_CTAS_PER_TILE + 2, capi.STREAM_CTAS_PER_TILE + 149))


# By the CTAs of 148 SMs: one 256-k unit per CTA and as many partners as units (16384 x 64); a last unit that is only partly there
# (8256 x 320); tiles shared by 7 or 8 CTAs, of which most hold one unit (19 tiles of 8 units); by 2 or 3, with a CTA in the middle
# (75 tiles of 8 units); whole tiles after shared ones (300 tiles of 2 units); S % 128 = 64.  Up to 6 rows of tiles whose other shares
# all came early in their CTAs' ranges are summed by the epilogue warps alone (two of the 75 and the 300 tiles)
@pytest.mark.parametrize("n,s,g", [(16384, 64, 128), (8256, 320, 192), (2048, 2432, -1), (2048, 9536, 64), (512, 38400, 128)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16, 17, 31, 32])
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


@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
@pytest.mark.parametrize("batch", [1, 2, 4, 16, 32])
def test_matvec_route_adds_into_outs_of_several_tiles_per_cta(fmt, batch):
    """Tiles that a CTA sums before its last one (300 tiles of 2 units) read the old outputs as well."""
    bits, sparse = fmt
    n, s = 512, 38400
    p = oracle.make_packed_problem(bits, n, s, 1, 64, sparse=sparse, batch=batch, seed=41)
    base = np.random.default_rng(3).standard_normal((batch, 1, s)).astype(np.float16)
    got = run_problem(p, path=P, outs_in=base, route="vec")
    cols = np.unique(np.concatenate([np.arange(0, s, 128), np.arange(127, s, 128)]))         # both edges of every tile
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base[..., cols]))
    assert_parity(got[..., cols], want, bound, f"accumulate {fmt}")


# shared tiles; whole tiles and shared ones; a few-row kernel's call (path 0)
@pytest.mark.parametrize("n,s", [(8256, 320), (512, 38400), (2048, 1024)])
@pytest.mark.parametrize("m", [1, 2, 5, 16, 17, 32, 48])
@pytest.mark.parametrize("path", [capi.PATH_AUTO, P])
@pytest.mark.parametrize("fmt", [(4, False), (4, True)], ids=fmt_id)
def test_several_destinations_hold_the_same_bits(fmt, path, m, n, s):
    """Three ordinary local buffers as the gathering entry's destinations, with rows longer than S: each holds what one call with one
    destination gives, and nothing else is written."""
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, 64, sparse=sparse, seed=n + m)
    w = {k: to_dev(p[k]) if p[k] is not None else None for k in ("matrix", "mask", "scales", "zeros", "x")}
    want = torch.empty((1, m, s), dtype=torch.float16, device="cuda")
    getattr(ops, f"quant_int{bits}_linear_mult_mtx")(want, w["matrix"], w["x"], w["scales"], w["zeros"], 64, w["mask"], path=path)
    lib, ld, stream = capi.load(), s + 64, torch.cuda.current_stream()
    shape = lib.i4mm_last_launch_shape()
    bufs = [torch.full((m, ld), 7.0, dtype=torch.float16, device="cuda") for _ in range(3)]
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), stream)
    status = lib.i4mm_quant_matmul_gather(bits, path, (ctypes.c_void_p * 3)(*[b.data_ptr() for b in bufs]), 3, ld, 1, 0, 1,
                                          w["matrix"].data_ptr(), w["mask"].data_ptr() if sparse else None, w["x"].data_ptr(),
                                          w["scales"].data_ptr(), w["zeros"].data_ptr(), m, n, s, p["scales"].shape[0], 64,
                                          ws.data_ptr(), ws.numel(), stream.cuda_stream)
    assert status == capi.OK and lib.i4mm_last_launch_shape() == shape
    torch.cuda.synchronize()
    for b in bufs:
        assert torch.equal(b[:, :s], want[0]) and (b[:, s:] == 7.0).all()


# more than 64 rows with several destinations: the whole-tile shapes, in K parts (8256 x 320) and in whole tiles (512 x 38400), single CTAs and pairs
@pytest.mark.parametrize("n,s,schedule", [(8256, 320, capi.K_PARTS), (512, 38400, capi.WHOLE_TILES)])
@pytest.mark.parametrize("m", [100, 300])
def test_several_destinations_of_many_rows(m, n, s, schedule):
    p = oracle.make_packed_problem(4, n, s, m, 64, seed=n + m)
    w = {k: to_dev(p[k]) for k in ("matrix", "scales", "zeros", "x")}
    lib, ld, stream = capi.load(), s + 64, torch.cuda.current_stream()
    bufs = [torch.full((m, ld), 7.0, dtype=torch.float16, device="cuda") for _ in range(3)]
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), stream)
    status = lib.i4mm_quant_matmul_gather(4, P, (ctypes.c_void_p * 3)(*[b.data_ptr() for b in bufs]), 3, ld, 1, 0, 1, w["matrix"].data_ptr(), None,
                                          w["x"].data_ptr(), w["scales"].data_ptr(), w["zeros"].data_ptr(), m, n, s, p["scales"].shape[0], 64,
                                          ws.data_ptr(), ws.numel(), stream.cuda_stream)
    assert status == capi.OK and lib.i4mm_last_launch_schedule() == schedule
    assert (lib.i4mm_last_launch_shape() % 10000 > 1000) == (m >= 128)
    torch.cuda.synchronize()
    cols = np.unique(np.concatenate([np.arange(64), s - 1 - np.arange(64), np.random.default_rng(m).integers(0, s, 60)]))
    want, bound = oracle.expected_columns(4, p["matrix"], None, p["scales"], p["zeros"], 64, p["x"], cols)
    assert_parity(bufs[0][:, :s].cpu().numpy()[None, :, cols], want, bound, f"{n}x{s} m={m}")
    for b in bufs:
        assert torch.equal(b[:, :s], bufs[0][:, :s]) and (b[:, s:] == 7.0).all()
    assert int(ws.count_nonzero()) == 0


# 33..64 rows: every number of row groups per warpgroup (groups of 4 rows, ragged last ones), on the same sizes
@pytest.mark.parametrize("n,s,g", [(16384, 64, 128), (8256, 320, 192), (2048, 2432, -1), (2048, 9536, 64), (512, 38400, 128)])
@pytest.mark.parametrize("m", [33, 36, 47, 48, 49, 61, 64])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_shared_tiles_of_33_to_64_rows(fmt, m, n, s, g):
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p, path=P)
    assert capi.load().i4mm_last_launch_shape() == 64
    cols = np.unique(np.concatenate([np.arange(64), s - 1 - np.arange(64), np.random.default_rng(m).integers(0, s, 60)]))
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], g, p["x"], cols)
    assert_parity(got[..., cols], want, bound, f"{fmt} m={m} {n}x{s} g{g}")
    again = run_problem(p, path=P)
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("n,s", [(512, 38400), (4096, 192)])
@pytest.mark.parametrize("batch", [33, 50, 64])
def test_matvec_route_adds_33_to_64_rows_into_outs(batch, n, s):
    p = oracle.make_packed_problem(4, n, s, 1, 64, batch=batch, seed=43)
    base = np.random.default_rng(4).standard_normal((batch, 1, s)).astype(np.float16)
    got = run_problem(p, path=P, outs_in=base, route="vec")
    cols = np.unique(np.concatenate([np.arange(0, s, 128), np.arange(63, s, 64)]))
    want, bound = oracle.expected_columns(4, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base[..., cols]))
    assert_parity(got[..., cols], want, bound, f"accumulate {batch} {n}x{s}")


@pytest.mark.parametrize("m", [1, 4, 7, 16, 32, 50, 100])
def test_partial_sums_of_zero_infinity_and_nan_are_delivered(m):
    """A shared tile's partial sums travel as words that are never zero: rows of zeros (of either sign), infinities and NaN."""
    n, s = 8192, 320
    p = oracle.make_packed_problem(4, n, s, m, 128, seed=m)
    p["zeros"][:] = 8                                                 # no weight row is all of one sign
    x = p["x"]
    for row in range(m):
        kind = (row + (m == 1)) % 5
        if kind == 0:
            x[0, row] = 0.0
        elif kind == 1:
            x[0, row] = -0.0
        elif kind == 2:
            x[0, row, n // 2] = np.inf
        elif kind == 3:
            x[0, row, 3] = np.nan
    got = run_problem(p, path=P, route="mtx")[0]
    want, bound = oracle.expected_columns(4, p["matrix"], p["mask"], p["scales"], p["zeros"], 128, x, np.arange(s))
    for row in range(m):
        kind = (row + (m == 1)) % 5
        if kind <= 1:
            assert not got[row].any()
        elif kind == 3:
            assert np.isnan(got[row]).all()
        elif kind == 2:
            assert np.array_equal(np.isnan(got[row]), np.isnan(want[0, row])) and np.array_equal(np.isposinf(got[row]), np.isposinf(want[0, row]))
        else:
            assert_parity(got[None, row:row + 1], want[:, row:row + 1], bound[:, row:row + 1], f"row {row}")
    ops.check_device_status()
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("m", [1, 5, 32])
def test_the_streaming_path_leaves_the_scratch_to_the_other_kernels(m):
    p = oracle.make_packed_problem(4, 8192, 320, m, 128, seed=m)
    want = run_problem(p, path=P)
    assert_parity(run_problem(p, path=capi.PATH_STREAM), want, np.full(want.shape, np.abs(want.astype(np.float32)).max()), "streaming path")
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0
    assert np.array_equal(run_problem(p, path=P).view(np.uint16), want.view(np.uint16))


# 65..128 rows: tiles shared by up to 64 and by 3 or 4 CTAs, a CTA that goes on to the next tile, two accumulators in turn (1.35 tiles a
# CTA), S % 128 = 64; and whole tiles of the other shape (75 tiles of 16 units)
@pytest.mark.parametrize("n,s,g,m", [(16384, 64, 128, m) for m in (65, 100, 128)] + [(8256, 320, 192, m) for m in (65, 77, 127, 128)] +
                         [(4096, 5056, -1, m) for m in (66, 96, 128)] + [(8192, 9536, 64, 97), (2048, 9536, 64, 97)] + [(4096, 25600, 128, m) for m in (65, 127)])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_shared_tiles_of_65_to_128_rows(fmt, n, s, g, m):
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p, path=P)
    assert capi.load().i4mm_last_launch_shape() == 128
    whole = (n, s) == (2048, 9536)                     # 75 tiles of 16 units: whole ones of the other shape
    assert capi.load().i4mm_last_launch_schedule() in ((capi.WHOLE_TILES,) if whole else STREAMED)
    cols = np.unique(np.concatenate([np.arange(64), s - 1 - np.arange(64), np.random.default_rng(m).integers(0, s, 60)]))
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], g, p["x"], cols)
    assert_parity(got[..., cols], want, bound, f"{fmt} m={m} {n}x{s} g{g}")
    again = run_problem(p, path=P)
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0


@pytest.mark.parametrize("n,s", [(4096, 25600), (8192, 192)])
@pytest.mark.parametrize("batch", [65, 128])
def test_matvec_route_adds_65_to_128_rows_into_outs(batch, n, s):
    p = oracle.make_packed_problem(4, n, s, 1, 64, batch=batch, seed=47)
    base = np.random.default_rng(5).standard_normal((batch, 1, s)).astype(np.float16)
    got = run_problem(p, path=P, outs_in=base, route="vec")
    cols = np.unique(np.concatenate([np.arange(0, s, 128), np.arange(63, s, 64)]))
    want, bound = oracle.expected_columns(4, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base[..., cols]))
    assert_parity(got[..., cols], want, bound, f"accumulate {batch} {n}x{s}")


# More than 128 rows: row tiles of 128 beside each other (a ragged last one of 1, 5, 72 and 122 rows), a CTA whose range goes over from
# one row tile to the next, two and three tiles a CTA; K in one unit and with a last unit that is only partly there
@pytest.mark.parametrize("n,s,g,m", [(8256, 320, 192, 133), (8192, 2432, -1, 200), (8192, 2432, 64, 257), (4096, 5056, 64, 129), (13824, 2048, 128, 378)])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_row_tiles_of_the_streaming_shape(fmt, n, s, g, m):
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, g, sparse=sparse, seed=n + s + m)
    got = run_problem(p, path=P)
    assert capi.load().i4mm_last_launch_shape() == 128 and capi.load().i4mm_last_launch_schedule() in STREAMED
    cols = np.unique(np.concatenate([np.arange(32), s - 1 - np.arange(32), np.random.default_rng(m).integers(0, s, 40)]))
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], g, p["x"], cols)
    assert_parity(got[..., cols], want, bound, f"{fmt} m={m} {n}x{s} g{g}")
    again = run_problem(p, path=P)
    assert np.array_equal(got.view(np.uint16), again.view(np.uint16))
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0


def test_matvec_route_adds_more_than_128_rows_into_outs():
    n, s, batch = 13824, 2048, 200
    p = oracle.make_packed_problem(4, n, s, 1, 64, batch=batch, seed=53)
    base = np.random.default_rng(6).standard_normal((batch, 1, s)).astype(np.float16)
    got = run_problem(p, path=P, outs_in=base, route="vec")
    assert capi.load().i4mm_last_launch_shape() == 128
    cols = np.unique(np.concatenate([np.arange(0, s, 128), np.arange(63, s, 64)]))
    want, bound = oracle.expected_columns(4, p["matrix"], p["mask"], p["scales"], p["zeros"], 64, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base[..., cols]))
    assert_parity(got[..., cols], want, bound, f"accumulate {batch} {n}x{s}")


# The same number of CTAs for every tile: 20 tiles of 13 units (26 of 128 k), the last one only partly there, cut into parts that are not
# equal; 37 tiles of which the last is half a one; 7 tiles; one tile cut into far fewer parts than units
@pytest.mark.parametrize("n,s", [(3264, 2560), (3264, 4672), (6400, 896), (16384, 128)])
@pytest.mark.parametrize("m", [1, 3, 4, 16, 20, 50, 100, 128])
@pytest.mark.parametrize("fmt", FORMATS, ids=fmt_id)
def test_tiles_of_as_many_ctas_each(fmt, m, n, s):
    bits, sparse = fmt
    p = oracle.make_packed_problem(bits, n, s, m, 192, sparse=sparse, seed=n + s + m)
    base = np.random.default_rng(m).standard_normal((1, 1, s)).astype(np.float16) if m == 1 else None
    kw = dict(outs_in=base, route="vec") if m == 1 else {}
    got = run_problem(p, path=P, **kw)
    assert capi.load().i4mm_last_launch_schedule() > capi.STREAM_CTAS_PER_TILE
    cols = np.unique(np.concatenate([np.arange(32), s - 1 - np.arange(32), np.random.default_rng(m).integers(0, s, 60)]))
    want, bound = oracle.expected_columns(bits, p["matrix"], p["mask"], p["scales"], p["zeros"], 192, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base[..., cols]) if m == 1 else None)
    assert_parity(got[..., cols], want, bound, f"{fmt} m={m} {n}x{s}")
    assert np.array_equal(got.view(np.uint16), run_problem(p, path=P, **kw).view(np.uint16))
    ws = ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    assert int(ws.count_nonzero()) == 0
