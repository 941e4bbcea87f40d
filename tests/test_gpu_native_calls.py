"""The compiled fast path of the Python entries (ops, QuantLinear) against the same calls through ctypes: equal results for
everything both accept, and the same exceptions for what the entries refuse."""
import dataclasses
import threading
import time

import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops, packing, sharding
from int4matmul_kernels_b200.quantize import QuantLinear

pytestmark = pytest.mark.gpu


def both(monkeypatch, call):
    """call() through the compiled module and through ctypes."""
    assert ops.native()
    fast = call()
    with monkeypatch.context() as m:
        m.setattr(ops, "_native", False)
        slow = call()
    return fast, slow


def weights(bits, n, s, g, sparse=False):
    w = packing.synthetic_weights(bits, n, s, g, sparse=sparse, seed=bits)
    return w["matrix"], w["scales"], w["zeros"], w["mask"]


@pytest.mark.parametrize("bits,sparse", [(4, False), (3, False), (2, False), (4, True)])
@pytest.mark.parametrize("shape", [(256,), (1, 256), (5, 256), (2, 3, 256), (2, 1, 70, 256)])
def test_quant_linear_shapes(monkeypatch, bits, sparse, shape):
    m, s, z, k = weights(bits, 256, 192, 128, sparse)
    layer = QuantLinear(bits, 256, 192, 128, m, s, z, k)
    x = torch.randn(shape, generator=torch.Generator().manual_seed(1)).half().cuda()
    for inp in (x, x.float(), torch.stack([x, x], dim=-1)[..., 0]):            # as it is, converted, strided
        fast, slow = both(monkeypatch, lambda: layer(inp))
        assert fast.shape == slow.shape == (*shape[:-1], 192) and torch.equal(fast, slow)


def test_static_weights_flag_and_second_stream(monkeypatch):
    m, s, z, _ = weights(4, 512, 128, 64)
    x = torch.randn(1, 3, 512, generator=torch.Generator().manual_seed(2)).half().cuda()

    def call():
        out = torch.empty((1, 3, 128), dtype=torch.float16, device="cuda")
        ops.quant_int4_linear_mult_mtx(out, m, x, s, z, 64, None)
        return out
    want, _ = both(monkeypatch, call)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    ops.set_static_weights(True)
    try:
        with torch.cuda.stream(side):
            got = [call() for _ in range(3)]
    finally:
        ops.set_static_weights(False)
    side.synchronize()
    assert all(torch.equal(want, g) for g in got)


@pytest.mark.parametrize("mode,n_in", [(0, 1), (1, 3), (2, 2), (3, 2), (4, 2)])
def test_row_norm_operands(monkeypatch, mode, n_in):
    big = torch.randn(4, 3 * 320, generator=torch.Generator().manual_seed(3)).half().cuda()
    for args in ([big[:, i * 320:(i + 1) * 320] for i in range(n_in)], [big[:, :320].contiguous()] * n_in):
        fast, slow = both(monkeypatch, lambda: ops.row_norm(mode, *args))
        assert torch.equal(fast, slow)
    for bad in (big[:, :320].float(), big[:, ::3], big[:2, :320]):
        with pytest.raises((ValueError, ops.Int4MatmulError)):
            ops.row_norm(2, big[:, :320], bad)


def test_refusals_are_the_same(monkeypatch):
    m, s, z, _ = weights(4, 256, 128, 128)
    x = torch.zeros((1, 2, 256), dtype=torch.float16, device="cuda")
    out = torch.zeros((1, 2, 128), dtype=torch.float16, device="cuda")
    cases = [
        lambda: ops.quant_matmul(5, out, m, x, s, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x.float(), s, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x.cpu(), s, z, 128, None),
        lambda: ops.quant_matmul(4, out[..., ::2], m, x, s, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x, s[:, :64].contiguous(), z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x, s, z, 96, None),
        lambda: ops.quant_matmul(4, out, m, x, s, z, 64, None),                  # too few groups for this group size
        lambda: ops.quant_matmul(3, out, m, x, s, z, 128, None),
        lambda: ops.quant_matmul(2, out, m, x, s, z, 128, m),
        lambda: ops.quant_int4_linear_mult_vec(out, m, x, s, z, 128, None),
        # arguments of another kind: the entry's own diagnosis, not that of the compiled function's signature
        lambda: ops.quant_matmul(4, out, m, None, s, z, 128, None),
        lambda: ops.quant_matmul(4, None, m, x, s, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x.cpu().numpy(), s, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x, None, z, 128, None),
        lambda: ops.quant_matmul(4, out, m, x, s, z, None, None),
        lambda: ops.quant_matmul(4, out, m, x, s, z, 128, False),
        lambda: QuantLinear(4, 256, 128, None, m, s, z)(x),
        lambda: QuantLinear(4, 256, 128, 128, m, s, z)(None),
        lambda: ops.row_norm(2, x[0]),
        lambda: ops.row_norm(0, None),
        lambda: ops.row_norm(2, x[0], 1.0),
    ]
    for call in cases:
        seen = []
        for native in (ops.native(), False):
            with monkeypatch.context() as mp:
                mp.setattr(ops, "_native", native)
                with pytest.raises(Exception) as e:
                    call()
                seen.append((type(e.value), str(e.value)))
        assert seen[0] == seen[1]


@pytest.mark.parametrize("kind", [float, int, np.int64, torch.tensor])
def test_group_size_of_any_kind_that_int_takes(monkeypatch, kind):
    m, s, z, _ = weights(4, 256, 128, 128)
    layer = QuantLinear(4, 256, 128, kind(128), m, s, z)
    x = torch.randn((3, 256), generator=torch.Generator().manual_seed(4)).half().cuda()
    fast, slow = both(monkeypatch, lambda: layer(x))
    assert torch.equal(fast, slow) and torch.equal(fast, QuantLinear(4, 256, 128, 128, m, s, z)(x))


def test_other_threads_run_while_a_launch_waits_for_room_in_the_queue():
    m, s, z, _ = weights(4, 256, 128, 128)
    layer = QuantLinear(4, 256, 128, 128, m, s, z)
    x = torch.zeros((1, 256), dtype=torch.float16, device="cuda")
    layer(x)
    ops.row_norm(0, x)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.005)
    thread = threading.Thread(target=tick)
    thread.start()
    try:
        for call in (lambda: layer(x), lambda: ops.row_norm(0, x)):
            torch.cuda._sleep(2_000_000_000)                                    # about a second during which nothing is taken from the queue
            for _ in range(3000):
                call()
            torch.cuda.synchronize()
    finally:
        stop.set()
        thread.join()
    gap = max(b - a for a, b in zip(ticks, ticks[1:]))
    assert gap < 0.5, gap


def test_threads_that_share_a_stream_do_not_mix_their_launches():
    """Multiplies cut into K parts are two launches with sums in the stream's scratch between them (tiles of 128 and 160 rows: this
    matrix fills few pairs); beside them one-launch multiplies that share tiles through the same scratch."""
    problems = []
    lib = capi.load()
    m, s, z, _ = weights(4, 4096, 512, 128)
    layer = QuantLinear(4, 4096, 512, 128, m, s, z)
    for i, (rows, height) in enumerate(((40, 128), (100, 128), (150, 160), (300, 160), (48, 0), (8, 0))):
        x = torch.randn((rows, 4096), generator=torch.Generator().manual_seed(i)).half().cuda()

        def multiply(x=x, rows=rows, height=height):
            if not height:
                return layer(x)
            out = torch.empty((1, rows, 512), dtype=torch.float16, device="cuda")
            ops.quant_int4_linear_mult_mtx(out, m, x.unsqueeze(0), s, z, 128, None, path=capi.PATH_TCGEN05 | (height << 8))
            return out[0]
        before = lib.i4mm_launch_count()
        want = multiply()
        assert lib.i4mm_launch_count() - before == (2 if height else 1)
        assert (lib.i4mm_last_launch_schedule() == capi.K_PARTS) == bool(height)
        problems.append((multiply, want))
    torch.cuda.synchronize()
    bad = []

    def run(multiply, want):
        try:
            outs = [multiply() for _ in range(300)]
            torch.cuda.synchronize()
            bad.extend(i for i, o in enumerate(outs) if not torch.equal(o, want))
        except Exception as e:
            bad.append(e)
    threads = [threading.Thread(target=run, args=p) for p in problems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, (len(bad), bad[0])
    ops.check_device_status()


@pytest.mark.parametrize("rows", [1, 40, 300])
def test_the_first_cuda_call_of_a_thread_may_be_a_multiply(rows):
    """With weights that no call has seen, so that tensor maps are encoded, which needs the thread to have a CUDA context."""
    m, s, z, _ = weights(4, 5120, 3072, 128)
    x = torch.randn((1, rows, 5120), generator=torch.Generator().manual_seed(rows)).half().cuda()
    out, results = torch.empty((1, rows, 3072), dtype=torch.float16, device="cuda"), []
    ops.workspace(torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream())
    torch.cuda.synchronize()

    def run():
        try:
            results.append(ops.quant_int4_linear_mult_mtx(out, m, x, s, z, 128, None, path=capi.PATH_TCGEN05))
        except Exception as e:
            results.append(e)
    thread = threading.Thread(target=run)
    thread.start()
    thread.join()
    assert results == [None]
    want = torch.empty_like(out)
    ops.quant_int4_linear_mult_mtx(want, m, x, s, z, 128, None, path=capi.PATH_TCGEN05)
    assert torch.equal(out, want)


def small_stack(bits, sparse, rows):
    """Two layers of 256 (inner width 448) with weights of one format, and rows of activations."""
    cfg = sharding.StackConfig(hidden=256, mlp=448, layers=2, bits=4, group_size=64)
    stack = sharding.DecoderStack(cfg, 0, 1, "cuda", layers=0)
    stack.layers = []
    for layer in range(2):
        mats = {}
        for i, (name, n, s) in enumerate((("qkv", 256, 768), ("o", 256, 256), ("gate_up", 256, 896), ("down", 448, 256))):
            w = packing.synthetic_weights(bits, n, s, 64, sparse=sparse, seed=10 * layer + i)
            mats[name] = sharding.QuantWeights(bits, n, s, 64, w["matrix"], w["scales"], w["zeros"], w["mask"])
        stack.layers.append(mats)
    return stack, torch.randn((rows, 256), generator=torch.Generator().manual_seed(rows)).half().cuda()


@pytest.mark.parametrize("bits,sparse", [(4, False), (3, False), (2, False), (4, True)])
@pytest.mark.parametrize("rows", [1, 5, 40])
def test_stack_layers_in_one_call(monkeypatch, bits, sparse, rows):
    stack, h = small_stack(bits, sparse, rows)
    stack.forward(h)                                                    # (allocates this stream's scratch)
    lib = capi.load()
    for static in (False, True):
        ops.set_static_weights(static)
        try:
            before = lib.i4mm_launch_count()
            fast, slow = both(monkeypatch, lambda: stack.forward(h))
            assert lib.i4mm_launch_count() - before == 2 * (1 + 2 * 8)
        finally:
            ops.set_static_weights(False)
        assert torch.equal(fast, slow)
    side = torch.cuda.Stream()                                          # no scratch there yet: the single calls allocate it
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        outs = [stack.forward(h) for _ in range(2)]
    side.synchronize()
    assert all(torch.equal(o, slow) for o in outs)


def test_stack_layers_leave_everything_else_to_the_single_calls(monkeypatch):
    stack, h = small_stack(4, False, 3)
    want = stack.forward(h)
    called = []
    monkeypatch.setattr(ops, "stack_layer", lambda *a: called.append(a))        # (a layer refused: None)
    assert torch.equal(stack.forward(h), want) and len(called) == 2
    called.clear()
    stack.multiply = lambda w, x: sharding.cuda_multiply(w, x)                  # another multiply, a replaced step
    assert torch.equal(stack.forward(h), want)
    stack.multiply = sharding.cuda_multiply
    stack._linear = lambda *a: sharding.DecoderStack._linear(stack, *a)
    assert torch.equal(stack.forward(h), want) and not called
    monkeypatch.undo()
    del stack._linear
    strided = torch.stack([h, h], dim=-1)[..., 0]
    for broken in ("scales", "s", "group_size"):
        mats = dict(stack.layers[1])
        old = mats["down"]
        mats["down"] = dataclasses.replace(old, **{broken: {"scales": old.scales.float(), "s": old.s + 64, "group_size": 100}[broken]})
        other, _ = small_stack(4, False, 3)
        other.layers = [stack.layers[0], mats]
        messages = []
        for native in (True, False):
            with monkeypatch.context() as m:
                if not native:
                    m.setattr(ops, "_native", False)
                with pytest.raises((ValueError, TypeError, RuntimeError)) as e:
                    other.forward(h)
                messages.append((type(e.value), str(e.value)))
        assert messages[0] == messages[1]
    rows_apart = torch.cat([h, h], dim=1)[:, :h.shape[1]]                        # a row stride: taken by the single calls
    fast, slow = both(monkeypatch, lambda: stack.forward(rows_apart))
    assert torch.equal(fast, want) and torch.equal(slow, want)
    messages = []                                                               # an element stride: refused
    for native in (ops.native(), False):
        with monkeypatch.context() as m:
            m.setattr(ops, "_native", native)
            with pytest.raises(ValueError) as e:
                stack.forward(strided)
            messages.append(str(e.value))
    assert messages[0] == messages[1]
