"""Every multiply may be launched while the kernel before it is still finishing; without the static-weights promise nothing
may be read before that kernel has completed.  The preceding kernels here write the weight-side tensors."""
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops, packing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,sparse", [(4, False), (3, False), (4, True)])
@pytest.mark.parametrize("m,path", [(1, 0), (1, 2), (8, 0), (8, 2), (24, 0), (64, 0), (200, 0)])
def test_weights_written_by_the_preceding_kernel_are_seen(bits, sparse, m, path):
    n, s = 2048, 1536
    w = [packing.synthetic_weights(bits, n, s, 128, sparse=sparse, seed=i) for i in range(2)]
    # scales from a row-norm launch: that kernel lets its successor start before it has written anything
    raw = [torch.rand((n // 128, s), generator=torch.Generator().manual_seed(i)).half().cuda() * 0.01 for i in range(2)]
    x = torch.randn((1, m, n), generator=torch.Generator().manual_seed(5)).half().cuda()
    matrix = w[0]["matrix"].clone()

    def step(i, sync):
        matrix.copy_(w[i]["matrix"])
        scales = ops.row_norm(0, raw[i])
        if sync:
            torch.cuda.synchronize()
        out = torch.empty((1, m, s), dtype=torch.float16, device="cuda")
        getattr(ops, f"quant_int{bits}_linear_mult_mtx")(out, matrix, x, scales, w[i]["zeros"], 128, w[i]["mask"], path=path)
        assert (capi.load().i4mm_last_launch_shape() == 8) == (path == 0 and m <= 8)      # few-row kernel
        return out
    want = [step(i, True) for i in range(2)]
    torch.cuda.synchronize()
    got = [step(i % 2, False) for i in range(40)]
    torch.cuda.synchronize()
    bad = [i for i, o in enumerate(got) if not torch.equal(o, want[i % 2])]
    assert not bad, bad


def _multiply(w, x, scales=None, path=0):
    out = torch.empty((1, x.shape[1], w["matrix"].shape[1]), dtype=torch.float16, device="cuda")
    ops.quant_int4_linear_mult_mtx(out, w["matrix"], x, w["scales"] if scales is None else scales, w["zeros"], 128, w["mask"], path=path)
    return out


@pytest.mark.parametrize("between", ["row_norm", 1, 8, 24, 64, 200])
@pytest.mark.parametrize("m,s", [(1, 1536), (8, 1536), (8, 12288), (64, 1536), (200, 1536)])
def test_the_promise_is_about_the_preceding_kernel_only(between, m, s):
    """A kernel writes scales, another one follows, then a multiply with the static-weights promise reads those scales: the
    kernel between has not written them, so the promise holds, and the call must see them complete.  Ahead of all three runs
    a long kernel, which a successor let through too early would overtake."""
    n = 2048
    long_w, other = (packing.synthetic_weights(4, 4096, 8192, 128, seed=8), packing.synthetic_weights(4, n, 1024, 128, seed=9))
    w = packing.synthetic_weights(4, n, s, 128, seed=1)
    gen = torch.Generator().manual_seed(5)
    long_x = torch.randn((1, 512, 4096), generator=gen).half().cuda()
    x = torch.randn((1, m, n), generator=gen).half().cuda()
    raw = [torch.rand((n // 128, s), generator=torch.Generator().manual_seed(i)).half().cuda() * 0.01 for i in range(2)]
    between_x = torch.randn((1, between if between != "row_norm" else 1, n), generator=gen).half().cuda()

    def step(i, sync):
        y = _multiply(long_w, long_x)
        scales = ops.row_norm(0, raw[i])
        if sync:
            torch.cuda.synchronize()
        other_out = ops.row_norm(0, between_x[0]) if between == "row_norm" else _multiply(other, between_x)
        return _multiply(w, x, scales, path=capi.PATH_STATIC_WEIGHTS), y, other_out
    want = [step(i, True)[0] for i in range(2)]
    torch.cuda.synchronize()
    got = [step(i % 2, False)[0] for i in range(20)]
    torch.cuda.synchronize()
    bad = [i for i, o in enumerate(got) if not torch.equal(o, want[i % 2])]
    assert not bad, bad
    ops.check_device_status()
