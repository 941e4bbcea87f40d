"""Every multiply may be launched while the kernel before it is still finishing; without the static-weights promise nothing
may be read before that kernel has completed.  The preceding kernels here write the weight-side tensors."""
import pytest
import torch

from int4matmul_kernels_b200 import ops, packing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,sparse", [(4, False), (3, False), (4, True)])
@pytest.mark.parametrize("m", [1, 8, 24, 64, 200])
def test_weights_written_by_the_preceding_kernel_are_seen(bits, sparse, m):
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
        getattr(ops, f"quant_int{bits}_linear_mult_mtx")(out, matrix, x, scales, w[i]["zeros"], 128, w[i]["mask"])
        return out
    want = [step(i, True) for i in range(2)]
    torch.cuda.synchronize()
    got = [step(i % 2, False) for i in range(40)]
    torch.cuda.synchronize()
    bad = [i for i, o in enumerate(got) if not torch.equal(o, want[i % 2])]
    assert not bad, bad
