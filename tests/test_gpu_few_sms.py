"""Multiplies while another stream's kernel holds nearly all SMs: the CTAs that share a tile cannot be resident together then, and a launch has
to get through all the same, with the same results."""
import time

import numpy as np
import pytest
import torch

from int4matmul_kernels_b200 import capi, ops
from oracle import reference_oracle as oracle

from helpers import assert_parity, device_problem

pytestmark = pytest.mark.gpu

HOLD_SECONDS, HOLD_SHARED_BYTES = 0.6, 200 * 1024
_HOLD = """
extern "C" __global__ void hold(int ms) {
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < 20000000; ++i) {                       // ends by itself, whatever the timer says
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t - t0 > 1000000ull * ms) break;
        __nanosleep(1000);
    }
}
"""


@pytest.fixture(scope="module")
def hold():
    """hold(sms): a kernel on a stream of its own that takes the shared memory of `sms` SMs for HOLD_SECONDS; its end as an event."""
    kernel = torch.cuda._compile_kernel(_HOLD, "hold")
    kernel.set_shared_memory_config(HOLD_SHARED_BYTES)
    stream = torch.cuda.Stream()

    def start(sms):
        kernel(grid=(sms, 1, 1), block=(32, 1, 1), args=[int(HOLD_SECONDS * 1000)], shared_mem=HOLD_SHARED_BYTES, stream=stream)
        end = torch.cuda.Event()
        end.record(stream)
        time.sleep(0.05)                                       # its blocks are resident
        return end
    return start


# one tile cut into parts; three tiles; more tiles than half of the CTAs, with CTAs that go on to a next tile; two accumulators in turn; row tiles
# beside each other; old outputs.  (Rows up to 32: one CTA of a tile waits for the others; above: those that sum wait for each other.)
@pytest.mark.parametrize("n,s,m", [(16384, 64, 1), (16384, 128, 16), (4096, 9536, 5), (16384, 64, 33), (16384, 128, 64), (4096, 9536, 48), (16384, 128, 65),
                                   (8256, 320, 100), (4096, 5056, 128), (4096, 25600, 127), (13824, 2048, 378)])
@pytest.mark.parametrize("free", [1, 5])
def test_a_launch_gets_through_beside_a_kernel_that_holds_the_other_sms(hold, free, n, s, m):
    p = oracle.make_packed_problem(4, n, s, m, 192, seed=n + s + m)
    w = device_problem(p)
    dev, stream = torch.device("cuda", torch.cuda.current_device()), torch.cuda.current_stream()
    base = torch.randn((1, m, s), generator=torch.Generator().manual_seed(m)).half().cuda() if m == 1 else None

    def multiply(out):
        (ops.quant_int4_linear_mult_vec if m == 1 else ops.quant_int4_linear_mult_mtx)(
            out, w["matrix"], w["x"], w["scales"], w["zeros"], 192, None, path=capi.PATH_TCGEN05)
        return out
    quiet = multiply(base.clone() if m == 1 else torch.empty((1, m, s), dtype=torch.float16, device=dev))
    assert capi.load().i4mm_last_launch_schedule() == capi.STREAM_EQUAL_RANGES or capi.load().i4mm_last_launch_schedule() > capi.STREAM_CTAS_PER_TILE
    beside = base.clone() if m == 1 else torch.empty_like(quiet)
    torch.cuda.synchronize()
    cols = np.unique(np.concatenate([np.arange(16), s - 1 - np.arange(16)]))
    want, bound = oracle.expected_columns(4, p["matrix"], None, p["scales"], p["zeros"], 192, p["x"], cols,
                                          outs_in=np.ascontiguousarray(base.cpu().numpy()[..., cols]) if m == 1 else None)
    assert_parity(quiet.cpu().numpy()[..., cols], want, bound, f"{n}x{s} m={m}")

    held = hold(torch.cuda.get_device_properties(dev).multi_processor_count - free)
    multiply(beside)
    stream.synchronize()
    before_the_end = not held.query()
    held.synchronize()
    assert before_the_end, "the multiply waited for the other kernel"
    assert torch.equal(beside, quiet)
    ops.check_device_status()
    assert int(ops.workspace(dev, stream).count_nonzero()) == 0
