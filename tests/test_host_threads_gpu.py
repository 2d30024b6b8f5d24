"""The native entry points give up the interpreter lock: while one thread's launch waits for a place in a full queue, the others run."""

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["entry point", "lane_matmul", "prefill_matmul"])
def test_a_full_queue_stops_no_other_thread(lib, call):
    from tensorfold_b200 import _lib, lane_qmm, prefill_qmm, synthetic

    x = torch.randn((1, 128), device="cuda").to(torch.bfloat16)
    w = synthetic.random_q4(torch.Generator(device="cuda").manual_seed(1), 256, 128, 64, "cuda")
    wide = prefill_qmm.tile_weight(*lane_qmm.untile_weight(w), 64)
    packed = lane_qmm.new_packed(1, 128, 64, x.device)
    one = {"entry point": lambda: lib.tf_pack_rows(x, packed.data, None, 1, 128, 64, _lib.stream()),
           "lane_matmul": lambda: lane_qmm.lane_matmul(x, w), "prefill_matmul": lambda: prefill_qmm.prefill_matmul(x, wide)}[call]
    one()
    torch.cuda.synchronize()
    took = []

    def fill():
        start = time.perf_counter()
        torch.cuda._sleep(2_000_000_000)                     # about a second of the GPU
        for _ in range(3000):                                # more launches than the queue holds
            one()
        took.append(time.perf_counter() - start)

    t = threading.Thread(target=fill)
    t.start()
    longest, last = 0.0, time.perf_counter()
    while t.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        longest, last = max(longest, now - last), now
    t.join()
    torch.cuda.synchronize()
    assert took[0] > 0.5, "the queue was never full: the test shows nothing"
    assert longest < 0.3, f"this thread stood still for {longest:.2f} s"


def test_f32_is_a_truth_value(lib):
    """Any object with a truth value, as before the checks went into native code."""

    import numpy as np

    from tensorfold_b200 import lane_qmm, prefill_qmm, synthetic

    x = torch.randn((2, 128), device="cuda").to(torch.bfloat16)
    w = synthetic.random_q4(torch.Generator(device="cuda").manual_seed(1), 256, 128, 64, "cuda")
    wide = prefill_qmm.tile_weight(*lane_qmm.untile_weight(w), 64)
    for yes, no in ((np.True_, np.False_), ("yes", ""), ([1], None)):
        for call, q in ((lane_qmm.lane_matmul, w), (prefill_qmm.prefill_matmul, wide)):
            assert call(x, q, f32=yes).dtype == torch.float32 and call(x, q, f32=no).dtype == torch.bfloat16
