"""GPU: calls from several Python threads. The native module gives up Python's lock while it plans, allocates and launches, so a call that
waits (a launch into a full queue) keeps no other thread from running, and calls of two threads on two streams do not disturb each other."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


def test_other_threads_run_while_a_launch_waits_for_the_queue(aclnn):
    import torch

    from gpu_util import DEV

    x = torch.randn((64, 1024), device=DEV).to(torch.bfloat16)
    y = torch.empty((64, 1024), dtype=torch.uint8, device=DEV)
    s = torch.empty((64, 16, 2), dtype=torch.uint8, device=DEV)
    d = (aclnn.from_torch(x), aclnn.from_torch(y, "float8_e4m3fn"), aclnn.from_torch(s, "float8_e8m0"))
    aclnn.dynamic_mx_quant(*d, "float8_e4m3fn")
    torch.cuda.synchronize()
    took = []

    def calls():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_200_000_000)  # clocks: 0.6 s and more that the launches behind it have to wait for
            t0 = time.monotonic()
            for _ in range(4000):
                aclnn.dynamic_mx_quant(*d, "float8_e4m3fn")
            took.append(time.monotonic() - t0)

    worker = threading.Thread(target=calls)
    worker.start()
    longest, last = 0.0, time.monotonic()
    while worker.is_alive():
        time.sleep(0.001)
        now = time.monotonic()
        longest, last = max(longest, now - last), now
    torch.cuda.synchronize()
    assert took and took[0] > 0.4, "the queue took all launches at once: nothing was shown"
    assert longest < 0.2, longest


def test_calls_of_two_threads_on_two_streams(pkg):
    import torch

    from gpu_util import DEV

    api = pkg.torch_api
    gen = torch.Generator(device=DEV).manual_seed(5)
    k, n, g = 2048, 4096, 128
    w = torch.randint(-2 ** 31, 2 ** 31, (k, n // 8), generator=gen, device=DEV, dtype=torch.int32)
    sc = (torch.rand((k // g, n), generator=gen, device=DEV) * 0.01 + 0.005).to(torch.bfloat16)
    q1 = torch.randint(-127, 128, (96, k), generator=gen, device=DEV, dtype=torch.int8)
    q2 = torch.randint(-127, 128, (k, n), generator=gen, device=DEV, dtype=torch.int8)
    s1, s2 = torch.rand(96, generator=gen, device=DEV) * 0.01, torch.rand(n, generator=gen, device=DEV) * 0.01
    xs = [torch.randn((m, k), generator=gen, device=DEV).to(torch.bfloat16) for m in (1, 16, 40, 200)]

    def both(i):
        return (api.npu_weight_quant_batchmatmul(xs[i % 4], w, sc, antiquant_group_size=g),
                api.npu_quant_matmul(q1, q2, s2, pertoken_scale=s1, output_dtype=torch.bfloat16))

    want = [both(i) for i in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def thread(first):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got = [both(first + i) for i in range(40)]
                torch.cuda.current_stream().synchronize()
                for i, pair in enumerate(got):
                    if not all(torch.equal(a, b) for a, b in zip(pair, want[(first + i) % 4])):
                        wrong.append((first, i))
        except Exception as e:  # shown by the assertion below
            wrong.append(repr(e))

    threads = [threading.Thread(target=thread, args=(f,)) for f in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
