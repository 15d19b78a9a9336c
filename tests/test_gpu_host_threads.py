"""The native host path beside other Python threads."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_call_that_blocks_lets_other_threads_run(dev):
    """With the GPU busy, launches block once the queue is full (some thousand of them).  Another thread keeps ticking."""
    from omnimem_b200 import ops
    x = torch.randn(1, 64, 1, 64, device=dev).to(torch.bfloat16)
    ops.pool_rows(x, 64)
    torch.cuda.synchronize()
    gaps, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=tick)
    thread.start()
    start = time.perf_counter()
    torch.cuda._sleep(2_000_000_000)                                       # about a second
    for _ in range(4000):
        ops.pool_rows(x, 64)
    blocked = time.perf_counter() - start
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert blocked > 0.5, "the queue took all launches: the test needs more of them"
    assert max(gaps) < 0.25 * blocked


def test_results_of_calls_from_several_threads(dev):
    from omnimem_b200 import ops
    from omnimem_b200.nsa.ops import selection_attention
    ids = torch.arange(2, dtype=torch.int32, device=dev).expand(1, 2, 2, 2).contiguous()
    inputs = [torch.randn(1, 128, 2, 128, device=dev, generator=torch.Generator(device=dev).manual_seed(i)).to(torch.bfloat16)
              for i in range(4)]

    def work(x):
        q = x.clone().requires_grad_(True)
        out = selection_attention(q, x, x, ids, 2, 64, group_size=64)
        return ops.pool_rows(x, 64), out.detach(), torch.autograd.grad(out, q, x)[0]

    want, got = [work(x) for x in inputs], [[] for _ in inputs]

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                got[i].append(work(inputs[i]))
            torch.cuda.current_stream().synchronize()

    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(len(g) == 50 and all(map(torch.equal, r, w)) for g, w in zip(got, want) for r in g)
