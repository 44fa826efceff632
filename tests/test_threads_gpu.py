"""Two host threads, each on its own stream, call the same operator with sizes that need different amounts of shared memory."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _attention_int8(T, gen, cuda, S):
    x = torch.randint(-127, 128, (S, 1, 3 * 64), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    return lambda: T.mha(x, 1, S, 1, scale_bmm1=1e-4, scale_softmax=127.0, scale_bmm2=1.0 / 127)


def _separate_int8(T, gen, cuda, S):
    q, k, v = (torch.randint(-127, 128, (1, 1, S, 64), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8) for _ in range(3))
    return lambda: T.attention_bnsd(q, k, v, scale_bmm1=1e-4, scale_softmax=127.0, scale_bmm2=1.0 / 127)


def _attention_odd_head(T, gen, cuda, S):
    x = torch.randn((S, 1, 3 * 6), device=cuda, generator=gen)
    return lambda: T.mha(x, 1, S, 1, 6)


def _skip_ln_int8(T, gen, cuda, ld):
    x = torch.randint(-127, 128, (4, ld), device=cuda, generator=gen, dtype=torch.int32).to(torch.int8)
    g = torch.ones(ld, device=cuda, dtype=torch.float16)
    return lambda: T.skip_layer_norm_dqq(x, x, g, g, g, 0.02, 0.02, 30.0)


@pytest.mark.parametrize("make,large,small,calls", [(_attention_int8, 512, 100, 2000), (_separate_int8, 512, 100, 2000),
                                                    (_attention_odd_head, 4000, 3100, 100), (_skip_ln_int8, 8192, 7168, 2000)])
def test_two_threads_with_different_sizes(cuda, make, large, small, calls):
    import tensorrt_b200 as T

    gen = torch.Generator(device=cuda).manual_seed(large)
    work = [make(T, gen, cuda, size) for size in (large, small)]
    want = [w() for w in work]
    torch.cuda.synchronize()
    start, failed = threading.Barrier(2), [None, None]

    def run(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(10)
                for _ in range(calls):
                    out = work[i]()
                torch.cuda.current_stream().synchronize()
            assert torch.equal(out, want[i])
        except Exception as e:  # noqa: BLE001 (reported by the test's own thread)
            failed[i] = e

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert failed == [None, None], failed
