"""M-token launches from other host threads than the one that set the device up."""
import threading

import numpy as np
import pytest

from tests import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,N,K", [(32, 256, 512), (300, 4096, 512)])
def test_first_cuda_call_of_a_thread(M, N, K):
    """Tensor maps are encoded by the driver, which wants a context in the calling thread."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    ops.init()
    qw, sc, x = (util.to_dev(a) for a in (synth.packed_weights(M, "t", N, K), synth.scales(M, "t", N, K), synth.activations(M, "t", M, K)))
    y = [torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2)]
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    errors = []

    def work():
        try:
            ops.launch_gemm_prefill_w4a16(qw, sc, x, None, y[0], M, N, K, stream)
        except Exception as e:      # noqa: BLE001  (it would be lost in the thread)
            errors.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not errors, errors
    ops.launch_gemm_prefill_w4a16(qw, sc, x, None, y[1], M, N, K, stream)
    torch.cuda.synchronize()
    assert torch.equal(y[0].view(torch.int16), y[1].view(torch.int16))


# (tokens, rows, K): few tokens with K over a cluster, streaming with a K split (partials in memory of their own and on top
# of the rings), CTA pairs
SIZES = [(4, 1536, 8960), (16, 1536, 8960), (47, 1536, 8960), (115, 1536, 1536), (128, 7680, 8960), (600, 4096, 1024)]


def test_two_threads_on_two_streams_give_the_bits_of_one():
    """What the kernels exchange inside their clusters (partial sums on the peers' mbarriers, tensor memory) and the plans both
    threads ask for stay apart."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    ops.init()
    jobs = []
    for M, N, K in SIZES:
        t = [util.to_dev(a) for a in (synth.packed_weights(M, "c", N, K), synth.scales(M, "c", N, K), synth.activations(M, "c", M, K),
                                      synth.activations(M, "r", M, N))]
        jobs.append((M, N, K, *t))
    torch.cuda.synchronize()
    rounds, errors = 12, []
    outs = [[[torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda") for _ in range(rounds)] for M, N, *_ in jobs] for _ in range(2)]
    start = threading.Barrier(2)

    def work(who):
        try:
            stream = torch.cuda.Stream()
            start.wait()
            for i in range(rounds):
                for j in (range(len(jobs)) if who == 0 else reversed(range(len(jobs)))):
                    M, N, K, qw, sc, x, r = jobs[j]
                    ops.launch_gemm_prefill_w4a16(qw, sc, x, r, outs[who][j][i], M, N, K, stream)
            stream.synchronize()
        except Exception as e:      # noqa: BLE001  (an assertion in a thread would be lost)
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(who,)) for who in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for j, (M, N, K, qw, sc, x, r) in enumerate(jobs):
        alone = torch.empty((M, N), dtype=torch.float16, device="cuda")
        ops.launch_gemm_prefill_w4a16(qw, sc, x, r, alone, M, N, K)
        want = util.to_np(alone).view(np.int16)
        for who in range(2):
            for y in outs[who][j]:
                assert np.array_equal(util.to_np(y).view(np.int16), want), (M, N, K, who)
    assert ops.debug_counter(0) == 0
