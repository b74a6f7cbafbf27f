"""M-token launches from other host threads than the one that set the device up."""
import threading

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
