"""The CTA-pair prefill kernel at the edges of its tiles: one accumulator and two, ragged token and row tiles, an odd number of
128-row tiles, rows that cannot be stored in pairs, scales on both sides of the limit of the short dequantisation."""
import numpy as np
import pytest

import oracle
from tests import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture()
def pairs():
    import qwen_engine_b200 as ops
    ops.set_option(ops.OPT_GEMM_FORM, 2)
    yield ops
    ops.set_option(ops.OPT_GEMM_FORM, 0)
    assert ops.debug_counter(0) == 0


def _pick(rng, n):
    return np.unique(np.concatenate([[0, n - 1], rng.choice(n, size=min(n, 24), replace=False)])).astype(np.int32)


@pytest.mark.parametrize("M,N,K,scale_max,res", [
    (1, 128, 256, 0.02, False), (16, 256, 512, 0.5, True), (17, 384, 256, 0.02, True), (129, 1536, 1536, 0.07, False),
    (300, 20000, 256, 0.02, True), (511, 17920, 512, 0.02, False), (770, 18944, 768, 0.5, True), (513, 1001, 512, 0.02, True),
    (257, 131, 8960, 0.02, False),
])
def test_pair_kernel_matches_oracle(pairs, M, N, K, scale_max, res):
    from qwen_engine_b200 import synth
    seed = M * 31 + N + K
    rng = np.random.default_rng(seed)
    qw, x = synth.packed_weights(seed, "p", N, K), synth.activations(seed, "p", M, K)
    sc = rng.uniform(0.002, scale_max, size=(N, K // 128)).astype(np.float16)
    r = rng.standard_normal((M, N)).astype(np.float16) if res else None
    y = torch.full((M * N + 64,), float("nan"), dtype=torch.float16, device="cuda")
    pairs.launch_gemm_prefill_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), util.to_dev(r) if res else None, y, M, N, K)
    torch.cuda.synchronize()
    got = util.to_np(y)
    assert np.isnan(got[M * N:]).all(), "wrote past the output"
    m_idx, n_idx = _pick(rng, M), _pick(rng, N)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx, residual=r)
    acc = ref64 - r[np.ix_(m_idx, n_idx)].astype(np.float64) if res else None
    util.assert_fp16_close(got[:M * N].reshape(M, N)[np.ix_(m_idx, n_idx)], ref64, what=f"{M}x{N}x{K}", magnitude=acc)


@pytest.mark.parametrize("col", [130, 131])      # word-aligned and not
def test_pair_kernel_block_with_peer_copies(pairs, col):
    """A column block of a wider matrix, also stored into matrices standing in for peer GPUs' memory."""
    from qwen_engine_b200 import synth
    M, N, K, ldc = 290, 384, 512, 1024
    qw, sc, x = synth.packed_weights(5, "b", N, K), synth.scales(5, "b", N, K), synth.activations(5, "b", M, K)
    d = [util.to_dev(v) for v in (qw, sc, x)]
    want = torch.empty((M, N), dtype=torch.float16, device="cuda")
    pairs.launch_gemm_prefill_w4a16(*d, None, want, M, N, K)
    mats = [torch.full((M, ldc), 7.0, dtype=torch.float16, device="cuda") for _ in range(3)]
    pairs.gemm_prefill_w4a16_block(*d, None, mats[0].data_ptr() + 2 * col, ldc, [m.data_ptr() + 2 * col for m in mats[1:]], M, N, K)
    torch.cuda.synchronize()
    for m in mats:
        assert torch.equal(m[:, col:col + N], want)
        assert (m[:, :col] == 7.0).all() and (m[:, col + N:] == 7.0).all()


@pytest.mark.parametrize("M,I,K,scale_max", [(260, 640, 512, 0.5), (700, 8960, 256, 0.02), (513, 4480, 1536, 0.07), (1030, 5000, 768, 0.02)])
def test_pair_kernel_swiglu_with_both_accumulators(pairs, M, I, K, scale_max):
    """Tiles of one accumulator and of two (the second one goes through shared memory), several tiles a pair, fewer steps than ring slots."""
    from qwen_engine_b200 import synth
    seed = M * 31 + I + K
    rng = np.random.default_rng(seed)
    qw, x = synth.packed_weights(seed, "s", 2 * I, K), synth.activations(seed, "s", M, K)
    sc = rng.uniform(0.002, scale_max, size=(2 * I, K // 128)).astype(np.float16)
    y = torch.full((M * I + 64,), float("nan"), dtype=torch.float16, device="cuda")
    pairs.launch_gemm_prefill_dual_gate_up_swiglu_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), y, M, None, K, I)
    torch.cuda.synchronize()
    got = util.to_np(y)
    assert np.isnan(got[M * I:]).all(), "wrote past the output"
    m_idx, n_idx = _pick(rng, M), _pick(rng, I)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx, swiglu=True)
    util.assert_fp16_close(got[:M * I].reshape(M, I)[np.ix_(m_idx, n_idx)], ref64, what=f"swiglu {M}x{I}x{K}")


@pytest.mark.parametrize("M,K", [(700, 256), (2400, 1024)])      # tiles of one accumulator, of two
def test_pair_kernel_swiglu_quotient(pairs, M, K):
    from tests import test_gpu_gemm_stream as stream
    stream.test_swiglu_quotient_over_its_range(M, K)
    stream.test_swiglu_with_an_infinite_up(M, K)
