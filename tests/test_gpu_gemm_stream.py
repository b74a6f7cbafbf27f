"""The weight-streaming tcgen05 kernel (up to 256 tokens) at the edges of its tiles: token tiles of 16 to 128, one and two of
them, K ranges of two steps and of many, split and not, rows past the last whole tile, scales on both sides of the limit
of the short dequantisation."""
import numpy as np
import pytest

import oracle
from tests import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,N,K,scale_max,res", [
    (17, 128, 256, 0.02, False), (47, 1536, 8960, 0.02, True), (48, 520, 512, 0.5, True), (64, 2048, 1536, 0.02, False),
    (65, 20000, 256, 0.02, True), (112, 384, 2304, 0.07, True), (115, 1536, 1536, 0.02, True), (128, 17920, 768, 0.02, False),
    (129, 1536, 1536, 0.5, True), (203, 17920, 1536, 0.02, False), (255, 132, 8960, 0.02, True), (256, 300, 1024, 0.02, False),
    # 128-token tiles with a K split leave no room beside the rings: the partial sums go on top of them
    (120, 7680, 8960, 0.02, True), (256, 4600, 8960, 0.5, False),
])
def test_stream_kernel_matches_oracle(M, N, K, scale_max, res):
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    seed = M * 31 + N + K
    rng = np.random.default_rng(seed)
    qw, x = synth.packed_weights(seed, "s", N, K), synth.activations(seed, "s", M, K)
    sc = rng.uniform(0.002, scale_max, size=(N, K // 128)).astype(np.float16)
    r = rng.standard_normal((M, N)).astype(np.float16) if res else None
    y = torch.full((M * N + 64,), float("nan"), dtype=torch.float16, device="cuda")
    ops.launch_gemm_prefill_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), util.to_dev(r) if res else None, y, M, N, K)
    torch.cuda.synchronize()
    got = util.to_np(y)
    assert np.isnan(got[M * N:]).all(), "wrote past the output"
    pick = lambda n: np.unique(np.concatenate([[0, n - 1], rng.choice(n, size=min(n, 24), replace=False)])).astype(np.int32)  # noqa: E731
    m_idx, n_idx = pick(M), pick(N)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx, residual=r)
    acc = ref64 - r[np.ix_(m_idx, n_idx)].astype(np.float64) if res else None
    util.assert_fp16_close(got[:M * N].reshape(M, N)[np.ix_(m_idx, n_idx)], ref64, what=f"{M}x{N}x{K}", magnitude=acc)
    assert ops.debug_counter(0) == 0


@pytest.mark.parametrize("M", [33, 130])
def test_stream_kernel_swiglu_and_qkv_routing(M):
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    H, I = 512, 640
    x = synth.activations(M, "x", M, H)
    qw, sc = synth.packed_weights(M, "gu", 2 * I, H), synth.scales(M, "gu", 2 * I, H)
    y = torch.empty((M, I), dtype=torch.float16, device="cuda")
    ops.launch_gemm_prefill_dual_gate_up_swiglu_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), y, M, None, H, I)
    m_idx, n_idx = np.arange(0, M, 7, dtype=np.int32), np.arange(0, I, 13, dtype=np.int32)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx, swiglu=True)
    util.assert_fp16_close(util.to_np(y)[np.ix_(m_idx, n_idx)], ref64, what="swiglu")
    # q, k, v as three tensors of 384, 128 and 128 rows = the rows of one
    qkv = [(util.to_dev(qw[a:b].copy()), util.to_dev(sc[a:b].copy()), torch.empty((M, b - a), dtype=torch.float16, device="cuda"))
           for a, b in ((0, 384), (384, 512), (512, 640))]
    ops.launch_gemm_prefill_qkv_w4a16(ops.QKVProjectionView(*[t for p in qkv for t in p]), util.to_dev(x), M, None, H, 3, 1, 128)
    n_idx = np.arange(0, 640, 11, dtype=np.int32)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx)
    got = np.concatenate([util.to_np(p[2]) for p in qkv], axis=1)
    util.assert_fp16_close(got[np.ix_(m_idx, n_idx)], ref64, what="qkv")


@pytest.mark.parametrize("M,N,K,scale_max,res", [
    # token counts that come to it from the few-token forms: 6 to 16, 2 on long K, 4 on rows that are no whole groups of 16
    (6, 17920, 1536, 0.02, False), (8, 1536, 8960, 0.02, True),
    (9, 1536, 1536, 0.02, True), (16, 17920, 1536, 0.5, False), (13, 2048, 8960, 0.02, True), (2, 264, 8192, 0.02, False),
    (4, 130, 512, 0.07, True), (3, 8200, 8192, 0.02, False),
    # one more step than token slots, steps beyond both rings, an odd number of steps in a CTA (two issuing threads)
    (40, 20000, 1792, 0.02, False), (33, 19000, 3328, 0.5, True), (64, 19100, 1792, 0.02, False), (47, 384, 8960, 0.02, True),
])
def test_stream_kernel_few_tokens_and_ring_lengths(M, N, K, scale_max, res):
    test_stream_kernel_matches_oracle(M, N, K, scale_max, res)


@pytest.mark.parametrize("M", [16, 64, 700])
def test_swiglu_quotient_over_its_range(M, K=256):
    """Gate and up values planted through tokens with one nonzero element, from 1e-4 to the ends of fp16's range, against 64 bits.
    exp (2 ulp), the sum, the quotient and the product leave at most 6 * 2^-24 of a value, so an output is the nearest fp16
    value except within that of a midpoint, two neighbours of which are 2^-11 apart: 0.2 % of them, and by one step."""
    import qwen_engine_b200 as ops
    I = 512
    rng = np.random.default_rng(M)
    q, sc = rng.integers(0, 16, 2 * I), rng.uniform(0.002, 0.05, (2 * I, K // 128)).astype(np.float16)
    qw = np.zeros((2 * I, K // 8), dtype=np.uint32)
    qw[:, 0] = q                                   # element 0 is the word's lowest nibble
    x = np.zeros((M, K), dtype=np.float16)
    x[:, 0] = (rng.standard_normal(M) * np.logspace(-2, 3, M)).astype(np.float16)
    w = ((q - 8) * sc[:, 0].astype(np.float32)).astype(np.float16).astype(np.float64)

    def run(xs):
        y = torch.empty((M, I), dtype=torch.float16, device="cuda")
        ops.launch_gemm_prefill_dual_gate_up_swiglu_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(xs), y, M, None, K, I)
        torch.cuda.synchronize()
        with np.errstate(all="ignore"):
            acc = (xs[:, :1].astype(np.float64) * w[None, :]).astype(np.float32).astype(np.float64)
            return util.to_np(y), acc[:, 0::2] / (1.0 + np.exp(-acc[:, 0::2])) * acc[:, 1::2]
    got, ref = run(x)
    ok = (np.abs(ref) > 1e-4) & (np.abs(ref) < 6e4)
    with np.errstate(over="ignore"):
        near = ref.astype(np.float16)
    steps = np.abs(got[ok].view(np.int16).astype(np.int32) - near[ok].view(np.int16).astype(np.int32))
    assert steps.max() <= 1 and np.mean(steps != 0) <= 2e-3, (steps.max(), np.mean(steps != 0))
    # infinite accumulators: -inf / (1 + inf) is NaN, inf / 1 is inf, whatever up makes of them
    x[:, 0] = np.where(np.arange(M) % 2 == 0, np.inf, -np.inf).astype(np.float16)
    got, ref = run(x)
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isposinf(got), np.isposinf(ref)) and np.array_equal(np.isneginf(got), np.isneginf(ref))


@pytest.mark.parametrize("M", [4, 16, 64, 700])
def test_swiglu_with_an_infinite_up(M, K=256):
    """Gates around the one from which e^-gate is infinite (-88.7), and of both signs: an infinity where IEEE arithmetic has one."""
    import qwen_engine_b200 as ops
    gates = np.concatenate([np.linspace(-91, -86, 448), np.linspace(-80, 80, 64)]).astype(np.float16)
    I = len(gates)
    qw, sc = np.full((2 * I, K // 8), 0x88888888, dtype=np.uint32), np.ones((2 * I, K // 128), dtype=np.float16)
    qw[0::2, 0], sc[0::2, 0] = 0x88888889, gates               # one weight of a gate row is its scale, the others are zero
    qw[1::2, :16], sc[1::2, 0] = 0x99999999, np.inf            # a group of infinite weights
    x = np.ones((M, K), dtype=np.float16)
    y = torch.empty((M, I), dtype=torch.float16, device="cuda")
    ops.launch_gemm_prefill_dual_gate_up_swiglu_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), y, M, None, K, I)
    torch.cuda.synchronize()
    g = gates.astype(np.float32)
    with np.errstate(all="ignore"):
        ref = (g / (np.float32(1) + np.exp(-g)) * np.float32(np.inf)).astype(np.float16)
    assert np.array_equal(util.to_np(y), np.broadcast_to(ref, (M, I)), equal_nan=True)
