"""The few-token kernel (2-16 tokens) at the edges of its cut: one CTA per row block and clusters, K of one step pair and of many,
row groups that do not fill a CTA, scales on both sides of the limit of the short dequantisation; and the RMSNorm + Q8_1 launch
at the ends of its register form."""
import numpy as np
import pytest

import oracle
from tests import util

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("M,N,K,scale_max", [(2, 16, 256, 0.02), (3, 48, 8960, 0.5), (7, 1536, 8960, 0.02), (8, 2064, 1536, 0.07),
                                             (9, 17920, 1536, 0.02), (13, 272, 4096, 0.5), (16, 1536, 8960, 0.02), (16, 30000, 512, 0.02)])
def test_few_token_kernel_matches_oracle(M, N, K, scale_max):
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    seed = M * 31 + N + K
    rng = np.random.default_rng(seed)
    qw, x = synth.packed_weights(seed, "f", N, K), synth.activations(seed, "f", M, K)
    sc = rng.uniform(0.002, scale_max, size=(N, K // 128)).astype(np.float16)
    r = rng.standard_normal((M, N)).astype(np.float16)
    y = torch.full((M * N + 64,), float("nan"), dtype=torch.float16, device="cuda")
    y[:M * N] = util.to_dev(r).reshape(-1)
    ops.launch_gemm_prefill_w4a16(util.to_dev(qw), util.to_dev(sc), util.to_dev(x), y, y, M, N, K)
    torch.cuda.synchronize()
    got = util.to_np(y)
    assert np.isnan(got[M * N:]).all(), "wrote past the output"
    n_idx = np.unique(np.concatenate([[0, N - 1], rng.choice(N, size=min(N, 48), replace=False)])).astype(np.int32)
    m_idx = np.arange(M, dtype=np.int32)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx, residual=r)
    util.assert_fp16_close(got[:M * N].reshape(M, N)[:, n_idx], ref64, what=f"{M}x{N}x{K}",
                           magnitude=ref64 - r[:, n_idx].astype(np.float64))
    assert ops.debug_counter(0) == 0


@pytest.mark.parametrize("hidden,offset", [(128, 0), (1536, 0), (1664, 0), (8192, 0), (8320, 0), (1536, 4)])
def test_rmsnorm_q8_1_sizes(hidden, offset):
    """offset: elements by which the input misses its 16-byte alignment (the shared-memory form takes it)."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    x = (synth.activations(hidden, "r", hidden).astype(np.float32) * 3).astype(np.float16)
    g = (1 + 0.1 * synth.activations(hidden, "g", hidden).astype(np.float32)).astype(np.float16)
    d_x = torch.empty(hidden + offset, dtype=torch.float16, device="cuda")[offset:]
    d_x.copy_(util.to_dev(x))
    q8 = torch.empty(hidden, dtype=torch.int8, device="cuda")
    xs = torch.empty(hidden // 128, dtype=torch.float32, device="cuda")
    s8 = torch.empty(hidden // 8, dtype=torch.int32, device="cuda")
    y = torch.empty(hidden, dtype=torch.float16, device="cuda")
    ops.launch_rmsnorm_q8_1(d_x, util.to_dev(g), y, q8, xs, s8, None, hidden)
    torch.cuda.synchronize()
    # the normed vector, then the quantiser the oracle has for it
    inv = np.float16(np.float32(1) / np.sqrt(np.float32(np.mean(x.astype(np.float64) ** 2)) + np.float32(1e-6)))
    want = ((x * inv).astype(np.float16) * g).astype(np.float16)
    assert np.array_equal(util.to_np(y).view(np.uint16), want.view(np.uint16))
    w8, ws, wsum = oracle.quantize_q8_1(want)
    assert np.array_equal(util.to_np(q8), w8) and np.array_equal(util.to_np(xs), ws) and np.array_equal(util.to_np(s8), wsum)


def test_rmsnorm_q8_1_gain_written_by_the_launch_in_front():
    """The gain is read as the launch in front left it: here a row of an embedding table, another one each time."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    H, V = 1536, 64
    table, sc = util.to_dev(synth.packed_weights(9, "e", V, H)), util.to_dev(synth.scales(9, "e", V, H))
    x, tokens = util.to_dev(synth.activations(9, "e", H)), torch.arange(V, dtype=torch.int32, device="cuda")
    gain = torch.zeros(H, dtype=torch.float16, device="cuda")

    def launch(t, y, gain):
        q8 = (torch.empty(H, dtype=torch.int8, device="cuda"), torch.empty(H // 128, dtype=torch.float32, device="cuda"),
              torch.empty(H // 8, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        ops.launch_embed_lookup_w4a16(table, sc, tokens[t:], gain, None, 1, None, H, V)
        return q8, lambda: ops.launch_rmsnorm_q8_1(x, gain, y, *q8, None, H)

    y = torch.empty((2, V, H), dtype=torch.float16, device="cuda")
    for t in range(V):
        q8, norm = launch(t, y[0, t], gain)
        norm()
        want8, norm = launch(t, y[1, t], torch.zeros_like(gain))
        torch.cuda.synchronize()      # the gain is there before the launch
        norm()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(q8, want8))
    assert torch.equal(y[0].view(torch.int16), y[1].view(torch.int16))


@pytest.mark.parametrize("M,N,K,scale_max", [(7, 1536, 8960, 0.02), (8, 17920, 1536, 0.5), (9, 17920, 1536, 0.02), (13, 272, 4096, 0.5), (16, 1536, 8960, 0.02), (16, 30000, 512, 0.07)])
def test_few_token_kernel_asked_for(M, N, K, scale_max):
    """6 to 16 tokens through this kernel whatever the matrix (by default only the smaller ones)."""
    import qwen_engine_b200 as ops
    ops.set_option(ops.OPT_GEMM_MMA_MAX_TOKENS, 16)
    try:
        test_few_token_kernel_matches_oracle(M, N, K, scale_max)
    finally:
        ops.set_option(ops.OPT_GEMM_MMA_MAX_TOKENS, 0)


@pytest.mark.parametrize("M,N,K", [(2, 8208, 4096), (3, 9456, 4096), (3, 9376, 3584)])
def test_large_matrix_below_the_first_tokens_of_tcgen05(M, N, K):
    test_few_token_kernel_matches_oracle(M, N, K, 0.02)


@pytest.mark.parametrize("M,K,q_heads,kv_heads", [(9, 1536, 24, 5), (16, 1024, 15, 3), (6, 4096, 64, 9)])
def test_qkv_of_heads_of_64(M, K, q_heads, kv_heads):
    """Widths that are no multiples of 128, which the tcgen05 kernels refuse."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    rows = [64 * q_heads, 64 * kv_heads, 64 * kv_heads]
    qw, sc, x = synth.packed_weights(M, "q", sum(rows), K), synth.scales(M, "q", sum(rows), K), synth.activations(M, "q", M, K)
    cut = np.cumsum([0, *rows])
    qkv = [(util.to_dev(qw[a:b].copy()), util.to_dev(sc[a:b].copy()), torch.full((M, b - a), float("nan"), dtype=torch.float16, device="cuda"))
           for a, b in zip(cut, cut[1:])]
    ops.launch_gemm_prefill_qkv_w4a16(ops.QKVProjectionView(*[t for p in qkv for t in p]), util.to_dev(x), M, None, K, q_heads, kv_heads, 64)
    m_idx, n_idx = np.arange(M, dtype=np.int32), np.unique(np.concatenate([np.arange(0, sum(rows), 29), cut[1:] - 1, cut[:-1]])).astype(np.int32)
    ref64, _ = oracle.gemm_prefill(qw, sc, x, m_idx, n_idx)
    got = np.concatenate([util.to_np(p[2]) for p in qkv], axis=1)
    assert not np.isnan(got).any()
    util.assert_fp16_close(got[:, n_idx], ref64, what="qkv")
    assert ops.debug_counter(0) == 0
