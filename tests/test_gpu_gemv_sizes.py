"""Batch-1 projections at the sizes where the streaming kernels take over from the register form: both sides of each line,
rows that do not fill the last block, K that does not fill the last slice.  Every entry point gives the bits of the register
form, and those are within tolerance of the oracle."""
import numpy as np
import pytest

import oracle
from tests import util

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [
    (4736, 2304), (4737, 2304), (5000, 4096),                    # one block per SM, K > 2048
    (5919, 1024), (5921, 768), (9472, 1024), (9473, 1024),       # one block per CTA, few steps
    (9472, 1536), (9473, 1280), (10001, 2048), (13000, 512),     # a second wave of the register form
]


@pytest.mark.parametrize("N,K", SIZES)
def test_plain_projection_bits_do_not_depend_on_the_form(N, K):
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    ops.init()
    qw_h, sc_h = synth.packed_weights(5, "t", N, K), synth.scales(5, "t", N, K)
    qw, sc = util.to_dev(qw_h), util.to_dev(sc_h)
    rng = np.random.Generator(np.random.Philox(key=N + K))
    x_h = rng.standard_normal(K).astype(np.float16)
    x, gamma = util.to_dev(x_h), util.to_dev((rng.random(K) * 0.02 + 0.04).astype(np.float16))
    res = util.to_dev(rng.standard_normal(N).astype(np.float16))
    act = (torch.empty(K, dtype=torch.int8, device="cuda"), torch.empty(K // 128, dtype=torch.float32, device="cuda"),
           torch.empty(K // 8, dtype=torch.int32, device="cuda"))
    ops.launch_quantize_fp16_to_q8_1(x, *act, K)

    heads = x.float() * 1.1

    def outputs():
        y = torch.full((4, N + 16), float("nan"), dtype=torch.float16, device="cuda")
        ops.launch_gemv_w4a8(qw, sc, *act, None, y[0], N, K)
        ops.launch_gemv_w4a16(qw, sc, x, res, y[1], N, K)
        ops.launch_gemv_rmsnorm_w4a16(qw, sc, x, gamma, None, y[2], N, K)
        ops.gemv_attn_heads_f32_w4a16(qw, sc, heads, res, y[3], N, K)
        torch.cuda.synchronize()
        return y

    got = outputs()
    try:
        ops.set_option(ops.OPT_GEMV_FORM, ops.GEMV_FORM_REGISTERS)
        want = outputs()
    finally:
        ops.set_option(ops.OPT_GEMV_FORM, ops.GEMV_FORM_AUTO)
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert torch.isnan(got[:, N:]).all()
    y64, _ = oracle.gemv_q8(qw_h, sc_h, util.to_np(act[0]), util.to_np(act[1]))
    util.assert_fp16_close(util.to_np(got[0, :N]), y64)


@pytest.mark.parametrize("inter,K", [(4800, 512), (5921, 1536), (9473, 1024), (9500, 1536), (11841, 2048)])
def test_gate_up_bits_do_not_depend_on_the_form(inter, K):
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    ops.init()
    qw, sc = util.to_dev(synth.packed_weights(6, "t", 2 * inter, K)), util.to_dev(synth.scales(6, "t", 2 * inter, K))
    rng = np.random.Generator(np.random.Philox(key=inter + K))
    x = util.to_dev(rng.standard_normal(K).astype(np.float16))
    gamma = util.to_dev((rng.random(K) * 0.02 + 0.04).astype(np.float16))
    outs = []
    try:
        for form in (ops.GEMV_FORM_REGISTERS, ops.GEMV_FORM_AUTO):
            ops.set_option(ops.OPT_GEMV_FORM, form)
            y = torch.full((inter + 16,), float("nan"), dtype=torch.float16, device="cuda")
            ops.launch_gemv_dual_gate_up_swiglu_rmsnorm_w4a16(qw, sc, x, gamma, y, K, inter)
            torch.cuda.synchronize()
            outs.append(y)
    finally:
        ops.set_option(ops.OPT_GEMV_FORM, ops.GEMV_FORM_AUTO)
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    assert torch.isfinite(outs[1][:inter]).all() and torch.isnan(outs[1][inter:]).all()


@pytest.mark.parametrize("K", [256, 1024, 1280, 2048, 2304, 4352, 16384, 16640, 33024])
@pytest.mark.parametrize("offset", [0, 4])
def test_fp16_staging_equals_the_stand_alone_quantisers(K, offset):
    """One and several rounds of groups, one and several turns of the raw buffer, x on an 8-byte boundary only."""
    import qwen_engine_b200 as ops
    from qwen_engine_b200 import synth
    ops.init()
    N = 40
    qw, sc = util.to_dev(synth.packed_weights(7, "t", N, K)), util.to_dev(synth.scales(7, "t", N, K))
    rng = np.random.Generator(np.random.Philox(key=K + offset))
    x = util.to_dev(rng.standard_normal(K + offset).astype(np.float16))[offset:]
    gamma = util.to_dev((rng.random(K) * 0.02 + 0.04).astype(np.float16))
    act = (torch.empty(K, dtype=torch.int8, device="cuda"), torch.empty(K // 128, dtype=torch.float32, device="cuda"),
           torch.empty(K // 8, dtype=torch.int32, device="cuda"))
    y = torch.empty((4, N), dtype=torch.float16, device="cuda")
    ops.launch_gemv_w4a16(qw, sc, x, None, y[0], N, K)
    ops.launch_quantize_fp16_to_q8_1(x, *act, K)
    ops.launch_gemv_w4a8(qw, sc, *act, None, y[1], N, K)
    ops.launch_gemv_rmsnorm_w4a16(qw, sc, x, gamma, None, y[2], N, K)
    ops.launch_rmsnorm_q8_1(x, gamma, None, *act, hidden_size=K)
    ops.launch_gemv_w4a8(qw, sc, *act, None, y[3], N, K)
    torch.cuda.synchronize()
    assert torch.equal(y[0].view(torch.int16), y[1].view(torch.int16))
    assert torch.equal(y[2].view(torch.int16), y[3].view(torch.int16))
