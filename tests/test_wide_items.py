"""GPU parity of the 128-row items of the GEMM with decoded weights in tensor memory where a tile is
cut or a ring comes round (test_gemm_forms.py: where its dispatch changes).  The oracle and its
tolerances are those of test_gpu_parity.py."""
import numpy as np
import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from parity_util import compare, compare_sampled, gemm_form, oracle_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,E,K,T", [
    (64, 64, 8, 2, 228),     # just above the 64-row items; one chunk of K
    (256, 192, 8, 2, 300),   # 4 and 3 chunks of K: a step that is cut, a step that is full
    (320, 128, 8, 2, 440),   # experts above 128 rows: two equal items
    (192, 64, 40, 4, 1100),
])
@pytest.mark.parametrize("skew", [False, True])
def test_wide_items(H, I, E, K, T, skew):
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + E + T)
    if skew:  # most rows to two experts, which then need many items; empty experts
        lw.b_router[:] = np.linspace(-2.0, 2.0, E, dtype=np.float32)
    x_bits = synth.make_tokens(T, H, seed=T)
    ref = oracle_case(lw, x_bits)
    res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05)
    compare(res, ref, K, f"{(H, I, E, K, T, skew)}")


@pytest.mark.parametrize("H,I,E,K,T", [
    (2880, 2880, 32, 4, 777),   # on CTA pairs: 12 steps per item
    (1088, 832, 64, 4, 1600),   # one CTA per item: 6 and 5 steps, the last one cut in both launches
])
@pytest.mark.parametrize("skew", [False, True])
def test_wide_items_reuse_their_rings(H, I, E, K, T, skew):
    """CTAs that walk several items of many steps: every slot of the weight, activation and
    tensor-memory rings, both accumulator sets and the parities of their barriers come round
    again.  All rows against the cross-check GEMM (the same rounding points, another fp32
    order: the bound of test_tcgen05_equals_mma_sync_at_prefill_size), a sample against the
    oracle."""
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + T, **(dict(zipf_s=1.1, zipf_gain=synth.ZIPF_GAIN_4X) if skew else {}))
    x_bits = synth.make_tokens(T, H, seed=T)
    res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05)  # asserts the status word
    items = sum(-(-c // 128) for c in res["counts"])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, ctas = gemm_form(H, I, E, sum(res["counts"]))
    assert rows == 128
    for m_tiles, k in ((-(-2 * I // 128), H), (-(-H // 128), I)):
        assert items * -(-m_tiles // ctas) >= 3 * (sms // ctas)  # three items and more to a CTA or pair
        assert -(-k // 64 // (2 + ctas)) > 4  # steps of three or four chunks: more than the rings hold
    if skew:
        assert max(res["counts"]) > 256  # more than two items of one expert
    ref = run_gpu(shape, lw, x_bits, capi.GEMM_MMA_SYNC)
    assert np.array_equal(ref["topk_i"], res["topk_i"])
    d = ref["out"].astype(np.float64) - res["out"].astype(np.float64)
    assert np.linalg.norm(d) / np.linalg.norm(ref["out"].astype(np.float64)) < 5e-4
    sample = np.linspace(0, T - 1, 16).astype(int)
    compare_sampled({k: res[k][sample] for k in ("out", "topk_i", "topk_w", "h_bits")}, lw, x_bits[sample],
                    lw.w_router, lw.b_router, K, f"{(H, I, E, K, T, skew)}")
