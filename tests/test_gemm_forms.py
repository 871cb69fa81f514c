"""Which form of the expert GEMM a call takes, and the two forms of its 128-row items, one CTA each
or a CTA pair, on both sides of the line between them."""
import statistics

import numpy as np
import pytest

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from parity_util import compare_sampled, gemm_form, run_gpu


@pytest.mark.parametrize("hidden,intermediate,n_local,ctas", [
    (2880, 2880, 128, 2), (2880, 2880, 32, 2), (2880, 2880, 16, 2), (2048, 768, 128, 2), (1024, 1408, 69, 2),
    # little to decode: the fixed cost of a pair is more than it saves
    (2880, 2880, 8, 1), (512, 256, 16, 1), (512, 512, 32, 1), (4096, 256, 32, 1), (64, 64, 1, 1), (64, 64, 256, 1),
    # odd numbers of weight tiles: the last pair of a matrix decodes one for nothing
    (2816, 448, 95, 1), (704, 1088, 48, 1),
])
def test_form_of_128_row_items(hidden, intermediate, n_local, ctas):
    for rows in (57, 128):
        assert gemm_form(hidden, intermediate, n_local, rows * n_local) == (128, ctas)
    assert gemm_form(hidden, intermediate, n_local, 57 * n_local - 1) == (64, 1)
    assert gemm_form(hidden, intermediate, n_local, 129 * n_local) == (256, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("ctas,H,I,E,K", [
    (2, 256, 2048, 256, 8),   # one step of four chunks; eight
    (2, 4096, 128, 256, 8),   # 16 steps; one cut step
    (2, 2880, 2880, 16, 4),   # odd numbers of weight tiles in both launches; 12 steps, the last of one chunk
    (1, 1088, 832, 64, 4),    # three chunks per step: 6 and 5 steps, the last one cut
    (1, 704, 1088, 48, 3),
])
@pytest.mark.parametrize("avg,few", [(57, False), (128, True), (129, False)])
def test_128_row_items_in_both_forms(ctas, H, I, E, K, avg, few):
    """All rows against the cross-check GEMM (the same rounding points, another fp32 order: the bound
    of test_tcgen05_equals_mma_sync_at_prefill_size), a sample against the oracle.  `few`: hardly any
    rows for the last expert, so that boxes of its item lie past the last row of the buffer."""
    T = -(-avg * E // K)
    assert gemm_form(H, I, E, T * K) == ((128, ctas) if avg <= 128 else (256, 2))
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + avg)
    if few:  # logits are N(0, 0.0004 H) over the experts: about six tokens choose the last one
        z = statistics.NormalDist(0, 0.02 * H ** 0.5).inv_cdf
        lw.b_router[-1] = z(1 - K / E) - z(1 - 6 / T)
    x_bits = synth.make_tokens(T, H, seed=avg)
    res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05)  # asserts the status word
    if few:
        assert 1 <= res["counts"][-1] <= 16
    ref = run_gpu(shape, lw, x_bits, capi.GEMM_MMA_SYNC)
    assert np.array_equal(ref["topk_i"], res["topk_i"])
    d = ref["out"].astype(np.float64) - res["out"].astype(np.float64)
    assert np.linalg.norm(d) / np.linalg.norm(ref["out"].astype(np.float64)) < 5e-4
    sample = np.linspace(0, T - 1, 8).astype(int)
    compare_sampled({k: res[k][sample] for k in ("out", "topk_i", "topk_w", "h_bits")}, lw, x_bits[sample],
                    lw.w_router, lw.b_router, K, f"{(H, I, E, K, avg)}")
