"""GPU parity of the GEMM with decoded weights in tensor memory where its rings are cut: K of one
chunk (64 columns), one less and one more than a step holds, and items of one row; 64-row items and
128-row items with one CTA each (on CTA pairs: test_gemm_forms.py).  The oracle and its tolerances are
those of test_gpu_parity.py."""
import pytest

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from parity_util import compare, oracle_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 20, 200, 300, 440])  # 8 experts, top 2: up to 110 rows per expert on average
@pytest.mark.parametrize("h_chunks,i_chunks", [(1, 2), (3, 1), (4, 5), (6, 7), (8, 13), (5, 3)])
def test_ring_cuts(h_chunks, i_chunks, T):
    H, I, E, K = 64 * h_chunks, 64 * i_chunks, 8, 2
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + I + T)
    x_bits = synth.make_tokens(T, H, seed=T)
    res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05)
    compare(res, oracle_case(lw, x_bits), K, f"{(H, I, T)}")
