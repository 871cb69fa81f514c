"""GPU parity of the 128-row variant of the small-batch GEMM, at the sizes where its dispatch
changes or a tile is cut.  The oracle and its tolerances are those of test_gpu_parity.py."""
import numpy as np
import pytest

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from parity_util import compare, oracle_case, run_gpu

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
