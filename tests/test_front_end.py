"""GPU parity of the one-launch front end (up to 16 tokens), at the sizes where its dispatch
changes or its K split is uneven.  The oracle and its tolerances are those of
test_gpu_parity.py."""
import numpy as np
import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth
from oracle import oracle
from parity_util import compare, oracle_case, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,E,K,T", [
    (64, 64, 4, 1, 1),       # one chunk of K: seven of the eight CTAs of the cluster have none
    (576, 64, 20, 4, 15),    # nine chunks: CTA 0 has two
    (128, 64, 33, 8, 16),    # the most tokens; E just above an expert tile
    (192, 64, 100, 2, 7),
    (1088, 64, 200, 4, 16),  # eight expert tiles
    (576, 64, 20, 4, 17),    # one token more: the separate kernels
])
@pytest.mark.parametrize("form", ["bf16", "f32", "norm"])
def test_front_end(H, I, E, K, T, form):
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + E + T)
    if form != "norm":
        x_bits = synth.make_tokens(T, H, seed=T)
        ref = oracle_case(lw, x_bits)
        res = run_gpu(shape, lw, x_bits, capi.GEMM_TCGEN05, dtype=form)
    else:
        g = torch.Generator().manual_seed(T)
        x = (3.0 * torch.randn(T, H, generator=g)).float()
        w = (1.0 + 0.2 * torch.randn(H, generator=g)).float()
        x_bits = synth.bf16_bits(torch.from_numpy(oracle.rmsnorm(x.numpy(), w.numpy())))
        ref = oracle_case(lw, x_bits)
        with pkg.MoEEngine(shape, max_tokens=T) as eng:
            eng.load_layer(0, lw)
            out, sc, ti, tw = eng.forward_norm(0, x.cuda(), w.cuda(), side=True)
            h = eng.last_intermediate(T)
            torch.cuda.synchronize()
            assert eng.device_status() == 0
            res = {"out": out.cpu().numpy(), "score": sc.cpu().numpy(), "topk_i": ti.cpu().numpy(),
                   "topk_w": tw.cpu().numpy(), "h_bits": h.cpu().numpy().view(np.uint16),
                   "counts": eng.last_expert_counts()}
    compare(res, ref, K, f"{(H, I, E, K, T, form)}")
    assert np.abs(res["score"] - ref["router_score"]).max() < 1e-5
    assert list(np.bincount(ref["topk_i"].reshape(-1), minlength=E)) == res["counts"]


def _row_at_a_rounding_edge(H):
    """A row and the weight of its first column for which the order of the norm's additions
    shows.  Sum of squares = a float midpoint m (the squares of columns 0 and 1) and twelve
    squares of a quarter of m's ulp in double, in three groups of four: added to m one by one
    they are all lost, group by group they are not.  Which of the two is stored moves the
    scale by one ulp, and the weight puts column 0 on a bf16 rounding edge between the two."""
    x = np.zeros(H, np.float32)
    x[0], x[1] = np.float32(1109804032.0), np.float32(2.0**18)
    for k in (32, 64, 96):  # float4 columns: one lane of a warp in both kernels
        x[4 * k:4 * k + 4] = 8.0
    m = float(x[0] * x[0]) + float(x[1] * x[1])
    scales = [np.float32(1.0) / np.sqrt(np.float32((m + d) / H + float(np.float32(1e-5)))) for d in (0.0, 768.0)]
    assert scales[0] != scales[1]
    w = np.float32(0.99)
    for _ in range(1 << 17):
        rows = torch.tensor([float(np.float32(float(w) * (float(s) * float(x[0])))) for s in scales])
        if rows.bfloat16()[0] != rows.bfloat16()[1]:
            return torch.from_numpy(x), float(w)
        w = np.nextafter(w, np.float32(2.0))
    raise AssertionError("no weight found")


@pytest.mark.parametrize("H,E,T,edge", [(512, 8, 16, True), (512, 8, 16, False), (2880, 32, 16, False),
                                        (4160, 20, 8, False)])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
def test_a_row_does_not_depend_on_the_kernel_that_normed_it(H, E, T, edge, w_dtype):
    """The first T rows in a batch of T (one launch) and of T + 1 (rows_to_bf16_kernel)."""
    shape = pkg.MoEShape(hidden=H, intermediate=64, n_experts=E, top_k=2)
    g = torch.Generator().manual_seed(H)
    x = (3.0 * torch.randn(T + 1, H, generator=g)).float()
    w = (1.0 + 0.2 * torch.randn(H, generator=g)).float()
    if edge:
        x[0], w[0] = _row_at_a_rounding_edge(H)
    with pkg.MoEEngine(shape, max_tokens=T + 1) as eng:
        eng.load_layer(0, synth.make_layer(shape, seed=H))
        w = w.to(w_dtype).cuda()
        a = [v.cpu() for v in eng.forward_norm(0, x[:T].cuda(), w, side=True)]
        assert eng.last_launch_count() == 4
        b = [v.cpu()[:T] for v in eng.forward_norm(0, x.cuda(), w, side=True)]
        assert eng.last_launch_count() == 6
        assert eng.device_status() == 0
    for p, q in zip(a, b):
        assert torch.equal(p, q)


@pytest.mark.parametrize("H,I,E,K,T,launches", [
    (576, 64, 20, 4, 1, 4),
    (576, 64, 20, 4, 16, 4),
    # Long rows, with an intermediate of 256: the parity rule allows one rounding flip of h in
    # 1000 elements, about 1 in 2000 is expected at this length, and 9 x 4 x 64 elements are too
    # few to tell the two apart (3 flips against a limit of 2.3).
    (4096, 256, 20, 4, 8, 4),   # a long row for every warp
    (4096, 256, 20, 4, 9, 6),   # one more: the separate kernels
    (4032, 256, 20, 4, 16, 4),  # the longest rows of which a warp takes two
    (2560, 64, 256, 2, 16, 4),  # the largest rows that fit shared memory with 256 experts
    (2624, 64, 256, 2, 16, 6),  # one chunk more: the separate kernels
    (4160, 64, 20, 4, 17, 6),   # rows above 4096 columns: weights fetched after the sum too
])
@pytest.mark.parametrize("w_dtype", [torch.float32, torch.bfloat16])
def test_norm_and_residual_update(H, I, E, K, T, launches, w_dtype):
    """forward_norm against the oracle with both weight types, the path it took, and the
    engine's in-place x += MoE(rmsnorm(x)): one fp32 addition to the same result."""
    shape = pkg.MoEShape(hidden=H, intermediate=I, n_experts=E, top_k=K)
    lw = synth.make_layer(shape, seed=H + E + T)
    g = torch.Generator().manual_seed(T)
    x = (3.0 * torch.randn(T, H, generator=g)).float()
    w = (1.0 + 0.2 * torch.randn(H, generator=g)).to(w_dtype)
    x_bits = synth.bf16_bits(torch.from_numpy(oracle.rmsnorm(x.numpy(), w.float().numpy())))
    ref = oracle_case(lw, x_bits)
    with pkg.MoEEngine(shape, max_tokens=T) as eng:
        eng.load_layer(0, lw)
        out, sc, ti, tw = eng.forward_norm(0, x.cuda(), w.cuda(), side=True)
        assert eng.last_launch_count() == launches
        h = eng.last_intermediate(T)
        stream = x.cuda()
        eng.forward_norm(0, stream, w.cuda(), out=stream, accumulate=True)
        torch.cuda.synchronize()
        assert eng.device_status() == 0
        res = {"out": out.cpu().numpy(), "topk_i": ti.cpu().numpy(), "topk_w": tw.cpu().numpy(),
               "h_bits": h.cpu().numpy().view(np.uint16)}
        assert torch.equal(stream.cpu(), x + out.cpu())
    compare(res, ref, K, f"{(H, I, E, K, T, w_dtype)}")


@pytest.mark.parametrize("H", [576, 4160])
def test_norm_with_early_and_late_weights(H):
    """rows_to_bf16_kernel fetches its norm weights ahead of the sum up to three rows per SM: the
    last batch that does and the first that does not give the same bits (both are 28 routing
    blocks on 148 SMs, so the router splits K alike)."""
    T = 3 * torch.cuda.get_device_properties(0).multi_processor_count
    shape = pkg.MoEShape(hidden=H, intermediate=64, n_experts=20, top_k=2)
    g = torch.Generator().manual_seed(H)
    x = (3.0 * torch.randn(T + 1, H, generator=g)).float().cuda()
    w = (1.0 + 0.2 * torch.randn(H, generator=g)).float().cuda()
    with pkg.MoEEngine(shape, max_tokens=T + 1) as eng:
        eng.load_layer(0, synth.make_layer(shape, seed=H))
        early = eng.forward_norm(0, x[:T], w, side=True)
        late = eng.forward_norm(0, x, w, side=True)
        torch.cuda.synchronize()
        assert eng.device_status() == 0
    for p, q in zip(early, late):
        assert torch.equal(p, q[:T])
