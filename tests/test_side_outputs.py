"""The routing that the combine kernel stores for the caller: both arrays, one of them, and pointers
that no 4-byte store may take (those are copied), in front of the small kernels, the permute's plan
and the plan kernel."""
import ctypes

import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 16, 17, 300, 900])
@pytest.mark.parametrize("K", [1, 4, 8])
def test_routing_for_the_caller(T, K):
    shape = pkg.MoEShape(hidden=128, intermediate=64, n_experts=32, top_k=K)
    lw = synth.make_layer(shape, seed=K)
    x = torch.from_numpy(synth.bf16_bits_to_f32(synth.make_tokens(T, 128, seed=T))).cuda().to(torch.bfloat16)
    with pkg.MoEEngine(shape, max_tokens=T) as eng:
        eng.load_layer(0, lw)
        out, score, ti, tw = eng.forward(0, x, side=True)
        want = score.topk(K, dim=-1)
        assert torch.equal(ti.long(), want.indices)
        assert torch.allclose(tw, torch.softmax(want.values, dim=-1), rtol=1e-5, atol=0)  # fp32, a few roundings
        for shift, with_i, with_w in [(0, True, False), (0, False, True), (1, True, True), (2, True, True)]:
            buf = [torch.full((T * K * 4 + 8,), 0x5A, dtype=torch.uint8, device="cuda") for _ in range(2)]
            ptr = [ctypes.c_void_p(b.data_ptr() + shift) if on else None for b, on in zip(buf, (with_i, with_w))]
            again = torch.empty_like(out)
            capi.check(eng._lib.moe_b200_forward(
                eng._h, 0, ctypes.c_void_p(x.data_ptr()), capi.DTYPE_BF16, T, ctypes.c_void_p(again.data_ptr()), 0,
                None, ptr[0], ptr[1], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), eng._h, eng._lib)
            assert torch.equal(again, out)
            for b, on, ref in zip(buf, (with_i, with_w), (ti, tw)):
                end = shift + T * K * 4
                if on:
                    assert torch.equal(b[shift:end].clone().view(torch.int32), ref.flatten().view(torch.int32))
                assert bool((b[:shift] == 0x5A).all()) and bool((b[end if on else 0:] == 0x5A).all())
