"""Which memory the combine kernel stores the caller's routing to itself, and which gets a copy.  A
copy reaches memory that no store of the handle's device may touch -- another GPU's without peer
access -- and answers with an error code where a store would fault."""
import ctypes

import pytest
import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import capi, synth

UNREGISTERED, HOST, DEVICE, MANAGED = range(4)  # cudaMemoryType


@pytest.mark.parametrize("kind,owner,address,stored", [
    (DEVICE, 0, 0x7F0000000000, True),
    (DEVICE, 0, 0x7F0000000004, True),
    (DEVICE, 0, 0x7F0000000002, False),
    (DEVICE, 0, 0x7F0000000001, False),
    (DEVICE, 1, 0x7F0000000000, False),  # another GPU
    (HOST, 0, 0x7F0000000000, False),
    (MANAGED, 0, 0x7F0000000000, False),
    (UNREGISTERED, -1, 0x7F0000000000, False),  # a plain host pointer
    (UNREGISTERED, -2, 0x7F0000000000, False),
    (DEVICE, 0, 0, False),  # not asked for
])
def test_where_a_kernel_may_store(kind, owner, address, stored):
    f = capi.lib(test_aids=True).moe_b200_test_word_store
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_ulonglong, ctypes.c_int]
    assert f(kind, owner, address, 0) == int(stored)
    assert f(kind, owner + 3, address, 3) == int(stored)


@pytest.mark.gpu
def test_pinned_host_memory_and_capture():
    """The routing in pinned host memory, and in device memory from a captured call."""
    T, K = 40, 4
    shape = pkg.MoEShape(hidden=128, intermediate=64, n_experts=32, top_k=K)
    x = torch.from_numpy(synth.bf16_bits_to_f32(synth.make_tokens(T, 128, seed=1))).cuda().to(torch.bfloat16)
    with pkg.MoEEngine(shape, max_tokens=T) as eng:
        eng.load_layer(0, synth.make_layer(shape, seed=2))
        out, _, ti, tw = eng.forward(0, x, side=True)
        pinned = torch.zeros(T, K, dtype=torch.int32).pin_memory()
        capi.check(eng._lib.moe_b200_forward(
            eng._h, 0, ctypes.c_void_p(x.data_ptr()), capi.DTYPE_BF16, T, ctypes.c_void_p(out.data_ptr()), 0, None,
            ctypes.c_void_p(pinned.data_ptr()), None, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
            eng._h, eng._lib)
        torch.cuda.synchronize()
        assert torch.equal(pinned, ti.cpu())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out2, _, ti2, tw2 = eng.forward(0, x, side=True)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out2, out) and torch.equal(ti2, ti) and torch.equal(tw2, tw)
