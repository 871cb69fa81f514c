"""What the performance of this framework is measured on: the calls that an inference
engine makes into the MoE block, from one token of a single stream to a full prefill
batch, over both model shapes of the benchmark (32 and 128 experts, top-4, hidden =
intermediate = 2880) and a generic narrower one.

A case is a dict of plain values:

  op        "forward"  MoEEngine.forward, device buffers in and out
            "norm"     MoEEngine.forward_norm with accumulate: x += MoE(rmsnorm(x))
            "host"     MoEEngine.forward_host, pinned host buffers in and out
            "unpack"   mxfp4_unpack of whole expert matrices to bf16
  H I E K   hidden, intermediate, experts, experts per token
  layers    layers walked in one pass, each with weights and token rows of its own (the
            attention between two layers is the caller's and not part of this framework)
  tokens    rows per call ("unpack": rows of the matrix)
  dtype     activations, "bf16" or "f32" ("norm": the norm weight, the stream is fp32)
  side      router scores, indices and routing weights are asked for too
  zipf      skewed router (busiest expert about four times the mean)

Values are those of the benchmark's synthetic checkpoint (synth.py): N(0, 1) activations,
uniform e2m1 codes, scale exponents -8..-4, small biases; everything follows from the seed.
"""
import math

import torch

import gpt_oss_amd_b200 as pkg
from gpt_oss_amd_b200 import synth

_BASE = dict(op="forward", H=2880, I=2880, E=32, K=4, layers=1, tokens=64, dtype="bf16", side=False, zipf=False)


def _case(**kw):
    return {**_BASE, **kw}


def listed():
    return [
        # one user's generation: every layer streams the four experts of a single token
        _case(name="single_stream", op="norm", layers=24, tokens=1, dtype="f32"),
        # the serving loop at its usual batch: all experts of all layers are streamed once
        _case(name="decode_256x24", layers=24, tokens=256),
        # one layer with the engine's side buffers, a half-empty serving batch
        _case(name="layer_64_side", tokens=64, side=True),
        # the larger model's decode batch, residual update with the engine's bf16 norm weights
        _case(name="decode_e128_200", op="norm", E=128, layers=2, tokens=200, dtype="bf16"),
        # a ragged mixed batch (some prompts, some decodes), fp32 activations
        _case(name="mixed_777_f32", tokens=777, dtype="f32"),
        # a short prefill chunk of the larger model, residual update, odd length
        _case(name="chunk_e128_3001", op="norm", E=128, tokens=3001, dtype="f32"),
        # skewed prefill: a few experts take most of the rows
        _case(name="prefill_zipf_8192", tokens=8192, zipf=True),
        # the largest batch, uniform routing
        _case(name="prefill_e128_16384", E=128, tokens=16384),
        # an engine that keeps its activations on the host: a small step and a full batch
        _case(name="host_48_f32", op="host", tokens=48, dtype="f32", side=True),
        _case(name="host_e128_16384", op="host", E=128, tokens=16384),
        # another model shape: narrow experts, eight of 128 per token
        _case(name="narrow_k8_1500", H=2048, I=768, E=128, K=8, tokens=1500),
        # a layer's gate/up matrices unpacked to bf16 for another consumer
        _case(name="unpack_layer", op="unpack", E=32, tokens=32 * 5760),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = max(work(c)["flops"] for c in listed())
    while True:
        op = rng.choice(["forward", "forward", "forward", "norm", "norm", "host", "unpack"])
        c = _case(op=op, dtype=rng.choice(["bf16", "f32"]), side=rng.random() < 0.3, tokens=log_int(1, 16384))
        shape = rng.random()
        if shape < 0.35:
            c["E"] = 128
        elif shape < 0.65:
            c.update(H=64 * rng.randint(8, 64), I=64 * rng.randint(4, 45), E=rng.randint(16, 128), K=rng.randint(2, 8))
        c["zipf"] = rng.random() < 0.2
        if op == "unpack":
            c.update(tokens=log_int(64, 32 * 5760), H=32 * rng.randint(8, 128), side=False, zipf=False, dtype="bf16")
        elif c["tokens"] <= 256 and c["E"] <= 64:
            c["layers"] = rng.randint(1, 8)
        if op == "host":
            c["layers"] = 1
        if work(c)["flops"] <= most:
            return c


def _shape(case):
    return pkg.MoEShape(hidden=case["H"], intermediate=case["I"], n_experts=case["E"], top_k=case["K"])


def _random_bytes(shape, gen):
    n = math.prod(shape)
    words = torch.randint(-2**63, 2**63 - 1, ((n + 7) // 8,), generator=gen, device="cuda", dtype=torch.int64)
    return words.view(torch.uint8)[:n].view(shape)


def _scales(shape, gen):
    return torch.randint(127 - 8, 127 - 4 + 1, shape, generator=gen, device="cuda", dtype=torch.uint8)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 + seed)
    H, I, E, L, T = case["H"], case["I"], case["E"], case["layers"], case["tokens"]
    if case["op"] == "unpack":
        return {"case": case, "blocks": _random_bytes((T, H // 32, 16), gen), "scales": _scales((T, H // 32), gen)}

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    eng = pkg.MoEEngine(_shape(case), n_layers=L, max_tokens=T)
    for layer in range(L):
        zipf = dict(zipf_s=1.1, zipf_gain=synth.ZIPF_GAIN_4X) if case["zipf"] else {}
        eng.set_router(layer, *synth.make_router(_shape(case), seed=seed * 64 + layer, **zipf))
        experts = (_random_bytes((E, 2 * I, H // 32, 16), gen), _scales((E, 2 * I, H // 32), gen),
                   0.01 * randn(E, 2 * I), _random_bytes((E, H, I // 32, 16), gen),
                   _scales((E, H, I // 32), gen), 0.01 * randn(E, H))
        torch.cuda.synchronize()  # the upload runs on a stream of its own
        eng.set_experts(layer, 0, *experts)
    del experts
    state = {"case": case, "eng": eng}
    if case["op"] == "norm":
        state["x"] = randn(L, T, H)
        w = 1.0 + 0.1 * randn(L, H)
        state["w"] = w.to(torch.bfloat16) if case["dtype"] == "bf16" else w
    else:
        state["x"] = randn(L, T, H).to(torch.bfloat16)
        if case["dtype"] == "f32":
            state["x"] = randn(L, T, H)
    state["out"] = torch.empty(L, T, H, dtype=torch.float32, device="cuda")
    if case["op"] == "host":
        state["x"] = state["x"][0].cpu().pin_memory()
        state["out"] = torch.empty(T, H, dtype=torch.float32).pin_memory()
        if case["side"]:
            state["topk_i"] = torch.empty(T, case["K"], dtype=torch.int32).pin_memory()
            state["topk_w"] = torch.empty(T, case["K"], dtype=torch.float32).pin_memory()
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "unpack":
        return pkg.mxfp4_unpack(state["blocks"], state["scales"])
    eng, x, out = state["eng"], state["x"], state["out"]
    if op == "host":
        ti, tw = state.get("topk_i"), state.get("topk_w")
        eng.forward_host(0, x, out, ti, tw)
        return (out, ti, tw) if case["side"] else out
    if op == "norm":
        out.copy_(x)  # the residual stream that the attention in front of the block leaves
    side = []
    for layer in range(case["layers"]):
        if op == "norm":
            r = eng.forward_norm(layer, out[layer], state["w"][layer], out=out[layer], accumulate=True,
                                 side=case["side"])
        else:
            r = eng.forward(layer, x[layer], out=out[layer], side=case["side"])
        if case["side"]:
            side.append(r[1:])
    return (out, side) if case["side"] else out


def _active_experts(case):
    """Experts that at least one token picks: expected value for uniform routing."""
    return case["E"] * (1.0 - (1.0 - case["K"] / case["E"]) ** case["tokens"])


def work(case):
    H, I, E, K, L, T = (case[k] for k in ("H", "I", "E", "K", "layers", "tokens"))
    if case["op"] == "unpack":
        return {"bytes": T * H * (0.5 + 1 / 32 + 2), "flops": 0}
    per_expert = 3 * I * H * (0.5 + 1 / 32) + (2 * I + H) * 4
    x_bytes = 4 if case["op"] == "norm" or case["dtype"] == "f32" else 2
    per_layer = _active_experts(case) * per_expert + E * H * 2 + E * 4 + T * H * (x_bytes + 4)
    if case["op"] == "norm":
        per_layer += H * (2 if case["dtype"] == "bf16" else 4)
    if case["side"]:
        per_layer += T * (K * 8 + (0 if case["op"] == "host" else E * 4))
    return {"bytes": L * per_layer, "flops": L * synth.moe_flops(T, _shape(case))}


def tolerance(case):
    if case["op"] == "unpack":
        return "exact"  # every e2m1 x e8m0 value is a bf16 number
    # Two correct fp32 evaluations of the gate/up contraction differ in the last bits, so a
    # few of the bf16 intermediates land on the neighbouring value.
    return {"rel": 2e-4, "differ": 2e-4}


_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _dequant64(blocks, scales):
    """[rows, G, 16] e2m1 pairs (even column in the low half) and [rows, G] e8m0 bytes -> [rows, 32 G]."""
    table = torch.tensor(_E2M1, dtype=torch.float64, device=blocks.device)
    v = torch.stack((table[(blocks & 15).long()], table[(blocks >> 4).long()]), dim=-1).flatten(-2)
    return (v * torch.exp2(scales.double() - 127.0).unsqueeze(-1)).flatten(-2)


def exact(case, seed):
    """What run() returns, in 64 bits.  The two roundings to bf16 that the block's contract
    names (its input, and the SwiGLU output in front of the down projection) are part of the
    result; everything between them is not rounded."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000 + seed)
    H, I, E, K, L, T = (case[k] for k in ("H", "I", "E", "K", "layers", "tokens"))
    if case["op"] == "unpack":
        return None  # bytes, compared as they are

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    layers = []
    for layer in range(L):
        zipf = dict(zipf_s=1.1, zipf_gain=synth.ZIPF_GAIN_4X) if case["zipf"] else {}
        wr, br = synth.make_router(_shape(case), seed=seed * 64 + layer, **zipf)
        router = (torch.from_numpy(synth.bf16_bits_to_f32(wr)).cuda().double(), torch.from_numpy(br).cuda().double())
        layers.append((router, (_random_bytes((E, 2 * I, H // 32, 16), gen), _scales((E, 2 * I, H // 32), gen),
                                0.01 * randn(E, 2 * I), _random_bytes((E, H, I // 32, 16), gen),
                                _scales((E, H, I // 32), gen), 0.01 * randn(E, H))))
    x = randn(L, T, H)
    if case["op"] == "norm":
        w = 1.0 + 0.1 * randn(L, H)
        w = w.to(torch.bfloat16) if case["dtype"] == "bf16" else w
    elif case["dtype"] == "f32":
        x = randn(L, T, H)

    out, side = [], []
    for layer, ((wr, br), (b1, s1, c1, b2, s2, c2)) in enumerate(layers):
        t = x[layer].double()
        if case["op"] == "norm":
            t = w[layer].double() * (t / torch.sqrt((t * t).mean(dim=-1, keepdim=True) + 1e-5))
        t = t.float().to(torch.bfloat16).double()
        scores = t @ wr.T + br
        top, index = scores.topk(K, dim=-1)
        weight = torch.softmax(top, dim=-1)
        y = x[layer].double() if case["op"] == "norm" else torch.zeros(T, H, dtype=torch.float64, device="cuda")
        for e in index.unique().tolist():
            rows, k = (index == e).nonzero(as_tuple=True)
            g = t[rows] @ _dequant64(b1[e], s1[e]).T + c1[e].double()
            gate, up = g[:, 0::2].clamp(max=7.0), g[:, 1::2].clamp(-7.0, 7.0)
            h = (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)).to(torch.bfloat16).double()
            y[rows] += weight[rows, k].unsqueeze(-1) * (h @ _dequant64(b2[e], s2[e]).T + c2[e].double())
        out.append(y)
        side.append((scores, None, weight))
    if case["op"] == "host":
        return (out[0], None, side[0][2]) if case["side"] else out[0]
    out = torch.stack(out)
    return (out, side) if case["side"] else out
