"""The work that a user of this package has it do, as cases that can be timed and compared.

Layer shapes are the K x N of the decoder, vision-tower and action-head linears of the benchmark
and of the synthetic policy; codebook layouts are the mixed-bit set of the benchmark and the
dim-4 / 64-wide-scale-group layouts that the tests call deployed; token counts go from one decode
token to the batched sweep's 8,192.  Weights are N(0, 0.02) cut into vectors and assigned to the
nearest of a sampled codebook, activations N(0, 1) with 1 % of the channels twenty times larger.

A case is a dict: `op` names the entry point, `m` tokens, `k` x `n` the layer, `d`, `codebook` and
`group` (0: one scale per output row) its layout, `bias` whether it has one.  A transformer block has
`k` as its hidden and `n` as its MLP width, `heads` query and `kv_heads` key/value heads, a gated or a
GELU MLP, and modulated or affine norms."""
import math

import torch
import torch.nn.functional as F

from sacq_b200 import (PrecomputedPackedVectorCodebookLinear, act_quantize_rows, index_bits_for, layernorm_quantize_rows,
                       linear_a8_multi, quantize_rows)

DEVICE = "cuda:0"

# K x N of the linears: decoder q/o, k/v, gate/up, down; vision tower; action head
SHAPES = ((2048, 2048), (2048, 1024), (2048, 6144), (6144, 2048), (1024, 1024), (1024, 4096), (4096, 1024), (1536, 1536),
          (2048, 1536), (1536, 6144), (6144, 1536))
# (vector dim, codebook entries, scale group): 1, 1.5, 2 and 3 bits per weight, and the deployed dim-4 layouts
LAYOUTS = ((8, 4096, 0), (8, 256, 0), (8, 65536, 0), (4, 4096, 0), (4, 64, 64), (4, 128, 64), (4, 1024, 64), (4, 2048, 64))
MOST_TOKENS = 8192
MOST_BLOCK_TOKENS = 1024
# transformer blocks of the synthetic policy: language model, vision tower, action head
BLOCKS = ({"k": 2048, "n": 6144, "heads": 16, "kv_heads": 8, "gated": True, "modulated": False},
          {"k": 1024, "n": 4096, "heads": 16, "kv_heads": 16, "gated": False, "modulated": False},
          {"k": 1536, "n": 6144, "heads": 12, "kv_heads": 12, "gated": False, "modulated": True})


def _case(name, op, m, k, n, d=8, codebook=4096, group=0, bias=False):
    return {"name": name, "op": op, "m": m, "k": k, "n": n, "d": d, "codebook": codebook, "group": group, "bias": bias}


def listed():
    return [
        # one token through the smallest projection of a decoder: nothing but latency
        _case("decode_kv_m1", "linear", 1, 2048, 1024),
        # a small decode batch through a gate/up projection
        _case("decode_gate_up_m16", "linear", 16, 2048, 6144),
        # a large decode batch through the deep down projection
        _case("decode_down_m64", "linear", 64, 6144, 2048),
        # a control loop that hands over host activations and reads host results (pinned buffers)
        _case("host_q_m4", "host", 4, 2048, 2048),
        # the 2 bits per weight layer: a codebook that does not fit on chip
        _case("two_bit_m16", "linear", 16, 2048, 6144, codebook=65536),
        # a deployed dim-4 layout with grouped scales and a bias, ragged token count
        _case("deployed_m41", "linear", 41, 2048, 2048, d=4, codebook=1024, group=64, bias=True),
        # the same kind of layer on INT8 activations, an action head's 16 steps
        _case("int8_activations_m16", "linear_int8", 16, 1536, 1536, d=4, codebook=1024, group=64),
        # the deployed INT8 recipe (8-bit weight rows, exact integer sums), ragged prefill
        _case("int8_recipe_m149", "int8_recipe", 149, 2048, 6144, d=4, codebook=1024, group=64),
        # the FP8 recipe on a batch of prefills
        _case("fp8_recipe_m1024", "fp8_recipe", 1024, 6144, 2048),
        # a transformer block of the action head on its 16-step horizon: modulated norms, attention, GELU MLP
        dict(_case("action_block_m16", "block", 16, 0, 0), **BLOCKS[2]),
        # a language-model block on a 300-token prefill: grouped-query attention, gated MLP
        dict(_case("prefill_block_m300", "block", 300, 0, 0), **BLOCKS[0]),
        # the batched throughput sweep's largest call
        _case("batched_gate_up_m8192", "linear", 8192, 2048, 6144),
    ]


def draw(rng):
    op = rng.choice(("linear",) * 6 + ("host", "linear_int8", "int8_recipe", "fp8_recipe", "block"))
    k, n = rng.choice(SHAPES)
    most = MOST_TOKENS
    if op == "block":
        most = MOST_BLOCK_TOKENS
    elif op == "host":
        most = 256
    elif rng.random() < 0.1:
        n -= rng.randint(1, 63)                       # an output width that is no multiple of anything
    m = max(1, min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1))))))
    # half of the layers have the 1.5 bits per weight layout
    d, codebook, group = LAYOUTS[0] if rng.random() < 0.5 else rng.choice(LAYOUTS[1:])
    case = _case("", op, m, k, n, d, codebook, group, rng.random() < 0.3)
    if op == "block":
        case.update(rng.choice(BLOCKS))
    del case["name"]
    return case


# ----------------------------------------------------------------------------- inputs

def _pack(indices, bits):
    """The little-endian bit stream of flat indices (on the GPU)."""
    planes = ((indices.unsqueeze(1) >> torch.arange(bits, device=indices.device)) & 1).to(torch.uint8).reshape(-1)
    if planes.numel() % 8:
        planes = torch.cat([planes, planes.new_zeros(8 - planes.numel() % 8)])
    weights = (1 << torch.arange(8, device=indices.device)).to(torch.uint8)
    return (planes.reshape(-1, 8) * weights).sum(dim=1, dtype=torch.uint8)


def _layer(gen, k, n, d, codebook, group, bias):
    group = group or k
    w = (torch.randn(n, k, generator=gen, device=DEVICE) * 0.02).reshape(n, k // group, group)
    scales = w.abs().amax(dim=2, keepdim=True)
    vectors = (w / scales).reshape(-1, d)
    centers = vectors[torch.randint(0, vectors.shape[0], (codebook,), generator=gen, device=DEVICE)].to(torch.bfloat16)
    if codebook > 4096:                               # too many to search: any codeword will do
        indices = torch.randint(0, codebook, (vectors.shape[0],), generator=gen, device=DEVICE)
    else:
        c = centers.float()
        half = 0.5 * (c * c).sum(1)
        indices = torch.cat([(half - v @ c.t()).argmin(dim=1) for v in vectors.split(max(1, (1 << 26) // codebook))])
    bits = index_bits_for(codebook)
    payload = {"format": "packed_vector_codebook_v1", "codebook": centers, "scales": scales.squeeze(-1).to(torch.bfloat16),
               "shift": torch.zeros((), dtype=torch.bfloat16), "in_features": k, "out_features": n, "group_size": group,
               "vector_dim": d, "packed_indices": _pack(indices, bits), "index_bits": bits,
               "index_shape": (n, k // group, group // d)}
    b = (torch.randn(n, generator=gen, device=DEVICE) * 0.05).to(torch.bfloat16) if bias else None
    return PrecomputedPackedVectorCodebookLinear(payload, b, DEVICE)


def _activations(gen, m, k):
    x = torch.randn(m, k, generator=gen, device=DEVICE)
    x[:, torch.randperm(k, generator=gen, device=DEVICE)[:k // 100]] *= 20.0
    return x.to(torch.bfloat16)


def prepare(case, seed):
    op = case["op"]
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    m, k, n = case["m"], case["k"], case["n"]
    layout = (case["d"], case["codebook"], case["group"], case["bias"])
    x = _activations(gen, m, k)
    state = {"op": op, "x": x}
    if op == "block":
        vec = lambda at: (torch.randn(k, generator=gen, device=DEVICE) * 0.1 + at).to(torch.bfloat16)  # noqa: E731
        kv = k // case["heads"] * case["kv_heads"]
        state["heads"] = case["heads"]
        # per norm: weight, bias, epsilon, modulation scale and shift
        state["norms"] = [(None, None, 1e-5, vec(0.0), vec(0.0)) if case["modulated"] else (vec(1.0), vec(0.0), 1e-5, None, None)
                          for _ in range(2)]
        state["qkv"] = [_layer(gen, k, width, *layout) for width in (k, kv, kv)]
        state["o"] = _layer(gen, k, k, *layout)
        state["up"] = [_layer(gen, k, n, *layout) for _ in range(2 if case["gated"] else 1)]
        state["down"] = _layer(gen, n, k, *layout)
        return state
    layer = state["layer"] = _layer(gen, k, n, *layout)
    if op == "host":
        state["x"] = x.cpu().pin_memory()
        state["y"] = torch.empty(m, n, dtype=torch.bfloat16).pin_memory()
    elif op in ("int8_recipe", "fp8_recipe"):
        state["mode"] = "int8_symmetric" if op == "int8_recipe" else "fp8_e4m3fn"
        state["row_scale"] = layer.weight_row_scale(state["mode"])      # kept with the layer, like its other scales
    return state


@torch.no_grad()
def run(state):
    op = state["op"]
    if op == "linear":
        return state["layer"](state["x"])
    if op == "host":
        return state["layer"].forward_host(state["x"], state["y"])
    if op == "linear_int8":
        return state["layer"].forward_int8(state["x"])
    if op == "int8_recipe":
        q, s = quantize_rows(state["x"], state["mode"])
        return state["layer"].linear_w8a8_int8(q, s, state["row_scale"])
    if op == "fp8_recipe":
        q, s = quantize_rows(state["x"], state["mode"])
        return state["layer"].linear_w8a8_fp8(q, s, state["row_scale"])
    return _block(state)


def _block(state):
    x, heads = state["x"], state["heads"]
    m, k = x.shape
    q, s = layernorm_quantize_rows(x, *state["norms"][0])
    qh, kh, vh = (t.view(1, m, -1, k // heads).transpose(1, 2) for t in linear_a8_multi(state["qkv"], q, s))
    a = F.scaled_dot_product_attention(qh, kh, vh, enable_gqa=kh.shape[1] != heads)
    x = state["o"].forward_residual(a.transpose(1, 2).reshape(m, k), x)
    q, s = layernorm_quantize_rows(x, *state["norms"][1])
    if len(state["up"]) == 2:
        q, s = act_quantize_rows("silu_mul", *linear_a8_multi(state["up"], q, s))
    else:
        q, s = act_quantize_rows("gelu", state["up"][0].linear_a8(q, s))
    return state["down"].linear_a8(q, s, residual=x)


# ----------------------------------------------------------------------------- what a pass cannot do without

def _layer_bytes(case, k, n):
    """Packed indices, codebook, scales and bias of one layer."""
    d, codebook = case["d"], case["codebook"]
    return (n * (k // d) * index_bits_for(codebook) / 8 + codebook * d * 2 + n * (k // (case["group"] or k)) * 2
            + (2 * n if case["bias"] else 0))


def work(case):
    op, m, k, n = case["op"], case["m"], case["k"], case["n"]
    if op == "block":
        kv = k // case["heads"] * case["kv_heads"]
        linears = [(k, k), (k, kv), (k, kv), (k, k)] + [(k, n)] * (2 if case["gated"] else 1) + [(n, k)]
        return {"bytes": sum(_layer_bytes(case, *kn) for kn in linears) + 2 * m * k * 2 + 4 * k * 2,
                "flops": sum(2.0 * m * a * b for a, b in linears) + 4.0 * m * m * k}
    kept = 4 * n if op in ("int8_recipe", "fp8_recipe") else 0                 # the recipe's row scales
    return {"bytes": _layer_bytes(case, k, n) + m * k * 2 + m * n * 2 + kept, "flops": 2.0 * m * n * k}


def tolerance(case):
    op = case["op"]
    if op == "int8_recipe":
        return "exact"                                # integer sums and a fixed order of roundings behind them
    if op == "block":
        # three e4m3 roundings (6 % steps) follow a product: a last bit that differs in front of one moves a few
        # per cent of its values by a step
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 5e-3, "max": 5e-2}                 # sums in fp32, one bf16 rounding of the result
