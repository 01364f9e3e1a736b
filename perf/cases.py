"""The work that this framework is used for, as cases that can be timed and compared.

A case is one call of a compiled graph through ``DAGExecutor.execute`` with its inputs on the GPU: a
decode step or a prompt of the Qwen2.5-1.5B architecture (bf16), or a batch of images through a
ResNet (fp16).  ``listed`` names the sizes that matter by name, ``draw`` takes others from the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` makes the call, ``work``
counts what the call cannot do without and ``tolerance`` bounds how far another correct
implementation may be away.
"""

from __future__ import annotations

import functools
import sys
from pathlib import Path

import torch

# the package of the tree in the working folder, whichever tree this file itself lies in
sys.path.insert(0, str(Path.cwd() / "pytorch-apple_b200"))

import model_zoo as mz  # noqa: E402
from cuda_compiler import compile_subgraph, is_cuda_op_supported  # noqa: E402
from cuda_runtime import CUDABackend, CUDABuffer  # noqa: E402
from ir_export import extract_ir  # noqa: E402
from npu_compiler import partition  # noqa: E402
from npu_runtime import DAGExecutor  # noqa: E402

LAYERS = 28          # depth of the language model in every case
MAX_KV_ROWS = 64 * 4352   # rows of one layer's cache over all sequences, largest decode case
MAX_PROMPT = 2048    # tokens of a prompt over all sequences, largest prefill case
MAX_IMAGES = 256


def listed() -> list[dict]:
    return [
        # one chat user: a single sequence with a few thousand tokens behind it
        _decode("decode_b1", 1, 4352, 4096),
        # one sequence over the longest cache the model has, well filled: summarising a long document
        _decode("decode_b1_long", 1, 32768, 20000),
        # a small server: eight sequences in lock step
        _decode("decode_b8", 8, 4352, 4096),
        # odd batch, short cache of an odd length, half filled: the middle of a chat with few users
        _decode("decode_b19_ragged", 19, 1111, 613),
        # the throughput case: 64 sequences with 4096 tokens each
        _decode("decode_b64", 64, 4352, 4096),
        # a short question, the prompt length that the decode sweep uses before its first token
        _prefill("prefill_t128", 1, 128),
        # the prompt length of the headline prefill number
        _prefill("prefill_t512", 1, 512),
        # a prompt as it comes, not padded to anything
        _prefill("prefill_t777", 1, 777),
        # a long prompt: a document with a question
        _prefill("prefill_t2048", 1, 2048),
        # one image at a time: an interactive classifier
        _resnet("resnet50_b1", 50, 1),
        # a server's batch
        _resnet("resnet50_b32", 50, 32),
        # offline classification
        _resnet("resnet50_b256", 50, 256),
    ]


def _decode(name: str, batch: int, cache: int, filled: int) -> dict:
    return {"name": name, "kind": "decode", "batch": batch, "cache": cache, "filled": filled}


def _prefill(name: str, batch: int, tokens: int) -> dict:
    return {"name": name, "kind": "prefill", "batch": batch, "tokens": tokens}


def _resnet(name: str, depth: int, batch: int) -> dict:
    return {"name": name, "kind": "resnet", "depth": depth, "batch": batch}


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number from lo to hi, evenly over its logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "resnet"))
    if kind == "decode":
        batch = _spread(rng, 1, 64)
        cache = _spread(rng, 300, min(32768, MAX_KV_ROWS // batch))
        case = _decode("", batch, cache, rng.randrange(cache // 8, cache))
    elif kind == "prefill":
        tokens = _spread(rng, 16, MAX_PROMPT)
        case = _prefill("", min(rng.choice((1, 1, 2, 4)), MAX_PROMPT // tokens), tokens)
    else:
        case = _resnet("", rng.choice((18, 50, 50)), _spread(rng, 1, MAX_IMAGES))
    del case["name"]
    return case


# The graph is what a program reads from its IR file; exporting it again for each set of inputs would
# only repeat the exporter.
@functools.lru_cache(maxsize=None)
def _ir(kind: str, *size: int) -> dict:
    if kind == "resnet":
        depth, batch = size
        return extract_ir(mz.resnet(depth, device="meta"), (torch.zeros(batch, 3, 224, 224, device="meta"),), f"resnet{depth}")
    cfg = mz.qwen2_config(num_layers=LAYERS)
    model = mz.qwen2_model(cfg)
    if kind == "decode":
        batch, cache = size
        return extract_ir(mz.QwenDecodeWrapper(model, LAYERS), mz.qwen2_example_inputs(cfg, batch, 1, cache), "qwen2_decode")
    batch, tokens = size
    return extract_ir(mz.QwenPrefillWrapper(model), mz.qwen2_example_inputs(cfg, batch, tokens, None), "qwen2_prefill")


def _graph(case: dict) -> dict:
    keys = {"decode": ("batch", "cache"), "prefill": ("batch", "tokens"), "resnet": ("depth", "batch")}[case["kind"]]
    return _ir(case["kind"], *(case[k] for k in keys))


@functools.lru_cache(maxsize=None)
def _resnet_checkpoint(depth: int) -> dict:
    return mz.state_dict_numpy(mz.resnet(depth, seed=0).state_dict())


def _qwen_checkpoint(cfg, device) -> dict:
    """Seeded weights in which, as in a trained network, a layer changes the residual stream by a small
    share.  With the equal scales that the zoo draws, every layer remakes the stream: rounding is then
    amplified until two correct bf16 evaluations of 28 layers are 4.5 % apart in the logits (1.5 % here)."""
    weights = mz.qwen2_weights(cfg, seed=0, device=str(device))
    for name, w in weights.items():
        if "o_proj" in name:
            w.mul_(0.1)
        elif "down_proj" in name:
            w.mul_(0.005)
    return weights


def prepare(case: dict, seed: int) -> dict:
    """The executor with its weights loaded, and one call's inputs on the GPU."""
    device = torch.device("cuda", 0)
    ir = _graph(case)
    names = [s["name"] for s in ir["graph_inputs"]]
    g = torch.Generator(device=device).manual_seed(seed)
    if case["kind"] == "resnet":
        weights = _resnet_checkpoint(case["depth"])
        inputs = [torch.randn(case["batch"], 3, 224, 224, device=device, generator=g).half()]
    else:
        cfg = mz.qwen2_config(num_layers=LAYERS)
        weights = {k: CUDABuffer(v) for k, v in _qwen_checkpoint(cfg, device).items()}
        batch = case["batch"]
        if case["kind"] == "decode":   # every sequence holds `filled` tokens and gets its next one
            pos, q_len, kv_len = case["filled"], 1, case["cache"]
        else:
            pos, q_len, kv_len = 0, case["tokens"], case["tokens"]
        at = torch.arange(pos, pos + q_len, device=device)
        inputs = [torch.randint(0, cfg.vocab_size, (batch, q_len), device=device, generator=g),
                  mz.causal_mask(batch, q_len, kv_len, pos).to(device), at[None].expand(batch, q_len).contiguous(), at]
        while len(inputs) < len(names):   # key and value caches
            inputs.append((torch.randn(batch, cfg.num_key_value_heads, kv_len, 128, device=device, generator=g) * 0.5).bfloat16())
    dag = DAGExecutor(partition(ir, is_cuda_op_supported), CUDABackend(device.index), compile_subgraph)
    dag.load_weights(weights)
    return {"dag": dag, "inputs": {n: CUDABuffer(t) for n, t in zip(names, inputs)}}


def run(state: dict) -> dict:
    """Logits and key / value caches of a language model, logits of a classifier."""
    return {name: buf.native_handle for name, buf in state["dag"].execute(state["inputs"]).items()}


def work(case: dict) -> dict:
    """Weights, inputs and outputs once each; of a cache the rows in use and the row that is new.  A
    causal mask leaves half of the score matrix."""
    if case["kind"] == "resnet":
        ir = _graph(case)
        flops = params = 0
        for node in ir["nodes"]:
            shapes = [t["shape"] for t in node["inputs"]]
            if node["op_type"].startswith(("aten.conv2d", "aten.linear")):
                out = node["outputs"][0]["shape"]
                per_out = functools.reduce(lambda a, b: a * b, shapes[1][1:], 1)
                flops += 2 * per_out * functools.reduce(lambda a, b: a * b, out, 1)
                params += per_out * shapes[1][0]
        images = case["batch"]
        return {"bytes": 2 * (params + images * (3 * 224 * 224 + 1000)), "flops": flops}
    cfg = mz.qwen2_config(num_layers=LAYERS)
    H, I, V, L = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, cfg.num_hidden_layers
    heads, kv = cfg.num_attention_heads, cfg.num_key_value_heads * 128
    layer = 2 * H * H + 2 * kv * H + 3 * H * I
    weights = 2 * (L * (layer + H + 2 * kv + 2 * H) + V * H + H)
    batch = case["batch"]
    if case["kind"] == "decode":
        rows = case["filled"] + 1
        moved = batch * (L * 2 * kv * rows * 2 + L * 2 * kv * 2 + 2 * V + 2 * case["cache"])
        flops = batch * (2 * (L * layer + V * H) + L * heads * 4 * rows * 128)
    else:
        T = case["tokens"]
        moved = batch * T * (L * 2 * kv * 2 + 2 * V + 2 * T)
        flops = batch * (2 * T * (L * layer + V * H) + L * heads * 2 * T * (T + 1) * 128)
    return {"bytes": weights + moved, "flops": flops}


def tolerance(case: dict) -> dict:
    """From the compiler's fused and unfused evaluations of the same inputs (other orders of the sums, and
    for decode other rounding points): decode logits 1.5 % apart and single values up to 0.10 of the rms,
    prompts 1.0 % and 0.06, ResNet-50 0.09 % and 0.003 (0.07 % from float64)."""
    if case["kind"] == "resnet":
        return {"rel": 0.0035, "max": 0.0125}
    return {"rel": 0.03, "max": 0.4 if case["kind"] == "decode" else 0.25}
