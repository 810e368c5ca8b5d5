"""Workloads that the framework's performance is measured on: what a user's program has it do on one GPU, through the
calls that such a program makes.

* ``step``: one optimizer step of ``TrainEngine`` (token batch from pinned host memory, forward, backward, AdamW, loss
  back on the host), on the named shapes of ``models/config.py`` with fewer layers, so that several states fit a GPU:
  a layer is what repeats, and embedding, head, loss and optimizer are there once as in the full model.
* ``attention``: causal grouped-query attention forward and backward at sequence lengths and head sizes that the steps
  above do not reach (long context, many short sequences).
* ``v1_encode`` / ``v1_decode``: the drop-in codec of ``zipccl.hopper_fastzip2`` as the all-gather hook calls it: a rank
  encodes its shard as one work and decodes the streams of all ranks.
* ``v2_encode`` / ``v2_decode``: the codec of the compressed collectives (bit-plane and nibble records).
* ``int8``: quantise and dequantise as the int8 all-gather does.
"""
from __future__ import annotations

import dataclasses
import math
import os
import socket

import torch

from fsdp_comm_opt_b200.engine import EngineConfig, TrainEngine
from fsdp_comm_opt_b200.models import get_config
from fsdp_comm_opt_b200.ops import attention, codec, quant
from fsdp_comm_opt_b200.utils.dist import init_distributed
from zipccl import hopper_fastzip2 as zip2

# Elements of one decoder layer of the Llama-3-8B shape: the bucket that its all-gather moves (218 112 000).
LAYER_8B = 218_112_000

# shape -> (fewest layers, most layers, most tokens) of a drawn step
STEP_SHAPES = {
    "tiny": (2, 4, 4096), "small": (2, 4, 4096), "gpt2-xl": (2, 6, 4096), "llama3-8b": (1, 2, 4096),
    "llama2-13b": (1, 2, 4096), "34b": (1, 1, 4096),
}


def _step(model, layers, batch, seq, act_ckpt=False, master="bf16", **name):
    return {**name, "kind": "step", "model": model, "layers": layers, "batch": batch, "seq": seq,
            "act_ckpt": act_ckpt, "master": master}


def listed() -> list:
    return [
        # the plumbing configuration (d_model 256, batch 4 x 128): the smallest step, where launches and host work count
        _step("tiny", 2, 4, 128, name="step tiny 4x128"),
        # a small model at an ordinary length: fine-tuning, debugging, hyper-parameter search
        _step("small", 4, 1, 1024, name="step small 1x1024"),
        # the shipped run: GPT-2-XL, batch 2 x 1024 (LayerNorm, biases, head size 64, ragged vocabulary, tied embedding)
        _step("gpt2-xl", 4, 2, 1024, name="step gpt2-xl 4L 2x1024"),
        # the headline run: Llama-3-8B at 4096 tokens
        _step("llama3-8b", 2, 1, 4096, name="step llama3-8b 2L 1x4096"),
        # the largest shape, which is trained with activation checkpointing
        _step("34b", 1, 1, 4096, act_ckpt=True, name="step 34b 1L 1x4096 ckpt"),
        # long-context training of the 8B shape: attention is most of such a step
        {"name": "attention 1x16384 gqa", "kind": "attention", "batch": 1, "seq": 16384, "q_heads": 32, "kv_heads": 8, "dim": 128},
        # many short sequences, GPT-2-XL heads
        {"name": "attention 8x1024 d64", "kind": "attention", "batch": 8, "seq": 1024, "q_heads": 25, "kv_heads": 25, "dim": 64},
        # a rank's shard of an 8B layer on eight ranks, with the base exponent refreshed from its statistics
        {"name": "v1 encode 27M", "kind": "v1_encode", "numel": LAYER_8B // 8, "works": 1, "data": "params", "refresh": True},
        # the whole layer from eight ranks' streams
        {"name": "v1 decode 8x27M", "kind": "v1_decode", "numel": LAYER_8B // 8, "works": 8, "data": "params"},
        # gradients of two layers-worth of a reduce-scatter bucket, smallest wire
        {"name": "v2 encode 2^27 planes", "kind": "v2_encode", "numel": 1 << 27, "data": "grads", "nibble": False},
        # a small ragged tensor in the default records: latency
        {"name": "v2 decode 1M nibble", "kind": "v2_decode", "numel": 1_000_003, "data": "params", "nibble": True},
        # int8 all-gather of a shard of the 8B layer, eight ranks' contributions dequantised
        {"name": "int8 8x27M", "kind": "int8", "numel": LAYER_8B // 8, "ranks": 8, "dtype": "bf16"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["step"] * 5 + ["attention"] * 2 + ["v1_encode", "v1_decode", "v2_encode", "v2_decode", "int8"])
    if kind == "step":
        model = rng.choice(sorted(STEP_SHAPES))
        lo, hi, most = STEP_SHAPES[model]
        batch = rng.choice([1, 2, 4])
        tokens = _log_int(rng, 256, most)
        seq = min(tokens // batch, get_config(model).max_seq)
        if rng.random() < 0.5:  # packed to a round length, or whatever the longest text of the batch has
            seq = max(64, seq // 64 * 64)
        act_ckpt = model == "34b" or rng.random() < 0.2
        return _step(model, rng.randint(lo, hi), batch, seq, act_ckpt=act_ckpt,
                     master="fp32" if model in ("tiny", "small") and rng.random() < 0.25 else "bf16")
    if kind == "attention":
        dim = rng.choice([64, 128])
        kv, group = (rng.choice([(25, 1), (8, 1)]) if dim == 64 else rng.choice([(8, 4), (8, 8), (40, 1), (2, 4)]))
        seq = _log_int(rng, 256, 16384)
        if rng.random() < 0.5:
            seq = max(256, seq // 128 * 128)
        q = kv * group
        # no more work than the longest listed case, no more tokens than 32768
        most = min(8, 32768 // seq, int(32 * 128 * 16384 ** 2 / (q * dim * seq ** 2)))
        if most < 1:
            seq = int(16384 * math.sqrt(32 * 128 / (q * dim))) - rng.randint(0, 200)
            most = 1
        return {"kind": "attention", "batch": rng.randint(1, most), "seq": seq, "q_heads": q, "kv_heads": kv, "dim": dim}
    data = rng.choice(["params", "grads"])
    if kind in ("v1_encode", "v1_decode"):
        works = rng.choice([1, 2, 4, 8])
        n = _log_int(rng, 20_000, LAYER_8B // works)
        if rng.random() < 0.5:
            n = max(4096, n // 4096 * 4096)
        case = {"kind": kind, "numel": n, "works": works, "data": data}
        if kind == "v1_encode":
            case["refresh"] = rng.random() < 0.5
        return case
    if kind == "int8":
        ranks = rng.choice([2, 4, 8])
        return {"kind": "int8", "numel": _log_int(rng, 50_000, LAYER_8B // ranks), "ranks": ranks,
                "dtype": rng.choice(["bf16", "bf16", "fp32"])}
    n = _log_int(rng, 50_000, 1 << 28)
    if rng.random() < 0.5:
        n = max(1024, n // 1024 * 1024)
    return {"kind": kind, "numel": n, "data": data, "nibble": rng.random() < 0.5}


# --------------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------------

def _device() -> torch.device:
    """``cuda:0`` with the one-rank process group that a training program starts with."""
    if not torch.distributed.is_initialized():
        if "MASTER_PORT" not in os.environ:
            with socket.socket() as s:
                s.bind(("127.0.0.1", 0))
                os.environ["MASTER_PORT"] = str(s.getsockname()[1])
        os.environ["MASTER_ADDR"] = "127.0.0.1"
        init_distributed("cuda")
    return torch.device("cuda:0")


def _values(n: int, data: str, gen, device) -> torch.Tensor:
    """Parameter-like N(0, 0.02), or gradient-like N(0, 1e-3) with 1 % of the entries a hundred times larger."""
    x = torch.empty(n, dtype=torch.bfloat16, device=device)
    step = 1 << 25
    for lo in range(0, n, step):
        m = min(step, n - lo)
        v = torch.randn(m, generator=gen, device=device)
        if data == "params":
            v.mul_(0.02)
        else:
            v.mul_(1e-3)
            v = torch.where(torch.rand(m, generator=gen, device=device) < 0.01, v * 100.0, v)
        x[lo:lo + m] = v
    return x


def _zeros(n: int, dtype, device) -> torch.Tensor:
    return torch.zeros(n, dtype=dtype, device=device)


def _v1_state(case, gen, dev) -> dict:
    """Buffers of an encode of ``works`` dense segments of ``numel`` elements each, padded to whole codec blocks."""
    n, works = case["numel"], case["works"]
    padded = codec.pad_to_block(n)
    st = {
        "x": _values(n * works, case["data"], gen, dev), "n": n, "works": works, "padded": padded,
        "n_8": torch.full((works,), padded, dtype=torch.int32, device=dev),
        "orig": torch.full((works,), n, dtype=torch.int32, device=dev),
        "bases": torch.full((256,), 122, dtype=torch.int32, device=dev),
        "det": _zeros(works * codec.v1_det_bytes(padded), torch.uint8, dev),
        "scratch": _zeros(works * padded, torch.uint8, dev),
        "esc": _zeros(works * codec.align128(padded), torch.uint8, dev),
        "counts": _zeros(works, torch.int32, dev),
    }
    codec.v1_base_from_std(st["x"], st["bases"])
    return st


def _v1_encode(st) -> None:
    if st["works"] == 1:
        zip2.compress_split_store(st["x"], st["n_8"], st["bases"], st["det"], st["scratch"], st["esc"], st["counts"], 1)
    else:
        zip2.compress_split_store_pad(st["x"], st["n_8"], st["orig"], st["bases"], st["det"], st["scratch"], st["esc"],
                                      st["counts"], st["padded"] * st["works"], st["works"])


def prepare(case: dict, seed: int) -> dict:
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "step":
        cfg = dataclasses.replace(get_config(case["model"]), n_layers=case["layers"])
        st["engine"] = TrainEngine(EngineConfig(
            model=cfg, seed=seed, act_ckpt=case["act_ckpt"],
            master_dtype=torch.float32 if case["master"] == "fp32" else torch.bfloat16), dev)
        host = torch.Generator().manual_seed(seed)
        st["ids"] = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), generator=host).pin_memory()
    elif kind == "attention":
        hq, hkv, d = case["q_heads"], case["kv_heads"], case["dim"]
        shape = (case["batch"], case["seq"])
        st.update(hq=hq, hkv=hkv)
        st["qkv"] = torch.randn(*shape, hq + 2 * hkv, d, generator=gen, device=dev, dtype=torch.bfloat16).requires_grad_()
        st["do"] = torch.randn(*shape, hq, d, generator=gen, device=dev, dtype=torch.bfloat16)
    elif kind == "v1_encode":
        st.update(_v1_state(case, gen, dev), refresh=case["refresh"])
    elif kind == "v1_decode":
        enc = _v1_state(case, gen, dev)
        _v1_encode(enc)
        # the outlier streams arrive padded to the longest of them, as the ranks gather them
        counts = enc["counts"].tolist()
        stride = codec.align128(max(counts))
        esc = _zeros(max(stride, 128) * enc["works"], torch.uint8, dev)
        at = 0
        for i, c in enumerate(counts):
            esc[i * stride:i * stride + c] = enc["esc"][at:at + c]
            at += codec.align128(c)
        st.update(det=enc["det"], esc=esc, n_8=enc["n_8"], n=enc["n"], works=enc["works"],
                  nbytes=torch.full((enc["works"],), stride, dtype=torch.int32, device=dev),
                  out=_zeros(enc["n"] * enc["works"], torch.bfloat16, dev))
    elif kind in ("v2_encode", "v2_decode"):
        n = case["numel"]
        nc = codec.v2_num_chunks(n)
        st.update(n=n, nibble=case["nibble"], x=_values(n, case["data"], gen, dev),
                  rec=_zeros(nc * codec.V2_SLOT, torch.uint8, dev), hdr=_zeros(nc, torch.int32, dev))
        if kind == "v2_decode":
            codec.v2_encode(st.pop("x"), st["rec"], st["hdr"], nibble=st["nibble"])
            st["out"] = _zeros(n, torch.bfloat16, dev)
    elif kind == "int8":
        n, ranks = case["numel"], case["ranks"]
        dt = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
        st.update(n=n, x=_values(n, "params", gen, dev).to(dt),
                  gathered=_zeros(ranks * quant.packed_bytes(n), torch.uint8, dev).view(ranks, -1),
                  out=_zeros(n * ranks, dt, dev))
        for r in range(1, ranks):  # what the other ranks sent
            quant.quantize_pack(_values(n, "params", gen, dev).to(dt), st["gathered"][r])
    else:
        raise ValueError(kind)
    return st


# --------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------

def run(st: dict):
    kind = st["kind"]
    if kind == "step":
        eng = st["engine"]
        loss = eng.step(st["ids"])
        moments = eng.optimizer.state[eng.flat.master_param]
        return {"loss": loss, "params": eng.flat.master, "grads": eng.flat.grad_master,
                "exp_avg": moments["exp_avg"], "exp_avg_sq": moments["exp_avg_sq"]}
    if kind == "attention":
        o = attention.causal_attention(st["qkv"], st["hq"], st["hkv"])
        (dqkv,) = torch.autograd.grad(o, st["qkv"], st["do"])
        return {"o": o.detach(), "dqkv": dqkv}
    if kind == "v1_encode":
        if st["refresh"]:
            codec.v1_base_from_std(st["x"], st["bases"])
        _v1_encode(st)
        return {"det": st["det"], "esc": st["esc"], "counts": st["counts"], "base": st["bases"]}
    if kind == "v1_decode":
        zip2.decompress_split_store_unpad(st["det"], st["esc"], st["n_8"], st["nbytes"], st["out"], st["n"], st["works"])
        return st["out"].view(torch.int16)
    if kind == "v2_encode":
        rec, hdr = codec.v2_encode(st["x"], st["rec"], st["hdr"], nibble=st["nibble"])
        return {"records": rec, "headers": hdr}
    if kind == "v2_decode":
        return codec.v2_decode(st["rec"], st["hdr"], st["n"], st["out"], nibble=st["nibble"]).view(torch.int16)
    quant.quantize_pack(st["x"], st["gathered"][0])
    quant.dequantize_unpack(st["gathered"], st["n"], st["out"])
    return {"packed": st["gathered"], "out": st["out"]}


# --------------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------------

def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "step":
        cfg = dataclasses.replace(get_config(case["model"]), n_layers=case["layers"])
        tokens = case["batch"] * case["seq"]
        # matrices take part in three products of 2 x tokens x elements each; embedding rows are looked up
        lookups = cfg.vocab_size * cfg.d_model if not cfg.tie_embeddings else 0
        if cfg.family == "gpt2":
            lookups += cfg.max_seq * cfg.d_model
        n = cfg.num_params()
        att = 7 * case["batch"] * cfg.n_layers * cfg.n_heads * cfg.head_dim * case["seq"] ** 2
        size = 4 if case["master"] == "fp32" else 2
        # parameters and both moments read and written, gradients written
        return {"bytes": n * (6 * size + 2) + tokens * 8, "flops": 6 * (n - lookups) * tokens + att}
    if kind == "attention":
        b, s, hq, hkv, d = (case[k] for k in ("batch", "seq", "q_heads", "kv_heads", "dim"))
        # qkv and do in, o and dqkv out; half of the scores are masked: 2 products forward, 5 backward
        return {"bytes": b * s * d * 2 * (2 * (hq + 2 * hkv) + 2 * hq), "flops": 7 * b * hq * d * s * s}
    n = case["numel"]
    # bytes per element of the coded form (measured on these distributions)
    if kind in ("v1_encode", "v1_decode"):
        coded = 1.40 if case["data"] == "params" else 1.57
        return {"bytes": n * case["works"] * (2 + coded), "flops": 0}
    if kind in ("v2_encode", "v2_decode"):
        coded = 1.50 if case["nibble"] else (1.40 if case["data"] == "params" else 1.41)
        return {"bytes": n * (2 + coded), "flops": 0}
    size = 4 if case["dtype"] == "fp32" else 2
    return {"bytes": n * (size + 1) + n * case["ranks"] * (1 + size), "flops": 0}


def tolerance(case: dict):
    kind = case["kind"]
    if kind == "step":
        # bf16 activations and gradients through a chain of products; the squared gradient doubles the relative error
        return {"rel": 2e-2}
    if kind == "attention":
        return {"rel": 1e-2}
    return "exact"
