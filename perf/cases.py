"""What a server built on this package has it do, as cases that can be timed and compared.

A decode step walks the model's MoE layers with the tokens of its concurrent slots; a prefill call pushes a prompt chunk through
one layer; a drop-in caller of the operator entries runs them one by one.  Layer shapes, weight types and routing variants are the
package's own configurations, weights and inputs are drawn as those configurations draw them.  A decode case walks several layers,
as a model does, so that the weights of a call come from device memory and not from what the call before left in the L2.

A case: config (a configuration's name), entry (how the layers are called), tokens, layers.
  decode     forward_moe on device tensors, call by call
  graph      the same calls captured once in a CUDA graph and replayed, as bench.py measures them
  host       forward_moe_host: pinned host rows in and out, every call waited for
  half       forward_moe_residual_norm: residual add + RMSNorm + layer; from PREFILL_FROM tokens on with the prefill weights
  prefill    forward_moe_prefill
  operators  the operator entries of the reference's interface on raw ggml blocks, one token at a time
"""
import math

import numpy as np
import torch

from chimere_b200 import abi, configs, formats
from chimere_b200.layer import (MoeScratch, MoeWeightsPrefill, MoeWeightsTiled, forward_moe, forward_moe_host, forward_moe_prefill,
                                forward_moe_residual_norm)

CONFIGS = {c.name: c for c in configs.CONFIGS + [configs.QWEN_IQ3S_Q5K]}
PREFILL_FROM = 65      # a server's slots are decoded together up to 64 tokens; longer batches are prompt chunks
MAX_PREFILL = 8192     # the largest chunk of the prefill configuration; the wider Nemotron-H-style layer does as much at a quarter of it


def _case(name, config, entry, tokens, layers):
    return {"name": name, "config": config.name, "entry": entry, "tokens": tokens, "layers": layers}


def listed():
    return [
        # the drop-in operator interface, one token of the production mix: quantise, batched expert products, the shared expert's GEMVs
        _case("operators-1", configs.QWEN_IQ3S_Q5K, "operators", 1, 4),
        # one user's token through four layers: latency of the smallest call
        _case("decode-1", configs.QWEN_IQ3S, "decode", 1, 4),
        # the production mix (Q5_K shared expert) the way the model's forward calls it, two slots
        _case("half-2", configs.QWEN_IQ3S_Q5K, "half", 2, 4),
        # the Nemotron-H-style layer at one token: fewer, wider experts, no gate matrix
        _case("decode-1-nemotron", configs.NEMOTRON_Q4_0, "decode", 1, 4),
        # five slots through the host-buffer entry
        _case("host-5", configs.QWEN_IQ3S, "host", 5, 4),
        # eight slots, replayed from a graph: the headline workload of bench.py
        _case("graph-8", configs.QWEN_IQ3S, "graph", 8, 4),
        # the CPU-runnable configuration's batch
        _case("decode-16", configs.QWEN_Q4_0, "decode", 16, 2),
        # an almost full set of slots with skewed routing: popular experts hold dozens of tokens, the tail one or two
        _case("decode-61-zipf", configs.QWEN_Q4_0_ZIPF, "decode", 61, 2),
        # the Nemotron-H-style layer's prompt chunk: every expert touched, about twelve tokens each
        _case("prefill-256-nemotron", configs.NEMOTRON_Q4_0, "prefill", 256, 1),
        # a ragged prompt of the production mix, called as the model's forward calls it
        _case("half-777", configs.QWEN_IQ3S_Q5K, "half", 777, 1),
        # the prefill configuration: Q8_0 experts, skewed routing, a short prompt chunk and the largest one
        _case("prefill-512-zipf", configs.QWEN_Q8_0, "prefill", 512, 1),
        _case("prefill-8192-zipf", configs.QWEN_Q8_0, "prefill", 8192, 1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["operators", "decode", "decode", "half", "host", "graph", "prefill", "prefill", "half-prefill"])
    config = CONFIGS[rng.choice(sorted(CONFIGS))]
    if entry == "operators":
        return {"config": config.name, "entry": entry, "tokens": rng.randint(1, 4), "layers": rng.randint(1, 4)}
    if entry in ("prefill", "half-prefill"):
        most = MAX_PREFILL if config is not configs.NEMOTRON_Q4_0 else MAX_PREFILL // 4
        return {"config": config.name, "entry": entry.split("-")[0], "tokens": _log_int(rng, PREFILL_FROM, most), "layers": 1}
    return {"config": config.name, "entry": entry, "tokens": _log_int(rng, 1, PREFILL_FROM - 1), "layers": rng.randint(2, 4)}


def _is_prefill(case):
    return case["entry"] == "prefill" or (case["entry"] == "half" and case["tokens"] >= PREFILL_FROM)


def _rows(T, H, gen):
    return torch.randn(T, H, generator=gen, device="cuda", dtype=torch.float32)


def prepare(case, seed):
    cfg, T, L, entry = CONFIGS[case["config"]], case["tokens"], case["layers"], case["entry"]
    gen = torch.Generator(device="cuda").manual_seed(7919 * seed + T)
    if entry == "operators":
        return {"entry": entry, "layers": [_operator_layer(cfg, T, seed * L + i, gen) for i in range(L)]}
    weights, prefill = [], []
    for i in range(L):
        raw = configs.make_layer(cfg, device="cuda", seed=seed * L + i)
        weights.append(MoeWeightsTiled(raw, keep_raw=False))
        prefill.append(MoeWeightsPrefill(raw) if _is_prefill(case) else None)
        del raw
    scratch = MoeScratch(weights[0], T)     # one workspace per stream, shared by the layers of the walk
    if _is_prefill(case):
        scratch.enable_prefill()
    s = {"entry": entry, "weights": weights, "prefill": prefill, "scratch": scratch,
         "x": [_rows(T, cfg.H, gen) for _ in range(L)], "y": [torch.empty(T, cfg.H, device="cuda") for _ in range(L)]}
    if entry == "half":
        s["residual"] = [_rows(T, cfg.H, gen) for _ in range(L)]
        s["norm"] = [1.0 + 0.1 * torch.randn(cfg.H, generator=gen, device="cuda") for _ in range(L)]
    elif entry == "host":
        s["x"] = [x.cpu().pin_memory() for x in s["x"]]
        s["y"] = [torch.empty(T, cfg.H).pin_memory() for _ in range(L)]
    elif entry == "graph":
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            _decode(s)                      # (kernel attributes are set on the first call, outside the capture)
            stream.synchronize()
            with torch.cuda.graph(s["graph"], stream=stream):
                _decode(s)
        torch.cuda.current_stream().wait_stream(stream)
    return s


def _decode(s):
    for w, x, y in zip(s["weights"], s["x"], s["y"]):
        forward_moe(w, s["scratch"], x, y)
    return s["y"]


def run(s):
    entry = s["entry"]
    if entry == "decode":
        return _decode(s)
    if entry == "graph":
        s["graph"].replay()
        return s["y"]
    if entry == "host":
        for w, x, y in zip(s["weights"], s["x"], s["y"]):
            forward_moe_host(w, s["scratch"], x, y)
        return s["y"]
    if entry == "prefill":
        for w, pw, x, y in zip(s["weights"], s["prefill"], s["x"], s["y"]):
            forward_moe_prefill(w, pw, s["scratch"], x, y)
        return s["y"]
    if entry == "half":
        for w, pw, x, r, n, y in zip(s["weights"], s["prefill"], s["x"], s["residual"], s["norm"], s["y"]):
            forward_moe_residual_norm(w, s["scratch"], x, r, n, 1e-6, y, pw)
        return {"y": s["y"], "residual": s["residual"]}
    return [out for layer in s["layers"] for out in _run_operators(layer)]


# ---- the operator entries: per token quantise, expert products by id, the shared expert's GEMVs (the activations between are the caller's) ----
_BATCHED = {formats.TYPE_IQ3_S: "chimere_mmvq_iq3s_batched", formats.TYPE_Q4_0: "chimere_mmvq_q4_0_batched", formats.TYPE_Q8_0: "chimere_mmvq_q8_0_batched"}
_SINGLE = {formats.TYPE_IQ3_S: "chimere_mmvq_iq3s", formats.TYPE_Q4_0: "chimere_mmvq_q4_0", formats.TYPE_Q8_0: "chimere_mmvq_q8_0",
           formats.TYPE_Q5_K: "chimere_mmvq_q5k"}


def _pad512(n):
    return (n + 511) // 512 * 512           # quantised rows are padded to 512 values, as the reference's buffers are


def _q8_1_bytes(n):
    return _pad512(n) // 32 * formats.Q8_1_BYTES


def _operator_layer(cfg, T, seed, gen):
    raw = configs.make_layer(cfg, device="cuda", seed=seed)
    k, H, F, Fs = cfg.top_k, cfg.H, cfg.F, cfg.F_s
    u8 = lambda *shape: torch.empty(*shape, dtype=torch.uint8, device="cuda")      # noqa: E731
    f32 = lambda *shape: torch.empty(*shape, device="cuda")                        # noqa: E731
    return {"raw": raw, "T": T, "k": k, "H": H, "F": F, "Fs": Fs,
            "x": _rows(T, H, gen), "inter": _rows(T * k, F, gen).reshape(T, k, F), "inter_sh": _rows(T, Fs, gen),
            "ids": torch.stack([torch.randperm(cfg.E, generator=gen, device="cuda")[:k] for _ in range(T)]).to(torch.int32).contiguous(),
            "x_q8": u8(T, _q8_1_bytes(H)), "inter_q8": u8(T, k, _q8_1_bytes(F)), "inter_sh_q8": u8(T, _q8_1_bytes(Fs)),
            "gate": f32(T, k, F), "up": f32(T, k, F), "down": f32(T, k, H), "gate_sh": f32(T, Fs), "up_sh": f32(T, Fs), "down_sh": f32(T, H)}


def _run_operators(l):
    lib, raw, st = abi.load(), l["raw"], torch.cuda.current_stream().cuda_stream
    k, H, F, Fs = l["k"], l["H"], l["F"], l["Fs"]
    gate_up, down = getattr(lib, _BATCHED[raw.type_up]), getattr(lib, _BATCHED[raw.type_down])
    sh_gate_up, sh_down = getattr(lib, _SINGLE[raw.type_sh_up]), getattr(lib, _SINGLE[raw.type_sh_down])
    nb = lambda n: _pad512(n) // 32                                                # noqa: E731
    for t in range(l["T"]):
        xq, ids = l["x_q8"][t].data_ptr(), l["ids"][t].data_ptr()
        lib.chimere_quantize_q8_1(l["x"][t].data_ptr(), xq, H, _pad512(H), st)
        if raw.gate_exps_raw is not None:
            gate_up(raw.gate_exps_raw.data_ptr(), xq, l["gate"][t].data_ptr(), ids, H, F, nb(H), raw.expert_bytes_gate, 0, k, st)
        gate_up(raw.up_exps_raw.data_ptr(), xq, l["up"][t].data_ptr(), ids, H, F, nb(H), raw.expert_bytes_up, 0, k, st)
        iq = l["inter_q8"][t]
        lib.chimere_quantize_q8_1_batched(l["inter"][t].data_ptr(), iq.data_ptr(), F, _pad512(F), k, st)
        down(raw.down_exps_raw.data_ptr(), iq.data_ptr(), l["down"][t].data_ptr(), ids, F, H, nb(F), raw.expert_bytes_down, _q8_1_bytes(F), k, st)
        if raw.shexp_gate_raw is not None:
            sh_gate_up(raw.shexp_gate_raw.data_ptr(), xq, l["gate_sh"][t].data_ptr(), H, Fs, nb(H), st)
        sh_gate_up(raw.shexp_up_raw.data_ptr(), xq, l["up_sh"][t].data_ptr(), H, Fs, nb(H), st)
        sq = l["inter_sh_q8"][t].data_ptr()
        lib.chimere_quantize_q8_1(l["inter_sh"][t].data_ptr(), sq, Fs, _pad512(Fs), st)
        sh_down(raw.shexp_down_raw.data_ptr(), sq, l["down_sh"][t].data_ptr(), Fs, H, nb(Fs), st)
    written = ["x_q8", "inter_q8", "inter_sh_q8", "up", "down", "up_sh", "down_sh"] + (["gate", "gate_sh"] if raw.gate_exps_raw is not None else [])
    return [l[n] for n in written]


# ---- what a pass cannot do without ----
def _distinct_experts(cfg, T):
    """Experts that T tokens select: logits of inputs ~N(0, 1) and router rows ~N(0, 0.02) are ~N(0, 0.0004 H), plus the configuration's bias."""
    rng = np.random.default_rng(1)
    z = rng.standard_normal((T, cfg.E), dtype=np.float32) * (0.02 * math.sqrt(cfg.H))
    if cfg.zipf_bias:
        z -= 2.2 * np.log(np.arange(1, cfg.E + 1, dtype=np.float32))
    return int(np.unique(np.argpartition(z, cfg.E - cfg.top_k, axis=1)[:, cfg.E - cfg.top_k:]).size)


def work(case):
    cfg, T, L, entry = CONFIGS[case["config"]], case["tokens"], case["layers"], case["entry"]
    if entry == "operators":
        n_gu = 2 if cfg.act == abi.ACT_SWIGLU else 1
        sh_gu, sh_dn = cfg.type_sh_gate_up or cfg.type_gate_up, cfg.type_sh_down or cfg.type_down
        weights = cfg.top_k * (n_gu * cfg.F * formats.row_bytes(cfg.type_gate_up, cfg.H) + cfg.H * formats.row_bytes(cfg.type_down, cfg.F))
        weights += n_gu * cfg.F_s * formats.row_bytes(sh_gu, cfg.H) + cfg.H * formats.row_bytes(sh_dn, cfg.F_s)
        rows_in = cfg.H + cfg.top_k * cfg.F + cfg.F_s
        rows_out = n_gu * (cfg.top_k * cfg.F + cfg.F_s) + (cfg.top_k + 1) * cfg.H
        q8 = _q8_1_bytes(cfg.H) + cfg.top_k * _q8_1_bytes(cfg.F) + _q8_1_bytes(cfg.F_s)
        return {"bytes": L * T * (weights + 4 * (rows_in + rows_out) + q8), "flops": L * configs.int8_ops(cfg, T)}
    extra = (12 * T + 4) * cfg.H if entry == "half" else 0      # (hidden takes the place of x; residual read and written, the norm's weight)
    return {"bytes": L * (configs.algorithmic_bytes(cfg, T, _distinct_experts(cfg, T)) + extra), "flops": L * configs.int8_ops(cfg, T)}


def tolerance(case):
    if case["entry"] == "operators":
        return {"rel": 1e-5, "max": 2e-4}   # fp32 sums of exact integer block dots; the quantised bytes are the same
    # fp32 sums again, but the intermediates between the two products are rounded to 8 bits: another order of additions moves a few of
    # them by one step
    return {"rel": 1e-3, "max": 2e-2}
