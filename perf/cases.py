"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values; ``kind`` says which public entry points one pass goes through:

  gemv      f32 activations -> Q8_1 -> Q4_K projection                        (bkQuantQ8_1 + bkGemvQ4K)
  gdn       conv1d + gated-DeltaNet step(s), recurrent state updated in place   (bkGdnStep)
  attn      decode attention over a filled KV cache                             (bkAttnDecode)
  quantize  bf16 / f32 checkpoint rows -> Q4_K rows, the loader's inner step    (bkQuantizeQ4K)
  generate  one request batch: reset, prompt, greedy tokens fed back on the GPU (DecodeModel.prefill + run)
  loop      the same, every token through the host                              (runGraphDecode)
  chat      prompt, then sampled tokens, each read by the host and fed back     (DecodeModel.prefill + step, bkSample)

Shapes are those of the two benchmark models, of the small test model, or log-uniform over the ranges between
them.  Weights, activations and state are random with the distributions of ``bunker_b200.synth``, drawn on the GPU.
"""
import math
import random

import numpy as np
import torch

from bunker_b200 import model as M
from bunker_b200 import ops
from bunker_b200 import runtime as R

CONFIGS = {"tiny": M.CONFIG_TINY, "24l": M.CONFIG_HYBRID_24L, "64l": M.CONFIG_HYBRID_64L}


def listed():
    return [
        # the smallest library call in the hot path: one projection of one token, launch latency included
        {"name": "gemv_4096_b1", "kind": "gemv", "N": 4096, "K": 4096, "B": 1},
        # the recurrent layer of eight sequences on its own (16 key / 32 value heads): state traffic
        {"name": "gdn_b8", "kind": "gdn", "B": 8, "Hk": 16, "Hv": 32, "T": 1},
        # long-context attention, the largest cache of the benchmark set, eight sequences
        {"name": "attn_b8_32768", "kind": "attn", "B": 8, "L": 32768, "Hq": 16, "Hkv": 2},
        # loading a checkpoint: one gate or up matrix of the 64-layer model, bf16
        {"name": "quantize_17408x5120", "kind": "quantize", "rows": 17408, "K": 5120, "bf16": True},
        # the small model driven token by token by the host: launches and host work only
        {"name": "loop_tiny_b1", "kind": "loop", "config": "tiny", "batch": 1, "prompt": 9, "new": 24},
        # interactive use: a short odd prompt, sampled tokens that the host sees one by one
        {"name": "chat_24l_b1", "kind": "chat", "config": "24l", "batch": 1, "prompt": 17, "new": 48, "top_k": 40, "top_p": 0.9,
         "temperature": 0.7},
        # the benchmark workload, one sequence and eight
        {"name": "generate_24l_b1", "kind": "generate", "config": "24l", "batch": 1, "prompt": 32, "new": 256},
        {"name": "generate_24l_b8", "kind": "generate", "config": "24l", "batch": 8, "prompt": 32, "new": 256},
        # a full server batch, and one that fills no power of two
        {"name": "generate_24l_b32", "kind": "generate", "config": "24l", "batch": 32, "prompt": 32, "new": 64},
        {"name": "generate_24l_b13", "kind": "generate", "config": "24l", "batch": 13, "prompt": 21, "new": 50},
        # reading a long prompt (summarising, retrieval): prefill is the work, one token comes out
        {"name": "prefill_24l_1000", "kind": "generate", "config": "24l", "batch": 1, "prompt": 1000, "new": 1},
        # the large model, one sequence
        {"name": "generate_64l_b1", "kind": "generate", "config": "64l", "batch": 1, "prompt": 64, "new": 32},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["gemv", "gemv", "gdn", "attn", "quantize", "loop", "chat", "generate", "generate", "generate", "generate"])
    if kind == "gemv":
        return {"kind": kind, "N": _log(rng, 32, 40000), "K": 256 * _log(rng, 1, 68), "B": _log(rng, 1, 64)}
    if kind == "gdn":
        hk, hv = rng.choice([(16, 32), (16, 48), (2, 4), (8, 8)])
        b = _log(rng, 1, 32)
        return {"kind": kind, "B": b, "Hk": hk, "Hv": hv, "T": _log(rng, 1, 64 // b)}
    if kind == "attn":
        hq, hkv = rng.choice([(16, 2), (24, 4), (4, 1)])
        return {"kind": kind, "B": _log(rng, 1, 8), "L": _log(rng, 64, 32768), "Hq": hq, "Hkv": hkv}
    if kind == "quantize":
        return {"kind": kind, "rows": _log(rng, 32, 17408), "K": 256 * _log(rng, 1, 20), "bf16": rng.random() < 0.7}
    if kind == "loop":
        return {"kind": kind, "config": rng.choice(["tiny", "24l"]), "batch": _log(rng, 1, 8), "prompt": _log(rng, 1, 20), "new": _log(rng, 4, 64)}
    if kind == "chat":
        return {"kind": kind, "config": "24l", "batch": _log(rng, 1, 16), "prompt": _log(rng, 4, 200), "new": _log(rng, 8, 48),
                "top_k": rng.randint(1, 64), "top_p": round(rng.uniform(0.5, 1.0), 2), "temperature": round(rng.uniform(0.3, 1.3), 2)}
    config = rng.choice(["tiny", "24l", "24l", "24l", "64l"])
    if config == "64l":
        return {"kind": kind, "config": config, "batch": _log(rng, 1, 8), "prompt": _log(rng, 1, 64), "new": _log(rng, 2, 24)}
    batch = _log(rng, 1, 64)
    return {"kind": kind, "config": config, "batch": batch, "prompt": _log(rng, 1, max(2, 1200 // batch)), "new": _log(rng, 1, 200 if batch <= 8 else 48)}


# ---- inputs ------------------------------------------------------------------------

def _gen(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + stream) & 0x7FFFFFFF)
    return g


def _bytes(n, g):
    return torch.randint(-2**31, 2**31, ((n + 3) // 4,), dtype=torch.int32, device="cuda", generator=g).view(torch.uint8)[:n]


def _q4k(buf, N, K, g):
    """Random Q4_K rows in place: every byte uniform, then f16 d and dmin = |N(0, 1e-3)|."""
    w = buf[:N * (K // 256) * 144].view(N * (K // 256), 144)
    d = (torch.randn((w.shape[0], 2), device="cuda", generator=g) * 1e-3).abs().half()
    w[:, :4] = d.view(torch.uint8)
    return buf


def _bf16(shape, g, std=1.0):
    return (torch.randn(shape, device="cuda", generator=g) * std).bfloat16()


def _f32(shape, g, std=1.0, mean=0.0):
    return torch.randn(shape, device="cuda", generator=g) * std + mean


class _Slab:
    """Device memory that holds a model's weights (what the loader's DeviceBuffer is to DecodeModel.from_device)."""

    def __init__(self, nbytes, g):
        self.t = _bytes(nbytes, g)
        self.ptr = self.t.data_ptr()

    def free(self):
        self.t = None


class _Loaded:
    """Owns a model; it is destroyed when neither the request state nor an output tensor refers to it any more."""

    def __init__(self, gm):
        self.gm = gm

    def __del__(self):
        self.gm.destroy()


class _Device:
    """A library-owned device buffer as something torch can read without a copy; keeps its owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False), "version": 3}


class _Served:
    """A loaded model and the request it gets."""

    def __init__(self, case, seed):
        self.case = dict(case)
        g = _gen(seed, 1)
        B, T, G = case["batch"], case["prompt"], case["new"]
        self.cfg = cfg = CONFIGS[case["config"]].with_(max_len=(T + G + 63) // 64 * 64)
        specs, offs, total = M.tensor_specs(cfg), {}, 0
        size = {"q4k": lambda s: s[0] * s[1] // 256 * 144, "bf16": lambda s: 2 * math.prod(s), "f32": lambda s: 4 * math.prod(s)}
        for name, kind, shape in specs:
            offs[name] = (total, size[kind](shape))
            total += (offs[name][1] + 255) // 256 * 256
        slab = _Slab(total, g)
        for name, kind, shape in specs:
            at, n = offs[name]
            t = slab.t[at:at + n]
            if kind == "q4k":
                _q4k(t, shape[0], shape[1], g)
            elif name.endswith("A_log"):
                t.view(torch.float32)[:] = torch.rand(shape, device="cuda", generator=g) * 2.0 - 2.0
            elif kind == "f32":
                t.view(torch.float32)[:] = _f32(shape, g, 0.02, 1.0)
            else:
                std = 1.0 if name.endswith("dt_bias") else 0.3 if name.endswith("conv1d.weight") else 0.02
                t.view(torch.bfloat16)[:] = _bf16(shape, g, std).view(-1)
        self.prompt = torch.randint(0, cfg.vocab, (T, B), dtype=torch.int32, device="cuda", generator=g).cpu().numpy()
        torch.cuda.synchronize()
        self.gm = gm = M.DecodeModel.from_device(cfg, {n: (slab.ptr + at, nb) for n, (at, nb) in offs.items()}, slab, batch=B)
        self.loaded = _Loaded(gm)
        self.logits = torch.as_tensor(_Device(self.loaded, gm.buffer("logits"), (B, cfg.vocab), "<f4"), device="cuda")
        self.idx = torch.zeros(B, dtype=torch.int32, device="cuda")
        self.host_idx = np.zeros(B, np.int32)
        torch.cuda.synchronize()


def prepare(case, seed):
    R.cu(0)
    kind = case["kind"]
    if kind in ("generate", "loop", "chat"):
        return _Served(case, seed)
    g = _gen(seed, 2)
    s = {"case": dict(case)}
    if kind == "gemv":
        N, K, B = case["N"], case["K"], case["B"]
        s["W"] = _q4k(_bytes(N * (K // 256) * 144, g), N, K, g)
        s["x"] = _f32((B, K), g)
        s["xq"] = torch.zeros((B, K // 32, 36), dtype=torch.uint8, device="cuda")
        s["y"] = torch.zeros((B, N), device="cuda")
    elif kind == "gdn":
        B, Hk, Hv, T = case["B"], case["Hk"], case["Hv"], case["T"]
        C = (2 * Hk + Hv) * 128
        s.update(qkv=_bf16((T * B, C), g), z=_bf16((T * B, Hv * 128), g), a=_f32((T * B, Hv), g), b=_f32((T * B, Hv), g),
                 conv_w=_bf16((C, 4), g, 0.3), A_log=torch.rand(Hv, device="cuda", generator=g) * 2.0 - 2.0, dt_bias=_bf16((Hv,), g, 0.5),
                 norm_w=_f32((128,), g, 0.02, 1.0), S=_f32((B, Hv, 128, 128), g, 0.02), conv=[_bf16((B, 3, C), g), _bf16((B, 3, C), g)],
                 out=torch.zeros((T * B, Hv * 128), dtype=torch.bfloat16, device="cuda"), turn=0)
    elif kind == "attn":
        B, L, Hq, Hkv, HD = case["B"], case["L"], case["Hq"], case["Hkv"], 256
        cos_t, sin_t = ops.rope_tables(L)
        split_len, _ = ops.attn_plan(L, B, Hkv)
        s.update(qg=_bf16((B, Hq * 2 * HD), g), k=_bf16((B, Hkv * HD), g), v=_bf16((B, Hkv * HD), g), q_norm_w=_bf16((HD,), g, 0.02),
                 k_norm_w=_bf16((HD,), g, 0.02), k_cache=_bf16((B, Hkv, L, HD), g), v_cache=_bf16((B, Hkv, L, HD), g),
                 cos=torch.from_numpy(cos_t).cuda(), sin=torch.from_numpy(sin_t).cuda(), split_len=split_len,
                 pos=torch.full((B,), L - 1, dtype=torch.int32, device="cuda"),
                 scratch=torch.zeros(ops.attn_scratch_bytes(B, Hq, HD, L, split_len), dtype=torch.uint8, device="cuda"),
                 out=torch.zeros((B, Hq * HD), dtype=torch.bfloat16, device="cuda"))
    else:
        rows, K = case["rows"], case["K"]
        s["x"] = _bf16((rows, K), g, 0.02) if case["bf16"] else _f32((rows, K), g, 0.02)
        s["W"] = torch.zeros((rows, K // 256 * 144), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return s


# ---- one pass ----------------------------------------------------------------------

def run(state):
    if isinstance(state, _Served):
        return _run_model(state)
    s, c = state, state["case"]
    if c["kind"] == "gemv":
        ops.quant_q8_1(s["x"].data_ptr(), c["K"], c["B"], s["xq"].data_ptr())
        ops.gemv_simple(s["W"].data_ptr(), c["N"], c["K"], s["xq"].data_ptr(), c["B"], s["y"].data_ptr())
        return {"xq": s["xq"], "y": s["y"]}
    if c["kind"] == "gdn":
        t = s["turn"]
        s["turn"] = t ^ 1
        ops.gdn_step(qkv=s["qkv"].data_ptr(), z=s["z"].data_ptr(), a=s["a"].data_ptr(), b=s["b"].data_ptr(), conv_w=s["conv_w"].data_ptr(),
                     conv_state_in=s["conv"][t].data_ptr(), conv_state_new=s["conv"][t ^ 1].data_ptr(), A_log=s["A_log"].data_ptr(),
                     dt_bias=s["dt_bias"].data_ptr(), norm_w=s["norm_w"].data_ptr(), S_in=s["S"].data_ptr(), S_new=s["S"].data_ptr(),
                     out=s["out"].data_ptr(), B=c["B"], Hk=c["Hk"], Hv=c["Hv"], apply_conv=1, n_tokens=c["T"])
        return {"out": s["out"], "S": s["S"], "conv": s["conv"][t ^ 1]}
    if c["kind"] == "attn":
        ops.attn_decode(qg=s["qg"].data_ptr(), k=s["k"].data_ptr(), v=s["v"].data_ptr(), q_norm_w=s["q_norm_w"].data_ptr(),
                        k_norm_w=s["k_norm_w"].data_ptr(), cos_t=s["cos"].data_ptr(), sin_t=s["sin"].data_ptr(),
                        k_cache=s["k_cache"].data_ptr(), v_cache=s["v_cache"].data_ptr(), pos=s["pos"].data_ptr(), out=s["out"].data_ptr(),
                        scratch=s["scratch"].data_ptr(), B=c["B"], Hq=c["Hq"], Hkv=c["Hkv"], HD=256, rot_half=32, max_len=c["L"],
                        split_len=s["split_len"], max_pos=c["L"] - 1, scale=1.0 / 16.0, fused_norm_rope=1)
        return {"out": s["out"], "k_row": s["k_cache"][:, :, c["L"] - 1], "v_row": s["v_cache"][:, :, c["L"] - 1]}
    ops.quantize_q4k(s["x"].data_ptr(), c["rows"], c["K"], s["W"].data_ptr(), bf16=c["bf16"])
    return {"W": s["W"]}


def _run_model(s):
    c, gm = s.case, s.gm
    gm.reset()
    if c["kind"] == "loop":
        tokens = M.runGraphDecode(gm, s.prompt, c["new"])
    elif c["kind"] == "generate":
        gm.prefill(s.prompt, read=False)
        gm.run(c["new"] - 1)
        tokens = gm.tokens(c["prompt"] - 1, c["new"])
    else:
        gm.prefill(s.prompt, read=False)
        got = []
        for i in range(c["new"]):
            ops.sample(s.logits.data_ptr(), s.cfg.vocab, c["batch"], s.idx.data_ptr(), temperature=c["temperature"], top_k=c["top_k"],
                       top_p=c["top_p"], seed=11, step_add=i)
            R.cuDtoH(s.host_idx, s.idx.data_ptr())
            got.append(s.host_idx.copy())
            if i + 1 < c["new"]:
                gm.step(s.host_idx, read=False)
        tokens = np.stack(got)
    return {"tokens": tokens, "logits": s.logits}


# ---- what a pass cannot do without ----------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "gemv":
        N, K, B = case["N"], case["K"], case["B"]
        return {"bytes": N * K // 256 * 144 + B * K * 4 + B * K // 32 * 36 + B * N * 4, "flops": 2 * N * K * B}
    if kind == "gdn":
        B, Hk, Hv, T = case["B"], case["Hk"], case["Hv"], case["T"]
        C = (2 * Hk + Hv) * 128
        per_token = C * 2 + Hv * 128 * 4 + Hv * 8
        return {"bytes": B * (2 * Hv * 128 * 128 * 4 + 2 * 3 * C * 2 + T * per_token) + C * 8, "flops": B * T * Hv * 128 * 128 * 7}
    if kind == "attn":
        B, L, Hq, Hkv = case["B"], case["L"], case["Hq"], case["Hkv"]
        return {"bytes": B * (2 * Hkv * L * 512 + Hq * 3 * 512), "flops": B * L * Hq * 256 * 4}
    if kind == "quantize":
        n = case["rows"] * case["K"]
        return {"bytes": n * (2 if case["bf16"] else 4) + n // 256 * 144, "flops": 0}
    cfg, B, T, G = CONFIGS[case["config"]], case["batch"], case["prompt"], case["new"]
    wb = M.weight_bytes(cfg)
    head = cfg.vocab * cfg.hidden // 256 * 144
    n_full = cfg.n_layers // cfg.full_attn_interval
    state = 2 * (cfg.n_layers - n_full) * (cfg.gdn_v_heads * 128 * 128 * 4 + 3 * cfg.conv_width * 2)
    kv = n_full * cfg.attn_kv_heads * 256 * 4
    # the prompt's weights and state once (token by token in the host loop), then once per further token
    passes = T + G - 1 if kind == "loop" else G
    rows = (T + T + G) * G // 2
    flops = 2 * (wb - head) // 144 * 256 * B * (T + G - 1) + 2 * head // 144 * 256 * B * passes
    return {"bytes": wb * passes + B * (state * passes + kv * (rows + T) + passes * cfg.vocab * 4), "flops": flops}


def tolerance(case):
    if case["kind"] == "gemv":
        return {"rel": 1e-5}   # 32-bit sums; the Q8_1 bytes are exact
    if case["kind"] in ("gdn", "attn"):
        return {"rel": 4e-3}   # outputs rounded to bf16
    return "exact"             # bytes; token streams, which a changed logit bit could turn
