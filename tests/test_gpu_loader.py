"""GPU: the loader's Q4_K quantiser against the oracle, bit for bit, and a checkpoint in the reference's naming loaded
into a decode model."""
import os

import numpy as np
import pytest

from bunker_b200 import loader as L
from bunker_b200 import model as M
from bunker_b200 import ops, synth
from bunker_b200 import runtime as R
from oracle import oracle as O
from oracle.model_oracle import OracleModel
from tests.util import assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
def test_quantize_q4k_matches_oracle(bk, bf16):
    rng = np.random.default_rng(21)
    N, K = 37, 1024
    x = rng.normal(0, 0.02, (N, K)).astype(np.float32)
    x[0, :256] = 0.0                                   # all-zero superblock
    x[1, :32] = 0.5                                    # constant sub-block
    x[2] = np.abs(x[2])                                # all positive: every min is zero
    x[3] = -np.abs(x[3])                               # all negative
    x[4, ::7] *= 40.0                                  # outliers that dominate their sub-blocks
    x[5] *= 1e-6                                       # scales near the f16 subnormal range
    if bf16:
        xb = synth.f32_to_bf16(x)
        x = synth.bf16_to_f32(xb)
        dx = R.DeviceBuffer.from_numpy(xb)
    else:
        dx = R.DeviceBuffer.from_numpy(x)
    out = R.DeviceBuffer(N * K // 256 * 144)
    ops.quantize_q4k(dx.ptr, N, K, out.ptr, bf16=bf16)
    assert R.cuSync() == 0
    got = out.download(np.uint8, (N, K // 256 * 144))
    assert_same_bits(got, O.q4k_quantize(x), "Q4_K superblocks")
    dx.free(), out.free()


@pytest.mark.parametrize("N,K", [(1, 256), (3, 256), (17, 256), (5, 768)])
def test_quantize_q4k_odd_superblock_counts_and_ties(bk, N, K):
    """Odd numbers of superblocks (two share a warp), and weights on rounding boundaries: multiples of half a step, where the
    quotient must be the correctly rounded one."""
    rng = np.random.default_rng(N * K)
    x = rng.normal(0, 0.02, (N, K)).astype(np.float32)
    x[0, :128] = (rng.integers(0, 31, 128) * 0.5).astype(np.float32)
    x[0, 0], x[0, 1] = 15.0, 0.0
    x[-1, 128:256] = (rng.integers(-15, 16, 128) * np.float32(0.125)).astype(np.float32)
    dx, out = R.DeviceBuffer.from_numpy(x), R.DeviceBuffer(N * K // 256 * 144)
    ops.quantize_q4k(dx.ptr, N, K, out.ptr)
    assert R.cuSync() == 0
    assert_same_bits(out.download(np.uint8, (N, K // 256 * 144)), O.q4k_quantize(x), "Q4_K superblocks")
    dx.free(), out.free()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n_sb", [1, 2, 3, 5, 31, 33])
def test_quantize_q4k_partial_groups_clamps_and_nans(bk, n_sb, bf16):
    """Four superblocks share a warp and 32 a thread block, the last of them incomplete here.  Sub-blocks whose scale is rounded far down (the clamp
    to 15), whose minimum is (the clamp to 0), and with NaNs, which become 0 and count for neither end."""
    rng = np.random.default_rng(40 + n_sb)
    x = rng.normal(0, 0.02, (n_sb, 256)).astype(np.float32)
    x[:, 32:64] *= 0.02 * rng.random((n_sb, 1)).astype(np.float32)      # scales of a few steps beside one of 63
    x[:, 64:96] = np.abs(x[:, 64:96]) * 0.05                            # no minimum, a small scale
    x[:, 96] = -0.3
    x[:, 129:160:3] = np.nan
    if bf16:
        xb = synth.f32_to_bf16(x)
        xb[:, 129:160:3] = 0x7FC0
        x = synth.bf16_to_f32(xb)
    dx, out = R.DeviceBuffer.from_numpy(xb if bf16 else x), R.DeviceBuffer(n_sb * 144)
    ops.quantize_q4k(dx.ptr, n_sb, 256, out.ptr, bf16=bf16)
    assert R.cuSync() == 0
    assert_same_bits(out.download(np.uint8, (n_sb, 144)), O.q4k_quantize(x), "Q4_K superblocks")
    dx.free(), out.free()


def _near_tie_weights(bf16: bool):
    """33 superblocks with d = dmin = 2^-5 exactly: sub-block 0 has the largest scale, 63 steps, sub-block 1 the largest minimum, the others whole
    numbers of both.  Weights on integers and on ties, all of them bf16 numbers; as f32 a third of those on ties is moved by an ulp to either side.
    Returns the weights and how far each quotient is from a tie."""
    rng = np.random.default_rng(77)
    x, off = np.empty((33, 8, 32), np.float32), np.empty((33, 8, 32))
    for sb in range(33):
        for j in range(8):
            s, m = (63, 1) if j == 0 else (8, 63) if j == 1 else (rng.choice([1, 2, 3, 4, 5, 6, 7, 8, 12, 16, 24, 32]), 0) if j < 6 else (rng.choice([2, 4, 8]), rng.integers(0, 63))
            n = rng.integers(0, 15, 32) + (0.5 if (sb + j) % 3 else rng.choice([0.0, 0.5], 32))
            if j == 0:
                n = rng.choice([0.5, 1.5], 32)
            if sb % 4 == 2 and j > 3:
                n = np.floor(n)      # no ties
            v = (n * s - m).astype(np.float32)
            v[rng.integers(0, 16)], v[16 + rng.integers(0, 16)] = -m, 15 * s - m
            if not bf16:
                t = (v + m) / s
                on = t != np.floor(t)
                v = np.where(on & (rng.random(32) < 1 / 3), np.nextafter(v, np.float32(rng.choice([-1e9, 1e9]))), v).astype(np.float32)
            x[sb, j] = v / 32
            t = (v.astype(np.float64) + m) / s
            off[sb, j] = np.abs(t - np.floor(t) - 0.5)
    return x.reshape(33, 256), off


@pytest.mark.parametrize("bf16", [False, True])
def test_quantize_q4k_many_near_ties(bk, bf16):
    """Several lanes of a warp (32 sub-blocks) have a quotient within 1e-5 of a tie, in each of the four chunks of eight weights, and others have none."""
    x, off = _near_tie_weights(bf16)
    assert np.array_equal(synth.bf16_to_f32(synth.f32_to_bf16(x)), x) == bf16
    near = off[:32].reshape(8, 32, 4, 8).min(axis=3) < 1e-5   # warp, lane, chunk
    assert near.sum(axis=1).min() >= 8 and (~near).sum(axis=1).min() >= 4
    assert (O.q4k_quantize(x).reshape(33, 144)[:, :4].copy().view(np.float16) == 2.0 ** -5).all()
    dx, out = R.DeviceBuffer.from_numpy(synth.f32_to_bf16(x) if bf16 else x), R.DeviceBuffer(33 * 144)
    ops.quantize_q4k(dx.ptr, 33, 256, out.ptr, bf16=bf16)
    assert R.cuSync() == 0
    assert_same_bits(out.download(np.uint8, (33, 144)), O.q4k_quantize(x), "Q4_K superblocks")
    dx.free(), out.free()


def test_checkpoint_load_matches_host_quantised_model(bk, tmp_path):
    """A bf16 checkpoint with the reference's tensor names (model.language_model.layers.L...., tied embed_tokens) is
    loaded through the device quantiser; the model must decode exactly like one built from the same weights quantised
    on the host by the oracle, and like the oracle itself."""
    cfg = M.CONFIG_TINY.with_(max_len=64)
    rng = np.random.default_rng(33)
    tensors, bf16_names, host = {}, set(), {}
    for name, kind, shape in M.tensor_specs(cfg):
        key = ("model.language_model.embed_tokens.weight" if name == "embed.weight" else
               "model.language_model.norm.weight" if name == "final.norm.weight" else
               "model.language_model." + name[len("model."):])
        if kind == "q4k":
            w = synth.normal_bf16(rng, shape, 0.03)
            tensors[key] = w
            bf16_names.add(key)
            host[name] = O.q4k_quantize(synth.bf16_to_f32(w))
        elif kind == "f32":
            a = (rng.uniform(-2, 0, shape) if name.endswith("A_log") else 1.0 + rng.normal(0, 0.02, shape)).astype(np.float32)
            tensors[key] = a
            host[name] = a
        else:
            w = synth.normal_bf16(rng, shape, 0.3 if name.endswith("conv1d.weight") else 0.02)
            tensors[key] = w.reshape(shape[0], 1, 4) if name.endswith("conv1d.weight") else w   # HF keeps [C, 1, 4]
            bf16_names.add(key)
            host[name] = w
    path = os.path.join(tmp_path, "tiny.safetensors")
    L.write_safetensors(path, tensors, bf16_names)
    gm = L.load_model(cfg, path, batch=1)
    ref = M.DecodeModel(cfg, host, batch=1)
    prompt = rng.integers(0, cfg.vocab, (6, 1)).astype(np.int32)
    a = M.runGraphDecode(gm, prompt, 24)
    b = M.runGraphDecode(ref, prompt, 24)
    assert np.array_equal(a, b)
    assert_same_bits(gm.logits(), ref.logits(), "logits, device-quantised vs host-quantised weights")
    info = gm.info()
    om = OracleModel(cfg, host, batch=1, split_len=info["split_len"], attn_warps=info["attn_warps"])
    assert np.array_equal(a, om.generate(prompt, 24))
    gm.destroy(), ref.destroy()
    # a checkpoint that lacks a tensor is refused by name
    del tensors["model.language_model.norm.weight"]
    L.write_safetensors(path, tensors, bf16_names)
    with pytest.raises(KeyError, match="final.norm.weight"):
        L.load_model(cfg, path)
