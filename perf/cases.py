"""What a user of this library has it do, as cases that can be timed and compared.

Five kinds of call, all through the C interface that ``capi`` binds:

* ``ncp``     -- coarse-to-fine generate from id prefixes, then codes -> token ids (what the gen / infer commands do);
* ``lm``      -- GPT-2 / Qwen2 shaped generation with a KV cache: prompt pass, then one step per new token;
* ``nll``     -- mean next-token likelihood of windows of text (the ppl commands): prompt pass and the head on every position;
* ``encode``  -- token rows -> latents -> residual-quantizer codes (the vq-encode command, data preparation);
* ``nearest`` -- flat nearest-code search of vectors in device memory against one codebook.

Shapes are this repository's configurations (``synth.spec_c1`` ... ``spec_qwen_05b``). Weights are N(0, 0.02) from a fixed
seed and are loaded once per process, as a serving program holds them; ids, prefixes and vectors come from the case's seed.
The gain of the last norm is set so that logits have a standard deviation of about 4, as those of trained checkpoints do:
with a gain of 1 they would have 0.5, every sampled distribution would be close to uniform, and a pick would hang on the
last bits of its logits.
"""
import ctypes as C
import dataclasses
import functools
import math
import os
import tempfile

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()
capi, synth = pkg.capi, pkg.synth

NCP_SPECS = {"c1": synth.spec_c1, "c2": synth.spec_c2, "c5": synth.spec_c5}
LM_SPECS = {"gpt2": synth.spec_gpt2_124m, "qwen": synth.spec_qwen_05b}
LAST_NORM = {"c1": "gen.transformer.ln_f.weight", "c2": "gen.transformer.ln_f.weight",
             "c5": "gen.transformer.ln_f.weight", "gpt2": "ln_f.weight", "qwen": "model.norm.weight"}
FIRST_BLOCK = ("gen.transformer.blocks.0.", "h.0.", "model.layers.0.")


def quantizer_spec():
    """The box-scale configuration's VQ-VAE (codebooks 16384 x 64, levels 1-4-16-32) with a one-layer transformer."""
    return synth.spec_c2(n_layer=1, vocab=16384, name="quantizer")


# ------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # one puzzle through the small model: the smallest call, all launches and latency
        {"name": "ncp_c1_b1", "kind": "ncp", "model": "c1", "B": 1, "temp": 0.0, "top_k": 0, "top_p": 1.0, "cfg": 0.0,
         "freq": 0.0, "ragged": False},
        # a handful of users' requests at once: odd batch, prefixes of different lengths, guidance and sampling on
        {"name": "ncp_c2_b19_ragged", "kind": "ncp", "model": "c2", "B": 19, "temp": 0.8, "top_k": 50, "top_p": 0.9,
         "cfg": 1.5, "freq": 0.2, "ragged": True},
        # the mid-size configuration at its stated batch (the benchmark's workload)
        {"name": "ncp_c2_b256", "kind": "ncp", "model": "c2", "B": 256, "temp": 0.8, "top_k": 50, "top_p": 0.9, "cfg": 1.5,
         "freq": 0.2, "ragged": False},
        # the box-scale model (24 x 1024, codebooks of 16384), a slice of its batch
        {"name": "ncp_c5_b160", "kind": "ncp", "model": "c5", "B": 160, "temp": 0.8, "top_k": 50, "top_p": 0.9, "cfg": 1.5,
         "freq": 0.2, "ragged": False},
        # one interactive GPT-2 shaped completion, greedy, fp32 weights
        {"name": "gpt2_b1", "kind": "lm", "model": "gpt2", "B": 1, "np": 128, "n_new": 64, "temp": 0.0, "top_k": 0, "top_p": 1.0},
        # the same model serving 64 prompts
        {"name": "gpt2_b64", "kind": "lm", "model": "gpt2", "B": 64, "np": 128, "n_new": 64, "temp": 0.0, "top_k": 0, "top_p": 1.0},
        # one interactive Qwen2 shaped completion, nucleus sampling over the whole vocabulary, bf16 weights
        {"name": "qwen_b1", "kind": "lm", "model": "qwen", "B": 1, "np": 512, "n_new": 64, "temp": 0.7, "top_k": 0, "top_p": 0.95},
        # a partly filled server: odd batch, odd prompt length
        {"name": "qwen_b27_odd", "kind": "lm", "model": "qwen", "B": 27, "np": 333, "n_new": 47, "temp": 0.7, "top_k": 0, "top_p": 0.95},
        # a full one, at the configuration's largest batch and prompt
        {"name": "qwen_b256", "kind": "lm", "model": "qwen", "B": 256, "np": 512, "n_new": 64, "temp": 0.7, "top_k": 0, "top_p": 0.95},
        # perplexity over text: 512-id windows of documents, the last of each shorter
        {"name": "qwen_nll", "kind": "nll", "model": "qwen", "B": 12, "T": 512},
        # preparing training rows: tokens -> codes
        {"name": "encode_rows", "kind": "encode", "B": 8192},
        # the stated quantizer sweep: 2^20 vectors against 16384 codes
        {"name": "nearest_1m", "kind": "nearest", "n": 1 << 20},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ncp", "ncp", "ncp", "lm", "lm", "lm", "nll", "encode", "nearest"])
    if kind == "ncp":
        model = rng.choice(["c1", "c2", "c5"])
        sampled = model != "c1" or rng.random() < 0.3
        guided = model != "c1" and rng.random() < 0.7
        return {"kind": kind, "model": model, "B": _log(rng, 1, 160 if model == "c5" else 256),
                "temp": 0.8 if sampled else 0.0, "top_k": rng.choice([20, 50, 100]) if sampled else 0,
                "top_p": rng.choice([0.9, 0.95, 1.0]) if sampled else 1.0, "cfg": 1.5 if guided else 0.0,
                "freq": 0.2 if guided and rng.random() < 0.7 else 0.0, "ragged": model != "c1" and rng.random() < 0.5}
    if kind == "lm":
        greedy = rng.random() < 0.4
        return {"kind": kind, "model": rng.choice(["gpt2", "qwen"]), "B": _log(rng, 1, 256), "np": _log(rng, 16, 512),
                "n_new": _log(rng, 8, 64), "temp": 0.0 if greedy else 0.7,
                "top_k": 0 if greedy else rng.choice([0, 0, 40]), "top_p": 1.0 if greedy else 0.95}
    if kind == "nll":
        return {"kind": kind, "model": rng.choice(["gpt2", "qwen"]), "B": _log(rng, 1, 12), "T": _log(rng, 64, 512)}
    if kind == "encode":
        return {"kind": kind, "B": _log(rng, 16, 8192)}
    return {"kind": kind, "n": _log(rng, 1 << 10, 1 << 20)}


# ------------------------------------------------------------------------------------------- models (once per process)

@functools.lru_cache(maxsize=None)
def library():
    lib = pkg.load_library()
    lib.arena_init_default()
    return lib


def _tensors(make, spec, key):
    """The spec's tensors. The package draws one block; the other layers' matrices are drawn on the GPU (quick)."""
    t = make(dataclasses.replace(spec, n_layer=1), 1234)
    gen = torch.Generator(device="cuda").manual_seed(1234)
    for name in [n for n in t if n.startswith(FIRST_BLOCK)]:
        first = next(p for p in FIRST_BLOCK if name.startswith(p))
        for b in range(1, spec.n_layer):
            a = t[name]
            if a.ndim > 1:
                w = torch.randn(a.shape, device="cuda", generator=gen) * 0.02
                if getattr(spec, "bf16_round", 0):
                    w = w.bfloat16().float()
                a = w.cpu().numpy()
            t[first.replace("0", str(b)) + name[len(first):]] = a
    if key in LAST_NORM:
        gain = 4.0 / (0.02 * math.sqrt(spec.n_embd))
        t[LAST_NORM[key]] = synth._round_bf16(t[LAST_NORM[key]] * np.float32(gain))
    return t


class _Ncp(capi.NcpModel):
    """NcpModel without its own arena (several models live in this process)."""

    def __init__(self, lib, conf, weights):
        self.lib = lib
        self.cfg = lib.load_config(conf)
        self.ws = lib.load_weights(weights)
        self.vqvae = lib.vqvae_load(self.cfg, C.byref(self.ws))
        self.ncp = lib.ncp_load(self.cfg, C.byref(self.ws), self.vqvae)
        self.vq = lib.vqvae_vq(self.vqvae)
        self.total = lib.vq_total_codes(self.vq)


@functools.lru_cache(maxsize=None)
def ncp_model(key):
    spec = quantizer_spec() if key == "quantizer" else NCP_SPECS[key]()
    with tempfile.TemporaryDirectory() as tmp:
        conf, w = os.path.join(tmp, "m.conf"), os.path.join(tmp, "m.ncm")
        synth.write_conf(conf, synth.ncp_conf(spec))
        synth.write_ncm(w, _tensors(synth.ncp_tensors, spec, key))
        return spec, _Ncp(library(), conf, w)


@functools.lru_cache(maxsize=None)
def lm_model(key):
    spec = LM_SPECS[key]()
    with tempfile.TemporaryDirectory() as tmp:
        conf, w = os.path.join(tmp, "m.conf"), os.path.join(tmp, "m.ncm")
        synth.write_conf(conf, synth.lm_conf(spec))
        (synth.write_ncm2 if spec.bf16_round else synth.write_ncm)(w, _tensors(synth.lm_tensors, spec, key))
        lib = library()
        handle = lib.ncmb_lm_open(lib.load_config(conf), w.encode(), int(spec.kind == "qwen"), int(spec.bf16_round))
        if not handle:
            raise RuntimeError(f"ncmb_lm_open failed: {key}")
        return spec, handle


# ------------------------------------------------------------------------------------------- states and passes

def prepare(case, seed):
    kind, lib = case["kind"], library()
    s = {"case": case, "seed": int(seed) % (1 << 31) + 1, "lib": lib}
    rng = np.random.default_rng(int(seed))
    if kind == "ncp":
        spec, s["model"] = ncp_model(case["model"])
        s["L"] = spec.L
        s["prefix"] = synth.ncp_prefixes(spec, case["B"], int(seed))
        if case["ragged"]:                                            # ids first, pads behind them
            n = rng.integers(spec.prefix_len // 4, spec.prefix_len + 1, size=(case["B"], 1))
            s["prefix"] = np.where(np.arange(spec.prefix_len)[None, :] < n, s["prefix"], spec.pad_id).astype(np.int32)
        s["allow"] = np.full(max(spec.vocab), 1.0 / max(spec.vocab)) if case["freq"] > 0 else None
    elif kind == "lm":
        spec, s["model"] = lm_model(case["model"])
        s["ids"] = np.ascontiguousarray(synth.lm_prompts(spec, case["B"], case["np"], int(seed)))
        s["out"] = np.zeros((case["B"], case["n_new"]), np.int32)
    elif kind == "nll":
        spec, s["model"] = lm_model(case["model"])
        s["ids"] = np.ascontiguousarray(synth.lm_prompts(spec, case["B"], case["T"], int(seed)))
        s["lens"] = np.full(case["B"], case["T"], np.int32)
        s["lens"][::4] = rng.integers(case["T"] // 4, case["T"] + 1, size=s["lens"][::4].shape)
        s["out"] = np.zeros(case["B"], np.float64)
    elif kind == "encode":
        spec, s["model"] = ncp_model("quantizer")
        s["ids"] = synth.zipf_ids(rng, case["B"] * spec.L, 2, spec.in_vocab).reshape(case["B"], spec.L)
        s["z"] = torch.empty((case["B"], spec.L, spec.vq_dim), device="cuda")
        s["codes"] = np.zeros((case["B"], spec.total), np.int32)
    else:
        spec, s["model"] = ncp_model("quantizer")
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        s["x"] = torch.randn((case["n"], spec.vq_dim), device="cuda", generator=g)
        s["idx"] = torch.empty(case["n"], device="cuda", dtype=torch.int32)
    return s


def run(s):
    case, lib, m = s["case"], s["lib"], s["model"]
    kind = case["kind"]
    if kind == "ncp":
        codes = m.generate(s["prefix"], temp=case["temp"], top_k=case["top_k"], top_p=case["top_p"], cfg=case["cfg"],
                           freq=case["freq"], allow=s["allow"], seed=s["seed"])
        return {"codes": codes, "tokens": m.decode_tokens(codes, s["L"])}
    if kind == "lm":
        lib.ncmb_lm_generate(m, s["ids"].ctypes.data, case["B"], case["np"], case["n_new"], case["temp"], case["top_k"],
                             case["top_p"], s["seed"], -1, s["out"].ctypes.data)
        return s["out"]
    if kind == "nll":
        lib.ncmb_lm_nll(m, s["ids"].ctypes.data, case["B"], case["T"], s["lens"].ctypes.data, s["out"].ctypes.data)
        return s["out"]
    if kind == "encode":
        lib.vqvae_encode_z(m.vqvae, s["ids"].ctypes.data, s["z"].data_ptr(), case["B"])
        lib.vq_z_to_idx(m.vq, s["z"].data_ptr(), case["B"], s["codes"].ctypes.data)
        return {"z": s["z"], "codes": s["codes"]}
    lib.ncmb_vq_nearest_dev(m.vq, 3, s["x"].data_ptr(), case["n"], s["idx"].data_ptr())
    return s["idx"]


# ------------------------------------------------------------------------------------------- work and tolerance

def _block_macs(n_embd, kv_dim, hidden, gated):
    return n_embd * (n_embd + 2 * kv_dim) + n_embd * n_embd + (3 if gated else 2) * n_embd * hidden


def work(case):
    """Multiply-adds of the dense layers and of attention over what is visible; bytes: the weights once per pass that
    needs them (once per step of a decode loop), the K/V cache once per step that reads it, ids and results."""
    kind = case["kind"]
    if kind == "ncp":
        spec = NCP_SPECS[case["model"]]()
        kvd = spec.n_kv_heads * (spec.n_embd // spec.n_head)
        gated = bool(spec.swiglu or spec.geglu)
        per = _block_macs(spec.n_embd, kvd, spec.mlp_hidden or 4 * spec.n_embd, gated)
        P = spec.prefix_len * (0.625 if case["ragged"] else 1.0)
        B, sides = case["B"], 2 if case["cfg"] > 0 else 1
        macs = B * P * spec.n_layer * (per + P * spec.n_embd * 2)
        macs += B * sum(n * spec.n_layer * (per * sides + 2 * spec.n_embd * (P + n + (sides - 1) * (n + 1))) for n in spec.levels)
        macs += B * sides * sum(n * v * spec.n_embd for n, v in zip(spec.levels, spec.vocab))
        macs += B * spec.L * (spec.dec_layers * 12 * spec.vq_dim ** 2 + spec.vq_dim * spec.in_vocab)
        weights = spec.n_layer * per + sum(spec.vocab) * (spec.n_embd + spec.vq_dim) + spec.in_vocab * spec.vq_dim
        return {"bytes": 4.0 * (weights + B * (spec.prefix_len + spec.total + spec.L)), "flops": 2.0 * macs}
    if kind in ("lm", "nll"):
        spec = LM_SPECS[case["model"]]()
        kvd = spec.n_kv_heads * (spec.n_embd // spec.n_head)
        per = spec.n_layer * _block_macs(spec.n_embd, kvd, spec.n_inner, spec.kind == "qwen")
        head, B = spec.vocab * spec.n_embd, case["B"]
        wbytes = (2.0 if spec.bf16_round else 4.0) * (per + head)
        T = case["np"] if kind == "lm" else case["T"]
        att = spec.n_layer * 2 * spec.n_embd
        if kind == "nll":
            return {"bytes": wbytes + 4.0 * B * T, "flops": 2.0 * B * T * (per + head + att * (T + 1) / 2)}
        steps = case["n_new"] - 1
        ctx = T + (steps + 1) / 2
        macs = B * T * (per + att * (T + 1) / 2) + B * head + steps * B * (per + head + att * ctx)
        kv = 4.0 * spec.n_layer * 2 * kvd * B * ctx
        return {"bytes": wbytes * (1 + steps) + steps * kv + 4.0 * B * (T + case["n_new"]), "flops": 2.0 * macs}
    spec = quantizer_spec()
    D, V = spec.vq_dim, spec.vocab[0]
    if kind == "encode":
        n = case["B"] * spec.L
        macs = n * (spec.enc_layers * (12 * D * D + 2 * spec.L * D)) + case["B"] * spec.total * V * D
        return {"bytes": 4.0 * (n * (1 + D) + case["B"] * spec.total + len(spec.levels) * V * D), "flops": 2.0 * macs}
    return {"bytes": 4.0 * (case["n"] * (D + 1) + V * D), "flops": 2.0 * case["n"] * V * D}


def tolerance(case):
    """Ids and codes are whole: two fp32-grade implementations differ at near-ties, and after one the rest of that row may.
    Latents and likelihoods are fp32-grade sums."""
    if case["kind"] == "nll":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] == "encode":
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
    if case["kind"] == "nearest":
        return {"rel": 0.0, "differ": 1e-3}
    return {"rel": 0.0, "differ": 0.01}
