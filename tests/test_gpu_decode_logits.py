"""Logits of decode steps (the loop of reference src/gpt2.c:179, src/qwen.c:209) against float64, early and late in a run and at every
row count where another kernel takes over: the persistent step (1 row), fp32 products (2 to 16), fp16-pair products (17 to 640), and the
decode attention's two to four warps a block."""
import numpy as np
import pytest
import torch

import helpers
import ref64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import capi
    return capi.NcmLib(helpers.CUDA_LIB)


def _open(cuda, spec, d, change=None):
    import synth
    t = synth.lm_tensors(spec, 4321)
    if change:
        change(t)
    conf, w = f"{d}/{spec.name}.conf", f"{d}/{spec.name}.ncm"
    synth.write_ncm(w, t)
    synth.write_conf(conf, synth.lm_conf(spec))
    return t, cuda.ncmb_lm_open(cuda.load_config(conf), w.encode(), int(spec.kind == "qwen"), spec.bf16_round)


def _errors(cuda, spec, t, m, B, np_, steps, n_last, plain=False):
    """relative 2-norm error of the logits of the last n_last of `steps` steps, [rows][n_last], for at most 24 rows of the batch; plain:
    and that of torch's fp32 arithmetic"""
    import synth
    ids = np.ascontiguousarray(synth.lm_prompts(spec, B, np_ + steps, 7))
    out = np.zeros((n_last, B, spec.vocab), np.float32)
    assert cuda.ncmb_lm_decode_logits(m, ids.ctypes.data, B, np_, steps, n_last, out.ctypes.data) == 0
    rows = sorted(set(np.linspace(0, B - 1, min(B, 24)).astype(int)))
    at = list(range(np_ + steps - n_last, np_ + steps))
    want = ref64.lm_logits(t, spec, ids[rows], at)
    got = out.transpose(1, 0, 2)[rows]
    assert np.isfinite(got).all()
    error = lambda x: np.sqrt(((x - want) ** 2).sum(-1) / (want ** 2).sum(-1))
    return (error(got), error(ref64.lm_logits(t, spec, ids[rows], at, dtype=torch.float32))) if plain else error(got)


@pytest.fixture(scope="module")
def models(cuda, tmp_path_factory):
    import synth
    # the widths of the GPT-2 124M and Qwen2-0.5B shapes, two layers; a gated projection small enough to be cut into slices of K; a width
    # that fills no block of K
    specs = {"gpt2": synth.LMSpec("gpt2_w", "gpt2", 2, 768, 12, 12, 3072, 1009, 64, rand_affine=1),
             "qwen": synth.LMSpec("qwen_w", "qwen", 2, 896, 14, 2, 4864, 1009, 64, rand_affine=1),
             "qwen_bf16": synth.LMSpec("qwen_w16", "qwen", 2, 896, 14, 2, 4864, 1009, 64, rand_affine=1, bf16_round=1),
             "gated_slices": synth.LMSpec("qwen_s", "qwen", 2, 512, 8, 2, 696, 301, 64, rand_affine=1),
             "ragged": synth.LMSpec("qwen_r", "qwen", 2, 80, 5, 5, 328, 301, 64, rand_affine=1)}
    made = {k: (s, *_open(cuda, s, str(tmp_path_factory.mktemp(k)))) for k, s in specs.items()}
    cuda.ncmb_set_lm_persistent(1)
    yield made
    for _, _, m in made.values():
        cuda.ncmb_lm_close(m)


# What the arithmetic leaves after two layers. fp32: a dozen roundings of 2^-24 (6e-8) on the way of a value, mostly independent.
# fp16 pairs: the tensor core's accumulator truncates, so an MMA step loses 2^-24 of what has been summed so far, on average half of the
# result, always towards zero; a product over K has K / 16 steps of two or three MMAs. The prompt's pass is not cut into slices of K.
FP32_BOUND = 6e-7


def _pair_bound(spec):
    return 3 * spec.n_inner / 16 * 2.0 ** -25


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 65, 129, 240, 256, 300, 641])
@pytest.mark.parametrize("kind", ["gpt2", "qwen", "qwen_bf16", "gated_slices", "ragged"])
def test_decode_logits_against_float64(cuda, models, kind, B):
    spec, t, m = models[kind]
    for steps in (1, 40):                                     # a prompt of one id: up to 16 rows, all of it is fp32
        e = _errors(cuda, spec, t, m, B, 1, steps, min(steps, 2))
        print(f"{kind} B={B} step {steps}: relative error mean {e.mean():.2e} max {e.max():.2e}")
        assert e.max() < (FP32_BOUND if B <= 16 else _pair_bound(spec))


def _large_inner(t):
    """units whose inner activation is about 6000 to 9000, and a down-projection that uses them"""
    for name in t:
        if name.endswith("mlp.c_fc.bias"):
            t[name][::97] = np.linspace(6000, 9000, len(t[name][::97]), dtype=np.float32)
        if name.endswith(("mlp.gate_proj.weight", "mlp.up_proj.weight")):
            t[name][::97] *= 150


@pytest.mark.parametrize("B", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("kind", ["gpt2", "qwen"])
def test_inner_activations_beyond_the_pair_range_keep_their_value(cuda, tmp_path, kind, B):
    """fp16 pairs end at 4094; calls of up to 16 rows hold activations in fp32."""
    import synth
    if kind == "gpt2":
        spec = synth.LMSpec("gpt2_large", "gpt2", 2, 192, 3, 3, 768, 301, 48, rand_affine=1)
    else:
        spec = synth.LMSpec("qwen_large", "qwen", 2, 192, 3, 1, 776, 301, 48, rand_affine=1)
    t, m = _open(cuda, spec, str(tmp_path), _large_inner)
    e, plain = _errors(cuda, spec, t, m, B, 1, 6, 3, plain=True)
    cuda.ncmb_lm_close(m)
    print(f"{kind} B={B}: relative error max {e.max():.2e}, plain fp32 {plain.max():.2e}")
    # rows whose large terms cancel amplify every rounding: plain fp32 shows by how much (clipped values are off by 1e-2 and more)
    assert e.max() < 4 * plain.max() + FP32_BOUND


@pytest.mark.parametrize("B", [1, 2, 16])
def test_partial_sums_meet_before_the_residual(cuda, tmp_path, B):
    """A hidden state much larger than what a layer adds to it: each rounding of it counts, so a product's partial sums must not be added to
    it one by one. Twelve layers with one rounding each are what plain fp32 has."""
    import synth
    spec = synth.LMSpec("gpt2_res", "gpt2", 12, 768, 12, 12, 3072, 1009, 64, rand_affine=1)

    def large_state(t):
        t["wte.weight"] *= 400
        t["wpe.weight"] *= 400
    t, m = _open(cuda, spec, str(tmp_path), large_state)
    e, plain = zip(*(_errors(cuda, spec, t, m, B, 1, steps, 3, plain=True) for steps in (9, 20, 40)))
    cuda.ncmb_lm_close(m)
    e, plain = np.mean(e), np.mean(plain)
    print(f"B={B}: relative error mean {e:.2e}, plain fp32 {plain:.2e}")
    assert e < 1.5 * plain
