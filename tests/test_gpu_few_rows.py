"""Decode steps of 1 to 641 rows (the loop of reference src/gpt2.c:179, src/qwen.c:209): the persistent kernel at one row, the
few-row products and their folded reductions up to 640, the general path above -- at the edges of their row tiles (16, 32, 64,
128), with widths that fill no tile, and with two to four warps a block of the decode attention (500 rows: three). Greedy ids of a few rows against the oracle's independent runs."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import capi
    return capi.NcmLib(helpers.CUDA_LIB)


@pytest.fixture(scope="module")
def models(cuda, tmp_path_factory):
    import orc
    import synth
    made = {}
    for kind in ("gpt2", "qwen", "qwen_bf16"):
        d = str(tmp_path_factory.mktemp(kind))
        if kind == "gpt2":
            spec = synth.LMSpec(kind, "gpt2", 3, 192, 3, 3, 200, 301, 48, rand_affine=1)
        else:
            spec = synth.LMSpec(kind, "qwen", 3, 192, 3, 1, 200, 301, 48, rope_theta=1e6, rand_affine=1, bf16_round=int(kind == "qwen_bf16"))
        conf, w = synth.write_lm(spec, d)
        made[kind] = (spec, cuda.ncmb_lm_open(cuda.load_config(conf), w.encode(), int(kind != "gpt2"), spec.bf16_round),
                      orc.LM(conf, w, kind != "gpt2"))
    yield made
    for _, m, _ in made.values():
        cuda.ncmb_lm_close(m)
    cuda.ncmb_set_lm_persistent(1)                            # the default


@pytest.mark.parametrize("B", [1, 2, 4, 5, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257, 500, 640, 641])
@pytest.mark.parametrize("kind", ["gpt2", "qwen", "qwen_bf16"])
def test_greedy_ids(cuda, models, kind, B):
    import synth
    spec, m, om = models[kind]
    cuda.ncmb_set_lm_persistent(1)
    n_new = 6
    P = np.ascontiguousarray(synth.lm_prompts(spec, B, 35, B))
    out = np.zeros((B, n_new), np.int32)
    cuda.ncmb_lm_generate(m, P.ctypes.data, B, P.shape[1], n_new, 0.0, 0, 1.0, 0, -1, out.ctypes.data)
    for b in sorted({0, B // 2, B - 1}):
        want = om.generate(P[b], n_new, temp=0.0)
        assert (out[b] == want).all(), (kind, B, b, out[b], want)
    assert cuda.ncmb_gemm_tc_check() == 0


@pytest.mark.parametrize("C,H,inner", [(896, 14, 4864), (768, 12, 8192)])
def test_one_row_whose_down_projection_rows_do_not_fit_the_ring_together(cuda, tmp_path, C, H, inner):
    """fp32: 7 x 4864 and 6 x 8192 floats a CTA against a ring of 32768; the rows are given back in groups."""
    import orc
    import synth
    spec = synth.LMSpec("ring", "qwen", 3, C, H, 2, inner, 301, 64, rope_theta=1e6, rand_affine=1)
    conf, w = synth.write_lm(spec, str(tmp_path))
    m = cuda.ncmb_lm_open(cuda.load_config(conf), w.encode(), 1, 0)
    om = orc.LM(conf, w, True)
    cuda.ncmb_set_lm_persistent(1)
    n_new = 12
    P = np.ascontiguousarray(synth.lm_prompts(spec, 1, 35, 4))
    out = np.zeros((1, n_new), np.int32)
    for kw in (dict(temp=0.0, top_k=0, top_p=1.0, seed=0), dict(temp=0.7, top_k=0, top_p=0.95, seed=9)):
        cuda.ncmb_lm_generate(m, P.ctypes.data, 1, P.shape[1], n_new, kw["temp"], kw["top_k"], kw["top_p"], kw["seed"], -1, out.ctypes.data)
        assert cuda.ncmb_gemm_tc_check() == 0
        want = om.generate(P[0], n_new, **kw)
        assert (out[0] == want).all(), (C, kw, out[0], want)
    cuda.ncmb_lm_close(m)


@pytest.mark.parametrize("B", [1, 3])
def test_a_wait_that_ran_out_ends_a_generate_without_ids(cuda, models, B, capfd):
    """The persistent step gives up at once when the error word is set and the chain's kernels run on; neither passes its ids on."""
    import synth
    spec, m, _ = models["qwen"]
    cuda.ncmb_set_lm_persistent(1)
    P = np.ascontiguousarray(synth.lm_prompts(spec, B, 35, 2))
    out = np.zeros((B, 6), np.int32)
    args = (m, P.ctypes.data, B, P.shape[1], 6, 0.0, 0, 1.0, 0, -1, out.ctypes.data)
    assert cuda.ncmb_lm_generate(*args) == 6
    want = out.copy()
    cuda.ncmb_gemm_tc_raise(61)
    assert cuda.ncmb_lm_generate(*args) == -1
    assert (out == -1).all()
    assert "code 61" in capfd.readouterr().err
    assert cuda.ncmb_lm_generate(*args) == 6 and (out == want).all()       # the word is clear again
