"""Nearest-code search (reference src/vq.c:420-450): the coarse fp16 pass, its fp32 refinement, the full scan and the fp16-pair
products of many undecided rows must give the argmin of float64 distances (lowest index among equal codes), whatever the scales
and however close codes lie."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import capi
    return capi.NcmLib(helpers.CUDA_LIB)


# (rows, codes, dims, codebook): the last scanned and the first two-pass row count, ragged row blocks and code tiles,
# one and two k-blocks, dims the tensor-core pass does not take, codes too close for the coarse pass, repeated codes
CASES = [(1, 512, 64, "normal"), (256, 1000, 64, "normal"), (257, 1000, 64, "normal"), (5000, 16384, 64, "normal"),
         (40000, 513, 64, "normal"), (3001, 700, 32, "normal"), (1500, 260, 128, "normal"), (600, 100, 20, "normal"),
         (2000, 1024, 64, "close"), (700, 4096, 128, "close"), (4097, 512, 64, "repeated"), (300, 40, 8, "repeated"),
         # undecided rows through the pair products: a second wave of blocks, two k-blocks, a tile that is not full, dims below a k-block
         (40000, 600, 64, "close"), (1500, 1100, 128, "close"), (3001, 700, 32, "repeated"), (1024, 16384, 64, "close"), (9000, 300, 64, "dead"),
         (500, 1000, 64, "shifted"), (900, 600, 128, "shifted")]

# What separates the pick's distance from the smallest, against |e| (|x| + |e|): fp32 sums 1e-6. Pairs: three roundings or dropped
# products of 2^-22 a dot product and twelve truncating MMA steps of 2^-24 (twice that for 128 dims), twice that in a distance, of two codes.
FP32, PAIR = 1e-6, 4 * (3 * 2.0 ** -22 + 24 * 2.0 ** -24)


@pytest.mark.parametrize("rows,V,D,book", CASES)
def test_nearest_codes(cuda, tmp_path, rows, V, D, book):
    import capi
    import synth
    spec = dataclasses.replace(synth.spec_c2(n_layer=1, n_embd=64, n_head=1, n_kv=1, vocab=V, name="near"), vq_dim=D, l1_cascade=[],
                               l1_norm=0, in_vocab=32)
    conf, w = synth.write_ncp(spec, str(tmp_path))
    m = capi.NcpModel(cuda, conf, w, arena_mb=64)
    rng = np.random.default_rng(rows + V + D)
    E = (rng.standard_normal((V, D)) * 0.05).astype(np.float32)
    if book == "close":
        E = (E[:1] + E * 1e-3).astype(np.float32)
    if book == "repeated":
        E = E[rng.integers(0, V // 7 + 1, V)]
    if book == "dead":
        E[V // 8:] *= 1e-3
    if book == "shifted":
        E += 3 * rng.standard_normal(D).astype(np.float32)
    t = C.cast(cuda.weights_get(C.byref(m.ws), b"tok.vq.embeddings.3.weight"), C.POINTER(capi.Tensor)).contents
    cuda.mem_h2d(t.data, E.ctypes.data, E.nbytes)
    x = (rng.standard_normal((rows, D)) * np.exp(rng.uniform(-18, 6, size=(rows, 1)))).astype(np.float32)
    x[::3] = E[rng.integers(0, V, len(x[::3]))] + 0.01 * rng.standard_normal((len(x[::3]), D)).astype(np.float32)
    x[rows // 2] = 0
    xd, idx_d = cuda.to_backend(x), cuda.alloc(rows)
    cuda.ncmb_vq_nearest_dev(m.vq, 3, xd, rows, idx_d)
    got = cuda.to_host(idx_d, (rows,), np.int32)
    assert cuda.ncmb_gemm_tc_check() == 0
    assert got.min() >= 0 and got.max() < V
    E64, x64 = E.astype(np.float64), x.astype(np.float64)
    cn = (E64 * E64).sum(1)
    size = np.sqrt(cn.max()) * (np.sqrt((x64 * x64).sum(1)) + np.sqrt(cn.max()))
    for r0 in range(0, rows, 4096):
        d = cn - 2 * x64[r0:r0 + 4096] @ E64.T
        i = np.arange(len(d))
        assert (d[i, got[r0:r0 + 4096]] - d.min(1) <= (PAIR if book in ("close", "dead", "repeated") and rows >= 1024 else FP32) * size[r0:r0 + 4096]).all()
    if book == "shifted":
        # rows of about the codes' length are compared by sums of (x - e)^2: D roundings of the distance itself, however long x and e are
        d = ((x64[::3, None] - E64[None]) ** 2).sum(2)
        assert (d[np.arange(len(d)), got[::3]] <= d.min(1) * (1 + D * 2.0 ** -23)).all()
    if book == "repeated":
        first = {e.tobytes(): j for j, e in reversed(list(enumerate(E)))}
        assert all(first[E[j].tobytes()] == j for j in got)
    cuda.ncp_free(m.ncp)
    cuda.vqvae_free(m.vqvae)
    cuda.weights_free(C.byref(m.ws))
