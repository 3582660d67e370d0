"""Quantizer and VQ-VAE entry points at the edges of what they take (reference src/vq.c, src/vqvae.c): no rows, buffers that start at any
float, contexts longer than a level's interpolation table has room for."""
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


def _model(cuda, d, **over):
    import capi
    import synth
    spec = dataclasses.replace(synth.spec_c2(n_layer=1, n_embd=64, n_head=1, n_kv=1, vocab=300, name="edges"), in_vocab=40, **over)
    conf, w = synth.write_ncp(spec, d)
    return spec, conf, w, capi.NcpModel(cuda, conf, w, arena_mb=64)


@pytest.fixture(scope="module")
def model(cuda, tmp_path_factory):
    return _model(cuda, str(tmp_path_factory.mktemp("edges")))


def test_no_rows(cuda, model):
    spec, _, _, m = model
    z, idx = cuda.to_backend(np.zeros(64, np.float32)), cuda.to_backend(np.full(64, 77, np.int32))
    host = np.full(64, 77, np.int32)
    cuda.ncmb_vq_nearest_dev(m.vq, 3, z, 0, idx)
    cuda.ncmb_vq_encode_dev(m.vq, z, 0, idx)
    cuda.vq_z_to_idx(m.vq, z, 0, host.ctypes.data)
    assert (cuda.to_host(idx, (64,), np.int32) == 77).all() and (host == 77).all()


@pytest.mark.parametrize("B", [1, 5, 70])
def test_buffers_that_start_at_any_float(cuda, model, B):
    """Device buffers of a caller that are aligned for a float but not for 16 bytes: the results of aligned ones, to fp32 rounding (other
    kernels take them)."""
    spec, _, _, m = model
    n = B * spec.L * spec.vq_dim
    rng = np.random.default_rng(B)
    close = lambda a, b: np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
    ids = rng.integers(2, spec.in_vocab, (B, spec.L)).astype(np.int32)
    z, z1 = cuda.alloc(n + 4), cuda.alloc(n + 4) + 4
    cuda.vqvae_encode_z(m.vqvae, ids.ctypes.data, z, B)
    cuda.vqvae_encode_z(m.vqvae, ids.ctypes.data, z1, B)
    zh = cuda.to_host(z, (n,))
    assert close(cuda.to_host(z1, (n,)), zh)
    zh = (zh + 0.05 * rng.standard_normal(n)).astype(np.float32)
    cuda.mem_h2d(z, zh.ctypes.data, zh.nbytes)
    cuda.mem_h2d(z1, zh.ctypes.data, zh.nbytes)
    total = sum(spec.levels)
    got, want = np.zeros((2, B, total), np.int32)
    cuda.vq_z_to_idx(m.vq, z, B, want.ctypes.data)
    cuda.vq_z_to_idx(m.vq, z1, B, got.ctypes.data)
    assert (got == want).all() and np.array_equal(cuda.to_host(z1, (n,)), zh)
    lg, lg1 = (cuda.alloc(B * spec.L * spec.in_vocab) for _ in range(2))
    cuda.vqvae_decode(m.vqvae, z, lg, B)
    cuda.vqvae_decode(m.vqvae, z1, lg1, B)
    shape = (B * spec.L * spec.in_vocab,)
    assert close(cuda.to_host(lg1, shape), cuda.to_host(lg, shape))
    codes = np.ascontiguousarray(want[:, 1:5])
    nx = B * spec.levels[2] * spec.vq_dim
    out = {}
    for dz, dx in ((0, 0), (4, 0), (0, 4), (4, 4)):
        zb, xb = cuda.alloc(n + 4) + dz, cuda.alloc(nx + 4) + dx
        cuda.mem_h2d(zb, zh.ctypes.data, zh.nbytes)
        cuda.vq_next_input(m.vq, codes.ctypes.data, 1, zb, xb, B)
        out[dz, dx] = cuda.to_host(zb, (n,)), cuda.to_host(xb, (nx,))
    for v in out.values():
        assert close(v[0], out[0, 0][0]) and close(v[1], out[0, 0][1])


@pytest.mark.parametrize("L", [3072, 4096])
def test_long_contexts(cuda, tmp_path, L):
    """A level's interpolation weights are tabled in shared memory up to 3072 positions (48 KB)."""
    import orc
    spec, conf, w, m = _model(cuda, str(tmp_path), levels=[1, 5, L], vocab=[300] * 3, l1_cascade=[], l1_norm=0, enc_layers=1, dec_layers=1)
    z = (0.05 * np.random.default_rng(L).standard_normal((2, L, spec.vq_dim))).astype(np.float32)
    idx = np.zeros((2, L + 6), np.int32)
    cuda.vq_z_to_idx(m.vq, cuda.to_backend(z), 2, idx.ctypes.data)
    want = orc.Model(conf, w).z_to_idx(z)
    assert (idx != want).mean() <= 1e-3                      # codes at near-ties
    assert (idx[:, :6] == want[:, :6]).all()
    zh = [cuda.alloc(z.size) for _ in range(3)]
    cuda.vq_idx_to_zhats(m.vq, want.ctypes.data, 2, (C.c_void_p * 3)(*zh))
    for got, ref in zip(zh, orc.Model(conf, w).idx_to_zhats(want, 3)):
        assert np.abs(cuda.to_host(got, z.shape) - ref).max() <= 1e-6 * np.abs(ref).max() + 1e-7
