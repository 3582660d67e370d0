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
