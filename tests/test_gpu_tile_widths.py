"""linear_fwd (reference src/ncm.h:146) on the fp16-pair engine's 192- and 224-column tiles, with weights that need their
second half and with weights that do not (bf16 values: the stage then has no second weight tile)."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import capi
    lib = capi.NcmLib(helpers.CUDA_LIB)
    yield lib
    lib.ncmb_set_gemm_mode(3)


@pytest.mark.parametrize("bn", [128, 192, 224, 256])
@pytest.mark.parametrize("shape", [(129, 1344, 64), (700, 1344, 136), (40000, 1344, 64)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("bf16", [0, 1])
def test_wide_tiles(cuda, shape, bn, bf16, monkeypatch):
    M, N, K = shape
    monkeypatch.setenv("NCM_B200_H3_BN", str(bn))
    rng = np.random.default_rng(M + N + K + bn)
    x = rng.standard_normal((M, K)).astype(np.float32)
    W = (rng.standard_normal((N, K)) * 0.05).astype(np.float32)
    if bf16:
        W = (W.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)
    b = rng.standard_normal(N).astype(np.float32)
    rows = np.unique(np.r_[0:min(M, 300), M - 200:M])
    want = x[rows].astype(np.float64) @ W.astype(np.float64).T + b
    scale = np.abs(x[rows]).astype(np.float64) @ np.abs(W).astype(np.float64).T + np.abs(b)
    y = cuda.alloc(M * N)
    cuda.ncmb_set_gemm_mode(3)
    cuda.linear_fwd(cuda.to_backend(x), cuda.to_backend(W), cuda.to_backend(b), y, M, N, K)
    cuda.ncmb_sync()
    assert cuda.ncmb_gemm_tc_check() == 0
    err = np.abs(cuda.to_host(y, (M, N))[rows] - want) / scale
    assert err.max() <= 2e-6
