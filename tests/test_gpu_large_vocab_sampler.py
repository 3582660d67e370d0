"""Device row sampler over vocabularies larger than one CTA holds (rule of reference src/kernels.c:794-825): candidates by parts
for top_k, mass by distance and lists for the nucleus alone. Against the same walk in fp64 with the same uniforms."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import capi
    lib = capi.NcmLib(helpers.CUDA_LIB)
    if not lib.has("ncmb_sample_rows_dev"):
        pytest.skip("device row sampler not exported")
    return lib


def walk(row, temp, top_k, top_p, u):
    w = (row / np.float32(temp)).astype(np.float32).astype(np.float64)
    order = np.argsort(-w, kind="stable")[:top_k or row.size]
    p = np.exp(w[order] - w[order[0]])
    p /= p.sum()
    cum = np.cumsum(p)
    cut = np.nonzero(cum - 2 * p > top_p)[0]
    n = int(cut[0]) if cut.size else p.size
    x = u * cum[n - 1]
    j = min(int(np.searchsorted(cum[:n], x, side="left")), n - 1)
    near = np.abs(cum[max(0, j - 1):j + 1] - x).min() < 1e-9       # a draw on a boundary may fall on either side
    return order[j], near


@pytest.mark.parametrize("V", [4097, 16385, 50257, 151936])
@pytest.mark.parametrize("B", [1, 5, 300])
@pytest.mark.parametrize("top_k,top_p", [(1, 0.9), (40, 0.95), (256, 0.5), (0, 0.95), (0, 1.0)])
def test_picks(cuda, V, B, top_k, top_p):
    rng = np.random.default_rng(V + B + top_k)
    lg = (rng.standard_normal((B, V)) * 4).astype(np.float32)
    if B >= 5:
        lg[1] = 0.75                                               # every entry tied: no list holds them
        lg[2] = np.round(lg[2])                                    # thousands of ties per value
        lg[3] *= 0.01                                              # close to uniform
        lg[4, V - 1] = 200.0                                       # the rest has no mass
    u = rng.random(B)
    d_lg, d_u, d_out = cuda.to_backend(lg), cuda.to_backend(u), cuda.alloc(B)
    cuda.ncmb_sample_rows_dev(d_lg, B, V, 0.7, top_k, top_p, d_u, d_out)
    got = cuda.to_host(d_out, (B,), np.int32)
    for b in list(range(min(B, 6))) + ([B - 1] if B > 6 else []):
        want, near = walk(lg[b], 0.7, top_k, top_p, u[b])
        assert got[b] == want or near, (b, got[b], want)
