"""The persistent decode step streams a CTA's weights through a ring of 16 chunks in shared memory. A product that needs more chunks
than that before it gives any back waits for ever; this walks the order in which the kernel waits and gives back, on the host."""
import helpers

RING_CHUNKS = 16
QWEN2_05B = (896, 2, 4864, 24, 151936, 1)               # C, kv heads, I, layers, V, gated
GPT2_124M = (768, 12, 3072, 12, 50257, 0)


def test_no_accepted_shape_needs_more_than_the_ring():
    import capi
    lib = capi.NcmLib(helpers.CUDA_LIB)
    for shape in (QWEN2_05B, GPT2_124M):
        for esz in (2, 4):
            assert 0 < lib.ncmb_lm_persistent_ring(*shape, esz, 148) <= RING_CHUNKS, (shape, esz)
    taken = 0
    for C in range(64, 1025, 64):
        for inner in (152, 200, C * 4, C * 4 + 8, 4864, 5632, 8184, 8192):
            for kv in {1, C // 64}:
                for gated, esz, sms in ((0, 4, 148), (1, 4, 148), (1, 2, 148), (0, 4, 132), (1, 4, 160)):
                    need = lib.ncmb_lm_persistent_ring(C, kv, inner, 3, 1009, gated, esz, sms)
                    assert need <= RING_CHUNKS, (C, inner, kv, gated, esz, sms, need)
                    taken += need > 0
    assert taken > 400


def test_every_block_of_the_step_owns_mlp_rows():
    """An exchange buffer is free to be written again because each block has since given the MLP something it computed after its
    read; a block without MLP rows could still be waiting for what is overwritten."""
    import capi
    lib = capi.NcmLib(helpers.CUDA_LIB)
    for sms in (132, 148, 160):
        for inner in range(8, 320, 8):
            need = lib.ncmb_lm_persistent_ring(192, 3, inner, 3, 301, 0, 4, sms)
            assert (need > 0) == (inner >= sms), (sms, inner)
