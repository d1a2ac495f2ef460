"""Where q4x_moe's scratch is carved (host code alone): the tiled f16 activations have room for whole tiles of 16 slots. A tile's
slots are interleaved every 32 bytes, so the slots of a last, partial tile reach to the whole tile's end - which once lay in the
gate's outputs."""
import pytest

import libosmos_b200
from libosmos_b200 import api, synth


@pytest.mark.parametrize("n_exp,k,dim,ff,n", [(96, 6, 2048, 2048, 85), (128, 4, 4096, 1536, 2048), (8, 2, 512, 256, 1), (20, 3, 256, 768, 33)])
def test_activations_have_whole_tiles(n_exp, k, dim, ff, n):
    lib = libosmos_b200.load()
    layer = api.Q4xMoeLayer()
    layer.dim, layer.ff, layer.n_exp, layer.k = dim, ff, n_exp, k
    for j in range(3):
        layer.type[j], layer.base[j], layer.bytes[j] = synth.TYPE_ID["MXFP4"], 1 << 20, 1 << 20
    need = lib.q4x_moe_scratch_bytes(layer, n)
    s = api.Q4xMoeScratch()
    assert need and lib.q4x_moe_scratch_bind(layer, n, 1 << 20, need, s)  # (addresses only: nothing is read or written)
    slots = n * k + 15 * min(n * k, n_exp)
    assert s.ga - s.xe16 >= (slots + 15) // 16 * 16 * max(dim, ff) * 2
    assert not lib.q4x_moe_scratch_bind(layer, n, 1 << 20, need - 1, s)
