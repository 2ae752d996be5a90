"""GPU: the warp-per-chunk repack at the edges of its work split (a single k-tile, tile counts that do not divide
by the tiles a warp takes, one and three 64-column chunks), every source and width, bit for bit.  4-bit AWQ and
small 4-bit GPTQ matrices take the staged form."""

import numpy as np
import pytest
import torch

from oracle import quant as oq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", ((16, 64), (80, 192), (1040, 64), (1040, 2112)))   # (the last: GPTQ 4-bit, from 2 Mi weights on)
@pytest.mark.parametrize("bits", (4, 8))
@pytest.mark.parametrize("source", ("gptq", "awq"))
def test_repack_edges(source, bits, k, n):
    from infiniops_b200 import capi

    q = np.random.default_rng(k + n + bits).integers(0, 1 << bits, size=(k, n), dtype=np.uint8)
    expect = torch.from_numpy(oq.marlin_pack(q, bits, False))
    out = torch.full((expect.shape[0] + 1, expect.shape[1]), -7, dtype=torch.int32, device="cuda")
    if source == "gptq":
        capi.gptq_marlin_repack(torch.from_numpy(oq.gptq_pack(q, bits)).cuda(), None, k, n, bits, False, out[:-1])
    else:
        capi.awq_marlin_repack(torch.from_numpy(oq.awq_pack(q, bits)).cuda(), k, n, bits, False, out[:-1])
    assert torch.equal(out[:-1].cpu(), expect)
    assert bool((out[-1] == -7).all())   # nothing behind the last tile


@pytest.mark.parametrize("bits", (4, 8))
@pytest.mark.parametrize("source", ("gptq", "awq"))
def test_repack_words_off_a_16_byte_boundary(source, bits):
    """The source may sit on any word: a view one word into a larger buffer."""
    from infiniops_b200 import capi

    k, n = 80, 192
    q = np.random.default_rng(bits).integers(0, 1 << bits, size=(k, n), dtype=np.uint8)
    packed = torch.from_numpy((oq.gptq_pack if source == "gptq" else oq.awq_pack)(q, bits)).flatten()
    buffer = torch.zeros(packed.numel() + 1, dtype=torch.int32, device="cuda")
    buffer[1:] = packed.cuda()
    words = buffer[1:]
    assert words.data_ptr() % 16 == 4
    expect = torch.from_numpy(oq.marlin_pack(q, bits, False))
    out = torch.full(expect.shape, -7, dtype=torch.int32, device="cuda")
    if source == "gptq":
        capi.gptq_marlin_repack(words, None, k, n, bits, False, out)
    else:
        capi.awq_marlin_repack(words, k, n, bits, False, out)
    assert torch.equal(out.cpu(), expect)
