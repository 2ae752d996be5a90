"""GPU: the warp-per-chunk repack at the edges of its work split (a single k-tile, tile counts that do not divide
by the tiles a warp takes, one and three 64-column chunks), every source and width, bit for bit."""

import numpy as np
import pytest
import torch

from oracle import quant as oq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,n", ((16, 64), (80, 192), (1040, 64)))
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
