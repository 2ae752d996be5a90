"""GPU: the GEMMs may start before the kernel in front of them has ended (programmatic dependent launch), so what that
kernel wrote -- weights, by a repack or a copy, as well as activations -- must be read after the dependency wait.

One weight buffer is rewritten in front of every GEMM of a chain whose activations are the previous GEMM's result,
nothing waited for on the host; the results must have the bits that the same calls give one at a time."""

import pytest
import torch

from oracle import quant as oq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("writer", ("repack", "copy"))
@pytest.mark.parametrize("bits", (4, 8))
@pytest.mark.parametrize("m", (1, 16, 17, 64, 300))   # both token tiles of the register-operand kernel, then tensor-memory tiles
def test_weights_written_right_in_front(m, bits, writer):
    from infiniops_b200 import capi

    size, links, dtype = 1024, 6, torch.bfloat16
    qtype = capi.QTYPE_UINT4B8 if bits == 4 else capi.QTYPE_UINT8B128
    gen = torch.Generator().manual_seed(m + bits)
    qs = [torch.randint(0, 1 << bits, (size, size), generator=gen, dtype=torch.int32).numpy().astype("uint8") for _ in range(links)]
    sources = [torch.from_numpy(oq.gptq_pack(q, bits)).cuda() for q in qs]
    packed = [torch.from_numpy(oq.marlin_pack(q, bits, False)).cuda() for q in qs]
    scales = torch.full((size // 128, size), 2.0 ** (-7 if bits == 4 else -11), dtype=dtype, device="cuda")
    x = torch.randn((m, size), generator=gen).to(dtype).cuda()

    def gemm(a, w, out):
        capi.marlin_gemm(a, w, None, scales, None, qtype, m, size, size, out)

    want, a = [], x
    for w in packed:
        out = torch.empty((m, size), dtype=dtype, device="cuda")
        gemm(a, w, out)
        torch.cuda.synchronize()
        want.append(out)
        a = out
    w = torch.empty_like(packed[0])
    got = [torch.empty((m, size), dtype=dtype, device="cuda") for _ in range(4 * links)]
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        link = i % links
        if writer == "repack":
            capi.gptq_marlin_repack(sources[link], None, size, size, bits, False, w)
        else:
            w.copy_(packed[link])
        gemm(x if link == 0 else got[i - 1], w, out)
    torch.cuda.synchronize()
    assert all(torch.isfinite(t.float()).all() for t in want)
    assert all(torch.equal(out, want[i % links]) for i, out in enumerate(got))
