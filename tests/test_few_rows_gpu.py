"""GPU: the register-operand GEMM (at most 16 activation rows per weight matrix or routing block) at the edges
of its tiles -- 8 / 9 / 16 rows, one K chunk, K chunks that do not divide over warps and blocks, 64-column tails,
two groups per chunk -- against the fp32 oracle.

Tolerance: the products of 16-bit activations and exact integers are summed in fp32 on both sides, so what
remains is the one rounding of the result, half an ulp (at most 2^-8 bfloat16, 2^-11 float16 of the value) and fp32
sums, below k * 2^-24 of the sum of magnitudes (k <= 2560: 1.5e-4, of which a random sum sees a few per cent)."""

import pytest
import torch

from oracle import moe as omoe
from oracle import quant as oq
from tests.helpers import make_quantized, rel_max_err

pytestmark = pytest.mark.gpu
TOL = {torch.bfloat16: 2.0 ** -8 + 1.5e-4, torch.float16: 2.0 ** -11 + 1.5e-4}


def _weights(bits, k, n, group, dtype, zeros, seed):
    """(q, scales, zero points) and their device forms."""
    q, scales, z = make_quantized(k, n, group, dtype, zeros, seed)
    if bits == 8:
        gen = torch.Generator().manual_seed(seed)
        q = torch.randint(0, 256, (k, n), generator=gen, dtype=torch.int32).numpy().astype("uint8")
        z = torch.randint(0, 256, tuple(scales.shape), generator=gen, dtype=torch.int32).numpy().astype("uint8") if zeros else None
    dev = (torch.from_numpy(oq.marlin_pack(q, bits, False)).cuda(), scales.cuda(),
           None if z is None else torch.from_numpy(oq.pack_zeros(z, bits)).cuda())
    return (q, scales, z), dev


def _qtype(bits, zeros):
    from infiniops_b200 import capi

    return {(4, True): capi.QTYPE_UINT4, (4, False): capi.QTYPE_UINT4B8, (8, True): capi.QTYPE_UINT8,
            (8, False): capi.QTYPE_UINT8B128}[bits, zeros]


@pytest.mark.parametrize("dtype", (torch.bfloat16, torch.float16))
@pytest.mark.parametrize("bits,zeros", ((4, True), (4, False), (8, True), (8, False)))
@pytest.mark.parametrize("m,k,n,group", (
    (1, 128, 64, 128),      # one chunk, one tile: seven of eight warps idle
    (8, 640, 192, 64),      # five chunks, two groups in each
    (9, 1152, 64, 128),     # nine chunks: the first row of the second token tile
    (16, 2560, 320, -1),    # twenty chunks over a cluster, one group
    (5, 2304, None, 256),   # a tile more than one round of blocks (two per SM): the others whole, that one over a cluster
))
def test_dense_edges(m, k, n, group, bits, zeros, dtype):
    from infiniops_b200 import capi

    n = n or 64 * (2 * torch.cuda.get_device_properties(0).multi_processor_count + 1)
    (q, scales, z), (w, s, zd) = _weights(bits, k, n, group, dtype, zeros, m + k)
    gen = torch.Generator().manual_seed(m)
    a, bias = torch.randn((m, k), generator=gen).to(dtype), torch.randn(n, generator=gen).to(dtype)
    out = torch.full((m + 1, n), float("nan"), dtype=dtype, device="cuda")
    capi.marlin_gemm(a.cuda(), w, bias.cuda(), s, zd, _qtype(bits, zeros), m, n, k, out)
    torch.cuda.synchronize()
    assert torch.isnan(out[m].float()).all()   # nothing behind the last row
    assert rel_max_err(out[:m], oq.w4a16_gemm(a, q, scales, z, bits, bias=bias)) <= TOL[dtype]


@pytest.mark.parametrize("m", (1, 9, 16))
def test_placed_without_peers(m):
    """Columns [n, 2n) of a 3n-wide matrix: the bits of the plain call, nothing beside them -- and the batched call's
    result, which another kernel computes, to the rounding of each."""
    from infiniops_b200 import capi

    k, n, dtype = 1152, 192, torch.bfloat16
    _, (w, s, z) = _weights(4, k, n, 128, dtype, True, 60 + m)
    a = torch.randn((m, k), generator=torch.Generator().manual_seed(m)).to(dtype).cuda()
    plain, batched = (torch.empty((m, n), dtype=dtype, device="cuda") for _ in range(2))
    capi.marlin_gemm(a, w, None, s, z, capi.QTYPE_UINT4, m, n, k, plain)
    wide = torch.full((m, 3 * n), 7.0, dtype=dtype, device="cuda")
    scratch = torch.zeros(max(capi.lib().infiniops_b200_marlin_gemm_scratch_bytes(m, n, k),
                              capi.lib().infiniops_b200_marlin_gemm_batch_scratch_bytes()), dtype=torch.uint8, device="cuda")
    capi.marlin_gemm_placed(capi.gemm_problem(a, w, None, s, z, wide, m, n, k, out_ld=3 * n, out_col0=n), dtype,
                            capi.QTYPE_UINT4, scratch)
    capi.marlin_gemm_batch(capi.problem_array([capi.gemm_problem(a, w, None, s, z, batched, m, n, k)]), dtype,
                           capi.QTYPE_UINT4, scratch)
    torch.cuda.synchronize()
    assert torch.equal(wide[:, n:2 * n], plain)
    assert bool((wide[:, :n] == 7.0).all()) and bool((wide[:, 2 * n:] == 7.0).all())
    assert rel_max_err(batched, plain) <= 2 * TOL[dtype]


@pytest.mark.parametrize("block", (8, 16))
@pytest.mark.parametrize("dtype,group,zeros", ((torch.bfloat16, 128, True), (torch.float16, 64, False)))
@pytest.mark.parametrize("by_product", (False, True))   # rows read where they are / through the gather
@pytest.mark.parametrize("tokens,experts,k,n,bits", ((1, 8, 512, 128, 4), (11, 4, 1152, 192, 8), (40, 3, 256, 64, 4), (70, 3, 256, 64, 4)))
def test_routed_edges(tokens, experts, k, n, bits, by_product, dtype, group, zeros, block):
    from infiniops_b200 import capi

    top_k = 2
    hosts, devs = zip(*[_weights(bits, k, n, group, dtype, zeros, 50 + e) for e in range(experts)])
    w, s, z = (torch.stack(x) if x[0] is not None else None for x in zip(*devs))
    gen = torch.Generator().manual_seed(tokens)
    ids = torch.randint(0, experts, (tokens, top_k), generator=gen, dtype=torch.int32)
    x = torch.randn((tokens, k), generator=gen).to(dtype)
    bias = torch.randn((experts, n), generator=gen).to(dtype)
    tw = torch.rand(tokens * top_k, generator=gen)
    rows = tokens * top_k
    size, blocks = omoe.padded_sizes(rows, experts, block)
    sorted_ids = torch.empty(size, dtype=torch.int32, device="cuda")
    expert_ids = torch.empty(blocks, dtype=torch.int32, device="cuda")
    npost = torch.empty(1, dtype=torch.int32, device="cuda")
    capi.moe_align_block_size(ids.cuda(), None, experts, block, sorted_ids, expert_ids, npost)
    extra = {"block_rows": torch.empty(blocks + 1, dtype=torch.int32, device="cuda")} if by_product else {}
    args = (x.cuda(), w, bias.cuda(), s, z, sorted_ids, expert_ids, npost, tw.cuda(), block, top_k)
    out = torch.full((rows, n), float("nan"), dtype=dtype, device="cuda")
    capi.moe_wna16_marlin_gemm(*args, True, _qtype(bits, zeros), tokens, n, k, out, **extra)
    in_order = torch.full((size, n), float("nan"), dtype=dtype, device="cuda")
    capi.moe_wna16_marlin_gemm(*args, False, _qtype(bits, zeros), tokens, n, k, in_order, out_sorted=True, **extra)
    torch.cuda.synchronize()
    ref = torch.cat([oq.w4a16_gemm(x[r // top_k:r // top_k + 1], *hosts[int(ids.view(-1)[r])], bits,
                                   bias=bias[int(ids.view(-1)[r])]) for r in range(rows)])
    assert rel_max_err(out, ref * tw[:, None]) <= TOL[dtype]
    order = sorted_ids[:int(npost)].cpu().long()
    live = order < rows
    assert rel_max_err(in_order[:len(order)][live.cuda()], ref[order[live]]) <= TOL[dtype]
