"""What the W4A16 linear and MoE path is measured on.

Four kinds of work, each through the entry points a program uses:

* ``linears``  one decoder layer's quantised linears (qkv, o, gate_up, down), issued one after the other
  through ``infini.ops.marlin_gemm`` -- the decode step and the prefill of a dense model;
* ``batch``    independent decode-sized linears as one ``capi.marlin_gemm_batch`` call (several sequences or
  adapters at once);
* ``moe``      a mixture-of-experts layer, as the operator chain of ``infini.ops`` (router, sort, expert
  GEMM, silu_and_mul, expert GEMM, sum) or through ``moe_layer.layer_from_logits``;
* ``repack``   the load-time shuffle of a layer's checkpoint words into the kernel's layout.

Weights are random words, as good as any checkpoint's for time and traffic; scales are |N(0,1)| * 0.01 + 1e-3
and activations N(0,1), so products and intermediates have ordinary magnitudes.
"""

import math

import torch

UINT4, UINT4B8, UINT8B128, FLOAT8 = 1125899906843648, 1125899907892224, 1125899923621888, 2814749767172868
QTYPE = {"awq4": UINT4, "gptq4": UINT4B8, "gptq8": UINT8B128, "fp8": FLOAT8}
DTYPE = {"bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    llama = {"hidden": 4096, "inter": 14336, "qkv": 6144, "group": 128, "act_order": False}
    mixtral = {"experts": 8, "top_k": 2, "hidden": 4096, "inter": 14336, "router": "softmax", "weights": "gptq4",
               "dtype": "bf16"}
    deepseek = {"experts": 256, "top_k": 8, "hidden": 7168, "inter": 2048, "router": "grouped", "weights": "awq4",
                "dtype": "bf16"}
    return [
        # one user, one token at a time: the smallest calls, one pass over the weights
        {"name": "linears_m1", "kind": "linears", "m": 1, "weights": "awq4", "dtype": "bf16", **llama},
        # a small batch of an 8-bit checkpoint, an odd number of sequences
        {"name": "linears_m7_int8", "kind": "linears", "m": 7, "weights": "gptq8", "dtype": "bf16", **llama},
        # ordinary batched decode, float16 GPTQ checkpoint
        {"name": "linears_m16", "kind": "linears", "m": 16, "weights": "gptq4", "dtype": "f16", **llama},
        # a full decode batch
        {"name": "linears_m64", "kind": "linears", "m": 64, "weights": "awq4", "dtype": "bf16", **llama},
        # a ragged chunk of a prompt with an activation-order (desc_act) checkpoint
        {"name": "linears_m333_act_order", "kind": "linears", "m": 333, "weights": "gptq4", "dtype": "f16", **llama,
         "act_order": True},
        # a whole prompt: compute-bound prefill
        {"name": "linears_m4096", "kind": "linears", "m": 4096, "weights": "gptq4", "dtype": "bf16", **llama},
        # sixteen independent decode linears in one call
        {"name": "batch_m1_4_16_64", "kind": "batch", "rows": "1,4,16,64", "weights": "awq4", "dtype": "bf16",
         "hidden": 4096, "inter": 14336, "qkv": 6144, "group": 128},
        # one token through a layer of few large experts: latency, launches and two experts' weights
        {"name": "moe_chain_e8_t1", "kind": "moe", "entry": "operators", "tokens": 1, **mixtral},
        # a prompt chunk through the same chain
        {"name": "moe_chain_e8_t1024", "kind": "moe", "entry": "operators", "tokens": 1024, **mixtral},
        # a decode batch over many small experts: nearly every row meets an expert of its own
        {"name": "moe_layer_e256_t16", "kind": "moe", "entry": "layer", "tokens": 16, **deepseek},
        # the largest call: a long prompt over many small experts
        {"name": "moe_layer_e256_t8192", "kind": "moe", "entry": "layer", "tokens": 8192, **deepseek},
        # loading a layer's weights
        {"name": "repack_gptq4", "kind": "repack", "format": "gptq", "bits": 4, "act_order": False, "hidden": 4096,
         "inter": 14336, "qkv": 6144},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi, step):
    return max(lo, min(hi, step * round(_log(rng, lo, hi) / step)))


def draw(rng):
    kind = rng.choices(("linears", "moe", "batch", "repack"), (5, 4, 1, 1))[0]
    dtype = rng.choice(("bf16", "bf16", "f16"))
    hidden = _size(rng, 1024, 8192, 128)
    inter = _size(rng, 1536, 16384, 128)
    qkv = hidden + 2 * rng.choice((64, 128, 256, 512, 1024))
    if kind == "linears":
        m = max(1, round(_log(rng, 1, 4096)))
        weights = rng.choice(("awq4", "awq4", "gptq4", "gptq4", "gptq8", "fp8"))
        group = rng.choice((128, 128, 64, 256 if hidden % 256 == 0 and inter % 256 == 0 else 128))
        return {"kind": kind, "m": m, "weights": weights, "dtype": dtype, "hidden": hidden, "inter": inter, "qkv": qkv,
                "group": group, "act_order": weights == "gptq4" and rng.random() < 0.3}
    if kind == "batch":
        rows = ",".join(str(max(1, round(_log(rng, 1, 64)))) for _ in range(rng.randint(1, 4)))
        return {"kind": kind, "rows": rows, "weights": rng.choice(("awq4", "gptq4")), "dtype": dtype, "hidden": hidden,
                "inter": inter, "qkv": qkv, "group": 128}
    if kind == "repack":
        form = rng.choice(("gptq", "awq"))
        return {"kind": kind, "format": form, "bits": rng.choice((4, 4, 8)), "act_order": form == "gptq" and rng.random() < 0.3,
                "hidden": hidden, "inter": inter, "qkv": qkv}
    experts = rng.choice((8, 16, 32, 64, 128, 256))
    top_k = rng.choice((1, 2, 2, 4)) if experts < 64 else rng.choice((4, 6, 8, 8))
    entry = rng.choice(("operators", "layer"))
    # many experts are small ones: the layer's weights stay within the largest listed layer's
    inter = min(inter, max(512, 128 * int(256 * 7168 * 2048 / (experts * hidden) / 128)))
    most = (8192 * 8 * 7168 * 2048 * (0.3 if entry == "operators" else 0.8)) / (top_k * hidden * inter)
    tokens = max(1, round(_log(rng, 1, min(8192, most))))
    return {"kind": kind, "entry": entry, "tokens": tokens, "experts": experts, "top_k": top_k, "hidden": hidden, "inter": inter,
            "router": "grouped" if experts >= 64 and rng.random() < 0.7 else "softmax",
            "weights": rng.choice(("awq4", "gptq4")), "dtype": dtype}


def _linears(case):
    """(K, N) of the layer's four linears."""
    h, i = case["hidden"], case["inter"]
    return [(h, case["qkv"]), (h, h), (h, 2 * i), (i, h)]


class _Maker:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, shape, dtype=torch.float32):
        return torch.randn(shape, generator=self.gen, device="cuda", dtype=dtype)

    def words(self, shape):
        return torch.randint(-(1 << 31), 1 << 31, shape, generator=self.gen, device="cuda", dtype=torch.int32)

    def scales(self, shape, dtype):
        return self.normal(shape).abs_().mul_(0.01).add_(1e-3).to(dtype)

    def order(self, k):
        return torch.randperm(k, generator=self.gen, device="cuda", dtype=torch.int32)

    def weights(self, kind, shape, groups, dtype):
        """Packed words [.., K/16, N * 16 / pack], scales [.., groups, N], zero points or None; `shape` = (.., K, N)."""
        *lead, k, n = shape
        pack = 4 if kind in ("gptq8", "fp8") else 8
        words = self.words((*lead, k // 16, n * 16 // pack))
        if kind == "fp8":   # the two NaN bytes are no weights
            raw = words.view(torch.uint8)
            raw[(raw & 0x7F) == 0x7F] = 0x38
        zeros = self.words((*lead, groups, n // 8)) if kind == "awq4" else None
        return words, self.scales((*lead, groups, n), dtype), zeros


def _prepare_linears(case, make):
    dtype, m = DTYPE[case["dtype"]], case["m"]
    calls = []
    workspace = torch.zeros(432, dtype=torch.int32, device="cuda")
    for k, n in _linears(case):
        w, s, z = make.weights(case["weights"], (k, n), k // case["group"], dtype)
        g_idx = perm = None
        if case["act_order"]:
            perm = make.order(k)
            g_idx = torch.arange(k, device="cuda", dtype=torch.int32) // case["group"]
        x = make.normal((m, k), dtype)
        out = torch.empty((m, n), dtype=dtype, device="cuda")
        calls.append((x, w, None, s, None, None, z, g_idx, perm, workspace, QTYPE[case["weights"]], m, n, k, True, False,
                      True, False, out))
    return {"kind": "linears", "calls": calls}


def _prepare_batch(case, make):
    from infiniops_b200 import capi

    dtype = DTYPE[case["dtype"]]
    problems, keep, outs = [], [], []
    for m in map(int, case["rows"].split(",")):
        for k, n in _linears(case):
            w, s, z = make.weights(case["weights"], (k, n), k // case["group"], dtype)
            x, out = make.normal((m, k), dtype), torch.empty((m, n), dtype=dtype, device="cuda")
            problems.append(capi.gemm_problem(x, w, None, s, z, out, m, n, k))
            keep.append((x, w, s, z))
            outs.append(out)
    scratch = torch.zeros(capi.lib().infiniops_b200_marlin_gemm_batch_scratch_bytes(), dtype=torch.uint8, device="cuda")
    return {"kind": "batch", "problems": capi.problem_array(problems), "dtype": dtype, "qtype": QTYPE[case["weights"]],
            "scratch": scratch, "outs": outs, "keep": keep}


def _prepare_repack(case, make):
    pack = 32 // case["bits"]
    calls = []
    for k, n in _linears(case):
        out = torch.empty((k // 16, n * 16 // pack), dtype=torch.int32, device="cuda")
        if case["format"] == "gptq":
            perm = make.order(k) if case["act_order"] else torch.empty(0, dtype=torch.int32, device="cuda")
            calls.append((make.words((k // pack, n)), perm, k, n, case["bits"], False, out))
        else:
            calls.append((make.words((k, n // pack)), k, n, case["bits"], False, out))
    return {"kind": "repack", "format": case["format"], "calls": calls}


def _operator_block(case):
    """Rows per routing block, 8..64 as the operators' callers choose it: the smallest that an expert's share fills."""
    share = case["tokens"] * case["top_k"] / case["experts"]
    return next((b for b in (8, 16, 32, 48) if share / b < 0.9), 64)


def _prepare_moe(case, make):
    from infiniops_b200 import moe_layer

    dtype = DTYPE[case["dtype"]]
    t, e, k, h, i = (case[x] for x in ("tokens", "experts", "top_k", "hidden", "inter"))
    w13, s13, z13 = make.weights(case["weights"], (e, h, 2 * i), h // 128, dtype)
    w2, s2, z2 = make.weights(case["weights"], (e, i, h), i // 128, dtype)
    x, logits = make.normal((t, h), dtype), make.normal((t, e))
    bias = make.normal((e,)).mul_(0.01)
    router = {"kind": "softmax", "top_k": k, "renormalize": True}
    if case["router"] == "grouped":
        router = {"kind": "grouped", "top_k": k, "bias": bias, "groups": 8, "topk_group": 4, "scaling": 2.5}
    state = {"kind": "moe", "entry": case["entry"], "x": x, "logits": logits, "router": router}
    if case["entry"] == "layer":
        weights = moe_layer.ExpertWeights(w13, s13, z13, w2, s2, z2, h, i)
        state["experts"] = moe_layer.RoutedExperts(weights, moe_layer.routing_block(t * k, e, h * i))
        return state
    block = _operator_block(case)
    size, blocks = moe_layer.padded_sizes(t * k, e, block)

    def empty(shape, kind=dtype):
        return torch.empty(shape, dtype=kind, device="cuda")

    state.update(block=block, qtype=QTYPE[case["weights"]], sizes=(t, e, k, h, i), w13=w13, s13=s13, z13=z13, w2=w2, s2=s2, z2=z2,
                 tw=empty((t, k), torch.float32), ids=empty((t, k), torch.int32), tei=empty((t, k), torch.int32),
                 sorted=empty((size,), torch.int32), eids=empty((blocks,), torch.int32), npost=empty((1,), torch.int32),
                 g=empty((t * k, 2 * i)), h=empty((t * k, i)), y=empty((t * k, h)), out=empty((t, h)),
                 workspace=torch.zeros(432, dtype=torch.int32, device="cuda"))
    return state


def prepare(case, seed):
    make = _Maker(seed)
    return {"linears": _prepare_linears, "batch": _prepare_batch, "repack": _prepare_repack, "moe": _prepare_moe}[case["kind"]](case, make)


def _run_chain(s, ops, stream):
    t, e, k, h, i = s["sizes"]
    r = s["router"]
    if r["kind"] == "softmax":
        ops.topk_softmax(s["logits"], None, None, True, s["tw"], s["ids"], s["tei"], stream=stream)
    else:
        ops.grouped_topk(s["logits"], r["bias"], r["groups"], r["topk_group"], k, True, r["scaling"], 1, s["tw"], s["ids"],
                         stream=stream)
    ops.moe_align_block_size(s["ids"], None, e, s["block"], s["sorted"], s["eids"], s["npost"], stream=stream)
    ops.moe_wna16_marlin_gemm(s["x"], s["w13"], None, s["s13"], None, None, s["z13"], None, None, s["workspace"], s["sorted"],
                              s["eids"], s["npost"], s["tw"], s["block"], k, False, s["qtype"], t, 2 * i, h, True, False, True,
                              False, -1, -1, -1, s["g"], stream=stream)
    ops.silu_and_mul(s["g"], s["h"], stream=stream)
    ops.moe_wna16_marlin_gemm(s["h"], s["w2"], None, s["s2"], None, None, s["z2"], None, None, s["workspace"], s["sorted"],
                              s["eids"], s["npost"], s["tw"], s["block"], 1, True, s["qtype"], t * k, h, i, True, False, True,
                              False, -1, -1, -1, s["y"], stream=stream)
    ops.moe_sum(s["y"].view(t, k, h), s["out"], stream=stream)
    return s["out"], s["tw"], s["ids"]


def run(state):
    import infini.ops as ops
    from infiniops_b200 import capi, moe_layer

    stream = torch.cuda.current_stream().cuda_stream
    kind = state["kind"]
    if kind == "linears":
        for args in state["calls"]:
            ops.marlin_gemm(*args, stream=stream)
        return [args[-1] for args in state["calls"]]
    if kind == "batch":
        capi.marlin_gemm_batch(state["problems"], state["dtype"], state["qtype"], state["scratch"], stream=stream)
        return state["outs"]
    if kind == "repack":
        repack = ops.gptq_marlin_repack if state["format"] == "gptq" else ops.awq_marlin_repack
        for args in state["calls"]:
            repack(*args, stream=stream)
        return [args[-1] for args in state["calls"]]
    if state["entry"] == "operators":
        return _run_chain(state, ops, stream)
    return moe_layer.layer_from_logits(state["x"], state["logits"], state["router"], state["experts"], stream=stream)


def _gemm_bytes(case, m, k, n, group, weights):
    per_weight = 1.0 if weights in ("gptq8", "fp8") else 0.5
    zeros = n / 2 if weights == "awq4" else 0
    return k * n * per_weight + (k // group) * (2 * n + zeros) + 2 * m * (k + n)


def work(case):
    kind = case["kind"]
    if kind in ("linears", "batch"):
        rows = [case["m"]] if kind == "linears" else [int(m) for m in case["rows"].split(",")]
        shapes = [(m, k, n) for m in rows for k, n in _linears(case)]
        return {"bytes": sum(_gemm_bytes(case, m, k, n, case["group"], case["weights"]) for m, k, n in shapes),
                "flops": sum(2.0 * m * k * n for m, k, n in shapes)}
    if kind == "repack":
        return {"bytes": sum(2 * k * n * case["bits"] / 8 + (4 * k if case["act_order"] else 0) for k, n in _linears(case)),
                "flops": 0}
    t, e, k, h, i = (case[x] for x in ("tokens", "experts", "top_k", "hidden", "inter"))
    touched = e * (1 - (1 - k / e) ** t)   # experts that get a row, expected for even routing
    expert = 3 * h * i / 2 + 3 * h * i / 128 * (2.5 if case["weights"] == "awq4" else 2)
    return {"bytes": touched * expert + 4 * t * h + 4 * t * e, "flops": 6.0 * t * k * h * i}


def tolerance(case):
    """Relative error of one 16-bit rounding of the weights (another order of scaling) and one of the result, of two
    implementations against each other; the MoE layer rounds its intermediates too.  Repacking moves bits."""
    if case["kind"] == "repack":
        return "exact"
    if case["kind"] == "moe":
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
    return {"rel": 5e-3 if case["dtype"] == "bf16" else 1e-3}
