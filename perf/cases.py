"""Performance cases: the work users of this package have it do, through its public entry points.

Three entry points carry everything: ``frisk_b200.gemm`` and ``frisk_b200.attention_forward`` on CUDA tensors,
and ``frisk_b200.execute`` for a kernel built with the IR builders.  A case names its kind:

* ``gemm``       16-bit or fp32 product(s) C <- op(A).op(B); with ``panels`` = 2 the K extent arrives as two
                 panels, the second accumulated into C (``clear_accum=False``)
* ``fused``      a built kernel that fills C, multiplies into it and reduces C along its rows
* ``graph``      a built kernel that holds the attention graph of one query tile
* ``attention``  batched attention forward on compact BHSD tensors, in either softmax mode
"""
import math

import torch

import frisk_b200 as F

_DTYPE = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
_SIZE = {"fp16": 2, "bf16": 2, "fp32": 4}


def _gemm(m, n, k, dtype, out=None, ta=False, tb=True, panels=1, **name):
    return dict(name, kind="gemm", m=m, n=n, k=k, dtype=dtype, out=out or dtype, ta=ta, tb=tb, panels=panels)


def _fused(m, n, k, reduce, fill, **name):
    return dict(name, kind="fused", m=m, n=n, k=k, dtype="fp16", out="fp16", reduce=reduce, fill=fill)


def _graph(n_q, n_kv, d, dtype, out, **name):
    return dict(name, kind="graph", b=1, h=1, s_q=n_q, s_kv=n_kv, d=d, dtype=dtype, out=out, causal=False)


def _attention(b, h, s_q, s_kv, d, dtype, causal, normalized=False, out=None, **name):
    return dict(name, kind="attention", b=b, h=h, s_q=s_q, s_kv=s_kv, d=d, dtype=dtype, out=out or dtype,
                causal=causal, normalized=normalized)


def listed():
    return [
        # one 64-query attention tile, built as IR and executed: the smallest call, all latency
        _graph(64, 64, 64, "fp16", "fp32", name="attention_graph_tile"),
        # fill, gemm and row maximum in one built kernel, at the size of an operator's tile-level test
        _fused(512, 384, 256, "max", 0.5, name="fused_fill_gemm_max"),
        # the headline product of the benchmark
        _gemm(4096, 4096, 4096, "fp16", name="gemm_f16_4096"),
        # one rank's slice of the deep-K product (131072 over 8 ranks): fp32 partials for the reduction
        _gemm(8192, 8192, 16384, "bf16", out="fp32", name="gemm_bf16_deep_k_partial"),
        # a ragged activation-by-weight product whose K arrives in two panels, weights stored [K, N]
        _gemm(3000, 2056, 1032, "bf16", tb=False, panels=2, name="gemm_bf16_ragged_accumulate"),
        # decoding a batch of 16 against one large weight matrix
        _gemm(16, 28672, 8192, "bf16", name="gemm_bf16_decode_16"),
        # decoding a batch of 64: still bound by the weights, too many rows for the decode kernel's 16
        _gemm(64, 8192, 8192, "bf16", name="gemm_bf16_decode_64"),
        # the fp32 product of the benchmark
        _gemm(1024, 1024, 1024, "fp32", tb=False, name="gemm_f32_1024"),
        # an fp32 product of odd sizes with both operands stored transposed
        _gemm(515, 771, 1003, "fp32", ta=True, tb=True, name="gemm_f32_ragged"),
        # the benchmark's causal prefill
        _attention(8, 32, 4096, 4096, 128, "bf16", True, name="attention_prefill"),
        # one new token per sequence against a cache of 4000
        _attention(4, 32, 1, 4000, 128, "bf16", True, name="attention_decode"),
        # the two-pass mode at the largest sequence of its original envelope (64 to 1025 tokens, D = 64)
        _attention(2, 8, 1025, 1025, 64, "fp16", False, normalized=True, out="fp32", name="attention_normalized"),
    ]


def _log(rng, lo, hi, step=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v // step * step))


def draw(rng):
    kind = rng.choice(["gemm16", "gemm16", "decode", "gemm32", "fused", "graph", "prefill", "attn_decode", "normalized"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind == "gemm16":
        # row pitches of 16-bit operands are multiples of 8 elements; M is free unless A is stored [K, M]
        ta, tb = rng.choice([(False, True), (False, True), (False, False), (True, False), (True, True)])
        step = rng.choice([1, 8, 64])
        m, n = _log(rng, 64, 8192, max(step, 8) if ta else step), _log(rng, 64, 8192, step if tb else max(step, 8))
        k = _log(rng, 64, 16384, 8)
        out = rng.choice([dtype, dtype, "fp32"])
        return _gemm(m, n, k, dtype, out=out, ta=ta, tb=tb, panels=rng.choice([1, 1, 2]) if k <= 8192 else 1)
    if kind == "decode":
        return _gemm(rng.choice([rng.randint(1, 16), rng.randint(17, 128)]), _log(rng, 1024, 32768, rng.choice([1, 64])),
                     _log(rng, 1024, 16384, 8), dtype)
    if kind == "gemm32":
        step = rng.choice([1, 8])
        m, n, k = (_log(rng, 64, 2048, step) for _ in range(3))
        return _gemm(m, n, k, "fp32", ta=rng.random() < 0.3, tb=rng.random() < 0.5)
    if kind == "fused":
        step = rng.choice([1, 8, 64])
        return _fused(_log(rng, 64, 4096, step), _log(rng, 64, 4096, step), _log(rng, 64, 4096, 8),
                      rng.choice(["max", "min", "add"]), rng.choice([0.0, 0.5, -1.5]))
    if kind == "graph":
        # the IR's row reductions take powers of two
        return _graph(2 ** rng.randint(4, 9), 2 ** rng.randint(4, 11), rng.choice([64, 128]), dtype, rng.choice([dtype, "fp32"]))
    if kind == "prefill":
        d, s = rng.choice([64, 128, 128]), _log(rng, 128, 8192)
        heads = rng.randint(4, 32)
        most = max(1, min(16, int(2 ** 32 / (s * s * heads))))  # at most the pairs of the listed prefill
        return _attention(rng.randint(1, most), heads, s, s, d, dtype, rng.random() < 0.7)
    if kind == "attn_decode":
        s_kv, heads = _log(rng, 256, 16384), rng.choice([8, 16, 32])
        most = max(1, min(16, int(2 ** 20 / (s_kv * heads))))
        return _attention(rng.randint(1, most), heads, rng.choice([1, 1, rng.randint(2, 16)]), s_kv,
                          rng.choice([64, 128, 128]), dtype, True)
    n = rng.randint(64, 1025)
    return _attention(rng.randint(1, 4), rng.randint(1, 16), n, n, 64, "fp16", False, normalized=True, out="fp32")


def _normal(gen, shape, dtype, scale):
    return (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * scale).to(_DTYPE[dtype])


def _operand(gen, rows, cols, dtype, scale):
    """A large operand is drawn in row blocks, so that its fp32 draw never needs much memory."""
    t = torch.empty(rows, cols, dtype=_DTYPE[dtype], device="cuda")
    step = max(1, (1 << 26) // cols)
    for r in range(0, rows, step):
        t[r:r + step] = _normal(gen, t[r:r + step].shape, dtype, scale)
    return t


def _fused_module(case):
    s = F.create_session()
    m, n, k = case["m"], case["n"], case["k"]
    types = [s.memref_type(shape, "fp16") for shape in ([m, k], [n, k], [m, n], [m])]
    _, entry = s.new_kernel("fused", types)
    a, b, c, r = (entry.get_argument(i) for i in range(4))
    par = s.builder.create_parallel_op([4, 4], 128)
    s.builder.set_insertion_point_to_start(par.add_entry_block())

    def body(builder, iv):
        builder.create_fill_op(c, case["fill"], "fp16")
        builder.create_gemm_op(a, b, c, False, True, False)
        builder.create_reduce_op(c, r, case["reduce"], 1, True)
    s.builder.create_for_op(0, 1, 1, body)
    return s.module


def _graph_module(case):
    s = F.create_session()
    element = {"fp16": s.builder.get_f16_ty, "bf16": s.builder.get_bf16_ty, "fp32": s.builder.get_f32_ty}
    F.build_attention_kernel(s.builder, s.module, "attention", case["s_q"], case["s_kv"], case["d"],
                             element[case["dtype"]](), case["d"] ** -0.5, element[case["out"]]())
    return s.module


def _inputs(case, seed):
    """The operands of a case, made from the seed alone: [(A, B), ...] of a product, (q, k, v) of an attention."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] in ("gemm", "fused"):
        m, n, k, dtype = case["m"], case["n"], case["k"], case["dtype"]
        ta, tb = case.get("ta", False), case.get("tb", True)
        # activations N(0, 1) against weights N(0, 1/K): results of unit size, as in a model
        return [(_operand(gen, *((k, m) if ta else (m, k)), dtype, 1.0),
                 _operand(gen, *((n, k) if tb else (k, n)), dtype, k ** -0.5)) for _ in range(case.get("panels", 1))]
    return tuple(_normal(gen, (case["b"], case["h"], s, case["d"]), case["dtype"], 1.0)
                 for s in (case["s_q"], case["s_kv"], case["s_kv"]))


def prepare(case, seed):
    inputs = _inputs(case, seed)
    if case["kind"] in ("gemm", "fused"):
        c = torch.empty(case["m"], case["n"], dtype=_DTYPE[case["out"]], device="cuda")
        state = dict(kind=case["kind"], pairs=inputs, c=c, ta=case.get("ta", False), tb=case.get("tb", True))
        if case["kind"] == "fused":
            state.update(module=_fused_module(case), r=torch.empty(case["m"], dtype=c.dtype, device="cuda"))
        return state
    q, k, v = inputs
    o = torch.empty(q.shape, dtype=_DTYPE[case["out"]], device="cuda")
    if case["kind"] == "graph":
        return dict(kind="graph", module=_graph_module(case), tensors=[t[0, 0] for t in (q, k, v, o)])
    spec = dict(B=case["b"], H=case["h"], N=case["s_q"], D=case["d"], N_kv=case["s_kv"])
    return dict(kind="attention", spec=spec, tensors=[q, k, v, o], causal=case["causal"], normalized=case["normalized"])


def run(state):
    kind = state["kind"]
    if kind == "gemm":
        for i, (a, b) in enumerate(state["pairs"]):
            F.gemm(a, b, state["c"], trans_a=state["ta"], trans_b=state["tb"], clear_accum=i == 0)
        return state["c"]
    if kind == "fused":
        F.execute(state["module"], *state["pairs"][0], state["c"], state["r"])
        return state["c"], state["r"]
    if kind == "graph":
        return F.execute(state["module"], *state["tensors"])
    q, k, v, o = state["tensors"]
    return F.attention_forward(state["spec"], q, k, v, o, causal=state["causal"], normalize_p=state["normalized"])


def work(case):
    s_in, s_out = _SIZE[case["dtype"]], _SIZE[case["out"]]
    if case["kind"] in ("gemm", "fused"):
        m, n, k, panels = case["m"], case["n"], case["k"], case.get("panels", 1)
        reduced = m * s_out if case["kind"] == "fused" else 0
        return {"bytes": panels * (m + n) * k * s_in + m * n * s_out + reduced, "flops": 2 * m * n * k * panels}
    b, h, s_q, s_kv, d = (case[x] for x in ("b", "h", "s_q", "s_kv", "d"))
    # causal: query i sees s_kv - s_q + i + 1 keys
    pairs = s_q * (s_kv - s_q) + s_q * (s_q + 1) // 2 if case["causal"] else s_q * s_kv
    return {"bytes": b * h * d * (s_q * (s_in + s_out) + 2 * s_kv * s_in), "flops": 4 * b * h * d * pairs}


def tolerance(case):
    if case["kind"] in ("graph", "attention"):
        # probabilities are rounded to the input type before they meet V
        return {"rel": {"fp16": 1.2e-3, "bf16": 9e-3}[case["dtype"]]}
    if case["out"] == "fp32":
        # the fp32 accumulation error alone, which grows with the length of the sum
        return {"rel": max(2e-6, 5e-9 * case["k"] * case["panels"])}
    # one rounding to the stored type for each panel
    return {"rel": {"fp16": 1e-3, "bf16": 8e-3}[case["out"]]}


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits."""
    inputs = _inputs(case, seed)
    if case["kind"] in ("gemm", "fused"):
        c = torch.full((case["m"], case["n"]), case.get("fill", 0.0), dtype=torch.float64, device="cuda")
        for a, b in inputs:
            c += (a.T if case.get("ta", False) else a).double() @ (b.T if case.get("tb", True) else b).double()
        if case["kind"] == "gemm":
            return c
        return c, {"max": lambda: c.amax(1), "min": lambda: c.amin(1), "add": lambda: c.sum(1)}[case["reduce"]]()
    q, k, v = (t.flatten(0, 1) for t in inputs)
    s_q, s_kv = case["s_q"], case["s_kv"]
    o = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    for i in range(q.shape[0]):
        kd, vd = k[i].double(), v[i].double()
        for r in range(0, s_q, 2048):  # query i sees s_kv - s_q + i + 1 keys where the case is causal
            s = (q[i, r:r + 2048].double() @ kd.T) * case["d"] ** -0.5
            if case["causal"]:
                rows = torch.arange(r, r + s.shape[0], device="cuda")[:, None]
                s.masked_fill_(torch.arange(s_kv, device="cuda")[None] > rows + (s_kv - s_q), -math.inf)
            o[i, r:r + 2048] = torch.softmax(s, 1) @ vd
    return o[0] if case["kind"] == "graph" else o.view(inputs[0].shape)
