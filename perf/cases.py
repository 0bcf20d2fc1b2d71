"""The work this framework is used for, as measurable cases.

A case is one call sequence through the public operators of ``gcnasm_b200.api``, of one of these kinds:

linear   a quantised layer of a served model: bf16 activations, fused activation quantiser, fp8 GEMM on weights that
         were quantised (and, for ``flat``, pre-shuffled) once at load time; block scales or MXFP8
gemm     the fp8 GEMM alone on operands that are quantised already: no scale, per-tensor or block scales, batches,
         row-major or pre-shuffled weights, bf16 or fp32 result
gemm16   the bf16 sibling
weights  what a loader does with one fp32 weight matrix: 128x128 quantisation, then the pre-shuffle
host     the host-buffer entry: operands and result in host memory, copies included

Sizes are those of the benchmark configurations and tests (18432x7168 and 7168x2048 layers, the 16384x7168x8192
shard, 8192 cubes, the 256x512x1024 call) and ragged neighbours of them.
"""
import torch

from gcnasm_b200 import _lib as L
from gcnasm_b200 import api


def _case(kind, m, n, k, **more):
    c = {"kind": kind, "m": m, "n": n, "k": k, "scale": "block", "layout": "row", "out": "bf16", "batch": 1, "pinned": False}
    c.update(more)
    return c


def listed():
    return [
        # one small call of the per-tensor GEMM: launch latency and host time
        _case("gemm", 256, 512, 1024, name="tensor 256x512x1024", scale="tensor"),
        # token generation: one sequence, a small layer at 16 sequences, a large layer at 64; pre-shuffled weights
        _case("linear", 1, 18432, 7168, name="decode m1 18432x7168", layout="flat"),
        _case("linear", 16, 7168, 2048, name="decode m16 7168x2048", layout="flat"),
        _case("linear", 64, 18432, 7168, name="decode m64 18432x7168", layout="flat"),
        # a short, ragged prompt (or a chunk of one)
        _case("linear", 333, 7168, 2048, name="chunk m333 7168x2048"),
        # prompt processing: the ordinary layer, and the largest one, a rank's shard of the column-parallel layer
        _case("linear", 4096, 7168, 2048, name="prefill m4096 7168x2048"),
        _case("linear", 16384, 7168, 8192, name="prefill m16384 7168x8192"),
        # MXFP8 at its benchmark size
        _case("linear", 8192, 8192, 8192, name="mx 8192 cube", scale="mx"),
        # batched unscaled product on pre-shuffled weights with an fp32 result, ragged in every dimension
        _case("gemm", 700, 2064, 1152, name="flat batch4 700x2064x1152", scale="none", layout="flat", out="f32", batch=4),
        # bf16 operands
        _case("gemm16", 4096, 4096, 4096, name="bf16 4096 cube", scale="none"),
        # loading a model: one large weight matrix
        _case("weights", 0, 18432, 7168, name="weights 18432x7168", layout="flat"),
        # a program that keeps everything in (pageable) host memory, as the reference's drivers do
        _case("host", 4096, 7168, 2048, name="host 4096x7168x2048"),
    ]


_MAX_FLOPS = 2 * 16384 * 7168 * 8192


def _between(rng, lo, hi, multiple=1):
    """Log-uniform over [lo, hi], rounded down to a multiple."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return max(multiple, v // multiple * multiple)


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["gemm", "gemm", "gemm16", "weights", "host"])
    while True:
        layout = rng.choice(["row", "flat"])
        if kind == "linear":
            scale = rng.choice(["block", "block", "block", "mx"])
            m = _between(rng, 1, 16384) if rng.random() < 0.6 else _between(rng, 1, 64)
            n = _between(rng, 512, 18432, 128) if scale == "block" else _between(rng, 512, 8192, 8)
            layout = layout if scale == "block" else "row"      # the MX operator takes row-major weights
            c = _case(kind, m, n, _between(rng, 512, 8192, 128), scale=scale, layout=layout)
        elif kind == "gemm":
            scale = rng.choice(["none", "tensor", "tensor", "block"])
            batch = rng.choice([1, 1, 1, 2, 4, 8])
            n = _between(rng, 256, 8192, 128 if scale == "block" else (16 if layout == "flat" else 8))
            k = _between(rng, 256, 8192, 128 if scale == "block" or layout == "flat" else 16)
            c = _case(kind, _between(rng, 1, 8192), n, k, scale=scale, layout=layout, batch=batch, out=rng.choice(["bf16", "bf16", "f32"]))
        elif kind == "gemm16":
            k = _between(rng, 256, 8192, 64 if layout == "flat" else 8)
            n = _between(rng, 256, 8192, 16 if layout == "flat" else 8)
            c = _case(kind, _between(rng, 1, 8192), n, k, scale="none", layout=layout, out=rng.choice(["bf16", "f32"]))
        elif kind == "weights":
            c = _case(kind, 0, _between(rng, 512, 18432, 128), _between(rng, 512, 8192, 128), layout="flat")
        else:
            c = _case(kind, _between(rng, 1, 4096), _between(rng, 512, 8192, 128), _between(rng, 512, 4096, 128), scale=rng.choice(["block", "tensor"]),
                      pinned=rng.random() < 0.5)
        flops = 2 * c["m"] * c["n"] * c["k"] * c["batch"]
        if flops * (2 if kind == "gemm16" else 1) <= _MAX_FLOPS and c["batch"] * c["n"] * (c["m"] + c["k"]) <= 1 << 29:
            return c


def _out_dtype(case):
    return torch.bfloat16 if case["out"] == "bf16" else torch.float32


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)

    kind, m, n, k, batch = case["kind"], case["m"], case["n"], case["k"], case["batch"]
    s = dict(case)
    if kind == "weights":
        s["w"] = normal(n, k)
        return s
    if kind == "linear":
        s["x"] = normal(m, k, dtype=torch.bfloat16)
        if case["scale"] == "mx":
            w, _, s["sfb"] = api.quantize_mx32(normal(n, k))
        else:
            w, s["sfb"] = api.quantize_128x128(normal(n, k))
        s["b"] = api.shuffle_b(w, "nk") if case["layout"] == "flat" else w
        return s
    if kind == "gemm16":
        s["a"], b = normal(m, k, dtype=torch.bfloat16), normal(n, k, dtype=torch.bfloat16)
        s["b"] = api.shuffle_b_bf16(b, "nk") if case["layout"] == "flat" else b
        return s
    # gemm and host: operands quantised beforehand
    parts = {"a": [], "b": [], "sfa": [], "sfb": []}
    for _ in range(batch):
        if case["scale"] == "block":
            (a, sfa), (b, sfb) = api.quantize_1x128(normal(m, k)), api.quantize_128x128(normal(n, k))
        elif case["scale"] == "tensor":
            (a, sfa), (b, sfb) = api.quantize_tensor(normal(m, k)), api.quantize_tensor(normal(n, k))
        else:
            a, b = api.cast_e4m3(normal(m, k)), api.cast_e4m3(normal(n, k))
            sfa = sfb = None
        if case["layout"] == "flat":
            b = api.shuffle_b(b, "nk")
        for name, t in (("a", a), ("b", b), ("sfa", sfa), ("sfb", sfb)):
            parts[name].append(t)
    if case["scale"] == "tensor":           # one scale per operand, whatever the batch
        parts["sfa"], parts["sfb"] = parts["sfa"][:1], parts["sfb"][:1]
    for name, ts in parts.items():
        s[name] = None if ts[0] is None else (ts[0] if len(ts) == 1 else torch.stack(ts))
    if kind == "host":
        def host(t):
            t = t.cpu()
            return (t.pin_memory() if case["pinned"] else t).numpy()

        for name in parts:
            s[name] = host(s[name])
        s["result"] = torch.zeros(m, n, dtype=torch.bfloat16, pin_memory=case["pinned"])
        s["c"] = s["result"].view(torch.int16).numpy()
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        if s["scale"] == "mx":
            q, atoms = api.quantize_act_bf16_mx32(s["x"])
            return api.gemm_a8w8_mx(q, s["b"], atoms, s["sfb"])
        q, sfa = api.quantize_act_bf16_1x128(s["x"])
        return api.gemm_a8w8_blockscale(q, s["b"], sfa, s["sfb"], b_flat_n=s["n"] if s["layout"] == "flat" else None)
    if kind == "gemm":
        if s["scale"] == "block":
            return api.gemm_a8w8_blockscale(s["a"], s["b"], s["sfa"], s["sfb"], out_dtype=_out_dtype(s),
                                            b_flat_n=s["n"] if s["layout"] == "flat" else None)
        if s["layout"] == "flat":
            return api.flatmm_a8w8(s["a"], s["b"], s["n"], s["sfa"], s["sfb"], out_dtype=_out_dtype(s))
        return api.gemm_a8w8(s["a"], s["b"], s["sfa"], s["sfb"], out_dtype=_out_dtype(s))
    if kind == "gemm16":
        return api.gemm_a16w16(s["a"], s["b"], n=s["n"], flat=s["layout"] == "flat", out_dtype=_out_dtype(s))
    if kind == "weights":
        q, sfb = api.quantize_128x128(s["w"])
        return api.shuffle_b(q, "nk"), sfb
    if s["scale"] == "block":
        api.gemm_a8w8_host(s["a"], s["b"], s["c"], sfa=s["sfa"], sfb=s["sfb"], scale_mode=L.SCALE_BLOCK)
    else:
        api.gemm_a8w8_host(s["a"], s["b"], s["c"], scale_a=s["sfa"], scale_b=s["sfb"], scale_mode=L.SCALE_TENSOR)
    return s["result"]


def work(case):
    m, n, k, batch = case["m"], case["n"], case["k"], case["batch"]
    if case["kind"] == "weights":           # fp32 in; bytes and block scales out
        return {"bytes": 4 * n * k + n * k + n * k // 4096, "flops": 0}
    a_item = 2 if case["kind"] in ("linear", "gemm16") else 1
    b_item = 2 if case["kind"] == "gemm16" else 1
    moved = a_item * m * k + b_item * n * k + (2 if case["out"] == "bf16" else 4) * m * n
    if case["scale"] == "block":
        moved += n * k // 4096 + (0 if case["kind"] == "linear" else 4 * m * (k // 128))
    elif case["scale"] == "mx":
        moved += n * k // 32
    return {"bytes": batch * moved, "flops": 2 * batch * m * n * k}


def tolerance(case):
    if case["kind"] == "weights":
        return "exact"
    if case["out"] == "f32":                # fp32 sums in another order
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 4e-3, "max": 1.6e-2}     # a bf16 result: one rounding step apart where the fp32 sums differ
