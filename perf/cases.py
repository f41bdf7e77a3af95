"""The work that programs built on venom_b200 have it do, as a list of measurable cases.

  layer       nmv.SrnmSpmm(x): a torch.nn.Linear held in V:N:M form inside a model (BERT encoder, GPT decoder block);
              decoding brings 8 .. 256 tokens a call, prefill and encoder batches 512 .. 16384
  product     capi.Prepared.spmm(B): the bare sparse x dense product, [K,N] in and [M,N] out
  host        capi.Prepared.spmm_host(B, C): the same product for operands that live in pinned host memory
  sparsify    nmv.MagnitudeSparsifier(weight): prune by magnitude, then compress (once for every weight of a model)
  compress    capi.compress(dense, column-loc): values and 2:4 metadata of a matrix that is pruned already
  decompress  capi.decompress(values, metadata, column-loc): back to the dense matrix

Everything is fp16 with fp32 accumulation, n = 2; V is 32, 64 or 128 and m (columns a group) 4 to 32.
"""
import math

import torch

from venom_b200 import capi
from venom_b200.nmv import MagnitudeSparsifier, SrnmSpmm
from venom_b200.synth import random_vnm_dense_cuda, vnm_sizes


def listed():
    return [
        # one decoding step of a small model, where launches and host work count: BERT-large's square projections
        dict(name="layer-decode-small", kind="layer", M=1024, K=1024, V=64, m=8, N=8, bias=True),
        # one decoding step of sixteen sequences through the widest attention projection of a GPT-3-shaped block
        dict(name="layer-decode-gpt", kind="layer", M=36864, K=12288, V=128, m=16, N=16, bias=True),
        # BERT-large's first feed-forward layer, batch 32 x sequence 512
        dict(name="layer-bert", kind="layer", M=4096, K=1024, V=64, m=8, N=16384, bias=True),
        # one sequence of 2048 tokens through the output projection of a GPT-3-shaped block
        dict(name="layer-gpt", kind="layer", M=12288, K=12288, V=128, m=16, N=2048, bias=True),
        # a layer with no round number in it: the last tile of every dimension is ragged; no bias
        dict(name="layer-ragged", kind="layer", M=2976, K=2040, V=32, m=8, N=1368, bias=False),
        # the benchmark's single product at BERT size
        dict(name="product-single", kind="product", M=1024, K=4096, V=64, m=8, N=4096),
        # high sparsity at BERT-large's second feed-forward shape
        dict(name="product-sparse", kind="product", M=1024, K=4096, V=128, m=32, N=16384),
        # the benchmark's headline product
        dict(name="product-large", kind="product", M=49152, K=12288, V=128, m=8, N=32768),
        # a product for a caller whose activations live on the host
        dict(name="host", kind="host", M=4096, K=1024, V=64, m=8, N=16384),
        # model preparation: a GPT-3-sized weight is pruned and compressed
        dict(name="sparsify", kind="sparsify", M=12288, K=12288, V=128, m=16, fp32=False),
        # the benchmark's compressor matrix
        dict(name="compress", kind="compress", M=49152, K=12288, V=128, m=8, count=False),
        # the dense copy of a stored GPT-3-sized weight
        dict(name="decompress", kind="decompress", M=12288, K=12288, V=128, m=16),
    ]


MOST_WEIGHT = 49152 * 12288
MOST_PRODUCT = 2.0 * 49152 * 12288 * 32768 * (2 / 8)


def _log(rng, lo, hi, multiple):
    """A multiple of `multiple` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["layer"] * 7 + ["product"] * 4 + ["host", "sparsify", "sparsify", "compress", "compress", "decompress", "decompress"])
    while True:
        m = rng.choice([4, 8, 8, 8, 16, 16, 20, 32])
        V = rng.choice([32, 64, 128])
        c = dict(kind=kind, M=_log(rng, 512, 49152, V), K=_log(rng, 512, 12288, math.lcm(m, 8)), V=V, m=m)
        weight = c["M"] * c["K"]
        if kind in ("layer", "product", "host"):
            c["N"] = _log(rng, 8, 16384, 8)
            if kind == "layer":
                c["bias"] = rng.random() < 0.7
            if kind == "host" and 2 * c["N"] * (c["M"] + c["K"]) > 1 << 28:
                continue
            if 2.0 * weight * c["N"] * 2 / m > MOST_PRODUCT:
                continue
        if kind == "sparsify":
            c["fp32"] = rng.random() < 0.5
        if kind == "compress":
            c["count"] = rng.random() < 0.5
        # the pruner scores every quadruple of a group's columns: C(m,4) of them
        if kind in ("layer", "sparsify") and weight * math.comb(m, 4) / m > 12288 * 12288 * math.comb(16, 4) / 16 * (4 if kind == "layer" else 1):
            continue
        if weight > MOST_WEIGHT:
            continue
        return c


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weight(c, seed, dtype):
    """An initialised weight, N(0, 0.02), as torch.nn.Linear holds it: [out features, in features]."""
    w = torch.empty((c["M"], c["K"]), dtype=dtype, device="cuda")
    return w.normal_(0, 0.02, generator=_generator(seed))


def _layer(c, seed):
    linear = torch.nn.utils.skip_init(torch.nn.Linear, c["K"], c["M"], bias=c["bias"], device="cuda", dtype=torch.float16)
    linear.requires_grad_(False)
    linear.weight.copy_(_weight(c, seed, torch.float16))
    if c["bias"]:
        linear.bias.normal_(0, 0.02, generator=_generator(seed + 1))
    return SrnmSpmm(linear, 2, c["m"], c["V"], sparsifier=MagnitudeSparsifier(2, c["m"], c["V"]))


def _operand(c, seed):
    """A seeded V:2:m matrix with uniform values and its compressed arrays."""
    dense, colloc = random_vnm_dense_cuda(c["M"], c["K"], c["V"], c["m"], seed=seed)
    values, meta, _ = capi.compress(dense, colloc, c["V"], c["m"], count_violations=False)
    return dense, colloc, values, meta


def prepare(case, seed):
    c, kind = case, case["kind"]
    M, K, V, m, N = c["M"], c["K"], c["V"], c["m"], c.get("N")
    s = dict(case=c)
    if kind == "layer":
        s["layer"] = _layer(c, seed)
        s["x"] = torch.randn((N, K), device="cuda", generator=_generator(seed + 2)).half()
    elif kind in ("product", "host"):
        _, colloc, values, meta = _operand(c, seed)
        s["operand"] = capi.Prepared(values, meta, colloc, M, K, V, m)
        b = torch.empty((K, N), dtype=torch.float16, device="cuda").uniform_(-1, 1, generator=_generator(seed + 2))
        if kind == "product":
            s["b"] = b
        else:
            s["b"] = b.cpu().pin_memory()
            s["out"] = torch.empty((M, N), dtype=torch.float16, pin_memory=True)
    elif kind == "sparsify":
        s["weight"] = _weight(c, seed, torch.float32 if c["fp32"] else torch.float16)
        s["sparsifier"] = MagnitudeSparsifier(2, m, V)
    elif kind == "compress":
        s["dense"], s["colloc"], _, _ = _operand(c, seed)
    elif kind == "decompress":
        _, s["colloc"], s["values"], s["meta"] = _operand(c, seed)
    else:
        raise ValueError("unknown kind %r" % kind)
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "layer":
        return state["layer"](state["x"])
    if kind == "product":
        return state["operand"].spmm(state["b"])
    if kind == "host":
        return state["operand"].spmm_host(state["b"], state["out"])
    if kind == "sparsify":
        t = state["sparsifier"](state["weight"])
        return {"values": t.values, "metadata": t.metadata, "columns": t.columns, "violations": t.violations}
    if kind == "compress":
        values, meta, bad = capi.compress(state["dense"], state["colloc"], c["V"], c["m"], count_violations=c["count"])
        return {"values": values, "metadata": meta, "violations": bad}
    return capi.decompress(state["values"], state["meta"], state["colloc"], c["M"], c["K"], c["V"], c["m"])


def work(case):
    M, K, V, m, N = case["M"], case["K"], case["V"], case["m"], case.get("N")
    _, nv, nm, nc = vnm_sizes(M, K, V, m)
    packed = 2 * nv + 4 * nm + 4 * nc
    kind = case["kind"]
    if kind in ("layer", "product", "host"):
        # two kept entries a group and row
        return {"bytes": packed + 2 * K * N + 2 * M * N + (2 * M if case.get("bias") else 0), "flops": 2.0 * M * N * 2 * -(-K // m)}
    if kind == "sparsify":
        # the score of a quadruple sums two magnitudes of each row of the block
        return {"bytes": (4 if case["fp32"] else 2) * M * K + packed, "flops": 2.0 * M * (K // m) * math.comb(m, 4)}
    return {"bytes": 2 * M * K + packed, "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("layer", "product", "host"):
        # fp32 sums rounded to fp16 once (twice with a bias)
        return {"rel": 1e-3, "max": 1e-2}
    return "exact"
