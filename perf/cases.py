"""What users of this package have it do, as measurable cases.

A case is one call (or one captured decode step) through the package's own modules: palettized
projections, the merged Q/K/V and gated-MLP modules, the embedding, the K-grouped variant. Sizes
are those of the 9B hybrid model the package is built around (hidden 4096, MLP 12288, heads of
1024 to 8192 rows, a vocabulary of 248320) or generic ones of the same ranges; weights, palettes
and activations are synthetic with the distributions the parity tests use (uniform codes, sorted
0.02 * randn palettes, randn activations).

listed() holds the named cases, draw(rng) one more case of the same ranges, prepare() what a
program holds before the call, run() the call, work() what the call cannot do without, tolerance()
how far two correct implementations of the same precision may lie apart.
"""
from __future__ import annotations

import importlib
import math

import torch

pkg = importlib.import_module("rag-cache-engineering-qwen35-9b-flute_b200")
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
HIDDEN, INTERMEDIATE, VOCAB = 4096, 12288, 248320
FULL_ATTENTION_EVERY = 4           # layers 3, 7, ... of the hybrid model are full attention
LARGEST_FLOPS = 2.0 * 2048 * 3 * HIDDEN * INTERMEDIATE

DEFAULTS = dict(dtype="bf16", bits=4, bits2=0, group=128, rank=0, rotated=False, bias=False, hadamard=0)


def listed():
    return [
        # one attention output projection of a decode step, one sequence
        dict(name="proj_m1", op="linear", M=1, N=4096, K=4096),
        # a deployed two-stream artifact in the loader's default dtype: 4 + 1 bit gate projection,
        # wide palette groups, rank-32 residual, rotated input, one sequence
        dict(name="proj_two_stream_m1", op="linear", M=1, N=12288, K=4096, bits=4, bits2=1, group=512, rank=32,
             rotated=True, dtype="fp16"),
        # the output head of a decode step, one sequence: the largest single weight
        dict(name="lm_head_m1", op="linear", M=1, N=VOCAB, K=HIDDEN),
        # hybrid palettization: a 3-bit projection with 64-row groups under a batch of 16 sequences
        dict(name="proj_3bit_m16", op="linear", M=16, N=12288, K=4096, bits=3, group=64),
        # the gated MLP of a decode step, eight sequences
        dict(name="mlp_m8", op="mlp", M=8, K=4096, I=12288),
        # the projections of eight decoder layers as a server replays them, one CUDA graph per step:
        # a single sequence, and a batch of 64
        dict(name="decode_step_m1", op="layers", M=1, layers=8),
        dict(name="decode_step_m64", op="layers", M=64, layers=8),
        # a short prompt of odd length through the merged attention projections of an artifact with
        # rank-32 residuals
        dict(name="qkv_prompt_333", op="qkv", M=333, K=4096, Nq=8192, Nk=1024, Nv=1024, rank=32, dtype="fp16"),
        # a long prompt through one MLP
        dict(name="mlp_prompt_2048", op="mlp", M=2048, K=4096, I=12288),
        # a long prompt through one projection behind the 128-point block Hadamard transform
        dict(name="proj_prompt_2048_hadamard", op="linear", M=2048, N=12288, K=4096, hadamard=128),
        # the prompt's token rows out of the palettized embedding table
        dict(name="embed_prompt_2048", op="embed", M=2048, N=VOCAB, K=HIDDEN),
        # palettes grouped along the input axis, one sequence
        dict(name="kgrouped_m1", op="kgrouped", M=1, N=4096, K=4096),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], evenly spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choices(("linear", "head", "qkv", "mlp", "layers", "embed", "kgrouped"), (35, 5, 15, 20, 10, 5, 10))[0]
    dtype = rng.choice(("bf16", "fp16"))
    bits = rng.choices((2, 3, 4), (10, 25, 65))[0]
    group = rng.choices((64, 128, 256, 512), (20, 50, 15, 15))[0]
    rank = rng.choices((0, 16, 32), (65, 10, 25))[0]
    rotated = rng.random() < 0.2
    M = _log_int(rng, 1, 2048)
    if op == "layers":
        return dict(op=op, M=_log_int(rng, 1, 256), layers=rng.randint(2, 8), dtype=dtype)
    if op == "embed":
        return dict(op=op, M=_log_int(rng, 1, 4096), N=128 * _log_int(rng, 64, VOCAB // 128), K=HIDDEN, bits=bits,
                    dtype=dtype, group=group)
    if op == "head":
        return dict(op="linear", M=_log_int(rng, 1, 16), N=128 * _log_int(rng, 256, VOCAB // 128), K=HIDDEN,
                    dtype=dtype, group=group)
    K = 64 * _log_int(rng, 16, 192)
    if op == "kgrouped":
        return dict(op=op, M=_log_int(rng, 1, 1024), N=128 * _log_int(rng, 8, 96), K=128 * (K // 128), dtype=dtype)
    if op == "qkv":
        c = dict(op=op, K=K, Nq=128 * _log_int(rng, 8, 64), Nk=128 * _log_int(rng, 8, 32), Nv=128 * _log_int(rng, 8, 32))
        per_row = 2.0 * K * (c["Nq"] + c["Nk"] + c["Nv"])
    elif op == "mlp":
        c = dict(op=op, K=K, I=128 * _log_int(rng, 8, 96))
        per_row = 6.0 * K * c["I"]
    else:
        c = dict(op=op, K=K, N=128 * _log_int(rng, 8, 96), bias=rng.random() < 0.2)
        two = rng.random() < 0.2
        c["bits2"] = rng.choice((1, 2, 3, 4)) if two else 0
        c["hadamard"] = 128 if K % 128 == 0 and not rotated and rng.random() < 0.15 else 0
        per_row = 2.0 * K * c["N"] * (2 if two else 1)
    c.update(M=max(1, min(M, int(LARGEST_FLOPS / per_row))), bits=bits, group=group, rank=rank, rotated=rotated,
             dtype=dtype)
    return c


# --------------------------------------------------------------------------- what a program holds

def _linear(c, N, K, seed, rotation_seed=5):
    """One palettized projection on the device, as the loader leaves it."""
    dt = DTYPES[c["dtype"]]
    groups = -(-N // c["group"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    kw = {}
    if c["bits2"]:
        kw.update(indices2=pkg.synthetic.random_blob_on_device(N, K, c["bits2"], seed + 1, "cuda"),
                  lut2=pkg.synthetic.make_lut(groups, c["bits2"], dt, seed + 1, std=0.005).cuda(), bitwidth2=c["bits2"])
    if c["rank"]:
        kw.update(resA=(0.05 * torch.randn(N, c["rank"], device="cuda", generator=g)).to(dt),
                  resB=(0.05 * torch.randn(c["rank"], K, device="cuda", generator=g)).to(dt))
    if c["rotated"]:
        kw.update(rotation_seed=rotation_seed, rotation_k=K)
    if c["bias"]:
        kw["bias"] = (0.1 * torch.randn(N, device="cuda", generator=g)).to(dt)
    blob = pkg.synthetic.random_blob_on_device(N, K, c["bits"], seed, "cuda")
    lut = pkg.synthetic.make_lut(groups, c["bits"], dt, seed).cuda()
    return pkg.PalettizedLinear(blob, lut, c["bits"], c["group"], N, K, **kw).cuda()


def _qkv(c, rows, K, seed):
    return pkg.SplitQKV(*(_linear(c, n, K, seed + 10 * i) for i, n in enumerate(rows)))


def _mlp(c, K, I, seed):
    return pkg.FusedPalettizedMLP(_linear(c, I, K, seed), _linear(c, I, K, seed + 10), _linear(c, K, I, seed + 20),
                                  torch.nn.SiLU())


def _decoder_layer(c, i, seed):
    """The palettized modules of decoder layer i: the projections that read the layer's input."""
    if (i + 1) % FULL_ATTENTION_EVERY == 0:
        mods = [_qkv(c, (8192, 1024, 1024), HIDDEN, seed)]
    else:
        mods = [_qkv(c, (2048, 2048, 4096), HIDDEN, seed), _linear(c, 4096, HIDDEN, seed + 30)]
    return mods + [_linear(c, HIDDEN, HIDDEN, seed + 40), _mlp(c, HIDDEN, INTERMEDIATE, seed + 50)]


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    s = 1000 * (seed % 1000003)
    dt, M = DTYPES[c["dtype"]], c["M"]
    g = torch.Generator(device="cuda").manual_seed(s + 7)
    if c["op"] == "embed":
        groups = -(-c["N"] // c["group"])
        blob = pkg.synthetic.random_blob_on_device(c["N"], c["K"], c["bits"], s, "cuda")
        lut = pkg.synthetic.make_lut(groups, c["bits"], dt, s).cuda()
        return dict(mod=pkg.PalettizedEmbedding(blob, lut, c["bits"], c["group"], c["N"], c["K"]).cuda(),
                    x=torch.randint(0, c["N"], (M,), device="cuda", generator=g))
    K = HIDDEN if c["op"] == "layers" else c["K"]
    state = dict(x=torch.randn(M, K, device="cuda", generator=g).to(dt), hadamard=c["hadamard"])
    if c["op"] == "linear":
        state["mod"] = _linear(c, c["N"], K, s)
    elif c["op"] == "qkv":
        state["mod"] = _qkv(c, (c["Nq"], c["Nk"], c["Nv"]), K, s)
    elif c["op"] == "mlp":
        state["mod"] = _mlp(c, K, c["I"], s)
    elif c["op"] == "kgrouped":
        lut_k = (0.02 * torch.randn(K // 128, c["N"], 1 << c["bits"], device="cuda", generator=g)).sort(dim=-1).values
        blob = pkg.synthetic.random_blob_on_device(c["N"], K, c["bits"], s, "cuda")
        state["mod"] = pkg.KGroupedPalettizedLinear(blob, lut_k.to(dt), c["bits"], c["N"], K).cuda()
    else:
        mods = [m for i in range(c["layers"]) for m in _decoder_layer(c, i, s + 100 * i)]
        state.update(mods=mods, x_in=torch.empty_like(state["x"]))
        _capture(state)
    return state


def _capture(state):
    """A server's decode step: one warm-up, then the step's launches in a CUDA graph. Every module
    reads the step's input rows (attention, norms and residual adds are not this package's)."""
    x_in = state["x_in"]
    x_in.copy_(state["x"])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(side):
        for m in state["mods"]:
            m(x_in)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.no_grad(), torch.cuda.graph(graph):
        outs = [m(x_in) for m in state["mods"]]
    state.update(graph=graph, outs=outs)


def run(state):
    if "graph" in state:
        state["x_in"].copy_(state["x"])
        state["graph"].replay()
        return state["outs"]
    x = state["x"]
    with torch.no_grad():
        if state.get("hadamard"):
            x = pkg.fht.fht_block(x, state["hadamard"])
        return state["mod"](x)


# --------------------------------------------------------------------------- what it takes

def _weight_bytes(c, N, K):
    """Codes, palettes, residual factors, bias, rotation signs of one projection."""
    groups = -(-N // c["group"])
    b = N * K * c["bits"] / 8 + groups * (2 << c["bits"]) + 2 * c["rank"] * (N + K) + (2 * N if c["bias"] else 0)
    if c["bits2"]:
        b += N * K * c["bits2"] / 8 + groups * (2 << c["bits2"])
    return b + (4 * K if c["rotated"] else 0)


def _flops(c, N, K, M):
    return 2.0 * M * N * K * (2 if c["bits2"] else 1) + 2.0 * M * c["rank"] * (N + K)


def work(case):
    """Each code, palette, activation and result moved once; two operations per weight and row
    (per stream, as the streams' sums are added in fp32)."""
    c = dict(DEFAULTS, **case)
    M = c["M"]
    if c["op"] == "embed":
        return dict(bytes=M * (8 + c["K"] * c["bits"] / 8 + (2 << c["bits"]) + 2 * c["K"]), flops=0)
    if c["op"] == "kgrouped":
        N, K = c["N"], c["K"]
        return dict(bytes=N * K * c["bits"] / 8 + (K // 128) * N * (2 << c["bits"]) + 2 * M * (N + K), flops=2.0 * M * N * K)
    if c["op"] == "layers":
        total = dict(bytes=2.0 * M * HIDDEN, flops=0.0)
        for i in range(c["layers"]):
            full = (i + 1) % FULL_ATTENTION_EVERY == 0
            heads = (8192, 1024, 1024) if full else (2048, 2048, 4096, 4096)
            shapes = [(n, HIDDEN) for n in heads + (HIDDEN, INTERMEDIATE, INTERMEDIATE)] + [(HIDDEN, INTERMEDIATE)]
            for N, K in shapes:
                total["bytes"] += _weight_bytes(c, N, K)
                total["flops"] += _flops(c, N, K, M)
            total["bytes"] += 2.0 * M * (sum(heads) + 2 * HIDDEN)
        return total
    K = c["K"]
    if c["op"] == "mlp":
        shapes, out = [(c["I"], K), (c["I"], K), (K, c["I"])], K
    elif c["op"] == "qkv":
        shapes = [(c["Nq"], K), (c["Nk"], K), (c["Nv"], K)]
        out = c["Nq"] + c["Nk"] + c["Nv"]
    else:
        shapes, out = [(c["N"], K)], c["N"]
    return dict(bytes=sum(_weight_bytes(c, n, k) for n, k in shapes) + 2.0 * M * (K + out),
                flops=sum(_flops(c, n, k, M) for n, k in shapes))


def tolerance(case):
    """A gather returns palette entries as they are. Everything else sums in fp32 and rounds its
    results, and a few intermediate values (the gated product, the transformed input, the residual's
    first factor), to the 16-bit operand type: 2^-9 per bf16 rounding, 2^-12 per fp16 rounding."""
    if case["op"] == "embed":
        return "exact"
    return {"rel": 1e-2 if case.get("dtype", "bf16") == "bf16" else 2e-3}
