"""The native host layer (csrc/host) against the Python route it stands in for: the same launches,
so the same bits, over the row counts where the route changes (decode, tensor-core GEMM) and the
options it carries; and what makes it let go of a module (replaced palette, swapped bias storage,
other dtype or device state), where results have to follow the module."""
from __future__ import annotations

import copy
import random

import pytest
import torch

from helpers import TOL, Case, pkg, rel_err

pytestmark = pytest.mark.gpu

OPTIONS = (dict(), dict(bias=True, residual=16), dict(rotation_seed=3), dict(rotation_seed=3, residual=8, awq=True),
           dict(bits2=2, bias=True), dict(bits2=4))


@pytest.mark.parametrize("opts", range(len(OPTIONS)))
@pytest.mark.parametrize("M", (1, 8, 9, 16, 17, 130))
def test_linear_equals_the_python_route(M, opts):
    case = Case(256, 192, 64, 4, torch.float16, seed=70 + opts, **OPTIONS[opts])
    mod = case.module()
    x = case.x(M).cuda()
    want = mod._forward_route(x)
    mod(x)
    assert mod._native is not None
    got = pkg._lib.host.linear(mod.__dict__, x, True)
    if got is not None:                     # None: this row count needs the Python route
        assert torch.equal(got, want)
    assert torch.equal(mod(x.view(1, M, 192)).view(M, -1), want)
    assert rel_err(want, case.oracle(case.x(M))) <= TOL


@pytest.mark.parametrize("M", (1, 8, 16, 40))
@pytest.mark.parametrize("opts", (0, 1, 2))
def test_merged_modules_equal_the_python_route(M, opts):
    K = 256
    mk = lambda n, k, s: Case(n, k, 128, 4, torch.bfloat16, seed=s, **OPTIONS[opts]).module()     # noqa: E731
    qkv = pkg.SplitQKV(mk(256, K, 1), mk(128, K, 2), mk(128, K, 3))
    mlp = pkg.FusedPalettizedMLP(mk(384, K, 4), mk(384, K, 5), mk(K, 384, 6), torch.nn.SiLU())
    x = torch.randn(M, K, device="cuda").bfloat16()
    for mod in (qkv, mlp):
        want = mod._forward_route(x)
        mod(x)
        assert torch.equal(mod(x), want)
        host = pkg._lib.host.qkv if mod is qkv else pkg._lib.host.mlp
        assert torch.equal(host(mod.__dict__, x, True), want)


def test_a_changed_module_is_described_anew():
    case = Case(256, 128, 128, 4, torch.bfloat16, seed=9, bias=True)
    mod = case.module()
    x = case.x(3).cuda()
    first = mod(x)
    assert torch.equal(mod(x), first)
    mod.lut = (2 * mod.lut.float()).bfloat16()
    assert pkg._lib.host.linear(mod.__dict__, x, True) is None
    assert torch.equal(mod(x), mod._forward_route(x)) and not torch.equal(mod(x), first)
    mod.bias.data = torch.zeros_like(mod.bias.data)
    assert torch.equal(mod(x), mod._forward_route(x))
    other = copy.deepcopy(mod)
    assert torch.equal(other(x), mod(x))
    mod.reference = True
    assert rel_err(mod(x), mod._forward_route(x)) == 0.0 and pkg._lib.host.linear(mod.__dict__, x, True) is None
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
        assert torch.equal(other(x), other._forward_route(x))
        torch.cuda.current_stream().synchronize()
    with pytest.raises(ValueError, match="feature dim"):
        other(x[:, :64])


def test_scratch_of_a_captured_graph_is_its_own():
    case = Case(1024, 512, 128, 4, torch.bfloat16, seed=12)
    mod = case.module()
    x = case.x(64).cuda()
    want = mod(x)
    graphs, outs = [], []
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(mod(x))
        graphs.append(g)
    for g, o in zip(graphs * 2, outs * 2):
        g.replay()
        assert torch.equal(mod(x), want)
        torch.cuda.synchronize()
        assert torch.equal(o, want)


class _Doubled(pkg.PalettizedLinear):
    def forward(self, x):
        return 2 * super().forward(x)


def _double_forward(m):
    plain = m.forward
    m.forward = lambda x: 2 * plain(x)


@pytest.mark.parametrize("attach", (
    lambda m: m.register_forward_hook(lambda mod, args, out: 2 * out),
    lambda m: m.register_forward_pre_hook(lambda mod, args: (2 * args[0],)),
    lambda m: torch.nn.modules.module.register_module_forward_hook(lambda mod, args, out: 2 * out if mod is m else None),
    _double_forward,
    lambda m: setattr(m, "__class__", _Doubled),
), ids=("hook", "pre_hook", "global_hook", "instance_forward", "subclass"))
@pytest.mark.parametrize("M", (1, 16, 40))
def test_what_is_attached_to_the_down_projection_runs_in_every_call(M, attach):
    K, inner = 256, 384
    mk = lambda n, k, s: Case(n, k, 128, 4, torch.bfloat16, seed=s).module()     # noqa: E731
    mlp = pkg.FusedPalettizedMLP(mk(inner, K, 4), mk(inner, K, 5), mk(K, inner, 6), torch.nn.SiLU())
    x = torch.randn(M, K, device="cuda").bfloat16()
    want = 2 * mlp(x)                                   # exact: a power of two
    mlp(x)
    handle = attach(mlp.down_proj)
    try:
        for _ in range(3):
            assert torch.equal(mlp(x), want)
    finally:
        if hasattr(handle, "remove"):
            handle.remove()


def _merged_with_residuals(K=256, inner=384):
    mk = lambda n, k, s, r: Case(n, k, 128, 4, torch.float16, seed=s, residual=r).module()     # noqa: E731
    return (pkg.SplitQKV(mk(256, K, 1, 16), mk(128, K, 2, 0), mk(128, K, 3, 8)),
            pkg.FusedPalettizedMLP(mk(inner, K, 4, 8), mk(inner, K, 5, 24), mk(K, inner, 6, 16), torch.nn.SiLU()))


@pytest.mark.parametrize("which", (0, 1), ids=("qkv", "mlp"))
@pytest.mark.parametrize("warm_up_rows", (4, 40))          # 40: the decode step's first call is the captured one
def test_residuals_of_graphs_and_eager_calls_do_not_depend_on_a_replay(which, warm_up_rows):
    mod = _merged_with_residuals()[which]
    xs = [torch.randn(m, 256, device="cuda").half() for m in (2, 3)]
    wants = [_merged_with_residuals()[which](x) for x in xs]
    mod(torch.randn(warm_up_rows, 256, device="cuda").half())
    torch.cuda.synchronize()
    graphs, outs = [], []
    for x in xs:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(mod(x))
        graphs.append(g)
    for _ in range(2):                                      # eager calls before any replay
        assert all(torch.equal(mod(x), w) for x, w in zip(xs, wants))
    for i in (1, 0, 1):                                     # the second graph first
        graphs[i].replay()
        torch.cuda.synchronize()
        assert torch.equal(outs[i], wants[i])
    assert all(torch.equal(mod(x), w) for x, w in zip(xs, wants))


@pytest.mark.parametrize("which", (0, 1), ids=("qkv", "mlp"))
def test_a_residual_factor_written_in_place_is_followed(which):
    mod = _merged_with_residuals()[which]
    x = torch.randn(3, 256, device="cuda").half()
    mod(x), mod(x)
    first = mod.q_proj if which == 0 else mod.gate_proj
    other = _merged_with_residuals()[which]
    for m in (first, other.q_proj if which == 0 else other.gate_proj):
        m.resB.mul_(-3)
    want = other(x)                                         # stacked after the change
    assert torch.equal(mod(x), want) and torch.equal(mod._forward_route(x), want) and torch.equal(mod(x), want)


@pytest.mark.parametrize("value,off", ((" 1 ", True), ("true", True), ("True\n", True), ("TRUE", False), ("10", False), ("", False)))
def test_the_merge_switch_reads_as_in_the_python_route(value, off, monkeypatch):
    mk = lambda n, s: Case(n, 256, 128, 4, torch.bfloat16, seed=s).module()     # noqa: E731
    qkv = pkg.SplitQKV(mk(256, 1), mk(128, 2), mk(128, 3))
    x = torch.randn(4, 256, device="cuda").bfloat16()
    qkv(x), qkv(x)
    monkeypatch.setenv("FLUTE_NO_MERGE", value)
    assert (pkg._lib.host.qkv(qkv.__dict__, x, True) is None) == off


def test_a_tensor_changed_in_place_is_described_anew():
    case = Case(256, 128, 128, 4, torch.float16, seed=31, residual=128)     # a square second factor
    mod = case.module()
    x = case.x(3).cuda()
    mod(x), mod(x)
    mod.resB.t_()                                           # same object, same storage, other strides
    case.resB = case.resB.t().contiguous()
    assert rel_err(mod(x), case.oracle(case.x(3))) <= TOL


def test_a_tied_table_follows_the_codes_of_its_head():
    head, other = (Case(256, 128, 128, 4, torch.bfloat16, seed=s) for s in (32, 33))
    lm = head.module()
    emb = pkg.PalettizedEmbedding.tied_to(lm).cuda()
    ids = torch.arange(256, device="cuda")
    emb(ids), emb(ids)
    lm.indices, lm._packed = other.blob.cuda(), None        # new codes under the same palettes
    want = other.codes.astype("int64")
    pal = head.lut.float()[torch.arange(256) // 128]
    assert torch.equal(emb(ids).float().cpu(), pal.gather(1, torch.from_numpy(want)))


def test_other_python_threads_run_while_a_launch_waits_for_room_in_the_queue():
    # the device sleeps for a quarter of a second; the launches behind it fill the stream's queue and block
    import threading
    import time
    case = Case(128, 128, 128, 4, torch.bfloat16, seed=41)
    mod = case.module()
    x = case.x(1).cuda()
    mod(x), mod(x)
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
    t = threading.Thread(target=tick)
    t.start()
    t0 = time.perf_counter()
    torch.cuda._sleep(500_000_000)
    for _ in range(8000):
        mod(x)
    blocked = time.perf_counter() - t0
    stop.set()
    t.join()
    torch.cuda.synchronize()
    assert blocked > 0.1, "the queue never filled"
    assert max(gaps) < 0.08


def test_threads_of_one_stream_do_not_mix_their_two_stream_launches():
    import threading
    mods = [Case(256, 256, 128, 4, torch.float16, seed=s, bits2=2).module() for s in (51, 52)]
    x = torch.randn(40, 256, device="cuda").half()
    wants = [m(x) for m in mods]
    assert all(pkg._lib.host.linear(m.__dict__, x, True) is not None for m in mods)
    torch.cuda.synchronize()
    bad = []

    def work(i):
        outs = [mods[i](x) for _ in range(1500)]
        torch.cuda.synchronize()
        bad.append(sum(not torch.equal(o, wants[i]) for o in outs))
    threads = [threading.Thread(target=work, args=(i % 2,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert bad == [0] * 4


@pytest.mark.parametrize("opts", range(len(OPTIONS)))
@pytest.mark.parametrize("M", (1, 8, 9, 16, 17, 130))
def test_the_native_route_serves_every_option(M, opts):
    case = Case(256, 192, 64, 4, torch.float16, seed=70 + opts, **OPTIONS[opts])
    mod = case.module()
    x = case.x(M).cuda()
    mod(x)
    got = pkg._lib.host.linear(mod.__dict__, x, True)
    assert got is not None and torch.equal(got, mod._forward_route(x))


@pytest.mark.parametrize("seed", range(24))
def test_rules_of_the_two_routes_agree(seed):
    # the same C entries, so the same bits, wherever the native layer does not leave the call alone
    rng = random.Random(seed)
    bits, gs, dt = rng.choice((1, 2, 3, 4)), rng.choice((32, 64, 128, 256)), rng.choice((torch.float16, torch.bfloat16))
    K = 64 * rng.randint(1, 9)
    opts = dict(bias=rng.random() < 0.5, residual=rng.choice((0, 0, 8, 12, 72)), bits2=rng.choice((None, None, 1, 2, 3, 4)))
    if rng.random() < 0.4:
        opts.update(rotation_seed=rng.randint(0, 99), awq=rng.random() < 0.5)
    a, b = (Case(256, K, gs, bits, dt, seed=2 * seed + i, **opts) for i in range(2))
    qkv = pkg.SplitQKV(a.module(), b.module(), b.module())
    mlp = pkg.FusedPalettizedMLP(a.module(), b.module(), Case(128, 256, gs, bits, dt, seed=seed, **opts).module(),
                                 torch.nn.SiLU())
    for M in (1, 3, 8, 9, 16, 17, 33, 130):
        x = (0.5 * torch.randn(M, K, generator=torch.Generator().manual_seed(M))).to(dt).cuda()
        for mod in (qkv.q_proj, qkv, mlp):
            want = mod._forward_route(x)
            mod(x)
            assert torch.equal(mod(x), want), (M, type(mod).__name__)


@pytest.mark.parametrize("kind", ("kgrouped", "two_stream"))
def test_scratch_of_captured_graphs_and_of_many_streams(kind):
    # two graphs of their own capture and eager calls between their replays; then more streams than the
    # pool keeps buffers for, each used again after its buffer may have gone
    N, K, M, dt = 512, 1024, 300, torch.float16
    if kind == "kgrouped":
        assert pkg._lib.lib().b200lut_gemm_workspace_bytes(M, N, K) > 0
        lut_k = (0.02 * torch.randn(K // 128, N, 16, generator=torch.Generator().manual_seed(1))).to(dt)
        blob = torch.randint(0, 256, (N * K // 2,), dtype=torch.uint8, generator=torch.Generator().manual_seed(2))
        mod = pkg.KGroupedPalettizedLinear(blob, lut_k, 4, N, K).cuda()
    else:
        mod = Case(N, K, 128, 4, dt, seed=61, bits2=2).module()
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(3)).to(dt).cuda()
    mod(x)
    want = mod(x)
    graphs, outs = [], []
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(mod(x))
        graphs.append(g)
    for g, o in zip(graphs * 2, outs * 2):
        g.replay()
        assert torch.equal(mod(x), want)
        torch.cuda.synchronize()
        assert torch.equal(o, want)
    streams = [torch.cuda.Stream() for _ in range(40)]
    for _ in range(2):
        got = []
        for s in streams:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(mod(x))
        torch.cuda.synchronize()
        assert all(torch.equal(g, want) for g in got)
