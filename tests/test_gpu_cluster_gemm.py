"""The tensor-core GEMM for batches and short prompts (csrc/gemm_cluster.cu) where it can go wrong: token
counts at the edges of its 16- to 128-token tiles, odd and few k-blocks per CTA, cuts of K over up to eight
CTAs per cluster with one tile each and with several one after the other, two palettes per tile, every code
width, merged projections, residual k-blocks that start in the middle of a stage, unaligned outputs."""
from __future__ import annotations

import pytest
import torch

from helpers import TOL, Case, pkg, rel_err

pytestmark = pytest.mark.gpu
L = pkg._lib


@pytest.fixture(autouse=True)
def _no_device_error():
    yield
    torch.cuda.synchronize()
    assert L.lib().b200lut_device_status() == 0


@pytest.mark.parametrize("N,K,gs,bits,dtype,M,opts", (
    (128, 128, 128, 4, torch.bfloat16, 17, {}),                       # two k-blocks, one tile
    (128, 4160, 128, 4, torch.bfloat16, 33, {}),                      # 65 k-blocks over eight CTAs
    (256, 2112, 64, 4, torch.float16, 128, dict(bias=True)),          # 33 k-blocks, two palettes, a full tile
    (384, 1984, 128, 3, torch.bfloat16, 129, {}),                     # 31 k-blocks, two token tiles
    (640, 1024, 64, 3, torch.float16, 250, dict(bias=True)),
    (256, 1536, 256, 2, torch.bfloat16, 64, {}),
    (512, 320, 512, 1, torch.float16, 65, dict(bias=True)),           # five k-blocks
    (128, 2048, 128, 4, torch.bfloat16, 48, dict(residual=32)),
    (256, 1088, 64, 4, torch.float16, 100, dict(residual=72, bias=True)),   # 17 k-blocks, two residual blocks
    (384, 192, 128, 4, torch.bfloat16, 20, dict(residual=8)),         # the residual opens a stage after three k-blocks
    (19200, 128, 128, 4, torch.bfloat16, 31, {}),                     # 150 row tiles: more than one per CTA
    (1280, 128, 128, 4, torch.float16, 900, {}),                      # 80 tiles of eight token tiles
))
def test_forward_matches_oracle(N, K, gs, bits, dtype, M, opts):
    case = Case(N, K, gs, bits, dtype, seed=N + 3 * K + M, **opts)
    mod = case.module()
    x = case.x(M).cuda()
    got = mod(x)
    assert rel_err(got, case.oracle(case.x(M))) <= TOL
    assert torch.equal(mod(x), got)                                    # ascending-k exchange: deterministic


@pytest.mark.parametrize("M", (24, 127))
def test_cut_and_whole_tiles_agree(M):
    # the same products in fp32, summed in parts: n terms in any order differ by at most n * 2^-24 of the
    # sum of magnitudes, far below one bf16 step; so the two roundings give the same or neighbouring values,
    # and neighbours in bf16 (8 significant bits) lie at most 2^-7 of their size apart
    case = Case(256, 4096, 128, 4, torch.bfloat16, seed=M)
    mod = case.module()
    mod._ensure_packed()
    x = case.x(M).cuda()
    outs = []
    for split in (True, False):
        o = torch.full((M, 256 + 3), float("nan"), dtype=case.dtype, device="cuda")     # odd stride: unaligned rows
        L.gemm(x, L.make_segments([dict(packed=mod._packed, lut=mod.lut, N=256, group_size=128, n_groups=2, bits=4,
                                        out=o, ldo=259)]), split=split)
        assert torch.isnan(o[:, 256:].float()).all()
        outs.append(o[:, :256])
    assert rel_err(outs[0], outs[1].cpu()) <= 2.0 ** -7
    assert rel_err(outs[0], case.oracle(case.x(M))) <= TOL


def test_merged_projections_with_and_without_a_residual():
    K, M, dt = 1344, 40, torch.float16                                 # 21 k-blocks
    cases = [Case(n, K, 128, 4, dt, seed=80 + i, bias=(i == 0), residual=16 * i) for i, n in enumerate((256, 128, 384))]
    qkv = pkg.SplitQKV(*(c.module() for c in cases))
    x = cases[0].x(M)
    want = torch.cat([c.oracle(x) for c in cases], dim=-1)
    assert rel_err(qkv(x.cuda()), want) <= TOL


@pytest.mark.parametrize("N,K,gs,bits,dtype,M,bias", (
    (128, 128, 128, 4, torch.bfloat16, 9, False),                      # the fewest k-blocks
    (256, 4160, 128, 4, torch.float16, 16, True),                      # eight CTAs share four token quads
    (384, 1984, 64, 3, torch.bfloat16, 13, True),
    (128, 832, 256, 2, torch.float16, 12, False),
    (256, 1088, 512, 1, torch.bfloat16, 16, True),
    (19200, 192, 128, 4, torch.bfloat16, 10, False),                   # 150 row tiles
    (128 * 1000, 128, 128, 4, torch.bfloat16, 3, False),               # few rows of many row tiles (not this kernel)
))
def test_batched_decode(N, K, gs, bits, dtype, M, bias):
    case = Case(N, K, gs, bits, dtype, seed=N + K + M, bias=bias)
    x = case.x(M)
    got = case.module()(x.cuda())
    assert rel_err(got, case.oracle(x)) <= TOL


@pytest.mark.parametrize("N,K,gs,bits,dtype,M,aligned", (
    (128, 128, 128, 4, torch.bfloat16, 9, True),
    (256, 4160, 64, 4, torch.float16, 16, False),                      # a cut over eight CTAs, two palettes, odd stride
    (384, 1984, 128, 3, torch.bfloat16, 11, True),
    (19328, 128, 128, 2, torch.float16, 16, True),                     # 151 pairs of tiles
))
def test_batched_gated_pair(N, K, gs, bits, dtype, M, aligned):
    gate, up = (Case(N, K, gs, bits, dtype, seed=7 * N + K + i, bias=(i == 0)) for i in range(2))
    x = gate.x(M)
    mods = [gate.module(), up.module()]
    ld = N if aligned else N + 3
    out = torch.full((M, ld), float("nan"), dtype=dtype, device="cuda")
    descs = []
    for m in mods:
        m._ensure_packed()
        descs.append(dict(packed=m._packed, lut=m.lut, N=N, group_size=gs, n_groups=m.lut.shape[0], bits=bits,
                          bias=m.bias, out=out, ldo=ld))
    L.gemv_multi(x.cuda(), L.make_segments(descs), 2, epilogue=L.EPI_SILU_MUL)
    g, u = (torch.nn.functional.linear(x.double(), c.w1.double(), None if c.bias is None else c.bias.double()) for c in (gate, up))
    want = torch.nn.functional.silu(g) * u                             # fp32 sums, one rounding: 2^-8 of a value in bf16
    assert rel_err(out[:, :N], want.float()) <= 2.0 ** -8
    assert torch.isnan(out[:, N:].float()).all()


@pytest.mark.parametrize("M", (20, 128))
def test_more_row_tiles_than_the_token_tiles_pay_for(M):
    case = Case(128 * 700, 128, 128, 4, torch.bfloat16, seed=M)        # 700 row tiles
    x = case.x(M)
    assert rel_err(case.module()(x.cuda()), case.oracle(x)) <= TOL


def _synthetic(N, K, bits, gs, dtype=torch.float16, seed=0):
    g = torch.Generator().manual_seed(N + K + seed)
    blob = pkg.synthetic.random_blob_on_device(N, K, bits, N + K + seed, "cuda")
    lut = (0.02 * torch.randn(-(-N // gs), 1 << bits, generator=g)).sort(dim=1).values.to(dtype).cuda()
    return pkg.PalettizedLinear(blob, lut, bits, gs, N, K)


@pytest.mark.parametrize("N,K,bits,M,dtype", (                         # on 148 SMs:
    (19200, 4096, 4, 9, torch.bfloat16),                               # cut 2, three tiles per cluster
    (19200, 6144, 3, 16, torch.float16),                               # cut 3, four tiles; one or two token quads per CTA
    (12800, 12288, 4, 17, torch.bfloat16),                             # cut 5, four tiles
    (19200, 12288, 4, 64, torch.bfloat16),                             # cut 6, seven tiles
    (11776, 6144, 2, 128, torch.float16),                              # cut 4, three full tiles
))
def test_cut_tiles_one_after_the_other(N, K, bits, M, dtype):
    # the exchange's barriers change phase with every tile of a cluster, the accumulators with every other one
    mod = _synthetic(N, K, bits, 128, dtype)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(dtype).cuda()
    got = mod(x)
    want = x.double() @ (mod._quantized_weight().double()).t()
    assert rel_err(got, want.float()) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)   # one rounding
    for _ in range(20):
        assert torch.equal(mod(x), got)


@pytest.mark.parametrize("N,M", ((6400, 9), (12800, 16)))
def test_cut_gated_tiles_one_after_the_other(N, M):
    K, dt = 12288, torch.bfloat16                                      # cut 5: four and eight tiles per cluster
    mods = [_synthetic(N, K, 4, 128, dt, seed=i) for i in range(2)]
    x = (0.1 * torch.randn(M, K, generator=torch.Generator().manual_seed(M))).to(dt).cuda()
    out = torch.empty(M, N, dtype=dt, device="cuda")
    segs = L.make_segments([m._segment_desc(out) for m in mods])
    g, u = (x.double() @ m._quantized_weight().double().t() for m in mods)
    for _ in range(20):
        out.fill_(float("nan"))
        L.gemv_multi(x, segs, 2, epilogue=L.EPI_SILU_MUL)
        assert rel_err(out, (torch.nn.functional.silu(g) * u).float()) <= 2.0 ** -8


def _missed(mod, x, **kw):
    """Share of fp16 outputs that are not the rounding of the 64-bit sums (one launch of `mod` over x)."""
    mod._ensure_packed()
    out = torch.empty(x.shape[0], mod.N, dtype=x.dtype, device="cuda")
    seg = L.make_segments([mod._segment_desc(out)])
    L.gemv_multi(x, seg, 1, **kw) if x.shape[0] <= 16 else L.gemm(x, seg, **kw)
    want = x.double() @ mod._quantized_weight().double().t()
    return (out != want.to(x.dtype)).double().mean().item(), out


@pytest.mark.parametrize("N,K,bits,gs,M", (
    (12288, 4096, 3, 64, 16),        # one CTA per tile: eight chains
    (4096, 4096, 4, 128, 9),         # cut tiles
    (4096, 12288, 4, 128, 12),
    (1024, 1024, 2, 128, 16),        # single k-blocks
))
def test_batched_decode_sums_no_less_exactly_than_the_tile_kernel(N, K, bits, gs, M):
    # both truncate at every accumulation of the tensor core and round where chains are added; with chains
    # of equal length the shares are those of two samples of one population, four deviations apart at most
    # (one chain per CTA: 5 to 10 times the tile kernel's share)
    mod = _synthetic(N, K, bits, gs)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).half().cuda()
    here, tile = _missed(mod, x)[0], _missed(mod, x, flags=L.FLAG_TILE_KERNEL)[0]
    assert here <= tile + 4 * (2 * max(tile, 1 / (M * N)) / (M * N)) ** 0.5


@pytest.mark.parametrize("N,K,bits,gs,M", ((4096, 4096, 4, 128, 64), (4096, 4096, 4, 128, 128), (1024, 1024, 2, 128, 700)))
def test_short_prompts_sum_in_chains_of_a_quarter_of_k(N, K, bits, gs, M):
    # the whole-tile kernel's split schedule cuts these tiles into four parts or more: a quarter of the
    # truncations behind one another; the fp32 additions of the parts round (2^-24 of the value each, 2^-13
    # of fp16's spacing, a few of them on partial sums up to a few times the result: 1.5e-3 at most)
    mod = _synthetic(N, K, bits, gs)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).half().cuda()
    assert _missed(mod, x)[0] <= _missed(mod, x, split=False)[0] / 4 + 1.5e-3


@pytest.mark.parametrize("M", (3, 8))
def test_a_head_of_few_rows_has_the_bits_of_the_row_range_kernel(M):
    mod = _synthetic(128 * 1000, 128, 4, 128)
    x = torch.randn(M, 128, generator=torch.Generator().manual_seed(M)).half().cuda()
    assert torch.equal(_missed(mod, x)[1], _missed(mod, x, flags=L.FLAG_ROWS_KERNEL)[1])


def test_a_launch_behind_a_long_exchange_wait_does_not_give_up():
    # the exchange waits 60 ms for rows that nobody pushes (it reports that, and ends); the launch behind it
    # starts early on the SMs that are free, and its own waits are bounded by 10 ms
    from importlib import import_module
    exchange = import_module(pkg.__name__ + ".exchange")
    M, dt = 16, torch.bfloat16
    arena = exchange.PeerArena.emulated(1 << 16, 2, "cuda")[0]
    cons = _synthetic(128, 256, 4, 128, dt)
    mod = _synthetic(4096, 1024, 4, 128, dt)
    for m in (cons, mod):
        m._ensure_packed()
    x = torch.randn(M, 1024, generator=torch.Generator().manual_seed(1)).to(dt).cuda()
    y, out, want = (torch.zeros(M, n, dtype=dt, device="cuda") for n in (128, 4096, 4096))
    L.gemv_multi(x, L.make_segments([mod._segment_desc(want)]), 1)
    torch.cuda.synchronize()
    blocks = L.gemv_launch_blocks(M, 256, L.make_segments([cons._segment_desc(None)]), 1)
    chan = exchange.Channel(arena, M, 256, dt, blocks)
    chan.wait.wait_ms = 60
    L.gemv_exchange(chan.act, L.make_segments([cons._segment_desc(y)]), 1, chan.wait)
    L.gemv_multi(x, L.make_segments([mod._segment_desc(out)]), 1, flags=L.FLAG_PDL)
    torch.cuda.synchronize()
    assert L.lib().b200lut_device_status() in (0x7000, 0x7001)        # the exchange's, not a pipeline wait's
    assert torch.equal(out, want)
