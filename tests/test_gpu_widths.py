"""Channel widths and row counts at which the conv kernels change form: rows that end in a half chunk of 32 channels, and accumulator
widths that are no power of two.

Bounds.  Inputs are rounded to the storage type, the oracle sums in fp32 (tap by tap, channel by channel).  A result of K = 27 Ci
products with |y| about 1 carries at most half a rounding step of the storage type from its own rounding and as much from
the oracle's, plus K * 2^-24 * sum|x w| from either order of summation (fp32 legs: that alone)."""
import numpy as np
import pytest
import torch

import oracle
from trellis2_cuda_b200 import scenes

pytestmark = pytest.mark.gpu
TD = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
STEP = {"f16": 2.0 ** -10, "bf16": 2.0 ** -7, "f32": 2.0 ** -23}


@pytest.fixture(scope="module")
def sp():
    import trellis2_cuda_b200 as m
    m.context()
    return m


def scene(n, Ci, Co, dt, seed=0, slots=1):
    rng = np.random.default_rng([n, Ci, Co, seed])
    res = max(4, int(round((n / 0.3) ** (1 / 3))))
    cells = rng.choice(res ** 3, size=n, replace=False)
    c = np.stack([np.zeros_like(cells), cells // (res * res), cells // res % res, cells % res], 1).astype(np.int32)
    x = oracle.round_to(rng.standard_normal((n, Ci), dtype=np.float32), dt)
    w = oracle.round_to(scenes.kaiming_uniform_weight(slots * Co, Ci, seed), dt)
    b = oracle.round_to(0.1 * rng.standard_normal(slots * Co).astype(np.float32), dt)
    return c, x, w, b


def check(y, want, Ci, dt, what, steps=1.0, bias=None):
    """`bias` [columns]: the sum was rounded once before the bias went in, at a size of up to |want| + |bias|."""
    got, want = y.float().cpu().numpy().astype(np.float64), np.asarray(want, np.float64)
    most = np.maximum(np.abs(want), np.abs(got)) + (0 if bias is None else np.abs(bias))
    size = 2.0 ** np.floor(np.log2(np.maximum(most, 2.0 ** -6)))
    order = 27 * Ci * 2.0 ** -24 * 8.0                 # sum |x w| stays below 8 for Kaiming weights and unit features
    allow = order + (0 if dt == "f32" else steps * STEP[dt] * size)
    bad = np.abs(got - want) > allow
    assert np.isfinite(got).all() and not bad.any(), f"{what}: {bad.sum()} of {bad.size}, worst {np.abs(got - want).max():.3e}"


@pytest.mark.parametrize("dt,n,Ci,Co", [("bf16", 700, 32, 32), ("f16", 129, 96, 160), ("bf16", 1000, 160, 96), ("f16", 385, 224, 224), ("bf16", 640, 32, 256),
                                        ("bf16", 300, 64, 192), ("f16", 257, 288, 320)])
def test_half_chunks_and_accumulator_widths(sp, dt, n, Ci, Co):
    c, x, w, b = scene(n, Ci, Co, dt)
    nbr, _, _, _ = oracle.build_neighbors(c)
    want = oracle.conv_block(x, w, b, nbr, dt)
    xd, wd, bd = (torch.from_numpy(t).cuda().to(TD[dt]) for t in (x, w, b))
    for tile_rows in (128, 256):
        cache = sp.build_neighbors(torch.from_numpy(c).cuda(), tile_rows=tile_rows)
        y = sp.subm_conv(xd, wd, bd, cache)
        sp.context().device_status()
        check(y, want, Ci, dt, f"{dt} {n} {Ci}->{Co} tile {tile_rows}", steps=2.0, bias=b)     # conv and bias are rounded one after the other


def test_subdivision_conv_with_half_chunks(sp):
    """8 weight sets, rows of 96 channels."""
    Ci, Cc, dt = 96, 96, "bf16"
    c, x, w, b = scene(400, Ci, Cc, dt, slots=8)
    sub = np.random.default_rng(3).standard_normal((400, 8)).astype(np.float16)
    parent = sp.build_neighbors(torch.from_numpy(c).cuda())
    level = sp.subdivide(parent, torch.from_numpy(sub).cuda())
    y = sp.subdiv_conv(*(torch.from_numpy(t).cuda().to(TD[dt]) for t in (x, w, b)), level)
    nbr, _, _, _ = oracle.build_neighbors(c)
    full = oracle.conv_block(x, w, b, nbr, dt).reshape(400 * 8, Cc)
    src = level.src.cpu().numpy()
    check(y, full[src], Ci, dt, "subdivision", steps=2.0, bias=b.reshape(8, Cc)[src % 8])


@pytest.mark.parametrize("n,Ci,Co", [(1, 32, 64), (63, 32, 64), (64, 64, 10), (65, 64, 64), (300, 32, 130), (2500, 64, 64), (9000, 32, 64), (29000, 32, 32)])
def test_fp32_splits(sp, n, Ci, Co):
    """The fp32 kernel splits a tile's taps over clusters of 1, 2, 4 and 8 CTAs by the number of tiles."""
    c, x, w, b = scene(n, Ci, Co, "f32")
    nbr, _, _, _ = oracle.build_neighbors(c)
    res = np.random.default_rng(1).standard_normal((n, Co), dtype=np.float32)
    want = oracle.conv_block(x, w, b, nbr, "f32", act_kind="silu", residual=res)
    for tile_rows in (128, 256):
        cache = sp.build_neighbors(torch.from_numpy(c).cuda(), tile_rows=tile_rows)
        args = [torch.from_numpy(t).cuda() for t in (x, w, b)]
        y = sp.subm_conv(*args, cache, act="silu", residual=torch.from_numpy(res).cuda())
        sp.context().device_status()
        check(y, want, Ci, "f32", f"f32 {n} {Ci}->{Co} tile {tile_rows}")
        assert torch.equal(y, sp.subm_conv(*args, cache, act="silu", residual=torch.from_numpy(res).cuda()))     # ranks add in a fixed order


@pytest.mark.parametrize("dt", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("n,C", [(1, 8), (10007, 32), (19001, 40), (10007, 64), (33, 72), (10007, 128), (777, 136), (5003, 256), (1000, 264), (601, 1024), (301, 1032)])
def test_row_pass_over_its_lane_groups(sp, dt, n, C):
    """Rows of 4, 8, 16 and 32 lanes, partly filled ones, and more rows than one sweep of the grid.  Against 64 bits with the pass's
    rounding points: LayerNorm, activation and residual each round once, a flipped rounding of one moves the next by as
    much again; fp32 adds the sums over C."""
    g = torch.Generator(device="cuda").manual_seed(n + C)
    x, r = (torch.randn((n, C), generator=g, device="cuda").to(TD[dt]) for _ in range(2))
    gamma, beta = torch.rand(C, generator=g, device="cuda") + 0.5, torch.randn(C, generator=g, device="cuda")
    y = sp.row_epilogue(x, ln=(gamma, beta, 1e-6), act="silu", residual=r)
    v = torch.nn.functional.layer_norm(x.double(), (C,), eps=1e-6) * gamma.double()
    h = torch.nn.functional.silu((v + beta.double()).to(TD[dt]).double()).to(TD[dt]).double()
    want = h + r.double()
    size = v.abs() + beta.double().abs() + want.abs() + r.double().abs()        # the terms of every sum along the way
    assert ((y.double() - want).abs() <= (4 if dt != "f32" else 16) * STEP[dt] * (size + 2.0 ** -6)).all()
    assert torch.equal(sp.row_epilogue(x, ln=(gamma, beta, 1e-6), act="silu", residual=r, out=x), y)        # in place


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("act", ["silu", "gelu", "gelu_tanh"])
def test_row_pass_gives_the_same_bits_at_any_alignment(sp, dt, act):
    """A tensor that starts in the middle of 16 bytes takes the element-by-element kernel.  The values reach past the point where
    exp(-x) leaves fp32's normal range."""
    n, C = 501, 64
    x = torch.linspace(-100, 100, n * C, device="cuda").to(TD[dt]).view(n, C)
    shifted = torch.empty(n * C + 1, dtype=TD[dt], device="cuda")[1:].view(n, C).copy_(x)
    assert torch.equal(sp.row_epilogue(x, act=act), sp.row_epilogue(shifted, act=act))


@pytest.mark.parametrize("C", [8, 40, 128, 256, 264, 1024, 2048])
def test_row_pass_adds_up_a_row_in_one_order(sp, C):
    """A lane adds its 8-channel pieces in order, the lanes meet in a butterfly: the same sums in fp32, operation by operation
    (a product and an addition that round once go through 64 bits, where the product is exact)."""
    x = torch.randn((501, C), generator=torch.Generator(device="cuda").manual_seed(C), device="cuda") + 3
    pieces = torch.zeros((501, -(-C // 256) * 32, 8), device="cuda")
    pieces.view(501, -1)[:, :C] = x
    have = torch.arange(pieces.shape[1], device="cuda") * 8 < C

    def total(term):
        s = torch.zeros((501, 32), device="cuda")
        for k in range(pieces.shape[1] // 32):
            for i in range(8):
                s = torch.where(have[32 * k:32 * k + 32], term(s, pieces[:, 32 * k:32 * k + 32, i]), s)
        for o in (16, 8, 4, 2, 1):
            s = s + s[:, torch.arange(32, device="cuda") ^ o]
        return s[:, :1]
    width = torch.full((1, 1), float(C), device="cuda")           # (dividing by a Python number multiplies by its reciprocal)
    mean = total(lambda s, v: s + v) / width
    var = total(lambda s, v: ((v - mean).double() ** 2 + s.double()).float()) / width
    want = torch.rsqrt(var + 1e-6) * (x - mean)
    assert torch.equal(sp.row_epilogue(x, ln=(None, None, 1e-6)), want)


@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("Co", [96, 160, 192, 224])
def test_layer_norm_over_widths_between_powers_of_two(sp, dt, Co):
    """Two passes over the row, as for any width that the epilogue does not hold: a first value far from the others must not cost the
    variance its bits.  The fused call gives the bits of the conv (the Linear layer) and then the row pass."""
    c, x, w, b = scene(700, 64, Co, dt)
    b[0] = 3000
    xd, wd, bd = (torch.from_numpy(t).cuda().to(TD[dt]) for t in (x, w, b))
    ln = (torch.rand(Co, device="cuda") + 0.5, torch.randn(Co, device="cuda"), 1e-6)
    cache = sp.build_neighbors(torch.from_numpy(c).cuda())
    assert torch.equal(sp.subm_conv(xd, wd, bd, cache, ln=ln, act="silu"), sp.row_epilogue(sp.subm_conv(xd, wd, bd, cache), ln=ln, act="silu"))
    wl = wd[:, 0].contiguous()
    assert torch.equal(sp.linear(xd, wl, bd, ln=ln), sp.row_epilogue(sp.linear(xd, wl, bd), ln=ln))


@pytest.mark.parametrize("Co", [64, 130])
def test_fp32_sums_do_not_depend_on_the_rows_beside_them(sp, Co):
    """The first rows of a map by themselves, at numbers of rows that split the taps over 8, 4 and 1 CTAs: the bits of the whole."""
    n, Ci = 30000, 64
    c, x, w, b = scene(n, Ci, Co, "f32")
    x, w, b = (torch.from_numpy(t).cuda() for t in (x, w, b))
    whole = sp.build_neighbors(torch.from_numpy(c).cuda())
    want = sp.subm_conv(x, w, b, whole)
    for m in (1, 700, 2500, 6000, 9000, 15000, 28000):
        part = sp.cache_from_map(whole.coords[:m], whole.nbr[:m].contiguous(), whole.gray[:m].contiguous())
        assert torch.equal(sp.subm_conv_local(x, w, b, part), want[:m]), m


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a second GPU")
def test_fp32_conv_on_a_device_that_is_not_current(sp):
    """Every launch of the call, the check of the plan's table included, goes to the context's device."""
    c, x, w, b = (torch.from_numpy(t) for t in scene(700, 64, 64, "f32"))
    want = sp.subm_conv(x.cuda(0), w.cuda(0), b.cuda(0), sp.build_neighbors(c.cuda(0)))
    xd, wd, bd, cd = (t.cuda(1) for t in (x, w, b, c))
    torch.cuda.synchronize(1)
    with torch.cuda.device(1):
        cache = sp.build_neighbors(cd)
    assert torch.cuda.current_device() == 0
    y = sp.subm_conv(xd, wd, bd, cache)
    torch.cuda.synchronize(1)
    assert torch.equal(y.cpu(), want.cpu())


@pytest.mark.parametrize("dt,n,Ci,Co", [("bf16", 700, 32, 64), ("f16", 3000, 96, 160), ("bf16", 129, 224, 256), ("f16", 257, 96, 128)])
def test_half_chunks_give_the_same_bits_on_either_schedule(sp, dt, n, Ci, Co):
    """128- and 256-row tiles add up a row's products in one order."""
    c, x, w, b = scene(n, Ci, Co, dt)
    xd, wd, bd = (torch.from_numpy(t).cuda().to(TD[dt]) for t in (x, w, b))
    y = [sp.subm_conv(xd, wd, bd, sp.build_neighbors(torch.from_numpy(c).cuda(), tile_rows=r)) for r in (128, 256)]
    sp.context().device_status()
    assert torch.equal(*y)
