"""A subdivided level's map read off its parents' against the hashed one, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from trellis2_cuda_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sp():
    import trellis2_cuda_b200 as m
    m.context()
    return m


def cube(n, res, seed, origin=0, batches=2):
    rng = np.random.default_rng([n, res, seed])
    cells = rng.choice(batches * res ** 3, size=n, replace=False)
    b, r = np.divmod(cells, res ** 3)
    return np.stack([b, r // (res * res) + origin, r // res % res + origin, r % res + origin], 1).astype(np.int32)


@pytest.mark.parametrize("name,coords,extent,derived", [
    ("one parent", cube(1, 1, 0), 4096, True), ("33 parents", cube(33, 4, 1), 4096, True), ("dense", cube(900, 8, 2), 8, True),
    ("odd grid", cube(700, 9, 3), 9, True), ("at the end of the grid", cube(500, 8, 4, origin=2040), 4096, True),
    ("children outside the grid", cube(500, 8, 5, origin=2044), 4096, False), ("parents outside their map's grid", cube(500, 8, 6), 7, False),
    ("two parents at one place", np.concatenate([cube(300, 8, 7), cube(300, 8, 7)[5:9]]), 4096, False)])
def test_child_map_from_the_parents(sp, name, coords, extent, derived):
    n = len(coords)
    sub = np.random.default_rng(n).standard_normal((n, 8)).astype(np.float16)
    sub[n // 2] = -1
    sub[0] = 1
    d = torch.from_numpy(coords).cuda()
    parent, flags, launches = sp.build_neighbors(d, extent, extent, extent), torch.from_numpy(sub).cuda(), sp.context().launch_count()
    lv = sp.subdivide(parent, flags)
    assert sp.context().launch_count() - launches == (3 if derived else 4), name          # count, emit, and one kernel for the map or two for the hash
    cc, src = oracle.subdivide(coords, sub.astype(np.float32) > 0)
    assert np.array_equal(lv.coords.cpu().numpy(), cc) and np.array_equal(lv.src.cpu().numpy(), src), name
    want = sp.build_neighbors(lv.coords, want_sorted=False)
    assert torch.equal(lv.nb.nbr, want.nbr) and torch.equal(lv.nb.gray, want.gray), name
    if derived:
        nbr, gray, _, _ = oracle.build_neighbors(cc)
        assert np.array_equal(lv.nb.nbr.cpu().numpy().view(np.uint32), nbr) and np.array_equal(lv.nb.gray.cpu().numpy(), gray), name


def test_child_map_follows_what_the_caller_changed(sp):
    c = torch.from_numpy(cube(400, 8, 9)).cuda()
    sub = torch.ones((400, 8), dtype=torch.uint8, device="cuda")
    parent = sp.build_neighbors(c)
    parent.nbr.fill_(-1)                      # the map is not what it was built as: the children's comes from their coordinates
    lv = sp.subdivide(parent, sub)
    assert torch.equal(lv.nb.nbr, sp.build_neighbors(lv.coords).nbr)
    with torch.inference_mode():
        lv = sp.subdivide(sp.build_neighbors(c), sub)
        assert torch.equal(lv.nb.nbr, sp.build_neighbors(lv.coords).nbr)


@pytest.mark.parametrize("n,Ci,dt", [(1, 64, torch.float16), (129, 128, torch.bfloat16), (1500, 192, torch.float16)])
def test_subdivision_conv_over_the_parents_tiles(sp, n, Ci, dt):
    """Every slot of every parent, kept children stored, against the children's own tiles: the same products in the same order."""
    g = torch.Generator(device="cuda").manual_seed(n)
    coords = torch.from_numpy(cube(n, max(2, round((n / 1.2) ** (1 / 3))), 1)).cuda()
    sub = (torch.rand((n, 8), generator=g, device="cuda") < 0.6).to(torch.uint8)
    sub[0] = 1
    if n > 8:
        sub[5] = 0
    x = torch.randn((n, Ci), generator=g, device="cuda").to(dt)
    w = (torch.randn((8 * 64, 27, Ci), generator=g, device="cuda") * 0.03).to(dt)
    b = torch.randn(8 * 64, generator=g, device="cuda").to(dt)
    gamma, beta = torch.rand(64, generator=g, device="cuda") + 0.5, torch.randn(64, generator=g, device="cuda")
    level = sp.subdivide(sp.build_neighbors(coords), sub)
    assert level._from_parents(x, 64)
    for kw in (dict(), dict(ln=(None, None, 1e-6), act="silu"), dict(ln=(gamma, beta, 1e-6), act="gelu")):
        for bias in (b, None):
            assert torch.equal(sp.subdiv_conv(x, w, bias, level, **kw), sp.subdiv_conv(x, w, bias, level, variant="umma", **kw)), kw
    sp.context().device_status()
    level.src = level.src.clone()             # no longer the list its parents' children were counted for
    assert not level._from_parents(x, 64)


@pytest.mark.parametrize("Cin,Co,n", [(128, 64, 700), (512, 256, 300), (2048, 1024, 200), (256, 32, 700), (128, 128, 700), (64, 32, 333), (128, 32, 500)])
def test_fused_skip_is_conv_then_add(sp, Cin, Co, n):
    """rep = 4 in one load per block (8 or 16 bytes apart), other factors element by element, in the conv's epilogue and in the row pass: the
    bits of the conv followed by add_skip."""
    rep = Co // (Cin // 8)
    g = torch.Generator(device="cuda").manual_seed(Cin + Co)
    cache = sp.build_neighbors(torch.from_numpy(cube(n, 8, 4)).cuda())
    x, parent = (torch.randn((m, c), generator=g, device="cuda").to(torch.bfloat16) for m, c in ((n, 64), (40, Cin)))
    src = torch.randint(0, 40 * 8, (n,), generator=g, device="cuda", dtype=torch.int32)
    w = (torch.randn((Co, 27, 64), generator=g, device="cuda") * 0.03).to(torch.bfloat16)
    for kw in (dict(), dict(ln=(None, None, 1e-6))):
        assert torch.equal(sp.subm_conv(x, w, None, cache, skip=(parent, src, rep), **kw), sp.add_skip(sp.subm_conv(x, w, None, cache, **kw), parent, src, rep))


def test_two_sm_variant_of_the_subdivision_conv(sp):
    """It takes 256-row tiles, which the other variants of a subdivided level do not: the same bits from either."""
    g = torch.Generator(device="cuda").manual_seed(3)
    n, Ci, Cc = 700, 128, 256
    level = sp.subdivide(sp.build_neighbors(torch.from_numpy(cube(n, 8, 5)).cuda()), (torch.rand((n, 8), generator=g, device="cuda") < 0.5).to(torch.uint8))
    x = torch.randn((n, Ci), generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn((8 * Cc, 27, Ci), generator=g, device="cuda") * 0.03).to(torch.bfloat16)
    b = torch.randn(8 * Cc, generator=g, device="cuda").to(torch.bfloat16)
    for kw in (dict(), dict(ln=(None, None, 1e-6), act="silu")):
        y = sp.subdiv_conv(x, w, b, level, variant="umma_pair", **kw)
        sp.context().device_status()
        assert torch.equal(y, sp.subdiv_conv(x, w, b, level, variant="umma", **kw))


@pytest.mark.parametrize("derived", [True, False])
def test_a_level_belongs_to_the_stream_it_is_made_on(sp, derived):
    """Convs over the children run on the stream that was current when the level was made, whether their map was read off the parents' or
    hashed, and the parent's stream has filled it by then."""
    c = torch.from_numpy(cube(3000, 16, 7)).cuda()
    sub = torch.ones((3000, 8), dtype=torch.uint8, device="cuda")
    parent = sp.build_neighbors(c)
    if not derived:
        parent = sp.cache_from_map(c, parent.nbr, parent.gray)
    want = sp.build_neighbors(sp.subdivide(parent, sub).coords, want_sorted=False)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        level = sp.subdivide(parent, sub)
        assert level.nb.ctx is sp.context() and level.nb.ctx is not parent.ctx
        same = torch.equal(level.nb.nbr, want.nbr) and torch.equal(level.nb.gray, want.gray)
    torch.cuda.synchronize()
    assert same and (level._info is not None) == derived


def test_subdivision_conv_follows_a_map_changed_after_the_parents_plan(sp):
    """The parents' plan is made by a conv on them; a map written to after that is not what it holds, and the subdivision conv has to
    go by the map, as it does with a plan of its own."""
    n = 900
    g = torch.Generator(device="cuda").manual_seed(9)
    parent = sp.build_neighbors(torch.from_numpy(cube(n, 9, 11)).cuda())
    x = torch.randn((n, 64), generator=g, device="cuda").half()
    w = (torch.randn((8 * 64, 27, 64), generator=g, device="cuda") * 0.03).half()
    sp.subm_conv(x, w[:64].contiguous(), None, parent)
    level = sp.subdivide(parent, torch.ones((n, 8), dtype=torch.uint8, device="cuda"))
    assert level._from_parents(x, 64)
    parent.nbr[:, 0] = -1
    assert not level._from_parents(x, 64)
    alone = sp.cache_from_map(parent.coords, parent.nbr, parent.gray)
    want = sp.subdiv_conv(x, w, None, sp.Level(level.coords, level.src, level.nb, alone))
    assert torch.equal(sp.subdiv_conv(x, w, None, level), want)
