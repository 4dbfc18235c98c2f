"""Convs of small maps with wide rows: one sum per output, whoever runs it.  The bits do not depend on the mask array after the plan
is made, on scratch that other calls use, on whether a part of the plan or the whole of it runs, or on where the caller's arrays lie."""
import numpy as np
import pytest
import torch

from trellis2_cuda_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sp():
    import trellis2_cuda_b200 as m
    m.context()
    return m


def scene(n, C, seed=0):
    rng = np.random.default_rng([n, C, seed])
    res = max(4, round((n / 0.35) ** (1 / 3)))
    cells = np.sort(rng.choice(res ** 3, size=n, replace=False))
    c = torch.from_numpy(np.stack([0 * cells, cells // (res * res), cells // res % res, cells % res], 1).astype(np.int32))
    x = torch.from_numpy(rng.standard_normal((n, C), dtype=np.float32)).to(torch.bfloat16)
    w = torch.from_numpy(scenes.kaiming_uniform_weight(C, C, seed)).to(torch.bfloat16)
    return c, x, w


def test_masks_written_after_the_plan_do_not_matter(sp):
    c, x, w = (t.cuda() for t in scene(1000, 512))
    built = sp.build_neighbors(c)
    gray = built.gray.clone()
    cache = sp.spconv.cache_from_map(c, built.nbr, gray)
    want = sp.subm_conv(x, w, None, cache)
    gray.zero_()                              # one buffer for many levels: the next one's masks
    assert torch.equal(sp.subm_conv(x, w, None, cache), want)


def test_captured_conv_outlives_the_scratch_of_other_calls(sp):
    """A conv on a kept plan touches the plan and the caller's arrays only, so a graph that holds it stays good when later calls grow the
    context's scratch."""
    c, x, w = (t.cuda() for t in scene(1000, 512))
    big = scene(150000, 64)[0].cuda()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        cache = sp.build_neighbors(c)
        want = sp.subm_conv(x, w, None, cache)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        y = sp.subm_conv(x, w, None, cache)
    with torch.cuda.stream(s):
        for _ in range(2):
            sp.build_neighbors(big).plan
        y.zero_()
        graph.replay()
        eager = sp.subm_conv(x, w, None, cache)
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(eager, want)


def test_parts_give_the_bits_of_the_whole(sp):
    c, x, w = (t.cuda() for t in scene(1000, 512))
    cache = sp.build_neighbors(c)
    want = sp.subm_conv(x, w, None, cache)
    plan = cache.split_plan_for(512, 512, 600)
    out = torch.full_like(want, float("nan"))
    for part in ("interior", "boundary"):
        sp.spconv.subm_conv_split(x, w, None, cache, plan, part, out=out)
    assert torch.equal(out, want)


@pytest.mark.parametrize("pinned", [True, False])
def test_host_call_gives_the_bits_of_the_device_call(sp, pinned):
    """8 MB and more each way, where pinned buffers are copied in chunks and pageable ones whole."""
    c, x, w = scene(8000, 1024)
    if pinned:
        c, x, w = (t.pin_memory() for t in (c, x, w))
    out = torch.empty_like(x, pin_memory=pinned)
    want = sp.subm_conv(x.cuda(), w.cuda(), None, sp.build_neighbors(c.cuda(), want_sorted=False))
    assert torch.equal(sp.subm_conv_host(c, x, w, None, out=out).cuda(), want)
