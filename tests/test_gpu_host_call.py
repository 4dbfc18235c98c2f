"""The host-buffer call that overlaps its copies gives the bits of the same operator on device buffers."""
import numpy as np
import pytest
import torch

from trellis2_cuda_b200 import scenes

pytestmark = pytest.mark.gpu


def test_results_over_the_features():
    """The first results lie where the last features do: nothing of them may arrive before those have been read."""
    import trellis2_cuda_b200 as sp
    n, C = 200000, 64
    g = torch.Generator().manual_seed(0)
    cells = torch.arange(n)
    c = torch.stack([0 * cells, cells // 3600, cells // 60 % 60, cells % 60], 1).to(torch.int32).pin_memory()
    buf = torch.empty((2 * n, C), dtype=torch.bfloat16).pin_memory()
    x, y = buf[:n], buf[n * 7 // 8:n * 15 // 8]
    features = torch.randn((n, C), generator=g).to(torch.bfloat16)
    w = torch.from_numpy(scenes.kaiming_uniform_weight(C, C, 1)).to(torch.bfloat16).pin_memory()
    want = sp.subm_conv(features.cuda(), w.cuda(), None, sp.build_neighbors(c.cuda(), want_sorted=False))
    for _ in range(5):
        x.copy_(features)
        assert torch.equal(sp.subm_conv_host(c, x, w, None, out=y).cuda(), want)


@pytest.mark.parametrize("dt,C,n,order", [(torch.bfloat16, 256, 20001, "morton"), (torch.float32, 128, 65536, "morton"), (torch.float16, 64, 140001, "morton"),
                                          (torch.bfloat16, 256, 30000, "random"), (torch.bfloat16, 64, 5000, "morton"), (torch.float16, 256, 20001, "pageable")])
def test_host_call_overlaps_and_gives_the_same_bits(dt, C, n, order):
    """2, 8 and 4 chunks; a scene in random order, whose rows nearly all wait for the last chunk; one too small for chunks; pageable memory."""
    import trellis2_cuda_b200 as sp
    rng = np.random.default_rng(n)
    res = int(np.ceil((n / 0.35) ** (1 / 3)))
    cells = rng.choice(res ** 3, size=n, replace=False)
    c = np.stack([np.zeros_like(cells), cells // (res * res), cells // res % res, cells % res], 1).astype(np.int32)
    if order != "random":
        key = np.zeros(n, np.int64)
        for bit in range(8):
            for ax in range(3):
                key |= ((c[:, 1 + ax].astype(np.int64) >> bit) & 1) << (3 * bit + 2 - ax)
        c = c[np.argsort(key)]
    pin = (lambda t: t) if order == "pageable" else (lambda t: t.pin_memory())
    x = pin(torch.from_numpy(rng.standard_normal((n, C), dtype=np.float32)).to(dt))
    w = pin(torch.from_numpy(scenes.kaiming_uniform_weight(C, C, 1)).to(dt))
    b = pin(torch.from_numpy(rng.standard_normal(C).astype(np.float32)).to(dt))
    c = torch.from_numpy(c)
    out = pin(torch.full((n, C), float("nan"), dtype=dt))
    want = sp.subm_conv(x.cuda(), w.cuda(), b.cuda(), sp.build_neighbors(c.cuda(), want_sorted=False), variant="auto")
    for _ in range(2):
        out.fill_(float("nan"))
        got = sp.subm_conv_host(c, x, w, b, out=out)
        assert torch.equal(got.cuda(), want)
