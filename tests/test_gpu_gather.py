"""Nearest maps on the tensor cores, rows fetched by the TMA unit: odd and even slice counts, one to three pixel tiles and
many, 2-D tiles, tiles that cross images, taps that read nothing, narrow column chunks (few tiles), against the oracle."""
import pytest
import torch

import helpers as H
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,K,B,size,grid", [
    (64, 64, 7, 1, (1, 40), (1, 40)),       # one partial tile, 7 slices (padded to 8 in the weight gradient)
    (64, 128, 7, 3, (1, 333), (1, 333)),    # tiles across images
    (128, 256, 5, 2, (9, 31), (8, 32)),     # 2-D tiles, two slices per tap, chunks of 64 columns
    (256, 256, 7, 1, (1, 200), (1, 150)),   # 28 slices, streamed weights
    (64, 72, 9, 2, (20, 30), (17, 23)),     # padded columns
    (192, 64, 3, 2, (16, 16), (16, 16)),    # three slices per tap
    (64, 64, 1, 2, (10, 10), (24, 48)),     # one slice per tile: steps of a warp lie in different tiles
    (64, 128, 7, 4, (1, 9000), (1, 10242)), # several tiles per block
])
def test_nearest_layers_against_oracle(cin, cout, K, B, size, grid):
    from mappedconvolutions_b200 import host
    (IH, IW), (OH, OW) = size, grid
    g = torch.Generator().manual_seed(cin + cout + K)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)
    m = (torch.rand(OH, OW, K, 2, generator=g) * torch.tensor([IW + 1.0, IH + 1.0]) - 1.0).contiguous()
    x, gy, b = bf(B, cin, IH, IW), bf(B, cout, OH, OW), bf(cout)
    w = (torch.randn(cout, cin, K, generator=g) / (cin * K) ** 0.5).to(torch.bfloat16)
    cl = lambda t: t.cuda().contiguous(memory_format=torch.channels_last)
    want = oracle.mapped_conv_forward(x.float(), m, w.float(), b.float(), K, 0)
    want_gw, want_gb = oracle.mapped_conv_backward(gy.float(), m, x.float(), w.float(), b.float(), K, 0)[1:]
    xd, gd, md = cl(x), cl(gy), m.cuda()
    for _ in range(4):  # (the ring is handed over by timing-dependent steps: same result each time)
        y = host.impl.mapped_conv_forward(xd, md, w.cuda(), b.cuda(), K, 0)
        _, gw, gb = host.impl.mapped_conv_backward(gd, md, xd, w.cuda(), b.cuda(), K, 0)
        for name, a, r in (("y", y, want), ("gw", gw, want_gw), ("gb", gb, want_gb)):
            H.assert_close(a.float(), r, H.TOL[torch.bfloat16], name)
    assert host.impl.device_status() == 0
