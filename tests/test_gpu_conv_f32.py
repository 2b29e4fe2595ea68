"""float32 layers on the (tap, channel)-ordered kernels: channel counts around the padding and tile edges, both
pixel tiles, both layouts, plain and weighted maps, against the oracle in double precision."""
import pytest
import torch

import helpers as H
from oracle import oracle

pytestmark = pytest.mark.gpu


def _check(B, cin, cout, size, grid, K, interp, layout, P=0):
    from mappedconvolutions_b200 import host
    g = torch.Generator().manual_seed(cin * 100 + cout + P)
    (IH, IW), (OH, OW) = size, grid
    x, gy = torch.randn(B, cin, IH, IW, generator=g), torch.randn(B, cout, OH, OW, generator=g)
    w, b = torch.randn(cout, cin, K, generator=g) / (cin * K) ** 0.5, torch.randn(cout, generator=g)
    # (taps beyond every edge of the image; half of the rows step by one pixel, so that neighbouring samples
    # share corners, a part of the samples lies on whole pixels)
    shape = (OH, OW, K, P, 2) if P else (OH, OW, K, 2)
    m = torch.rand(*shape, generator=g) * torch.tensor([IW + 3.0, IH + 3.0]) - 2.0
    m[::2, 1:] = m[::2, :1]
    m[::2, ..., 0] += torch.arange(OW).view(1, OW, *([1] * (m.dim() - 3))) % IW
    m[:, ::5] = m[:, ::5].round()
    m = m.contiguous()
    iw = torch.rand(OH, OW, K, P, generator=g) if P else None
    lay = (lambda t: t.cuda().contiguous(memory_format=torch.channels_last)) if layout == "nhwc" else (lambda t: t.cuda())
    pre = "weighted_mapped_conv" if P else "mapped_conv"
    maps, mapsd = ((m.cuda(), iw.cuda()), (m.double(), iw.double())) if P else ((m.cuda(),), (m.double(),))
    y = getattr(host.impl, pre + "_forward")(lay(x), *maps, w.cuda(), b.cuda(), K, interp)
    got = getattr(host.impl, pre + "_backward")(lay(gy), *maps, lay(x), w.cuda(), b.cuda(), K, interp)
    want = getattr(oracle, pre + "_forward")(x.double(), *mapsd, w.double(), b.double(), K, interp)
    wantg = getattr(oracle, pre + "_backward")(gy.double(), *mapsd, x.double(), w.double(), b.double(), K, interp)
    for name, a, r in (("y", y, want), ("gx", got[0], wantg[0]), ("gw", got[1], wantg[1]), ("gb", got[2], wantg[2])):
        H.assert_close(a, r, H.TOL[torch.float32], name)


# Cin <= 4 (two taps per thread), multiples of 8 and not, of 4 (vector gathers) and not; Cout around 16 / 32 / 64
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("interp", [0, 1, 2])
@pytest.mark.parametrize("cin,cout", [(1, 8), (3, 16), (4, 17), (5, 33), (8, 32), (12, 64), (40, 65), (33, 7)])
def test_small_tiles(cin, cout, interp, layout):
    _check(2, cin, cout, (10, 13), (9, 17), 7, interp, layout)


# 128-pixel tiles; grids whose pixel count is and is not a multiple of four (16-byte stores)
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("cin,cout,grid", [(3, 10, (150, 132)), (9, 20, (151, 131)), (4, 3, (149, 135)),
                                           (20, 40, (90, 220))])
def test_wide_tiles(cin, cout, grid, layout):
    _check(2, cin, cout, (70, 90), grid, 5, 1, layout)


@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("P,interp", [(1, 0), (3, 0), (4, 0), (5, 0), (2, 1)])  # (the last two: generic kernels)
def test_weighted_maps(P, interp, layout):
    _check(2, 12, 24, (6, 11), (8, 9), 4, interp, layout, P)
