"""bf16 layers whose channel counts are not multiples of 64 (padded MMA columns, packed gathers), in both
layouts, and the layout change itself."""
import pytest
import torch

import helpers as H
from oracle import oracle

pytestmark = pytest.mark.gpu


def _case(cin, cout, interp, seed):
    g = torch.Generator().manual_seed(seed)
    B, IH, IW, OH, OW, K = 2, 10, 13, 9, 17, 5
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)
    m = (torch.rand(OH, OW, K, 2, generator=g) * torch.tensor([IW + 1.0, IH + 1.0]) - 1.0).contiguous()
    # tap 1 reads the same place from six grid pixels in a row: inverse lists beyond a table record's four
    # entries.  (Not from all of them: the gathered sum is rounded to bf16, so that a list of n entries of
    # N(0, 1) adds an error of 2^-9 sqrt(n) |w| sqrt(C_out) to an output of about sqrt(K C_out) |w| - 1e-3
    # of it for six, and beyond the tolerance at its tails for all 153.)
    flat = m.view(OH * OW, K, 2)
    flat[:, 1] = flat[(torch.arange(OH * OW) // 6) * 6, 1]
    w = (torch.randn(cout, cin, K, generator=g) / (cin * K) ** 0.5).to(torch.bfloat16)
    return bf(B, cin, IH, IW), bf(B, cout, OH, OW), w, bf(cout), m, K, interp


# below / above one tile of 64 columns, several chunks, counts that are no multiple of 8
@pytest.mark.parametrize("layout", ["nchw", "nhwc"])
@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("cin,cout", [(32, 32), (96, 64), (64, 96), (8, 200), (40, 24), (72, 8), (16, 20), (64, 1),
                                      (320, 72)])
def test_odd_channel_counts_against_oracle(cin, cout, interp, layout):
    from mappedconvolutions_b200 import host
    x, gy, w, b, m, K, interp = _case(cin, cout, interp, cin + cout)
    lay = (lambda t: t.cuda().contiguous(memory_format=torch.channels_last)) if layout == "nhwc" else (lambda t: t.cuda())
    y = host.impl.mapped_conv_forward(lay(x), m.cuda(), w.cuda(), b.cuda(), K, interp)
    g = host.impl.mapped_conv_backward(lay(gy), m.cuda(), lay(x), w.cuda(), b.cuda(), K, interp)
    assert y.is_contiguous(memory_format=torch.channels_last if layout == "nhwc" and cout > 1 else torch.contiguous_format)
    want = oracle.mapped_conv_forward(x.float(), m, w.float(), b.float(), K, interp)
    want_g = oracle.mapped_conv_backward(gy.float(), m, x.float(), w.float(), b.float(), K, interp)
    for name, a, r in (("y", y, want), ("gx", g[0], want_g[0]), ("gw", g[1], want_g[1]), ("gb", g[2], want_g[2])):
        H.assert_close(a.float(), r, H.TOL[torch.bfloat16], name)
    assert host.impl.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,C,H_,W_", [(1, 64, 8, 8), (3, 65, 7, 9), (2, 17, 1, 130), (2, 3, 5, 7), (1, 200, 3, 3), (5, 16, 1, 1),
                                       (1, 20, 64, 65)])
def test_layout_change_is_exact(dtype, B, C, H_, W_):
    from mappedconvolutions_b200 import _lib
    x = torch.randn(B, C, H_, W_, device="cuda").to(dtype)
    esz, st = x.element_size(), torch.cuda.current_stream().cuda_stream
    for pad in (C, (C + 7) // 8 * 8):
        y = torch.full((B, H_ * W_, pad), 7.0, device="cuda", dtype=dtype)
        _lib.check(_lib.lib().mc_transpose(esz, B, C, H_ * W_, x.data_ptr(), y.data_ptr(), pad, st))
        want = torch.zeros_like(y)
        want[:, :, :C] = x.reshape(B, C, -1).transpose(1, 2)
        assert torch.equal(y, want)
    z = torch.empty_like(x)
    y = x.reshape(B, C, -1).transpose(1, 2).contiguous()
    _lib.check(_lib.lib().mc_transpose(esz, B, H_ * W_, C, y.data_ptr(), z.data_ptr(), H_ * W_, st))
    assert torch.equal(z, x)
