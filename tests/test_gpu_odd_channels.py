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
    # tap 1 reads the same place from six grid pixels in a row: inverse lists beyond a table record's four entries
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


def _run(x, gy, w, b, m, K, interp, iw=None):
    from mappedconvolutions_b200 import host
    cl = lambda t: t.cuda().contiguous(memory_format=torch.channels_last)
    maps, pre = ((m.cuda(),), "mapped_conv") if iw is None else ((m.cuda(), iw.cuda()), "weighted_mapped_conv")
    y = getattr(host.impl, pre + "_forward")(cl(x), *maps, w.cuda(), b.cuda(), K, interp)
    g = getattr(host.impl, pre + "_backward")(cl(gy), *maps, cl(x), w.cuda(), b.cuda(), K, interp)
    assert host.impl.device_status() == 0
    return [t.float().cpu() for t in (y, g[0], g[1])]


def _oracle(x, gy, w, b, m, K, interp, iw=None):
    maps, pre = ((m,), "mapped_conv") if iw is None else ((m, iw), "weighted_mapped_conv")
    y = getattr(oracle, pre + "_forward")(x, *maps, w, b, K, interp)
    return [y] + list(getattr(oracle, pre + "_backward")(gy, *maps, x, w, b, K, interp)[:2])


# Padded channel counts keep float32 products and sums up to the one rounding of the result.  Bound: that rounding
# (2^-8 of the value), plus 2^-15 of the sum of the terms' magnitudes: 2^-16 for values that reach the tensor
# cores as two bf16 parts, and as much for float32 sums of up to 1600 terms, whose errors mostly cancel.
@pytest.mark.parametrize("interp,P", [(0, 0), (1, 0), (2, 0), (0, 3)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (96, 64), (64, 96), (32, 64), (128, 200), (3, 40), (12, 72), (8, 8)])
def test_odd_channel_counts_round_once(cin, cout, interp, P):
    x, gy, w, b, m, K, _ = _case(cin, cout, interp, cin + cout)
    g = torch.Generator().manual_seed(1)
    # tap 2 reads one place from every grid pixel: lists of 153 entries
    m.view(-1, K, 2)[:, 2] = torch.tensor([4.25, 3.5])
    iw = None
    if P:
        m = (m.unsqueeze(3) + torch.rand(*m.shape[:3], P, 2, generator=g) * 3).contiguous()
        iw = torch.rand(*m.shape[:3], P, generator=g)
    d = lambda *ts: [None if t is None else t.double() for t in ts]
    got = _run(x, gy, w, b, m, K, interp, iw)
    xd, gd, wd, bd, md, iwd = d(x, gy, w, b, m, iw)
    want = _oracle(xd, gd, wd, bd, md, K, interp, iwd)
    size = _oracle(xd.abs(), gd.abs(), wd.abs(), bd.abs(), md, K, interp, iwd)
    for name, a, r, s in zip(("y", "gx", "gw"), got, want, size):
        if name != "gx" and cout % 64 == 0 and (interp or P):
            continue  # (only the image's channels are padded: interpolated taps are bf16 there, as in whole blocks)
        over = ((a.double() - r).abs() / (2.0 ** -8 * r.abs() + 2.0 ** -15 * s + 1e-30)).max().item()
        assert over <= 1.0, (name, over)


@pytest.mark.parametrize("interp", [0, 1])
@pytest.mark.parametrize("cin,cout", [(32, 32), (64, 96), (8, 40), (3, 24)])
def test_infinities_reach_what_uses_them(cin, cout, interp):
    x, gy, w, b, m, K, _ = _case(cin, cout, interp, cin)
    x[0, 0, 0, 0], x[1, 1, 5, 7], gy[0, 0, 0, 0], gy[1, 2, 4, 4] = float("inf"), float("nan"), float("inf"), -float("inf")
    f = [t.float() for t in (x, gy, w, b)]
    for name, a, r in zip(("y", "gx", "gw"), _run(x, gy, w, b, m, K, interp), _oracle(*f, m, K, interp)):
        assert torch.equal(a.isnan(), r.isnan()) and torch.equal(a.isinf(), r.isinf()), name
        assert torch.equal(a[a.isinf()], r[r.isinf()]), name


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("cout", [64, 40])
def test_fused_activation_keeps_nan(cout, weighted):
    from mappedconvolutions_b200 import nn as mnn
    x, _, w, b, m, K, _ = _case(64, cout, 0, 3)
    x[0, 5, 4, 4] = float("nan")
    args = (m.cuda(),)
    if weighted:
        args = (m.unsqueeze(3).repeat(1, 1, 1, 3, 1).cuda(), torch.rand(*m.shape[:3], 3).cuda())
    layers = [mnn.MappedConvolution(64, cout, K, "nearest", activation=a).cuda().bfloat16() for a in (None, "relu")]
    layers[1].load_state_dict(layers[0].state_dict())
    xc = x.cuda().contiguous(memory_format=torch.channels_last)
    want, got = torch.relu(layers[0](xc, *args)), layers[1](xc, *args)
    assert want.isnan().any() and torch.equal(want.isnan(), got.isnan())
    assert torch.equal(want.nan_to_num(), got.nan_to_num())


@pytest.mark.parametrize("shift,ws", [(0, False), (1, True), (1, False), (0, True)])
def test_c_entry_points_without_workspace_or_alignment(shift, ws):
    """Multiples of 8 that are not multiples of 64: any element-aligned pointer, workspace or not, same result up
    to the order of the sums."""
    import ctypes
    from mappedconvolutions_b200 import _lib
    L = _lib.lib()
    x, gy, w, b, m, K, interp = _case(16, 40, 1, 5)
    d = _lib.McDesc(2, 16, 40, 10, 13, 9, 17, K, 0, 1, _lib.MC_BF16, _lib.MC_NHWC)

    def dev(t):  # channels-last, off a 16-byte boundary by `shift` elements
        t = t.permute(0, 2, 3, 1).contiguous()
        buf = torch.empty(t.numel() + 16, dtype=t.dtype, device="cuda")
        out = buf[shift:shift + t.numel()].view(t.shape)
        out.copy_(t)
        return out

    xd, gd, wd, bd, md = dev(x), dev(gy), w.cuda(), b.cuda(), m.cuda()
    y = dev(torch.zeros(2, 40, 9, 17, dtype=torch.bfloat16))
    gw, gb = torch.empty(40, 16, K, device="cuda"), torch.empty(40, device="cuda")
    n = L.mc_conv_fwd_workspace_bytes(ctypes.byref(d))
    buf = torch.empty(n, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(L.mc_conv_fwd(ctypes.byref(d), xd.data_ptr(), md.data_ptr(), None, wd.data_ptr(), bd.data_ptr(), y.data_ptr(),
                             buf.data_ptr() if ws else None, n if ws else 0, st))
    _lib.check(L.mc_conv_wgrad(ctypes.byref(d), gd.data_ptr(), xd.data_ptr(), md.data_ptr(), None, gw.data_ptr(),
                               gb.data_ptr(), None, 0, st))
    f = [t.float() for t in (x, gy, w, b)]
    want = oracle.mapped_conv_forward(f[0], m, f[2], f[3], K, 1)
    _, want_gw, want_gb = oracle.mapped_conv_backward(f[1], m, f[0], f[2], f[3], K, 1)
    H.assert_close(y.float().permute(0, 3, 1, 2), want, 2.0 ** -7, "y")  # (one rounding)
    H.assert_close(gw, want_gw, 1e-4, "gw")  # (float32 sums of values that keep 16 bits)
    H.assert_close(gb, want_gb, 1e-5, "gb")


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
