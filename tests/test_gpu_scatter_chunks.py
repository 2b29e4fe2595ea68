"""Max unpooling of whole planes and images with few and many values each: bf16 in 42 MB chunks of float32 sums (full
ones and a remainder) whose buffer is used again, the other types in one go.  Whole-number gradients, so that sums are
exact in any order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(7, 9), (400, 500)], ids=["few", "many"])
@pytest.mark.parametrize("dtype,layout,shape", [
    (torch.bfloat16, "nchw", (3, 7, 1024, 1024)),  # planes of 4 MB: chunks of 10, 10 and 1
    (torch.bfloat16, "nhwc", (3, 5, 1024, 1024)),  # images of 20 MB: chunks of 2 and 1
    (torch.bfloat16, "nhwc", (5, 4, 700, 900)),    # images of 10 MB: chunks of 4 and 1
    (torch.bfloat16, "nchw", (2, 2, 4000, 3000)),  # planes of 48 MB: beyond a chunk each
    (torch.float32, "nchw", (3, 7, 1024, 1024)), (torch.float32, "nhwc", (3, 5, 1024, 1024)),
    (torch.float64, "nchw", (2, 3, 1024, 1024)), (torch.float32, "nchw", (2, 2, 4000, 3000)),
])
def test_max_unpool_in_chunks(dtype, layout, shape, grid):
    from mappedconvolutions_b200 import host
    B, C, IH, IW = shape
    OH, OW = grid
    g = torch.Generator(device="cuda").manual_seed(OH)
    md = torch.float64 if dtype == torch.float64 else torch.float32
    m = (torch.rand(OH, OW, 4, 2, generator=g, device="cuda") * torch.tensor([IW + 1.0, IH + 1.0], device="cuda") - 1.0).to(md)
    tap = torch.randint(0, 4, (B, C, OH, OW), generator=g, device="cuda")
    entry = torch.arange(OH * OW, device="cuda").view(OH, OW) * 4 + tap  # (pixel, tap) that won, stored as a map offset
    gy = torch.randint(-3, 4, (B, C, OH, OW), generator=g, device="cuda").to(dtype)
    cl = (lambda t: t.contiguous(memory_format=torch.channels_last)) if layout == "nhwc" else (lambda t: t)
    got = host.impl.mapped_max_unpool(cl(gy), cl(2 * entry), m, IH, IW, 4, 0)
    at = m.view(-1, 2)[entry]
    at = at.double()
    at = torch.where(at >= 0, (at + 0.5).floor(), (at - 0.5).ceil())
    inside = (at[..., 0] >= 0) & (at[..., 0] < IW) & (at[..., 1] >= 0) & (at[..., 1] < IH)
    flat = torch.where(inside, at[..., 1] * IW + at[..., 0], 0).long()
    want = torch.zeros(B, C, IH * IW, dtype=torch.float32, device="cuda")
    want.scatter_add_(2, flat.view(B, C, -1), (gy.float() * inside).view(B, C, -1))
    assert torch.equal(got.reshape(B, C, -1), want.to(dtype))


def test_workspace_is_one_chunk():
    import ctypes
    from mappedconvolutions_b200 import _lib
    n = lambda B, C, H, W, lay: _lib.lib().mc_scatter_workspace_bytes(
        ctypes.byref(_lib.McDesc(B, C, C, H, W, 4, 4, 4, 0, 0, _lib.MC_BF16, lay)))
    assert n(2, 3, 10, 20, _lib.MC_NCHW) == 2 * 3 * 200 * 4 and n(2, 3, 10, 20, _lib.MC_NHWC) == 2 * 3 * 200 * 4
    assert n(32, 128, 1, 163842, _lib.MC_NCHW) == (42 << 20) // (163842 * 4) * 163842 * 4
    assert n(32, 128, 1, 163842, _lib.MC_NHWC) == 128 * 163842 * 4
    assert n(1, 1, 4000, 3000, _lib.MC_NCHW) == 4000 * 3000 * 4
