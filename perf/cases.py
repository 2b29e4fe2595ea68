"""The work whose speed matters to users of this library, as cases that can be timed and compared.

Every case goes through the public layer API (`mapped_convolution.nn`, `mapped_convolution.util`)
the way a program would: layers and sample maps exist before the call, the batch is on the GPU,
and one pass is a forward call or a forward and backward call.  Sample maps depend on the mesh or
image geometry only, so a program builds one and uses it for every batch: they are made once per
geometry here and shared by all states; data and weights come from the seed.

  encoder    icosphere encoder, convolutions 3 -> 64 -> 128 -> 256 -> 256 on 7-tap one-ring maps with
             fused ReLU, average pooling between the mesh levels; inference, or training with the
             gradient that the network behind it hands back
  conv       one mapped convolution on an image: spherical kernels (translation invariant along
             rows), a lens-corrected grid, a jittered (learned-offset-like) grid
  meshconv   weighted mapped convolution between icospheres, gnomonic 3 x 3 kernels whose taps are
             barycentric mixtures of three vertices
  upconv     transposed mapped convolution from one mesh level to the next finer one
  pool       mapped max / average pooling from one mesh level to the next coarser one and back
  resample   panorama -> mesh vertices (bilinear gather) and vertices -> panorama (scatter)
  colour     panorama -> vertices and vertices -> panorama with barycentric weights (three points
             per pixel), what the colour-transfer utilities of the library do per call
  knn        k nearest neighbours among points on the sphere, used to build sample maps
"""
import functools

import torch

from mapped_convolution import nn as mnn
from mapped_convolution import util as mutil

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
SIZE = {"bf16": 2, "f32": 4}
ENC_CH = (3, 64, 128, 256, 256)


def vertices(level):
    return 10 * 4 ** level + 2


def enc_levels(level):
    """Mesh level of the four convolutions of an encoder that starts at `level`."""
    return (level, level - 1, level - 2, level - 2)


# ---- the cases ---------------------------------------------------------------------------------------

def listed():
    return [
        # one small sphere through the encoder: a robot or a viewer that waits for the answer
        dict(name="encoder_infer_1", kind="encoder", level=5, batch=1, train=False),
        # training step of the same encoder at the finest mesh and the full batch
        dict(name="encoder_train_64", kind="encoder", level=7, batch=64, train=True),
        # spherical convolution layer on full panoramas, training (the headline benchmark)
        dict(name="pano_conv_train", kind="conv", map="gnomonic", height=512, stride=1, batch=8, cin=64, cout=64,
             dtype="bf16", layout="nhwc", train=True),
        # the smallest convolution of the benchmark: one fp32 image, first layer, inference
        dict(name="conv_f32_infer_1", kind="conv", map="jitter", height=64, stride=1, batch=1, cin=3, cout=16,
             dtype="f32", layout="nchw", train=False),
        # a spherical layer trained in torch's default type and layout
        dict(name="pano_conv_f32_train", kind="conv", map="gnomonic", height=128, stride=1, batch=4, cin=32, cout=64,
             dtype="f32", layout="nchw", train=True),
        # convolution on lens-distorted images: no structure in the map, odd image size, NCHW
        dict(name="lens_conv_train", kind="conv", map="lens", height=250, stride=1, batch=4, cin=64, cout=128,
             dtype="bf16", layout="nchw", train=True),
        # mesh layer with barycentric taps, training
        dict(name="mesh_conv_train", kind="meshconv", level=6, batch=8, cin=64, cout=64, dtype="bf16",
             layout="nhwc", train=True),
        # decoder layer: level 5 -> level 6, training
        dict(name="mesh_upconv_train", kind="upconv", level=6, batch=8, cin=128, cout=64, dtype="bf16",
             layout="nhwc", train=True),
        # pooling of the benchmark, both directions
        dict(name="mesh_max_pool_f32", kind="pool", op="max", level=7, batch=32, channels=128, dtype="f32",
             layout="nchw"),
        # resampling of the benchmark: 16 panoramas to the vertices and back
        dict(name="pano_resample_16", kind="resample", height=512, level=7, batch=16, channels=3),
        # colour transfer of one panorama
        dict(name="pano_colour_1", kind="colour", height=512, level=7, batch=1, channels=3),
        # neighbour search over all vertices of the finest mesh
        dict(name="knn_163842", kind="knn", points=163842, queries=163842, batch=1, k=9),
    ]


def _log(rng, lo, hi):
    """A whole number, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _fit(rng, lo, hi, most):
    """The same with an upper end that keeps the case within the largest listed one."""
    return _log(rng, lo, max(lo, min(hi, int(most))))


def draw(rng):
    kind = rng.choice(("encoder", "encoder", "conv", "conv", "conv", "meshconv", "upconv", "pool", "pool",
                       "resample", "colour", "knn"))
    if kind == "encoder":
        level = rng.randint(4, 7)
        return dict(kind=kind, level=level, batch=_fit(rng, 1, 64, 63 * vertices(7) / vertices(level)),
                    train=rng.random() < 0.6)
    if kind == "conv":
        dtype = rng.choice(("bf16", "bf16", "f32"))
        stride = rng.choice((1, 1, 2))
        if dtype == "bf16":
            height, cin, cout = _log(rng, 48, 512), rng.choice((32, 64, 96, 128)), rng.choice((32, 64, 96, 128))
            most = 7 * 512 * 512 * 64 * 64 / (height * height * cin * cout)
        else:
            height, cin, cout = _log(rng, 32, 256), _log(rng, 3, 64), _log(rng, 8, 64)
            most = 8 * 128 * 128 * 64 * 64 / (height * height * cin * cout)
        return dict(kind=kind, map=rng.choice(("gnomonic", "gnomonic", "lens", "jitter")), height=height, stride=stride,
                    batch=_fit(rng, 1, 8, most), cin=cin, cout=cout, dtype=dtype,
                    layout=rng.choice(("nchw", "nhwc")), train=rng.random() < 0.7)
    if kind in ("meshconv", "upconv"):
        dtype = rng.choice(("bf16", "bf16", "f32"))
        level = rng.randint(3, 6 if dtype == "bf16" else 5)
        cin, cout = ((rng.choice((32, 64, 128)), rng.choice((64, 128))) if dtype == "bf16"
                     else (_log(rng, 8, 64), _log(rng, 8, 64)))
        return dict(kind=kind, level=level, batch=_fit(rng, 1, 16, 4 * 16 * 4 ** (6 - level)), cin=cin, cout=cout,
                    dtype=dtype, layout="nhwc" if dtype == "bf16" else "nchw", train=rng.random() < 0.7)
    if kind == "pool":
        level, channels = rng.randint(4, 7), _log(rng, 16, 256)
        return dict(kind=kind, op=rng.choice(("max", "avg")), level=level, channels=channels,
                    batch=_fit(rng, 1, 32, 31 * 128 * vertices(7) / (channels * vertices(level))),
                    **rng.choice((dict(dtype="f32", layout="nchw"), dict(dtype="bf16", layout="nhwc"),
                                  dict(dtype="f32", layout="nhwc"))))
    if kind == "resample":
        return dict(kind=kind, height=_log(rng, 64, 768), level=rng.randint(4, 7), batch=_log(rng, 1, 16),
                    channels=rng.choice((1, 3, 3, 4, 8)))
    if kind == "colour":
        return dict(kind=kind, height=_log(rng, 64, 512), level=rng.randint(4, 7), batch=_log(rng, 1, 4),
                    channels=rng.choice((1, 3, 3, 4)))
    return dict(kind=kind, points=_log(rng, 600, 160000), queries=_log(rng, 200, 160000), batch=rng.choice((1, 1, 1, 2)),
                k=rng.choice((1, 3, 7, 9, 16)))


# ---- maps: one per geometry --------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def kernel_map(level):
    return mutil.vertex_kernel_map(level).to(DEV)


@functools.lru_cache(maxsize=64)
def pooling_map(level):
    return mutil.pooling_map(level).to(DEV)


@functools.lru_cache(maxsize=64)
def image_map(kind, height, stride):
    """(OH, OW, 9, 2) map of a 3 x 3 kernel on a height x 2 height image."""
    h, w = height, 2 * height
    if kind == "gnomonic":
        m = mutil.get_projection_map((h, w), (3, 3), "gnomonic", stride)
    else:
        m = mutil.get_perspective_projection_map((h, w), (3, 3), stride)
        if kind == "jitter":
            m = m + torch.rand(m.shape, generator=torch.Generator().manual_seed(0)) - 0.5
        else:  # radial lens distortion about the image centre
            c = torch.tensor([(w - 1) / 2.0, (h - 1) / 2.0])
            d = (m - c) / h
            m = c + h * d * (1.0 + 0.05 * (d * d).sum(-1, keepdim=True))
    return m.float().contiguous().to(DEV)


@functools.lru_cache(maxsize=64)
def mesh_map(level):
    """Vertices (1, V, 9, 3, 2) and barycentric weights (1, V, 9, 3) of a gnomonic 3 x 3 kernel."""
    m, w = mutil.vertex_to_vertex_kernel_map(mutil.generate_icosphere(level), 3, 3, level)
    return m.contiguous().to(DEV), w.contiguous().to(DEV)


@functools.lru_cache(maxsize=64)
def vertex_map(height, level):
    return mutil.image_to_sphere_resample_map((height, 2 * height), mutil.generate_icosphere(level)).contiguous().to(DEV)


@functools.lru_cache(maxsize=64)
def colour_map(height, level):
    m, w = mutil.sphere_to_image_resample_map(level, (height, 2 * height))
    return m.contiguous().to(DEV), w.contiguous().to(DEV)


# ---- states ------------------------------------------------------------------------------------------

def _randn(g, shape, case):
    t = torch.randn(shape, generator=g, device=DEV).to(DTYPES[case["dtype"]])
    return t.contiguous(memory_format=torch.channels_last) if case["layout"] == "nhwc" else t


def _grid(case):
    """Grid that the map of a conv case has: every stride-th pixel of the image."""
    s = case["stride"]
    return -(-case["height"] // s), -(-2 * case["height"] // s)


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    torch.manual_seed(seed)  # (initialisation of the layers)
    kind = case["kind"]
    s = dict(kind=kind, train=case.get("train", True))
    if kind == "encoder":
        case = dict(case, dtype="bf16", layout="nhwc")
        lv, n = enc_levels(case["level"]), case["batch"]
        s["convs"] = torch.nn.ModuleList(
            [mnn.MappedConvolution(ENC_CH[i], ENC_CH[i + 1], 7, "nearest", activation="relu")
             for i in range(4)]).to(DEV).to(torch.bfloat16)
        s["pool"] = mnn.MappedAvgPool(7, "nearest")
        s["maps"] = [kernel_map(l) for l in lv]
        s["pools"] = [pooling_map(lv[0]), pooling_map(lv[1])]
        s["x"] = _randn(g, (n, 3, 1, vertices(lv[0])), case)
        s["gy"] = _randn(g, (n, 256, 1, vertices(lv[3])), case)
        s["params"] = list(s["convs"].parameters())
    elif kind == "conv":
        h, (oh, ow) = case["height"], _grid(case)
        s["layer"] = mnn.MappedConvolution(case["cin"], case["cout"], 9, "bilinear").to(DEV).to(DTYPES[case["dtype"]])
        s["map"], s["iw"] = image_map(case["map"], h, case["stride"]), None
        s["x"] = _randn(g, (case["batch"], case["cin"], h, 2 * h), case).requires_grad_(case["train"])
        s["gy"] = _randn(g, (case["batch"], case["cout"], oh, ow), case)
    elif kind == "meshconv":
        n = vertices(case["level"])
        s["layer"] = mnn.MappedConvolution(case["cin"], case["cout"], 9, "nearest").to(DEV).to(DTYPES[case["dtype"]])
        s["map"], s["iw"] = mesh_map(case["level"])
        s["x"] = _randn(g, (case["batch"], case["cin"], 1, n), case).requires_grad_(case["train"])
        s["gy"] = _randn(g, (case["batch"], case["cout"], 1, n), case)
    elif kind == "upconv":
        n, fine = vertices(case["level"] - 1), vertices(case["level"])
        s["layer"] = mnn.MappedTransposedConvolution(case["cin"], case["cout"], 7, "nearest").to(DEV).to(
            DTYPES[case["dtype"]])
        s["map"], s["out"] = pooling_map(case["level"]), (1, fine)
        s["x"] = _randn(g, (case["batch"], case["cin"], 1, n), case).requires_grad_(case["train"])
        s["gy"] = _randn(g, (case["batch"], case["cout"], 1, fine), case)
    elif kind == "pool":
        n, coarse = vertices(case["level"]), vertices(case["level"] - 1)
        s["layer"] = (mnn.MappedMaxPool(7, "nearest", return_indices=True) if case["op"] == "max"
                      else mnn.MappedAvgPool(7, "nearest"))
        s["op"], s["map"] = case["op"], pooling_map(case["level"])
        s["x"] = _randn(g, (case["batch"], case["channels"], 1, n), case).requires_grad_(True)
        s["gy"] = _randn(g, (case["batch"], case["channels"], 1, coarse), case)
    elif kind == "resample":
        h = case["height"]
        s["down"], s["up"] = mnn.Unresample("bilinear"), mnn.Resample("bilinear")
        s["map"], s["shape"] = vertex_map(h, case["level"]), (h, 2 * h)
        s["x"] = torch.rand((case["batch"], case["channels"], h, 2 * h), generator=g, device=DEV)
    elif kind == "colour":
        h = case["height"]
        s["down"], s["up"] = mnn.Resample("bispherical"), mnn.Unresample("bispherical")
        (s["map"], s["iw"]), s["shape"] = colour_map(h, case["level"]), (1, vertices(case["level"]))
        s["x"] = torch.rand((case["batch"], case["channels"], h, 2 * h), generator=g, device=DEV)
    else:  # points spread over the unit sphere: mesh vertices where there is a mesh of that size
        q, _ = torch.linalg.qr(torch.randn((3, 3), generator=g, device=DEV))
        level = next((l for l in range(8) if vertices(l) == case["points"]), None)
        if level is not None:
            p = mutil.generate_icosphere(level).get_vertices().to(DEV).t().unsqueeze(0).expand(case["batch"], -1, -1)
        else:
            p = torch.randn((case["batch"], 3, case["points"]), generator=g, device=DEV)
            p = p / p.norm(dim=1, keepdim=True)
        s["ref"] = torch.matmul(q, p).contiguous()
        if case["queries"] == case["points"]:
            s["query"] = s["ref"]
        else:
            p = torch.randn((case["batch"], 3, case["queries"]), generator=g, device=DEV)
            s["query"] = (p / p.norm(dim=1, keepdim=True)).contiguous()
        s["k"] = case["k"]
    return s


# ---- one pass ----------------------------------------------------------------------------------------

def _encode(s):
    c, m, p = s["convs"], s["maps"], s["pools"]
    h = s["pool"](c[0](s["x"], m[0]), p[0])
    h = s["pool"](c[1](h, m[1]), p[1])
    return c[3](c[2](h, m[2]), m[3])


def run(s):
    kind = s["kind"]
    if kind == "encoder":
        if not s["train"]:
            with torch.no_grad():
                return _encode(s)
        h = _encode(s)
        return (h.detach(),) + torch.autograd.grad(h, s["params"], s["gy"])
    if kind == "resample":
        v = s["down"](s["x"], s["map"])
        return v, s["up"](v, s["map"], s["shape"])
    if kind == "colour":
        v = s["down"](s["x"], s["map"], s["shape"], s["iw"])
        return v, s["up"](v, s["map"], s["iw"])
    if kind == "knn":
        return mutil.knn(s["ref"], s["query"], s["k"])
    if kind == "pool":
        y = s["layer"](s["x"], s["map"])
        y, idx = y if s["op"] == "max" else (y, None)
        return (y.detach(), idx) + torch.autograd.grad(y, (s["x"],), s["gy"])
    layer, x = s["layer"], s["x"]
    args = (x,) + (s["out"] if kind == "upconv" else ()) + (s["map"],) + ((s["iw"],) if s.get("iw") is not None else ())
    if not s["train"]:
        with torch.no_grad():
            return layer(*args)
    y = layer(*args)
    return (y.detach(),) + torch.autograd.grad(y, (x, layer.weight, layer.bias), s["gy"])


# ---- what a pass cannot do without -------------------------------------------------------------------

def _layer_work(b, n_in, n_out, cin, cout, k, points, size, train, input_grad=True):
    """One (transposed) convolution: every tensor once, the contraction 2 b n k cin cout flops per direction."""
    x, y, w = b * n_in * cin * size, b * n_out * cout * size, cin * cout * k * size
    gemm = 2.0 * b * max(1, min(n_in, n_out) if points < 0 else n_out) * k * cin * cout
    maps = (n_in if points < 0 else n_out) * k * max(1, points) * (8 if points <= 0 else 12)
    if not train:
        return x + y + w + maps, gemm
    # forward: x, w -> y; backward: gy, x, w -> gx, gw
    return (x + y + w + maps) + (y + x + 2 * w) + (x if input_grad else 0), gemm * (3 if input_grad else 2)


def work(case):
    kind, b = case["kind"], case["batch"]
    size = SIZE[case.get("dtype", "bf16")]
    if kind == "encoder":
        lv, by, fl = enc_levels(case["level"]), 0, 0
        for i in range(4):
            n = vertices(lv[i])
            q, f = _layer_work(b, n, n, ENC_CH[i], ENC_CH[i + 1], 7, 0, 2, case["train"], i > 0)
            by, fl = by + q, fl + f
        for i in range(2):
            by += b * ENC_CH[i + 1] * (vertices(lv[i]) + vertices(lv[i] - 1)) * 2 * (2 if case["train"] else 1)
        return dict(bytes=by, flops=fl)
    if kind == "conv":
        oh, ow = _grid(case)
        q, f = _layer_work(b, 2 * case["height"] ** 2, oh * ow, case["cin"], case["cout"], 9, 0, size, case["train"])
        return dict(bytes=q, flops=f)
    if kind == "meshconv":
        n = vertices(case["level"])
        q, f = _layer_work(b, n, n, case["cin"], case["cout"], 9, 3, size, case["train"])
        return dict(bytes=q, flops=f)
    if kind == "upconv":
        q, f = _layer_work(b, vertices(case["level"] - 1), vertices(case["level"]), case["cin"], case["cout"], 7, -1,
                           size, case["train"])
        return dict(bytes=q, flops=f)
    if kind == "pool":
        n, m = vertices(case["level"]), vertices(case["level"] - 1)
        per = b * case["channels"]
        index = 2 * 8 * per * m if case["op"] == "max" else 0
        return dict(bytes=2 * per * (n + m) * size + index + m * 7 * 8, flops=2.0 * per * m * 7)
    if kind in ("resample", "colour"):
        n, v = 2 * case["height"] ** 2, vertices(case["level"])
        maps = v * 8 if kind == "resample" else n * 3 * 12
        return dict(bytes=2 * (b * case["channels"] * (n + v) * 4 + maps),
                    flops=4.0 * b * case["channels"] * (4 * v if kind == "resample" else 3 * n))
    return dict(bytes=b * (3 * 4 * (case["points"] + case["queries"]) + case["queries"] * case["k"] * 12),
                flops=9.0 * b * case["queries"] * case["k"])


def tolerance(case):
    if case["kind"] == "knn":
        return "exact"  # indices, and distances whose order decides near ties
    if case["kind"] == "encoder":  # bf16 activations rounded in each of four layers, and again on the way back
        return dict(rel=2e-2)
    if case.get("dtype") == "bf16":
        return dict(rel=1e-2)
    return dict(rel=1e-5)
