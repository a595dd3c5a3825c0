"""Performance cases of the PIV engine: the calls a user's program makes, over the range of
image sizes, window shapes and forms that the framework is used for.

  pair     one image pair through the whole multigrid loop (Engine.run_pair) and the filtered
           field read back: frames already on the GPU, or uploaded from pinned host memory
           (queue_images) in the same pass
  batch    pairs of uneven size and window shape in one call (Batch.run)
  learned  a pair whose grid-1 passes are replaced by the trained predictor
  train    one forward-and-backward call of the predictor's training
  mhe      contrast enhancement of one frame on its own (mhe_gpu)

Sizes are those of the repository's own workloads: the 6600x4400 recording (64 px windows, then
32 px), the uneven batch's frames (1024x1024, 2048x1536, 4096x2160) with 16, 24, 32 and 64 px
windows at 50 or 75 % overlap, the odd-sized small frames of its tests, and the training set's
64 pairs of 31x31 vectors.  Frames are seeded synthetic particle images (Gaussian spots of 0.6 px,
0.04 particles per pixel, a Lamb-Oseen vortex with shear, grey-level noise), drawn with PyTorch
in integer sums so that a seed gives the same frames every time.

exact() states the same pipeline in 64 bits with plain PyTorch.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "piv_xcorr2d_v1.0_b200"


def _package():
    """The framework (its folder's name is not a Python identifier)."""
    if "piv_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("piv_b200", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["piv_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["piv_b200"]


P = _package()

# ------------------------------------------------------------------------------
# The cases.
# ------------------------------------------------------------------------------


def _pair(Nx, Ny, w1, s1, n1, w2, s2, n2, mhe=True, host=False, kind="pair"):
    """A pair: window (x, y), spacing (x, y) and passes of both grids."""
    return {"kind": kind, "Nx": Nx, "Ny": Ny, "mhe": mhe, "host": host,
            "wx1": w1[0], "wy1": w1[1], "sx1": s1[0], "sy1": s1[1], "n1": n1,
            "wx2": w2[0], "wy2": w2[1], "sx2": s2[0], "sy2": s2[1], "n2": n2}


def _sq(a):
    return (a, a)


HEADLINE = (6600, 4400, _sq(64), _sq(32), 2, _sq(32), _sq(16), 3)


def listed():
    return [
        # a small odd-sized crop, as in a parameter search or a live view: launches and latency
        dict(_pair(333, 251, _sq(32), _sq(16), 1, _sq(16), _sq(8), 2), name="pair 333x251"),
        # one frame of a 1 Mpx camera, the usual multigrid settings
        dict(_pair(1024, 1024, _sq(64), _sq(32), 2, _sq(32), _sq(16), 3), name="pair 1024x1024"),
        # the same camera class with non-square windows along the flow (a boundary layer), no MHE
        dict(_pair(2048, 1536, (64, 32), (32, 16), 2, (48, 24), (24, 12), 2, mhe=False), name="pair 2048x1536 48x24"),
        # dense vectors from small windows: 16 px at 75 % overlap
        dict(_pair(2048, 1536, _sq(32), _sq(8), 2, _sq(16), _sq(4), 3), name="pair 2048x1536 16@4"),
        # a 4K sensor, windows that are no power of two
        dict(_pair(4096, 2160, _sq(48), _sq(24), 2, _sq(24), _sq(12), 3), name="pair 4096x2160 24@12"),
        # low seeding: wide windows, outside the fused shapes
        dict(_pair(2048, 1536, _sq(96), _sq(48), 2, _sq(40), _sq(20), 2), name="pair 2048x1536 40@20"),
        # the large recording, frames on the GPU
        dict(_pair(*HEADLINE), name="pair 6600x4400"),
        # the same from pinned host frames to the field in host memory
        dict(_pair(*HEADLINE, host=True), name="pair 6600x4400 host"),
        # the same with the trained predictor in place of the grid-1 passes
        dict(_pair(*HEADLINE, kind="learned"), name="learned 6600x4400"),
        # recordings of several cameras in one call
        {"name": "batch of 9", "kind": "batch", "pairs": 9, "pick": 0},
        # a training step's gradients: 64 pairs of 1024x1024, 31x31 vectors each
        {"name": "train 64x31x31", "kind": "train", "N": 64, "H": 31, "W": 31},
        # contrast enhancement alone, in front of another program
        {"name": "mhe 4096x2160", "kind": "mhe", "Nx": 4096, "Ny": 2160, "ws": 40, "thresh": 0.91},
    ]


SHAPES2 = [(16, 16), (24, 24), (32, 32), (48, 48), (64, 64), (48, 24), (24, 48), (32, 16), (64, 32), (40, 40), (36, 60)]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair"] * 6 + ["learned", "batch", "train", "mhe"])
    if kind == "train":
        n, h, w = _log(rng, 4, 64), rng.randint(17, 40), rng.randint(17, 40)
        return {"kind": "train", "N": max(1, min(n, 64 * 961 // (h * w))), "H": h, "W": w}
    if kind == "mhe":
        nx = _log(rng, 256, 6600)
        return {"kind": "mhe", "Nx": nx, "Ny": max(128, int(nx * rng.uniform(0.5, 1.0))),
                "ws": rng.choice([16, 24, 25, 32, 40, 64]), "thresh": 0.91}
    if kind == "batch":
        return {"kind": "batch", "pairs": rng.randint(2, 9), "pick": rng.randint(1, 1 << 20)}
    if kind == "learned":
        nx = _log(rng, 768, 6600)
        return _pair(nx, max(512, int(nx * rng.uniform(0.6, 1.0))), _sq(64), _sq(32), 2, _sq(32), _sq(16),
                     rng.randint(1, 3), kind="learned")
    w2 = rng.choice(SHAPES2)
    ov = rng.choice([0.5, 0.5, 0.75])
    w1 = tuple(min(2 * v, 64) if v < 64 else v for v in w2)
    s1 = tuple(max(4, int(round(v * (1 - ov)))) for v in w1)
    s2 = tuple(max(4, int(round(v * (1 - ov))) - (1 if rng.random() < 0.2 else 0)) for v in w2)
    nx = _log(rng, 300, 6600)
    c = _pair(nx, max(256, int(nx * rng.uniform(0.5, 1.0))), w1, s1, rng.randint(1, 2), w2, s2, rng.randint(1, 3),
              mhe=rng.random() < 0.7, host=rng.random() < 0.2)
    most = work(_pair(*HEADLINE))["flops"]
    if (w2[0] * w2[1]) % 1024 == 0 or w2 in ((16, 16), (48, 24), (24, 48)):
        limit = most
    else:
        limit = most / 4  # the general-size kernel and mixed radices take longer per window
    while work(c)["flops"] > limit:
        c["Nx"] = int(c["Nx"] * 0.8)
        c["Ny"] = max(200, int(c["Ny"] * 0.8))
    return c


BATCH_SIZES = [(1024, 1024), (2048, 1536), (4096, 2160)]


def _batch_pairs(case):
    """The pairs of a batch case: sizes in turn, window and overlap drawn, 2 + 3 passes."""
    rng = np.random.default_rng(17 + case["pick"])
    out = []
    for k in range(case["pairs"]):
        nx, ny = BATCH_SIZES[k % 3]
        w2 = int(rng.choice([16, 24, 32, 64]))
        ov = float(rng.choice([0.5, 0.75]))
        w1 = min(2 * w2, 64)
        if w2 == 16 and nx == 4096:
            ov = 0.5  # one 4K pair at 75 % overlap of 16 px would outweigh all others
        out.append(_pair(nx, ny, _sq(w1), _sq(int(round(w1 * (1 - ov)))), 2, _sq(w2), _sq(int(round(w2 * (1 - ov)))), 3))
    return out


# ------------------------------------------------------------------------------
# Inputs.
# ------------------------------------------------------------------------------


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _frames(c, seed):
    """Both frames [Ny][Nx] uint8: spots summed in 1/256 grey levels (integers: the order of
    the sums does not matter), background 10, noise of 2 grey levels."""
    Nx, Ny, dev = c["Nx"], c["Ny"], _device()
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 13)
    M = 20  # particles are drawn this far outside the image as well
    n = int(0.04 * (Nx + 2 * M) * (Ny + 2 * M))
    x = torch.rand(n, generator=g, device=dev) * (Nx + 2 * M) - M
    y = torch.rand(n, generator=g, device=dev) * (Ny + 2 * M) - M
    peak = 120.0 + 135.0 * torch.rand(n, generator=g, device=dev)
    # Lamb-Oseen vortex (at most 10 px, less for small windows) with a shear of 0.002 px/px
    a = min(10.0, 0.16 * min(c.get("wx1", 64), c.get("wy1", 64)))
    core = 0.14 * min(Nx, Ny)
    rx, ry = x - 0.5 * Nx, y - 0.5 * Ny
    r = torch.sqrt(rx * rx + ry * ry).clamp_min(1e-3)
    sp = a * 1.398 * (core / r) * (1 - torch.exp(-1.2564 * (r / core) ** 2)) / r
    u, v = -sp * ry + 0.002 * ry, sp * rx
    out = []
    for px, py in ((x, y), (x + u, y + v)):
        W, H = Nx + 8, Ny + 8
        img = torch.zeros(W * H, dtype=torch.int32, device=dev)
        ok = (px > -3) & (px < Nx + 2) & (py > -3) & (py < Ny + 2)
        px, py, pk = px[ok], py[ok], peak[ok]
        ix, iy = torch.round(px), torch.round(py)
        for dy in range(-2, 3):
            ey = torch.exp(-((iy + dy - py) ** 2) / 0.72)
            for dx in range(-2, 3):
                val = (256 * pk * ey * torch.exp(-((ix + dx - px) ** 2) / 0.72)).to(torch.int32)
                q = (iy + dy + 4).clamp(0, H - 1).to(torch.int64) * W + (ix + dx + 4).clamp(0, W - 1).to(torch.int64)
                img.index_add_(0, q, val)
        img = img.view(H, W)[4:4 + Ny, 4:4 + Nx].to(torch.float32) / 256
        img = img + 10 + 2 * torch.randn((Ny, Nx), generator=g, device=dev)
        out.append(img.round().clamp(0, 255).to(torch.uint8).contiguous())
    return out


def _params(c):
    return P.default_params(
        Nx=c["Nx"], Ny=c["Ny"], if_mhe=int(c["mhe"]), mhe_ws=40, mhe_thresh=0.91,
        ws_x1=c["wx1"], ws_y1=c["wy1"], spacing_x1=c["sx1"], spacing_y1=c["sy1"], Npass1=c["n1"],
        ws_x2=c["wx2"], ws_y2=c["wy2"], spacing_x2=c["sx2"], spacing_y2=c["sy2"], Npass2=c["n2"],
        insert_threshold_p1=2.0, insert_threshold_p2=2.0)


def _training_batch(case, seed):
    """Cost volumes as the features give them (a bump of 0.9 at the displacement, 0.1 of noise),
    their displacements (smooth, within 3 downsampled px) and a mask with 5 % holes."""
    N, H, W, dev = case["N"], case["H"], case["W"], _device()
    g = torch.Generator(device=dev).manual_seed(int(seed) * 104729 + 7)
    yy = torch.arange(H, device=dev).view(1, 1, H, 1) / H
    xx = torch.arange(W, device=dev).view(1, 1, 1, W) / W
    k = torch.rand((4, N, 2, 1, 1), generator=g, device=dev)
    label = 3 * (torch.sin(6.28 * (xx * k[0] + yy * k[1] + k[2])) * k[3])
    s = torch.arange(9, device=dev, dtype=torch.float32) - 4
    bx = torch.exp(-0.5 * (s.view(1, 9, 1, 1) - label[:, 0:1]) ** 2)
    by = torch.exp(-0.5 * (s.view(1, 9, 1, 1) - label[:, 1:2]) ** 2)
    x = 0.9 * (by.unsqueeze(2) * bx.unsqueeze(1)).reshape(N, 81, H, W)
    x = x + 0.1 * torch.randn((N, 81, H, W), generator=g, device=dev)
    mask = (torch.rand((N, H, W), generator=g, device=dev) < 0.95).float()
    return x.contiguous(), label.contiguous(), mask.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "train":
        st["x"], st["label"], st["mask"] = _training_batch(case, seed)
        st["net"] = P.PredictorNet(seed=1 + seed % 97)
    elif kind == "mhe":
        st["frame"] = _frames(case, seed)[0]
        st["mhe"] = P.mhe_gpu()
        assert st["mhe"].init(case["Nx"], case["Ny"], case["ws"], case["thresh"])
    elif kind == "batch":
        pairs = _batch_pairs(case)
        st["batch"] = P.Batch([_params(c) for c in pairs])
        st["frames"] = [_frames(c, seed * 64 + k) for k, c in enumerate(pairs)]
        torch.cuda.synchronize()
        for e, (a, b) in zip(st["batch"].engines, st["frames"]):
            e.set_device_images(a.data_ptr(), b.data_ptr())
    else:
        a, b = _frames(case, seed)
        st["engine"] = P.Engine(_params(case))
        if case["host"]:
            st["frames"] = (a.cpu().pin_memory(), b.cpu().pin_memory())
        else:
            st["frames"] = (a, b)
        if kind == "learned":
            st["net"] = P.PredictorNet(weights=PKG / "weights" / "predictor.bin")
    torch.cuda.synchronize()
    if "engine" in st and not case["host"]:
        st["engine"].set_device_images(st["frames"][0].data_ptr(), st["frames"][1].data_ptr())
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind == "train":
        net, c = st["net"], st["case"]
        loss = net.loss_grad(st["x"], st["label"], st["mask"], c["N"], c["H"], c["W"])
        return {"loss": loss, "grads": net.grads()}
    if kind == "mhe":
        assert st["mhe"].processsing(st["frame"])
        return st["mhe"].d_enhanced
    if kind == "batch":
        st["batch"].run()
        st["batch"].synchronize()
        return [dict(zip(FIELD, e.field(3))) for e in st["batch"].engines]
    e = st["engine"]
    if kind == "learned":
        judged = e.run_pair_learned(st["net"])
        return {**judged, **dict(zip(FIELD, e.field(3)))}
    if st["case"]["host"]:
        e.queue_images(*st["frames"])
        e.run_pair()
        return dict(zip(FIELD, e.field_wait(e.field_async(3))))
    e.run_pair()
    return dict(zip(FIELD, e.field(3)))


FIELD = ("x", "y", "dx", "dy", "valid")


# ------------------------------------------------------------------------------
# What a pass cannot do without.
# ------------------------------------------------------------------------------


def _vectors(N, sp):
    t1 = (N - sp // 2 - 1) // sp
    t2 = N - (sp // 2 + 1 + t1 * sp)
    while t2 < sp // 2 - 1:
        t1, t2 = t1 - 1, t2 + sp
    return t1 + 1


# (input channels, output channels, stride, level of the output) of the predictor's layers
LAYERS = ((81, 32, 1, 0), (32, 32, 1, 0), (32, 64, 2, 1), (64, 64, 1, 1), (64, 96, 2, 2), (96, 96, 1, 2),
          (96, 128, 2, 3), (128, 128, 1, 3), (224, 96, 1, 2), (96, 96, 1, 2), (160, 64, 1, 1), (96, 32, 1, 0),
          (32, 2, 1, 0))


def _net_macs(H, W):
    dims = [(H, W)]
    for _ in range(3):
        dims.append(((dims[-1][0] + 1) // 2, (dims[-1][1] + 1) // 2))
    return sum(9 * ci * co * dims[lv][0] * dims[lv][1] for ci, co, _, lv in LAYERS)


def work(case):
    """Bytes: frames (or network inputs) read once, results written once.  Flops: per window and
    pass the transforms of two real frames and of a real correlation (1.5 complex transforms of
    5 N log2 N) and the product; two per multiply-add of the network, three times in training."""
    kind = case["kind"]
    if kind == "train":
        N, H, W = case["N"], case["H"], case["W"]
        return {"bytes": 4.0 * N * H * W * 84 + 4 * 881922, "flops": 6.0 * N * _net_macs(H, W)}
    if kind == "mhe":
        return {"bytes": 2.0 * case["Nx"] * case["Ny"], "flops": 0.0}
    if kind == "batch":
        each = [work(c) for c in _batch_pairs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    flops = 0.0
    for k, n in (("1", 0 if kind == "learned" else case["n1"]), ("2", case["n2"])):
        pts = case["wx" + k] * case["wy" + k]
        nv = _vectors(case["Nx"], case["sx" + k]) * _vectors(case["Ny"], case["sy" + k])
        flops += n * nv * (1.5 * 5 * pts * math.log2(pts) + 8 * pts)
    if kind == "learned":
        nv = (_vectors(case["Nx"], case["sx1"]), _vectors(case["Ny"], case["sy1"]))
        flops += 2.0 * _net_macs(nv[1], nv[0]) + 2.0 * 81 * nv[0] * nv[1] * case["wx1"] * case["wy1"] / 16
    return {"bytes": 2.0 * case["Nx"] * case["Ny"] + 17.0 * nv_out(case), "flops": flops}


def nv_out(case):
    return _vectors(case["Nx"], case["sx2"]) * _vectors(case["Ny"], case["sy2"])


# ------------------------------------------------------------------------------
# The same in 64 bits with plain PyTorch.
# ------------------------------------------------------------------------------

D = torch.float64


def _mhe(img, ws, thresh):
    """Tile histograms summed over the 3x3 neighbourhood, thresholded and stretched to a lookup
    table per tile; whole numbers throughout."""
    Ny, Nx = img.shape
    wd, ht = ws * (Nx // ws), ws * (Ny // ws)
    xs, ys = (0, 0) if (wd, ht) == (Nx, Ny) else ((Nx - wd) // 2, (Ny - ht) // 2)
    I, J = ht // ws, wd // ws
    t = img[ys:ys + ht, xs:xs + wd].reshape(I, ws, J, ws).permute(0, 2, 1, 3).reshape(I * J, ws * ws).to(torch.int64)
    hist = torch.zeros((I * J, 256), dtype=torch.int64, device=img.device).scatter_add_(1, t, torch.ones_like(t))
    pad = torch.zeros((I + 2, J + 2, 256), dtype=torch.int64, device=img.device)
    pad[1:-1, 1:-1] = hist.view(I, J, 256)
    tr = sum(pad[a:a + I, b:b + J] for a in range(3) for b in range(3))
    iy, ix = torch.arange(I, device=img.device).view(I, 1), torch.arange(J, device=img.device).view(1, J)
    inner = (ix >= 1) & (ix <= J - 2) & (iy >= 1) & (iy <= I - 2)
    corner = ((ix == 0) | (ix == J - 1)) & ((iy == 0) | (iy == I - 1))
    cnt = torch.where(inner, 9, torch.where(corner, 4, 6)).view(I, J, 1)
    trash = int(np.floor(np.float32(ws * ws) * np.float32(thresh) + np.float32(0.5)))
    cum = (tr.cumsum(2) - cnt * trash).clamp_min(0)
    lut = (cum * 255 // (cnt * (ws * ws - trash))).clamp_max(255)
    lut[..., 0], lut[..., 255] = 0, 255
    out = torch.zeros_like(img)
    res = lut.view(I * J, 256).gather(1, t).to(torch.uint8)
    out[ys:ys + ht, xs:xs + wd] = res.view(I, J, ws, ws).permute(0, 2, 1, 3).reshape(ht, wd)
    return out


class _Grid:
    def __init__(self, c, k):
        self.w, self.s = (c["wx" + k], c["wy" + k]), (c["sx" + k], c["sy" + k])
        size = (c["Nx"], c["Ny"])
        self.n = tuple(_vectors(size[i], self.s[i]) for i in range(2))
        h = tuple(v // 2 for v in self.w)
        self.left = tuple(max(0, h[i] - self.s[i] // 2) for i in range(2))
        last = tuple(self.s[i] // 2 + 1 + (self.n[i] - 1) * self.s[i] for i in range(2))
        right = tuple(max(0, last[i] + h[i] - 1 - size[i]) for i in range(2))
        self.aug = tuple(size[i] + self.left[i] + right[i] for i in range(2))
        self.border = tuple(max(1, h[i] - int(math.floor(float(np.float32(self.w[i]) * np.float32(0.4)) + 0.5)))
                            for i in range(2))
        self.h = h

    def extent(self, frame):
        """The frame with the grid's zero margins, [aug_y][aug_x]."""
        out = torch.zeros((self.aug[1], self.aug[0]), dtype=D, device=frame.device)
        out[self.left[1]:self.left[1] + frame.shape[0], self.left[0]:self.left[0] + frame.shape[1]] = frame
        return out

    def windows(self, ext):
        v = ext.unfold(0, self.w[1], self.s[1]).unfold(1, self.w[0], self.s[0])
        return v[:self.n[1], :self.n[0]]


def _cell(field, nx, ny, ix, iy):
    return field[(iy - 3).clamp(0, ny - 1), (ix - 3).clamp(0, nx - 1)]


def _bilinear(field, g, X, Y, x_st, y_st):
    """The field [ny][nx] between its vectors, edge values outside, at the outer product Y, X."""
    ax, ay = (X - x_st) / g.s[0], (Y - y_st) / g.s[1]
    ix, iy = torch.floor(ax), torch.floor(ay)
    fx, fy = (ax - ix).view(1, -1), (ay - iy).view(-1, 1)
    ix, iy = ix.long().view(1, -1), iy.long().view(-1, 1)
    nx, ny = g.n
    return ((1 - fx) * (1 - fy) * _cell(field, nx, ny, ix, iy) + fx * (1 - fy) * _cell(field, nx, ny, ix + 1, iy) +
            (1 - fx) * fy * _cell(field, nx, ny, ix, iy + 1) + fx * fy * _cell(field, nx, ny, ix + 1, iy + 1))


def _deform(img, g, fx, fy):
    dev = img.device
    X = torch.arange(g.aug[0], device=dev, dtype=D)
    Y = torch.arange(g.aug[1], device=dev, dtype=D)
    ax = X.view(1, -1) + _bilinear(fx, g, X, Y, g.h[0] - 3 * g.s[0], g.h[1] - 3 * g.s[1])
    ay = Y.view(-1, 1) + _bilinear(fy, g, X, Y, g.h[0] - 3 * g.s[0], g.h[1] - 3 * g.s[1])
    ix, iy = torch.floor(ax), torch.floor(ay)
    ax, ay = ax - ix, ay - iy
    ix, iy = ix.long() - g.left[0], iy.long() - g.left[1]
    Ny, Nx = img.shape
    flat, out = img.reshape(-1), torch.zeros_like(ax)
    for dy in range(2):
        for dx in range(2):
            c, r = ix + dx, iy + dy
            ok = (c >= 0) & (c < Nx) & (r >= 0) & (r < Ny)
            v = flat[torch.where(ok, r * Nx + c, 0)] * ok
            out += (ax if dx else 1 - ax) * (ay if dy else 1 - ay) * v
    return out


def _candidates(g, e1, e2, px, py, peaks=4):
    """The highest local maxima of every window's correlation with their sub-pixel positions:
    dx, dy, valid as [peaks][ny][nx]."""
    (wx, wy), (nx, ny) = g.w, g.n
    w1, w2 = g.windows(e1), g.windows(e2)
    rows = max(1, int(2.5e7 // (nx * wx * wy)))
    out = []
    for r0 in range(0, ny, rows):
        a, b = w1[r0:r0 + rows], w2[r0:r0 + rows]
        m = a.shape[0]
        dead = (a.sum((2, 3)) == 0) | (b.sum((2, 3)) == 0)
        c = torch.fft.irfft2(torch.conj(torch.fft.rfft2(a)) * torch.fft.rfft2(b), s=(wy, wx)).abs()
        c = torch.where(dead[:, :, None, None], 0.0, torch.roll(c, (wy // 2, wx // 2), (2, 3)))
        by, bx = g.border[1], g.border[0]
        y0, y1, x0, x1 = max(by, 1), min(wy - by, wy - 1), max(bx, 1), min(wx - bx, wx - 1)
        mid = c[:, :, y0:y1, x0:x1]
        top = ((mid > 0) & (mid >= c[:, :, y0:y1, x0 - 1:x1 - 1]) & (mid >= c[:, :, y0:y1, x0 + 1:x1 + 1]) &
               (mid >= c[:, :, y0 - 1:y1 - 1, x0:x1]) & (mid >= c[:, :, y0 + 1:y1 + 1, x0:x1]))
        v, at = torch.where(top, mid, -1.0).reshape(m, nx, -1).topk(peaks, 2)
        j, i = y0 + at // (x1 - x0), x0 + at % (x1 - x0)
        flat = c.reshape(m, nx, wy * wx)

        def part(step):
            q = j * wx + i
            f0, fm, fp = (flat.gather(2, q + d) for d in (0, -step, step))
            return (torch.log(fm) - torch.log(fp)) / torch.log(fm / f0 * (fp / f0)) * 0.5

        dx = i + part(1) - wx / 2 + px[r0:r0 + m].unsqueeze(2)
        dy = j + part(wx) - wy / 2 + py[r0:r0 + m].unsqueeze(2)
        ok = (v > 0) & torch.isfinite(dx) & torch.isfinite(dy) & (dx.abs() <= 100) & (dy.abs() <= 100)
        out.append((torch.where(ok, dx, 0.0), torch.where(ok, dy, 0.0), ok))
        del a, b, c, flat, mid, top
    return tuple(torch.cat(t).permute(2, 0, 1).contiguous() for t in zip(*out))


def _shifted(f, r, fill):
    """[(2r+1)^2][ny][nx] neighbours in raster order."""
    ny, nx = f.shape
    p = torch.full((ny + 2 * r, nx + 2 * r), fill, dtype=f.dtype, device=f.device)
    p[r:r + ny, r:r + nx] = f
    return torch.stack([p[a:a + ny, b:b + nx] for a in range(2 * r + 1) for b in range(2 * r + 1)])


def _median(v, n):
    """Median of the n finite values along dimension 0 (the rest is +inf)."""
    s = v.sort(0).values
    hi = s.gather(0, (n // 2).clamp_max(len(s) - 1).unsqueeze(0))[0]
    lo = s.gather(0, (n // 2 - 1).clamp_min(0).unsqueeze(0))[0]
    return torch.where(n % 2 == 1, hi, 0.5 * (hi + lo))


def _validate(cand, thr=2.0, passes=2, least=5):
    """Normalised median test (5x5), hole fill, 3x3 mean; also how many vectors the test rejected."""
    cx, cy, ok = cand
    fx, fy, fv = cx[0], cy[0], ok[0]
    for _ in range(passes):
        nv = _shifted(fv, 2, False)
        nv[12] = False
        n = nv.sum(0)
        gx, gy = (torch.where(nv, _shifted(f, 2, 0.0), math.inf) for f in (fx, fy))
        mx, my = _median(gx, n), _median(gy, n)
        sx, sy = _median(torch.where(nv, (gx - mx).abs(), math.inf), n), _median(torch.where(nv, (gy - my).abs(), math.inf), n)
        good = ok & ((cx - mx).abs() / (sx + 0.1) < thr) & ((cy - my).abs() / (sy + 0.1) < thr) & (n >= least)
        first = good.to(torch.uint8).argmax(0).unsqueeze(0)
        fv = good.any(0)
        fx, fy = (torch.where(fv, c.gather(0, first)[0], 0.0) for c in (cx, cy))
    rejected = int((~fv).sum())
    while not bool(fv.all()):
        nv = _shifted(fv, 1, False)
        n = nv.sum(0)
        new = ~fv & (n > 0)
        if not bool(new.any()):
            break
        fx, fy = (torch.where(new, (_shifted(f, 1, 0.0) * nv).sum(0) / n.clamp_min(1), f) for f in (fx, fy))
        fv = fv | new
    n = _shifted(torch.ones_like(fx), 1, 0.0).sum(0)
    return _shifted(fx, 1, 0.0).sum(0) / n, _shifted(fy, 1, 0.0).sum(0) / n, fv, rejected


def _upsample(g1, g2, f):
    dev = f.device
    X = torch.arange(g2.n[0], device=dev, dtype=D) * g2.s[0] + g2.s[0] // 2
    Y = torch.arange(g2.n[1], device=dev, dtype=D) * g2.s[1] + g2.s[1] // 2
    return _bilinear(f, g1, X, Y, g1.s[0] // 2 - 3 * g1.s[0], g1.s[1] // 2 - 3 * g1.s[1])


def _exact_pair(c, seed):
    f1, f2 = _frames(c, seed)
    if c["mhe"]:
        f1, f2 = _mhe(f1, 40, 0.91), _mhe(f2, 40, 0.91)
    g1, g2 = _Grid(c, "1"), _Grid(c, "2")
    i2 = f2.to(D)
    if c["kind"] == "learned":
        fx, fy = _predicted(g1, f1, f2)
    else:
        e1, e2 = g1.extent(f1.to(D)), g1.extent(i2)
        fx = torch.zeros((g1.n[1], g1.n[0]), dtype=D, device=f1.device)
        fy = fx.clone()
        for j in range(c["n1"]):
            d = e2 if j == 0 else _deform(i2, g1, fx, fy)
            fx, fy, fv, _ = _validate(_candidates(g1, e1, d, fx, fy))
    fx, fy = _upsample(g1, g2, fx), _upsample(g1, g2, fy)
    px, py, rejected = fx, fy, 0
    e1 = g2.extent(f1.to(D))
    for _ in range(c["n2"]):
        fx, fy, fv, rejected = _validate(_candidates(g2, e1, _deform(i2, g2, fx, fy), fx, fy))
    X = (torch.arange(g2.n[0]) * g2.s[0] + g2.s[0] // 2).repeat(g2.n[1])
    Y = (torch.arange(g2.n[1]) * g2.s[1] + g2.s[1] // 2).repeat_interleave(g2.n[0])
    out = {"x": X.to(D), "y": Y.to(D), "dx": fx.reshape(-1), "dy": fy.reshape(-1), "valid": fv.to(torch.uint8).reshape(-1)}
    if c["kind"] == "learned":
        rms = float(torch.sqrt(((px - fx) ** 2 + (py - fy) ** 2).mean()))
        frac = rejected / (g2.n[0] * g2.n[1])
        out.update(fell_back=not (frac <= 0.05 and rms <= 0.5), reject_frac=frac, rms_px=rms)
    return out


def _weights(flat):
    """(weight, bias) of the layers of a flat parameter vector; weights rounded to BF16, as the
    network defines them."""
    out, o = [], 0
    for ci, co, _, _ in LAYERS:
        w, b = flat[o:o + co * ci * 9], flat[o + co * ci * 9:o + co * (ci * 9 + 1)]
        o += co * (ci * 9 + 1)
        out.append((w.to(torch.bfloat16).to(D).view(co, ci, 3, 3).requires_grad_(), b.to(D).requires_grad_()))
    return out


def _net(ws, x):
    def conv(k, x):
        y = torch.nn.functional.conv2d(x, ws[k][0], ws[k][1], stride=LAYERS[k][2], padding=1)
        return y if k == 12 else torch.nn.functional.leaky_relu(y, 0.1)

    def up(a, b):
        a = a.repeat_interleave(2, 2).repeat_interleave(2, 3)[:, :, :b.shape[2], :b.shape[3]]
        return torch.cat([a, b], 1)

    t2 = conv(1, conv(0, x))
    t4 = conv(3, conv(2, t2))
    t6 = conv(5, conv(4, t4))
    t8 = conv(7, conv(6, t6))
    t10 = conv(9, conv(8, up(t8, t6)))
    return conv(12, conv(11, up(conv(10, up(t10, t4)), t2)))


def _predicted(g, f1, f2):
    """The predictor's grid-1 field: cost volume of the 4x box averages, network, times 4."""
    dev = f1.device
    raw = np.fromfile(PKG / "weights" / "predictor.bin", np.float32, offset=16)
    ws = _weights(torch.from_numpy(raw).to(dev))
    H4, W4 = f1.shape[0] // 4, f1.shape[1] // 4
    d = [f[:4 * H4, :4 * W4].to(D).view(H4, 4, W4, 4).mean((1, 3)) / 255 for f in (f1, f2)]
    M = 64
    d = [torch.nn.functional.pad(v - v.mean(), (M, M, M, M)) for v in d]
    wd = [v // 4 for v in g.w]
    at = [((torch.arange(g.n[i], device=dev) * g.s[i] - g.left[i] + g.w[i] // 2 + 2) >> 2) - wd[i] // 2 + M
          for i in range(2)]
    cols = (at[0].view(-1, 1) + torch.arange(wd[0], device=dev)).view(1, g.n[0], 1, wd[0])
    rows = (at[1].view(-1, 1) + torch.arange(wd[1], device=dev)).view(g.n[1], 1, wd[1], 1)
    a = d[0][rows, cols]
    e = (a * a).sum((2, 3)) * (d[1][rows, cols] ** 2).sum((2, 3))
    sc = torch.where(e > 0, 1 / torch.sqrt(e), 0.0)
    cv = torch.stack([(a * d[1][rows + dy, cols + dx]).sum((2, 3)) * sc
                      for dy in range(-4, 5) for dx in range(-4, 5)])
    with torch.no_grad():
        out = 4 * _net(ws, cv.unsqueeze(0))[0]
    return out[0], out[1]


def _exact_train(case, seed):
    net = P.PredictorNet(seed=1 + seed % 97)  # only its initial weights, an input of the pass
    flat = torch.from_numpy(net.params()).to(_device())
    net.close()
    x, label, mask = _training_batch(case, seed)
    ws = _weights(flat)
    loss = 0.0
    n = float(mask.sum())
    for k in range(0, case["N"], 16):
        e = _net(ws, x[k:k + 16].to(D)) - label[k:k + 16].to(D)
        part = ((torch.sqrt(e * e + 1e-4) - 0.01) * mask[k:k + 16].to(D).unsqueeze(1)).sum() / n
        part.backward()
        loss += float(part)
    return {"loss": loss, "grads": torch.cat([t.grad.reshape(-1) for w in ws for t in w])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "mhe":
        return _mhe(_frames(case, seed)[0], case["ws"], case["thresh"])
    if kind == "batch":
        return [_exact_pair(c, seed * 64 + k) for k, c in enumerate(_batch_pairs(case))]
    return _exact_pair(case, seed)
