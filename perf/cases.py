"""The library's work as its users run it: which calls, on which sizes, with which data.

Every case goes through the package's public entry points (opencliper_gb300.api): the
reconstructions without iteration (SimpleMRIRecon, SimpleMRIReconSOS), the operator processes a
caller's own solver is built from, the tTV-NESTA solve on phase-encode masks and on pixel masks,
alone, in a batch behind one CUDA graph and with motion compensation, and the motion estimate.

A solve here runs up to 20 inner iterations per continuation step.  A clinical run takes 100; the
iteration is the same, but past about 30 of them FP32 rounding alone moves the image by more than
FP32 resolution (two summation orders of the same algorithm part by 7e-5 after 50 and 8e-4 after
100 iterations of the 256 x 256 x 20 workload), so that results could no longer be compared.

`exact` restates each path in torch, in 64 bits, from the reference's published algorithm.
"""
import math

import numpy as np
import torch

import opencliper_gb300 as g
from opencliper_gb300 import api, synth

DEV = "cuda:0"
SEED48 = (0x330E, 0xABCD, 0x1234)  # drand48's own start, so that every solve draws the same restart vector

_ctx = None


def context():
    """One context for the process, as a program has it."""
    global _ctx
    if _ctx is None:
        _ctx = g.Context(0)
    return _ctx


# ---- which cases -----------------------------------------------------------------------------

def listed():
    return [
        # one fully sampled image, the smallest call there is (8 coils, 256 x 256)
        {"name": "recon_256x256c8", "kind": "simple", "W": 256, "H": 256, "F": 1, "C": 8},
        # a cine series without coil maps: backward FFT and root sum of squares; a ragged size
        {"name": "sos_192x160x20c12", "kind": "sos", "W": 192, "H": 160, "F": 20, "C": 12},
        # E and E^H of the benchmark's series, what a caller's own solver iterates on
        {"name": "encode_256x256x20c12", "kind": "encode", "W": 256, "H": 256, "F": 20, "C": 12, "R": 8.0},
        # the FFT process on whole KData, there and back, the largest matrix of the configurations
        {"name": "fft_384x384x30c4", "kind": "fft", "W": 384, "H": 384, "F": 30, "C": 4},
        # the element-wise processes one by one: temporal TV, normalisation, coil product, mask, sum
        {"name": "operators_224x200x16c10", "kind": "operators", "W": 224, "H": 200, "F": 16, "C": 10},
        # a small solve with the reference driver's rules (continuation, stopping test, statistics)
        {"name": "nesta_64x48x6c4", "kind": "nesta", "W": 64, "H": 48, "F": 6, "C": 4, "R": 4.0, "mask": "rows",
         "loops": 2, "iters": 15, "stop": 1},
        # the benchmark's reconstruction
        {"name": "nesta_256x256x20c12", "kind": "nesta", "W": 256, "H": 256, "F": 20, "C": 12, "R": 8.0,
         "mask": "rows", "loops": 1, "iters": 20, "stop": 0},
        # the largest single reconstruction of the configurations
        {"name": "nesta_384x384x30c16", "kind": "nesta", "W": 384, "H": 384, "F": 30, "C": 16, "R": 8.0,
         "mask": "rows", "loops": 1, "iters": 20, "stop": 0},
        # sampling that varies along the readout (a pixel mask): the row transforms are needed
        {"name": "pixmask_240x224x12c8", "kind": "nesta", "W": 240, "H": 224, "F": 12, "C": 8, "R": 6.0,
         "mask": "pixels", "loops": 1, "iters": 20, "stop": 0},
        # uneven reconstructions of one scanner queue, solved together by one graph launch
        {"name": "batch_uneven8", "kind": "batch", "iters": 20,
         "members": "128x128x30x20x6,192x192x27x29x9,256x256x16x12x8,256x256x24x8x5,"
                    "320x320x20x16x5,384x384x12x12x8,128x128x40x21x4,192x192x26x32x6"},
        # the motion-compensated solve of the benchmark's series
        {"name": "motion_256x256x20c12", "kind": "motion", "W": 256, "H": 256, "F": 20, "C": 12, "R": 8.0,
         "iters": 20},
        # the motion estimate that feeds it, with the reference driver's parameters
        {"name": "registration_256x20", "kind": "registration", "W": 256, "H": 256, "F": 20, "radius": 40,
         "nmax": 100},
    ]


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


# the FFT process's lengths, from 24 on: row masks sample 16 central rows at least
LENGTHS = [n for n in range(24, 513, 8) if _smooth(n)]
MOST = 384 * 384 * 30 * 16 * 20.0  # pixel-coil-frame-iterations of the largest listed solve


def _size(rng, lo, hi):
    """A supported length, spread over the logarithm."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((n for n in LENGTHS if lo <= n <= hi), key=lambda n: abs(n - want))


def _int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.499)))))))


def draw(rng):
    kind = rng.choice(["simple", "sos", "encode", "fft", "operators", "nesta", "nesta", "nesta", "nesta", "batch",
                       "motion", "registration"])
    while True:
        W, H = _size(rng, 24, 512), _size(rng, 32, 512)
        F, C = _int(rng, 3, 40), _int(rng, 1, 32)
        vol = float(W) * H * F * C
        if kind == "simple":
            F = 1 if rng.random() < 0.5 else F
            c = {"kind": kind, "W": W, "H": H, "F": F, "C": C}
        elif kind in ("sos", "fft", "operators"):
            c = {"kind": kind, "W": W, "H": H, "F": F, "C": C}
        elif kind == "encode":
            c = {"kind": kind, "W": W, "H": H, "F": F, "C": C, "R": round(rng.uniform(2, 10), 1)}
        elif kind == "nesta":
            stop = 1 if rng.random() < 0.3 else 0
            c = {"kind": kind, "W": W, "H": H, "F": F, "C": C, "R": round(rng.uniform(4, 10), 1),
                 "mask": "pixels" if rng.random() < 0.3 else "rows", "loops": 2 if stop else 1,
                 "iters": rng.randint(8, 15 if stop else 20), "stop": stop}
            vol *= c["iters"] * c["loops"] * (2 if c["mask"] == "pixels" else 1)
        elif kind == "batch":
            mem, vol, it = [], 0.0, rng.randint(8, 20)
            sizes = [(_size(rng, 48, 384), _size(rng, 48, 384)) for _ in range(3)]
            for _ in range(rng.randint(2, 9)):
                (w, h), f, cc = rng.choice(sizes), _int(rng, 4, 40), _int(rng, 2, 32)
                mem.append("%dx%dx%dx%dx%d" % (w, h, f, cc, rng.randint(4, 10)))
                vol += float(w) * h * f * cc * it
            c = {"kind": kind, "iters": it, "members": ",".join(mem)}
        elif kind == "motion":
            W, H = max(W, 64), max(H, 64)
            c = {"kind": kind, "W": W, "H": H, "F": F, "C": C, "R": round(rng.uniform(4, 10), 1),
                 "iters": rng.randint(8, 20)}
            vol = 2.0 * W * H * F * C * c["iters"]
        else:
            N = 8 * rng.randint(12, 48)
            c = {"kind": kind, "W": N, "H": N, "F": F, "radius": rng.randint(N // 8, N // 4),
                 "nmax": rng.randint(20, 100)}
            vol = float(N) * N * F * 20
        if vol <= MOST * (1.0 if kind in ("nesta", "batch", "motion") else 0.1):
            return c


# ---- inputs ----------------------------------------------------------------------------------

def _gen(seed, salt=0):
    r = torch.Generator(device=DEV)
    r.manual_seed(int(seed) * 64 + salt)
    return r


def _uni(r, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(shape, generator=r, device=DEV, dtype=torch.float64)


def _series(W, H, F, r):
    """A beating phantom [F][H][W]: ten ellipses that move over 20 frames, under a smooth phase."""
    sc = min(W, H) / 256.0
    n = 10
    cx, cy = _uni(r, 0.15, 0.85, n) * W, _uni(r, 0.15, 0.85, n) * H
    ax, ay = _uni(r, 10, 80, n) * sc, _uni(r, 10, 80, n) * sc
    rot, amp, ph = _uni(r, 0, math.pi, n), _uni(r, 0.2, 1.0, n), _uni(r, 0, 2 * math.pi, n)
    k = torch.randn(6, generator=r, device=DEV, dtype=torch.float64)
    u = torch.linspace(-1, 1, W, device=DEV, dtype=torch.float64)[None, :]
    v = torch.linspace(-1, 1, H, device=DEV, dtype=torch.float64)[:, None]
    phi = k[0] + k[1] * u + k[2] * v + k[3] * u * u + k[4] * u * v + k[5] * v * v
    phi = (phi - phi.min()) / (phi.max() - phi.min()).clamp_min(1e-12) * 2 * math.pi - math.pi
    yy = torch.arange(H, device=DEV, dtype=torch.float64)[None, :, None]
    xx = torch.arange(W, device=DEV, dtype=torch.float64)[None, None, :]
    f = torch.arange(F, device=DEV, dtype=torch.float64)
    img = torch.zeros(F, H, W, device=DEV)
    for e in range(n):
        wob = (5.0 * sc * torch.sin(2 * math.pi * f / 20.0 + ph[e]))[:, None, None]
        dx, dy = xx - (cx[e] + wob), yy - (cy[e] + wob)
        c, s = torch.cos(rot[e]), torch.sin(rot[e])
        a, b = (ax[e] + wob).clamp_min(1.0), (ay[e] + wob).clamp_min(1.0)
        img += (amp[e] * (((c * dx + s * dy) / a) ** 2 + ((c * dy - s * dx) / b) ** 2 <= 1.0)).float()
    return img * torch.polar(torch.ones_like(phi), phi).to(torch.complex64)


def _coils(W, H, C):
    """C Gaussian coils on a circle around the field of view, sum_c |S_c|^2 = 1."""
    fov = float(min(W, H))
    ang = 2 * math.pi * torch.arange(C, device=DEV, dtype=torch.float64) / C
    px, py = W / 2 + 0.5 * fov * torch.cos(ang), H / 2 + 0.5 * fov * torch.sin(ang)
    yy = torch.arange(H, device=DEV, dtype=torch.float64)[None, :, None]
    xx = torch.arange(W, device=DEV, dtype=torch.float64)[None, None, :]
    e = -((xx - px[:, None, None]) ** 2 + (yy - py[:, None, None]) ** 2) / (2 * (0.4 * fov) ** 2)
    m = torch.exp(e - e.amax(0, keepdim=True))
    m = m / m.square().sum(0, keepdim=True).sqrt()
    return torch.polar(m, ang[:, None, None].expand(m.shape).contiguous()).to(torch.complex64).contiguous()


def _mask(W, H, F, R, seed, pixels):
    """Phase-encode rows with variable density and 16 central rows; `pixels`: of the rows outside
    the centre only part of the readout is sampled."""
    rm = synth.row_masks(H, F, R, np.random.default_rng(seed))
    m = torch.from_numpy((rm.astype(np.uint8) * 255)).to(DEV)[:, :, None].expand(F, H, W).contiguous()
    if pixels:
        keep = torch.rand((F, H, W), generator=_gen(seed, 7), device=DEV) < 0.6
        keep[:, :8] = True
        keep[:, H - 8:] = True
        m = m * keep
    return m.contiguous()


def _kspace(x, S, r, norm="ortho"):
    """FFT2(S_c x_f) plus complex noise of 1e-3 of its maximum, frame by frame."""
    F, (C, H, W) = x.shape[0], S.shape
    y = torch.empty((F, C, H, W), dtype=torch.complex64, device=DEV)
    for f in range(F):
        y[f] = torch.fft.fft2(x[f][None] * S, norm=norm)
    top = 1e-3 * float(torch.view_as_real(y).square().sum(-1).max().sqrt()) / math.sqrt(2)
    for f in range(F):
        y[f] += top * torch.view_as_complex(torch.randn((C, H, W, 2), generator=r, device=DEV))
    return y


def _data(c, seed):
    """x, S, mask and y of a sampled acquisition."""
    r = _gen(seed)
    W, H, F, C = c["W"], c["H"], c["F"], c["C"]
    x, S = _series(W, H, F, r), _coils(W, H, C)
    m = _mask(W, H, F, c["R"], seed, c.get("mask") == "pixels")
    y = _kspace(x, S, r)
    for f in range(F):
        y[f] *= (m[f] != 0)
    return x, S, m, y


def _members(c):
    for i, t in enumerate(c["members"].split(",")):
        W, H, F, C, R = (int(v) for v in t.split("x"))
        yield i, {"W": W, "H": H, "F": F, "C": C, "R": float(R), "mask": "rows", "iters": c["iters"], "loops": 1,
                  "stop": 0}


def _arr(t):
    """The library's view of a tensor."""
    dt = {torch.complex64: np.complex64, torch.uint8: np.uint8, torch.float32: np.float32,
          torch.int32: np.int32}[t.dtype]
    return api.DeviceArray(context(), tuple(t.shape), dt, ptr=t.data_ptr())


class _View:
    """An array the library returned, for torch.as_tensor: the tensor holds on to it, and so to the memory."""

    def __init__(self, d):
        self.array = d
        self.__cuda_array_interface__ = {"shape": d.shape, "typestr": d.dtype.str, "data": (d.ptr, False),
                                         "version": 3, "strides": None}


def _tensor(d):
    return torch.as_tensor(_View(d), device=DEV)


def _params(c):
    return dict(lambda_i=0.01, mu_f=1e-3, La=1.0, maxIntIter=c.get("loops", 1), tolVar=3e-4, maxIter=c["iters"],
                stoptest=c.get("stop", 0), miniter=7)


def _motion(c, seed):
    xn, xm, bb = synth.make_motion(c["W"], c["H"], c["F"], seed=seed)
    return torch.from_numpy(xn).to(DEV), torch.from_numpy(xm).to(DEV), [int(v) for v in bb]


def prepare(case, seed):
    c, ctx = case, context()
    kind = c["kind"]
    s = {"kind": kind, "case": c, "keep": []}

    def give(**tensors):
        for k, t in tensors.items():
            s["keep"].append(t)
            s[k + "_t"], s[k] = t, _arr(t)

    def empty(*shape):
        return torch.zeros(shape, dtype=torch.complex64, device=DEV)

    if kind in ("simple", "sos", "fft"):
        W, H, F, C = c["W"], c["H"], c["F"], c["C"]
        r = _gen(seed)
        S = _coils(W, H, C)
        give(y=_kspace(_series(W, H, F, r), S, r, "backward"), S=S)
        if kind == "fft":
            give(a=empty(F, C, H, W), b=empty(F, C, H, W))
        else:
            give(x=empty(F, H, W))
    elif kind == "encode":
        x, S, m, _ = _data(c, seed)
        give(x=x.contiguous(), S=S, m=m, k=empty(c["F"], c["C"], c["H"], c["W"]), z=empty(*x.shape))
    elif kind == "operators":
        W, H, F, C = c["W"], c["H"], c["F"], c["C"]
        r = _gen(seed)
        x, S = _series(W, H, F, r), _coils(W, H, C)
        x = x + 0.05 * torch.view_as_complex(torch.randn((F, H, W, 2), generator=r, device=DEV))
        m = _mask(W, H, F, 4.0, seed, True)
        give(x=x.contiguous(), S=S, m=m)
        give(d=empty(F, H, W), u=empty(F, H, W), v=empty(F, H, W), k=empty(F, C, H, W), q=empty(F, C, H, W),
             z=empty(F, H, W), a=empty(F, H, W))
    elif kind == "nesta":
        _, S, m, y = _data(c, seed)
        give(y=y, S=S, m=m, x=empty(c["F"], c["H"], c["W"]))
        s["problem"] = g.Problem(ctx, s["y"], s["S"], s["m"])
        s["params"] = g.nesta_params(**_params(c))
    elif kind == "batch":
        probs, prms, s["outs"] = [], [], []
        for i, mc in _members(c):
            _, S, m, y = _data(mc, seed * 16 + i)
            x = empty(mc["F"], mc["H"], mc["W"])
            s["keep"] += [S, m, y, x]
            s["outs"].append(x)
            probs.append(g.Problem(ctx, _arr(y), _arr(S), _arr(m)))
            prms.append(g.nesta_params(**_params(mc)))
        torch.cuda.synchronize()
        s["batch"] = g.Batch(ctx, probs, prms, [_arr(x) for x in s["outs"]])
        s["batch"].capture()
    elif kind == "motion":
        _, S, m, y = _data(c, seed)
        x0 = (torch.fft.ifft2(y, norm="ortho") * S.conj()[None]).sum(1).contiguous()
        xn, xm, bb = _motion(c, seed)
        give(y=y, S=S, m=m, x0=x0, x=torch.zeros_like(x0), xn=xn, xm=xm)
        s["problem"] = g.Problem(ctx, s["y"], s["S"], s["m"])
        s["problem"].set_motion(s["xn"], s["xm"], bb)
        s["params"] = g.nesta_params(**_params(c))
        s["stream"] = torch.cuda.ExternalStream(ctx.stream)
    else:
        r = _gen(seed)
        x = _series(c["W"], c["H"], c["F"], r)
        x = x + 0.01 * torch.view_as_complex(torch.randn(x.shape + (2,), generator=r, device=DEV))
        give(x=x.contiguous())
        s["params"] = g.registration_params(radius=c["radius"], nmax=c["nmax"])
    torch.cuda.synchronize()  # the library works on its own stream
    return s


# ---- the calls -------------------------------------------------------------------------------

def run(state):
    s, ctx, kind = state, context(), state["kind"]
    if kind == "simple":
        api.simple_recon(ctx, s["y"], s["S"], s["x"])
        return s["x_t"]
    if kind == "sos":
        api.simple_recon_sos(ctx, s["y"], s["x"])
        return s["x_t"]
    if kind == "fft":
        api.op_fft2(ctx, -1, s["y"], s["a"])
        api.op_fft2(ctx, 1, s["a"], s["b"])
        return {"forward": s["a_t"], "back": s["b_t"]}
    if kind == "encode":
        api.op_encode(ctx, s["x"], s["S"], s["m"], s["k"])
        api.op_encode_adjoint(ctx, s["k"], s["S"], s["z"])
        return {"k": s["k_t"], "x": s["z_t"]}
    if kind == "operators":
        api.op_ttv(ctx, 1, s["x"], s["d"])
        api.op_normalize(ctx, s["d"], s["u"], 0.03)
        api.op_ttv(ctx, 0, s["u"], s["v"])
        api.op_sensmul(ctx, False, s["x"], s["S"], s["k"])
        api.op_mask(ctx, s["k"], s["m"])
        api.op_sensmul(ctx, True, s["k"], s["S"], s["q"])
        api.op_coilsum(ctx, s["q"], s["z"])
        api.op_rss(ctx, s["k"], s["a"])
        return {n: s[n + "_t"] for n in ("d", "u", "v", "k", "q", "z", "a")}
    if kind == "nesta":
        ctx.seed48(SEED48)
        if not s["case"]["stop"]:
            s["problem"].run(s["params"], s["x"], stats=False)
            return s["x_t"]
        st = s["problem"].run(s["params"], s["x"])
        return {"x": s["x_t"], "inner_iters": st["inner_iters"], "kept_rows": st["kept_rows"],
                "normU": st["normU"]}
    if kind == "batch":
        ctx.seed48(SEED48)
        s["batch"].launch()
        return s["outs"]
    if kind == "motion":
        ctx.seed48(SEED48)
        with torch.cuda.stream(s["stream"]):
            s["x_t"].copy_(s["x0_t"])  # the image of the loop before
        s["problem"].run(s["params"], s["x"], stats=False)
        return s["x_t"]
    r = api.registration(ctx, s["x"], s["params"])
    return {"T": _tensor(r["T"]), "xn": _tensor(r["xn"]), "xmesh": _tensor(r["xmesh"]), "H": r["H"],
            "iterations": r["iterations"]}


# ---- what a pass cannot do without -----------------------------------------------------------

def work(case):
    c = case
    if c["kind"] == "batch":
        w = [work(dict(m, kind="nesta")) for _, m in _members(c)]
        return {"bytes": sum(v["bytes"] for v in w), "flops": sum(v["flops"] for v in w)}
    N, F, C = c["W"] * c["H"], c["F"], c.get("C", 1)
    K, X, S = 8.0 * N * F * C, 8.0 * N * F, 8.0 * N * C
    fft = 5.0 * N * math.log2(N) * F * C
    if c["kind"] == "simple":
        return {"bytes": K + S + X, "flops": fft + 8.0 * N * F * C}
    if c["kind"] == "sos":
        return {"bytes": K + X, "flops": fft + 4.0 * N * F * C}
    if c["kind"] == "fft":
        return {"bytes": 4 * K, "flops": 2 * fft}
    if c["kind"] == "encode":
        return {"bytes": 2 * X + 2 * S + N * F + 2 * K, "flops": 2 * fft + 16.0 * N * F * C}
    if c["kind"] == "operators":
        # each call's inputs read and outputs written: ttv, normalise, ttv; product, mask, product, sum, rss
        return {"bytes": 6 * X + (X + S + K) + (2 * K + N * F) + (2 * K + S) + (K + X) + (K + X),
                "flops": 20.0 * N * F + 22.0 * N * F * C}
    if c["kind"] == "registration":
        box = (2.0 * c["radius"]) ** 2 * F
        return {"bytes": X + 2 * 4.0 * N * F + 2 * 4.0 * N, "flops": c["nmax"] * box * (2 * 32 + 3 * 12 + 2 * 20)}
    # a solve: the column transforms there and back in every iteration (both axes on pixel masks), the coil
    # products, the temporal TV and the update; inputs and the image move once
    axis = math.log2(N) if c.get("mask") == "pixels" else math.log2(c["H"])
    it = c["iters"] * c.get("loops", 1)
    flops = it * (2 * 5.0 * N * axis * F * C + 16.0 * N * F * C + 40.0 * N * F)
    byts = K + S + N * F + X
    if c["kind"] == "motion":
        byts += X + 2 * 4.0 * N * F + 2 * 4.0 * N
        flops += it * 60.0 * N * F
    return {"bytes": byts, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------------------

def _d(t):
    return t.to(torch.complex128)


def _drand48(n, skip):
    """n values of drand48 after `skip` draws from its own start, by doubling: X -> a X + c modulo 2^48."""
    M = (1 << 48) - 1
    a, c, x = 0x5DEECE66D, 0xB, SEED48[0] | SEED48[1] << 16 | SEED48[2] << 32
    ja, jc, k = a, c, skip + 1
    while k:
        if k & 1:
            x = (ja * x + jc) & M
        ja, jc, k = (ja * ja) & M, (ja * jc + jc) & M, k >> 1
    v, ja, jc = torch.tensor([x], dtype=torch.int64, device=DEV), a, c  # (ja, jc): the jump over len(v) draws
    while len(v) < n:
        v = torch.cat([v, (v * ja + jc) & M])  # modulo 2^64, which 2^48 divides
        ja, jc = (ja * ja) & M, (ja * jc + jc) & M
    return v[:n].to(torch.float64) * 2.0 ** -48


def _warp_geometry(c, xn, xm, bb):
    W, H = c["W"], c["H"]
    m0, m1 = H // 40, W // 40
    rows = torch.arange(bb[1] - m0 - 2, bb[3] + m0 + 1, device=DEV)
    cols = torch.arange(bb[0] - m1 - 2, bb[2] + m1 + 1, device=DEV)
    nh = xn[0][:, rows[:, None], cols[None, :]].double() - 1
    nv = xn[1][:, rows[:, None], cols[None, :]].double() - 1
    ph, pv = torch.floor(nh).long(), torch.floor(nv).long()
    return rows, cols, ph, pv, nh - ph, nv - pv


def _operators(c, geo):
    """The sparsity operator U = D M and its adjoint (M the identity without motion)."""
    def D(x):
        return x - torch.roll(x, 1, 0)

    def Dt(d):
        return torch.roll(d, -1, 0) - d  # the reference's adjoint kernel: negated by its caller

    if geo is None:
        return D, Dt
    rows, cols, ph, pv, fh, fv = geo
    H, W, F = c["H"], c["W"], c["F"]
    fr = torch.arange(F, device=DEV)[:, None, None]
    four = [((fr * H + pv + b) * W + ph + a, (fh if a else 1 - fh) * (fv if b else 1 - fv)) for a in (0, 1) for b in (0, 1)]

    def M(x):
        out, flat = x.clone(), x.reshape(-1)
        out[:, rows[:, None], cols[None, :]] = sum(flat[i] * w for i, w in four)
        return out

    def Mt(v):
        out = v.clone()
        val = v[:, rows[:, None], cols[None, :]]
        out[:, rows[:, None], cols[None, :]] = 0
        flat = torch.view_as_real(out).reshape(-1, 2)
        for i, w in four:
            flat.index_add_(0, i.reshape(-1), torch.view_as_real((val * w).reshape(-1)))
        return out

    return lambda x: D(M(x)), lambda d: Mt(Dt(d))


def _norm_of(U, Ut, F, H, W, skip):
    """The reference's power method: all ones first, and drand48 where that maps to zero."""
    x = torch.ones((F, H, W), dtype=torch.complex128, device=DEV)
    e, e0, n = math.sqrt(F * H * W), 0.0, 0
    while abs(e - e0) > 1e-3 * e and n < 100:
        e0 = e
        v = U(x)
        if float(v.abs().sum()) <= 1e-9 * float(x.abs().sum()):
            v = _drand48(F * H * W, skip).float().double().reshape(F, H, W).to(torch.complex128)
        e = float(v.abs().square().sum().sqrt())
        x = Ut(v)
        x = x / float(x.abs().square().sum().sqrt())
        n += 1
    return e


def _solve(c, S, m, y, geo=None, x0=None, skip=0):
    """NESTA in 64 bits: (x, ||U||)."""
    p = _params(c)
    W, H, F = c["W"], c["H"], c["F"]
    S, keep = _d(S), m != 0
    U, Ut = _operators(c, geo)

    def adjoint(f, k):
        return (torch.fft.ifft2(k, norm="ortho") * S.conj()).sum(0)

    x = torch.stack([adjoint(f, _d(y[f])) for f in range(F)]) if x0 is None else _d(x0)
    top, topU = float(x.abs().max()), float(U(x).abs().max())
    lam, muf, mu = p["lambda_i"] * top, p["mu_f"] * top, 0.9 * topU
    normU = _norm_of(U, Ut, F, H, W, skip)
    mu = max(mu, lam / p["La"])
    gamma, gammat, tol = (muf / mu) ** (1.0 / p["maxIntIter"]), (p["tolVar"] / 0.1) ** (1.0 / p["maxIntIter"]), 0.1
    n, last = p["miniter"], [0.0] * p["miniter"]
    for _ in range(p["maxIntIter"]):
        mu, tol = mu * gamma, tol * gammat
        L1 = 1.0 / (lam * normU / mu + p["La"])
        xk, w, hit, k = x.clone(), torch.zeros_like(x), False, 0
        last[n - 1] = float(np.float32(2 ** 63))
        while k < p["maxIter"]:
            d = U(xk)
            u = d / d.abs().clamp_min(mu)
            df = -lam * Ut(u)
            l2 = 0.0
            for f in range(F):
                r = torch.fft.fft2(xk[f][None] * S, norm="ortho") * keep[f] - _d(y[f])
                l2 += float(torch.view_as_real(r).square().sum())
                df[f] += adjoint(f, r)
            if p["stoptest"]:
                fx = 0.5 * l2 + lam * (float((u.conj() * d).real.sum()) - 0.5 * mu * float(u.abs().square().sum()))
                stop = False
                if k >= n:
                    mean = sum(last) / n
                    if (mean - fx) / mean <= tol:
                        k, hit, stop = p["maxIter"] if hit else k, True, True
                if not stop:
                    last[(n - 1) - ((k + 1) % n)] = fx
            yk = xk - L1 * df
            w += 0.5 * (k + 1.0) * df
            t = 2.0 / (k + 3.0)
            xk = t * (x - L1 * w) + (1.0 - t) * yk
            k += 1
        x = xk
    return x, normU


def _spline(v):
    """The reference's cubic B-spline, its constant 0.6666 included."""
    v = v.abs()
    return torch.where(v < 1, 0.5 * v ** 3 - v ** 2 + 0.6666, torch.where(v < 2, (2 - v) ** 3 / 6, torch.zeros_like(v)))


def _register(c, x):
    """Groupwise registration in 64 bits: gradient descent on the temporal variance inside a circle."""
    N, F, rad, Dp = c["W"], c["F"], c["radius"], 4
    pos = torch.arange(N, device=DEV, dtype=torch.float64)
    d2 = (pos + 1 - (N + 1) / 2) ** 2
    roi = (d2[:, None] + d2[None, :] <= rad * rad).double()
    inside = torch.nonzero(roi.amax(0)).reshape(-1)
    lo, hi = int(inside[0]), int(inside[-1])
    box = torch.arange(lo, hi + 1, device=DEV)
    L = hi - lo + 1
    mid = (lo + hi + 2) / 2
    C0 = math.floor((mid - (lo + 1) + 8) / Dp)
    Cp = C0 + math.floor((hi + 1 - mid + 8) / Dp) + 1
    arg = (pos + 1 - mid) / Dp
    kmin = torch.floor(arg).long() - 1
    first = kmin - kmin[lo + 1]
    R = torch.zeros(N, Cp, device=DEV, dtype=torch.float64)  # pixel -> its four control points
    for b in range(4):
        R[box, first[box] + b] = _spline(arg - (kmin + b))[box]
    P = torch.zeros(N, Cp, device=DEV, dtype=torch.float64)  # control point -> its 17-pixel support
    for n in range(Cp):
        q = torch.arange(17, device=DEV) + math.ceil(mid + Dp * (n - C0) - 8) - 1
        P[q, n] = _spline((q.double() + 1 - (mid + Dp * (n - C0))) / Dp)
    R, Pb, roib = R[box], P[box], roi[box][:, box]
    a = _d(x).abs()
    I = a * (500.0 / float(a.max()))
    g1, g2 = torch.empty_like(I), torch.empty_like(I)
    g1[:, :, 1:-1], g2[:, 1:-1] = (I[:, :, 2:] - I[:, :, :-2]) / 2, (I[:, 2:] - I[:, :-2]) / 2
    g1[:, :, 0], g1[:, :, -1] = I[:, :, 1] - I[:, :, 0], I[:, :, -1] - I[:, :, -2]
    g2[:, 0], g2[:, -1] = I[:, 1] - I[:, 0], I[:, -1] - I[:, -2]
    fr = torch.arange(F, device=DEV)[:, None, None]

    def at(img, h, v):
        ph, pv = torch.floor(h).long(), torch.floor(v).long()
        b, d, flat = h - ph, v - pv, img.reshape(-1)
        i = (fr * N + pv) * N + ph
        return (1 - d) * ((1 - b) * flat[i] + b * flat[i + 1]) + d * ((1 - b) * flat[i + N] + b * flat[i + N + 1])

    T = torch.zeros(2, F, Cp, Cp, device=DEV, dtype=torch.float64)

    def mesh():
        u = R @ T @ R.T
        return u[0] + box[None, None, :], u[1] + box[None, :, None]

    def cost(w):
        return float((w.var(0, unbiased=False) * roib).sum())

    w = I[:, box[:, None], box[None, :]]
    H = [cost(w)]
    step, tolT, tolH = 1.0 / float(roi.sum()), 0.01 * F * 2, H[0] * 0.005
    h, v = mesh()
    for it in range(1, c["nmax"] + 1):
        dy = (w - w.mean(0)) * (2.0 / F) * roib
        dH = torch.stack([Pb.T @ (dy * at(gd, h, v)) @ Pb for gd in (g1, g2)])
        dif = step * (dH - dH.mean(1, keepdim=True))
        T = T - dif
        h, v = mesh()
        w = at(I, h, v)
        H.append(cost(w))
        down = H[-2] - H[-1]
        step = step * 1.2 if down > 0 else step / 2
        if float(dif.square().sum().sqrt()) < tolT and down < tolH:
            break
    xn = torch.empty(2, F, N, N, device=DEV, dtype=torch.float64)
    xn[0], xn[1] = pos[None, None, :] + 1, pos[None, :, None] + 1
    xn[0][:, lo:hi + 1, lo:hi + 1], xn[1][:, lo:hi + 1, lo:hi + 1] = h + 1, v + 1
    return T, xn, H


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("simple", "sos", "fft"):
        W, H, F, C = c["W"], c["H"], c["F"], c["C"]
        r = _gen(seed)
        S = _coils(W, H, C)
        y = _kspace(_series(W, H, F, r), S, r, "backward")
        if kind == "simple":
            return torch.stack([(torch.fft.ifft2(_d(y[f])) * _d(S).conj()).sum(0) for f in range(F)])
        if kind == "sos":
            return torch.stack([torch.fft.ifft2(_d(y[f])).abs().square().sum(0).sqrt() + 0j for f in range(F)])
        return {"forward": torch.fft.fft2(_d(y)), "back": _d(y)}
    if kind == "encode":
        x, S, m, _ = _data(c, seed)
        k = torch.fft.fft2(_d(x)[:, None] * _d(S)[None], norm="ortho") * (m != 0)[:, None]
        return {"k": k, "x": (torch.fft.ifft2(k, norm="ortho") * _d(S).conj()[None]).sum(1)}
    if kind == "operators":
        s = prepare(c, seed)
        x, S, m = _d(s["x_t"]), _d(s["S_t"]), s["m_t"] != 0
        d = x - torch.roll(x, 1, 0)
        u = d / d.abs().clamp_min(float(np.float32(0.03)))
        k = x[:, None] * S[None] * m[:, None]
        q = k * S.conj()[None]
        return {"d": d, "u": u, "v": torch.roll(u, -1, 0) - u, "k": k, "q": q, "z": q.sum(1),
                "a": k.abs().square().sum(1).sqrt() + 0j}
    if kind == "nesta":
        _, S, m, y = _data(c, seed)
        x, e = _solve(c, S, m, y)
        return {"x": x, "inner_iters": None, "kept_rows": None, "normU": e} if c["stop"] else x
    if kind == "batch":
        out, skip = [], 0  # a member's restart vector follows the draws of the members before it
        for i, mc in _members(c):
            _, S, m, y = _data(mc, seed * 16 + i)
            out.append(_solve(mc, S, m, y, skip=skip)[0])
            skip += mc["W"] * mc["H"] * mc["F"]
        return out
    if kind == "motion":
        _, S, m, y = _data(c, seed)
        x0 = (torch.fft.ifft2(y, norm="ortho") * S.conj()[None]).sum(1)
        xn, xm, bb = _motion(c, seed)
        return _solve(c, S, m, y, _warp_geometry(c, xn, xm, bb), x0)[0]
    s = prepare(c, seed)
    T, xn, H = _register(c, s["x_t"])
    return {"T": T, "xn": xn, "xmesh": None, "H": np.array(H), "iterations": None}
