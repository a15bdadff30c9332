"""The workloads whose speed this framework is measured by.

A case is a dict of plain values.  `listed()` holds one case per kind of work that a program does
with the framework (an encode, a decode, a batch, a transform, a training step), at sizes from a
single small image to the largest one of its benchmark; `draw()` gives more cases of the same
ranges.  `prepare()` makes what such a program has in hand before the call, `run()` is one pass
through the public entry points, `work()` the bytes and operations that a pass cannot do without,
and `exact()` the 64-bit value of the outputs that are computed in floating point (every other
output is an integer or a byte and has to stay what it is).

Images are seeded sums of sinusoids plus Gaussian noise, 8 bits a sample, the channels of a colour
image correlated (the same distribution as roger_b200.synth, made on the GPU).
"""
import ctypes
import math

import numpy as np
import torch

from roger_b200 import _lib as L
from roger_b200 import batch, codec, diff97, synth

DEVICE = "cuda"
RD_SEED, RD_LAMBDA = 7, 0.01


# -- the cases -----------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: one gray tile handed over as a host array, its code-blocks read back
        dict(name="encode_gray_512", op="encode", w=512, h=512, ncomp=1, lossy=False, levels=5, cb=64, host=True,
             style=0, bpp=0.0),
        # the largest single image: a colour frame already on the GPU, coded without loss
        dict(name="encode_rgb_4096", op="encode", w=4096, h=4096, ncomp=3, lossy=False, levels=6, cb=64, host=False,
             style=0, bpp=0.0),
        # an ordinary photograph of odd size, irreversible transform, small code-blocks
        dict(name="encode_rgb_odd_lossy", op="encode", w=1999, h=1501, ncomp=3, lossy=True, levels=5, cb=32,
             host=False, style=0, bpp=0.0),
        # the same kind of image cut to a byte budget and written as a codestream
        dict(name="encode_rgb_rate", op="encode", w=2048, h=2048, ncomp=3, lossy=True, levels=5, cb=64, host=False,
             style=0, bpp=1.0),
        # every coding pass a segment of its own (contexts reset, codeword terminated)
        dict(name="encode_rgb_styled", op="encode", w=2048, h=2048, ncomp=3, lossy=False, levels=5, cb=64,
             host=False, style=L.CBLK_RESET | L.CBLK_TERMALL, bpp=0.0),
        # many images of uneven size through one batched encoder
        dict(name="batch_mixed", op="batch", n=256, lo=64, hi=2048, layout=300),
        # the largest decode, code-blocks on the host, pixels into a page-locked array
        dict(name="decode_rgb_4096", op="decode", w=4096, h=4096, ncomp=3, lossy=False, levels=6, cb=64),
        # a small gray image of odd size, dequantised
        dict(name="decode_gray_odd_lossy", op="decode", w=1237, h=989, ncomp=1, lossy=True, levels=5, cb=64),
        # many codestreams decoded by one call
        dict(name="decode_streams", op="streams", n=24, lo=64, hi=1024, layout=41),
        # the reversible transform of three planes, forward and back
        dict(name="dwt53_planes_4096", op="dwt", kernel=53, n=3, w=4096, h=4096, levels=6),
        # the irreversible one on planes of odd size
        dict(name="dwt97_planes_odd", op="dwt", kernel=97, n=3, w=2047, h=3001, levels=5),
        # one rate-distortion training step: the loss and its gradients
        dict(name="rd_step_1024", op="rd", n=16, w=1024, h=1024, levels=5),
    ]


def _log(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _levels(w, h, most):
    return max(1, min(most, int(math.log2(min(w, h))) - 3))


def draw(rng):
    op = rng.choice(["encode", "encode", "decode", "decode", "batch", "streams", "dwt", "rd"])
    if op in ("encode", "decode"):
        w, h = _log(rng, 64, 4096), _log(rng, 64, 4096)
        lossy = rng.random() < 0.5
        c = dict(op=op, w=w, h=h, ncomp=rng.choice([1, 3]), lossy=lossy, levels=_levels(w, h, 6),
                 cb=rng.choice([32, 64]))
        if op == "encode":
            way = rng.random()
            c.update(host=rng.random() < 0.3, style=L.CBLK_RESET | L.CBLK_TERMALL if way < 0.2 else 0,
                     bpp=round(rng.uniform(0.25, 2.0), 2) if way > 0.8 else 0.0)
        return c
    if op in ("batch", "streams"):
        return dict(op=op, n=rng.randint(4, 32 if op == "batch" else 24), lo=64, hi=rng.randint(256, 1024),
                    layout=rng.randint(1, 10 ** 6))
    if op == "dwt":
        w, h = _log(rng, 64, 4096), _log(rng, 64, 4096)
        return dict(op=op, kernel=rng.choice([53, 97]), n=rng.choice([1, 3]), w=w, h=h, levels=_levels(w, h, 6))
    if rng.random() < 0.5:
        w, h = 64 << rng.randint(0, 4), 64 << rng.randint(0, 4)
    else:
        w, h = _log(rng, 64, 1024), _log(rng, 64, 1024)
    return dict(op=op, n=rng.randint(1, 16), w=w, h=h, levels=_levels(w, h, 5))


# -- inputs --------------------------------------------------------------------------------------

def _field(w, h, rng):
    """A zero-mean sum of 8 sinusoids, evaluated separably."""
    theta, lam = rng.uniform(0.0, math.pi, 8), np.exp(rng.uniform(math.log(4.0), math.log(128.0), 8))
    amp, phi = rng.uniform(10.0, 40.0, 8), rng.uniform(0.0, 2.0 * math.pi, 8)
    kx, ky = 2.0 * math.pi * np.cos(theta) / lam, 2.0 * math.pi * np.sin(theta) / lam
    ax, ay = np.outer(kx, np.arange(w)) + phi[:, None], np.outer(ky, np.arange(h))
    left = np.concatenate([np.cos(ay), np.sin(ay)]).T
    right = np.concatenate([amp[:, None] * np.sin(ax), amp[:, None] * np.cos(ax)])
    return torch.from_numpy(left).to(DEVICE, torch.float32) @ torch.from_numpy(right).to(DEVICE, torch.float32)


def _image(w, h, ncomp, seed):
    """(h, w) or (h, w, 3) uint8 on the GPU."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    shared = _field(w, h, rng) if ncomp == 3 else None
    planes = []
    for _ in range(ncomp):
        f = _field(w, h, rng)
        if ncomp == 3:
            f = math.sqrt(0.8) * shared + math.sqrt(0.2) * f
        f = f + 128.0 + 6.0 * torch.randn(h, w, device=DEVICE, generator=g)
        planes.append(f.round_().clamp_(0, 255).to(torch.uint8))
    return planes[0] if ncomp == 1 else torch.stack(planes, dim=-1).contiguous()


def _set(case, seed):
    """The images of a batch, (descriptor, pixels on the GPU) each; the descriptors depend on the
    case alone."""
    descs = synth.mixed_set(case["n"], case["layout"], case["lo"], case["hi"])
    for d in descs:
        d["steps"] = codec.default_steps(d["w"], d["h"], d["levels"]) if d["kernel"] == 97 else None
    return descs, [_image(d["w"], d["h"], d["ncomp"], seed * 1000 + i) for i, d in enumerate(descs)]


def _pinned(shape):
    return torch.zeros(shape, dtype=torch.uint8, pin_memory=True).numpy()


def _sinks(blocks, samples):
    """Page-locked room for the descriptors and the codewords of an encode, which a program that
    calls the C interface hands in."""
    return dict(descs=_pinned(blocks * L.CB_DESC.itemsize), data=_pinned(samples * 5 // 4 + 65536))


def prepare(case, seed):
    op = case["op"]
    s = dict(case)
    if op == "encode":
        img = _image(case["w"], case["h"], case["ncomp"], seed)
        s.update(img=img.cpu().numpy() if case["host"] else img, enc=codec.OCLEncoder(lossy=case["lossy"]),
                 target=int(case["bpp"] * case["w"] * case["h"] / 8) + 1024 if case["bpp"] else 0)
        if case["bpp"]:
            s["stream"] = _pinned(s["target"])
        else:
            s.update(_sinks(case["ncomp"] * codec.codeblock_count(case["w"], case["h"], case["levels"], case["cb"],
                                                                  case["cb"]), case["w"] * case["h"] * case["ncomp"]))
    elif op == "decode":
        enc = codec.OCLEncoder(lossy=case["lossy"])
        enc.run_rgb(_image(case["w"], case["h"], case["ncomp"], seed), levels=case["levels"], cbw=case["cb"],
                    cbh=case["cb"])
        d, b = enc.get_codeblocks()
        s.update(descs=d, data=b, dec=codec.OCLDecoder(lossy=case["lossy"]),
                 out=_pinned((case["h"], case["w"], case["ncomp"])))
    elif op == "batch":
        descs, images = _set(case, seed)
        s.update(images=images, enc=batch.BatchEncoder(descs),
                 **_sinks(sum(d["ncomp"] * codec.codeblock_count(d["w"], d["h"], d["levels"], d["cb"], d["cb"])
                              for d in descs), sum(d["w"] * d["h"] * d["ncomp"] for d in descs)))
    elif op == "streams":
        descs, images = _set(case, seed)
        encs = {k: codec.OCLEncoder(lossy=k == 97) for k in (53, 97)}
        s["streams"] = []
        for d, im in zip(descs, images):
            e = encs[d["kernel"]].run_rgb(im, levels=d["levels"], cbw=d["cb"], cbh=d["cb"], steps=d["steps"])
            s["streams"].append(e.codestream())
        s["dec"] = codec.OCLDecoder()
    elif op == "dwt":
        px = [_image(case["w"], case["h"], 1, seed * 10 + k).to(torch.int32) - 128 for k in range(case["n"])]
        x = torch.stack(px)
        s["x"] = x if case["kernel"] == 53 else x.to(torch.float32)
    else:
        x, log_steps = _rd_inputs(case, seed, torch.float32)
        s.update(x=x.requires_grad_(True), log_steps=log_steps.requires_grad_(True))
    return s


def _rd_inputs(case, seed, dtype):
    x = torch.stack([_image(case["w"], case["h"], 1, seed * 100 + k).to(torch.float32) / 255.0
                     for k in range(case["n"])])
    log_steps = torch.full((3 * case["levels"] + 1,), math.log(1.0 / 64.0), dtype=torch.float32, device=DEVICE)
    return x.to(dtype), log_steps.to(dtype)


# -- one pass ------------------------------------------------------------------------------------

def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def run(s):
    op = s["op"]
    if op == "encode":
        enc, got = s["enc"], ctypes.c_size_t()
        enc.run_rgb(s["img"], levels=s["levels"], cbw=s["cb"], cbh=s["cb"], target_bytes=s["target"],
                    cblk_style=s["style"])
        if s["target"]:
            out = s["stream"]
            L.check(L.lib().j2k_encoder_get_codestream(enc.h, _ptr(out), out.size, ctypes.byref(got)), enc.ctx.h)
            return out, got.value
        count = ctypes.c_size_t(s["descs"].size // L.CB_DESC.itemsize)
        L.check(L.lib().j2k_encoder_get_codeblocks(enc.h, _ptr(s["descs"]), ctypes.byref(count), _ptr(s["data"]),
                                                   s["data"].size, ctypes.byref(got)), enc.ctx.h)
        out = s["descs"], s["data"], got.value
        return (*out, enc.get_pass_ends()) if s["style"] else out
    if op == "decode":
        return s["dec"].run(s["descs"], s["data"], s["w"], s["h"], s["ncomp"], levels=s["levels"], cbw=s["cb"],
                            cbh=s["cb"], out=s["out"])
    if op == "batch":
        enc, got = s["enc"], ctypes.c_size_t()
        enc.encode(s["images"])
        L.check(L.lib().j2k_batch_pack(enc.h, ctypes.byref(got)), enc.ctx.h)
        L.check(L.lib().j2k_batch_read_packed(enc.h, _ptr(s["descs"]), _ptr(s["data"]), s["data"].size), enc.ctx.h)
        enc.ctx.sync()
        return s["descs"], s["data"], got.value
    if op == "streams":
        return codec.decode_codestreams(s["streams"], decoder=s["dec"])
    if op == "dwt":
        y = codec.dwt_forward(s["x"], s["levels"])
        return y, codec.dwt_inverse(y, s["levels"])
    s["x"].grad = s["log_steps"].grad = None
    loss = diff97.rd_loss(s["x"], s["log_steps"], s["levels"], RD_LAMBDA, RD_SEED)
    loss.backward()
    return loss.detach(), s["x"].grad, s["log_steps"].grad


# -- what a pass cannot do without -----------------------------------------------------------------

# additions and multiplications per sample of one 2-D lifting transform over all levels
# (4/3 of one level; per level two 1-D passes, 5/3: 4 additions and 2 shifts per pair of samples,
# 9/7: 4 lifting steps of 2 additions and 1 multiplication per pair, 2 scalings)
DWT_OPS = {53: 4 / 3 * 2 * 3, 97: 4 / 3 * 2 * 7}
# codeword bytes per sample of these images, and coding decisions per codeword byte with the
# interval update and state transition of each (about 8 operations)
CODED = {False: 0.7, True: 0.55}
DECISION_OPS = 8.5 * 8


def _coded_work(w, h, ncomp, lossy):
    n = w * h * ncomp
    coded = CODED[lossy] * n
    return n + coded, n * DWT_OPS[97 if lossy else 53] + coded * DECISION_OPS


def work(case):
    op = case["op"]
    if op in ("encode", "decode"):
        b, f = _coded_work(case["w"], case["h"], case["ncomp"], case["lossy"])
    elif op in ("batch", "streams"):
        parts = [_coded_work(d["w"], d["h"], d["ncomp"], d["kernel"] == 97)
                 for d in synth.mixed_set(case["n"], case["layout"], case["lo"], case["hi"])]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif op == "dwt":
        n = case["n"] * case["w"] * case["h"]
        b, f = 16 * n, 2 * n * DWT_OPS[case["kernel"]]  # each direction reads and writes 4 bytes a sample
    else:
        n = case["n"] * case["w"] * case["h"]
        b, f = 8 * n, n * (4 * DWT_OPS[97] + 30)  # pixels in, their gradient out
    return dict(bytes=b, flops=f)


# -- the 64-bit values -----------------------------------------------------------------------------

_P1, _U1, _P2, _U2 = -1.586134342, -0.05298011854, 0.8829110762, 0.4435068522
_KM, _KD = 1.23017410491400, 0.81289306611596153187273657637352


def _split(x):
    return x[..., 0::2], x[..., 1::2]


def _to_odd(e, n):
    """Sum of the two even neighbours of every odd sample (whole-sample symmetric ends)."""
    right = e[..., 1:] if n % 2 else torch.cat([e[..., 1:], e[..., -1:]], -1)
    return e[..., :n // 2] + right


def _to_even(o, n):
    """Sum of the two odd neighbours of every even sample."""
    left = torch.cat([o[..., :1], o], -1)
    right = torch.cat([o, o[..., -1:]], -1) if n % 2 else o
    return left[..., :(n + 1) // 2] + right


def _fwd1(x):
    n = x.shape[-1]
    if n == 1:
        return x
    e, o = _split(x)
    o = o + _P1 * _to_odd(e, n)
    e = e + _U1 * _to_even(o, n)
    o = o + _P2 * _to_odd(e, n)
    e = e + _U2 * _to_even(o, n)
    return torch.cat([e * _KD, o * _KM], -1)


def _inv1(c):
    n = c.shape[-1]
    if n == 1:
        return c
    k = (n + 1) // 2
    e, o = c[..., :k] * _KM, c[..., k:] * _KD
    e = e - _U2 * _to_even(o, n)
    o = o - _P2 * _to_odd(e, n)
    e = e - _U1 * _to_even(o, n)
    o = o - _P1 * _to_odd(e, n)
    x = torch.stack([e[..., :n // 2], o], -1).flatten(-2)
    return torch.cat([x, e[..., -1:]], -1) if n % 2 else x


def _columns(f, x):
    return f(x.transpose(-1, -2)).transpose(-1, -2)


def _dwt64(x, levels):
    if levels == 0:
        return x
    y = _fwd1(_columns(_fwd1, x))
    h, w = (x.shape[-2] + 1) // 2, (x.shape[-1] + 1) // 2
    top = torch.cat([_dwt64(y[..., :h, :w], levels - 1), y[..., :h, w:]], -1)
    return torch.cat([top, y[..., h:, :]], -2)


def _idwt64(y, levels):
    if levels == 0:
        return y
    h, w = (y.shape[-2] + 1) // 2, (y.shape[-1] + 1) // 2
    top = torch.cat([_idwt64(y[..., :h, :w], levels - 1), y[..., :h, w:]], -1)
    return _columns(_inv1, _inv1(torch.cat([top, y[..., h:, :]], -2)))


def _noise64(case, seed):
    """The relaxed quantiser's uniform noise: Philox4x32-10 keyed by seed + image, one block per
    four samples of a row (counter row * ceil(w / 4) + column / 4), 24 bits a word."""
    n, h, w = case["n"], case["h"], case["w"]
    groups = (w + 3) // 4
    low = 0xFFFFFFFF

    def mul(a, c):  # high and low word of a 32 x 32 bit product, in 16-bit halves of a
        p0, p1 = (a & 0xFFFF) * c, (a >> 16) * c
        mid = (p0 >> 16) + p1
        return (mid >> 16) & low, ((mid << 16) | (p0 & 0xFFFF)) & low

    ctr = torch.arange(h * groups, device=DEVICE, dtype=torch.int64).expand(n, -1)
    key = seed + torch.arange(n, device=DEVICE, dtype=torch.int64)[:, None]
    c0, c1 = ctr & low, ctr >> 32
    c2, c3 = torch.zeros_like(c0), torch.zeros_like(c0)
    k0, k1 = key & low, key >> 32
    for _ in range(10):
        h0, l0 = mul(c0, 0xD2511F53)
        h1, l1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    words = torch.stack([c0, c1, c2, c3], -1).view(n, h, groups * 4)[:, :, :w]
    return (words >> 8).to(torch.float64) / 16777216.0 - 0.5


def _step_map(log_steps, w, h, levels):
    """exp(log_step) of the subband that each coefficient belongs to."""
    idx = torch.zeros(h, w, dtype=torch.int64, device=DEVICE)
    for b, (x0, y0, bw, bh, _, _) in enumerate(_rects(w, h, levels)):
        idx[y0:y0 + bh, x0:x0 + bw] = b
    return torch.exp(log_steps)[idx]


def _rects(w, h, levels):
    """(x0, y0, width, height, orientation, level) of the subbands: the lowest one, then HL, LH
    and HH from the deepest level up."""
    ws, hs = [w], [h]
    for _ in range(levels):
        ws.append((ws[-1] + 1) // 2)
        hs.append((hs[-1] + 1) // 2)
    out = [(0, 0, ws[levels], hs[levels], 0, levels)]
    for k in range(levels, 0, -1):
        out += [(ws[k], 0, ws[k - 1] - ws[k], hs[k], 1, k), (0, hs[k], ws[k], hs[k - 1] - hs[k], 2, k),
                (ws[k], hs[k], ws[k - 1] - ws[k], hs[k - 1] - hs[k], 3, k)]
    return out


def exact(case, seed):
    if case["op"] == "dwt" and case["kernel"] == 97:
        s = prepare(case, seed)
        y = _dwt64(s["x"].double(), case["levels"])
        return y, _idwt64(y, case["levels"])
    if case["op"] == "rd":
        x, log_steps = (v.requires_grad_(True) for v in _rd_inputs(case, seed, torch.float64))
        step = _step_map(log_steps, case["w"], case["h"], case["levels"])
        t = _dwt64(x, case["levels"]) / step + _noise64(case, RD_SEED)
        d = _idwt64(t * step, case["levels"]) - x
        loss = (d * d).mean() + RD_LAMBDA * torch.log2(1.0 + t.abs()).sum()
        loss.backward()
        return loss.detach(), x.grad, log_steps.grad
    return None
