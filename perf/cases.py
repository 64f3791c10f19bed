"""Workloads that the speed of this framework is judged by: image pairs and
volume pairs through ``PIV``, the field clean-up that follows it, and a batch
plan's replay.  Sizes, windows and displacement fields are those of the
benchmark (``bench.py``, ``multi_quickpiv_b200/synth.py``) or of the package's
defaults; images are synthetic particle images, rendered on the GPU.

A case is a dict of plain values:

    kind      "pair" (one PIV call), "clean" (PIV with SN, then remove_low_SN
              and average), "batch" (one replay of a batch plan)
    shape     image or volume extents; alg, IS, SM, step, passes, SN, dtype:
              PIV's parameters (passes > 1: multi-pass refinement); th: the
              skip threshold
    mask      masked NSQECC with an ellipse mask
    order     "F": the images are column-major, as the kernels read them and
              as frames come from Julia; "C": plain torch tensors
    flow      displacement field: "shift", "vortex" or "shear"
    pairs     (batch) how many pairs the plan holds
"""
import math
import random

import numpy as np
import torch

import multi_quickpiv_b200 as mq
from multi_quickpiv_b200 import postprocessing as post
from multi_quickpiv_b200.batch import BatchPlan

BASE = dict(kind="pair", alg="nsqecc", IS=32, SM=16, step=16, passes=1, SN=False, dtype="float32", th=-1.0,
            mask=False, order="F", flow="vortex", pairs=1, h=0, w=0, d=0)


def _case(**kw):
    c = dict(BASE)
    c.update(kw)
    return c


def listed():
    return [
        # a small double-precision pair, as an interactive user or a test sends: launches and host work count
        _case(name="pair256_fft_f64", h=256, w=256, alg="fft", th=0.0, dtype="float64", flow="shift"),
        # a camera frame with the package's default parameters (interSize 32, margin 10, no overlap) in a plain tensor
        _case(name="frame512_default", h=512, w=512, SM=10, step=32, order="C"),
        # an ordinary camera frame at half-window overlap
        _case(name="frame1280_nsqecc", h=1024, w=1280, order="C"),
        # the benchmark's pair: dense vectors on a large frame
        _case(name="frame2048_nsqecc", h=2048, w=2048, step=8),
        # a measured field with its clean-up: SN ratios, low-SN vectors removed, smoothed
        _case(name="clean2048_sn", kind="clean", h=2048, w=2048, SN=True),
        # a cropped frame: odd extents, windows off the powers of two; ZNCC
        _case(name="ragged1501_zncc", h=1501, w=1999, alg="zncc", IS=24, SM=10, step=12),
        # a frame with a body or a wall masked out
        _case(name="masked1024", h=1024, w=1024, mask=True, flow="shift"),
        # three-pass refinement, windows halving from 64 to 16
        _case(name="refine1536_3pass", h=1536, w=2048, IS=16, SM=8, step=8, passes=3),
        # large displacements in one pass: the largest windows
        _case(name="window256", h=2048, w=2048, IS=128, SM=64, step=32),
        # the benchmark's volume pair
        _case(name="volume512_fft", h=512, w=512, d=256, alg="fft", flow="shear"),
        # a small volume refined over two passes
        _case(name="volume160_2pass", h=160, w=160, d=160, IS=16, SM=8, step=8, passes=2, flow="shear"),
        # a plan over mixed pairs, replayed: 2D and 3D, every algorithm, masks, three passes
        _case(name="batch_mixed", kind="batch", pairs=16, passes=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    order = rng.choice(["F", "C"])
    alg = rng.choice(["fft", "zncc", "nsqecc", "nsqecc"])
    kind = rng.choice(["frame", "frame", "frame", "frame", "clean", "mask", "refine", "large", "volume", "volume",
                       "refine3d", "batch"])
    dtype = "float64" if rng.random() < 0.15 else "float32"
    if kind in ("frame", "clean"):
        IS = rng.choice([16, 24, 31, 32, 32, 32])
        SM = rng.choice([IS // 4, IS // 3, IS // 2])
        step = rng.choice([IS // 4, IS // 2, IS])
        return _case(kind="clean" if kind == "clean" else "pair", h=_log_int(rng, 256, 2048), w=_log_int(rng, 256, 2048),
                     alg="nsqecc" if kind == "clean" and alg == "zncc" else alg, IS=IS, SM=SM, step=step, SN=kind == "clean" or rng.random() < 0.3, dtype=dtype,
                     th=rng.choice([-1.0, 0.0]), order=order, flow=rng.choice(["shift", "vortex"]))
    if kind == "mask":
        return _case(h=_log_int(rng, 512, 1536), w=_log_int(rng, 512, 1536), mask=True, flow="shift", order=order,
                     IS=rng.choice([16, 32]), SM=rng.choice([8, 12, 16]))
    if kind == "refine":
        IS = rng.choice([8, 16])
        return _case(h=_log_int(rng, 512, 2048), w=_log_int(rng, 512, 2048), alg=alg, IS=IS, SM=IS // 2, step=IS // 2,
                     passes=rng.choice([2, 3]), order=order)
    if kind == "large":
        IS = rng.choice([64, 96, 128])
        return _case(h=_log_int(rng, 768, 2048), w=_log_int(rng, 768, 2048), alg=alg, IS=IS,
                     SM=rng.choice([IS // 4, IS // 2]), step=rng.choice([IS // 4, IS // 2]), order=order)
    if kind == "volume":
        IS = rng.choice([16, 24, 32])
        return _case(h=_log_int(rng, 96, 320), w=_log_int(rng, 96, 320), d=_log_int(rng, 64, 192), alg=alg, IS=IS,
                     SM=IS // 2, step=rng.choice([IS // 2, IS]), SN=rng.random() < 0.3, order=order, flow="shear")
    if kind == "refine3d":
        IS = rng.choice([8, 16])
        return _case(h=_log_int(rng, 96, 192), w=_log_int(rng, 96, 192), d=_log_int(rng, 96, 160), alg=alg, IS=IS,
                     SM=IS // 2, step=IS // 2 if IS == 16 else IS, passes=2, order=order, flow="shear")
    return _case(kind="batch", pairs=rng.randint(6, 16), passes=rng.choice([1, 2, 3]))


# ---------------------------------------------------------------------------
# synthetic particle images
# ---------------------------------------------------------------------------
def _flow(pos, shape, flow):
    """Displacement per frame at `pos` (n, nd)."""
    nd = len(shape)
    if flow == "vortex" and nd == 2:  # Lamb-Oseen, core 200 px, peak 6 px
        r = pos - (torch.tensor(shape, dtype=pos.dtype, device=pos.device) - 1) / 2
        rr = r.norm(dim=1).clamp_min(1e-9)
        ut = 6.0 / 0.638 * (200.0 / rr) * (1 - torch.exp(-(rr / 200.0) ** 2))
        return torch.stack([ut * r[:, 1] / rr, -ut * r[:, 0] / rr], 1)
    d = torch.tensor([2.3, -1.7] if nd == 2 else [1.5, -0.8, 0.6], dtype=pos.dtype, device=pos.device).repeat(len(pos), 1)
    if flow == "shear":
        d[:, 0] += 0.01 * pos[:, -1]
    return d


def _render(shape, pos, peak, sigma):
    """Sum of Gaussian spots, in 64 bits.  Spots are added as whole numbers
    (units of 2^-20), so the sum does not depend on the order of additions."""
    nd = len(shape)
    R = int(math.ceil(4 * sigma))
    offs = torch.arange(-R, R + 1, device=pos.device)
    out = torch.zeros(int(np.prod(shape)), dtype=torch.int64, device=pos.device)
    for a in range(0, len(pos), 1 << 16):
        c, pk = pos[a:a + (1 << 16)], peak[a:a + (1 << 16)]
        base = c.floor().long()
        w = pk.view((-1,) + (1,) * nd)
        lin, ok = 0, True
        for d in range(nd):
            at = (base[:, d:d + 1] + offs).view([-1] + [len(offs) if k == d else 1 for k in range(nd)])
            w = w * torch.exp(-(at - c[:, d].view([-1] + [1] * nd)) ** 2 / (2 * sigma * sigma))
            ok = ok & (at >= 0) & (at < shape[d])
            lin = lin * shape[d] + at.clamp(0, shape[d] - 1)
        v = torch.where(ok, (w * (1 << 20)).round().long(), torch.zeros((), dtype=torch.int64, device=pos.device))
        out.index_add_(0, lin.reshape(-1), v.reshape(-1))
    return out.view(shape).double() / (1 << 20)


def _ordered(t, order):
    if order == "C":
        return t.contiguous()
    perm = tuple(range(t.dim() - 1, -1, -1))
    return t.permute(perm).contiguous().permute(perm)


def _images(shape, flow, dtype, order, mask, seed):
    """(img1, img2, mask or None) on the GPU."""
    g = torch.Generator().manual_seed(seed)
    nd = len(shape)
    density, sigma = (0.02, 1.2) if nd == 2 else (0.005, 1.0)
    size = torch.tensor(shape, dtype=torch.float64)
    n = int(density * float((size + 16).prod()))
    pos = (torch.rand((n, nd), generator=g, dtype=torch.float64) * (size + 16) - 8).cuda()
    peak = (500 + 500 * torch.rand(n, generator=g, dtype=torch.float64)).cuda()
    gain = 0.8 + 0.4 * torch.rand(2, generator=g, dtype=torch.float64)
    gc = torch.Generator(device="cuda").manual_seed(seed + 1)
    imgs = []
    for k in range(2):
        img = _render(shape, pos + _flow(pos, shape, flow) * k, peak, sigma)
        if flow == "vortex":  # uneven lighting
            img = (img + torch.linspace(0, 300, shape[1], dtype=torch.float64, device="cuda")) * float(gain[k])
        img += 10 * torch.randn(shape, generator=gc, dtype=torch.float64, device="cuda")
        imgs.append(_ordered(img.to(getattr(torch, dtype)), order))
    m = None
    if mask:
        m = torch.ones(shape, dtype=torch.bool, device="cuda")  # 1 = measured; bodies are left out
        for _ in range(5):
            c, ax = torch.rand(nd, generator=g), 0.08 + 0.16 * torch.rand(nd, generator=g)
            q = 0
            for d in range(nd):
                x = torch.arange(shape[d], device="cuda") / shape[d]
                q = q + (((x - float(c[d])) / float(ax[d])) ** 2).view([-1 if k == d else 1 for k in range(nd)])
            m &= q > 1
        m = _ordered(m.to(imgs[0].dtype), order)
    return imgs[0], imgs[1], m


def _shape(case):
    return (case["h"], case["w"], case["d"]) if case["d"] else (case["h"], case["w"])


def _params(case):
    nd = 3 if case["d"] else 2
    return mq.setPIVParameters(corr_alg=case["alg"], interSize=(case["IS"],) * nd, searchMargin=(case["SM"],) * nd,
                               step=(case["step"],) * nd, multipass=case["passes"], refine=case["passes"] > 1,
                               computeSN=case["SN"], threshold=case["th"], ndims=nd,
                               mask_threshold=0.5 if case["mask"] else -1.0)


def _members(case):
    """The pairs of a batch case, as cases: the benchmark's mix on smaller images."""
    rng = random.Random(case["pairs"] * 10 + case["passes"])
    out = []
    for i in range(case["pairs"]):
        IS = (8, 16, 16, 32)[i % 4]
        vol = i % 4 == 1
        mask = i % 4 == 3
        out.append(_case(h=_log_int(rng, 96, 128) if vol else _log_int(rng, 384, 1024),
                         w=_log_int(rng, 96, 128) if vol else _log_int(rng, 384, 1024),
                         d=_log_int(rng, 96, 128) if vol else 0, alg="nsqecc" if mask else ("fft", "zncc", "nsqecc")[i % 3],
                         IS=8 if vol else IS, SM=4 if vol else IS // 2, step=8 if vol else IS // 2, mask=mask,
                         passes=min(case["passes"], 2) if IS == 32 or vol else case["passes"], flow="shift"))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        pairs = []
        for i, m in enumerate(_members(case)):
            a, b, k = _images(_shape(m), m["flow"], m["dtype"], m["order"], m["mask"], seed * 1000 + i)
            pairs.append((a, b, _params(m)) + ((k,) if k is not None else ()))
        return {"plan": BatchPlan(pairs)}
    a, b, k = _images(_shape(case), case["flow"], case["dtype"], case["order"], case["mask"], seed * 1000)
    return {"args": (a, b) + ((k,) if k is not None else ()) + (_params(case),), "clean": case["kind"] == "clean"}


def run(state):
    if "plan" in state:
        state["plan"].run()
        return [VF for VF, _ in state["plan"].results()]
    VF, SN = mq.PIV(*state["args"])
    if state["clean"]:
        kept = post.remove_low_SN(SN, 1.2, VF)
        return VF, SN, kept, post.average(2, kept)
    return (VF,) if SN is None else (VF, SN)


# ---------------------------------------------------------------------------
# work and 64-bit values
# ---------------------------------------------------------------------------
def _field(shape, IS, step):
    return [max(0, (s - IS) // step + 1) for s in shape]


def _work(case):
    shape = _shape(case)
    nd, px = len(shape), 1
    for s in shape:
        px *= s
    size = 8 if case["dtype"] == "float64" else 4
    nbytes = px * size * (3 if case["mask"] else 2)
    flops = 0.0
    for level in range(case["passes"]):
        IS, SM, step = (case[k] << level for k in ("IS", "SM", "step"))
        ia = math.prod(_field(shape, IS, step))
        n, P = float((IS + 2 * SM) ** nd), float((2 * SM + 1) ** nd)
        half = n / (IS + 2 * SM) * ((IS + 2 * SM) // 2 + 1)
        # two real transforms forward, one back, the product, the similarity of every lag
        corr = 3 * 2.5 * n * math.log2(n) + 6 * half
        flops += ia * (corr * (2 if case["mask"] else 1) + (1 if case["alg"] == "fft" else 13) * P + 2 * IS ** nd)
        if level == 0:
            nbytes += ia * 8 * (nd + (1 if case["SN"] else 0))
            if case["kind"] == "clean":
                nbytes += 2 * ia * 8 * nd
                flops += ia * 25 * nd
    return {"bytes": nbytes, "flops": flops}


def work(case):
    parts = [_work(m) for m in _members(case)] if case["kind"] == "batch" else [_work(case)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def _axis(vf, step, IS, SM, size, shift):
    """Window geometry of every vector along one axis (src/utils/piv_ops.jl:38-76, 1-based there)."""
    T = 1 + vf * step
    vT, vB = T + shift, T + IS - 1 + shift
    top, bot = (vT - SM).clamp_min(1), (vB + SM).clamp_max(size)
    tlf, brb = (SM - 1 - vT).clamp_min(0), (vB + SM - size).clamp_min(0)
    return T - 1, top - 1 - tlf, tlf, tlf + (bot - top + 1).clamp_min(0), tlf, brb  # ir, g0, lo, hi, tlf, brb


def _windows(img, starts, lo, hi, length):
    """img[start + p] for p in [lo, hi) of every window and axis, 0 elsewhere."""
    nd, n = img.dim(), len(starts[0])
    p = torch.arange(length, device=img.device)
    idx, ok = [], True
    for d in range(nd):
        view = [n] + [length if k == d else 1 for k in range(nd)]
        idx.append((starts[d][:, None] + p).clamp(0, img.shape[d] - 1).view(view))
        ok = ok & ((p >= lo[d][:, None]) & (p < hi[d][:, None])).view(view)
    return img[tuple(idx)] * ok, ok


def _box(x, IS, P):
    """Sums over windows of IS per axis at the first P offsets."""
    for d in range(1, x.dim()):
        c = torch.cumsum(x, d)
        c = torch.cat([torch.zeros_like(c.narrow(d, 0, 1)), c], d)
        x = c.narrow(d, IS, P) - c.narrow(d, 0, P)
    return x


def _at(v, idx, P):
    """v (n, P, ..., P) at idx (list of (n,) per axis)."""
    lin = 0
    for i in idx:
        lin = lin * P + i
    return v.reshape(len(v), -1).gather(1, lin[:, None])[:, 0]


def _exact_pass(a, b, mask, case, level, prev):
    nd, shape = a.dim(), a.shape
    IS, SM, step = (case[k] << level for k in ("IS", "SM", "step"))
    vf, SS, P = _field(shape, IS, step), IS + 2 * SM, 2 * SM + 1
    n, dev = math.prod(vf), a.device
    VF = torch.zeros((n, nd), dtype=torch.float64, device=dev)
    SNv = torch.zeros(n, dtype=torch.float64, device=dev)
    dims = range(1, nd + 1)
    chunk = max(1, (1 << 25) // SS ** nd)
    for i0 in range(0, n, chunk):
        ia, v = torch.arange(i0, min(n, i0 + chunk), device=dev), []
        r = ia
        for d in range(nd):  # column-major
            v.append(r % vf[d])
            r = r // vf[d]
        shift = [torch.zeros_like(ia)] * nd
        if prev is not None:  # the nearest coarse vector, rounded, kept inside the image
            pv, pVF = prev
            near = [((2 * v[d] * step + IS - 1 - (2 * IS - 1) + 2 * step) // (4 * step)).clamp(0, pv[d] - 1)
                    for d in range(nd)]
            lin = 0
            for d in reversed(range(nd)):
                lin = lin * pv[d] + near[d]
            p = pVF[lin].nan_to_num(0.0, 0.0, 0.0)
            p = (p.sign() * (p.abs() + 0.5).floor()).long()
            shift = [torch.minimum(torch.maximum(p[:, d], -v[d] * step), shape[d] - IS - v[d] * step) for d in range(nd)]
        ax = [_axis(v[d], step, IS, SM, shape[d], shift[d]) for d in range(nd)]
        ir, g0, lo, hi, tlf, brb = ([x[k] for x in ax] for k in range(6))
        zero, full = [torch.zeros_like(ia)] * nd, [torch.full_like(ia, IS)] * nd
        F, _ = _windows(a, ir, zero, full, IS)
        G, ok = _windows(b, g0, lo, hi, SS)
        skip = (F.amax(tuple(dims)) < case["th"]) if case["th"] >= (1e-300 if case["mask"] else 0) else torch.zeros_like(ia, dtype=torch.bool)
        alg = case["alg"]
        if mask is not None:
            M, _ = _windows(mask, ir, zero, full, IS)
            skip = skip | (M.amax(tuple(dims)) < 0.5)
            F = F * M
            sumF = (F * F / torch.where(M > 0, M, torch.ones_like(M))).sum(tuple(dims))
        else:
            if alg == "zncc":
                F = F - F.mean(tuple(dims), keepdim=True)
                G = (G - G.sum(tuple(dims), keepdim=True) / ok.sum(tuple(dims), keepdim=True)) * ok
            sumF = (F * F).sum(tuple(dims))

        def corr(x, y):
            X, Y = torch.fft.rfftn(x, (SS,) * nd, tuple(dims)), torch.fft.rfftn(y, (SS,) * nd, tuple(dims))
            return torch.fft.irfftn(X.conj() * Y, (SS,) * nd, tuple(dims))[(slice(None),) + (slice(0, P),) * nd]

        c = corr(F, G)
        if alg != "fft" or mask is not None:
            S = corr(M, G * G).abs() if mask is not None else _box(G * G, IS, P).clamp_min(0)
            sF = sumF.view((-1,) + (1,) * nd)
            den = S.sqrt() * sF.sqrt()
            c = c / den if alg == "zncc" and mask is None else den / (den + sF + S - 2 * c)
        q, inp, ins, length = torch.arange(P, device=dev), True, True, 1.0
        for d in range(nd):
            view = [len(ia)] + [P if k == d else 1 for k in range(nd)]
            above, last = q >= tlf[d][:, None], 2 * SM - brb[d][:, None]
            inp = inp & (above & (q <= last)).view(view)
            ins = ins & (above & (q <= last - 1)).view(view)
            length = length * (2 * SM - brb[d] - tlf[d]).double()
        top = torch.where(ins, c, torch.full_like(c, -math.inf)).amax(tuple(dims))
        total = torch.where(ins, c, torch.zeros_like(c)).sum(tuple(dims))
        sn = top / ((total - top) / (length - 1))
        # the first maximum above 0 in column-major order: the axes reversed, then the first of the flat order
        w = torch.where(inp & (c > 0), c, torch.full_like(c, -math.inf)).permute([0] + list(reversed(dims))).reshape(len(ia), -1)
        best = w.amax(1, keepdim=True)
        first = torch.where(w == best, torch.arange(w.shape[1], device=dev), w.shape[1]).amin(1)
        has = best[:, 0] > 0
        first = torch.where(has, first, torch.zeros_like(first))
        peak = [(first // P ** d) % P for d in range(nd)]
        inside = has.clone()
        for d in range(nd):
            inside &= (peak[d] > tlf[d]) & (peak[d] < 2 * SM - brb[d])
        mid = [x.clamp(1, P - 2) if P > 2 else x * 0 for x in peak]
        near, lowest = {}, None
        for o in np.ndindex(*(3,) * nd):
            off = [k - 1 for k in o]
            val = _at(c, [(mid[d] + off[d]).clamp(0, P - 1) for d in range(nd)], P)
            lowest = val if lowest is None else torch.minimum(lowest, val)
            if sum(map(abs, off)) <= 1:
                near[tuple(off)] = val
        l0 = torch.log(1 + near[(0,) * nd] - lowest)
        for d in range(nd):
            unit = [int(k == d) for k in range(nd)]
            lm, lp = (torch.log(1 + near[tuple(s * u for u in unit)] - lowest) for s in (-1, 1))
            pos = peak[d] + torch.where(inside, (lm - lp) / (2 * lm - 4 * l0 + 2 * lp), torch.zeros_like(lm))
            pos = torch.where(has, pos, torch.full_like(pos, -1.0)) - SM + shift[d]
            VF[ia, d] = torch.where(skip, torch.zeros_like(pos), pos)
        SNv[ia] = torch.where(skip, torch.zeros_like(sn), sn)
    return vf, VF, SNv


def _exact_piv(case, images):
    a, b = images[0].double(), images[1].double()
    m = images[2].double() if images[2] is not None else None
    prev = None
    for level in reversed(range(case["passes"])):
        vf, VF, SN = _exact_pass(a, b, m, case, level, prev)
        prev = (vf, VF)
    nd = len(vf)
    back = list(reversed(range(nd)))
    VF = VF.view(list(reversed(vf)) + [nd]).permute([nd] + back)  # column-major vectors, component first
    return VF, SN.view(list(reversed(vf))).permute(back)


def _exact_average(VF, radius):
    n, total = torch.zeros_like(VF[0]), torch.zeros_like(VF)
    H, W = VF.shape[1:]
    for i in range(-radius, radius + 1):
        for j in range(-radius, radius + 1):
            to = (slice(max(0, -i), min(H, H - i)), slice(max(0, -j), min(W, W - j)))
            src = (slice(max(0, i), min(H, H + i)), slice(max(0, j), min(W, W + j)))
            total[(slice(None),) + to] += VF[(slice(None),) + src]
            n[to] += 1
    return total / n


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_piv(m, _images(_shape(m), m["flow"], m["dtype"], m["order"], m["mask"], seed * 1000 + i))[0]
                for i, m in enumerate(_members(case))]
    VF, SN = _exact_piv(case, _images(_shape(case), case["flow"], case["dtype"], case["order"], case["mask"], seed * 1000))
    if case["kind"] == "clean":
        kept = torch.where((SN < 1.2)[None], torch.zeros_like(VF), VF)
        return VF, SN, kept, _exact_average(kept, 2)
    return (VF, SN) if case["SN"] else (VF,)
