"""The work a user of this library has it do, as measurable cases.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what the caller holds before the call, run() is one pass through the
public entry points, work() counts the bytes and operations the pass cannot do
without, and exact() restates the computed values in FP64 with plain torch.

Stacks are seeded phantoms: sums of 6-12 Gaussian blobs, each particle its
class phantom mirrored with p = 0.5, rotated, shifted and covered with white
noise, normalised inside the mask.
"""
import math
import os
import random
import sys

import numpy as np
import torch

for _d in (os.getcwd(), *sys.path[:1]):
    _pkg = os.path.join(_d, "gpu-isac_gb300")
    if os.path.isdir(_pkg) and _pkg not in sys.path:
        sys.path.insert(0, _pkg)

import gpuisac  # noqa: E402
from gpuisac import align, assign, averages, learned, multigroup, prealign  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # a handful of particles against a few class averages: what a call costs by itself
        dict(name="align_tiny", kind="align", P=8, R=4, D=64, rings=29, shift=2, mode="fp32", L=256),
        # the drop-in call on host pointer arrays at the CPU-runnable configuration (64 x 64, 16 references)
        dict(name="host_align_2000x64", kind="host", P=2000, R=16, D=64, rings=29, shift=2, mode="fp32", L=256),
        # one main iteration's alignment, FP32 (the default arithmetic)
        dict(name="align_3000x76_fp32", kind="align", P=3000, R=200, D=76, rings=35, shift=3, mode="fp32", L=256),
        # the same with the tensor-core contraction, over several particle chunks
        dict(name="align_5000x76_split", kind="align", P=5000, R=200, D=76, rings=35, shift=3, mode="bf16x3", L=256),
        # large box: 61 rings, 81 shifts in two shift blocks, 500 references
        dict(name="align_400x128_split", kind="align", P=400, R=500, D=128, rings=61, shift=4, mode="bf16x3", L=256),
        # 512-sample rings (Numrinit's longest ring at 61 rings)
        dict(name="align_300x128_ring512", kind="align", P=300, R=60, D=128, rings=61, shift=2, mode="fp32", L=512),
        # uneven groups, each with its own references, in one pass
        dict(name="groups_32", kind="groups", n=32, lo=100, hi=1000, rlo=10, rhi=60, D=76, rings=35, shift=3, layout=1),
        # learned proposal in front of the search, about five per cent of the particles falling back
        dict(name="learned_4000x200", kind="learned", P=4000, R=200, D=76, rings=35, shift=3, k=16),
        # one training step of the proposal network: forward, backward, AdamW
        dict(name="train_500x200", kind="train", P=500, R=200, rings=35),
        # pre-alignment of a stack against one average, two rounds
        dict(name="prealign_4000x76", kind="prealign", P=4000, D=76, rings=35, shift=5, rounds=2),
        # stability test: classes of at most 100 members, filtered averages, six iterations
        dict(name="stability_3000x76", kind="stability", P=3000, R=30, D=76, rings=35, shift=2, iters=6),
        # what follows the alignment: equal-size group assignment, then the averages
        dict(name="assign_average_20000", kind="average", P=20000, R=200, D=76),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["align", "align", "align", "host", "groups", "learned", "train", "prealign", "stability", "average"])
    D = _log(rng, 48, 128)
    rings = max(8, D // 2 - rng.randint(3, 8))
    if kind in ("align", "host"):
        shift = rng.randint(1, 4)
        mode, L = rng.choice([("fp32", 256), ("fp32", 256), ("bf16x3", 256), ("bf16x3", 256), ("fp32", 512)])
        if kind == "host":
            mode, L = rng.choice([("fp32", 256), ("bf16x3", 256)])
        R = _log(rng, 3, 500 if L == 256 else 60)
        cap = 7e8 if L == 256 else 2.5e7  # rows x rings: below the largest listed case
        P = _log(rng, 5, max(6, min(5000, cap / (R * (2 * shift + 1) ** 2 * rings))))
        return dict(kind=kind, P=P, R=R, D=D, rings=rings, shift=shift, mode=mode, L=L)
    if kind == "groups":
        return dict(kind=kind, n=rng.randint(2, 32), lo=20, hi=_log(rng, 100, 700), rlo=4, rhi=rng.randint(8, 50),
                    D=min(D, 90), rings=min(rings, 40), shift=rng.randint(1, 3), layout=rng.randrange(1 << 20))
    if kind == "learned":
        D, rings = min(D, 90), min(rings, 40)
        return dict(kind=kind, P=_log(rng, 200, 4000), R=_log(rng, 40, 200), D=D, rings=rings, shift=rng.randint(1, 3),
                    k=rng.choice([8, 16]))
    if kind == "train":
        return dict(kind=kind, P=_log(rng, 100, 2048), R=_log(rng, 20, 500), rings=rings)
    if kind == "prealign":
        return dict(kind=kind, P=_log(rng, 100, 4000), D=min(D, 90), rings=min(rings, 40), shift=rng.randint(2, 5),
                    rounds=rng.randint(1, 2))
    if kind == "stability":
        R = rng.randint(2, 30)
        return dict(kind=kind, P=R * rng.randint(10, 100) + rng.randint(0, 9), R=R, D=min(D, 90), rings=min(rings, 40),
                    shift=rng.randint(1, 2), iters=rng.randint(3, 6))
    return dict(kind=kind, P=_log(rng, 300, 20000), R=_log(rng, 4, 200), D=min(D, 100))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _render(amp, sig, cx, cy, D):
    c = torch.arange(D, device=DEV, dtype=torch.float32) - D // 2
    inv = 1.0 / (2.0 * sig**2)
    gx = torch.exp(-((c - cx[..., None]) ** 2) * inv[..., None])
    gy = torch.exp(-((c - cy[..., None]) ** 2) * inv[..., None]) * amp[..., None]
    return torch.bmm(gy.transpose(1, 2), gx)


def _normalise(x, mask):
    v = x[:, mask]
    mean = v.mean(1)
    sd = (v - mean[:, None]).square().mean(1).sqrt()
    return ((x - mean[:, None, None]) / (sd + 1e-12)[:, None, None]).contiguous()


def _stack(P, R, D, rings, shift, seed, cls=None, snr=0.05):
    """particles [P][D][D], references [R][D][D], the particles' classes"""
    g = _gen(seed)

    def uni(lo, hi, *n):
        return torch.rand(*n, generator=g, device=DEV) * (hi - lo) + lo

    nb = torch.randint(6, 13, (R, 1), generator=g, device=DEV)
    amp = uni(0.5, 1.0, R, 12) * (torch.arange(12, device=DEV)[None, :] < nb)
    sig = uni(2.0, 8.0, R, 12)
    rad, th = (rings - 1) * uni(0.0, 1.0, R, 12).sqrt(), uni(0.0, 2 * math.pi, R, 12)
    cx, cy = rad * torch.cos(th), rad * torch.sin(th)
    c = torch.arange(D, device=DEV) - D // 2
    mask = c[None, :] ** 2 + c[:, None] ** 2 <= rings**2
    refs = _normalise(_render(amp, sig, cx, cy, D), mask)
    if cls is None:
        cls = torch.randint(0, R, (P,), generator=g, device=DEV)
    t = uni(0.0, 2 * math.pi, P, 1)
    sh = torch.randint(-shift, shift + 1, (P, 2), generator=g, device=DEV).float()
    flip = torch.where(torch.rand(P, 1, generator=g, device=DEV) < 0.5, -1.0, 1.0)
    px, py = cx[cls] * flip, cy[cls]
    parts = _render(amp[cls], sig[cls], torch.cos(t) * px - torch.sin(t) * py + sh[:, :1],
                    torch.sin(t) * px + torch.cos(t) * py + sh[:, 1:], D)
    var = parts[:, mask].var(1, unbiased=False)
    parts += torch.randn(parts.shape, generator=g, device=DEV) * (var / snr).sqrt()[:, None, None]
    base = uni(-1.0, 1.0, P, 2)  # sub-pixel shifts left by the previous iteration
    return _normalise(parts, mask), refs, cls, base


def _group_table(case):
    rng = random.Random(case["layout"])
    tbl, po, ro = [], 0, 0
    for _ in range(case["n"]):
        p, r = _log(rng, case["lo"], case["hi"]), rng.randint(case["rlo"], case["rhi"])
        tbl.append((po, p, ro, r))
        po, ro = po + p, ro + r
    return tbl


def _class_sizes(P, R):
    return [P // R + (1 if i < P % R else 0) for i in range(R)]


def _train_inputs(case, seed):
    g = _gen(seed)
    n_in = case["rings"] * learned.NK
    par = learned.init_params(n_in, learned.HIDDEN, learned.EMB, seed)
    n = sum(v.size for v in par.values())
    Xr = torch.randn(case["R"], n_in, generator=g, device=DEV)
    lab = torch.randint(0, case["R"], (case["P"],), generator=g, device=DEV, dtype=torch.int32)
    X = 0.6 * Xr[lab.long()] + 0.8 * torch.randn(case["P"], n_in, generator=g, device=DEV)
    m = 1e-3 * torch.randn(n, generator=g, device=DEV)  # moments of a training under way
    v = 1e-5 * (0.5 + torch.rand(n, generator=g, device=DEV))
    return par, X.contiguous(), lab, Xr.contiguous(), m, v


def _average_inputs(case, seed):
    P, R = case["P"], case["R"]
    g = _gen(seed)
    parts, _, cls, _ = _stack(P, R, case["D"], case["D"] // 2 - 3, 3, seed)
    d = torch.randn(R, P, generator=g, device=DEV)
    d[cls, torch.arange(P, device=DEV)] += 3.0
    peak = torch.empty(R, P, 4, device=DEV)
    peak[..., 0] = torch.rand(R, P, generator=g, device=DEV) * 360.0
    peak[..., 1:3] = torch.randint(-3, 4, (R, P, 2), generator=g, device=DEV).float()
    peak[..., 1:3] += torch.rand(1, P, 2, generator=g, device=DEV) - 0.5
    peak[..., 3] = (torch.rand(R, P, generator=g, device=DEV) < 0.5).float()
    return parts, d, peak


def prepare(case, seed):
    k = case["kind"]
    if k in ("align", "host"):
        parts, refs, _, base = _stack(case["P"], case["R"], case["D"], case["rings"], case["shift"], seed)
        if k == "host":
            parts, refs, base = parts.cpu().numpy(), refs.cpu().numpy(), base.cpu().numpy()
        return dict(case=case, parts=parts, refs=refs, base=base)
    if k == "groups":
        tbl = _group_table(case)
        nr = tbl[-1][2] + tbl[-1][3]
        cls = torch.cat([ro + torch.arange(pn, device=DEV) % rn for _, pn, ro, rn in tbl])
        parts, refs, _, base = _stack(cls.numel(), nr, case["D"], case["rings"], case["shift"], seed, cls)
        return dict(case=case, parts=parts, refs=refs, base=base, table=tbl)
    if k == "learned":
        parts, refs, _, _ = _stack(case["P"], case["R"], case["D"], case["rings"], case["shift"], seed)
        net = learned.ProposalNet(case["rings"], seed=seed)
        net.set_feature_stats(learned.ring_features(parts[:256], case["rings"], net.nk))
        emb = learned.reference_embeddings(net, refs, case["rings"])
        # the margin below which a particle is searched against every reference:
        # a small share of the largest possible peak
        bound = 256.0**2 * sum(range(1, case["rings"] + 1))
        return dict(case=case, parts=parts, refs=refs, net=net, emb=emb, margin=1e-3 * bound)
    if k == "train":
        par, X, lab, Xr, m, v = _train_inputs(case, seed)
        net = learned.ProposalNet(case["rings"], seed=seed)
        net.load_params(par)
        net.m.copy_(m)
        net.v.copy_(v)
        net.step_count = 100
        return dict(case=case, net=net, X=X, lab=lab, Xr=Xr)
    if k == "prealign":
        parts, refs, _, _ = _stack(case["P"], 1, case["D"], case["rings"], 2, seed)
        return dict(case=case, parts=parts.cpu().numpy(), ref=refs[0].cpu().numpy())
    if k == "stability":
        sizes = _class_sizes(case["P"], case["R"])
        cls = torch.repeat_interleave(torch.arange(case["R"], device=DEV), torch.tensor(sizes, device=DEV))
        parts, refs, _, _ = _stack(case["P"], case["R"], case["D"], case["rings"], 1, seed, cls, snr=0.3)
        return dict(case=case, parts=parts.cpu().numpy(), cid=cls.cpu().numpy(), avg=refs.cpu().numpy())
    parts, d, peak = _average_inputs(case, seed)
    return dict(case=case, parts=parts, d=d, peak=peak)


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "align":
        d, pk = align.multi_ref_align_device(state["parts"], state["refs"], case["rings"], case["shift"], case["shift"],
                                             base_shifts=state["base"], contraction_mode=case["mode"],
                                             ring_len=case["L"])
        return {"d": d, "peak": pk}
    if k == "host":
        pl, d = gpuisac.multi_ref_align(state["parts"], state["refs"], case["rings"], case["shift"], case["shift"],
                                        base_shifts=state["base"], contraction_mode=case["mode"])
        return {"d": d, "peak": pl.reshape(case["R"], case["P"], 4)}
    if k == "groups":
        d, pk, _ = align.multi_ref_align_groups_device(state["parts"], state["refs"], state["table"], case["rings"],
                                                       case["shift"], case["shift"], base_shifts=state["base"])
        return {"d": d, "peak": pk}
    if k == "learned":
        r = learned.learned_align(state["parts"], state["refs"], state["net"], case["rings"], case["shift"],
                                  case["shift"], k=case["k"], gap_margin=state["margin"], ref_embed=state["emb"])
        return {"ref": r.ref, "peak": r.peak, "params": r.params, "gap": r.gap, "fallback": r.fallback}
    if k == "train":
        net = state["net"]
        loss = net.loss_and_grad(state["X"], state["lab"], state["Xr"])
        net.adam(1e-3, wd=1e-4)
        return {"loss": loss, "grad": net.grad, "weights": net.flat}
    if k == "prealign":
        return {"params": prealign.pre_align(state["parts"], state["ref"], case["rings"], case["shift"],
                                             rounds=case["rounds"])}
    if k == "stability":
        prm, avg = multigroup.multigroup_refinement(state["parts"], state["cid"], case["rings"], case["shift"],
                                                    case["shift"], case["iters"], cutoff_freq=0.3, falloff=0.2,
                                                    init_averages=state["avg"], return_averages=True)
        return {"params": prm, "averages": avg}
    ids, bel, _ = assign.assign_groups_device(state["d"])
    avg, prm, members, shifts = averages.class_averages_device(state["parts"], state["peak"], bel, 0.3, 0.2)
    return {"ids": ids, "belongsto": bel, "averages": avg, "params": prm, "members": members, "shifts": shifts}


# ---------------------------------------------------------------- what a pass cannot do without
def _pair_flops(S, rings, L):
    """one particle against one reference: the ring-summed products of both mirrors, their inverse transforms, the scan"""
    return S * (8.0 * (L // 2 + 1) * rings + 2 * 2.5 * L * math.log2(L) + 2.0 * L)


def _row_flops(rings, L):
    """one polar row: bilinear samples, normalisation, ring transforms"""
    return rings * (12.0 * L + 2.5 * L * math.log2(L))


def work(case):
    k = case["kind"]
    img = 4.0 * case.get("D", 0) ** 2
    S = (2 * case.get("shift", 0) + 1) ** 2
    if k in ("align", "host"):
        P, R, L = case["P"], case["R"], case["L"]
        return {"bytes": img * (P + R) + 8.0 * P + 20.0 * P * R,
                "flops": P * R * _pair_flops(S, case["rings"], L) + (P * S + R) * _row_flops(case["rings"], L)}
    if k == "groups":
        t = _group_table(case)
        P, R, pr = sum(x[1] for x in t), sum(x[3] for x in t), sum(x[1] * x[3] for x in t)
        return {"bytes": img * (P + R) + 8.0 * P + 20.0 * pr,
                "flops": pr * _pair_flops(S, case["rings"], 256) + (P * S + R) * _row_flops(case["rings"], 256)}
    if k == "learned":
        P, R, K = case["P"], case["R"], case["k"]
        nin = case["rings"] * learned.NK
        rows = P * 2.0 * (nin * learned.HIDDEN + learned.HIDDEN * learned.EMB + learned.EMB * R)
        return {"bytes": img * (P + R) + 32.0 * P,
                "flops": P * K * _pair_flops(S, case["rings"], 256) + (P * S + R) * _row_flops(case["rings"], 256) + rows}
    if k == "train":
        n, R, nin = case["P"], case["R"], case["rings"] * learned.NK
        w = nin * learned.HIDDEN + learned.HIDDEN * learned.EMB
        return {"bytes": 4.0 * (n + R) * nin + 4.0 * 7 * w + 8.0 * n,
                "flops": (n + R) * 2.0 * (2 * nin * learned.HIDDEN + 3 * learned.HIDDEN * learned.EMB)
                + 6.0 * n * R * learned.EMB}
    if k == "prealign":
        P = case["P"]
        one = P * (_pair_flops(S, case["rings"], 256) + S * _row_flops(case["rings"], 256))
        return {"bytes": img * (P + 1) + 16.0 * P, "flops": case["rounds"] * one}
    if k == "stability":
        P, R = case["P"], case["R"]
        one = P * (_pair_flops(S, case["rings"], 256) + S * _row_flops(case["rings"], 256) + 20.0 * case["D"] ** 2)
        return {"bytes": img * (P + 2 * R) + 20.0 * P, "flops": case["iters"] * one}
    P, R = case["P"], case["R"]
    return {"bytes": 4.0 * R * P + img * (P + R) + 16.0 * P + 8.0 * P + 16.0 * P + 12.0 * R,
            "flops": 40.0 * P * case["D"] ** 2}


# ---------------------------------------------------------------- FP64 restatement
def _sbj_batch(P, R, shift, L):
    """particles per texture batch: the reference's size check (2^31 - 1 table entries)"""
    per = min(R, 100) * 2 * (2 * shift + 1) ** 2 * (L + 2)
    bs = 0
    for i in range(int(math.log2(P)), -1, -1):
        cand = min(bs + 2**i, P)
        if cand * per <= 2**31 - 1:
            bs = cand
    return max(1, bs)


def _pad_stack(imgs, batch, tex, m):
    """every image with m more rows and columns as the stacked, clamped textures hold them, and its place in its texture"""
    n, D = imgs.shape[0], imgs.shape[1]
    batch = min(batch, n)
    i = torch.arange(n, device=DEV)
    loc = i % batch
    slot = loc % tex
    alloc = torch.where(loc // tex == (batch - 1) // tex, batch - (loc // tex) * tex, tex)
    nxt = torch.where(i + 1 < torch.clamp((i // batch + 1) * batch, max=n), i + 1, i + 1 - batch).clamp(0, n - 1)
    above = torch.where((slot > 0)[:, None, None], imgs[(i - 1).clamp(min=0), D - m:], imgs[:, :1])
    below = torch.where((slot + 1 < alloc)[:, None, None], imgs[nxt, :m], imgs[:, -1:])
    full = torch.cat([above, imgs, below], 1)
    return torch.cat([full[..., :1].expand(-1, -1, m), full, full[..., -1:].expand(-1, -1, m)], 2), slot


def _ring_spectra(imgs, batch, rings, L, shifts, base, lo=0, hi=None):
    """normalised polar rows' ring transforms [image][shift][ring][L/2 + 1], FP64 from the texture unit's 8-bit weights"""
    D, m = imgs.shape[1], 12
    tex = 65000 // D
    pad, slot = _pad_stack(imgs, batch, tex, m)
    hi = imgs.shape[0] if hi is None else hi
    pad, slot = pad[lo:hi].double(), slot[lo:hi]
    f32 = torch.float32
    j = torch.arange(L, device=DEV, dtype=f32) / float(L)
    ang = (j.double() * 3.14159265358979 * 2).to(f32).double()
    r = torch.arange(1, rings + 1, device=DEV, dtype=f32)[:, None]
    ox = ((torch.cos(ang).to(f32) * r) * rings / rings).reshape(-1)
    oy = ((torch.sin(ang).to(f32) * r) * rings / rings).reshape(-1)
    wr = torch.arange(1, rings + 1, device=DEV, dtype=torch.float64)[:, None]
    n = pad.shape[0]
    flat, W = pad.reshape(n, -1), pad.shape[2]
    out = torch.empty(n, len(shifts), rings, L // 2 + 1, dtype=torch.complex128, device=DEV)
    yoff = (slot * D).to(f32)
    for s, (sx, sy) in enumerate(shifts):
        cx = torch.full((n,), float(D // 2 + sx), dtype=f32, device=DEV)
        cy = torch.full((n,), float(D // 2 + sy), dtype=f32, device=DEV)
        if base is not None:
            cx, cy = cx + base[lo:hi, 0], cy + base[lo:hi, 1]
        x = (cx + 0.5)[:, None] + ox[None]
        y = (yoff + (cy + 0.5))[:, None] + oy[None]
        qx = torch.floor((x - 0.5).double() * 256 + 0.5).long()
        qy = torch.floor((y - 0.5).double() * 256 + 0.5).long()
        ix, A = (qx >> 8) + m, (qx & 255)
        iy, B = (qy >> 8) - (slot * D)[:, None] + m, (qy & 255)
        at = (iy.clamp(0, pad.shape[1] - 2) * W + ix.clamp(0, W - 2))
        w11 = (A * B + 128) >> 8
        v = (flat.gather(1, at) * (256 - A - B + w11) + flat.gather(1, at + 1) * (A - w11)
             + flat.gather(1, at + W) * (B - w11) + flat.gather(1, at + W + 1) * w11) / 256.0
        v = v.reshape(n, rings, L)
        nn = wr.sum() * L
        avg = (v * wr).sum((1, 2)) / nn
        sd = ((v * v * wr).sum((1, 2)) / nn - avg * avg).abs().sqrt()
        out[:, s] = torch.fft.rfft((v - avg[:, None, None]) / (sd + 1e-7)[:, None, None], dim=2)
    return out


def _exact_peaks(parts, refs, base, rings, shift, L):
    """d [R][P]: the largest correlation over shift, angle and mirror"""
    P, R = parts.shape[0], refs.shape[0]
    shifts = [(x, y) for x in range(-shift, shift + 1) for y in range(-shift, shift + 1)]
    S, K = len(shifts), L // 2 + 1
    w = torch.arange(1, rings + 1, device=DEV, dtype=torch.float64)[:, None]
    rs = (_ring_spectra(refs, 100, rings, L, [(0, 0)], None)[:, 0] * w).permute(2, 1, 0).contiguous()  # [k][ring][ref]
    d = torch.empty(R, P, dtype=torch.float64, device=DEV)
    batch = _sbj_batch(P, R, shift, L)
    step = max(1, int(2.5e8 / (S * L * max(R, rings))))
    for p0 in range(0, P, step):
        p1 = min(P, p0 + step)
        sp = _ring_spectra(parts, batch, rings, L, shifts, base, p0, p1)
        sp = sp.reshape(-1, rings, K).permute(2, 0, 1).contiguous()  # [k][row][ring]
        best = None
        for z in (torch.bmm(sp.conj(), rs), torch.bmm(sp, rs).conj()):
            c = torch.fft.irfft(z.permute(1, 2, 0), n=L, dim=2, norm="forward").amax(2)
            best = c if best is None else torch.maximum(best, c)
        d[:, p0:p1] = best.reshape(p1 - p0, S, R).amax(1).t()
    return d


def _exact_train(case, seed):
    par, X, lab, Xr, m, v = _train_inputs(case, seed)
    p = {n: torch.tensor(a, dtype=torch.float64, device=DEV, requires_grad=True) for n, a in par.items()}

    def emb(x):
        z = torch.relu(x.double() @ p["W1"].t() + p["b1"]) @ p["W2"].t() + p["b2"]
        return z / z.square().sum(1, keepdim=True).sqrt()

    loss = torch.nn.functional.cross_entropy(learned.SCALE * emb(X) @ emb(Xr).t(), lab.long(), reduction="none")
    loss.mean().backward()
    flat = torch.cat([p[n].detach().reshape(-1) for n in ("W1", "b1", "W2", "b2")])
    g = torch.cat([p[n].grad.reshape(-1) for n in ("W1", "b1", "W2", "b2")])
    m, v = 0.9 * m.double() + 0.1 * g, 0.999 * v.double() + 0.001 * g * g
    mh, vh = m / (1 - 0.9**101), v / (1 - 0.999**101)
    return {"loss": loss.detach(), "grad": g, "weights": flat - 1e-3 * (mh / (vh.sqrt() + 1e-8) + 1e-4 * flat)}


def _greedy_groups(d):
    """each pair in order of its peak: the particle joins the group unless it is placed or the group is full"""
    R, P = d.shape
    most, left = P // R, P % R
    size, open_, bel = [0] * R, R, [-1] * P
    for at in torch.sort(d.reshape(-1), descending=True, stable=True).indices.cpu().numpy().tolist():
        r, i = divmod(at, P)
        if bel[i] >= 0 or size[r] < 0:
            continue
        bel[i] = r
        size[r] += 1
        if size[r] == (most if open_ > 1 else most + left):
            size[r] = -1
            open_ -= 1
            if not open_:
                break
    return torch.tensor(bel, device=DEV)


def _exact_average(case, seed):
    parts, d, peak = _average_inputs(case, seed)
    P, R, D = case["P"], case["R"], case["D"]
    f32, f64 = torch.float32, torch.float64
    bel = _greedy_groups(d)
    pk = peak[bel, torch.arange(P, device=DEV)].double()
    a = torch.deg2rad(pk[:, 0])
    c, s = torch.cos(a), -torch.sin(a)
    sx = (-pk[:, 1] * c + pk[:, 2] * s).to(f32)
    sy = (-pk[:, 1] * s - pk[:, 2] * c).to(f32)
    flip = pk[:, 3] > 0.5
    col, row = torch.arange(D, device=DEV)[None, None, :], torch.arange(D, device=DEV)[None, :, None]
    sums = torch.zeros(R, D, D, dtype=f64, device=DEV)
    h = float(D // 2)
    for p0 in range(0, P, 1000):
        q = slice(p0, min(P, p0 + 1000))
        ixs = torch.where(flip[q, None, None], (D - col) % D, col)
        co, si = torch.cos(a[q]).to(f32)[:, None, None], torch.sin(a[q]).to(f32)[:, None, None]
        x = ixs.to(f32) - (h + sx[q])[:, None, None]
        y = row.to(f32) - (h + sy[q])[:, None, None]
        xo, yo = (x * co - y * si) + h, (x * si + y * co) + h
        out = (xo < 0) | (xo >= D) | (yo < 0) | (yo >= D)
        xo, yo = torch.where(out, ixs.to(f32), xo).double(), torch.where(out, row.to(f32), yo).double()
        i, j = torch.floor(xo).long(), torch.floor(yo).long()
        dx, dy = xo - i, yo - j
        i, j = i % D, j % D
        ip, im, jp, jm = (i + 1) % D, (i - 1) % D, (j + 1) % D, (j - 1) % D
        f = parts[q].reshape(-1, D * D).double()

        def at(jj, ii):
            return f.gather(1, (jj * D + ii).reshape(f.shape[0], -1)).reshape(-1, D, D)

        f00 = at(j, i)
        c1, c3 = at(j, ip) - f00, at(jp, i) - f00
        c2, c4 = (c1 - f00 + at(j, im)) * 0.5, (c3 - f00 + at(jm, i)) * 0.5
        c5 = at(jp, ip) - f00 - c1 - c3
        sums.index_add_(0, bel[q], f00 + dx * (c1 + (dx - 1) * c2 + dy * c5) + dy * (c3 + (dy - 1) * c4))
    n = torch.bincount(bel, minlength=R).double()
    zero = torch.zeros(R, dtype=f64, device=DEV)
    mx = zero.index_add(0, bel, torch.where(flip, -sx, sx).double()).to(f32).double() / n
    my = zero.index_add(0, bel, sy.double()).to(f32).double() / n
    kx = torch.arange(D // 2 + 1, device=DEV, dtype=f64)[None, :]
    ky = torch.arange(D, device=DEV, dtype=f64)[:, None]
    ky = torch.where(ky > D // 2, ky - D, ky)
    rad, fl, ff = torch.sqrt((kx / D) ** 2 + (ky / D) ** 2), 0.3, 0.2
    t = math.pi / (2 * ff * fl)
    filt = 0.5 * (torch.tanh(t * (rad + fl)) - torch.tanh(t * (rad - fl)))
    ph = 2 * math.pi * (kx[None] * mx[:, None, None] + ky[None] * my[:, None, None]) / D
    avg = torch.fft.irfft2(torch.fft.rfft2(sums / n[:, None, None]) * filt * torch.polar(torch.ones_like(ph), ph), s=(D, D))
    prm = torch.stack([pk[:, 0], torch.where(flip, sx + mx[bel], sx - mx[bel]), sy - my[bel], pk[:, 3]], 1)
    return {"ids": None, "belongsto": bel.int(), "averages": avg, "params": prm, "members": n.int(),
            "shifts": torch.stack([mx, my], 1)}


def exact(case, seed):
    """run()'s computed values in FP64.  A peak's angle and shift are the place of a maximum among equals to within
    rounding: they have no value of this kind, nor has what the iterations of the host sessions build on them."""
    k = case["kind"]
    if k in ("align", "host"):
        parts, refs, _, base = _stack(case["P"], case["R"], case["D"], case["rings"], case["shift"], seed)
        return {"d": _exact_peaks(parts, refs, base, case["rings"], case["shift"], case["L"]), "peak": None}
    if k == "groups":
        s = prepare(case, seed)
        d = [_exact_peaks(s["parts"][po:po + pn], s["refs"][ro:ro + rn], s["base"][po:po + pn], case["rings"],
                          case["shift"], 256).reshape(-1) for po, pn, ro, rn in s["table"]]
        return {"d": torch.cat(d), "peak": None}
    if k == "train":
        return _exact_train(case, seed)
    if k == "average":
        return _exact_average(case, seed)
    return None
