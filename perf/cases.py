"""The work that a user of this framework has it do, as cases that can be timed and compared.

Three kinds of call make up the framework's use, and each case is one of them through its public entry point:

* ``search``: `Search`, one handle per observation format.  The block loop of a search pushes one block of samples (uint8
  from host or device memory, or float samples that the caller has preprocessed), waits for it and takes each ddplan row's
  points above the threshold and its clusters.  The handle is filled before the first pass, so that every pass yields
  output, as all blocks of an observation but its first few do; ``file`` cases search one short file from its start.
* ``boxcar``: `boxcar`, the matched filter over dedispersed series that the caller already has.
* ``replot``: `replot`, the per-candidate chain over a batch of cut-out candidates.

Data are seeded: 8-bit Gaussian noise (mean 128, sigma 12) with dispersed pulses and, where ``rfi`` is set, sinusoids in
5 % of the channels and zero-DM impulses.  A stream of `nblk` blocks repeats from pass to pass.
"""
import math

import numpy as np
import torch

import transientx_gb300 as tx

KDM = 4.148741601e3  # dispersion delay in s for DM in pc/cm^3 and frequencies in MHz


# ---- the cases ----------------------------------------------------------------------------------

def _search(name, nchans, fhi, flo, tsamp, ndump, plan, **more):
    c = dict(kind="search", nchans=nchans, fhi=fhi, flo=flo, tsamp=tsamp, ndump=ndump, plan=plan, precision="fp32", beams=1,
             blocks=1, cap=16384, source="device", file=0, rfi=False, dense=False, iqr=False, zapthre=4.0, thre=7.0, nsub=0)
    c.update(more)
    if name:
        c["name"] = name
    return c


RFI = " kadaneF 8 4 zdot"


def listed():
    return [
        # one small block with RFI zapping, the quick-look size: launches and host work are most of it
        _search("quicklook_64ch", 64, 1500.0, 1200.0, 256e-6, 2048, "1 1 0 1 100 0.1 0.02" + RFI, source="host", nsub=8, cap=2048),
        # the single-beam search of 256 channels to DM 1000, FP32, blocks from pageable host memory
        _search("search_256ch_dm1000", 256, 1500.5, 1244.5, 64e-6, 15625, "1 1 0 0.5 2000 0.1 0.05", source="host", nsub=16),
        # a short file of the same kind searched from its start with a handle that is used for file after file
        _search("file_256ch", 256, 1500.5, 1244.5, 64e-6, 15625, "1 1 0 0.5 1000 0.1 0.05" + RFI, source="pinned", file=6,
                nsub=16),
        # four 1024-channel beams of the 64-beam job, 16-bit subband storage, one block of each
        _search("beams_1024ch_fp16", 1024, 1712.0, 856.0, 76e-6, 13156,
                "1 1 0 0.1 5000 0.1 0.05" + RFI + "\n2 1 500 0.2 5000 0.1 0.05\n4 1 1500 0.5 3000 0.1 0.05", precision="fp16",
                beams=4),
        # the 4096-channel search with RFI, three ddplan rows to DM 3000, plain FP32
        _search("rfi_4096ch_fp32", 4096, 1712.0, 856.0, 76e-6, 13156,
                "1 1 0 0.1 5000 0.1 0.05" + RFI + "\n2 1 500 0.2 5000 0.1 0.05\n4 1 1500 0.5 3000 0.1 0.05", rfi=True),
        # the same data with bfloat16 subband storage
        _search("rfi_4096ch_bf16", 4096, 1712.0, 856.0, 76e-6, 13156,
                "1 1 0 0.1 5000 0.1 0.05" + RFI + "\n2 1 500 0.2 5000 0.1 0.05\n4 1 1500 0.5 3000 0.1 0.05", rfi=True,
                precision="bf16"),
        # the high-time-resolution search, 8192 channels at 16 us, five rows to DM 5000: the largest block
        _search("hires_8192ch_fp16", 8192, 1800.0, 1200.0, 16e-6, 62496,
                "1 1 0 0.05 2000 0.1 0.01" + RFI + "\n2 1 100 0.1 2000 0.1 0.01\n4 1 300 0.2 2000 0.1 0.01\n"
                "8 1 700 0.5 2000 0.1 0.01\n16 1 1700 1 3300 0.1 0.01", precision="fp16", rfi=True),
        # the class-compatible headers' path: preprocessed float blocks, the dense S/N map read back after each
        _search("float_dense_512ch", 512, 1500.0, 1200.0, 128e-6, 7812, "1 1 0 1 500 0.1 0.05 zdot", source="float", dense=True),
        # ragged sizes and the other filters: 1000 channels, downsampling in both axes, mask, kadaneT, zero-DM, IQR statistics
        _search("ragged_1000ch_filters", 1000, 1510.0, 1210.0, 100e-6, 9990,
                "2 2 0 0.7 701 0.1 0.03 mask 4 5 kadaneT 2 5 zero", rfi=True, iqr=True),
        # boxcar over series that the caller dedispersed, the points above the threshold wanted
        dict(name="boxcar_points", kind="boxcar", ndm=1000, n=8193, maxw=300, iqr=False, dense=False, thre=7.0),
        # one small candidate, the quick look that replot gives
        dict(name="replot_one", kind="replot", count=1, nchan=256, dm=120.0, width=1e-3, tbin=64e-6, fhi=1500.0, flo=1244.0,
             zdot=True, kadane=True, clip=False, fd=1, nopt=False),
        # a batch of candidates at the sampling of the 1024-channel beams
        dict(name="replot_batch", kind="replot", count=6, nchan=1024, dm=100.0, width=2e-3, tbin=76e-6, fhi=1712.0, flo=856.0,
             zdot=False, kadane=True, clip=True, fd=1, nopt=False),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.12:
        return dict(kind="boxcar", ndm=_logint(rng, 1, 1500), n=_logint(rng, 500, 70000 if rng.random() < 0.3 else 20000),
                    maxw=_logint(rng, 4, 400), iqr=rng.random() < 0.3, dense=rng.random() < 0.3, thre=rng.choice([6.5, 7.0, 8.0]))
    if pick < 0.3:
        return dict(kind="replot", count=rng.randint(1, 6), nchan=_logint(rng, 64, 1024), dm=round(rng.uniform(10.0, 110.0), 2),
                    width=round(math.exp(rng.uniform(math.log(5e-4), math.log(4e-3))), 5), tbin=rng.choice([64e-6, 76e-6, 128e-6]),
                    fhi=1712.0, flo=rng.choice([856.0, 1200.0]), zdot=rng.random() < 0.5, kadane=rng.random() < 0.7,
                    clip=rng.random() < 0.4, fd=rng.choice([1, 1, 2]), nopt=rng.random() < 0.25)
    nchans = _logint(rng, 48, 4096)
    if rng.random() < 0.6:
        nchans = max(64, nchans // 16 * 16)
    tsamp = rng.choice([64e-6, 76e-6, 100e-6, 128e-6, 256e-6])
    td0, fd0 = rng.choice([(1, 1), (1, 1), (1, 1), (2, 1), (1, 2), (3, 1)])
    nrows = rng.choice([1, 1, 2, 3])
    ndump = int(round(rng.uniform(0.25, 1.0) / tsamp)) // (td0 * 4) * (td0 * 4)
    fhi, flo = rng.choice([(1712.0, 856.0), (1500.0, 1200.0), (1800.0, 1200.0)])
    flt = rng.choice(["", " zdot", RFI, RFI, RFI, " mask 4 4 kadaneF 8 4", " zero kadaneT 4 4"])
    dms, ddm, lines = 0.0, rng.choice([0.1, 0.2, 0.5, 1.0]), []
    for r in range(nrows):
        ndm = _logint(rng, 40, 4000)
        lines.append("%d %d %g %g %d 0.1 %g%s" % (td0 * 2 ** r, fd0, dms, ddm, ndm, rng.choice([0.01, 0.03, 0.05]), flt if r == 0 else ""))
        dms, ddm = round(dms + ndm * ddm, 6), ddm * 2
        if dms > 2000:
            break
    c = _search("", nchans, fhi, flo, tsamp, ndump, "\n".join(lines), precision=rng.choice(["fp32", "fp16", "bf16"]),
                beams=rng.choice([1, 1, 2]), source=rng.choice(["device", "device", "host", "pinned", "float"]),
                iqr=rng.random() < 0.15, zapthre=rng.choice([0.0, 4.0]))
    c["rfi"] = flt == RFI and c["zapthre"] > 0 and c["source"] != "float"  # unfiltered RFI is all points, no search
    while not _modest(c):  # a shorter DM range, then fewer rows, until the case is no larger than the listed ones
        lines = c["plan"].split("\n")
        p = lines[-1].split()
        if int(p[4]) > 60:
            p[4] = str(int(p[4]) * 2 // 3)
            lines[-1] = " ".join(p)
        elif len(lines) > 1:
            lines.pop()
        else:
            c["nchans"] //= 2
        c["plan"] = "\n".join(lines)
    return c


def _modest(c):
    adds = ring = 0
    for p in _plans(c):
        if p["maxd1"] > 20000:  # a channel's delay within its subband has to fit in a kernel's window
            return False
        adds += c["beams"] * p["N"] * (p["C"] * p["ng"] + p["nsub"] * p["r"].ndm)
        ring += c["beams"] * 4 * (p["nsub"] * p["ng"] + 2 * p["C"]) * (p["offset"] + p["N"])
    return adds < 3e10 and ring < 12e9 and _fill(c) <= 40


# ---- inputs -------------------------------------------------------------------------------------

def _freqs(c):
    n = c["nchans"] if c["kind"] == "search" else c["nchan"]
    return c["fhi"] - (c["fhi"] - c["flo"]) / n * (np.arange(n) + 0.5)


def _delay(dm, fh, fl):
    return KDM * dm * (1.0 / (fl * fl) - 1.0 / (fh * fh))


def _rows(c):
    base = tx.SinglePulse(thre=c["thre"], iqr=c["iqr"], nsub=c["nsub"])
    return tx.parse_ddplan(c["plan"], base)


def _nblk(c):
    return c["file"] or 3


def _stream(c, seed, beam):
    """uint8 samples [nblk * ndump][nchans] on the GPU; pulses wrap around, so that the stream can repeat."""
    n, C, f, ts = _nblk(c) * c["ndump"], c["nchans"], _freqs(c), c["tsamp"]
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 2097143) + beam)
    rng = np.random.default_rng([seed, beam])
    raw = torch.empty((n, C), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 25) // C)
    for t in range(0, n, step):
        x = torch.randn((min(step, n - t), C), generator=g, device="cuda")
        raw[t:t + step] = x.mul_(12.0).add_(128.0).round_().clamp_(0, 255).to(torch.uint8)
    dmax = max(r.dms + r.ddm * r.ndm for r in _rows(c))
    for p in range(2):
        dm, snr = rng.uniform(0.02, 0.95) * dmax, rng.uniform(8, 16)
        w = max(1, int(math.exp(rng.uniform(math.log(3e-4), math.log(1e-2))) / ts))
        amp = 12.0 * snr / math.sqrt(C * w)
        d = torch.from_numpy(np.round((rng.uniform(0, n * ts) + _delay(dm, f.max(), f)) / ts).astype(np.int64)).cuda()
        at = (d[:, None] + torch.arange(w, device="cuda")[None, :]) % n * C + torch.arange(C, device="cuda")[:, None]
        add = torch.full(at.shape, math.floor(amp), device="cuda") + (torch.rand(at.shape, generator=g, device="cuda") < amp % 1.0)
        raw.view(-1)[at] = (raw.view(-1)[at].float() + add).clamp_(0, 255).to(torch.uint8)
    if c["rfi"]:
        t = torch.arange(n, device="cuda") * ts
        for j in rng.choice(C, size=max(1, C // 20), replace=False):
            a, per, ph = rng.uniform(10, 30), rng.uniform(2e-3, 0.2), rng.uniform(0, 2 * math.pi)
            raw[:, int(j)] = (raw[:, int(j)].float() + 12.0 * a * torch.sin(2 * math.pi / per * t + ph)).clamp_(0, 255).to(torch.uint8)
        for _ in range(int(rng.poisson(n * ts)) + 1):
            t0, k = int(rng.uniform(0, n)), int(rng.integers(1, 51))
            raw[t0:t0 + k] = (raw[t0:t0 + k].float() + 240.0).clamp_(0, 255).to(torch.uint8)
    return raw


def _float(raw):
    """What a caller's own preprocessing leaves: samples about zero, near unit variance."""
    return (raw.float() - 127.5) / 11.0


def _fill(c):
    """Blocks after which every row's next block gives output."""
    return 0 if c["file"] else max(-(-p["offset"] // p["N"]) for p in _plans(c))


def _candidates(c, seed):
    f = _freqs(c)
    dly = _delay(c["dm"], f.max(), f)
    nbin = int((dly.max() + 40 * c["width"]) / c["tbin"])
    out = []
    for k in range(c["count"]):
        g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 2097143) + k)
        x = torch.randn((c["nchan"], nbin), generator=g, device="cuda").mul_(10.0).add_(100.0).round_()
        d = torch.from_numpy(np.round((0.4 * nbin * c["tbin"] + dly) / c["tbin"]).astype(np.int64)).cuda()
        at = (d[:, None] + torch.arange(max(1, int(c["width"] / c["tbin"])), device="cuda")) % nbin
        x.scatter_add_(1, at, torch.full(at.shape, 3.0, device="cuda"))
        out.append(x)
    return f, out


def _series(c, seed):
    """Dedispersed series: noise of the sum of many channels, a slow drift in some, boxcar pulses."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 2097143))
    rng = np.random.default_rng(seed)
    x = torch.randn((c["ndm"], c["n"]), generator=g, device="cuda").mul_(16.0)
    for _ in range(1 + c["ndm"] // 16):
        k, w = int(rng.integers(c["ndm"])), int(min(c["n"] // 4, rng.integers(1, c["maxw"] + 1)))
        t = int(rng.integers(0, c["n"] - w + 1))
        x[k, t:t + w] += 16.0 * rng.uniform(8, 25) / math.sqrt(w)
    return x


def _widths(minw, maxw, snrloss, ts):
    """The boxcar widths in samples: each longer by 1/(1 - snrloss)^2, and by one at least."""
    w = [int(math.floor(max(float(np.float32(minw)), float(np.float32(ts)) if minw < ts else 0.0) / ts + 0.5))]
    factor = np.float32(1.0 / (1.0 - float(np.float32(snrloss))) ** 2)
    while True:
        n = max(int(np.float32(w[-1]) * factor), w[-1] + 1)
        if n * ts > float(np.float32(maxw)):
            return np.array(w, np.int32)
        w.append(n)


def prepare(case, seed):
    c = case
    if c["kind"] == "boxcar":
        return dict(c=c, tim=_series(c, seed).cpu().numpy(), vwn=_widths(1e-4, c["maxw"] * 1e-4, 0.1, 1e-4))
    if c["kind"] == "replot":
        f, xs = _candidates(c, seed)
        cands = []
        for x in xs:
            h = torch.empty(x.shape, dtype=torch.float32, pin_memory=True)
            h.copy_(x)
            cands.append({"data": h.numpy(), "frequencies": f, "tbin": c["tbin"], "dm": c["dm"], "width": c["width"], "keep": h})
        return dict(c=c, cands=cands)
    rows = _rows(c)
    flags = (tx.FLAG_DENSE | tx.FLAG_KEEP_SERIES if c["dense"] else 0) | tx.FLAG_CLUSTER
    s = tx.Search(rows, c["nchans"], c["tsamp"], _freqs(c), c["ndump"], nbeams=c["beams"], precision=c["precision"], flags=flags,
                  zapthre=c["zapthre"])
    blocks = []
    for b in range(c["beams"]):
        raw = _stream(c, seed, b)
        if c["source"] == "float":
            raw = _float(raw)
        if c["source"] == "pinned":
            h = torch.empty(raw.shape, dtype=raw.dtype, pin_memory=True)
            h.copy_(raw)
            raw = h
        elif c["source"] != "device":
            raw = raw.cpu()
        parts = [raw[k * c["ndump"]:(k + 1) * c["ndump"]] for k in range(_nblk(c))]
        blocks.append(parts if c["source"] == "device" else [p.numpy() for p in parts])
    st = dict(c=c, s=s, blocks=blocks, at=0, nrows=len(rows))
    torch.cuda.synchronize()  # the inputs are in place before the library's own streams read them
    for _ in range(_fill(c)):
        _push(st)
    s.sync(allow_overflow=True)
    for b in range(c["beams"]):
        for r in range(len(rows)):
            while s.pop_result(r, b) is not None:
                pass
    return st


def _push(st):
    c, s, i = st["c"], st["s"], st["at"] % _nblk(st["c"])
    for b in range(c["beams"]):
        blk = st["blocks"][b][i]
        if c["source"] == "device":
            s.push_block_device(blk.data_ptr(), b)
        elif c["source"] == "float":
            s.push_block_f32(blk, b)
        else:
            s.push_block(blk, b)
    st["at"] += 1


def _table(p, cap):
    """Points as a table of fixed length, its unused end zero: their (DM, sample, width) and their S."""
    t = np.zeros(cap, p.dtype)
    t[:len(p)] = p[:cap]
    return t.view(np.int32).reshape(-1, 4)[:, :3], t["S"]


def run(state):
    c = state["c"]
    if c["kind"] == "boxcar":
        S, W, p = tx.boxcar(state["tim"], state["vwn"], iqr=c["iqr"], thre=c["thre"], dense=c["dense"])
        return [S, W, *_table(p, 4096)]
    if c["kind"] == "replot":
        res = tx.replot(state["cands"], zdot=c["zdot"], kadane=(8, 4, 7) if c["kadane"] else None,
                        clip=(2, 2, 7) if c["clip"] else None, fd=c["fd"], nopt=c["nopt"], maps=True)
        return [[r["snrmap"], np.array([r["snr"], r["width"]], np.float32), np.array([r["dm_maxsnr"], r["dms"], r["ddm"]]),
                 np.array([r["maxtid"], r["nbin"], r["nchan"], r["ndm"]])] for r in res]
    s, out = state["s"], []
    if c["file"]:
        for b in range(c["beams"]):
            s.reset_beam(b)
    for _ in range(c["file"] or c["blocks"]):
        _push(state)
    s.sync(allow_overflow=True)
    for b in range(c["beams"]):
        for r in range(state["nrows"]):
            got = s.pop_result(r, b)
            while got is not None:
                res, pts, cl = got
                if res.gated:
                    out.append([*_table(pts, c["cap"]), *_table(cl, 128)])
                got = s.pop_result(r, b)
    if c["dense"]:
        out.append([a for r in range(state["nrows"]) for a in s.dense(r)])
    return out


# ---- the plan of a row, from its configuration alone ---------------------------------------------

def _subbands(f, nsub):
    C = len(f)
    sub = np.arange(C) * nsub // C
    fref = np.array([f[sub == s].max() for s in range(nsub)])
    flow = np.array([f[sub == s].min() for s in range(nsub)])
    return sub, fref, flow


def _group(f, nsub, ts, ddm, ndm):
    _, fref, flow = _subbands(f, nsub)
    k = _delay(1.0, fref, flow).max()
    if not ddm * k > 0.0:
        return ndm
    g = math.floor(2.0 * ts / (ddm * k))
    g = g // 8 * 8 if g >= 8 else g
    return int(min(max(g, 1), ndm))


def _round(x):
    return np.floor(np.asarray(x) + 0.5).astype(np.int64)  # delays are not negative


def _plans(c, tables=False):
    f0, out = _freqs(c), []
    for r in _rows(c):
        C, N, ts, ndm = c["nchans"] // r.fd, c["ndump"] // r.td, c["tsamp"] * r.td, r.ndm
        f = f0[:C * r.fd].reshape(C, r.fd).mean(1)
        nsub = min(r.nsub, C) if r.nsub > 0 else 0
        if not nsub:
            best = None
            for e in range(C.bit_length()):
                p = 1 << e
                if p <= C:
                    cost = C * -(-ndm // _group(f, p, ts, r.ddm, ndm)) + p * ndm
                    if best is None or cost < best:
                        best, nsub = cost, p
        G = _group(f, nsub, ts, r.ddm, ndm)
        ng = -(-ndm // G)
        sub, fref, _ = _subbands(f, nsub)
        dmc = np.array([r.dms + r.ddm * 0.5 * (g * G + min((g + 1) * G, ndm) - 1) for g in range(ng)])
        dmk = r.dms + r.ddm * np.arange(ndm)
        d1 = _round(_delay(dmc[-1:, None], fref[sub][None, :], f[None, :]) / ts)
        d2 = _round(_delay(dmk[-1:, None], f.max(), fref[None, :]) / ts)
        offset = -(-int(d1.max() + d2.max()) // N) * N
        p = dict(r=r, C=C, N=N, ts=ts, f=f, nsub=nsub, G=G, ng=ng, sub=sub, offset=offset, vwn=_widths(r.minw, r.maxw, r.snrloss, ts))
        if tables:
            p["d1"] = _round(_delay(dmc[:, None], fref[sub][None, :], f[None, :]) / ts)
            p["d2"] = _round(_delay(dmk[:, None], f.max(), fref[None, :]) / ts)
        p["maxd1"] = int(d1.max())
        out.append(p)
    return out


def work(case):
    """Bytes: each input read once, each output written once, and for a search the subband series of the rows, which have to
    be kept until their delayed samples are there, written and read once.  Operations: the additions of the two dedispersion
    stages at the row's plan, and one subtraction and one product for each sample and width of the boxcar."""
    c = case
    if c["kind"] == "boxcar":
        return {"bytes": 4.0 * c["ndm"] * c["n"] * (3 if c["dense"] else 1), "flops": 2.0 * c["ndm"] * c["n"] * len(_widths(1e-4, c["maxw"] * 1e-4, 0.1, 1e-4))}
    if c["kind"] == "replot":
        f = _freqs(c)
        nbin = int((_delay(c["dm"], f.max(), f).max() + 40 * c["width"]) / c["tbin"])
        cut = min(nbin, int(40 * c["width"] / c["tbin"]))
        rows = 1 if c["nopt"] else 2 ** math.ceil(math.log2(c["nchan"] // c["fd"]))
        nw = math.log(max(2.0, cut / 2)) / math.log(1 / 0.81)
        return {"bytes": 4.0 * c["count"] * (c["nchan"] * nbin + rows * cut),
                "flops": c["count"] * (12.0 * c["nchan"] * nbin + rows * cut * (math.log2(max(2, rows)) + 2 * nw))}
    by = fl = 0.0
    size = 2 if c["precision"] != "fp32" else 4
    for p in _plans(c):
        nb = max(0, c["file"] - p["offset"] // p["N"]) if c["file"] else c["blocks"]
        n1 = c["file"] or c["blocks"]
        by += size * p["nsub"] * p["ng"] * p["N"] * (n1 + nb)
        fl += p["N"] * (n1 * p["C"] * p["ng"] + nb * (p["nsub"] * p["r"].ndm + 2.0 * p["r"].ndm * len(p["vwn"])))
        by += 8.0 * p["r"].ndm * p["N"] if c["dense"] else 0.0
    raw = c["ndump"] * c["nchans"] * (4.0 if c["source"] == "float" else 1.0) * n1
    return {"bytes": c["beams"] * (by + raw), "flops": c["beams"] * fl}


# ---- 64-bit results -------------------------------------------------------------------------------

D = torch.float64


def _std(x):
    m = x.mean(-1, keepdim=True)
    v = (x * x).mean(-1, keepdim=True) - m * m
    return m, v


def _kadane(ds):
    """Largest-sum run of each row: (sum, first, last)."""
    P = torch.cumsum(ds, -1)
    Q = torch.cat([torch.zeros_like(P[:, :1]), P[:, :-1]], -1)
    lo, at = torch.cummin(Q, -1)
    best, e = (P - lo).max(-1)
    return best, at.gather(1, e[:, None])[:, 0], e


def _ds(x, td, fd):
    C, N = x.shape[0] // fd, x.shape[1] // td
    return x[:C * fd, :N * td].reshape(C, fd, N, td).sum((1, 3))


def _kadane_f(x, td, fd, thr2, limit):
    ds = _ds(x, td, fd)
    t = torch.arange(x.shape[1], device=x.device)
    for s in (1.0, -1.0):
        b, a, e = _kadane(ds * s)
        wn = e - a + 1
        hit = (wn > limit) & (b * b / (wn * td * fd) > thr2)
        z = hit[:, None] & (t >= (a * td)[:, None]) & (t < ((e + 1) * td)[:, None])
        x[:ds.shape[0] * fd][z.repeat_interleave(fd, 0)] = 0.0
    return x


def _quart(v):
    s = torch.sort(v.reshape(-1))[0]
    n = len(s)
    return s[n // 4], s[n - 1 - n // 4]


def _zdot(x):
    m, v = _std(x)
    n = (x - m) / torch.where(v > 0, v, torch.ones_like(v)).sqrt()
    s = n.mean(0)
    N = x.shape[1]
    xe, xs, se, ss = n.sum(1), n @ s, s.sum(), (s * s).sum()
    q = se * se - ss * N
    if float(q) == 0.0:
        return n
    return n - (((xe * se - xs * N) / q)[:, None] * s + ((xs * se - xe * ss) / q)[:, None])


def _preprocess(c, p, blk):
    """One block after downsampling, equalize, baseline and the row's filters, [C][N]."""
    r = p["r"]
    x = blk.T.to(D)
    if c["source"] != "float" and c["zapthre"] > 0:
        v = x - 128.0
        a, b, cc, d = (v.pow(k).mean(1) for k in (1, 2, 3, 4))
        m2, m3 = b - a * a, cc - 3 * a * b + 2 * a ** 3
        m4 = d - 4 * a * cc + 6 * a * a * b - 3 * a ** 4
        ok = m2 > 0
        sk, ku = torch.where(ok, m3 / m2.clamp_min(1e-300) ** 1.5, 0.0), torch.where(ok, m4 / m2.clamp_min(1e-300) ** 2 - 3.0, 0.0)
        for q in (sk, ku):
            q1, q3 = _quart(q)
            x[(q < q1 - c["zapthre"] * (q3 - q1)) | (q > q3 + c["zapthre"] * (q3 - q1))] = 0.0
        del v
    x = _ds(x, r.td, r.fd) if r.td * r.fd > 1 else x
    m, v = _std(x)
    live = v[:, 0] > 0
    x = (x - m) / torch.where(v > 0, v, torch.ones_like(v)).sqrt()
    nw = int(math.floor(float(np.float32(r.bswidth)) / p["ts"] + 0.5)) if r.bswidth > 0 else 0
    if nw > 0:
        x[live] -= _smooth(x.sum(0) / max(1, int(live.sum())), nw)
    for o in r.rfilist:
        td, fd = (int(o[1]), int(o[2])) if len(o) > 2 else (1, 1)
        if o[0] == "kadaneF":
            x = _kadane_f(x, td, fd, r.threKadaneF ** 2, int(r.widthlimit / (p["ts"] * td)))
        elif o[0] == "zdot":
            x = _zdot(x)
        elif o[0] == "zero":
            x[live] -= x.sum(0) / max(1, int(live.sum()))
        elif o[0] == "mask":
            ds = _ds(x, td, fd)
            q1, q3 = _quart(ds)
            bad = (ds < q1 - r.threMask * (q3 - q1)) | (ds > q3 + r.threMask * (q3 - q1))
            x[:ds.shape[0] * fd, :ds.shape[1] * td][bad.repeat_interleave(fd, 0).repeat_interleave(td, 1)] = 0.0
        else:
            bw = abs(p["f"][1] - p["f"][0])
            x = _kadane_f(x.T.contiguous(), fd, td, r.threKadaneT ** 2, int(r.bandlimitKT / (bw * fd))).T.contiguous()
    return x


def _smooth(z, nw):
    N, h = len(z), nw // 2
    c = torch.cat([torch.zeros(1, dtype=D, device=z.device), torch.cumsum(z, 0)])
    i = torch.arange(N, device=z.device)
    lo, hi = (i - h).clamp_min(0), (i + h).clamp_max(N - 1)
    return (c[hi + 1] - c[lo]) / (hi - lo + 1)


def _dedisperse(p, X, t0, k0, k1, g):
    """Series of the DMs k0..k1-1 of group g from absolute sample t0 on, of a stream that repeats."""
    dev, L, N = X.device, X.shape[1], p["N"]
    d2 = torch.from_numpy(p["d2"][k0:k1]).to(dev)
    sp = int((d2[-1] - d2[0]).max())
    sub = torch.from_numpy(p["sub"]).to(dev)
    base = t0 + d2[0][sub] + torch.from_numpy(p["d1"][g]).to(dev)
    u = torch.arange(N + sp, device=dev)
    S = torch.zeros((p["nsub"], N + sp), dtype=D, device=dev)
    for j in range(0, p["C"], 1024):
        S.index_add_(0, sub[j:j + 1024], X[j:j + 1024].gather(1, (base[j:j + 1024, None] + u) % L))
    n = torch.arange(N, device=dev)
    return torch.stack([S.gather(1, (d2[k] - d2[0])[:, None] + n).sum(0) for k in range(k1 - k0)])


def _match(x, vwn, iqr):
    """Largest S of each sample over the widths, [rows][n]."""
    n = x.shape[1]
    if iqr:
        s = torch.sort(x, 1)[0]
        m, v = s[:, n // 2, None], ((s[:, n - 1 - n // 4] - s[:, n // 4]) / 1.349)[:, None] ** 2
    else:
        m, v = _std(x)
    c = torch.cat([torch.zeros_like(x[:, :1]), torch.cumsum(x - m, 1)], 1)
    best = torch.zeros_like(x)
    for w in (int(w) for w in vwn):
        wl, wh = w // 2 + 1, (w - 1) // 2
        if n - wh > wl:
            S = (c[:, wl + wh + 1:n + 1] - c[:, 1:n - wh - wl + 1]) / (w * v).sqrt()
            best[:, wl:n - wh] = torch.maximum(best[:, wl:n - wh], S)
    return torch.where(v > 0, best, torch.zeros_like(best))


def _padded(v, cap):
    out = torch.zeros(cap, dtype=D, device=v.device)
    out[:len(v)] = v[:cap]
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "boxcar":
        x = _series(c, seed)
        S = torch.cat([_match(x[k:k + 256].to(D), _widths(1e-4, c["maxw"] * 1e-4, 0.1, 1e-4), c["iqr"]) for k in range(0, c["ndm"], 256)])
        return [S if c["dense"] else None, None, None, _padded(S[S > c["thre"]], 4096)]
    if c["kind"] == "replot":
        f, xs = _candidates(c, seed)
        return [[_replot(c, f, x.to(D)), None, None, None] for x in xs]
    if c["precision"] != "fp32" and not c["dense"] or c["beams"] * sum(p["N"] * (p["C"] * p["ng"] + p["nsub"] * p["r"].ndm) for p in _plans(c)) * max(c["blocks"], c["file"]) > 1.8e11:
        return None
    out, dense = [], []
    for b in range(c["beams"]):
        raw = _stream(c, seed, b)
        raw = _float(raw) if c["source"] == "float" else raw
        blocks = raw.split(c["ndump"])
        for p in _plans(c, True):
            r, N = p["r"], p["N"]
            X = torch.cat([_preprocess(c, p, blk) for blk in blocks], 1)
            first = p["offset"] // N + 1 if c["file"] else _fill(c) + 1
            for m in range(first, (c["file"] or first + c["blocks"] - 1) + 1):
                t0, got, S = m * N - N - p["offset"], [], []
                for g in range(p["ng"]):
                    k0, k1 = g * p["G"], min((g + 1) * p["G"], r.ndm)
                    best = _match(_dedisperse(p, X, t0, k0, k1, g), p["vwn"], r.iqr)
                    got.append(best[best > np.float32(r.thre)])
                    S.append(best if c["dense"] else None)
                # with 16-bit storage a point at the threshold may fall on either side, and the tables would not line up
                out.append([None, _padded(torch.cat(got), c["cap"]) if c["precision"] == "fp32" else None, None, None])
            if c["dense"]:
                dense += [torch.cat(S), None]
            del X
    return out + ([dense] if c["dense"] else [])


def _stats(x):
    """Each channel's quietest half (circular): mean, variance, skewness, kurtosis, lag-1 autocorrelation."""
    n = x.shape[1]
    h = n // 2
    cs = torch.cat([torch.zeros_like(x[:, :1]), torch.cumsum(torch.cat([x, x], 1), 1)], 1)
    a = (cs[:, h:h + n + 1] - cs[:, :n + 1]).argmin(1)
    y = x.gather(1, (a[:, None] + torch.arange(h, device=x.device)) % n)
    m, v = _std(y)
    t = y - m
    q = (t * t).mean(1)
    ac = (t[:, 1:] * t[:, :-1]).sum(1) / (h - 1)
    safe = torch.where(q > 0, q, torch.ones_like(q))
    return m, v, (t ** 3).mean(1) / safe ** 1.5, (t ** 4).mean(1) / safe ** 2 - 3.0, ac / safe


def _replot(c, f, x):
    dev, tbin, dm, n = x.device, c["tbin"], c["dm"], x.shape[1]
    if c["zdot"]:
        x = _zdot(x)
    _, _, sk, ku, ac = _stats(x)
    d = torch.from_numpy(_round(_delay(dm, f.max(), f) / tbin) % n).to(dev)
    x = x.gather(1, (torch.arange(n, device=dev) + d[:, None]) % n)
    factor = 8 if c["kadane"] else 1
    x = x[:, :min(n, int(40 * float(np.float32(c["width"])) / tbin) // factor * factor)].contiguous()
    n = x.shape[1]
    for q in (ku, sk, ac):
        s = torch.sort(q)[0]
        q1, q3 = s[len(s) // 4], s[len(s) - 1 - len(s) // 4]
        x[(q < q1 - 3 * (q3 - q1)) | (q > q3 + 3 * (q3 - q1))] = 0.0
    m, v, _, _, _ = _stats(x)
    x = (x - m) / torch.where(v > 0, v, torch.ones_like(v)).sqrt()
    if c["clip"]:
        ds = _ds(x, 2, 2)
        bad = (ds > 7 * 2.0).repeat_interleave(2, 0).repeat_interleave(2, 1)
        x[:bad.shape[0], :bad.shape[1]][bad] = 0.0
    if c["kadane"]:
        x = _kadane_f(x, 8, 4, 49.0, 0)
    if c["fd"] > 1:
        x = _ds(x, 1, c["fd"])
        f = f[:len(x) * c["fd"]].reshape(len(x), c["fd"]).mean(1)
    nc = len(x)
    if c["nopt"]:
        h = x.sum(0, keepdim=True)
    else:
        R = 2 ** math.ceil(math.log2(nc))
        span = n * tbin / _delay(1.0, f.max(), f.min())
        dms = max(0.0, dm - span / 2)
        ddm = (dm + span / 2 - dms) / R
        fp = np.concatenate([f, f[0] + np.arange(nc, R) * (f[1] - f[0])])
        h = torch.cat([x, torch.zeros((R - nc, n), dtype=D, device=dev)])
        i = torch.arange(n, device=dev)
        order, w = np.zeros(R, np.int64), 1
        while w < R:  # blocks of w rows merge into blocks of 2w
            order[w:2 * w] = order[:w] + R // (2 * w)
            top = np.arange(0, R, 2 * w)
            sh = KDM * (dms + order[None, :2 * w] * ddm - dm) * (1.0 / fp[top + w, None] ** 2 - 1.0 / fp[top, None] ** 2) / tbin
            sh = torch.from_numpy((np.sign(sh) * np.floor(np.abs(sh) + 0.5)).astype(np.int64) % n).to(dev)
            a, b = h.reshape(-1, 2, w, n).unbind(1)
            a, b = a.repeat(1, 2, 1), b.repeat(1, 2, 1)
            h = (a + b.gather(2, (i + sh[:, :, None]) % n)).reshape(R, n)
            w *= 2
        o = torch.empty_like(h)
        o[torch.from_numpy(order).to(dev)] = h
        h = o
    m, v = _std(h)
    y = h - m
    cs = torch.cumsum(torch.cat([y, y], 1), 1)
    best, wn, i = torch.zeros_like(h), 1, torch.arange(n, device=dev)
    factor = np.float32(1.0 / ((1.0 - float(np.float32(0.1))) ** 2))
    while True:
        wl, wh = wn // 2 + 1, (wn - 1) // 2
        at = torch.where(i >= wl, i, i + n)
        best = torch.maximum(best, (cs[:, at + wh] - cs[:, at - wl]) / (wn * v).sqrt())
        wn = max(int(np.float32(wn) * factor), wn + 1)
        if wn > n // 2:
            break
    return torch.where(v > 0, best, torch.zeros_like(best))
