"""Performance cases of the baseband hot path.

Each case is one piece of work that a user of the framework runs through the
Python entry points of dspsr_b200: a block through the fused pipeline (unpack,
optional filterbank, coherent dedispersion, detection, fold) and its profile
read back, the same steps one engine at a time, the filterbank with the
dedispersion inside it, the inverse filterbank, or spectral kurtosis.  Sizes
are those of the repository's own benchmark configurations (C1 .. C5, C2 with
-F 64:D) and of its tests, with whole and ragged block lengths.

  listed()            the named cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs (on the GPU) and the plan a program keeps
  run(state)          one pass, its outputs whole
  exact(case, seed)   the same outputs in 64 bits, by torch and numpy alone
  work(case)          the bytes and operations of one pass
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dspsr-kanyixia_b200"))
import dspsr_b200 as b2  # noqa: E402

START = (60000, 3600, 0.25)
EPOCH = (59999, 0, 0.0)
SPACING = 0.03                     # 8-bit digitiser: level x is worth (x + 0.5) * SPACING
INT8, INT16, FLOAT = b2.INT8_TFPD, b2.INT16_TFPD, b2.FLOAT_FPT


def _pipe(name, cf, bw, dm, nchan, fb, npol, nfft, kind, state, nbin, period, ndat, pos=None,
          neg=None):
    """A pipeline block: nchan input channels, each split into fb by the
    filterbank when fb > 1; nfft, pos and neg count samples of the
    dedispersed channels, ndat those of the input."""
    c = nchan * max(fb, 1)
    if pos is None:
        pos, neg, nfft = b2.dispersion_plan(cf, bw, dm, c, nfft)
    return dict(name=name, kind="pipe", cf=cf, bw=bw, dm=dm, nchan=nchan, fb=fb, npol=npol,
                nfft=nfft, pos=pos, neg=neg, input=kind, state=state, nbin=nbin, period=period,
                ndat=ndat)


def listed():
    half = b2.smearing_samples(1400.0, 256.0, 25.0, 64, 1)
    half500 = b2.smearing_samples(1400.0, 256.0, 500.0, 64, 1)
    return [
        # the shortest block a real-time loop hands over: latency and launches
        _pipe("block_4096_short", 1400.0, 16.0, 1.5, 1, 0, 2, 4096, INT8, b2.INTENSITY, 256,
              0.08933, 1 << 16),
        # one 16 MHz band, the reference's CPU-runnable configuration (C1)
        _pipe("band_2p17_c1", 1400.0, 16.0, 67.99, 1, 0, 2, 1 << 17, INT8, b2.INTENSITY, 1024,
              0.08933, 1 << 24),
        # the headline: 256 MHz into 64 channels, DM 500, full Stokes (C2)
        _pipe("fb64_2p16_stokes_c2", 1400.0, 256.0, 500.0, 1, 64, 2, 1 << 16, INT8, b2.STOKES,
              2048, 5.757e-3, 1 << 26),
        # beams of the 48-stream configuration (C3): 32 and 8 channels
        _pipe("beam_32x2p14", 1400.0, 32.0, 411.84, 32, 0, 2, 1 << 14, INT8, b2.INTENSITY, 1024,
              0.0317, 1 << 19),
        _pipe("beam_8x2p17", 1400.0, 32.0, 764.81, 8, 0, 2, 1 << 17, INT8, b2.INTENSITY, 2048,
              0.217, 1 << 21),
        # 16-bit data, one channel at the longest transform, coherence
        # products, a block length that is no multiple of anything
        _pipe("band_2p18_int16_ragged", 1400.0, 16.0, 150.0, 1, 0, 2, 1 << 18, INT16, b2.COHERENCE,
              512, 0.0451, 6000001),
        # float voltages through a 1024-channel filterbank (second half of C5)
        _pipe("fb1024_2p15_float_c5", 1400.0, 800.0, 1000.0, 1, 1024, 2, 1 << 15, FLOAT,
              b2.STOKES, 4096, 1.6e-3, 1 << 27),
        # the reference's engine-by-engine sequence on C1's shape: unpack,
        # convolve to voltages, detect, fold
        dict(name="engines_2p17", kind="engines", cf=1400.0, bw=16.0, dm=67.99, nchan=1, npol=2,
             nfft=1 << 17, pos=b2.smearing_samples(1400.0, 16.0, 67.99, 1, 1),
             neg=b2.smearing_samples(1400.0, 16.0, 67.99, 1, -1), state=b2.STOKES, nbin=1024,
             period=0.08933, ndat=1 << 21),
        # 256 oversampled PFB channels of 16-bit data back to one band (C5)
        dict(name="ifb_256x1024_c5", kind="ifb", nin=256, npol=2, lin=1024, disc=12288,
             input=INT16, ndat=260424),
        # the filterbank with the dedispersion inside it, small and large DM
        dict(name="fbd_64x4096_dm25", kind="fbd", cf=1400.0, bw=256.0, dm=25.0, npol=2, nsub=64,
             freq_res=4096, pos=half, neg=half, input=INT8, state=b2.STOKES, nbin=2048,
             period=5.757e-3, ndat=1 << 25),
        dict(name="fbd_64x65536_dm500", kind="fbd", cf=1400.0, bw=256.0, dm=500.0, npol=2,
             nsub=64, freq_res=65536, pos=half500, neg=half500, input=INT8, state=b2.STOKES,
             nbin=2048, period=5.757e-3, ndat=1 << 26),
        # RFI excision on 512 channels of voltages (C4's shape, an eighth of
        # its block)
        dict(name="sk_512x1024", kind="sk", nchan=512, npol=2, ndat=1 << 17, M=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pipe", "pipe", "pipe", "pipe", "engines", "ifb", "fbd", "sk"])
    cf = rng.uniform(700.0, 3000.0)
    bw = rng.choice([16.0, 32.0, 64.0, 128.0, 256.0])
    dm = rng.uniform(1.0, 1000.0)
    period = math.exp(rng.uniform(math.log(1.5e-3), math.log(0.5)))
    nbin = rng.choice([64, 256, 500, 1024, 2048, 4096])
    if kind in ("pipe", "engines"):
        npol = 1 if kind == "pipe" and rng.random() < 0.15 else 2
        nfft = 1 << rng.randint(12, 18)
        state = b2.INTENSITY if npol == 1 else rng.randint(0, 3)
        fb = rng.choice([0, 0, 64, 64, 16, 256, 1024]) if kind == "pipe" else 0
        nchan = rng.choice([1, 1, 2, 8, 32]) if fb == 0 else 1
        c = nchan * max(fb, 1)
        nfft = min(nfft, (1 << 26) // c)
        total = nfft * rng.uniform(0.02, 0.88)
        pos = int(total * rng.uniform(0.4, 0.6))
        neg = int(total) - pos
        keep = nfft - pos - neg
        # whole parts, bounded by the transformed points, and a ragged rest
        most = max(1, (1 << 27) // (c * npol * nfft))
        npart = _log(rng, 1, most)
        ndat = (pos + neg + npart * keep + rng.randint(0, keep - 1)) * max(fb, 1)
        case = dict(kind=kind, cf=cf, bw=bw, dm=dm, nchan=nchan, npol=npol, nfft=nfft, pos=pos,
                    neg=neg, state=state, nbin=nbin, period=period, ndat=ndat)
        if kind == "pipe":
            case.update(fb=fb, input=rng.choice([INT8, INT8, INT16, FLOAT]))
        return case
    if kind == "ifb":
        lin = rng.choice([128, 256, 512, 1024])
        nin = 256 if lin < 1024 else rng.choice([64, 128, 256])
        return dict(kind="ifb", nin=nin, npol=rng.choice([1, 2, 2]), lin=lin,
                    disc=nin * lin // 16, input=rng.choice([INT8, INT16, FLOAT]),
                    ndat=_log(rng, 4 * lin, 300000))
    if kind == "fbd":
        nsub, freq_res = rng.choice([(64, 1024), (64, 4096), (32, 4096), (16, 16384), (64, 16384),
                                     (128, 8192), (64, 65536)])
        pos = int(freq_res * rng.uniform(0.02, 0.3))
        neg = int(freq_res * rng.uniform(0.02, 0.3))
        step = nsub * (freq_res - pos - neg)
        npart = _log(rng, 1, max(2, (1 << 25) // (nsub * freq_res)))
        return dict(kind="fbd", cf=cf, bw=bw, dm=dm, npol=rng.choice([1, 2, 2]), nsub=nsub,
                    freq_res=freq_res, pos=pos, neg=neg, input=rng.choice([INT8, INT16, FLOAT]),
                    state=b2.INTENSITY, nbin=nbin, period=period,
                    ndat=nsub * (pos + neg) + npart * step + rng.randint(0, step - 1))
    M = rng.choice([64, 100, 256, 1000, 1024, 4096])
    nchan = rng.choice([16, 64, 128, 512])
    return dict(kind="sk", nchan=nchan, npol=rng.choice([1, 2, 2]), M=M,
                ndat=M * _log(rng, 4, max(5, (1 << 26) // (nchan * M))) + 2 * rng.randint(0, 20))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (seed + 1) + salt)
    return g


def _pulsed(ndat, rate, period, g):
    """Noise amplitude of each sample: a 3 % duty pulse once per period."""
    t = torch.arange(ndat, device="cuda", dtype=torch.float64) / rate / period
    on = torch.remainder(t - 0.3 - float(torch.rand(1, device="cuda", generator=g)), 1.0) < 0.03
    return 1.0 + 0.7 * on.float()


def _raw(kind, ndat, nchan, npol, rate, period, seed):
    """A block as the receiver delivers it: TFPD integers, or FPT voltages."""
    g = _gen(seed, 7 * ndat + nchan)
    amp = _pulsed(ndat, rate, period, g)
    if kind == FLOAT:
        x = torch.empty((nchan, npol, ndat, 2), device="cuda")
        for c in range(nchan):
            for p in range(npol):
                x[c, p] = torch.randn((ndat, 2), device="cuda", generator=g) * amp[:, None]
        return x
    sigma, lim, dt = (12.0, 127, torch.int8) if kind == INT8 else (300.0, 32767, torch.int16)
    out = torch.empty((ndat, nchan, npol, 2), dtype=dt, device="cuda")
    step = max(1, (1 << 24) // (nchan * npol * 2))
    for t0 in range(0, ndat, step):
        n = min(step, ndat - t0)
        v = torch.randn((n, nchan, npol, 2), device="cuda", generator=g)
        v *= sigma * amp[t0:t0 + n, None, None, None]
        out[t0:t0 + n] = v.round_().clamp_(-lim - 1, lim).to(dt)
    return out


def _voltages(case, seed):
    """Complex FPT voltages with interference in a few channels (SK)."""
    nchan, npol, ndat = case["nchan"], case["npol"], case["ndat"]
    g = _gen(seed, nchan + ndat)
    x = torch.empty((nchan, npol, ndat, 2), device="cuda")
    for c in range(nchan):
        x[c] = torch.randn((npol, ndat, 2), device="cuda", generator=g) * math.sqrt(0.5)
    t = torch.arange(ndat, device="cuda", dtype=torch.float64)
    for c in range(0, nchan, 23):                       # tones
        ph = 2 * math.pi * 0.37 * t
        x[c, :, :, 0] += (1.5 * torch.cos(ph)).float()
        x[c, :, :, 1] += (1.5 * torch.sin(ph)).float()
    for k in range(ndat // 8192):                       # broadband bursts
        t0 = int(torch.randint(0, ndat - 40, (1,), device="cuda", generator=g))
        x[:, :, t0:t0 + 8 + k % 32] *= 6.0
    return x


def _lut():
    x = np.arange(256, dtype=np.uint8).view(np.int8).astype(np.float32)
    return (x + np.float32(0.5)) * np.float32(SPACING)


def _rate(case):
    """Sampling rate of the input (complex samples per second)."""
    return case["bw"] * 1e6 / case.get("nchan", 1)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    ctx = b2.Context(0)
    st = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind == "pipe":
        cfg = b2.make_config(case["cf"], case["bw"], case["dm"], case["nchan"], case["npol"],
                             case["nfft"], case["pos"], case["neg"], case["nbin"],
                             case["period"], state=case["state"], input_kind=case["input"],
                             lut=_lut(), start_mjd=START, epoch_mjd=EPOCH,
                             filterbank_nchan=case["fb"])
        st["pipe"] = b2.Pipeline(ctx, cfg)
        st["prof"], st["hits"] = st["pipe"].profile_buffers()
        st["raw"] = _raw(case["input"], case["ndat"], case["nchan"], case["npol"], _rate(case),
                         case["period"], seed)
    elif kind == "engines":
        nchan, npol, ndat = case["nchan"], case["npol"], case["ndat"]
        conv = b2.Convolution(ctx, nchan, npol, case["nfft"], case["pos"], case["neg"])
        conv.set_dedispersion(case["cf"], case["bw"], case["dm"])
        n = conv.npart(ndat) * conv.nkeep
        st.update(conv=conv, n=n, lut=_lut(),
                  fold=b2.Fold(ctx, case["nbin"], nchan, b2.NOUT[case["state"]]),
                  raw=_raw(INT8, ndat, nchan, npol, _rate(case), case["period"], seed),
                  x=torch.empty((nchan, npol, ndat, 2), device="cuda"),
                  y=torch.empty((nchan, npol, n, 2), device="cuda"),
                  d=torch.empty((nchan, b2.NOUT[case["state"]], n), device="cuda"))
    elif kind == "ifb":
        ifb = b2.InverseFilterbank(ctx, case["nin"], 1, case["nin"], case["npol"], case["lin"],
                                   os=(4, 3), output_discard=(case["disc"], case["disc"]))
        n = ifb.npart(case["ndat"]) * ifb.info["out_step"]
        st.update(ifb=ifb, n=n, lut=_lut(),
                  raw=_raw(case["input"], case["ndat"], case["nin"], case["npol"], 1e6, 0.01, seed),
                  out=torch.empty((1, case["npol"], n, 2), device="cuda"))
    elif kind == "fbd":
        fbd = b2.FilterbankDuring(ctx, 1, case["npol"], case["nsub"], case["freq_res"],
                                  (case["pos"], case["neg"]))
        fbd.set_dedispersion(case["cf"], case["bw"], case["dm"])
        st.update(fbd=fbd, n=fbd.npart(case["ndat"]) * fbd.info["nkeep"], lut=_lut(),
                  fold=b2.Fold(ctx, case["nbin"], case["nsub"], b2.NOUT[case["state"]]),
                  raw=_raw(case["input"], case["ndat"], 1, case["npol"], _rate(case),
                           case["period"], seed))
    else:
        npart, cells = case["ndat"] // case["M"], case["ndat"] // case["M"] * case["nchan"]
        x = _voltages(case, seed)
        st.update(x=x, out=torch.zeros_like(x), npart=npart,
                  limits=b2.sk_limits(case["M"]),
                  sums=torch.empty((npart, case["nchan"], case["npol"], 2), device="cuda"),
                  counts=torch.empty(cells, dtype=torch.int32, device="cuda"),
                  mask=torch.empty(cells, dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    return st


def _phi(case, idat, rate):
    return b2.fold_phi(START, EPOCH, idat, rate, case["period"])


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "pipe":
        pipe = st["pipe"]
        pipe.reset()
        pipe.run(st["raw"], case["ndat"], case["ndat"] if case["input"] == FLOAT else 0)
        pipe.get_profiles_async(st["prof"], st["hits"])
        pipe.wait_profiles()
        return dict(profiles=st["prof"], hits=st["hits"])
    if kind == "engines":
        nchan, npol, ndat, n = case["nchan"], case["npol"], case["ndat"], st["n"]
        rate = _rate(case)
        ctx.unpack8(st["raw"], ndat, nchan, npol, 2, st["lut"], st["x"], 2 * ndat)
        st["conv"].perform(st["x"], ndat, ndat, st["y"], n)
        ctx.detect(st["y"], n, n, nchan, case["state"], st["d"], n)
        st["fold"].reset()
        st["fold"].set_bins(_phi(case, case["pos"], rate), 1.0 / rate / case["period"], n)
        st["fold"].fold(st["d"], n)
        profiles, hits = st["fold"].get_profiles()
        return dict(voltages=st["y"], detected=st["d"], profiles=profiles, hits=hits)
    if kind == "ifb":
        st["ifb"].perform(st["raw"], case["ndat"], st["out"], st["n"], input_kind=case["input"],
                          lut=st["lut"] if case["input"] == INT8 else None)
        return st["out"]
    if kind == "fbd":
        rate = _rate(case) / case["nsub"]
        st["fold"].reset()
        st["fold"].set_bins(_phi(case, case["pos"], rate), 1.0 / rate / case["period"], st["n"])
        st["fbd"].perform_fold(st["raw"], case["ndat"], st["fold"], case["state"],
                               input_kind=case["input"],
                               lut=st["lut"] if case["input"] == INT8 else None)
        profiles, hits = st["fold"].get_profiles()
        return dict(profiles=profiles, hits=hits)
    lo, hi = st["limits"]
    ndat = case["ndat"]
    ctx.sk(st["x"], ndat, ndat, case["nchan"], case["npol"], case["M"], lo, hi, st["out"], ndat,
           st["sums"], st["counts"], st["mask"])
    return dict(out=st["out"], sums=st["sums"], counts=st["counts"], mask=st["mask"])


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _unpacked(raw, kind):
    """Complex128 [chan][pol][t] of a block from _raw."""
    if kind == FLOAT:
        return torch.view_as_complex(raw.double())
    v = raw.permute(1, 2, 0, 3).double() + 0.5
    return torch.view_as_complex((v * float(np.float32(SPACING)) if kind == INT8 else v)
                                 .contiguous())


def _chirp(case, freq, nfft, swap, norm, bw=None):
    """Dispersion response [chan][nfft]: FP64 phases kept as floats, as the
    reference stores them."""
    bw = case["bw"]
    nchan = len(freq)
    width = bw / nchan
    ipt = torch.arange(nfft, device="cuda", dtype=torch.float64)
    if swap:
        ipt = torch.roll(ipt, nfft // 2)
    f = ipt * (width / nfft) - 0.5 * width
    out = torch.empty((nchan, nfft), device="cuda", dtype=torch.complex128)
    for c, fc in enumerate(freq):
        coeff = -2 * math.pi * (1e6 * case["dm"] / 2.41e-4) / (fc * fc)
        ph = (coeff * (f * f) / (fc + f)).float().double()
        out[c] = torch.polar(torch.full_like(ph, norm), ph)
    return out


def _centres(case, nchan, swap, dc):
    base = case["cf"] - 0.5 * case["bw"] + (0.0 if dc else 0.5 * case["bw"] / nchan)
    return [base + ((c + nchan // 2) % nchan if swap else c) * case["bw"] / nchan
            for c in range(nchan)]


def _convolved(case, x, h):
    """Overlap-save of x [chan][pol][t] with h [chan][nfft]."""
    nfft, pos, neg = case["nfft"], case["pos"], case["neg"]
    keep = nfft - pos - neg
    npart = (x.shape[2] - pos - neg) // keep if x.shape[2] >= nfft else 0
    y = torch.empty((x.shape[0], x.shape[1], npart * keep), device="cuda", dtype=torch.complex128)
    for c in range(x.shape[0]):
        for p0 in range(0, npart, 64):
            n = min(64, npart - p0)
            part = x[c, :, p0 * keep:(p0 + n - 1) * keep + nfft].unfold(1, nfft, keep)
            z = torch.fft.ifft(torch.fft.fft(part) * h[c], norm="forward")
            y[c, :, p0 * keep:(p0 + n) * keep] = z[..., pos:nfft - neg].flatten(1)
    return y


def _detected(y, state):
    p, q = y[:, 0], y[:, -1]
    pp, qq = p.real ** 2 + p.imag ** 2, q.real ** 2 + q.imag ** 2
    if state == b2.INTENSITY:
        return (pp + qq if y.shape[1] == 2 else pp)[:, None]
    if state == b2.PPQQ:
        return torch.stack([pp, qq], 1)
    x = p.conj() * q
    if state == b2.COHERENCE:
        return torch.stack([pp, qq, x.real, x.imag], 1)
    return torch.stack([pp + qq, pp - qq, 2 * x.real, 2 * x.imag], 1)


def _bins(case, idat, rate, n):
    """The reference's bin of each sample: a sequential double recurrence."""
    offset = (idat + 0.5) / rate
    whole = math.floor(offset)
    frac = START[2] + (offset - whole)
    sec = START[1] + int(whole)
    if frac >= 1.0:
        frac, sec = frac - 1.0, sec + 1
    day, sec = START[0] + sec // 86400, sec % 86400
    secs = float((day - EPOCH[0]) * 86400 + (sec - EPOCH[1])) + (frac - EPOCH[2])
    phi = math.fmod(secs, case["period"]) / case["period"] - 0.0
    step = 1.0 / rate / case["period"]
    out = np.empty(n, np.float64)
    for lo in range(0, n, 1 << 20):
        part = []
        for _ in range(min(1 << 20, n - lo)):
            phi -= math.floor(phi)
            part.append(phi)
            phi += step
        out[lo:lo + len(part)] = part
    return torch.from_numpy((out * case["nbin"]).astype(np.int64)).cuda()


def _folded(case, d, bins):
    nbin = case["nbin"]
    prof = torch.zeros((d.shape[0], d.shape[1], nbin), device="cuda", dtype=torch.float64)
    for c in range(d.shape[0]):
        prof[c].index_add_(1, bins, d[c])
    hits = torch.bincount(bins, minlength=nbin)
    return prof.cpu().numpy(), hits.cpu().numpy().astype(np.uint32)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sk":
        n = case["ndat"] // case["M"] * case["M"]
        x = _voltages(case, seed)[:, :, :n].double()
        s = (x ** 2).sum(-1).reshape(case["nchan"], case["npol"], -1, case["M"])
        sums = torch.stack([s.sum(-1), (s * s).sum(-1)], -1).permute(2, 0, 1, 3).contiguous()
        return dict(out=None, sums=sums, counts=None, mask=None)
    if kind == "ifb":
        return _exact_ifb(case, seed)
    rate = _rate(case)
    nchan = case.get("nchan", 1)
    x = _unpacked(_raw(case.get("input", INT8), case["ndat"], nchan, case["npol"], rate,
                       case["period"], seed), case.get("input", INT8))
    if kind == "fbd":
        return _exact_fbd(case, x, rate / case["nsub"])
    fb = case.get("fb", 0)
    if fb > 1:
        rate /= fb
        n = x.shape[2] // fb
        f = torch.empty((fb, case["npol"], n), device="cuda", dtype=torch.complex128)
        for p in range(case["npol"]):
            for t0 in range(0, n, 1 << 16):
                m = min(1 << 16, n - t0)
                blk = x[0, p, t0 * fb:(t0 + m) * fb].reshape(m, fb)
                f[:, p, t0:t0 + m] = torch.fft.fft(blk).T / math.sqrt(fb)
        x, nchan = f, fb
    freq = _centres(case, nchan, fb > 1, fb > 1)
    h = _chirp(case, freq, case["nfft"], True, 1.0 / math.sqrt(case["nfft"]))
    y = _convolved(case, x, h)
    del x
    d = _detected(y, case["state"])
    prof, hits = _folded(case, d, _bins(case, case["pos"], rate, y.shape[2]))
    if kind == "engines":
        return dict(voltages=torch.view_as_real(y), detected=d, profiles=prof, hits=hits)
    return dict(profiles=prof, hits=hits)


def _exact_fbd(case, x, rate):
    nsub, fr, pos, neg = case["nsub"], case["freq_res"], case["pos"], case["neg"]
    keep, nfft = fr - pos - neg, nsub * fr
    over = (pos + neg) * nsub
    npart = (x.shape[2] - over) // (nsub * keep)
    h = _chirp(case, _centres(case, nsub, True, False), fr, False,
               1.0 / math.sqrt(float(nfft) * fr))
    y = torch.empty((nsub, case["npol"], npart * keep), device="cuda", dtype=torch.complex128)
    for k in range(npart):
        for p in range(case["npol"]):
            t0 = k * nsub * keep
            z = torch.fft.fft(x[0, p, t0:t0 + nfft]).reshape(nsub, fr) * h
            z = torch.fft.ifft(z, norm="forward")
            y[:, p, k * keep:(k + 1) * keep] = z[:, pos:fr - neg]
    prof, hits = _folded(case, _detected(y, case["state"]), _bins(case, pos, rate, y.shape[2]))
    return dict(profiles=prof, hits=hits)


def _exact_ifb(case, seed):
    nin, lin, disc, npol = case["nin"], case["lin"], case["disc"], case["npol"]
    keep = lin * 3 // 4
    lout = nin * keep
    din = disc * 4 // (nin * 3)
    step_in, step_out = lin - 2 * din, lout - 2 * disc
    npart = (case["ndat"] - 2 * din) // step_in
    x = _unpacked(_raw(case["input"], case["ndat"], nin, npol, 1e6, 0.01, seed), case["input"])
    out = torch.empty((1, npol, npart * step_out), device="cuda", dtype=torch.complex128)
    for k in range(npart):
        spec = torch.fft.fft(x[:, :, k * step_in:k * step_in + lin])
        # bins [-keep/2, keep/2) of fine channel c at [c*keep - keep/2, c*keep + keep/2)
        kept = torch.cat([spec[..., lin - keep // 2:], spec[..., :keep // 2]], -1)
        s = torch.roll(kept.transpose(0, 1).reshape(npol, lout), -(keep // 2), dims=1)
        z = torch.fft.ifft(s, norm="forward")
        out[0, :, k * step_out:(k + 1) * step_out] = z[:, disc:lout - disc]
    return torch.view_as_real(out)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def work(case):
    """Input read once, outputs written once; radix-2 operation counts of the
    transforms that the requested lengths imply."""
    kind = case["kind"]
    npol, ndat = case["npol"], case["ndat"]
    size = {INT8: 2, INT16: 4, FLOAT: 8}
    if kind == "sk":
        samples = case["nchan"] * npol * ndat
        return dict(bytes=16.0 * samples, flops=8.0 * samples)
    if kind == "ifb":
        lin, lout = case["lin"], case["nin"] * case["lin"] * 3 // 4
        din = case["disc"] * 4 // (case["nin"] * 3)
        npart = (ndat - 2 * din) // (lin - 2 * din)
        out = npart * (lout - 2 * case["disc"]) * npol
        return dict(bytes=float(size[case["input"]] * case["nin"] * npol * ndat + 8 * out),
                    flops=npart * npol * (case["nin"] * _fft_flops(lin) + _fft_flops(lout)))
    nout = b2.NOUT[case["state"]]
    if kind == "fbd":
        nfft = case["nsub"] * case["freq_res"]
        keep = case["freq_res"] - case["pos"] - case["neg"]
        npart = (ndat - (case["pos"] + case["neg"]) * case["nsub"]) // (case["nsub"] * keep)
        flops = npart * (npol * (_fft_flops(nfft) + 6.0 * nfft
                                 + case["nsub"] * _fft_flops(case["freq_res"]))
                         + case["nsub"] * keep * 3.0 * npol * nout)
        return dict(bytes=float(size[case["input"]] * npol * ndat
                                + 4 * nout * case["nsub"] * case["nbin"]), flops=flops)
    fb = max(case.get("fb", 0), 1)
    c = case["nchan"] * fb
    nfft = case["nfft"]
    keep = nfft - case["pos"] - case["neg"]
    n = ndat // fb
    npart = (n - case["pos"] - case["neg"]) // keep if n >= nfft else 0
    flops = npart * c * (npol * (2 * _fft_flops(nfft) + 6.0 * nfft) + keep * 3.0 * npol * nout)
    if fb > 1:
        flops += n * npol * _fft_flops(fb)
    bytes_ = size[case.get("input", INT8)] * case["nchan"] * npol * ndat + 4 * c * nout * case["nbin"]
    if kind == "engines":
        # each engine's own input and output: that is what the caller asks for
        bytes_ += c * (npol * (16 * ndat + 16 * npart * keep) + 8 * nout * npart * keep)
    return dict(bytes=float(bytes_), flops=float(flops))
