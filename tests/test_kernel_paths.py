"""GPU parity of the kernels that one rule or another chooses: row lengths and
column passes of every size, the transposing load of many TFPD channels,
blocks that start between words, filterbanks and inverse filterbanks of every
warp-sized transform, folds whose bins are much longer or shorter than a
sample, and an engine whose rows change from FP32 to the tensor cores and back.

Tolerances are those of the same comparisons elsewhere: profiles 1e-5 of the
oracle chain's power (float sums of a few hundred samples per bin), voltages
5e-6 relative RMS of a 64-bit evaluation."""
import numpy as np
import pytest

import test_sk as sk
from test_gpu_pipeline import base_cfg, check, make_blocks, oracle_chain, run_pipeline

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

VOLTAGE_RTOL = 5e-6


def rel_rms(a, b):
    a, b = np.asarray(a, np.complex128), np.asarray(b, np.complex128)
    return float(np.sqrt(np.mean(np.abs(a - b) ** 2) / np.mean(np.abs(b) ** 2)))


# nfft, row length (0: the default, 4096 up to 2^17 points and 8192 above),
# channels, input kind (8-bit: affine table or not), state, nbin, samples per bin
PATHS = [
    (1 << 14, 4096, 1, "i8", 3, 64, 2000.0),      # n1 4, one column per row of samples
    (1 << 14, 8192, 2, "i8", 1, 512, 0.4),        # n1 2, bins shorter than a sample
    (1 << 15, 0, 8, "i8", 0, 128, 40.0),          # n1 8, eight channels: transposing load
    (1 << 15, 0, 16, "i16", 2, 256, 11.0),        # n1 8, the same for 16-bit samples
    (1 << 15, 0, 8, "lut", 3, 100, 7.0),          # a table that is not affine
    (1 << 16, 0, 3, "i16", 3, 256, 11.0),         # n1 16, channels that do not tile
    (1 << 16, 0, 8, "i8", 0, 64, 900.0),          # n1 16, transposing load
    (1 << 16, 8192, 1, "f", 2, 333, 3.0),         # n1 8 with 8192-point rows
    (1 << 17, 8192, 1, "i8", 3, 256, 33.0),       # n1 16, 8192-point rows
    (1 << 17, 0, 8, "i8", 2, 256, 90.0),          # n1 32, transposing load
    (1 << 17, 4096, 1, "i16", 1, 256, 100.0),     # n1 32, 4096-point rows
    (1 << 18, 0, 2, "lut", 3, 1024, 11.0),        # n1 32
    (1 << 18, 0, 1, "f", 0, 64, 5000.0),
]


def path_cfg(b2, nfft, row, nchan, kind, state, nbin, per_bin, npol=2):
    kinds = dict(i8=b2.INT8_TFPD, lut=b2.INT8_TFPD, i16=b2.INT16_TFPD, f=b2.FLOAT_FPT)
    bw = 16.0
    cfg = base_cfg(b2, bw=bw, nchan=nchan, npol=npol, nfft=nfft, dm=0.5, kind=kinds[kind],
                   state=state, nbin=nbin, period=per_bin * nbin * nchan / (bw * 1e6), row=row)
    if kind == "lut":
        x = np.arange(256, dtype=np.uint8).view(np.int8).astype(np.float32)
        cfg["lut"] = np.sign(x) * np.abs(x) ** np.float32(0.9)
    return cfg


@pytest.mark.parametrize("path", PATHS, ids=lambda p: "-".join(str(x) for x in p))
def test_pipeline_paths_match_oracle(ctx, b2, orc, path):
    nfft = path[0]
    cfg = path_cfg(b2, *path)
    rng = np.random.default_rng(nfft + path[2])
    nk = nfft - cfg["pos"] - cfg["neg"]
    # the second block starts with a carried prefix that parts straddle
    blocks = make_blocks(rng, cfg, [nfft + nk + 777, 2 * nk + 12345])
    prof, hits, total, info = run_pipeline(ctx, b2, blocks, cfg)
    n2 = path[1] or (4096 if nfft <= 1 << 17 else 8192)
    assert (info["n1"], info["n2"]) == (nfft // n2, n2)
    rprof, rhits, rtotal = oracle_chain(orc, b2, blocks, cfg)
    check(prof, hits, total, rprof, rhits, rtotal, cfg["state"])


@pytest.mark.parametrize("npol", [1, 2])
def test_default_row_lengths(ctx, b2, npol):
    """The split of each transform length when the caller names no row length."""
    most = (1 << 15) if npol == 1 else 1 << 17
    for lg in range(13, 19):
        nfft = 1 << lg
        want = 4096 if 1 << 14 <= nfft <= most else 8192
        for row, n2 in ((0, want), (8192, 8192)):
            pl = b2.Pipeline(ctx, b2.make_config(1400.0, 16.0, 0.1, 1, npol, nfft, 10, 10, 64, 0.01,
                                                 row_length=row))
            info = pl.info()
            pl.close()
            assert (info["n1"], info["n2"]) == (nfft // n2, n2), (nfft, row)


@pytest.mark.parametrize("nfft,kind", [(1 << 14, "i8"), (1 << 17, "i8"), (1 << 18, "i16")])
def test_one_polarisation_matches_oracle(ctx, b2, orc, nfft, kind):
    cfg = path_cfg(b2, nfft, 0, 1, kind, b2.INTENSITY, 128, 50.0, npol=1)
    rng = np.random.default_rng(nfft)
    blocks = make_blocks(rng, cfg, [2 * nfft + 99])
    prof, hits, total, _ = run_pipeline(ctx, b2, blocks, cfg)
    rprof, rhits, rtotal = oracle_chain(orc, b2, blocks, cfg)
    check(prof, hits, total, rprof, rhits, rtotal, cfg["state"])


@pytest.mark.parametrize("fb,nfft,kind,offset", [(0, 1 << 14, "i8", 2), (0, 1 << 17, "i16", 4),
                                                 (64, 1 << 15, "i8", 2), (64, 1 << 16, "i16", 4),
                                                 (64, 1 << 16, "i8", 4)])
def test_blocks_between_words(ctx, b2, fb, nfft, kind, offset):
    """A block at an address that is no multiple of a dual-polarisation
    sample's (or of 16 bytes) gives the profile of the same block aligned."""
    cfg = base_cfg(b2, bw=16.0 * (fb or 1), nfft=nfft, dm=0.5, fb=fb, nbin=128, period=0.0031,
                   kind=b2.INT8_TFPD if kind == "i8" else b2.INT16_TFPD, state=b2.STOKES)
    rng = np.random.default_rng(nfft + offset)
    raw = make_blocks(rng, cfg, [(2 * nfft + 64) * (fb or 1)])[0]
    ndat = (2 * nfft + 64) * (fb or 1)
    whole = torch.zeros(raw.nbytes + 16, dtype=torch.uint8, device="cuda")
    whole[offset:offset + raw.nbytes] = torch.from_numpy(raw.view(np.uint8)).cuda()
    out = []
    for d in (torch.from_numpy(raw.view(np.uint8)).cuda(), whole[offset:]):
        pl = b2.Pipeline(ctx, b2.make_config(
            cfg["cf"], cfg["bw"], cfg["dm"], 1, 2, nfft, cfg["pos"], cfg["neg"], cfg["nbin"],
            cfg["period"], state=cfg["state"], input_kind=cfg["kind"], lut=cfg["lut"],
            filterbank_nchan=fb))
        pl.run(d, ndat)
        out.append(pl.get_profiles())
        pl.close()
    assert np.array_equal(out[0][1], out[1][1])
    scale = np.abs(out[0][0][:, :1]) + 1e-30
    # two runs differ by the order of the atomic sums only
    assert np.max(np.abs(out[0][0] - out[1][0]) / scale) < 1e-5


@pytest.mark.parametrize("row", [4096, 8192])
@pytest.mark.parametrize("kind", ["i8", "lut", "i16"])
def test_fused_filterbank_row_lengths(ctx, b2, orc, row, kind):
    """The 64-channel filterbank inside the column pass, both splits."""
    nfft = 1 << 16
    cfg = base_cfg(b2, bw=64 * 4.0, nfft=nfft, dm=20.0, fb=64, nbin=256, period=0.0057,
                   state=b2.STOKES, kind=b2.INT16_TFPD if kind == "i16" else b2.INT8_TFPD, row=row)
    if kind == "lut":
        x = np.arange(256, dtype=np.uint8).view(np.int8).astype(np.float32)
        cfg["lut"] = np.sign(x) * np.abs(x) ** np.float32(0.9)
    rng = np.random.default_rng(row)
    nk = nfft - cfg["pos"] - cfg["neg"]
    blocks = make_blocks(rng, cfg, [64 * (nfft + 100), 64 * (nk + 50)])
    prof, hits, total, info = run_pipeline(ctx, b2, blocks, cfg)
    assert info["n2"] == row
    rprof, rhits, rtotal = oracle_chain(orc, b2, blocks, cfg)
    check(prof, hits, total, rprof, rhits, rtotal, cfg["state"])


@pytest.mark.parametrize("nsub", [128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("kind,npol,nchan", [("f", 2, 2), ("i8", 2, 1), ("i16", 1, 3), ("i16", 2, 5),
                                             ("i8", 1, 12)])
def test_filterbank_sizes(ctx, b2, nsub, kind, npol, nchan):
    """Output lengths around a tile's, against a 64-bit FFT."""
    kinds = dict(i8=b2.INT8_TFPD, i16=b2.INT16_TFPD, f=b2.FLOAT_FPT)
    lut, _ = b2.bittable8()
    rng = np.random.default_rng(nsub + nchan)
    for nblk in (1, 7, 65):
        ndat = nblk * nsub + 5
        if kind == "f":
            raw = rng.standard_normal((nchan, npol, ndat, 2)).astype(np.float32)
            x = raw.astype(np.float64).view(np.complex128)[..., 0]
        else:
            dt, s = (np.int8, 20) if kind == "i8" else (np.int16, 3000)
            raw = np.clip(np.round(rng.standard_normal((ndat, nchan, npol, 2)) * s), -127, 127 if
                          kind == "i8" else 32767).astype(dt)
            v = lut[raw.view(np.uint8)].astype(np.float64) if kind == "i8" else raw + 0.5
            x = np.ascontiguousarray(np.moveaxis(v, 0, 2)).view(np.complex128)[..., 0]
        out = torch.full((nchan * nsub, npol, nblk + 3, 2), 7.0, device="cuda")
        d = torch.from_numpy(raw).cuda()
        n = ctx.filterbank(kinds[kind], d, ndat, nchan, npol, nsub, out, nblk + 3,
                           in_span=ndat if kind == "f" else 0, lut=lut if kind == "i8" else None)
        ctx.synchronize()
        assert n == nblk
        got = out.cpu().numpy()
        assert np.all(got[:, :, nblk:] == 7.0)            # nothing past the output's end
        ref = np.fft.fft(x[:, :, :nblk * nsub].reshape(nchan, npol, nblk, nsub)) / np.sqrt(nsub)
        ref = np.transpose(ref, (0, 3, 1, 2)).reshape(nchan * nsub, npol, nblk)
        g = np.ascontiguousarray(got[:, :, :nblk]).view(np.complex64)[..., 0]
        assert rel_rms(g, ref) < VOLTAGE_RTOL


def test_filterbank_captured_at_its_first_call(b2):
    """Up to 1024 channels a call sets nothing up: its first one, at a length
    other than the last call's, can be captured."""
    st = torch.cuda.Stream()
    ctx = b2.Context(0, st.cuda_stream)
    ndat = 1 << 15
    d = torch.randn((1, 2, ndat, 2), device="cuda")
    out = torch.zeros((1024, 2, 300, 2), device="cuda")
    torch.cuda.synchronize()
    for nsub in (2048, 256, 1024, 128):
        want = torch.zeros_like(out)
        got = torch.zeros_like(out)
        torch.cuda.synchronize()
        if nsub > 1024:
            ctx.filterbank(b2.FLOAT_FPT, d, ndat, 1, 2, nsub, out, 300, in_span=ndat)
            ctx.synchronize()
            continue
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            ctx.filterbank(b2.FLOAT_FPT, d, ndat, 1, 2, nsub, got, 300, in_span=ndat)
        g.replay()
        ctx.filterbank(b2.FLOAT_FPT, d, ndat, 1, 2, nsub, want, 300, in_span=ndat)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and bool((want != 0).any())
    ctx.close()


@pytest.mark.parametrize("lin", [64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("kind,npol", [("i16", 2), ("i8", 1), ("f", 2)])
def test_inverse_filterbank_sizes(ctx, b2, orc, lin, kind, npol):
    """Fine-channel transforms of every size, channels that do not fill the
    last block, against the oracle in 64 bits."""
    kinds = dict(i8=b2.INT8_TFPD, i16=b2.INT16_TFPD, f=b2.FLOAT_FPT)
    nin = max(16384 // lin * 2, 16) if lin <= 1024 else 16
    while nin * lin * 3 // 4 > 196608 or (nin * lin * 3 // 4) % 4096:
        nin *= 2
    disc = nin * 3
    rng = np.random.default_rng(lin)
    ifb = b2.InverseFilterbank(ctx, nin, 1, nin, npol, lin, os=(4, 3), output_discard=(disc, disc))
    info = ifb.info
    ndat = 2 * info["in_step"] + info["in_discard_pos"] + info["in_discard_neg"] + 3
    lut, _ = b2.bittable8()
    if kind == "f":
        raw = rng.standard_normal((nin, npol, ndat, 2)).astype(np.float32)
        x = raw.view(np.complex64)[..., 0]
    else:
        dt, s = (np.int8, 20) if kind == "i8" else (np.int16, 3000)
        raw = np.clip(np.round(rng.standard_normal((ndat, nin, npol, 2)) * s), -127,
                      127 if kind == "i8" else 32767).astype(dt)
        v = lut[raw.view(np.uint8)] if kind == "i8" else (raw + np.float32(0.5)).astype(np.float32)
        x = np.ascontiguousarray(np.moveaxis(v, 0, 2)).view(np.complex64)[..., 0]
    cfg = dict(input_nchan=nin, output_nchan=1, pfb_nchan=nin, npol=npol, input_fft_length=lin,
               os_num=4, os_den=3, output_discard_pos=disc, output_discard_neg=disc,
               pfb_dc_chan=1, pfb_all_chan=1, dual_sideband=1)
    ref = orc.inverse_filterbank(x.astype(np.complex128), cfg, fp64=True)
    n = 2 * info["out_step"]
    out = torch.zeros((1, npol, n, 2), device="cuda")
    assert ifb.perform(torch.from_numpy(raw).cuda(), ndat, out, n, input_kind=kinds[kind],
                       lut=lut if kind == "i8" else None) == 2
    ctx.synchronize()
    assert rel_rms(out.cpu().numpy().view(np.complex64)[..., 0], ref) < VOLTAGE_RTOL


@pytest.mark.parametrize("lin,nin,npol", [(64, 512, 1), (128, 256, 2), (256, 128, 1), (512, 128, 2),
                                          (1024, 256, 1), (1024, 64, 2), (2048, 16, 2)])
@pytest.mark.parametrize("kind", ["i16", "f"])
def test_inverse_filterbank_windows(ctx, b2, orc, lin, nin, npol, kind):
    """Response and both windows, with rows of the stitched spectra shorter and
    longer than the threads of a transform, both splits of the transforms."""
    disc = nin * 3
    rng = np.random.default_rng(lin + nin)
    ifb = b2.InverseFilterbank(ctx, nin, 1, nin, npol, lin, os=(4, 3), output_discard=(disc, disc))
    info = ifb.info
    lout = info["lout"]
    resp = (np.exp(2j * np.pi * rng.random((1, lout))) * rng.uniform(0.5, 1.5, (1, lout))).astype(np.complex64)
    temporal = b2.apodization(b2.APOD_TUKEY, lin, info["in_discard_pos"], info["in_discard_neg"])
    spectral = b2.apodization(b2.APOD_HANNING, lout, swap_halves=True)
    ifb.copy_response(resp)
    ifb.set_apodization(temporal, spectral)
    ndat = 2 * info["in_step"] + info["in_discard_pos"] + info["in_discard_neg"]
    raw = np.clip(np.round(rng.standard_normal((ndat, nin, npol, 2)) * 3000), -32768, 32767).astype(np.int16)
    v = (raw + np.float32(0.5)).astype(np.float32)
    x = np.ascontiguousarray(np.moveaxis(v, 0, 2)).view(np.complex64)[..., 0]
    data = raw if kind == "i16" else x.view(np.float32)
    cfg = dict(input_nchan=nin, output_nchan=1, pfb_nchan=nin, npol=npol, input_fft_length=lin,
               os_num=4, os_den=3, output_discard_pos=disc, output_discard_neg=disc,
               pfb_dc_chan=1, pfb_all_chan=1, dual_sideband=1)
    ref = orc.inverse_filterbank(x, cfg, response=resp, temporal=temporal, spectral=spectral, fp64=True)
    n = 2 * info["out_step"]
    out = torch.zeros((1, npol, n, 2), device="cuda")
    assert ifb.perform(torch.from_numpy(data).cuda(), ndat, out, n,
                       input_kind=b2.INT16_TFPD if kind == "i16" else b2.FLOAT_FPT) == 2
    ctx.synchronize()
    assert rel_rms(out.cpu().numpy().view(np.complex64)[..., 0], ref) < VOLTAGE_RTOL
    ifb.close()


@pytest.mark.parametrize("npol,nbin,per_bin", [(1, 64, 700.0), (2, 500, 0.3), (3, 100, 9.0),
                                               (4, 128, 9.0), (4, 32, 3000.0), (5, 64, 1.0)])
def test_fold_runs_of_every_length(ctx, b2, orc, npol, nbin, per_bin):
    """Rows inside one bin, rows of single samples and rows in between."""
    nchan, ndat = 3, 20011
    rng = np.random.default_rng(nbin)
    data = rng.random((nchan, npol, ndat), dtype=np.float32) + np.float32(0.1)
    phi, pps = 0.123, 1.0 / (per_bin * nbin)
    plan = orc.fold_binplan(phi, pps, ndat, nbin)
    rprof, rhits = orc.fold_accumulate(data.astype(np.float64), plan, nbin)
    f = b2.Fold(ctx, nbin, nchan, npol)
    f.set_bins(phi, pps, ndat)
    f.fold(torch.from_numpy(data).cuda(), ndat)
    prof, hits = f.get_profiles()
    f.close()
    assert np.array_equal(hits, rhits)
    hit = rhits > 0
    assert np.all(prof[..., ~hit] == 0)
    assert np.max(np.abs(prof - rprof)[..., hit] / rprof[..., hit]) < 1e-5


@pytest.mark.parametrize("npol", [1, 2])
def test_fused_4096_side_by_side_and_in_turn(ctx, b2, orc, npol):
    """4096-point parts with one, two, three and five blocks per SM: the same
    bits however many parts a call has, and right against 64 bits."""
    nfft, pos, neg = 4096, 300, 211
    nk = nfft - pos - neg
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    counts = [nsm // 2, 2 * nsm, 2 * nsm + 1, 4 * nsm + 1]
    total = sum(counts)
    ndat = total * nk + pos + neg
    gen = torch.Generator(device="cuda").manual_seed(npol)
    d = torch.randn((1, npol, ndat, 2), device="cuda", generator=gen)
    rng = np.random.default_rng(npol)
    h = np.exp(2j * np.pi * rng.random((1, nfft))).astype(np.complex64) / np.float32(np.sqrt(nfft))
    c = b2.Convolution(ctx, 1, npol, nfft, pos, neg)
    c.copy_response(h)
    whole = torch.zeros((1, npol, total * nk, 2), device="cuda")
    assert c.perform(d, ndat, ndat, whole, total * nk) == total
    first = 0
    for n in counts:
        part = torch.zeros((1, npol, n * nk, 2), device="cuda")
        piece = d[:, :, first * nk:first * nk + n * nk + pos + neg].contiguous()
        assert c.perform(piece, piece.shape[2], piece.shape[2], part, n * nk) == n
        ctx.synchronize()
        assert torch.equal(part, whole[:, :, first * nk:(first + n) * nk])
        first += n
    c.close()
    x = d[:, :, :3 * nk + pos + neg].cpu().numpy().astype(np.float64).view(np.complex128)[..., 0]
    ref = orc.convolve(x, h.astype(np.complex128), nfft, pos, neg)
    got = whole[:, :, :3 * nk].cpu().numpy().view(np.complex64)[..., 0]
    assert rel_rms(got, ref) < VOLTAGE_RTOL


def test_rows_change_with_the_arithmetic(ctx, b2, orc):
    """An engine with its default rows, then tensor-core rows, then FP32
    again: the response follows the split."""
    nfft, pos, neg = 1 << 15, 1000, 500
    rng = np.random.default_rng(3)
    h = np.exp(2j * np.pi * rng.random((2, nfft))).astype(np.complex64) / np.float32(np.sqrt(nfft))
    nk = nfft - pos - neg
    ndat = nfft + nk
    x = (rng.standard_normal((2, 2, ndat)) + 1j * rng.standard_normal((2, 2, ndat))).astype(np.complex64)
    ref = orc.convolve(x.astype(np.complex128), h.astype(np.complex128), nfft, pos, neg)
    c = b2.Convolution(ctx, 2, 2, nfft, pos, neg)
    c.copy_response(h)
    d = torch.from_numpy(x.view(np.float32)).cuda()
    for mode in (b2.FFT_FP32, b2.FFT_BF16X3, b2.FFT_FP32):
        c.set_fft_precision(mode)
        assert np.array_equal(c.get_response(), h)
        out = torch.zeros((2, 2, 2 * nk), dtype=torch.complex64, device="cuda")
        assert c.perform(d, ndat, ndat, out, 2 * nk) == 2
        c.status()
        assert rel_rms(out.cpu().numpy(), ref) < VOLTAGE_RTOL
    c.close()


def test_change_of_the_arithmetic_then_of_the_stream(b2, orc):
    """The second split's response is in place before a call on another stream."""
    nfft, nchan = 1 << 16, 64
    rng = np.random.default_rng(9)
    h = np.exp(2j * np.pi * rng.random((nchan, nfft))).astype(np.complex64) / np.float32(np.sqrt(nfft))
    x = (rng.standard_normal((nchan, 2, nfft)) + 1j * rng.standard_normal((nchan, 2, nfft))).astype(np.complex64)
    ref = orc.convolve(x.astype(np.complex128), h.astype(np.complex128), nfft, 100, 100)
    streams = [torch.cuda.Stream() for _ in range(2)]
    ctx = b2.Context(0, streams[0].cuda_stream)
    c = b2.Convolution(ctx, nchan, 2, nfft, 100, 100)
    c.copy_response(h)
    d = torch.from_numpy(x.view(np.float32)).cuda()
    out = torch.zeros((nchan, 2, nfft - 200), dtype=torch.complex64, device="cuda")
    busy = torch.zeros(1 << 28, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        for _ in range(20):
            busy.add_(1.0)
    c.set_fft_precision(b2.FFT_BF16X3)
    ctx.set_stream(streams[1].cuda_stream)
    assert c.perform(d, nfft, nfft, out, nfft - 200) == 1
    torch.cuda.synchronize()
    assert rel_rms(out.cpu().numpy(), ref) < VOLTAGE_RTOL
    c.close()
    ctx.close()


def test_captured_calls_survive_a_change_of_the_arithmetic(b2, orc):
    """Graphs captured with one row length replay rightly after the engine has
    changed to the other, also with a response set in between."""
    nfft, pos, neg = 1 << 15, 700, 900
    rng = np.random.default_rng(8)
    h = np.exp(2j * np.pi * rng.random((2, 1, nfft))).astype(np.complex64) / np.float32(np.sqrt(nfft))
    nk = nfft - pos - neg
    ndat = nfft + 40 * nk
    x = (rng.standard_normal((1, 2, ndat)) + 1j * rng.standard_normal((1, 2, ndat))).astype(np.complex64)
    ref = [orc.convolve(x.astype(np.complex128), r.astype(np.complex128), nfft, pos, neg) for r in h]
    st = torch.cuda.Stream()
    ctx = b2.Context(0, st.cuda_stream)
    c = b2.Convolution(ctx, 1, 2, nfft, pos, neg)
    c.copy_response(h[0])
    d = torch.from_numpy(x.view(np.float32)).cuda()
    out = torch.zeros((1, 2, 41 * nk), dtype=torch.complex64, device="cuda")
    torch.cuda.synchronize()

    def perform():
        assert c.perform(d, ndat, ndat, out, 41 * nk) == 41

    def check(what, r):
        out.zero_()
        torch.cuda.synchronize()
        what()
        torch.cuda.synchronize()
        assert rel_rms(out.cpu().numpy(), ref[r]) < VOLTAGE_RTOL

    graphs = []
    for mode in (b2.FFT_FP32, b2.FFT_BF16X3):
        c.set_fft_precision(mode)
        check(perform, 0)                  # and what a first call sets up
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            perform()
        graphs.append(g)
    for g in graphs:
        check(g.replay, 0)
    c.copy_response(h[1])
    for g in graphs:
        check(g.replay, 1)
    c.set_fft_precision(b2.FFT_FP32)
    check(perform, 1)
    for g in graphs:
        check(g.replay, 1)
    assert np.array_equal(c.get_response(), h[1])
    c.status()
    del graphs, g
    c.close()
    ctx.close()


# spectral kurtosis: 8, 4, 2 and 1 blocks per thread block at the edges of the
# shared tile, counts that leave the last one partly empty
SK_EDGES = [(4, 2, 636, 9), (4, 2, 638, 9), (4, 2, 1276, 7), (4, 2, 1278, 7), (4, 2, 2556, 5),
            (4, 2, 2558, 5), (4, 1, 1276, 17), (4, 1, 1278, 17), (4, 2, 30, 49)]


@pytest.mark.parametrize("nchan,npol,M,npart", SK_EDGES)
@pytest.mark.parametrize("inplace", [False, True])
def test_sk_tiles_bit_exact(ctx, b2, orc, nchan, npol, M, npart, inplace):
    sk.test_sk_kernel_bit_exact(ctx, b2, orc, nchan, npol, M, npart * M + 6, 0, False, 1, inplace)
