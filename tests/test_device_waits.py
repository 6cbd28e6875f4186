"""Device-side waits that give up: the bound of the wait itself, and the
status that reaches whoever takes results after one has run out.  No test
makes a kernel fault: a barrier is left alone until its wait ends, or the
engine's status word is set as the row kernel sets it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dspsr-kanyixia_b200", "csrc")
OUT = os.path.join(ROOT, "tests", "cpp", "_build")
EXE = os.path.join(OUT, "wait_main")


def build():
    os.makedirs(OUT, exist_ok=True)
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "wait_main.cu"), "-o", EXE],
                   check=True, capture_output=True, text=True)


def test_wait_program_builds():
    build()
    assert os.path.exists(EXE)


@pytest.mark.gpu
def test_wait_gives_up_in_time():
    """A second, and what the last 16 polls may add to it."""
    if not os.path.exists(EXE):
        build()
    r = subprocess.run([EXE], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    done, left = [dict(kv.split("=") for kv in l.split()[1:]) for l in r.stdout.splitlines()]
    assert done["ok"] == "1" and float(done["ms"]) < 100.0
    assert left["ok"] == "0" and float(left["ms"]) < 3000.0


# ---- the status of a wait that gave up, seen by every caller -----------------

@pytest.fixture
def own(b2):
    """A context of its own: a status stays until its engine is destroyed."""
    c = b2.Context(0, None)
    yield c
    c.close()


def word_of(ctx, call, handle):
    w = ctypes.POINTER(ctypes.c_int)()
    ctx.check(call(handle, ctypes.byref(w)), "status_word")
    return w


def gave_up(b2):
    return pytest.raises(b2.B200Error, match="wait timed out")


@pytest.mark.gpu
def test_engine_status_reaches_its_callers(own, b2):
    torch = pytest.importorskip("torch")
    nfft, ndat = 1 << 14, 20000
    conv = b2.Convolution(own, 1, 2, nfft, 100, 100)
    conv.copy_response(np.ones((1, nfft), np.complex64))
    d = torch.zeros(ndat * 4, device="cuda")
    out = torch.zeros_like(d)
    conv.perform(d, ndat, ndat, out, ndat)
    fold = b2.Fold(own, 64, 1, 1)
    fold.set_bins(0.0, 1e-3, ndat)
    fold.fold(torch.zeros(ndat, device="cuda"), ndat)
    conv.status()
    own.synchronize()
    fold.get_profiles()
    word_of(own, own._lib.dspsr_b200_convolution_status_word, conv.handle)[0] = 1
    for call in (conv.status, own.synchronize, fold.get_profiles):
        with gave_up(b2):
            call()
    # a change of the arithmetic does not forget it
    conv.set_fft_precision(b2.FFT_BF16X3)
    with gave_up(b2):
        conv.status()
    conv.close()
    own.synchronize()


def pipeline(ctx, b2, **kw):
    nfft = 1 << 14
    return b2.Pipeline(ctx, b2.make_config(1400.0, 16.0, 1.0, 1, 2, nfft, 100, 100, 64, 0.004, **kw))


@pytest.mark.gpu
def test_pipeline_status_reaches_profiles(own, b2):
    torch = pytest.importorskip("torch")
    pl = pipeline(own, b2)
    d = torch.zeros(1 << 18, dtype=torch.uint8, device="cuda")
    pl.run(d, 1 << 16)
    pl.get_profiles()
    prof, hits = pl.profile_buffers()
    pl.get_profiles_async(prof, hits)
    pl.wait_profiles()
    word_of(own, own._lib.dspsr_b200_pipeline_status_word, pl.handle)[0] = 1
    with gave_up(b2):
        pl.get_profiles()
    pl.get_profiles_async(prof, hits)
    with gave_up(b2):
        pl.wait_profiles()
    pl.close()


@pytest.mark.gpu
def test_pipeline_status_reaches_subints(own, b2):
    """Sub-integrations of 4 ms: popped with the status, kept from the unloader."""
    torch = pytest.importorskip("torch")
    d = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    for unloader in (False, True):
        got = []
        pl = pipeline(own, b2, subint_seconds=0.004, subint_slots=8)
        if unloader:
            pl.set_unloader(lambda info, prof, hits: got.append(info["division"]))
        word = word_of(own, own._lib.dspsr_b200_pipeline_status_word, pl.handle)
        pl.run(d, 1 << 18)
        if unloader:
            pl.finish()
            seen = len(got)
            assert seen >= 2
        else:
            assert pl.subints_ready() >= 2
            pl.pop_subint()
        word[0] = 1
        with gave_up(b2):
            if unloader:
                pl.run(d, 1 << 18)
                pl.finish()
            else:
                pl.pop_subint()
        if unloader:
            assert len(got) == seen
        pl.close()
    own.synchronize()


@pytest.mark.gpu
def test_status_words_are_each_engines_own(own, b2):
    """Engines that come and go: each word starts at 0 and is seen by its own
    engine alone, also where another engine's set word was handed back."""
    engines = [b2.Convolution(own, 1, 2, 4096, 10, 10) for _ in range(1100)]
    words = [word_of(own, own._lib.dspsr_b200_convolution_status_word, c.handle) for c in engines]
    assert len({ctypes.addressof(w.contents) for w in words}) == len(engines)
    assert all(w[0] == 0 for w in words)
    words[7][0] = words[1050][0] = 1
    for i in (6, 8, 1049, 1051):
        engines[i].status()
    for i in (7, 1050):
        with gave_up(b2):
            engines[i].status()
        engines[i].close()
    own.synchronize()
    again = [b2.Convolution(own, 1, 2, 4096, 10, 10) for _ in range(3)]
    for c in again:
        c.status()
        assert word_of(own, own._lib.dspsr_b200_convolution_status_word, c.handle)[0] == 0
    for c in engines[:7] + engines[8:1050] + engines[1051:] + again:
        c.close()
