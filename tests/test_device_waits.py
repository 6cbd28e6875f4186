"""Device-side waits that give up: the bound of the wait itself, and the
status that reaches whoever takes results after one has run out.  No test
makes a kernel fault: a barrier is left alone until its wait ends, or the
engine's status word is set as the row kernel sets it."""
import os
import subprocess

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
