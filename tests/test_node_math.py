"""The scalar functions of the passes over frequency nodes (kg_log.cuh, kg_qp1.cuh,
kg_advance.cuh) against long double, built from tests/host/node_math.cu: on the host
in the CPU run, on the device in the GPU run.

Bounds, from the functions' terms (U = 2^-53):
  recip      the cubic step leaves e^3 <= 2^-60 of the approximation's 2^-20 and
             rounds once: within an ulp, 2 U relative;
  log        e log 2 and -log c from a table (each rounded), their sum and the
             series' sum: 4 U (1 + |log d|), for every d from 2^-32 to 2^32;
  neg_log1m  |z| <= 1/64: 1e-15 relative (the first term left out is 3.9e-16); else the
             logarithm's bound and 1 - z rounded, for ratios from 5e-9 to 1.9e8;
  step       what is left of the difference step along the iterate: the roundings of
             its nine terms;
  wave_bound the waves that a call may run: at least 11 passes of both forms for every
             iteration up to 2^40, whatever the limit (2 where it wraps);
  segments   the largest sum of signed digits in a 32-bit accumulator, of 2^31 (2 where a
             bin's segments are empty or leave stages out).
Errors are printed as fractions of these bounds."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def fractions(tmp_path, *args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "node_math")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(ROOT, "kestrel_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "host", "node_math.cu"), "-o", exe], check=True)
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    print(r.stdout)
    return {ln.split()[0]: float(ln.split()[1]) for ln in r.stdout.splitlines()}


def test_on_the_host(tmp_path):
    got = fractions(tmp_path)
    assert set(got) == {"recip", "log", "neg_log1m", "step", "wave_bound", "segments"}
    assert all(v <= 1.0 for v in got.values()), got


@pytest.mark.gpu
def test_on_the_device(tmp_path):
    got = fractions(tmp_path, "device")
    assert set(got) == {"recip", "log", "neg_log1m", "step", "wave_bound", "segments"}
    assert all(v <= 1.0 for v in got.values()), got
