"""Face lengths (scheme_math.cuh face_len) equal the reference's square root of
the summed squares bit for bit, also where the smaller component's square is
left out (host-compiled, CPU)."""
from __future__ import annotations

import subprocess

from test_native_math import ROOT, _nvcc


def test_face_len(tmp_path):
    exe = tmp_path / "check_face_len"
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off",
                    "-I", str(ROOT / "include"), "-I", str(ROOT / "mahyco_gb300" / "csrc"),
                    "-x", "cu", str(ROOT / "tests" / "native" / "check_face_len.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stdout + res.stderr
    checked, differ = map(int, res.stdout.split())
    assert checked == 12_000_000 and differ == 0
