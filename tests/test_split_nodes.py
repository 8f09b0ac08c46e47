"""The node launches' split grid (items.cuh) visits every node once, sides and
inner nodes apart, on small, ragged and long thin meshes (host-compiled,
CPU)."""
from __future__ import annotations

import subprocess

from test_native_math import ROOT, _nvcc


def test_split_nodes(tmp_path):
    exe = tmp_path / "check_split_nodes"
    subprocess.run([_nvcc(), "-std=c++17", "-O2", "-I", str(ROOT / "include"),
                    "-I", str(ROOT / "mahyco_gb300" / "csrc"),
                    "-x", "cu", str(ROOT / "tests" / "native" / "check_split_nodes.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    checked, bad = map(int, res.stdout.split())
    assert checked == 17 * 17 + 23 and bad == 0
