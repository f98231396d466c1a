"""The layout a caller's shader program is checked by names every structure that its launchers
take from the library: the arguments of VsOps' and PsOps' functions, read from the header."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OPS = os.path.join(ROOT, "softwarerenderer_gb300", "csrc", "swr_ops.h")


def test_every_argument_structure_is_in_the_layout(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = os.path.join(tmp_path, "layout")
    from softwarerenderer_gb300 import build
    r = subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-o", exe, os.path.join(ROOT, "tests", "cpp", "program_layout.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    layout = [int(x) for x in lines[0].split()[1:]]
    sizes = {k.replace("swr::", ""): int(v) for k, v in (line.split() for line in lines[1:])}
    text = open(OPS).read()
    ops = text[text.index("struct VsOps"):text.index("const VsOps* vs_ops")]
    taken = set(re.findall(r"\b(\w+Args|Swr\w+)\b", ops)) - {"SwrOverwrite", "SwrDepthMin", "SwrRasterSlices",
                                                             "SwrRasterChunk"}
    assert taken <= set(sizes), taken - set(sizes)
    for name, size in sizes.items():
        assert size in layout, name
    assert len(layout) == len(sizes)
