"""A caller's own shaders give the same bytes drawn in one call and in many
(tests/cpp/user_split_test.cu)."""
import os
import subprocess

import pytest

from .test_user_shader import ROOT, BUILD, _nvcc

pytestmark = pytest.mark.gpu


def test_one_draw_equals_many(gpu_lib, tmp_path):
    from softwarerenderer_gb300 import build
    build.build()
    exe = os.path.join(tmp_path, "user_split_test")
    cmd = [_nvcc(), *build.ARCH, "-O3", "-std=c++17", "-fmad=false", "-prec-div=true", "-prec-sqrt=true", "-ftz=false",
           "--expt-relaxed-constexpr", "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(ROOT, "tests", "cpp"), os.path.join(ROOT, "tests", "cpp", "user_split_test.cu"),
           "-L", BUILD, "-lswr_gb300", "-Xlinker", "-rpath=" + BUILD, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
