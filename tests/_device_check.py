"""Builds and runs a small CUDA program of tests/cpp against libsphgpu.so."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(name, out_dir):
    from spheral_gb300 import build
    lib = os.path.join(ROOT, "spheral_gb300")
    exe = os.path.join(str(out_dir), name)
    cmd = [build._nvcc()] + build.ARCH + ["-O2", "-std=c++17", "-I" + build.CSRC, "-I" + build.INCLUDE,
                                          os.path.join(ROOT, "tests", "cpp", name + ".cu"), "-o", exe,
                                          "-L" + lib, "-lsphgpu", "-Xlinker", "-rpath," + lib]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
