"""Compiles a small host program over the headers of the device code (their
__host__ __device__ functions) with the library's compiler, and runs it."""
import os
import subprocess

from mcmtop_b200 import build


def run(tmp_path, source: str, *flags: str) -> str:
    src, exe = os.path.join(tmp_path, "program.cu"), os.path.join(tmp_path, "program")
    with open(src, "w") as f:
        f.write(source)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Xcompiler",
                    "-ffp-contract=off", *flags, "-I", build.CSRC, src, "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout
