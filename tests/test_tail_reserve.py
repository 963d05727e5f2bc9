"""Radii can be set where there is no device memory for the marcher's list of
tail rays: renders then go without it.  Without a device every allocation
fails, so this needs none."""
import ctypes
import os
import subprocess

import torch

from renderer_ray_marching_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
OUT = os.path.join(HERE, "_build", "libtail_probe.so")


def test_no_memory_for_the_list_is_no_error():
    lib = build.build()
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + ".tmp%d" % os.getpid()
    subprocess.run([build._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "renderer_ray_marching_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(HERE, "tail_probe.cu"), "-o", tmp, lib,
                    "-Xlinker", "-rpath," + os.path.dirname(lib)], check=True)
    os.replace(tmp, OUT)
    assert ctypes.CDLL(OUT).tail_probe() == (1 if torch.cuda.is_available() else 0)
