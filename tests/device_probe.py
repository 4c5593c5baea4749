"""Builds and loads device_probe.cu (device functions called on host arrays)."""

import ctypes
import os
import subprocess

from ddhdg_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def load(directory):
    """The probe library, compiled into `directory`."""
    lib = os.path.join(str(directory), "device_probe.so")
    subprocess.check_call([build.nvcc()] + build.NVCC_FLAGS + ["-shared", "-I", build.CSRC, "-o", lib,
                                                               os.path.join(HERE, "device_probe.cu")])
    return ctypes.CDLL(lib)


def dptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
