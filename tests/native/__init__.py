"""Parts of the engine that need no GPU, compiled for the host with the
harnesses of this folder."""

import ctypes
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(os.path.dirname(HERE)), "imate_b200",
                    "csrc")


def load(name, folder):
    """Compile tests/native/<name>.cpp into the folder and load it."""
    lib = os.path.join(str(folder), name + ".so")
    subprocess.check_call(
        ["/usr/bin/g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC",
         "-shared", "-I" + CSRC, "-o", lib,
         os.path.join(HERE, name + ".cpp")])
    return ctypes.CDLL(lib)
