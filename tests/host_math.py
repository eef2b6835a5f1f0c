"""Compiles parts of the kernels' sources with the host's compiler, so that their index and
rounding arithmetic is checked without a GPU."""

from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

from terraingen_b200.build import CSRC, nvcc


def compiled(directory: Path, source: str) -> C.CDLL:
    """The functions of `source` (C++, its entry points extern "C") as a library."""
    unit, library = directory / "unit.cpp", directory / "unit.so"
    unit.write_text(source)
    cuda = Path(nvcc()).resolve().parents[1] / "include"
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC",
                    "-shared", "-w", "-I", str(CSRC), "-I", str(cuda), "-o", str(library),
                    str(unit)], check=True)
    return C.CDLL(str(library))
