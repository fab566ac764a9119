"""The library's host code over ``fake_cuda.cpp``: device memory is host memory, kernels do not
run, and every runtime call is recorded and may be failed.

The compiled units come from the library's own build (``_build/*.o``), so what is tested is
the object code that the library links.
"""

from __future__ import annotations

import ctypes
import importlib.util
import shutil
import subprocess
from dataclasses import dataclass
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "monki-gpu_gb300"


@dataclass(frozen=True)
class Event:
    call: str
    kernel: str = ""
    stream: int = 0
    pointer: int = 0
    value: int = 0  # bytes, dynamic shared memory of a launch, or the attribute's value
    grid: int = 0


_HOOK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_char_p, ctypes.c_char_p, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_uint64,
                         ctypes.c_uint64)


def build(directory: Path, units) -> Path:
    """Link the compiled ``units`` of the library with the runtime of host memory."""

    spec = importlib.util.spec_from_file_location("monki_build_native", PACKAGE / "build_native.py")
    native = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(native)
    if not shutil.which("g++"):
        pytest.skip("needs a host compiler")
    native.build()
    objects = [PACKAGE / "_build" / f"{unit}.o" for unit in units]
    if not all(o.is_file() for o in objects):
        native.build(force=True)
    output = directory / "libmonki_host.so"
    include = Path(native.nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{include}",
                    str(ROOT / "tests" / "fake_cuda.cpp"), *map(str, objects), "-o", str(output)], check=True)
    return output


class Runtime:
    """The calls of one test: ``events`` lists them; ``on_call(event)`` may return an error."""

    def __init__(self, library: Path):
        self.library = ctypes.CDLL(str(library))
        self.events: list[Event] = []
        self.on_call = lambda event: 0
        self._hook = _HOOK(self._record)
        self.library.fake_hook(self._hook)

    def _record(self, call, kernel, stream, pointer, value, grid):
        event = Event(call.decode(), kernel.decode(), stream, pointer, value, grid)
        self.events.append(event)
        return self.on_call(event) or 0

    def close(self):
        self.library.fake_hook(_HOOK())
