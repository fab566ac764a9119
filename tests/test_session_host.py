"""Host code of the single-scene session (csrc/session.cu) over a runtime of host memory."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

COUNT_WORDS, CLAIMED = 20, 16  # words of the read-back counts; index of the claim counter
LAUNCH_FAILED = 719


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    import fake_cuda

    return fake_cuda.build(tmp_path_factory.mktemp("host"), ("session", "tail"))


@pytest.mark.parametrize("config, failing", [("tail=0", "graph kernel"), ("tail=0,graphs=0", "launch"), ("", "tail"),
                                             ("engine=megakernel", "transport")])
def test_a_run_after_a_failed_one_starts_from_empty_tallies(library, config, failing):
    import fake_cuda
    import monki.scenes as scenes

    runtime = fake_cuda.Runtime(library)
    native = runtime.library
    native.monki_cuda_create.restype = ctypes.c_void_p
    native.monki_cuda_tally_count.restype = ctypes.c_size_t
    scene = scenes.box_cloud(2000, 1, nx=15, ny=11, box_x=(3, 8), box_y=(2, 6))
    tables = np.ascontiguousarray(scene.tables)
    photons = 2000 * 15 * 11
    f64p = ctypes.POINTER(ctypes.c_double)
    error = ctypes.create_string_buffer(2048)
    handle = native.monki_cuda_create(0, tables.ctypes.data_as(f64p), ctypes.c_size_t(tables.size), 1,
                                      f"pool=262144,{config}".encode(), error, ctypes.c_size_t(2048))
    assert handle, error.value
    handle = ctypes.c_void_p(handle)
    (banks,) = {(e.pointer, e.value) for e in runtime.events if e.call == "memset"}
    counts = [e.pointer for e in runtime.events if e.call == "malloc host" and e.value == 4 * COUNT_WORDS]
    out = np.zeros(native.monki_cuda_tally_count(handle))
    controls = (ctypes.c_uint32 * 8)(photons, 0, 1, 7, 100000, 0, photons, 1)
    kernel = {"tail": "wf_tail", "transport": "transport_kernel"}.get(failing, "wf_step")
    failures = [LAUNCH_FAILED]
    batches = []

    def on_call(event):
        if event.call == "copy" and event.pointer in counts:
            words = (ctypes.c_uint32 * COUNT_WORDS).from_address(event.pointer)
            ctypes.memset(words, 0, ctypes.sizeof(words))
            words[2] = 100 if not batches else 0
            words[CLAIMED] = photons
            batches.append(1)
        if kernel in event.kernel and failures:
            return failures.pop()
        return 0

    runtime.on_call = on_call
    run = lambda: native.monki_cuda_run(handle, controls, out.ctypes.data_as(f64p), error, ctypes.c_size_t(2048))  # noqa: E731
    assert run() == 1 and b"failed by the test" in error.value
    first = len(runtime.events)
    batches.clear()
    assert run() == 0, error.value
    events = runtime.events[first:]
    started = next(n for n, e in enumerate(events) if e.kernel)
    assert banks in {(e.pointer, e.value) for e in events[:started] if e.call == "memset"}
    # A run after a whole one does not clear them again.
    first = len(runtime.events)
    batches.clear()
    assert run() == 0, error.value
    events = runtime.events[first:]
    started = next(n for n, e in enumerate(events) if e.kernel)
    assert banks not in {(e.pointer, e.value) for e in events[:started] if e.call == "memset"}
    native.monki_cuda_close(handle)
    runtime.close()
