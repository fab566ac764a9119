"""Host code of the multi-scene session (csrc/multi.cu, csrc/tail.cu) over a runtime of host
memory: the order of its calls and what it does when one fails, with the read-back counts of
each wavefront batch supplied by the test.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

COUNT_WORDS, CLAIMED = 20, 16  # words per scene of the read-back counts; index of the claim counter
LAUNCH_FAILED = 719


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    import fake_cuda

    return fake_cuda.build(tmp_path_factory.mktemp("host"), ("multi", "tail"))


class Session:
    """A multi-scene session of one scene per group (I, and I/Q/U). ``live[group]`` lists the
    photons left after each batch, every photon claimed from the second batch on; a group whose
    list has ended has none left."""

    def __init__(self, library, config, live=((), ())):
        import fake_cuda
        import monki.scenes as scenes

        self.runtime = fake_cuda.Runtime(library)
        self.native = self.runtime.library
        self.native.monki_cuda_multi_create.restype = ctypes.c_void_p
        self.native.monki_cuda_multi_tally_count.restype = ctypes.c_size_t
        self.scenes = [scenes.clear_sky(2000, 1, nx=12, ny=10),
                       scenes.box_cloud(2000, 1, nx=15, ny=11, box_x=(3, 8), box_y=(2, 6))]
        self.photons = [s.photons_per_column * s.shape[1] * s.shape[2] for s in self.scenes]
        tables = [np.ascontiguousarray(s.tables) for s in self.scenes]
        f64p = ctypes.POINTER(ctypes.c_double)
        pointers = (f64p * 2)(*[t.ctypes.data_as(f64p) for t in tables])
        sizes = (ctypes.c_size_t * 2)(*[t.size for t in tables])
        self.error = ctypes.create_string_buffer(2048)
        self.handle = self.native.monki_cuda_multi_create(0, 2, pointers, sizes, 1, config.encode(), self.error, 2048)
        assert self.handle, self.error.value
        # The pinned count buffers: the groups' host_counts, in the order of their creation.
        self.counts = [e.pointer for e in self.runtime.events if e.call == "malloc host" and e.value == 4 * COUNT_WORDS]
        assert len(self.counts) == 2
        self.batches = [0, 0]
        self.live = live
        self.fail = lambda event: 0
        self.runtime.on_call = self._on_call

    def _on_call(self, event):
        if event.call == "copy" and event.pointer in self.counts:
            group = self.counts.index(event.pointer)
            words = (ctypes.c_uint32 * COUNT_WORDS).from_address(event.pointer)
            batch, left = self.batches[group], self.live[group]
            ctypes.memset(words, 0, ctypes.sizeof(words))
            words[2] = left[batch] if batch < len(left) else 0
            words[CLAIMED] = self.photons[group] if batch else 0
            self.batches[group] = batch + 1
        return self.fail(event)

    def run(self):
        controls = np.zeros((2, 8), dtype=np.uint32)
        for q, photons in enumerate(self.photons):
            controls[q] = [photons, 0, 1, 7, 100000, 0, photons, 1]
        outs = [np.zeros(self.native.monki_cuda_multi_tally_count(ctypes.c_void_p(self.handle), q)) for q in range(2)]
        f64p = ctypes.POINTER(ctypes.c_double)
        out = (f64p * 2)(*[o.ctypes.data_as(f64p) for o in outs])
        self.first = len(self.runtime.events)
        return self.native.monki_cuda_multi_run(ctypes.c_void_p(self.handle), controls.ctypes.data_as(ctypes.c_void_p),
                                                out, self.error, 2048)

    def of_run(self):
        return self.runtime.events[self.first :]

    def close(self):
        self.native.monki_cuda_multi_close(ctypes.c_void_p(self.handle))
        self.runtime.close()


def _grids(events, kernel):
    grids = []
    for e in events:
        if kernel in e.kernel and (not grids or grids[-1] != e.grid):
            grids.append(e.grid)
    return grids


def test_shrunk_launches_replay_a_graph(library):
    """The launches of a group that is draining cover its live entries, and stay graph replays:
    launched kernel by kernel, a drain without tail launches took longer than with full-size
    graphs (four small scenes 131 ms with those, 154 launched one by one)."""

    session = Session(library, "pool=262144,check_every=2,tail=0,graphs=1",
                      live=((240000, 100000, 5000, 300), (330000, 330000, 200)))
    assert session.run() == 0, session.error.value
    wavefront = [e for e in session.of_run() if "wf_step_multi" in e.kernel or "wf_peel_multi" in e.kernel]
    assert {e.call for e in wavefront} == {"graph kernel"}
    streams = list(dict.fromkeys(e.stream for e in wavefront))
    full = [-(-p // 256) for p in (240000, 262144)]
    for kernel in ("wf_step_multi", "wf_peel_multi"):
        first, second = ([e for e in wavefront if e.stream == s] for s in streams)
        assert _grids(first, kernel) == [full[0], -(-100000 // 256), -(-5000 // 256), 2]
        assert _grids(second, kernel) == [full[1], 1]
    session.close()


def test_without_graphs_shrunk_launches_are_launched_directly(library):
    session = Session(library, "pool=262144,check_every=2,tail=0,graphs=0", live=((240000, 100000, 5000), (200, 0)))
    assert session.run() == 0, session.error.value
    assert not [e for e in session.of_run() if e.call.startswith("graph")]
    step = [e for e in session.of_run() if "wf_step_multi" in e.kernel]
    first = [e for e in step if e.stream == step[0].stream]
    assert _grids(first, "wf_step_multi") == [-(-240000 // 256), -(-100000 // 256), -(-5000 // 256)]
    session.close()


@pytest.mark.parametrize("graphs", [1, 0])
@pytest.mark.parametrize("failing", ["launch", "shrink"])
def test_a_failed_run_waits_for_the_tails_it_launched(library, graphs, failing):
    """The first group's tail is launched, then a call of the second group fails: the run ends
    only after the tail, which writes the pool and the tally banks that the next run resets."""

    session = Session(library, f"pool=262144,check_every=2,tail=65536,graphs={graphs}",
                      live=((240000, 100), (330000, 300000, 100000, 80000)))

    def fail(event):
        events = session.of_run()
        if not any("wf_tail" in e.kernel for e in events):
            return 0
        if failing == "launch":
            return LAUNCH_FAILED if "wf_step_multi" in event.kernel or event.call == "graph launch" else 0
        return LAUNCH_FAILED if event.call == "copy" and event.pointer not in session.counts else 0

    session.fail = fail
    assert session.run() == 1
    assert b"failed by the test" in session.error.value
    events = session.of_run()
    tails = [n for n, e in enumerate(events) if "wf_tail" in e.kernel]
    assert tails
    for n in tails:
        assert any(e.call == "synchronize" and e.stream == events[n].stream for e in events[n:])
    session.close()


def test_close_waits_for_every_stream_before_it_frees(library):
    session = Session(library, "pool=262144,check_every=2", live=((240000, 100), (330000, 200)))
    streams = {e.stream for e in session.runtime.events if e.call == "stream"}
    assert session.run() == 0, session.error.value
    first = len(session.runtime.events)
    session.native.monki_cuda_multi_close(ctypes.c_void_p(session.handle))
    events = session.runtime.events[first:]
    freed = next(n for n, e in enumerate(events) if e.call.startswith("free"))
    assert {e.stream for e in events[:freed] if e.call == "synchronize"} == streams
    session.runtime.close()


def test_a_tail_launch_lowers_no_other_sessions_shared_memory_limit(library):
    """A kernel's dynamic shared-memory limit belongs to the kernel: sessions of other scenes
    launch it from other threads, so no launch may set it to its own scene's band."""

    session = Session(library, "pool=262144,check_every=2", live=((240000, 100), (330000, 200)))
    assert session.run() == 0, session.error.value
    tails = [e for e in session.of_run() if "wf_tail" in e.kernel and e.call == "launch"]
    assert any(e.value > 0 for e in tails)  # a staged band
    assert {e.value for e in session.runtime.events if e.call == "attribute"} <= {48 * 1024}
    session.close()


def test_a_run_after_a_failed_one_starts_from_empty_tallies(library):
    session = Session(library, "pool=262144,check_every=2", live=((240000, 100), (330000, 200)))
    banks = {(e.pointer, e.value) for e in session.runtime.events if e.call == "memset"}
    assert len(banks) == 2
    session.fail = lambda event: LAUNCH_FAILED if "wf_tail" in event.kernel else 0
    assert session.run() == 1
    session.fail = lambda event: 0
    session.batches = [0, 0]
    assert session.run() == 0, session.error.value
    events = session.of_run()
    started = next(n for n, e in enumerate(events) if "wf_" in e.kernel)
    assert banks <= {(e.pointer, e.value) for e in events[:started] if e.call == "memset"}
    session.close()
