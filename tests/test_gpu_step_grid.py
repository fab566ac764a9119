"""The step kernel serves one work-list entry per thread: a launch with fewer threads than its
lists hold must reject the round (failure flag 32) instead of losing photons."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QUEUE_CORRUPT = 32


@pytest.mark.parametrize("block", [64, 256])
@pytest.mark.parametrize("photons, short", [(256, 0), (256, 1), (3000, 0), (3000, 1), (3000, 5), (70000, 0), (70000, 100)])
def test_a_launch_too_small_for_its_lists_is_reported(native, device, block, photons, short):
    import monki.scenes as scenes
    from monki.execution.native import F64P

    scene = scenes.box_cloud(70000, 1, nx=12, ny=10, box_x=(3, 8), box_y=(2, 6))
    tables = np.ascontiguousarray(scene.tables)
    err = ctypes.create_string_buffer(2048)
    handle = native.monki_cuda_create(0, tables.ctypes.data_as(F64P), tables.size, 1, f"pool=66000,block={block}".encode(),
                                      err, len(err))
    assert handle, err.value
    try:
        entries = min(66000, (photons + 255) // 256 * 256)
        blocks = -(-entries // block) - short
        flag = (ctypes.c_uint32 * 1)()
        controls = (ctypes.c_uint32 * 8)(photons, 0, 1, 7, 100000, 0, photons, 1)
        if blocks < 1:
            return  # one block: nothing to leave out
        assert native.monki_cuda_probe_step(handle, controls, blocks, flag, err, len(err)) == 0, err.value
        assert flag[0] == (QUEUE_CORRUPT if short else 0)
        # The session is unharmed.
        out = np.zeros(int(native.monki_cuda_tally_count(handle)))
        assert native.monki_cuda_run(handle, controls, out.ctypes.data_as(F64P), err, len(err)) == 0, err.value
        assert out.sum() > 0
    finally:
        native.monki_cuda_close(handle)
