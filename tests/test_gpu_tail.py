"""The tail kernel at the edges of its blocks: the end of a round group run by blocks that list
their photons in shared memory, against the FP64 oracle on the same streams.

Group sizes: one photon per block, a block with a partly filled warp, and more photons than
one resident wave of blocks holds (blocks then take more slots as their photons end). The
fused step leaves scatterings pending, the separate kernels (``fused=0``) do not; split copies
wait in their slots. Tolerance: the oracle-parity one (rtol 1e-6), equal event counts.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(native, scene, config, seed=9):
    from monki.execution.native import F64P, U64P

    tables = np.ascontiguousarray(scene.tables)
    _, nx, ny, _, _ = scene.shape
    per_round = scene.photons_per_column * nx * ny
    err = ctypes.create_string_buffer(2048)
    handle = native.monki_cuda_create(0, tables.ctypes.data_as(F64P), tables.size, 1, config.encode(), err, len(err))
    assert handle, err.value
    try:
        out = np.zeros(int(native.monki_cuda_tally_count(handle)))
        controls = [per_round, 0, 1, seed, 100000, 0, per_round, 1]
        words = (ctypes.c_uint32 * 8)(*controls)
        assert native.monki_cuda_run(handle, words, out.ctypes.data_as(F64P), err, len(err)) == 0, err.value
        counters = np.zeros(6, dtype=np.uint64)
        native.monki_cuda_counters(handle, counters.ctypes.data_as(U64P))
        return out, int(counters[0]), controls
    finally:
        native.monki_cuda_close(handle)


@pytest.mark.parametrize("fused", [1, 0])
@pytest.mark.parametrize("nx, ny, ppc", [(3, 1, 1), (7, 5, 9), (20, 20, 500)])
def test_tail_block_edges_reproduce_oracle(native, oracle, device, nx, ny, ppc, fused):
    import monki.scenes as scenes

    scene = scenes.clear_sky(ppc, 1, nx=nx, ny=ny)
    out, scatters, controls = _run(native, scene, f"precision=fp64,check_every=2,tail={1 << 20},fused={fused}")
    expected, counters = oracle.run(scene.tables, controls, 8)
    assert scatters == counters["scatters"]
    np.testing.assert_allclose(out, expected[0], rtol=1e-6, atol=1e-12)


@pytest.mark.parametrize("fused", [1, 0])
def test_tail_runs_waiting_split_copies(native, oracle, device, fused):
    import monki.scenes as scenes
    from monki import Guided

    scene = scenes.box_cloud(6, 1, nx=12, ny=10, box_x=(3, 8), box_y=(2, 6))
    guide = Guided(0.0, 0.25, 0.0, 2.0)
    out, scatters, controls = _run(native, scene, f"precision=fp64,check_every=2,fused={fused}" + guide.config(), seed=5)
    expected, counters = oracle.run(scene.tables, controls, 8, guide=guide.oracle())
    assert scatters == counters["scatters"]
    np.testing.assert_allclose(out, expected[0][: out.size], rtol=1e-6, atol=1e-12)
