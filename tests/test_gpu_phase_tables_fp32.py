"""The node tables of plain particle species (the default) against the general tables of the same
particles in FP32 (``nodes=0``): single-scene kernels with and without layer paths, the tail
kernel, and the multi-scene kernels.

Both forms evaluate the same expressions, but in two places of a kernel, where the compiler may
contract them differently: a history that rounds differently now and then goes another way. As
for other FP32 kernels that inline the same functions: scatter counts within 0.05 %, and all but
0.1 % of the tally entries equal to FP32 summation order.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(angles, nmat, paths=False):
    import monki.scenes as scenes

    levels = np.array([0.0, 1.0, 2.0, 4.0, 10.0, 60.0])
    nx, ny = 5, 4
    depth = np.zeros((1, nx, ny, len(levels) - 1))
    depth[0, 1:4, 1:3, 1] = 3.0
    return np.ascontiguousarray(scenes.build_tables(
        nx=nx, ny=ny, levels_km=levels, nmat=nmat, solar_zenith=30.0, solar_azimuth=0.0, view_zeniths=[0.0, 40.0],
        view_azimuths=[0.0, 120.0], albedo=0.2, save_path=paths, gas_scattering=scenes.rayleigh_layers(levels),
        gas_absorption=scenes.ozone_layers(levels), particles=[(*scenes.henyey_greenstein_table(0.6, angles), 0.98)],
        particle_optical_depth=depth,
    ))


def _assert_alike(runs):
    (scatters, out), (other_scatters, other) = runs
    assert scatters > 0 and abs(scatters / other_scatters - 1.0) < 5e-4
    close = np.isclose(out, other, rtol=2e-4, atol=1e-7 * np.abs(other).max())
    assert np.mean(close) >= 0.999, (np.mean(close), np.abs(out - other).max())


@pytest.mark.parametrize("tail", [0, 65536])
@pytest.mark.parametrize("angles", [3, 181, 3601])
@pytest.mark.parametrize("nmat, paths", [(1, False), (3, False), (3, True)])
def test_node_tables_match_general_tables(native, device, angles, nmat, paths, tail):
    from monki.execution.native import F64P, U64P

    tables = _tables(angles, nmat, paths)
    photons = 40000
    runs = []
    for nodes in (1, 0):
        controls = (ctypes.c_uint32 * 8)(photons, 0, 1, 7, 100000, 0, photons, 1)
        err = ctypes.create_string_buffer(2048)
        handle = native.monki_cuda_create(0, tables.ctypes.data_as(F64P), tables.size, 1,
                                          f"pool=16384,tail={tail},nodes={nodes}".encode(), err, len(err))
        assert handle, err.value
        try:
            out = np.zeros(int(native.monki_cuda_tally_count(handle)))
            assert native.monki_cuda_run(handle, controls, out.ctypes.data_as(F64P), err, len(err)) == 0, err.value
            counters = np.zeros(6, dtype=np.uint64)
            native.monki_cuda_counters(handle, counters.ctypes.data_as(U64P))
        finally:
            native.monki_cuda_close(handle)
        runs.append((int(counters[0]), out))
    _assert_alike(runs)


def test_node_tables_match_general_tables_in_one_launch_sequence(native, device):
    from monki.execution.native import F64P, U64P

    batch = [_tables(181, nmat) for nmat in (1, 3)]
    photons = 40000
    pointers = (F64P * 2)(*[t.ctypes.data_as(F64P) for t in batch])
    sizes = (ctypes.c_size_t * 2)(*[t.size for t in batch])
    controls = np.array([[photons, 0, 1, 7, 100000, 0, photons, 1]] * 2, dtype=np.uint32)
    runs = []
    for nodes in (1, 0):
        err = ctypes.create_string_buffer(2048)
        handle = native.monki_cuda_multi_create(0, 2, pointers, sizes, 1, f"pool=16384,nodes={nodes}".encode(), err, len(err))
        assert handle, err.value
        try:
            outs = [np.zeros(int(native.monki_cuda_multi_tally_count(handle, q))) for q in range(2)]
            out = (F64P * 2)(*[o.ctypes.data_as(F64P) for o in outs])
            u32p = ctypes.POINTER(ctypes.c_uint32)
            assert native.monki_cuda_multi_run(handle, controls.ctypes.data_as(u32p), out, err, len(err)) == 0, err.value
            counters = np.zeros(6, dtype=np.uint64)
            native.monki_cuda_multi_counters(handle, counters.ctypes.data_as(U64P))
        finally:
            native.monki_cuda_multi_close(handle)
        runs.append((int(counters[0]), np.concatenate(outs)))
    _assert_alike(runs)
