"""The histories of the one-thread-per-history kernel in FP32 (``engine=megakernel``, the kernel
of the allocation-free call too): the scatter counts of fixed seeds.

A seed's run is one set of histories. What other kernels read (the wavefront's node tables of
plain species among it) must not change how this kernel rounds: histories that round differently
part ways, and the tallies of a fixed seed move by 1e-3. The counts were taken on one GB300.
Tolerance: the scene's tables are made with numpy, whose last bits may differ between versions;
an FP32 table entry that rounds the other way moves a history with a probability of about 1e-7
per scatter, 0.1 of the 120,000 histories here or 1e-6 of the count, so 3e-5 leaves room for
thirty of them. Reading the node tables moved these counts by 6e-5 to 4e-4.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(nmat, polarizing, paths):
    import monki.scenes as scenes
    from test_backward import polarizing_particle

    levels, nx, ny = scenes.layer_levels_km(), 30, 20
    profile = scenes.layer_fraction(levels, 1.0, 2.0) * np.diff(levels)
    cloud = np.zeros((nx, ny, len(levels) - 1))
    cloud[10:20, 6:13] = 8.0 * profile / profile.sum()
    return np.ascontiguousarray(scenes.build_tables(
        nx=nx, ny=ny, levels_km=levels, nmat=nmat, solar_zenith=40.0, solar_azimuth=0.0,
        view_zeniths=[0.0, 30.0, 60.0], view_azimuths=[0.0, 90.0, 180.0], albedo=0.1, save_path=paths,
        gas_scattering=scenes.rayleigh_layers(levels), gas_absorption=scenes.ozone_layers(levels),
        particles=[scenes.AEROSOL, polarizing_particle(3601) if polarizing else scenes.CLOUD],
        particle_optical_depth=np.stack([scenes.aerosol_depth(levels, nx, ny), cloud]),
    ))


@pytest.mark.parametrize("paths", [False, True])
@pytest.mark.parametrize("nmat, polarizing, scatters", [
    (1, False, 1196044), (1, True, 1194929), (3, False, 1192792), (3, True, 1189524),
])
def test_fixed_seed_keeps_its_histories(native, device, nmat, polarizing, scatters, paths):
    from monki.execution.native import F64P, U64P

    tables = _tables(nmat, polarizing, paths)
    per_round = 200 * 600
    err = ctypes.create_string_buffer(2048)
    handle = native.monki_cuda_create(0, tables.ctypes.data_as(F64P), tables.size, 1,
                                      b"precision=fp32,engine=megakernel,shards=1", err, len(err))
    assert handle, err.value
    try:
        out = np.zeros(int(native.monki_cuda_tally_count(handle)))
        controls = (ctypes.c_uint32 * 8)(per_round, 0, 1, 5, 100000, 0, per_round, 1)
        assert native.monki_cuda_run(handle, controls, out.ctypes.data_as(F64P), err, len(err)) == 0, err.value
        counters = np.zeros(6, dtype=np.uint64)
        native.monki_cuda_counters(handle, counters.ctypes.data_as(U64P))
    finally:
        native.monki_cuda_close(handle)
    assert abs(int(counters[0]) / scatters - 1.0) < 3e-5, (int(counters[0]), scatters)
