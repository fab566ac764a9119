"""The node tables of plain particle species (F22 = F33 = F11, F12 = 0) against the general
tables: the same histories and the same tallies.

A species is general when its F12 differs from zero anywhere, so the same particle with F12 of
1e-300 at one angle takes the general tables with the same physics. FP64 runs of both must
agree in every event; I and I/Q/U, and table sizes down to three angles (sampling and phase
function at the first and last brackets).
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(angles, nmat, plain):
    import monki.scenes as scenes

    levels = np.array([0.0, 1.0, 2.0, 4.0, 10.0, 60.0])
    nx, ny = 5, 4
    cosines, cdf, f11, f22, f33, f12 = scenes.henyey_greenstein_table(0.6, angles)
    if not plain:
        f12 = f12.copy()
        f12[angles // 2] = 1e-300
    depth = np.zeros((1, nx, ny, len(levels) - 1))
    depth[0, 1:4, 1:3, 1] = 3.0
    return scenes.build_tables(
        nx=nx, ny=ny, levels_km=levels, nmat=nmat, solar_zenith=30.0, solar_azimuth=0.0, view_zeniths=[0.0, 40.0],
        view_azimuths=[0.0, 120.0], albedo=0.2, save_path=False, gas_scattering=scenes.rayleigh_layers(levels),
        gas_absorption=scenes.ozone_layers(levels), particles=[(cosines, cdf, f11, f22, f33, f12, 0.98)],
        particle_optical_depth=depth,
    )


@pytest.mark.parametrize("angles", [3, 181, 3601])
@pytest.mark.parametrize("nmat", [1, 3])
def test_plain_species_tables_match_general_tables(native, device, angles, nmat):
    from monki.execution.native import F64P, U64P

    results = []
    for plain in (True, False):
        tables = np.ascontiguousarray(_tables(angles, nmat, plain))
        controls = (ctypes.c_uint32 * 8)(400, 0, 1, 7, 100000, 0, 400, 1)
        err = ctypes.create_string_buffer(2048)
        handle = native.monki_cuda_create(0, tables.ctypes.data_as(F64P), tables.size, 1, b"precision=fp64", err, len(err))
        assert handle, err.value
        try:
            out = np.zeros(int(native.monki_cuda_tally_count(handle)))
            assert native.monki_cuda_run(handle, controls, out.ctypes.data_as(F64P), err, len(err)) == 0, err.value
            counters = np.zeros(6, dtype=np.uint64)
            native.monki_cuda_counters(handle, counters.ctypes.data_as(U64P))
        finally:
            native.monki_cuda_close(handle)
        results.append((int(counters[0]), out))
    assert results[0][0] == results[1][0]
    np.testing.assert_allclose(results[0][1], results[1][1], rtol=1e-9, atol=1e-14)
