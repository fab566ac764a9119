"""The weight-gradient kernel (tcgen05, split-K, operands contracted over their rows) at the
edges of its slices and tiles.

* alone, against float64 products of the same BF16 values: fewer rows than a tile, one more and
  one less than a slice, several slices with a short last one; the device rows past the valid
  ones hold NaN. Tolerance: FP32 accumulation of n products of unit normals has an error of about
  sqrt(n) 2^-24 of the largest sum, and the slices' sums are added in any order: 1e-4 of the
  largest entry, as for the plain GEMM;
* in the network, every parameter's gradient against the CPU restatement for calls of many sizes
  on one network, smaller after larger and larger than any before. The hidden values round to
  BF16 on both sides, and a value near a rounding boundary may round the other way in each of
  three layers, 3 x 2^-8; the output's error enters relative to the rows' residuals. The same
  call on a fresh network differs only in the order of FP32 sums.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 256])
@pytest.mark.parametrize("rows, chunk", [(1, 1024), (63, 1024), (64, 1024), (65, 1024), (1023, 1024), (1024, 1024),
                                         (1025, 1024), (2500, 1024), (200, 64), (331, 192)])
def test_row_contraction_matches_float64_products(native, device, rows, chunk, n):
    from monki.execution.native import F32P
    from oracle import mlp

    m = 256
    rng = np.random.default_rng(rows + n)
    a, b = mlp.bf16(rng.normal(size=(rows, m))), mlp.bf16(rng.normal(size=(rows, n)))
    bits = [np.ascontiguousarray(v.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16) for v in (a, b)]
    u16 = ctypes.POINTER(ctypes.c_uint16)
    c = np.zeros((m, n), dtype=np.float32)
    err = ctypes.create_string_buffer(1024)
    status = native.monki_mlp_rows_probe(0, *(v.ctypes.data_as(u16) for v in bits), rows, m, n, chunk,
                                         c.ctypes.data_as(F32P), err, len(err))
    assert status == 0, err.value
    expected = a.T @ b
    np.testing.assert_allclose(c, expected, rtol=1e-4, atol=1e-4 * np.abs(expected).max())


def test_gradients_of_many_sizes_on_one_network_match_the_oracle(device):
    from monki.importance import ImportanceModel
    from oracle import mlp

    with ImportanceModel(rows=2560, seed=3) as model:
        params = model.params
        for rows in (65, 2500, 1, 63, 1025, 2500, 64, 2560):
            rng = np.random.default_rng(rows)
            x = rng.normal(size=(rows, 48)).astype(np.float32)
            t = (np.sin(x[:, 0]) + 0.5 * x[:, 1] ** 2 - x[:, 2] * x[:, 3]).astype(np.float32)
            w = rng.uniform(0.5, 1.5, size=rows).astype(np.float32)
            loss, grads = model.gradients(x, t, w)
            y = model.predict(x)
            y_ref, _ = mlp.forward(params, x)
            np.testing.assert_allclose(y, y_ref, rtol=2e-2, atol=2e-2 * np.abs(y_ref).max())
            loss_ref, grads_ref = mlp.gradients(params, x, t, w)
            residual = 2e-2 * np.abs(y_ref).max() / np.sqrt(np.mean((y_ref - t) ** 2))
            assert loss == pytest.approx(loss_ref, rel=1e-2 + 2 * residual)
            at = 0
            for name, shape in mlp.SHAPES:
                size = int(np.prod(shape))
                g, r = grads[at : at + size].astype(np.float64), grads_ref[at : at + size]
                at += size
                assert np.linalg.norm(g - r) < (2e-2 + residual) * np.linalg.norm(r), (rows, name)
            with ImportanceModel(rows=2560, params=params) as fresh:
                fresh_loss, fresh_grads = fresh.gradients(x, t, w)
            assert loss == pytest.approx(fresh_loss, rel=1e-5)
            assert np.linalg.norm(grads - fresh_grads) < 1e-5 * np.linalg.norm(fresh_grads)
