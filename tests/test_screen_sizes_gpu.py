"""The extrusion kernel at the edges of their tiles,
against a float64 numpy restatement."""
import numpy as np
import pytest
import torch

from dasp_gb300.infscreen import DeviceScreen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [3, 33, 63, 64, 65, 153, 305, 768, 769, 1217])
@pytest.mark.parametrize("axis", [0, 1, 2, 3])
def test_extruded_lines_match_numpy(length, axis):
    # one row per CTA up to the SM count, more beyond; chunks of 768 elements;
    # lengths around the 64 threads of an element
    rng = np.random.default_rng(length * 4 + axis)
    a = rng.standard_normal((length, 2 * length)) / length
    b = rng.standard_normal((length, length)) / length
    other = 5
    cols = axis in (0, 2)
    shape = (length, other) if cols else (other, length)
    init = rng.standard_normal(shape).astype(np.float32)
    mats = dict(ay=a, by=b) if cols else dict(ax=a, bx=b)
    scr = DeviceScreen(init, 20.0, seed=3, **mats)
    add = (scr.add_columns, scr.add_rows, scr.add_columns_start, scr.add_rows_start)[axis]
    want = init.astype(np.float64) if cols else init.T.astype(np.float64)
    coeff = (20.0 / 0.1) ** (5.0 / 6)
    for step in (0.5, 0.0):
        n = rng.standard_normal((3, length))
        add(3, 0.1, step=step, noise=n)
        for k in range(3):
            z = np.concatenate([want[:, 1], want[:, 0]] if axis >= 2 else [want[:, -2], want[:, -1]])
            new = (a @ z + (b @ n[k]) * coeff + (step if k == 0 else 0.0)).astype(np.float32).astype(np.float64)
            want = np.column_stack([new, want[:, :-1]] if axis >= 2 else [want[:, 1:], new])
    got = scr.numpy()
    # one float rounding per line (of inputs that may differ by one each)
    np.testing.assert_allclose(got if cols else got.T, want, rtol=0, atol=4e-7 * np.abs(want).max())
    # the device's own normals: the same lines whether queued one call or several
    scr.free()
    one, many = DeviceScreen(init, 20.0, seed=9, **mats), DeviceScreen(init, 20.0, seed=9, **mats)
    stream = torch.cuda.Stream()
    kinds = ("add_columns", "add_rows", "add_columns_start", "add_rows_start")
    getattr(one, kinds[axis])(7, 0.1, stream=stream)
    for _ in range(7):
        getattr(many, kinds[axis])(1, 0.1)
    stream.synchronize()
    np.testing.assert_array_equal(one.numpy(), many.numpy())
    assert np.isfinite(one.numpy()).all()
    one.free()
    many.free()
