"""The extrusion, window and pupil-phase kernels at the edges of their tiles,
against float64 numpy restatements."""
import numpy as np
import pytest
import torch

from dasp_gb300.infscreen import DeviceScreen, pupil_phase

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


@pytest.mark.parametrize("npup", [1, 15, 17, 63, 64, 65, 130, 301])
def test_pupil_phase_edges_and_window(npup):
    # tiles of 64 columns and 16 rows; screens whose circular starts wrap
    # inside the window; outputs that are not 16-byte aligned
    rng = np.random.default_rng(npup)
    n = npup + 6
    eye = np.hstack([np.zeros((n, n)), np.eye(n)])
    layers, total = [], np.zeros((npup, npup), np.float32)
    for q in range(3):
        init = rng.standard_normal((n, n)).astype(np.float32)
        mats = dict(ay=eye, by=np.zeros((n, n))) if q % 2 == 0 else dict(ax=eye, bx=np.zeros((n, n)))
        scr = DeviceScreen(init, 20.0, seed=q, **mats)
        (scr.add_columns if q % 2 == 0 else scr.add_rows)(2 + npup // 2, 0.1)
        now = scr.numpy()
        win = torch.empty((npup, npup), device="cuda")
        scr.window(q, 3, win)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(win.cpu().numpy(), now[q:q + npup, 3:3 + npup])
        ys, xs = np.float32(0.25 * q), np.float32(0.375)
        w = now[q:q + npup + 1, 3:3 + npup + 1]
        s = [np.float32((1.0 - float(xs)) * (1.0 - float(ys))), np.float32((1.0 - float(xs)) * float(ys)),
             np.float32(float(xs) * (1.0 - float(ys))), np.float32(xs * ys)]
        f = w[:-1, :-1] * s[0]
        f = f + w[1:, :-1] * s[1]
        f = f + w[:-1, 1:] * s[2]
        f = f + w[1:, 1:] * s[3]
        total = total + f
        layers.append((scr, q, 3, ys, xs))
    pup = (rng.random((npup, npup)) < 0.8).astype(np.float32)
    pup[0, 0] = 1.0
    store = torch.zeros(npup * npup + 1, device="cuda")
    for out in (store[:-1].view(npup, npup), store[1:].view(npup, npup)):
        for piston in (False, True):
            pupil_phase(layers, torch.from_numpy(pup).cuda(), out, remove_piston=piston, wavelength=640.0)
            torch.cuda.synchronize()
            # the float64 piston rounded to float may differ by one rounding
            p = np.float32((total.astype(np.float64) * pup).sum() / float(pup.sum(dtype=np.float64))) if piston \
                else np.float32(0)
            want = (total - p) * pup * np.float32(500.0 / 640.0)
            atol = 1.2e-7 * np.abs(total).max() if piston else 0.0
            np.testing.assert_allclose(out.cpu().numpy(), want, rtol=0, atol=atol)
    for ly in layers:
        ly[0].free()
