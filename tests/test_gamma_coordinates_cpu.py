"""``update_T`` places the beam by the first cell centre of the coordinate arrays
it is given: of these arrays, as they are now, whatever it was given before."""
import gc

import numpy as np
import pytest
import torch

from jax_am_gb300.cfd import gamma

NX, NY, NZ, DX, DY = 9, 7, 4, 2e-6, 1e-6


def grid(x0, y0, torch_=False, nx=NX, ny=NY):
    x, y, _ = np.meshgrid(x0 + DX * np.arange(nx), y0 + DY * np.arange(ny), np.arange(NZ),
                          indexing="ij")
    return (torch.from_numpy(x), torch.from_numpy(y)) if torch_ else (x, y)


def first(x, y, nx=NX, ny=NY):
    return gamma._first_centre(x, y, nx, ny, DX, DY)


@pytest.mark.parametrize("torch_", [False, True], ids=["numpy", "torch"])
def test_new_arrays_of_equal_spacing(torch_):
    for k in range(30):  # each freed before the next is made: ids come back
        x, y = grid(1e-5 * k, -1e-5 * k, torch_)
        got = first(x, y)
        assert got == (float(x[0, 0, -1]), float(y[0, 0, -1])), k
        assert first(x, y) == got
        del x, y
        gc.collect()


@pytest.mark.parametrize("torch_", [False, True], ids=["numpy", "torch"])
def test_arrays_changed_in_place(torch_):
    x, y = grid(0.0, 0.0, torch_)
    assert first(x, y) == (0.0, 0.0)
    x += 3e-6
    y -= 2e-6
    assert first(x, y) == (float(x[0, 0, -1]), float(y[0, 0, -1]))
    x *= 2.0  # another spacing
    with pytest.raises(ValueError):
        first(x, y)


def test_extents_and_spacing_are_checked_each_time():
    x, y = grid(0.0, 0.0)
    first(x, y)
    with pytest.raises(ValueError):
        first(x, y, nx=NX + 1)
    with pytest.raises(ValueError):
        gamma._first_centre(x, y, NX, NY, 2 * DX, DY)
    first(x, y)
    with pytest.raises(ValueError):
        first(y, x)


def test_arrays_are_not_kept():
    import weakref
    x, y = grid(0.0, 0.0)
    first(x, y)
    w = weakref.ref(x)
    del x, y
    gc.collect()
    assert w() is None


def test_lists():
    x, y = grid(5e-6, 0.0)
    assert first(x.tolist(), y.tolist()) == (5e-6, 0.0)
    x, y = grid(7e-6, 0.0)
    assert first(x.tolist(), y.tolist()) == (7e-6, 0.0)
