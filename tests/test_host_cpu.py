"""The native host side of render.py: parameter blocks, views and output tensors as ctypes and torch make them (no GPU)."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

from vet_b200 import _lib as L
from vet_b200.render import default_params, level_sizes
from vet_b200.scenes import View

pytestmark = pytest.mark.skipif(not (os.path.exists(L.HOST_PATH) and os.path.exists(L.LIB_PATH)), reason="libraries not built")


def test_parameter_block():
    params = default_params(render_mode=3, num_layers=5, num_channels=3, drop_out_radius_threshold=0.25, ghost_gradients=True,
                            depth_accept=np.float32(0.5), viewer_only=np.int64(1))
    want, got = L.Params(**{k: params[k] for k, _ in L.Params._fields_ if k != "num_channels"}), L.Params()
    want.num_channels = 4
    L.host().params(C.addressof(got), params, 4)
    for k, _ in L.Params._fields_:
        assert getattr(got, k) == getattr(want, k), k
    for k, _ in L.Params._fields_:
        with pytest.raises(KeyError):
            L.host().params(C.addressof(got), {n: v for n, v in params.items() if n != k}, 4)
    with pytest.raises(TypeError):
        L.host().params(C.addressof(got), dict(params, num_layers=4.0), 4)


def test_views():
    views = [View(96, 64, image_index=1, camera_index=2), View(33, 17, crop=(2, 3, 4, 5, 6), rot=(0.5, 1, 2, 3))]
    arr = (L.View * 2)()
    L.host().views(C.addressof(arr), views)
    for a, v in zip(arr, views):
        assert (a.w, a.h, a.image_index, a.camera_index, a.camera_model) == (v.w, v.h, v.image_index, v.camera_index, v.camera_model)
        assert list(a.crop) == [float(x) for x in v.crop] and list(a.rot) == [float(x) for x in v.rot]
    with pytest.raises(ValueError):
        L.host().views(C.addressof(arr), [View(8, 8, crop=(1,) * 6)])


@pytest.mark.parametrize("w, h", [(96, 64), (801, 603), (17, 16)])
def test_images(w, h):
    color, weight, mask, depth = L.host().images(torch.device("cpu"), 3, 4, w, h, 5, True, False, 1)
    sizes = level_sizes(w, h, 5)
    assert [tuple(t.shape) for t in color] == [(3, 4, b, a) for a, b in sizes]
    assert [tuple(t.shape) for t in weight] == [tuple(t.shape) for t in depth] == [(3, 1, b, a) for a, b in sizes]
    assert mask is None and all(t.dtype == torch.float32 and t.is_contiguous() for t in color + weight + depth)


def test_wrong_arguments_raise():
    t = torch.zeros(4)
    with pytest.raises(TypeError):
        L.host().images("cpu", 1, 4, 8, 8, 1, True, False, False)
    with pytest.raises(ValueError):
        L.host().images(torch.device("cpu"))
    with pytest.raises(TypeError):
        L.host().l1_loss_grad(8, [1.0], [t], [t], t)
    with pytest.raises(ValueError):
        L.host().l1_loss_grad(8, [t, t], [t], [t, t], t)  # a target too few
    assert L.host().l1_loss_grad(8, [t] * 6, [t] * 6, [t] * 6, t) == L.E_INVALID_ARG


def test_crop_and_rotation_with_too_many_entries():
    """The rasterizer answers as an array does that is given too many initialisers; fewer leave the rest at zero."""
    from vet_b200.render import Rasterizer

    for bad in (View(8, 8, crop=(1.0,) * 6), View(8, 8, rot=(1.0,) * 5)):
        with pytest.raises(IndexError):
            Rasterizer._views(None, [bad])
    arr = Rasterizer._views(None, [View(8, 8, crop=(1, 2, 3), rot=())])
    assert list(arr[0].crop) == [1, 2, 3, 0, 0] and list(arr[0].rot) == [0, 0, 0, 0]
