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


class _Array:
    """Device memory of another library: a tensor's methods, but not a torch.Tensor."""

    def __init__(self, t):
        self.t, self.shape = t, tuple(t.shape)

    def data_ptr(self):
        return self.t.data_ptr()

    def numel(self):
        return self.t.numel()

    def __getitem__(self, k):
        return _Array(self.t[k])


class _SubTensor(torch.Tensor):
    pass


@pytest.fixture
def recorded():
    """The native host side bound to functions that record what they are given; bound to the library again afterwards."""
    import vet_b200._lib as lib

    calls = []

    def fake(name, n):
        @C.CFUNCTYPE(C.c_int, *[C.c_void_p] * n)
        def f(*a):
            calls.append((name, a))
            return 0
        return f

    fakes = [fake("forward", 13), fake("backward", 20), fake("finalize", 14), fake("l1", 7), fake("zero", 4)]
    L.host().bind(*[C.cast(f, C.c_void_p).value for f in fakes])
    yield calls
    lib._bound = None
    lib.host()


def _levels(address, n):
    return [C.c_void_p.from_address(address + 8 * k).value for k in range(n)]


@pytest.mark.parametrize("kind", [lambda t: t, _Array, lambda t: t.as_subclass(_SubTensor), torch.nn.Parameter])
@pytest.mark.parametrize("b0", [0, 8])
def test_addresses_of_a_group_of_views(recorded, kind, b0):
    """Views from b0 on: images, drop-out flags and gradients start at view b0, whatever kind of tensor they come in."""
    host, views = L.host(), 11
    img = [torch.zeros(views, 4, 6 >> l, 8 >> l) for l in range(2)]
    plane = [torch.zeros(views, 1, 6 >> l, 8 >> l) for l in range(2)]
    drop = torch.zeros(views, 33)
    want = lambda ts: [t[b0:].data_ptr() for t in ts]  # noqa: E731
    frame = (1, 2, 3, 4, 5, 6, 3, b0, kind(drop), 7, 2)
    tables = {}  # the level tables live on the native stack, so they are read during the call

    @C.CFUNCTYPE(C.c_int, *[C.c_void_p] * 13)
    def forward(*a):
        tables["dropout"] = a[7]
        tables["forward"] = [_levels(p, 2) for p in a[9:13]]
        return 0

    @C.CFUNCTYPE(C.c_int, *[C.c_void_p] * 20)
    def backward(*a):
        tables["backward"] = [_levels(p, 2) for p in a[9:11]]
        tables["gradients"] = a[11:19]
        tables["dropout_backward"] = a[7]
        return 0

    names = ("vetr_finalize_gradients", "vetr_l1_loss_grad", "vetr_zero_buffers")
    host.bind(C.cast(forward, C.c_void_p).value, C.cast(backward, C.c_void_p).value,
              *[C.cast(getattr(L.lib(), n), C.c_void_p).value for n in names])
    ts = lambda x: [kind(t) for t in x]  # noqa: E731
    assert host.forward(*frame, ts(img), ts(plane), ts(plane), ts(plane)) == 0
    assert tables["dropout"] == drop[b0:].data_ptr()
    assert tables["forward"] == [want(img)] + [want(plane)] * 3
    grads = [torch.zeros(5, 4), torch.zeros(5), torch.zeros(9, 4), torch.zeros(4)]
    assert host.backward(*frame, ts(img), ts(img), *ts(grads), None, None, None, None, 3) == 0
    assert tables["backward"] == [want(img)] * 2 and tables["dropout_backward"] == drop[b0:].data_ptr()
    assert list(tables["gradients"]) == [t.data_ptr() for t in grads] + [None] * 4


@pytest.mark.parametrize("kind", [lambda t: t, _Array, lambda t: t.as_subclass(_SubTensor)])
def test_sizes_of_any_tensor(recorded, kind):
    host = L.host()
    out = host.finalize(1, torch.device("cpu"), 3, kind(torch.zeros(7, 4)), kind(torch.zeros(9, 4)), kind(torch.zeros(2, 6)),
                        kind(torch.zeros(2)), kind(torch.zeros(3, 13)), kind(torch.zeros(3)))
    assert tuple(out.shape) == (3, 7)
    name, a = recorded[-1]
    assert name == "finalize" and (a[2], a[5], a[8], a[11]) == (7, 9, 2, 3)
    image = [torch.zeros(2, 4, 3, 5)]
    assert host.l1_loss_grad(1, [kind(t) for t in image], [kind(t) for t in image], [kind(t) for t in image], kind(torch.zeros(()))) == 0
    assert recorded[-1][0] == "l1" and recorded[-1][1][1] == 1
    with pytest.raises(TypeError):
        host.l1_loss_grad(1, [np.zeros(4)], image, image, image[0])


@pytest.mark.parametrize("kind", [lambda t: t, _Array, lambda t: t.as_subclass(_SubTensor), torch.nn.Parameter])
@pytest.mark.parametrize("mode, w, h, layers, views", [(0, 40, 32, 4, 2), (1, 321, 200, 5, 8), (3, 5, 3, 2, 1), (1, 4, 4, 1, 3)])
def test_scene(kind, mode, w, h, layers, views):
    """Parameters, addresses, numbers of rows and the library's sizes in one call, whatever kind of tensor they come from."""
    params = default_params(render_mode=mode, num_layers=layers)
    position, index, texture, confidence = torch.zeros(33, 4), torch.zeros(33), torch.zeros(3, 35), torch.zeros(35)
    background, poses, intrinsics = torch.zeros(3), torch.zeros(5, 8).double(), torch.zeros(2, 13)
    tensors = (position, index, texture, confidence, background, poses, intrinsics)
    s, want = L.Scene(), L.Params()
    n, levels, pixels, capacity = L.host().scene(C.addressof(s), params, w, h, views, *[kind(t) for t in tensors])
    L.host().params(C.addressof(want), params, 3)
    assert bytes(s.params) == bytes(want) and s.params.num_channels == 3
    assert (n, levels, pixels) == (33, layers, L.lib().vetr_pyramid_pixels(w, h, layers))
    assert capacity == L.lib().vetr_list_capacity(33, views, w, h, C.byref(want))
    assert (s.cloud.position, s.cloud.index, s.cloud.n) == (position.data_ptr(), index.data_ptr(), 33)
    assert (s.texture.texture, s.texture.confidence, s.texture.background) == (texture.data_ptr(), confidence.data_ptr(), background.data_ptr())
    assert s.texture.n_tex == 35 and (s.cameras.poses_se3, s.cameras.n_img) == (poses.data_ptr(), 5)
    assert (s.cameras.intrinsics, s.cameras.n_cam) == (intrinsics.data_ptr(), 2)
    assert L.host().scene(C.addressof(s), params, 0, h, views, *tensors)[2:] == (-1, -1)
    with pytest.raises(KeyError):
        L.host().scene(C.addressof(s), {}, w, h, views, *tensors)
    with pytest.raises(TypeError):
        L.host().scene(C.addressof(s), params, w, h, views, 1.0, *tensors[1:])


def test_whole_numbers_are_cut_to_32_bits():
    params = default_params(debug_max_list_length=2**70 + 5, viewer_only=True)
    want, got = L.Params(**{k: params[k] for k, _ in L.Params._fields_}), L.Params()
    L.host().params(C.addressof(got), params, 4)
    assert got.debug_max_list_length == want.debug_max_list_length and got.viewer_only == want.viewer_only == 1


def test_native_host_side_is_built_anew_when_its_makers_change(monkeypatch, tmp_path):
    """Another torch, another interpreter, other flags, a changed source or a file of unknown origin: built again; else not.  With
    every variant of the library, and not at all where there is no torch."""
    import importlib.util
    import sys
    import sysconfig

    from vet_b200 import build as B

    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    assert L.HOST_PATH == B.HOST_PATH and B.HOST_PATH.endswith("_host" + suffix)
    target, source = tmp_path / ("_host" + suffix), tmp_path / "host.cpp"
    source.write_text("")
    commands = []

    def compiler(cmd):
        commands.append(cmd)
        if "-o" in cmd and cmd[cmd.index("-o") + 1] == str(target):
            target.write_text("built")

    monkeypatch.setattr(B.subprocess, "check_call", compiler)
    monkeypatch.setattr(B, "HOST_PATH", str(target))
    monkeypatch.setattr(B, "HOST_SOURCES", [str(source)])

    def built():
        n = len(commands)
        B.build_host()
        return len(commands) - n

    target.write_text("of unknown origin")
    assert (built(), built()) == (1, 0)
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0")
        assert (built(), built()) == (1, 0)
    assert built() == 1
    with monkeypatch.context() as m:
        m.setattr(sys, "version", "0.0")
        assert built() == 1
    with monkeypatch.context() as m:
        m.setattr(torch._C, "_GLIBCXX_USE_CXX11_ABI", not torch._C._GLIBCXX_USE_CXX11_ABI)
        assert built() == 1
    assert (built(), built()) == (1, 0)
    os.utime(source, (os.path.getmtime(target) + 10,) * 2)
    assert built() == 1
    # a variant of the library comes with it
    target.unlink()
    commands.clear()
    B.build(out=str(tmp_path / "variant.so"))
    assert len(commands) == 2 and target.exists()
    find = importlib.util.find_spec
    target.unlink()
    monkeypatch.setattr(importlib.util, "find_spec", lambda name, *a: None if name == "torch" else find(name, *a))
    B.build(out=str(tmp_path / "variant.so"))
    assert not target.exists()
