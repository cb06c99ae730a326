"""Sizes at which a kernel takes another path than in the other parity tests: ends of tiles, remainders, the cells of the
error grid that leave the row form.  Against the CPU oracle, with the bounds of the tests of the same function."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import util
from vet_b200 import scenes
from vet_b200.render import default_params, level_sizes, scene_to_device

pytestmark = pytest.mark.gpu


# ---- error grid: rows of cells, rows and cells that go through the per-pixel test


def _grid(cells, box):
    a = np.arange(cells, dtype=np.float32) * np.float32(2 * box / cells) - np.float32(box)
    m = np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
    return np.ascontiguousarray(m), np.full_like(m, np.float32(2 * box / cells))


@pytest.mark.parametrize("case", ["inside", "aligned", "distorted", "non_finite", "flat_boxes", "one_cell"])
def test_grid_loss_paths(rasterizer, case):
    """Coverage is exact whatever path a cell takes; values are sums of non-negative fp32 terms (1e-5)."""
    import torch

    w, h = 333, 251
    sc = scenes.config_planar(64, w, h, 200.0, n_views=1, seed=3)
    bb_min, bb_len = _grid(21, 10.0)  # the camera stands inside the grid: cells of a few pixels and of the whole image
    rng = np.random.default_rng(1)
    loss = rng.standard_normal((3, h, w)).astype(np.float32)
    if case == "aligned":  # edges on pixel rows and columns, faces seen edge-on
        sc.poses = np.array([[0, 0, 0, 1, 0, 0, 0, 0]], np.float64)
        bb_min, bb_len = _grid(16, 8.0)
    elif case == "distorted":
        sc.intrinsics[0, 5:] = (0.05, -0.02, 0.001, 0.01, 0.0, 0.0, 0.001, -0.002)
    elif case == "non_finite":
        loss[0, 100, 60], loss[1, 120, 200] = np.inf, np.nan
    elif case == "flat_boxes":
        bb_len = bb_len * rng.choice(np.array([0.0, 1e-4, 1.0], np.float32), size=bb_len.shape)
    elif case == "one_cell":
        bb_min, bb_len = np.array([[-1.0, -1.0, -1.0]], np.float32), np.array([[2.0, 2.0, 2.0]], np.float32)
    n = bb_min.shape[0]
    ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(n, device=rasterizer.device), torch.zeros(n, dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)
    assert ref_c.sum() > 0
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
    np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0, equal_nan=True)


@pytest.mark.parametrize("offset", [2e5, 1e6])
def test_grid_loss_far_from_the_origin(rasterizer, offset):
    """A scene far from the origin: the corners of a box are rounded to the grid of the world coordinates (1/64 of a unit at 2e5,
    where a cell is 0.4 units wide), so its faces bend and their diagonals stick out of the edges' outline; at 1e6 the projected box
    is no longer in one piece row by row.  Coverage stays exact."""
    import torch

    w, h, cells = 640, 360, 48
    sc = scenes.config_planar(64, w, h, 800.0, n_views=2, seed=5)
    bb_min, bb_len = _grid(cells, 10.0)
    shift = np.array([1.0, 0.7, -0.4]) * offset
    bb_min = (bb_min + shift).astype(np.float32)
    for pose in sc.poses:  # x -> R x + t seen from the shifted scene: t - R shift
        q, v = pose[:3], shift
        uv = 2 * np.cross(q, v)
        pose[4:7] -= v + pose[3] * uv + np.cross(q, uv)
    loss = np.random.default_rng(1).random((1, h, w)).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    for view in sc.views:
        ref_v, ref_c = O.grid_loss(sc, view, bb_min, bb_len, loss)
        value, count = torch.zeros(len(bb_min), device=rasterizer.device), torch.zeros(len(bb_min), dtype=torch.int32, device=rasterizer.device)
        rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), view, t(bb_min), t(bb_len), t(loss), value, count)
        assert (ref_c > 0).sum() > 1000
        np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
        np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


def test_grid_loss_wide_range(rasterizer):
    """Rows with one pixel of 1e12 among losses of 1e-3, and a block of zeros: what a cell covers beside that pixel keeps its
    relative accuracy (sums of non-negative fp32 terms, 1e-5), and a cell over zeros only stays exactly zero."""
    import torch

    w, h = 640, 360
    sc = scenes.config_planar(64, w, h, 800.0, n_views=1, seed=5)
    bb_min, bb_len = _grid(40, 10.0)
    rng = np.random.default_rng(2)
    loss = (1e-3 * rng.standard_normal((2, h, w))).astype(np.float32)
    loss[:, 100:200, 300:420] = 0
    loss[0, ::3, 40] = 1e12
    loss[1, 1::3, 290] = 1e12
    ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    assert ((ref_c > 0) & (ref_v == 0)).sum() > 50 and (ref_v > 1e11).sum() > 50
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(len(bb_min), device=rasterizer.device), torch.zeros(len(bb_min), dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
    np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


def test_grid_loss_recorded(rasterizer):
    """Recorded calls: a graph stays good when a larger image has come since, and an image larger than any before can be
    recorded (without room for its running sums the cells are walked pixel by pixel)."""
    import torch

    from vet_b200.render import Rasterizer

    rast = Rasterizer(0)
    bb_min, bb_len = _grid(21, 10.0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rast.device)  # noqa: E731

    def call(w, h, seed):
        sc = scenes.config_planar(64, w, h, 0.6 * w, n_views=1, seed=3)
        loss = np.random.default_rng(seed).random((3, h, w)).astype(np.float32)
        value, count = torch.zeros(len(bb_min), device=rast.device), torch.zeros(len(bb_min), dtype=torch.int32, device=rast.device)
        args = (t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)

        def check():
            torch.cuda.synchronize()
            ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
            np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
            np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)
            value.zero_(), count.zero_()

        return lambda: rast.grid_loss(*args), check

    run, check = call(160, 120, 1)
    run(), check()
    graphs = []
    for size, seed in (((160, 120), 2), ((400, 300), 3)):
        run, check = call(*size, seed)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run()
        graphs.append((graph, check, run))  # (run holds the graph's tensors)
    run, check = call(640, 480, 4)
    run(), check()
    for graph, check, _ in graphs:
        graph.replay(), check()
    rast.close()


# ---- lists of more than 256 fragments: their sort (runs of 32, merges, up to 2048 in shared memory), their fold (blocks of
# 1024), their sweeps (blocks of 768; mode 2: up to 1024, up to 4096)


@pytest.mark.parametrize("mode, opacity", [(1, 0.005), (3, 0.005), (3, 0.1), (2, 0.005)])
def test_long_list_lengths(rasterizer, mode, opacity):
    _check_lists(rasterizer, mode, opacity, (1, 255, 256, 257, 319, 511, 513, 767, 768, 769, 1023, 1024, 1025, 1537, 2047, 2048, 2049))


@pytest.mark.parametrize("mode", [1, 3])
def test_long_list_runs(rasterizer, mode):
    """Lists of several runs of 2048 fragments, the last run of one fragment, of almost all and in between."""
    _check_lists(rasterizer, mode, 0.002, (4095, 4096, 4097, 6144, 7000, 8191, 8193, 10241))


def _check_lists(rasterizer, mode, opacity, lengths):
    w, h, f = 64, 48, 50.0
    n = sum(lengths)
    sc = scenes.tiny_scene(n=n, w=w, h=h, n_views=1, seed=9)
    rng = np.random.default_rng(4)
    sc.poses = np.array([[0, 0, 0, 1, 0, 0, 0, 0]], np.float64)
    sc.intrinsics[0] = 0
    sc.intrinsics[0, :4] = f, f, w / 2, h / 2
    pixel = np.repeat(np.arange(len(lengths)), lengths)  # a list each, in columns of 16 x 2 pixels; mode 3: 2 x 2 lists
    u, v = 4 + 3 * (pixel % 16) + 0.2, 10 + 20 * (pixel // 16) + 0.3
    z = rng.integers(512, 1536, n).astype(np.float32) / 256  # with points at equal depth: the point index decides
    sc.position[:, 0], sc.position[:, 1], sc.position[:, 2] = (u - w / 2) / f * z, (v - h / 2) / f * z, z
    sc.position[:] = sc.position[rng.permutation(n)]
    sc.confidence[:] = (opacity * rng.random(sc.confidence.shape)).astype(np.float32)
    params = default_params(render_mode=mode, drop_out_points_by_radius=0, num_layers=1)
    ora = util.run_oracle(sc, params)
    grads = util.random_grads(ora["fwd"]["color"], seed=3)
    ora = util.run_oracle(sc, params, grads=grads)
    gpu = util.run_gpu(rasterizer, sc, params, grads=grads)
    assert gpu["longest"] == max(lengths)
    util.compare_forward(gpu, ora, exact_images=True)
    util.compare_backward(gpu["bwd_raw"], ora, sc.channels)


# ---- environment map: the backward kernel is compiled for up to four and for up to eight spheres


@pytest.mark.parametrize("spheres", [2, 5, 8])
def test_envmap_sphere_counts(rasterizer, spheres):
    levels = 2
    sc = util.env_scene(n_views=2, w=96, h=64, f=80.0)
    rng = np.random.default_rng(spheres)
    env = util.env_map(rng, S=spheres, R=32)
    weight = util.env_weights(rng, sc, levels)
    ref = O.envmap_forward(sc, sc.views, levels, env, weight)
    gout = [rng.standard_normal(r.shape).astype(np.float32) for r in ref]
    ref_d, ref_c, mag_d, mag_c = O.envmap_backward(sc, sc.views, levels, env, weight, gout)
    out, g_density, g_color = util.env_gpu_run(sc, env, levels, weight, 0, gout)
    tol = util.env_sample_tolerance(env)
    assert all(np.abs(o - r).max() <= tol for o, r in zip(out, ref))
    assert np.all(np.abs(g_density - ref_d) <= util.env_grad_tolerance(mag_d, env))
    assert np.all(np.abs(g_color - ref_c) <= util.env_grad_tolerance(mag_c, env))


# ---- zero fill of several buffers: partial last units, empty buffers, starts off a 16-byte boundary


def test_zero_buffers(rasterizer):
    import ctypes as C

    import torch

    from vet_b200 import _lib as L

    sizes = [0, 1, 3, 4, 5, 4096, 4097, 100_003, 2, 7]
    for shift in (0, 1):
        whole = [torch.ones(n + 2, device=rasterizer.device) for n in sizes]
        part = [t[shift:shift + n] for t, n in zip(whole, sizes)]
        ptrs = (C.c_void_p * len(sizes))(*[t.data_ptr() for t in part])
        nbytes = (C.c_int64 * len(sizes))(*[4 * n for n in sizes])
        rasterizer._sync_stream()
        assert L.lib().vetr_zero_buffers(rasterizer._ctx, ptrs, nbytes, len(sizes)) == L.OK
        for t, n in zip(whole, sizes):
            want = torch.ones_like(t)
            want[shift:shift + n] = 0
            assert torch.equal(t, want)
    assert L.lib().vetr_zero_buffers(rasterizer._ctx, ptrs, (C.c_int64 * 1)(6), 1) == L.E_INVALID_ARG
    assert L.lib().vetr_zero_buffers(rasterizer._ctx, None, None, 17) == L.E_INVALID_ARG


# ---- camera gradients: the image-space gradients of a point's fragments are summed in fp64


def test_pose_gradient_of_cancelling_fragments(rasterizer):
    """One point of mode 3 between four pixels, every product a power of two: the corners' gradients along x are 2^24, 1,
    -2^24 and 0.  Their sum is 1; a sum in fp32 gives 0."""
    import torch

    dev = rasterizer.device
    w = h = 16
    f32 = dict(dtype=torch.float32, device=dev)
    position = torch.tensor([[(6.5 - 8) / 64 * 2, (7.5 - 8) / 64 * 2, 2.0, 0.01]], **f32)
    index = torch.zeros(1, dtype=torch.int32, device=dev)
    texture, confidence, background = torch.tensor([[1.0], [0], [0], [0]], **f32), torch.ones(1, 1, **f32), torch.zeros(4, **f32)
    poses = torch.tensor([[0, 0, 0, 1, 0, 0, 0, 0]], dtype=torch.float64, device=dev)
    intrinsics = torch.tensor([[64.0, 64, 8, 8] + [0] * 9], **f32)
    params = default_params(render_mode=3, num_layers=1, drop_out_points_by_radius=0)
    rasterizer.forward(position, index, texture, confidence, background, poses, intrinsics, [scenes.View(w, h)], params)
    grad = torch.zeros(1, 4, h, w, **f32)
    grad[0, 0, 7, 6], grad[0, 0, 7, 7], grad[0, 0, 8, 6] = -2.0 ** 25, 2.0, 2.0 ** 25
    raw = rasterizer.backward_raw([grad])
    assert raw["points"][0, 3].item() == 4
    assert raw["pose"][0, 0].item() == 32.0  # f / z
    assert raw["intrinsics"][0, 2].item() == 0.5  # K_gradient_factor


# ---- mode 0: backward with the interleaved image copies, and without pixel scratch


@pytest.mark.parametrize("channels, ghost", [(4, 0), (3, 0), (4, 1)])
def test_mode0_backward_scratch(monkeypatch, channels, ghost):
    from vet_b200 import render

    sc = scenes.tiny_scene(n=9000, w=93, h=61, n_views=2, seed=13, channels=channels, crop=True)  # 7475 pixels a view
    dropout = (np.random.default_rng(2).random((2, sc.n)) < 0.2).astype(np.float32)
    params = default_params(render_mode=0, num_channels=channels, ghost_gradients=ghost)
    ora = util.run_oracle(sc, params, dropout=dropout)
    grads = util.random_grads(ora["fwd"]["color"], seed=3)
    ora = util.run_oracle(sc, params, grads=grads, dropout=dropout)
    for scratch in (True, False):
        if not scratch:
            monkeypatch.setattr(render.FragmentLists, "ensure_pixel_scratch", lambda self: None)
        rast = render.Rasterizer(0)
        gpu = util.run_gpu(rast, sc, params, grads=grads, dropout=dropout)
        # the forward image differs from the oracle's in the last bits (descriptors are summed in no fixed order), and an
        # addend (T - I) * G inherits that relative to |I * G|: the bound of the mode-0 parity tests
        util.compare_backward(gpu["bwd_raw"], ora, channels, rtol=2e-5, floor_rel=1e-6)
        rast.close()


def test_mode0_leaves_the_scratch_of_other_modes_alone(rasterizer):
    """vetr_backward in mode 0 does not touch lists->pixel_scratch, which it has no use for: a caller may keep a buffer of any
    size there."""
    import ctypes as C

    import torch

    from vet_b200 import _lib as L

    sc = scenes.tiny_scene(n=9000, w=93, h=61, n_views=2, seed=13)
    params = default_params(render_mode=0)
    grads = [torch.from_numpy(g).to(rasterizer.device) for g in
             util.random_grads(util.run_gpu(rasterizer, sc, params)["fwd"]["color"], seed=3)]
    want = rasterizer.backward_raw(grads)
    s = rasterizer._saved
    b0, b1, lists, views = s["groups"][0]
    lists.ensure_pixel_scratch()
    lists.pixel_scratch.fill_(7.0)
    got = {k: torch.zeros_like(v) for k, v in want.items()}
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    arr = lambda ts: (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])  # noqa: E731
    rc = L.lib().vetr_backward(rasterizer._ctx, C.byref(s["prm"]), C.byref(s["cloud"]), C.byref(s["tex"]), C.byref(s["cams"]),
                               views, b1 - b0, None, C.byref(lists.c), arr(s["color"]), arr(grads), p(got["desc"]),
                               p(got["conf"]), p(got["points"]), p(got["background"]), p(got["pose"]), p(got["pose_count"]),
                               p(got["intrinsics"]), p(got["intrinsics_count"]))
    assert rc == L.OK
    assert bool((lists.pixel_scratch == 7.0).all())
    assert torch.equal(got["points"][:, 3], want["points"][:, 3])
    for k in want:  # the same addends (sums in no fixed order)
        assert torch.allclose(got[k], want[k], rtol=1e-4, atol=1e-5 * float(want[k].abs().max())), k
    # the word for it goes with the per-fragment phase; other bits are refused as before
    for phases in (0, 4, 6, 8, 11):
        assert L.lib().vetr_backward_phase(rasterizer._ctx, C.byref(s["prm"]), C.byref(s["cloud"]), C.byref(s["tex"]),
                                           C.byref(s["cams"]), views, b1 - b0, None, C.byref(lists.c), arr(s["color"]),
                                           arr(grads), p(got["desc"]), p(got["conf"]), None, p(got["background"]), None, None,
                                           None, None, phases) == L.E_INVALID_ARG


# ---- per-point pass: several runs of 256 points per block (2 and the most, 8), several views, a partial last run


@pytest.mark.parametrize("mode", [1, 3])
@pytest.mark.parametrize("tiles, w, h, views", [(2, 320, 240, 3), (8, 640, 480, 2)])
def test_point_backward_tiles(rasterizer, mode, tiles, w, h, views):
    import torch

    per_tile = 256 * 4 * torch.cuda.get_device_properties(rasterizer.device).multi_processor_count
    n = tiles * per_tile + 257  # the rule: as many runs per block as leave four blocks per SM
    sc = scenes.config_planar(n, w, h, 0.9 * w, n_views=views, seed=17)
    rng = np.random.default_rng(6)  # gradients without cancellation inside a term: thin fragments of one sign, no background
    sc.texture[:], sc.background[:] = 0, 0
    sc.texture[0] = rng.uniform(1, 2, n)
    sc.confidence *= np.float32(0.002)
    params = default_params(render_mode=mode, num_layers=2)
    ora = util.run_oracle(sc, params)
    grads = util.l1_grads(ora["fwd"]["color"], seed=3)
    ora = util.run_oracle(sc, params, grads=grads)
    gpu = util.run_gpu(rasterizer, sc, params, grads=grads)
    util.compare_forward(gpu, ora, exact_images=True)
    util.compare_backward(gpu["bwd_raw"], ora, sc.channels)
    on = [torch.from_numpy(g).to(rasterizer.device) for g in grads]
    for want_pose in (True, False):  # the kernel without intrinsics, with and without a pose
        part = rasterizer.backward_raw(on, want_pose=want_pose, want_intrinsics=False)
        np.testing.assert_array_equal(part["points"].cpu().numpy(), gpu["bwd_raw"]["points"])  # one owner per point, fixed order
    pose = rasterizer.backward_raw(on, want_intrinsics=False)["pose"].cpu().numpy()
    np.testing.assert_allclose(pose, gpu["bwd_raw"]["pose"], rtol=1e-6, atol=1e-9 * np.abs(pose).max())


# ---- mode 2: groups of one, of a few, of the whole list, with the background (beyond a window of 1e5 every depth is in)


@pytest.mark.parametrize("accept", [1e-6, 0.003, 0.5, 9e4, 3e5])  # (0: an empty first group, 0 / 0 as in the reference)
@pytest.mark.parametrize("n, w, h", [(6000, 96, 64), (30000, 16, 12)])
def test_mode2_group_sizes(rasterizer, accept, n, w, h):
    sc = scenes.tiny_scene(n=n, w=w, h=h, n_views=1, seed=17)
    for env in (0, 1):
        params = default_params(render_mode=2, drop_out_points_by_radius=0, num_layers=3, depth_accept_blend=accept, use_environment_map=env)
        g = util.l1_grads(util.run_oracle(sc, params)["fwd"]["color"], seed=3)
        ora = util.run_oracle(sc, params, grads=g)
        gpu = util.run_gpu(rasterizer, sc, params, grads=g)
        util.compare_forward(gpu, ora, exact_images=True)
        util.compare_backward(gpu["bwd_raw"], ora, sc.channels)


# ---- error grid: groups of cells that are left out before their corners are projected


@pytest.mark.parametrize("crop", [False, True])
def test_grid_loss_cells_around_the_edges_of_the_view(rasterizer, crop):
    """Boxes of all sizes around the camera and the border of the image, in groups of four that lie across it or just beside it:
    none that covers a pixel may be left out (coverage is exact).  A number of cells that fills no group."""
    import torch

    w, h = 321, 243
    sc = scenes.config_planar(64, w, h, 200.0, n_views=1, seed=3)
    if crop:
        sc.views[0].crop = (1.3, 0.8, 12.0, -9.0, 0.05)
        sc.views[0].rot = (0.8, -0.6, 0.6, 0.8)
    rng = np.random.default_rng(2)
    n = 20_003
    centre = np.repeat(rng.uniform(-12, 12, size=(n // 4 + 1, 3)), 4, axis=0)[:n]  # neighbours close to each other, as in a grid
    size = np.repeat(10.0 ** rng.uniform(-2.5, 0.5, size=(n // 4 + 1, 1)), 4, axis=0)[:n]
    bb_min = (centre + size * rng.uniform(-1, 1, size=(n, 3))).astype(np.float32)
    bb_len = np.broadcast_to(size, (n, 3)).astype(np.float32).copy()
    loss = rng.standard_normal((3, h, w)).astype(np.float32)
    ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(n, device=rasterizer.device), torch.zeros(n, dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)
    assert (ref_c > 0).sum() > 1000 and (ref_c == 0).sum() > 1000
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
    np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


@pytest.mark.parametrize("w, h", [(321, 243), (147, 143)])
@pytest.mark.parametrize("n", [4 * 3551 - 1, 4 * 3551 + 1, 8 * 3552 - 4, 8 * 3552 + 1, 32 * 3552 - 4, 32 * 3552 + 1, 1_000_001])
def test_grid_loss_many_cells(rasterizer, n, w, h):
    """Cell numbers around those at which a warp of 148 SMs goes about its cells in another way: more groups of four than the stride from one of its
    groups to the next (3551), from twice to eight times as many as there are warps (two groups, eight groups at a time).  Small and large boxes around
    the camera and the border of the image; coverage is exact."""
    import torch

    sc = scenes.config_planar(64, w, h, 200.0, n_views=1, seed=3)
    rng = np.random.default_rng(n)
    centre = np.repeat(rng.uniform(-12, 12, size=(n // 4 + 1, 3)), 4, axis=0)[:n]
    size = np.repeat(10.0 ** rng.uniform(-2.5, 0.2, size=(n // 4 + 1, 1)), 4, axis=0)[:n]
    bb_min = (centre + size * rng.uniform(-1, 1, size=(n, 3))).astype(np.float32)
    bb_len = np.broadcast_to(size, (n, 3)).astype(np.float32).copy()
    loss = rng.standard_normal((3, h, w)).astype(np.float32)
    ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(n, device=rasterizer.device), torch.zeros(n, dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)
    assert (ref_c > 0).sum() > n // 100 and (ref_c == 0).sum() > n // 2
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
    np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


@pytest.mark.parametrize("n", [1, 3, 5, 31, 33, 130])
def test_grid_loss_rows_and_corners(rasterizer, n):
    """Boxes whose front face covers 1 to 200 rows, among them the numbers around a chunk of 64 rows, with corners on whole and half
    pixels (the front face stands at depth 1 of a focal length of 256, the back face at depth 2): exact coverage."""
    import torch

    w, h = 400, 300
    sc = scenes.config_planar(64, w, h, 256.0, n_views=1, seed=3)
    sc.poses = np.array([[0, 0, 0, 1, 0, 0, 0, 0]], np.float64)
    sc.intrinsics[0, :4] = 256.0, 256.0, 200.0, 150.0
    rng = np.random.default_rng(n)
    rows = np.resize(np.array([64, 65, 63, 128, 127, 129, 1, 2, 32, 33, 200, 192, 193]), n)
    u, v = rng.integers(32, 200, n), rng.integers(32, 60, n)
    columns = rng.integers(1, 150, n)
    bb_min = np.stack([(u - 200) / 256, (v - 150) / 256, np.ones(n)], 1).astype(np.float32)
    bb_len = np.stack([columns / 256, rows / 256, np.ones(n)], 1).astype(np.float32)
    loss = rng.standard_normal((3, h, w)).astype(np.float32)
    ref_v, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(n, device=rasterizer.device), torch.zeros(n, dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min), t(bb_len), t(loss), value, count)
    assert (ref_c > 0).any()
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
    np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


# Rotation of the camera, box, principal row: of the boxes with the outermost corner on a whole row (one in ten thousand of them) some for which
# the fp32 middles and halves of the segments that meet at the corner, as they are rounded, leave the row out.
_CORNERS_ON_ROWS = [
    ((0.30658183, 0.36946553, 0.5665552, -0.66971487), (4.2802687, -0.24014834, 1.4477539), (2.1629434, 1.3006504, 1.2766961), 350.27316),
    ((0.07821663, -0.5740086, -0.34341568, 0.7392307), (3.5538538, 1.9203218, -1.1163687), (1.498105, 1.3347545, 0.76249063), 349.79883),
    ((-0.22463317, -0.9429001, 0.18938075, 0.15688913), (-0.5152078, -3.4728684, -4.5743327), (1.0238084, 1.3970141, 1.3433175), 349.5322),
    ((-0.22463317, -0.9429001, 0.18938075, 0.15688913), (-0.6212897, -4.195308, -6.3612576), (1.0719604, 2.115874, 1.9900571), 349.7246),
    ((-0.7046612, -0.5607396, -0.15494646, 0.40622082), (3.4207447, -2.508509, -7.8716316), (2.3550122, 2.3201106, 3.090605), 350.05362),
    ((0.7350364, -0.5994996, 0.31396294, 0.041821703), (1.9027438, -1.8412875, -3.2669928), (1.125605, 1.089446, 1.4549216), 349.70297),
    ((-0.2781702, 0.555939, 0.44323123, -0.6458322), (3.2008967, 2.9440315, 1.6696035), (1.8064176, 2.9341648, 1.5898691), 349.9827),
    ((-0.42319033, 0.78361243, 0.22142796, 0.39727974), (-5.389095, 0.34001753, -5.5709224), (2.9694746, 1.5295297, 1.505763), 349.54324),
    ((-0.8119283, -0.18111958, 0.3197237, 0.4535911), (-2.4465358, -5.170887, -5.085798), (2.266861, 1.5348879, 2.192551), 350.13196),
    ((-0.5533877, 0.038533997, 0.70032746, 0.44924226), (-4.645606, -1.2301524, 1.5215195), (2.0896008, 1.491314, 0.97503215), 349.83658),
    ((0.79685336, -0.52456146, 0.21881467, 0.20489049), (2.2056577, -1.0097961, -2.7729173), (2.0048594, 0.9074665, 1.3701627), 350.31216),
    ((-0.62642443, 0.5759482, -0.31922892, 0.41709593), (-1.5578544, -6.227739, -1.2585564), (2.7273932, 2.3098223, 1.7034277), 350.2481),
    ((0.7696578, -0.5616687, 0.3031369, -0.01622326), (2.23646, -4.3709273, -4.1443353), (2.1590297, 1.5269341, 3.0312054), 350.3346),
    ((-0.5932387, -0.104229875, 0.67960924, 0.4187305), (-5.274751, -2.8566115, 0.8076543), (3.3586922, 1.9716004, 2.1268368), 350.19293),
]


def test_grid_loss_outermost_corner_on_a_row(rasterizer):
    """Boxes of 270 to 700 pixels whose leftmost or rightmost corner alone lies on a whole row: the run of that row ends at the corner
    and not at an inner segment (47 to 274 pixels less).  Coverage is exact."""
    import torch

    w, h = 1400, 700
    sc = scenes.config_planar(64, w, h, 700.0, n_views=1, seed=3)
    loss = np.random.default_rng(5).standard_normal((3, h, w)).astype(np.float32)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    on = t(loss)
    for quaternion, bb_min, bb_len, row in _CORNERS_ON_ROWS:
        sc.poses = np.array([quaternion + (0, 0, 0, 0)], np.float32).astype(np.float64)
        sc.intrinsics[:] = 0
        sc.intrinsics[0, :4] = 700.0, 700.0, 700.0, row
        box = [np.array([a], np.float32) for a in (bb_min, bb_len)]
        ref_v, ref_c = O.grid_loss(sc, sc.views[0], *box, loss)
        value, count = torch.zeros(1, device=rasterizer.device), torch.zeros(1, dtype=torch.int32, device=rasterizer.device)
        rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(box[0]), t(box[1]), on, value, count)
        assert ref_c[0] > 10_000
        np.testing.assert_array_equal(count.cpu().numpy(), ref_c)
        np.testing.assert_allclose(value.cpu().numpy(), ref_v, rtol=1e-5, atol=0)


@pytest.mark.parametrize("n, w, h, distorted", [(30, 1920, 1080, False), (4000, 1920, 1080, False), (20_000, 1920, 1080, False),
                                                (30, 1920, 1080, True), (30, 640, 480, True), (30, 333, 251, True)])
def test_grid_loss_chunks_of_the_per_pixel_form(rasterizer, n, w, h, distorted):
    """Boxes without depth (per-pixel form) of a few to 1.8 million pixels, around the sizes from which on a cell's chunks are larger; few of them, so many
    that all chunks are of the largest size, and more than the queue has room for.  A distorted camera in images of the three sizes that
    its chunks go by.  Coverage is exact."""
    import torch

    sc = scenes.config_planar(64, w, h, 1000.0, n_views=1, seed=3)
    sc.poses = np.array([[0, 0, 0, 1, 0, 0, 0, 0]], np.float64)
    sc.intrinsics[0, :4] = 1000.0, 1000.0, w / 2, h / 2
    if distorted:
        sc.intrinsics[0, 5:] = (0.05, -0.02, 0.001, 0.01, 0.0, 0.0, 0.001, -0.002)
    size = np.array([(3, 3), (8, 8), (9, 8), (64, 9), (256, 255), (256, 256), (257, 256), (256, 257), (512, 256), (513, 256), (512, 257), (512, 512),
                     (513, 513), (700, 700), (1800, 1000)], np.float32)
    bb_len = np.concatenate([size / 1000, np.zeros((len(size), 1))], 1).astype(np.float32)
    bb_min = np.tile(np.array([[(90.3 - w / 2) / 1000, (60.3 - h / 2) / 1000, 1.0]], np.float32), (len(size), 1))
    loss = np.ones((1, h, w), np.float32)
    _, ref_c = O.grid_loss(sc, sc.views[0], bb_min, bb_len, loss)
    assert ref_c.min() > 0 and n * ref_c.mean() / 512 > {30: 0, 4000: 2 ** 19, 20_000: 2 ** 22}[n]
    which = np.arange(n) % len(size)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device)  # noqa: E731
    value, count = torch.zeros(n, device=rasterizer.device), torch.zeros(n, dtype=torch.int32, device=rasterizer.device)
    rasterizer.grid_loss(t(sc.poses), t(sc.intrinsics), sc.views[0], t(bb_min[which]), t(bb_len[which]), t(loss), value, count)
    np.testing.assert_array_equal(count.cpu().numpy(), ref_c[which])
    np.testing.assert_array_equal(value.cpu().numpy(), ref_c[which].astype(np.float32))  # whole numbers below 2^24


# ---- mode 0 without camera gradients: the pixels of all levels are looked up together


@pytest.mark.parametrize("layers, ghost, by_radius", [(1, 0, 1), (4, 1, 1), (5, 0, 0), (5, 0, 1)])
def test_mode0_backward_without_cameras(rasterizer, layers, ghost, by_radius):
    """Against the oracle; counts of hits per point and which descriptors are reached are exact."""
    sc = scenes.tiny_scene(n=9000, w=93, h=61, n_views=2, seed=13, crop=True)
    dropout = (np.random.default_rng(2).random((2, sc.n)) < 0.2).astype(np.float32)
    params = default_params(render_mode=0, num_layers=layers, ghost_gradients=ghost, drop_out_points_by_radius=by_radius)
    ora = util.run_oracle(sc, params, dropout=dropout)
    grads = util.random_grads(ora["fwd"]["color"], seed=3)
    ora = util.run_oracle(sc, params, grads=grads, dropout=dropout)
    gpu = util.run_gpu(rasterizer, sc, params, grads=grads, dropout=dropout)
    import torch

    on = [torch.from_numpy(g).to(rasterizer.device) for g in grads]
    plain = rasterizer.backward_raw(on, want_pose=False, want_intrinsics=False)
    raw = dict(gpu["bwd_raw"], **{k: v.cpu().numpy() for k, v in plain.items()})
    # the bound of the other mode-0 tests (see test_mode0_backward_scratch)
    util.compare_backward(raw, ora, 4, rtol=2e-5, floor_rel=1e-6)
    assert np.array_equal(raw["points"][:, 3], gpu["bwd_raw"]["points"][:, 3]) and raw["points"][:, 3].sum() > 0


def test_calls_after_close_are_refused():
    """Every call of a closed rasterizer raises VetrError with the library's status for a missing context."""
    import torch
    from vet_b200 import _lib as L
    from vet_b200.render import Rasterizer, scene_to_device

    rast = Rasterizer(0)
    sc = scenes.tiny_scene(n=500, w=40, h=32, n_views=1, seed=3)
    tensors = scene_to_device(sc, rast.device)
    fwd = rast.forward(*tensors, sc.views, default_params())
    grads, loss = [torch.ones_like(c) for c in fwd["color"]], torch.zeros((), device=rast.device)
    raw = rast.backward_raw(grads)
    torch.cuda.synchronize()
    rast.close()
    calls = [lambda: rast.forward(*tensors, sc.views, default_params()), lambda: rast.backward_raw(grads),
             lambda: rast.backward_raw(grads, accum=raw), lambda: rast.finalize(raw),
             lambda: rast.l1_loss_grad(fwd["color"], grads, grads, loss)]
    for call in calls:
        with pytest.raises(L.VetrError) as e:
            call()
        assert e.value.status == L.E_INVALID_ARG


def test_follows_the_current_stream(monkeypatch):
    """Kernels go to torch's current stream, which is asked for through public interfaces only."""
    import torch
    from vet_b200.render import Rasterizer, scene_to_device

    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream")
    rast = Rasterizer(0)
    sc = scenes.tiny_scene(n=500, w=40, h=32, n_views=1, seed=3)
    tensors = scene_to_device(sc, rast.device)
    want = rast.forward(*tensors, sc.views, default_params())["color"][0].clone()
    assert rast._cur_stream == torch.cuda.current_stream(rast.device).cuda_stream
    torch.cuda.synchronize()
    side = torch.cuda.Stream(rast.device)
    with torch.cuda.stream(side):
        got = rast.forward(*tensors, sc.views, default_params())["color"][0]
        assert rast._cur_stream == side.cuda_stream != 0
        side.synchronize()  # nothing else is waited for
        assert torch.equal(got, want)
    rast.close()


@pytest.mark.parametrize("n", [500, 1])
@pytest.mark.parametrize("mode, forward, backward", [
    (0, 4, 1 + 2 + 1),  # clear, nearest depth, splat, combine; gradients cleared, pack or background, points, epilogue
    (1, 7, 1 + 4 + 1),  # clear, count, two of the scan, collect, two of sort + blend; pack, lists, long lists, points
    (2, 7, 1 + 5 + 1),  # long lists in two kernels
    (3, 7, 1 + 4 + 1)])
def test_launch_count(mode, forward, backward, n):
    """vetr_launch_count counts every kernel once."""
    from vet_b200.render import Rasterizer, scene_to_device
    import torch

    rast = Rasterizer(0)
    sc = scenes.tiny_scene(n=n, w=40, h=32, n_views=1, seed=3)
    tensors, params = scene_to_device(sc, rast.device), default_params(render_mode=mode)
    before = rast.launch_count()
    grads = [torch.ones_like(c) for c in rast.forward(*tensors, sc.views, params)["color"]]
    between = rast.launch_count()
    rast.finalize(rast.backward_raw(grads))
    assert (between - before, rast.launch_count() - between) == (forward, backward)
    rast.close()


def test_launch_count_of_an_empty_cloud():
    """Mode 0 without points: the clearing and combining kernels, then the background sum."""
    import torch
    from vet_b200.render import Rasterizer, scene_to_device

    class NoPoints:  # an empty tensor has no address, which the library wants
        shape = (0, 4)

        def __init__(self, t):
            self.data_ptr = t.data_ptr

    rast = Rasterizer(0)
    sc = scenes.tiny_scene(n=8, w=40, h=32, n_views=1, seed=3)
    position, index, *rest = scene_to_device(sc, rast.device)
    before = rast.launch_count()
    out = rast.forward(NoPoints(position), NoPoints(index), *rest, sc.views, default_params(render_mode=0))
    assert rast.launch_count() - before == 2
    rast.backward_raw([torch.ones_like(c) for c in out["color"]], want_points=False)
    assert rast.launch_count() - before == 2 + 1 + 1  # gradients cleared, background summed
    rast.close()


# ---- kernels that are set up while the one before them ends


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
def test_steps_follow_one_another(rasterizer, mode):
    """Steps that follow one another on the stream, each with inputs that were written just before it, give what the same steps give with
    the device waited for between all calls: no kernel starts on data that the one before it still works on."""
    import torch

    sc = scenes.config_planar(20_000, 200, 120, 125.0, n_views=2, seed=5)
    pos, index, tex, conf, bg, poses, intr = (torch.from_numpy(np.ascontiguousarray(a)).to(rasterizer.device) for a in (
        sc.position, sc.index, sc.texture, sc.confidence, sc.background, sc.poses, sc.intrinsics))
    prm = default_params(render_mode=mode, num_layers=4, num_channels=tex.shape[0])
    loss = torch.zeros((), device=rasterizer.device)
    given = [torch.randn(2, tex.shape[0], h, w, device=rasterizer.device) for w, h in level_sizes(200, 120, 4)]

    def steps(wait):
        p, t, q, results = pos.clone(), tex.clone(), poses.clone(), []
        for k in range(12):
            p[:, :3] += 0.01 * (-1) ** k
            q[:, 4] += 0.02
            t.mul_(0.9)
            wait()
            out = rasterizer.forward(p, index, t, conf, bg, q, intr, sc.views, prm)
            wait()
            targets = [torch.zeros_like(c) for c in out["color"]]
            grads = [torch.empty_like(c) for c in out["color"]]
            rasterizer.l1_loss_grad(out["color"], targets, grads, loss)
            wait()
            raw = rasterizer.backward_raw(given)  # (grads holds signs, which may differ where an image is next to nothing)
            wait()
            g = rasterizer.finalize(raw)
            results.append([c.clone() for c in out["color"]] + [loss.clone(), g["texture"].clone(), g["points"].clone(), g["pose"].clone()])
            wait()
        torch.cuda.synchronize()
        return results

    for a, b in zip(steps(torch.cuda.synchronize), steps(lambda: None)):
        for x, y in zip(a, b):  # the order of fp32 sums is not fixed
            assert torch.allclose(x, y, rtol=1e-4, atol=1e-5 * float(x.abs().max()))


# ---- items of sort + blend from a counter, long lists first


@pytest.mark.parametrize("mode, n", [(1, 270_000), (2, 270_000), (3, 70_000)])
def test_large_batches_are_their_halves(rasterizer, mode, n):
    """Eight views of a cloud that reach the number of fragments from which on long lists go first and items come from a counter, against the same
    views four at a time, below it: the same lists in the same order, the same images bit for bit."""
    import torch

    sc = scenes.config_planar(n, 160, 96, 100.0, n_views=8, seed=6)
    tensors = scene_to_device(sc, rasterizer.device)
    params = default_params(render_mode=mode, num_layers=3, drop_out_points_by_radius=0)
    whole = rasterizer.forward(*tensors, sc.views, params)
    fragments, longest = rasterizer.fragment_count()
    assert longest > 256  # some are left to the kernel for long lists
    lists = [rasterizer.lists_of(view, level) for view in range(8) for level in range(3)]
    seen = 0
    for first in (0, 4):
        half = rasterizer.forward(*tensors, sc.views[first:first + 4], params)
        seen += rasterizer.fragment_count()[0]
        for key in ("color", "weight"):
            for a, b in zip(whole[key], half[key]):
                assert torch.equal(a[first:first + 4], b)
        for view in range(4):
            for level in range(3):
                for a, b in zip(lists[3 * (first + view) + level], rasterizer.lists_of(view, level)):
                    assert torch.equal(a, b)
    assert seen == fragments


@pytest.mark.parametrize("mode, n", [(1, 262_145), (1, 1_048_577), (3, 262_145)])
def test_points_per_thread_same_lists(rasterizer, mode, n):
    """Eight views against four at a time, just above the points times views from which on a thread takes several points: mode 1 in counting, mode 1 in
    collecting (both count several), mode 3 in both."""
    test_large_batches_are_their_halves(rasterizer, mode, n)
