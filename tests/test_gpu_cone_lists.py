"""Renders through cone lists against renders that search the BVH from its root.

crRenderPosesDevice builds, for launches with many rays, a list per (pose,
ommatidium) of what that ommatidium's samples can hit first;
crRenderPosesDeviceNoAlloc never does.  Both find the same closest hits and
sum them in the same order, so their results are equal bit for bit, for any
eye and pose.
"""
import ctypes
import math

import numpy as np
import pytest

import eyeRendererHelperFunctions as eh
import scenes

pytestmark = pytest.mark.gpu

# spp: the fewest that use lists and a full segment of 8 and of 16 lanes
# (several lists a warp), the smallest whole-warp segment, tails of one sample,
# one chunk, several chunks in a block, chunks that no block holds.
SPP = [5, 8, 9, 16, 17, 31, 32, 33, 64, 96, 256, 300, 513]


def _eye(n, kind):
    rng = np.random.default_rng(n)
    d = scenes.fibonacci_sphere(n)
    omm = np.zeros((n, 8), np.float32)
    omm[:, 0:3], omm[:, 3:6] = d * 0.001, d
    omm[:, 6] = np.radians(rng.uniform(0.5, 6.0, n))
    if kind == "odd":  # axes on the coordinate planes, wide, narrow, negative and zero cones, offsets, long axes
        s = math.sqrt(0.5)
        omm[:6, 3:6] = [[0, 1, 0], [0, -1, 0], [s, 0, s], [1, 0, 0], [0, 0, -1], [-s, 0, -s]]
        omm[6:12, 6] = np.radians([60.0, 25.0, 0.0, -3.0, 1e-4, 179.0])
        omm[12:40, 7] = np.linspace(-0.01, 0.02, 28)
        omm[40:50, 3:6] *= np.linspace(0.5, 2.0, 10)[:, None].astype(np.float32)
        omm[50:60, 3:6] *= np.float32(1.0004)
        omm[60, 3:6] = 0.0
        omm[61, 6] = np.nan
    return omm


@pytest.fixture(scope="module")
def deep(tmp_path_factory):
    """A terrain with a deep tree (at least 16384 triangles): lists from 5
    samples on, sorted rounds in the adaptive render."""
    d = tmp_path_factory.mktemp("deep")
    return scenes.terrain_scene(str(d), cells=96, extent=60.0, cones=40, n_omm=500, poses=1)


def _load(lib, info):
    lib.setOmmatidia.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.loadGlTFscene(info["gltf"].encode())
    assert eh.lastError(lib) == ""
    assert "height_fn" not in info or lib.crGetTriangleCount() >= 16384
    eh.gotoFirstCompoundEye(lib)


def _poses(info, count, seed):
    rng = np.random.default_rng(seed)
    if "height_fn" in info:
        p = scenes.random_poses(info["height_fn"], count, rng, 20.0)
        boxes = np.array([[[-1.0, 0.0, -1.0], [1.0, 0.5, 1.0]]] * 2)
    else:
        boxes = info["boxes"]
        p = scenes.open_poses(boxes, count, rng)
    p16 = np.zeros((count, 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p[:, 3 * k:3 * k + 3]
    p16[0, 1] = 0.0  # on the ground plane
    p16[1, 0:3] = boxes[0].mean(axis=0)  # inside a box
    p16[2, 0:3] = boxes[1][1]  # on a box's corner
    p16[3, 4:7] *= 1.0004  # a frame within the lists' tolerance, and three outside it
    p16[4, 4:16] *= 2.0
    p16[5, 4:7] = p16[5, 8:11]
    p16[6, 8:11] = 0.0
    p16[7, 0:3] = [500.0, 300.0, -900.0]  # far outside
    p16[8, 0] = np.nan
    return p16


def _render(lib, fn, d_poses, P, n):
    import torch

    out = torch.full((P, n, 3), -1.0, device="cuda")
    torch.cuda.synchronize()
    assert fn(d_poses.data_ptr(), P, out.data_ptr()) == 0, eh.lastError(lib)
    assert lib.crSynchronize() == 0, eh.lastError(lib)
    return out.cpu().numpy()


def _both(lib, omm, spp, p16):
    """Frames of both entry points from the same random streams, after one
    frame through each path's set-up, and the streams they leave."""
    import torch

    n, P = len(omm), len(p16)
    d_poses = torch.from_numpy(p16).cuda()
    res = []
    for fn in (lib.crRenderPosesDevice, lib.crRenderPosesDeviceNoAlloc):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        _render(lib, lib.crRenderPosesDevice, d_poses, 1, n)  # one frame: odd, so a normal is cached
        held = lib.crGetDeviceMemoryHeld()
        a = _render(lib, fn, d_poses, P, n)
        b = _render(lib, fn, d_poses, 1, n)
        states = np.zeros(8 * n * spp, np.uint32)
        assert lib.crGetRandomStates(states) == 0
        res.append((a, b, states, lib.crGetDeviceMemoryHeld() - held))
    return res


@pytest.mark.parametrize("kind", ["plain", "odd"])
@pytest.mark.parametrize("spp", SPP)
def test_lists_change_no_bit(lib, small, deep, kind, spp):
    info, rays = (deep, 2 ** 20) if spp <= 16 else (small, 2 ** 21)  # just past the fewest rays that use lists
    _load(lib, info)
    n = 701 if spp > 16 else rays // (60 * spp) | 1
    P = 2 + rays // (n * spp)
    if P < 9:
        n, P = rays // (9 * spp) + 1, 9
    with_lists, without = _both(lib, _eye(n, kind), spp, _poses(info, P, spp))
    assert with_lists[3] >= 400 * n * P and without[3] == 0  # the first did build lists
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("segment", [8, 16])
def test_lists_of_narrow_segments(lib, deep, segment):
    """Many samples in segments of 8 or 16 lanes: chunk partials of several
    ommatidia a warp, with a last warp that is not full."""
    _load(lib, deep)
    assert lib.crSetRenderLayout(128, segment) == 0
    try:
        with_lists, without = _both(lib, _eye(701, "odd"), 50, _poses(deep, 31, 2))
    finally:
        lib.crSetRenderLayout(0, 32)
    assert with_lists[3] > 400 * 701 * 31
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("spp", [5, 8, 16, 20])
def test_feature_rows_with_and_without_lists(lib, deep, spp):
    """Feature rows and 8-sample means of the denoiser."""
    assert lib.crDenoiserInit(1) == 0
    n = 3001
    omm = _eye(n, "odd")
    P = 2 ** 20 // (n * spp) + 2
    p12 = scenes.random_poses(deep["height_fn"], P, np.random.default_rng(4), 20.0)
    got = []
    for lists in (True, False):
        _load(lib, deep)
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(1)
        x, base = np.zeros((P * n, 112), np.uint16), np.zeros((P * n, 3), np.float32)
        if not lists:  # the statistics and rows of the first run are still held
            assert lib.crSetDeviceMemoryCap(lib.crGetDeviceMemoryHeld() + (24 << 20)) == 0
        held = lib.crGetDeviceMemoryHeld()
        try:
            assert lib.crDenoiserFeatureRows(p12, P, spp, x, base) == 0, eh.lastError(lib)
        finally:
            lib.crSetDeviceMemoryCap(0)
        assert (lib.crGetDeviceMemoryHeld() - held > 400 * P * n) == lists
        got.append((x, base))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1], equal_nan=True)


def test_lists_of_a_single_leaf_scene(lib, tmp_path):
    """A scene that is one BVH leaf (the root's second child is a dummy)."""
    g = scenes.GltfBuilder()
    v, f = scenes.box_mesh([-1.0, 0.0, -1.0], [1.0, 1.0, 1.0])
    g.mesh("ground", v, f[:7], colours=np.random.default_rng(1).uniform(0, 1, (8, 4)))
    d = scenes.fibonacci_sphere(10)
    scenes.write_eye(str(tmp_path / "e.eye"), d * 0.001, d, 0.05, 0.0)
    g.compound_camera("eye", "e.eye")
    lib.setOmmatidia.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.loadGlTFscene(g.write(str(tmp_path / "one.gltf")).encode())
    assert eh.lastError(lib) == ""
    eh.gotoFirstCompoundEye(lib)
    p = np.zeros((64, 16), np.float32)
    rng = np.random.default_rng(2)
    p[:, 0:3] = rng.uniform(-2.0, 2.0, (64, 3))
    p[:, 4] = p[:, 9] = p[:, 14] = 1.0
    with_lists, without = _both(lib, _eye(1100, "plain"), 32, p)
    assert with_lists[3] > 0
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y)


def test_lists_give_way_under_a_memory_cap(lib, small):
    """Lists are dropped, not the render, when their memory is not to be had."""
    _load(lib, small)
    omm, p16 = _eye(800, "plain"), _poses(small, 90, 3)
    want = _both(lib, omm, 64, p16)[0][0]
    _load(lib, small)  # gives back every buffer
    lib.setOmmatidia(omm.ctypes.data, len(omm))
    lib.setCurrentEyeSamplesPerOmmatidium(64)
    import torch

    d_poses = torch.from_numpy(p16).cuda()
    _render(lib, lib.crRenderPosesDevice, d_poses, 1, len(omm))
    # room for the partials and pre-drawn numbers of the launch, not for the lists
    need = 4 * 90 * 800 * 2 * 3 + 8 * 90 * 800 * 64
    assert lib.crSetDeviceMemoryCap(lib.crGetDeviceMemoryHeld() + need + (1 << 20)) == 0
    try:
        got = _render(lib, lib.crRenderPosesDevice, d_poses, 90, len(omm))
    finally:
        lib.crSetDeviceMemoryCap(0)
    assert np.array_equal(got, want, equal_nan=True)


def test_batch_with_and_without_lists(lib, tmp_path):
    """A batch whose eyes partly go through lists (16 samples fill no warp
    segment) equals each eye's render without lists, frame by frame."""
    import torch

    P, spp = 5, [16, 48, 256, 1, 100]
    info = scenes.batch_scene(str(tmp_path), n_eyes=len(spp), poses_per_eye=P, n_min=600, n_max=3000)
    lib.loadGlTFscene(info["gltf"].encode())
    cams = np.arange(info["first_batch_camera"], info["first_batch_camera"] + len(spp), dtype=np.int32)
    p12 = info["poses"].reshape(-1, 12)
    p16 = np.zeros((len(p12), 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p12[:, 3 * k:3 * k + 3]
    assert sum(n * s for n, s in zip(info["n"], spp)) * P >= 2 ** 21
    d_poses = torch.from_numpy(p16).cuda()
    want = []
    for i, c in enumerate(cams):
        lib.gotoCamera(int(c))
        lib.setCurrentEyeSamplesPerOmmatidium(spp[i])
        _render(lib, lib.crRenderPosesDevice, d_poses[i * P:], 1, info["n"][i])
        lib.crSynchronize()
        want.append(_render(lib, lib.crRenderPosesDeviceNoAlloc, d_poses[i * P:], P, info["n"][i]))
    for i, c in enumerate(cams):  # the same streams again, one frame in
        lib.gotoCamera(int(c))
        lib.setCurrentEyeSamplesPerOmmatidium(spp[i])
        _render(lib, lib.crRenderPosesDevice, d_poses[i * P:], 1, info["n"][i])
    out = torch.full((3 * P * sum(info["n"]),), -1.0, device="cuda")
    torch.cuda.synchronize()
    held = lib.crGetDeviceMemoryHeld()
    h = lib.crBatchCreate(cams, len(cams), P, d_poses.data_ptr(), out.data_ptr())
    assert h > 0, eh.lastError(lib)
    assert lib.crGetDeviceMemoryHeld() - held >= 400 * P * sum(n for n, s in zip(info["n"], spp) if s > 16)
    assert lib.crBatchLaunch(h) == 0 and lib.crSynchronize() == 0, eh.lastError(lib)
    got = out.cpu().numpy()
    lat, total = np.zeros(len(cams), np.float32), ctypes.c_float(0.0)
    assert lib.crBatchLatencies(h, lat, ctypes.byref(total)) == 0
    assert (lat > 0).all() and total.value == lat.max()
    for i in range(len(cams)):
        o = lib.crBatchOutputOffset(h, i)
        assert np.array_equal(got[o:o + want[i].size].reshape(want[i].shape), want[i]), spp[i]
    lib.crBatchDestroy(h)


@pytest.mark.parametrize("on_deep", [False, True])
@pytest.mark.parametrize("spp", [16, 32, 64, 256, 512])
def test_adaptive_records_with_and_without_lists(lib, small, deep, on_deep, spp):
    """crAdaptiveRecord through lists and (under a memory cap) without: the
    same rays, hits, colours and sums.  Two entries a warp, one round, several,
    a pool's worth, two chunks; an odd number of entries."""
    info = deep if on_deep else small
    _load(lib, info)
    if on_deep:
        p12 = scenes.random_poses(info["height_fn"], 3, np.random.default_rng(5), 20.0)
    else:
        p12 = scenes.open_poses(small["boxes"], 3, np.random.default_rng(6))
    n = (2 ** (19 if on_deep else 21) // (3 * spp) + 2) | 1
    omm = _eye(n, "odd")
    lib.setOmmatidia(omm.ctypes.data, n)
    lib.setCurrentEyeSamplesPerOmmatidium(1)
    p12 = np.ascontiguousarray(p12, np.float32)
    rows = 3 * n
    got = []
    for lists in (True, False):
        rec = np.zeros((rows, spp), eh.RAY_RECORD_DTYPE)
        sums = np.zeros((rows, 3), np.float32)
        if lists:
            assert lib.crAdaptiveRecord(p12[:1], 1, 1, 9, np.zeros((n, 1), eh.RAY_RECORD_DTYPE).ctypes.data,
                                        np.zeros((n, 3), np.float32)) == 0, eh.lastError(lib)
        else:
            _load(lib, info)  # gives the lists back
            lib.setOmmatidia(omm.ctypes.data, n)
            lib.setCurrentEyeSamplesPerOmmatidium(1)
            assert lib.crAdaptiveRecord(p12[:1], 1, 1, 9, np.zeros((n, 1), eh.RAY_RECORD_DTYPE).ctypes.data,
                                        np.zeros((n, 3), np.float32)) == 0, eh.lastError(lib)
            need = rows * (4 + 12 + 12 * max(1, spp // 256) + 64 * spp) + rows * 100
            assert lib.crSetDeviceMemoryCap(lib.crGetDeviceMemoryHeld() + need) == 0
        held = lib.crGetDeviceMemoryHeld()
        try:
            assert lib.crAdaptiveRecord(p12, 3, spp, 9, rec.ctypes.data, sums) == 0, eh.lastError(lib)
        finally:
            lib.crSetDeviceMemoryCap(0)
        assert (lib.crGetDeviceMemoryHeld() - held >= rows * (64 * spp + 400)) == lists
        got.append((rec, sums))
    assert got[0][0].tobytes() == got[1][0].tobytes()
    assert np.array_equal(got[0][1], got[1][1], equal_nan=True)


def test_adaptive_render_with_and_without_lists(lib, deep):
    """The whole adaptive render with entries in several buckets."""
    import torch

    omm, P = _eye(2501, "plain"), 20
    p12 = scenes.random_poses(deep["height_fn"], P, np.random.default_rng(8), 20.0)
    p16 = np.zeros((P, 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p12[:, 3 * k:3 * k + 3]
    d_poses = torch.from_numpy(p16).cuda()
    res = []
    lib.crDenoiserRelease()
    assert lib.crAllocatorInit(3) == 0 and lib.crSetAllocatorHalvings(-4.0) == 0
    try:
        for lists in (True, False):
            _load(lib, deep)
            lib.setOmmatidia(omm.ctypes.data, len(omm))
            lib.setCurrentEyeSamplesPerOmmatidium(1)
            out = torch.full((P, len(omm), 3), -1.0, device="cuda")
            lev = torch.zeros((P, len(omm)), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            if not lists:  # buffers of the first render are still there; no room for lists
                assert lib.crSetDeviceMemoryCap(lib.crGetDeviceMemoryHeld() + (12 << 20)) == 0
            assert lib.crAdaptiveRenderPosesDevice(d_poses.data_ptr(), P, 8, out.data_ptr(),
                                                   lev.data_ptr(), None) == 0, eh.lastError(lib)
            assert lib.crSynchronize() == 0, eh.lastError(lib)
            res.append((out.cpu().numpy(), lev.cpu().numpy()))
    finally:
        lib.crSetDeviceMemoryCap(0)
        lib.crSetAllocatorHalvings(0.0)
    assert len(np.unique(res[0][1])) >= 2 and (res[0][1] != 255).mean() > 0.5
    assert np.array_equal(res[0][1], res[1][1]) and np.array_equal(res[0][0], res[1][0])


@pytest.mark.parametrize("n,spp,P", [(3, 5, 1025), (40, 32, 700), (701, 8, 513), (33, 513, 257)])
def test_long_launches_of_small_eyes(lib, small, n, spp, P):
    """More than 256 poses in one launch, and in launches of 256 when the
    memory for one is not to be had."""
    _load(lib, small)
    poses = _poses(small, P, n)
    long, usual = _both(lib, _eye(n, "plain"), spp, poses)
    for x, y in zip(long[:3], usual[:3]):
        assert np.array_equal(x, y, equal_nan=True)
    _load(lib, small)
    omm = _eye(n, "plain")
    import torch

    d_poses = torch.from_numpy(poses).cuda()
    for cap in (False, True):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        _render(lib, lib.crRenderPosesDevice, d_poses, 255, n)  # the buffers of a usual launch
        if cap:
            assert lib.crSetDeviceMemoryCap(lib.crGetDeviceMemoryHeld() + 8 * 10 * n * spp + 4096) == 0
        try:
            got = _render(lib, lib.crRenderPosesDevice, d_poses, P, n)
        finally:
            lib.crSetDeviceMemoryCap(0)
        if not cap:
            want = got
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("on_deep,spp", [(False, 32), (False, 100), (True, 8), (True, 33)])
def test_negative_focal_offsets(lib, small, deep, on_deep, spp):
    """Rays of a negative focal offset start ahead of the ommatidium and hit
    what lies between (the ground and boxes here), in every kind of launch."""
    info = deep if on_deep else small
    _load(lib, info)
    n, rays = 801, 2 ** 20 if on_deep else 2 ** 21
    P = max(9, rays // (n * spp) + 2)
    omm = _eye(n, "plain")
    omm[::10, 7] = -np.linspace(0.3, 3.0, len(omm[::10]), dtype=np.float32)
    poses = _poses(info, P, spp)
    with_lists, without = _both(lib, omm, spp, poses)
    assert with_lists[3] >= 400 * n * P
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y, equal_nan=True)
    omm[::10, 7] = 0.0  # the offsets do decide what is seen
    assert not np.array_equal(_both(lib, omm, spp, poses)[1][0][:, ::10], without[0][:, ::10], equal_nan=True)


@pytest.mark.parametrize("slack", [0, 40000, 90000])
def test_record_with_cuts_under_a_cap_that_fits_the_lists(lib, small, slack):
    """crAdaptiveRecord with a cut radius and a memory cap that has room for
    the lists, but (up to 69,360 bytes more) not for the lists and the cuts:
    the cuts come first, and the lists are left out."""
    P, spp = 256, 32
    p12 = np.ascontiguousarray(scenes.open_poses(small["boxes"], P, np.random.default_rng(6)), np.float32)
    n = 2 ** 21 // (P * spp) + 3
    rows = P * n
    assert lib.crSetCutRadius(1.0 / 32) == 0
    got = []
    try:
        for cap in (False, True):
            _load(lib, small)
            omm = _eye(n, "plain")
            lib.setOmmatidia(omm.ctypes.data, n)
            lib.setCurrentEyeSamplesPerOmmatidium(1)
            assert lib.crAdaptiveRecord(p12[:1], 1, 1, 9, np.zeros((n, 1), eh.RAY_RECORD_DTYPE).ctypes.data,
                                        np.zeros((n, 3), np.float32)) == 0, eh.lastError(lib)
            rec, sums = np.zeros((rows, spp), eh.RAY_RECORD_DTYPE), np.zeros((rows, 3), np.float32)
            held = lib.crGetDeviceMemoryHeld()
            if cap:  # entries, sums, records, poses (perhaps held already); the lists
                need = rows * (4 + 12 + 64 * spp) + 4 + 64 * (P - 1)
                lib.crSetDeviceMemoryCap(held + need + rows * 31 * 16 + slack)
            try:
                assert lib.crAdaptiveRecord(p12, P, spp, 9, rec.ctypes.data, sums) == 0, eh.lastError(lib)
            finally:
                lib.crSetDeviceMemoryCap(0)
            assert (lib.crGetDeviceMemoryHeld() - held >= rows * (64 * spp + 400)) == (not cap or slack > 272 * (P - 1))
            got.append((rec, sums))
    finally:
        lib.crSetCutRadius(0.0)
    assert got[0][0].tobytes() == got[1][0].tobytes() and np.array_equal(got[0][1], got[1][1])


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    """A scene whose linear BVH is nearly as deep as the traversal stack:
    every facet's Morton code shares one bit less with the origin's."""
    rng = np.random.default_rng(3)
    c = [rng.uniform(0, 2.0 ** -22, 3) for _ in range(8)]
    r = [2.0 ** -21] * 8
    for k in range(57):
        e = np.zeros(3)
        e[k % 3] = 1.2 * 2.0 ** -(1 + k // 3)
        c.append(e)
        r.append(0.4 * 2.0 ** -(1 + k // 3))
    for e in np.eye(3):  # the corners of the unit cube
        c.append(e)
        r.append(0.2)
    tri = np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]]) + np.zeros(3)
    v = np.concatenate([x + s * tri for x, s in zip(c, r)])
    d = tmp_path_factory.mktemp("chain")
    g = scenes.GltfBuilder()
    g.mesh("chain", v.astype(np.float32), np.arange(len(v)).reshape(-1, 3), colours=rng.uniform(0, 1, (len(v), 4)))
    a = scenes.fibonacci_sphere(10)
    scenes.write_eye(str(d / "e.eye"), a * 0.001, a, 0.05, 0.0)
    g.compound_camera("eye", "e.eye")
    return {"gltf": g.write(str(d / "chain.gltf"))}


@pytest.mark.parametrize("spp", [32, 100])
def test_lists_of_a_tree_as_deep_as_the_stack(lib, chain, spp):
    """A list's entries wait on the stack of a subtree's search, which needs no
    more of it than a search from the root."""
    n = 701
    P = max(12, 2 ** 21 // (n * spp) + 2)
    omm = _eye(n, "plain")
    rng = np.random.default_rng(5)
    axis = np.ones(3) / math.sqrt(3.0)
    omm[:600, 3:6] = axis  # most look along the diagonal, some exactly
    omm[200:600, 3:6] += rng.normal(0, 0.05, (400, 3))
    omm[200:600, 3:6] /= np.linalg.norm(omm[200:600, 3:6], axis=1)[:, None]
    omm[:, 0:3] = 0.0
    omm[100:300, 6] = 0.0
    p = np.zeros((P, 16), np.float32)
    p[:, 0:3] = -axis * 10.0 ** rng.uniform(-7, 0, (P, 1)) + rng.normal(0, 1, (P, 3)) * 10.0 ** rng.uniform(-9, -2, (P, 1))
    p[::3, 0:3] = -axis * 10.0 ** rng.uniform(-7, 0, (len(p[::3]), 1))
    p[:, 4] = p[:, 9] = p[:, 14] = 1.0
    assert lib.crSetBvhBuilder(1) == 0
    try:
        _load(lib, chain)
        with_lists, without = _both(lib, omm, spp, p)
    finally:
        lib.crSetBvhBuilder(0)
    depth = ctypes.c_uint32()
    lib.crGetBvhStats(None, None, ctypes.byref(depth))
    assert 54 <= depth.value <= 62
    assert with_lists[3] >= 400 * n * P and len(np.unique(without[0][0])) > 3
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n,spp,P,lists", [(2000, 256, 4, False), (101, 64, 1, False), (6000, 128, 2, False),
                                           (700, 512, 17, True), (900, 64, 300, True), (1100, 100, 40, True)])
def test_no_more_memory_than_without_lists(lib, small, n, spp, P, lists):
    """Chunk sums stay in the block with and without lists, or need no more
    scratch than without: under a cap of what the launch without lists holds,
    every call is accepted, before and after one with lists."""
    import torch

    _load(lib, small)
    omm, p16 = _eye(n, "plain"), _poses(small, max(P, 9), P)[:P]
    d_poses = torch.from_numpy(p16).cuda()
    got = []
    for capped in (True, False, True):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        _render(lib, lib.crRenderPosesDevice, d_poses, 1, n)
        held = lib.crGetDeviceMemoryHeld()
        if capped and not got:  # 8 bytes a ray where the poses are spread over the warps, for 256 poses at most
            chunks = (spp + 31) // 32
            split = P > 1 and n * chunks < 8192
            room = min(P, 256) * n * (8 * spp + 12 * chunks) if split else 0
            assert lists or split or room == 0
            lib.crSetDeviceMemoryCap(held + room)
        elif capped:
            lib.crSetDeviceMemoryCap(held)
        try:
            got.append(_render(lib, lib.crRenderPosesDevice, d_poses, P, n))
        finally:
            lib.crSetDeviceMemoryCap(0)
        if got[1:] and not capped:
            assert (lib.crGetDeviceMemoryHeld() - held > 400 * min(P, 256) * n) == lists
    for g in got[1:]:
        assert np.array_equal(g, got[0], equal_nan=True)


@pytest.mark.parametrize("n,spp,P", [(6000, 256, 1), (6000, 400, 1), (700, 512, 17), (900, 64, 300), (40, 32, 700)])
def test_capture_after_one_render(lib, small, deep, n, spp, P):
    """A render captured into a graph after the same render once outside: the
    capture allocates nothing, and its replay gives the next frames."""
    import torch

    info = deep if P == 1 else small  # a single frame with lists
    _load(lib, info)
    omm, p16 = _eye(n, "plain"), _poses(info, max(P, 9), P)[:P]
    d_poses = torch.from_numpy(p16).cuda()
    out = torch.zeros((P, n, 3), device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    res = []
    for captured in (False, True):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        assert lib.crSetStream(st.cuda_stream) == 0
        try:
            render = lambda: lib.crRenderPosesDevice(d_poses.data_ptr(), P, out.data_ptr())
            assert render() == 0
            held = lib.crGetDeviceMemoryHeld()
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st):
                    rc = render()
                assert rc == 0, eh.lastError(lib)
                assert lib.crGetDeviceMemoryHeld() == held
                for _ in range(2):
                    with torch.cuda.stream(st):
                        g.replay()
            else:
                assert render() == 0 and render() == 0
            assert lib.crSynchronize() == 0
        finally:
            lib.crSetStream(None)
        res.append(out.cpu().numpy())
    assert np.array_equal(res[0], res[1], equal_nan=True)


def test_captured_render_survives_longer_ones(lib, small):
    """A captured render of 256 poses keeps its buffers when renders of more
    poses follow outside the capture, with room for their own and without."""
    import torch

    _load(lib, small)
    n, spp, P = 901, 32, 256
    omm, p16 = _eye(n, "plain"), _poses(small, 1024, 3)
    d_poses = torch.from_numpy(p16).cuda()
    out = torch.zeros((1024, n, 3), device="cuda")
    other = torch.zeros((1024, n, 3), device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    res = []
    assert lib.crSetCutRadius(1.0 / 32) == 0 and lib.crSetStream(st.cuda_stream) == 0
    try:
        for captured in (False, True):
            lib.setOmmatidia(omm.ctypes.data, n)
            lib.setCurrentEyeSamplesPerOmmatidium(spp)
            render = lambda count, o: lib.crRenderPosesDevice(d_poses.data_ptr(), count, o.data_ptr())
            assert render(P, out) == 0
            if captured:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st):
                    rc = render(P, out)
                assert rc == 0, eh.lastError(lib)
            for cap in (0, 1):
                lib.crSetDeviceMemoryCap(cap and lib.crGetDeviceMemoryHeld())
                try:
                    assert render(1024, other) == 0, eh.lastError(lib)
                finally:
                    lib.crSetDeviceMemoryCap(0)
                assert render(1024, other) == 0 and lib.crSynchronize() == 0
                if captured:
                    with torch.cuda.stream(st):
                        g.replay()
                else:
                    assert render(P, out) == 0
                assert lib.crSynchronize() == 0
                res.append((out.cpu().numpy(), other.cpu().numpy()))
    finally:
        lib.crSetStream(None)
        lib.crSetCutRadius(0.0)
    for a, b in zip(res[:2], res[2:]):
        assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True)


@pytest.mark.parametrize("n,spp,P", [(3, 64, 257), (701, 9, 513), (2900, 8, 769), (40, 33, 1025)])
def test_tails_of_long_launches(lib, small, deep, n, spp, P):
    """A last launch of one pose after long ones, which sums in the block and
    draws for itself."""
    info = deep if spp < 17 else small
    _load(lib, info)
    long, usual = _both(lib, _eye(n, "plain"), spp, _poses(info, P, n))
    for x, y in zip(long[:3], usual[:3]):
        assert np.array_equal(x, y, equal_nan=True)


def test_poses_of_a_launch_without_lists(lib, small):
    """Renders that build no lists take 256 poses a launch, however many
    ommatidia the eye has (the launches of a captured render are counted)."""
    import torch

    _load(lib, small)
    n, spp, P = 100000, 4, 256
    omm = _eye(n, "plain")
    d_poses = torch.from_numpy(_poses(small, P, 1)).cuda()
    out = torch.zeros((P, n, 3), device="cuda")
    st = torch.cuda.Stream()
    cu = ctypes.CDLL("libcuda.so.1")
    s, graph, nodes = ctypes.c_void_p(st.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    torch.cuda.synchronize()
    lib.setOmmatidia(omm.ctypes.data, n)
    lib.setCurrentEyeSamplesPerOmmatidium(spp)
    assert lib.crSetStream(st.cuda_stream) == 0
    try:
        assert lib.crRenderPosesDevice(d_poses.data_ptr(), 1, out.data_ptr()) == 0 and lib.crSynchronize() == 0
        assert cu.cuStreamBeginCapture_v2(s, 1) == 0  # thread-local mode
        rc = lib.crRenderPosesDevice(d_poses.data_ptr(), P, out.data_ptr())
        assert cu.cuStreamEndCapture(s, ctypes.byref(graph)) == 0 and rc == 0
    finally:
        lib.crSetStream(None)
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(nodes)) == 0
    cu.cuGraphDestroy(graph)
    assert nodes.value == 1


def test_long_renders_on_two_streams(lib, tmp_path):
    """Renders of two eyes issued back to back on two streams share the memory
    of their lists; each gives the frames that it gives alone."""
    import torch

    P, spp, rounds = 9, 128, 6
    info = scenes.batch_scene(str(tmp_path), n_eyes=2, poses_per_eye=P, n_min=2600, n_max=3400)
    lib.loadGlTFscene(info["gltf"].encode())
    cams = [info["first_batch_camera"], info["first_batch_camera"] + 1]
    p12 = info["poses"].reshape(-1, 12)
    p16 = np.zeros((len(p12), 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p12[:, 3 * k:3 * k + 3]
    d_poses = torch.from_numpy(p16).cuda()
    assert all(4 * n >= 8192 and n * spp * P >= 2 ** 21 for n in info["n"])  # no pre-drawn numbers; lists
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    res = []
    try:
        for apart in (True, False):
            out = [torch.full((rounds, P, n, 3), -1.0, device="cuda") for n in info["n"]]
            for c in cams:
                lib.gotoCamera(c)
                for k in (1, spp):  # a change of the sample count restarts the streams
                    lib.setCurrentEyeSamplesPerOmmatidium(k)
                    assert lib.crRenderPosesDevice(d_poses.data_ptr(), 1, out[cams.index(c)].data_ptr()) == 0
                    assert lib.crSynchronize() == 0
            torch.cuda.synchronize()
            for k in range(rounds):
                for i, c in enumerate(cams):
                    lib.gotoCamera(c)
                    lib.crSetStream(streams[i].cuda_stream)
                    assert lib.crRenderPosesDevice(d_poses[i * P:].data_ptr(), P, out[i][k].data_ptr()) == 0
                    if apart:
                        assert lib.crSynchronize() == 0
            torch.cuda.synchronize()
            res.append([o.cpu().numpy() for o in out])
    finally:
        lib.crSetStream(None)
    for a, b in zip(*res):
        assert (a >= 0).all() and np.array_equal(a, b)


def test_batch_gives_its_lists_back(lib, tmp_path):
    """Under a memory cap that a batch's lists fill, a later render takes what
    it needs from them, and the batch goes on without."""
    import torch

    P, spp = 5, [33, 256, 100]
    info = scenes.batch_scene(str(tmp_path), n_eyes=len(spp), poses_per_eye=P, n_min=1500, n_max=3000)
    cams = np.arange(info["first_batch_camera"], info["first_batch_camera"] + len(spp), dtype=np.int32)
    p12 = info["poses"].reshape(-1, 12)
    p16 = np.zeros((len(p12), 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p12[:, 3 * k:3 * k + 3]
    d_poses = torch.from_numpy(p16).cuda()
    n0 = info["n"][0]
    lists = 31 * 16 * P * sum(info["n"])
    res = []
    for cap in (False, True):
        lib.loadGlTFscene(info["gltf"].encode())  # gives back every buffer
        for i, c in enumerate(cams):
            lib.gotoCamera(int(c))
            for k in (1, spp[i]):  # a change of the sample count restarts the streams
                lib.setCurrentEyeSamplesPerOmmatidium(k)
                _render(lib, lib.crRenderPosesDevice, d_poses[i * P:], 1, info["n"][i])
        lib.gotoCamera(int(cams[0]))
        out = torch.full((3 * P * sum(info["n"]),), -1.0, device="cuda")
        torch.cuda.synchronize()
        held = lib.crGetDeviceMemoryHeld()
        h = lib.crBatchCreate(cams, len(cams), P, d_poses.data_ptr(), out.data_ptr())
        assert h > 0, eh.lastError(lib)
        batch = lib.crGetDeviceMemoryHeld()
        assert batch - held >= lists
        frames = []
        try:
            for k in range(2):
                assert lib.crBatchLaunch(h) == 0 and lib.crSynchronize() == 0, eh.lastError(lib)
                frames.append(out.cpu().numpy())
                if cap:
                    lib.crSetDeviceMemoryCap(batch + 4096)
                frames.append(_render(lib, lib.crRenderPosesDevice, d_poses, 6 + k, n0))
        finally:
            lib.crSetDeviceMemoryCap(0)
        assert (lib.crGetDeviceMemoryHeld() < batch) == cap
        lib.crBatchDestroy(h)
        res.append(frames)
    for a, b in zip(*res):
        assert (a >= 0).all() and np.array_equal(a, b)


def test_batch_latencies_count_the_lists(lib, tmp_path):
    """crBatchLatencies counts from the start of the launch, the building of
    lists (over 0.1 ms of this batch) included."""
    import torch

    P = 50
    info = scenes.batch_scene(str(tmp_path), n_eyes=1, poses_per_eye=P, n_min=30000, n_max=30000)
    lib.loadGlTFscene(info["gltf"].encode())
    cams = np.array([info["first_batch_camera"]], np.int32)
    p16 = np.zeros((P, 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = info["poses"].reshape(-1, 12)[:, 3 * k:3 * k + 3]
    d_poses, out = torch.from_numpy(p16).cuda(), torch.zeros((P, 30000, 3), device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    lib.gotoCamera(int(cams[0]))
    lib.setCurrentEyeSamplesPerOmmatidium(17)
    assert lib.crSetStream(st.cuda_stream) == 0
    try:
        h = lib.crBatchCreate(cams, 1, P, d_poses.data_ptr(), out.data_ptr())
        assert h > 0, eh.lastError(lib)
        lat, total, apart = np.zeros(1, np.float32), ctypes.c_float(0.0), []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            assert lib.crBatchLaunch(h) == 0
            b.record(st)
            assert lib.crSynchronize() == 0
            assert lib.crBatchLatencies(h, lat, ctypes.byref(total)) == 0 and lat[0] == total.value
            apart.append(a.elapsed_time(b) - total.value)  # the counters' reset before, the launch itself
        lib.crBatchDestroy(h)
    finally:
        lib.crSetStream(None)
    assert -0.01 < min(apart) < 0.06, apart


def test_measured_traversal_of_long_renders(lib, deep):
    """crMeasureTraversal counts the search of the tree however many rays the
    render has: the mean of its poses' own counts."""
    import torch

    _load(lib, deep)
    n, spp, P = 1001, 32, 32
    omm = _eye(n, "plain")
    d_poses = torch.from_numpy(_poses(deep, P, 2)[9:]).cuda()
    P -= 9
    assert n * spp * P >= 2 ** 19
    torch.cuda.synchronize()
    counts = []
    for per in (P, 1):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        a = np.zeros(2)
        for k in range(0, P, per):
            nv, tt = ctypes.c_double(), ctypes.c_double()
            assert lib.crMeasureTraversal(d_poses[k:].data_ptr(), per, ctypes.byref(nv), ctypes.byref(tt)) == 0
            a += np.array([nv.value, tt.value]) * per / P
        counts.append(a)
    assert np.allclose(counts[0], counts[1], rtol=1e-12) and counts[0][0] > 5


# rays around each line of coneMaxAngle, for every segment width and depth of tree
@pytest.mark.parametrize("on_deep,n,spp,P", [(True, 1301, 32, 13), (True, 1301, 32, 50), (True, 1301, 32, 110),
                                             (True, 1301, 16, 30), (True, 1301, 16, 250), (True, 1301, 8, 200),
                                             (True, 1301, 8, 410), (False, 1301, 32, 55), (False, 1301, 32, 110),
                                             (False, 1301, 16, 210)])
def test_wide_cones(lib, small, deep, on_deep, n, spp, P):
    """Acceptance angles of 6 to 20 degrees: some get lists, some do not,
    depending on the launch."""
    info = deep if on_deep else small
    _load(lib, info)
    omm = _eye(n, "plain")
    omm[:, 6] = np.radians(np.random.default_rng(n).uniform(6.0, 20.0, n))
    with_lists, without = _both(lib, omm, spp, _poses(info, P, n))
    assert with_lists[3] >= 400 * n * min(P, 256)
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y, equal_nan=True)


def test_batch_of_odd_eyes(lib, tmp_path):
    """Odd eyes and poses in a batch with lists, against each eye's render
    without."""
    import torch

    P, spp = 9, [33, 128]
    info = scenes.batch_scene(str(tmp_path), n_eyes=2, poses_per_eye=P, n_min=2000, n_max=2000)
    lib.setOmmatidia.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.loadGlTFscene(info["gltf"].encode())
    cams = np.arange(info["first_batch_camera"], info["first_batch_camera"] + 2, dtype=np.int32)
    boxes = scenes.small_scene(str(tmp_path / "b"))["boxes"]
    d_poses = torch.from_numpy(np.concatenate([_poses({"boxes": boxes}, P, k) for k in (1, 2)])).cuda()
    omm = _eye(2000, "odd")
    out = torch.full((2, P, 2000, 3), -1.0, device="cuda")
    want = []
    for batch in (False, True):
        for i, c in enumerate(cams):
            lib.gotoCamera(int(c))
            lib.setOmmatidia(omm.ctypes.data, 2000)
            lib.setCurrentEyeSamplesPerOmmatidium(spp[i])
            _render(lib, lib.crRenderPosesDevice, d_poses[i * P:], 1, 2000)
            if not batch:
                want.append(_render(lib, lib.crRenderPosesDeviceNoAlloc, d_poses[i * P:], P, 2000))
    h = lib.crBatchCreate(cams, 2, P, d_poses.data_ptr(), out.data_ptr())
    assert h > 0 and lib.crBatchLaunch(h) == 0 and lib.crSynchronize() == 0, eh.lastError(lib)
    lib.crBatchDestroy(h)
    for i in range(2):
        assert np.array_equal(out[i].cpu().numpy(), want[i], equal_nan=True)


@pytest.mark.parametrize("spp", [17, 64])
def test_lit_renders_through_lists(lib, small, spp):
    _load(lib, small)
    n = 701
    P = max(9, 2 ** 21 // (n * spp) + 2)
    assert lib.crSetLighting(1) == 0
    try:
        with_lists, without = _both(lib, _eye(n, "odd"), spp, _poses(small, P, spp))
    finally:
        lib.crSetLighting(0)
    assert with_lists[3] >= 400 * n * P
    for x, y in zip(with_lists[:3], without[:3]):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("pose", [0, 1, 2, 3, 4, 5, 7])
def test_recorded_frames_through_lists(lib, small, deep, pose):
    """A recorded frame of an odd eye at odd poses: the colours of the same
    frame without lists, and records that add up to them."""
    import torch

    info = deep if pose % 2 else small
    _load(lib, info)
    n, spp = (6001, 350) if info is small else (3001, 200)
    omm, p = _eye(n, "odd"), _poses(info, 9, 4)[pose]
    d_pose = torch.from_numpy(p.reshape(1, 16)).cuda()
    got = []
    for record in (True, False):
        lib.setOmmatidia(omm.ctypes.data, n)
        lib.setCurrentEyeSamplesPerOmmatidium(spp)
        _render(lib, lib.crRenderPosesDevice, d_pose, 1, n)
        if record:
            lib.setCameraPosition(*[float(v) for v in p[0:3]])
            lib.setCameraLocalSpace(*[float(v) for k in (4, 8, 12) for v in p[k:k + 3]])
            rec, col = np.zeros((n, spp), eh.RAY_RECORD_DTYPE), np.zeros((n, 3), np.float32)
            assert lib.crRenderFrameRecorded(rec.ctypes.data) == 0, eh.lastError(lib)
            assert lib.getOmmatidialColoursF32(col) == 0
            got.append(col)
        else:
            got.append(_render(lib, lib.crRenderPosesDeviceNoAlloc, d_pose, 1, n)[0])
    assert np.array_equal(got[0], got[1], equal_nan=True)
    total = rec["rgb"].sum(1, dtype=np.float64) / spp
    ok = np.isfinite(got[0])
    assert np.allclose(total[ok], got[0][ok], rtol=1e-4, atol=1e-6)


def test_renders_of_an_empty_eye(lib, small):
    """No ommatidia: every render succeeds and writes nothing."""
    import torch

    _load(lib, small)
    d_poses = torch.from_numpy(_poses(small, 300, 1)).cuda()
    out = torch.full((300,), -1.0, device="cuda")
    torch.cuda.synchronize()
    lib.setOmmatidia(None, 0)
    for P in (1, 4, 300):
        assert lib.crRenderPosesDevice(d_poses.data_ptr(), P, out.data_ptr()) == 0, eh.lastError(lib)
    assert lib.crSynchronize() == 0
    assert (out.cpu().numpy() == -1.0).all()
