"""The host path of a call: where images come from, how results leave, and launches that are recorded as graphs. Needs a GPU.

The same frames must give the same bits whichever way their images take (inside the staging block, through the upload helpers,
straight from pinned memory, already on the device) and whether the chunk's kernels are launched one by one (a shape's first
call) or as a graph (the calls that follow)."""
import numpy as np
import pytest

import golden_io as G
from visualmesh_b200 import workloads as W
from visualmesh_b200.engine import Engine, FrameInput, Mesh, pinned_empty, pinned_free

pytestmark = pytest.mark.gpu


def _same(a, b):
    for name in ("pixel_coordinates", "global_indices", "neighbourhood", "classifications"):
        assert np.array_equal(G.bits(getattr(a, name)) if getattr(a, name).dtype == np.float32 else getattr(a, name),
                              G.bits(getattr(b, name)) if getattr(b, name).dtype == np.float32 else getattr(b, name)), name


# bytes of an RGBA frame: inside the staging block (up to 128 KB in all), one slice, around the 256 KB slices, many slices
@pytest.mark.parametrize("width,height", [(96, 64), (181, 181), (256, 256), (257, 256), (1280, 1024)])
def test_images_from_every_kind_of_memory_give_the_same_results(width, height):
    import torch
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    lens = W.Lens((width, height), W.EQUISOLID, 0.35 * width, (0.0, 0.0), (0.0, 0.0), np.pi)
    engine = Engine(case.network)
    code = W.fourcc("RGBA")
    image = W.random_bytes(7, width * height * 4)
    pinned = pinned_empty(image.size)
    pinned[:] = image
    device = torch.from_numpy(image).cuda()
    torch.cuda.synchronize()
    frames = {"pageable": FrameInput(mesh, case.frames[0]["Hoc"], lens, image, code, None),
              "pinned": FrameInput(mesh, case.frames[0]["Hoc"], lens, pinned, code, None),
              "device": FrameInput(mesh, case.frames[0]["Hoc"], lens, device.data_ptr(), code, None, True)}
    want = engine.run_batch([frames["device"]]).frame(0)
    assert len(want.global_indices) > 100
    for kind, frame in frames.items():
        for _ in range(3):
            _same(engine.run_batch([frame]).frame(0), want)
    # unaligned, and one batch of all three kinds
    shifted = np.empty(image.size + 1, np.uint8)[1:]
    shifted[:] = image
    order = ["pinned", "pageable", "device"]
    for _ in range(3):
        batch = engine.run_batch([frames[k] for k in order] + [FrameInput(mesh, case.frames[0]["Hoc"], lens, shifted, code, None)])
        for f in range(4):
            _same(batch.frame(f), want)
    engine.close()
    pinned_free(pinned)


def test_frames_pinned_one_by_one_that_lie_next_to_one_another():
    """Frames that follow one another in memory travel as one copy, but no copy reaches from one allocation into the next."""
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    lens = W.Lens((512, 512), W.EQUISOLID, 0.35 * 512, (0.0, 0.0), (0.0, 0.0), np.pi)
    engine = Engine(case.network)
    buffers = sorted((pinned_empty(512 * 512 * 4) for _ in range(24)), key=lambda b: b.ctypes.data)
    if not any(b.ctypes.data - a.ctypes.data == a.size for a, b in zip(buffers, buffers[1:])):
        pytest.skip("no two of these allocations lie next to one another")
    for i, b in enumerate(buffers):
        b[:] = W.random_bytes(50 + i, b.size)
    frames = [FrameInput(mesh, case.frames[i % 3]["Hoc"], lens, b, W.fourcc("RGBA"), None) for i, b in enumerate(buffers)]
    want = [engine.run_batch([fr]).frame(0) for fr in frames]
    for _ in range(3):
        batch = engine.run_batch(frames)
        for f, w in enumerate(want):
            _same(batch.frame(f), w)
    engine.close()
    for b in buffers:
        pinned_free(b)


def test_host_ranges_of_changing_poses_leave_nothing_behind():
    """With host ranges the node table is not cleared between calls: entries of an earlier pose must not be taken for points."""
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    engine = Engine(case.network)
    for f in (0, 1, 0, 2, 1, 0):
        fr = case.frames[f]
        out = engine.run_batch([FrameInput(mesh, fr["Hoc"], case.lens, fr["image"], case.format, fr["ranges"])]).frame(0)
        assert np.array_equal(out.global_indices, fr["global_indices"])
        assert np.array_equal(out.neighbourhood, fr["neighbourhood"])
    engine.close()


def test_a_recorded_graph_serves_one_layout_of_the_staging_block_only():
    """Two shapes whose staging blocks have the same size and all their launches the same grids, but the group counts in another
    place: 24576 bytes of images against 12288 of images and 12288 of range slots."""
    case = G.Case("ring4_rectilinear_grey")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    engine = Engine(case.network)
    Hoc, code = case.frames[0]["Hoc"], W.fourcc("GREY")
    everything = np.array([[0, mesh.n_nodes]], np.int32)

    def frame(width, height, ranges):
        lens = W.Lens((width, height), W.EQUISOLID, 0.35 * width, (0.0, 0.0), (0.0, 0.0), np.pi)
        return FrameInput(mesh, Hoc, lens, W.random_bytes(width, width * height), code, ranges)

    batches = [[frame(128, 96, None), frame(128, 96, None)], [frame(64, 96, None), frame(64, 96, everything)]]
    want = [[engine.run_batch([fr]).frame(0) for fr in batch] for batch in batches]
    assert all(len(w.global_indices) > 100 for batch in want for w in batch)
    for _ in range(3):
        for batch, expected in zip(batches, want):
            out = engine.run_batch(batch)
            for f in range(2):
                _same(out.frame(f), expected[f])
    engine.close()


def test_staging_blocks_of_every_size_reach_the_device_whole():
    """Frame constants, ranges and counts come by a copy when the images are on the device already, else they are read by a kernel:
    from one range to 16810 of one node each (204 KB, more than the kernel's threads read in one turn)."""
    import torch
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    lens = W.Lens((640, 512), W.EQUISOLID, 0.35 * 640, (0.0, 0.0), (0.0, 0.0), np.pi)
    engine = Engine(case.network)
    host = W.random_bytes(3, 5 * 640 * 512 * 4).reshape(5, -1)
    device = torch.from_numpy(host).cuda()
    torch.cuda.synchronize()
    nodes = np.arange(mesh.n_nodes, dtype=np.int32)
    for ranges in (None, np.array([[0, mesh.n_nodes]], np.int32), np.stack([nodes, nodes + 1], axis=1)[::7], np.stack([nodes, nodes + 1], axis=1)):
        frames = [[FrameInput(mesh, case.frames[f % 3]["Hoc"], lens, device[f].data_ptr() if there else host[f], W.fourcc("RGBA"), ranges, there)
                   for f in range(5)] for there in (True, False)]
        batch = engine.run_batch(frames[0])
        want = [batch.frame(f) for f in range(5)]
        assert min(len(w.global_indices) for w in want) > 100
        for _ in range(3):
            batch = engine.run_batch(frames[1])
            for f in range(5):
                _same(batch.frame(f), want[f])
    engine.close()


def test_many_frames_with_few_candidates_on_a_mesh_of_many_nodes():
    """The node tables of the batch's frames together pass 2^31 entries, their candidates are 205 k: a chunk is cut before its
    32-bit offsets into the node table overflow."""
    n_nodes, n_frames, part = 8_500_000, 257, 800
    assert n_nodes * (n_frames - 1) > 2**31
    rng = np.random.default_rng(7)
    rays = rng.uniform(-1.0, 1.0, (n_nodes, 3)).astype(np.float32)
    rays /= np.linalg.norm(rays, axis=1, keepdims=True)
    near = np.arange(n_nodes, dtype=np.int64)[:, None] + np.array([-2, -1, 1, 2])
    mesh = Mesh.from_arrays(rays, np.clip(near, 0, n_nodes - 1).astype(np.int32))
    lens = W.Lens((640, 480), W.EQUIDISTANT, 200.0, (0.0, 0.0), (0.0, 0.0), np.pi)
    engine = Engine()
    starts = np.linspace(0, n_nodes - part, n_frames).astype(np.int32)
    frames = [FrameInput(mesh, W.make_Hoc(-0.01 * f, 0.1, 1.0), lens, None, 0, np.array([[s, s + part]], np.int32)) for f, s in enumerate(starts)]
    batch = engine.run_batch(frames)
    got = [batch.frame(f) for f in range(n_frames)]
    assert sum(len(g.global_indices) for g in got) > 10 * n_frames
    for f in list(range(0, n_frames, 16)) + [n_frames - 2, n_frames - 1]:
        want = engine.run_batch([frames[f]]).frame(0)
        assert np.array_equal(G.bits(got[f].pixel_coordinates), G.bits(want.pixel_coordinates))
        assert np.array_equal(got[f].global_indices, want.global_indices) and np.array_equal(got[f].neighbourhood, want.neighbourhood)
    engine.close()


@pytest.mark.parametrize("n_frames", [1, 2, 37])
def test_batches_left_on_the_device_and_copied_to_the_host_agree(n_frames):
    """Results written to the host by the device (one small chunk), copied by the copy engines (several chunks) and left behind."""
    import ctypes
    import torch
    wl = W.config(1, n_frames=n_frames)
    mesh = Mesh.from_spec(wl.frames[0].mesh)
    engine = Engine(wl.network)
    images = torch.randint(0, 256, (n_frames, wl.frames[0].image_bytes), dtype=torch.uint8)
    frames = [FrameInput(mesh, fr.Hoc, fr.lens, images[i].numpy(), fr.format, None) for i, fr in enumerate(wl.frames)]
    on_device = images.cuda()
    torch.cuda.synchronize()
    device_frames = [FrameInput(mesh, fr.Hoc, fr.lens, on_device[i].data_ptr(), fr.format, None, True) for i, fr in enumerate(wl.frames)]
    for _ in range(3):
        left = engine.run_batch(device_frames, results_on_device=True)
        n_cls, total = left.n_classes, left.total_points

        class Array:
            def __init__(self, pointer, shape, kind):
                self.__cuda_array_interface__ = {"data": (ctypes.cast(pointer, ctypes.c_void_p).value, False), "shape": shape, "typestr": kind, "version": 3}
        cls = torch.as_tensor(Array(left.raw.classifications, (total + n_frames, n_cls), "<f4"), device="cuda").cpu().numpy()
        gi = torch.as_tensor(Array(left.raw.global_indices, (total,), "<i4"), device="cuda").cpu().numpy()
        nb = torch.as_tensor(Array(left.raw.neighbourhood, (total + n_frames, 6), "<i4"), device="cuda").cpu().numpy()
        for some in (frames, device_frames):
            batch = engine.run_batch(some)
            for f in range(n_frames):
                out = batch.frame(f, copy=False)
                p0, p1 = left.offsets[f], left.offsets[f + 1]
                assert np.array_equal(out.global_indices, gi[p0:p1])
                assert np.array_equal(out.neighbourhood, nb[p0 + f:p1 + f + 1])
                assert np.array_equal(G.bits(out.classifications), G.bits(cls[p0 + f:p1 + f + 1]))
    engine.close()


# frames per launch: beyond 64 (two turns of a warp over the table of tiles), and one more than a chunk holds
@pytest.mark.parametrize("n_frames", [130, 257])
@pytest.mark.parametrize("widths", [[16, 16, 8, 3], [32, 32, 32, 4]])
def test_batches_of_many_frames_equal_single_frames(n_frames, widths):
    import torch
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    engine = Engine(W.make_network(23, 6, widths))
    size = case.lens.dimensions[0] * case.lens.dimensions[1] * 4
    images = torch.from_numpy(W.random_bytes(29, n_frames * size).reshape(n_frames, size)).cuda()
    torch.cuda.synchronize()
    # from straight down to above the horizon: frames of many rows, few and none
    views = [W.make_Hoc(-1.5 + 3.1 * (7 * f % n_frames) / n_frames, 0.2, 1.0) for f in range(n_frames)]
    frames = [FrameInput(mesh, H, case.lens, images[f].data_ptr(), W.fourcc("RGBA"), None, True) for f, H in enumerate(views)]
    batch = engine.run_batch(frames)
    got = [batch.frame(f) for f in range(n_frames)]
    points = [len(g.global_indices) for g in got]
    assert min(points) < 10 and max(points) > 1000 and len(set(points)) > n_frames // 2
    for f in range(n_frames):
        _same(got[f], engine.run_batch([frames[f]]).frame(0))
    engine.close()


def test_call_looks_up_on_the_host_when_the_device_has_no_bsp():
    """vm_call on a mesh that was uploaded without its BSP: the host tables find the same nodes as the device does."""
    import ctypes as C
    from visualmesh_b200 import abi
    from visualmesh_b200.engine import _c_lens
    lib = abi.load()
    mesh = Mesh("XYGRID6", "CYLINDER", 0.2, 1.8, 1.0, 4.0, 12.0)
    lens = W.Lens((320, 240), W.RECTILINEAR, 190.0, (0.0, 0.0), (0.0, 0.0), 1.8)
    engine = Engine(W.make_network(5, 6, [8, 8, 3]))
    image = W.random_bytes(11, 320 * 240 * 4)
    handle = C.c_void_p()
    abi.check(lib.vm_mesh_upload(engine._ptr, mesh.rays.ctypes.data, mesh.neighbours.ctypes.data, mesh.n_nodes, mesh.n_neighbours, C.byref(handle)))
    most = 0
    for pitch in (-0.2, -0.6, -1.2, 1.5):
        Hoc = W.make_Hoc(pitch, 0.1, 1.0)
        want = engine(mesh, Hoc, lens, image, W.fourcc("RGBA"))
        most = max(most, len(mesh.lookup(Hoc, lens)))
        for _ in range(2):
            res = abi.vm_batch_result()
            abi.check(lib.vm_call(engine._ptr, handle, mesh._ptr, Hoc.ctypes.data, C.byref(_c_lens(lens)), image.ctypes.data, W.fourcc("RGBA"), C.byref(res)))
            n = res.offsets[1]
            assert n == len(want.global_indices)
            if n > 0:
                assert np.array_equal(np.ctypeslib.as_array(res.global_indices, (n,)), want.global_indices)
                assert np.array_equal(np.ctypeslib.as_array(res.neighbourhood, (n + 1, 6)), want.neighbourhood)
                assert np.array_equal(G.bits(np.ctypeslib.as_array(res.classifications, (n + 1, 3))), G.bits(want.classifications))
    assert most > 10
    bad = _c_lens(lens)
    bad.projection = 7
    status = lib.vm_call(engine._ptr, handle, mesh._ptr, Hoc.ctypes.data, C.byref(bad), image.ctypes.data, W.fourcc("RGBA"), C.byref(res))
    assert status == abi.VM_ERR_UNSUPPORTED_LENS
    engine.close()


def test_results_of_a_call_are_the_callers_own():
    """Results kept over later calls (more of them than the engine hands over without a copy), over the engine's end, and given
    back in another order."""
    case = G.Case("ring6_equisolid_rgba")
    mesh = Mesh.from_arrays(case.rays, case.nbrs, case.bsp)
    engine = Engine(case.network)
    frames = [case.frames[i] for i in (0, 1, 0, 1, 1, 0, 2)]
    kept = [engine(mesh, fr["Hoc"], case.lens, fr["image"], case.format, fr["ranges"]) for fr in frames]
    del kept[2]
    kept.insert(2, engine(mesh, frames[2]["Hoc"], case.lens, frames[2]["image"], case.format, "device"))
    columns = kept[1].pixel_coordinates[:, 0]
    engine.close()
    for out, fr in zip(kept, frames):
        assert np.array_equal(out.global_indices, fr["global_indices"]) and np.array_equal(out.neighbourhood, fr["neighbourhood"])
        assert out.pixel_coordinates.shape == fr["pixel_coordinates"].shape and np.abs(out.classifications - fr["classifications"]).max(initial=0.0) < 1e-4
    want = frames[1]["pixel_coordinates"][:, 0].copy()
    kept.clear()
    assert np.array_equal(columns, want)
