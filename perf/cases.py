"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case names an entry point, a mesh, a camera, a network and a number of frames:

  "call"     Engine(mesh, Hoc, lens, image, format): one camera frame in ordinary host memory, lookup on the host, results
             copied to arrays of the caller - the reference's own call
  "project"  Engine.run_batch on the poses of a rig of cameras, no images: projections only, results on the host
  "device"   Engine.run_prepared on frames that are in device memory, results left there: a ring of camera buffers
  "stream"   Engine.run_batch on frames in device memory whose poses (and meshes) differ in every batch, results left there
  "host"     Engine.run_prepared on frames in pinned host memory, results on the host: the whole path, copies included

The weights and the poses of a case are fixed, as a trained network and a camera's mounting are; the images and the order in
which the frames arrive come from the seed.
"""
import ctypes
import math
import random

import numpy as np
import torch

from visualmesh_b200 import workloads as W
from visualmesh_b200.engine import Engine, FrameInput, Mesh

# C_out of every layer; "," separates the groups (each begins with a gather), "+" the dense layers inside one.
NET_SMALL = "8,8,3"
NET_4 = "16,16,8,2"
NET_6 = "16,16,12,8,8,2"
NET_8 = "16,16,16,16,8,8,8,3"
NET_13 = "16,16,16,16,16,16,8,8,8,8,8,8,5"
NET_DENSE = "32,32,32,32,32,32,32,32,32,4"
NET_GROUPS = "16+16,16+8,8+3"
NET_ODD = "24,20,12,5"
NET_MIXED = "6+5,8+3"


def _case(name, entry, frames, model, shape, h, k, distance, heights, width, height, projection, code, net, activation="selu"):
    return {"name": name, "entry": entry, "frames": frames, "model": model, "shape": shape, "h": h, "k": k, "distance": distance,
            "heights": heights, "width": width, "height": height, "projection": projection, "code": code, "net": net,
            "activation": activation}


def listed():
    return [
        # the smallest call: a coarse mesh on a thumbnail, where only launches, copies and waits count
        _case("call_small", "call", 1, "RING4", "CIRCLE", 1.0, 2.0, 5.0, 1, 128, 96, "rectilinear", "GREY", "4,2"),
        # a robot's vision loop: one full frame after another through the reference's call
        _case("call_frame", "call", 1, "RING6", "SPHERE", 1.2, 6.0, 20.0, 1, 1280, 1024, "equisolid", "RGBA", NET_4),
        # the same loop with a network of the example model's shape on its half-resolution frames: thirteen small layers
        _case("call_model", "call", 1, "RING6", "SPHERE", 1.2, 4.0, 10.0, 1, 640, 512, "equisolid", "RGBA", NET_13),
        # one frame of the densest mesh: the largest single call
        _case("call_dense", "call", 1, "RING8", "SPHERE", 1.6, 12.0, 50.0, 1, 2592, 2048, "equisolid", "RGBA", NET_DENSE),
        # projection only, a rig of six cameras in one batch of new poses
        _case("project_rig", "project", 6, "RING6", "SPHERE", 1.2, 6.0, 20.0, 1, 1280, 1024, "equisolid", "RGBA", ""),
        # offline processing: batches of frames in pinned host memory, results back to the host
        _case("host_fisheye", "host", 32, "RING6", "SPHERE", 1.2, 6.0, 20.0, 1, 1280, 1024, "equidistant", "RGBA", NET_8),
        # frames that a capture card or a decoder leaves in device memory
        _case("device_fisheye", "device", 64, "RING6", "SPHERE", 1.2, 6.0, 20.0, 1, 1280, 1024, "equidistant", "RGBA", NET_8),
        # raw Bayer frames of a narrow lens: large images, few nodes on screen
        _case("device_bayer", "device", 32, "XYGRID6", "CYLINDER", 1.0, 4.0, 15.0, 1, 2048, 1536, "rectilinear", "RGGB", NET_6),
        # large frames on the densest mesh, ten 32-wide layers: the largest batch
        _case("device_dense", "device", 8, "RING8", "SPHERE", 1.6, 12.0, 50.0, 1, 2592, 2048, "equisolid", "RGBA", NET_DENSE),
        # cameras at four heights, a new pose and mesh for every frame
        _case("stream_heights", "stream", 128, "RING6", "SPHERE", 1.2, 6.0, 20.0, 4, 1280, 1024, "equisolid", "RGBA", NET_4),
        # groups of several dense layers behind one gather, eight neighbours, an odd frame size
        _case("device_groups", "device", 16, "RING8", "SPHERE", 1.2, 5.0, 15.0, 1, 641, 479, "equidistant", "BGRA", NET_GROUPS, "relu"),
        # widths that are no power of two, three bytes a pixel, four neighbours, a handful of frames
        _case("device_odd", "device", 5, "XYGRID4", "CYLINDER", 1.1, 5.0, 11.0, 1, 1000, 751, "rectilinear", "RGB8", NET_ODD, "tanh"),
    ]


# ---- sizes -------------------------------------------------------------------------------------------------------------

_SHAPES = {"SPHERE": (0.0949, 0.0), "CIRCLE": (0.1, 0.0), "CYLINDER": (0.2, 1.8)}
_BYTES = {"RGBA": 4, "BGRA": 4, "RGB8": 3, "BGR3": 3, "GREY": 1, "RGGB": 1, "GRBG": 1, "GBRG": 1, "BGGR": 1}
_PROJECTIONS = {"rectilinear": W.RECTILINEAR, "equisolid": W.EQUISOLID, "equidistant": W.EQUIDISTANT}
_ACTIVATIONS = {"selu": W.SELU, "relu": W.RELU, "tanh": W.TANH}


def _neighbours(case):
    return int(case["model"][-1])


def _layers(net, neighbours):
    """(slots, C_in, C_out) of every dense layer"""
    out, width = [], 4
    for group in net.split(",") if net else []:
        for i, c_out in enumerate(group.split("+")):
            out.append((neighbours + 1 if i == 0 else 1, width, int(c_out)))
            width = int(c_out)
    return out


def _products(net, neighbours):
    return sum(s * i * o for s, i, o in _layers(net, neighbours))


def _nodes(model, shape, h, k, distance):
    """About how many nodes a mesh has (from above)."""
    if model.startswith("RING"):
        return 150 * k * k * h * distance
    r = _SHAPES[shape][0]
    return 0.95 * math.pi * (distance * k / (2 * r)) ** 2


def draw(rng):
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        entry = rng.choice(["call", "call", "call", "project", "host", "device", "device", "stream"])
        model, shape = rng.choice([("RING4", "SPHERE"), ("RING6", "SPHERE"), ("RING6", "SPHERE"), ("RING8", "SPHERE"), ("XYGRID4", "CYLINDER"),
                                   ("XYGRID6", "CYLINDER"), ("XYGRID8", "CYLINDER")])
        h = round(rng.uniform(0.6, 1.6), 2)
        k = round(log(2.0, 12.0), 2)
        distance = round(log(5.0, 50.0), 1)
        width = int(log(128, 2592))
        height = max(96, int(width * rng.choice([0.6, 0.75, 0.8])))
        projection = rng.choice(list(_PROJECTIONS))
        code = rng.choice(["RGBA", "RGBA", "BGRA", "RGB8", "GREY", "RGGB", "GBRG"])
        net = rng.choice([NET_SMALL, NET_4, NET_6, NET_8, NET_13, NET_DENSE, NET_GROUPS, NET_ODD, NET_MIXED])
        activation = rng.choice(["selu", "selu", "relu", "tanh"])
        heights = 1
        if entry == "call":
            frames = 1
        elif entry == "project":
            frames, net = 6, ""
        elif entry == "stream":
            frames, heights = int(log(8, 128)), rng.choice([1, 4])
        else:
            frames = int(log(4, 64))
        nodes = _nodes(model, shape, h, k, distance)
        if nodes < 1000 or nodes > 1.5e6 or nodes * frames > 8e6:
            continue
        # no dearer than the largest listed case: in its contractions, in its pixels, and (few tensor-core shapes there) with odd widths
        if nodes * frames * _products(net, int(model[-1])) > 2e11 or width * height * frames > 1280 * 1024 * 64:
            continue
        if net in (NET_ODD, NET_MIXED) and nodes * frames > 1e6:
            continue
        case = _case("", entry, frames, model, shape, h, k, distance, heights, width, height, projection, code, net, activation)
        del case["name"]
        return case


# ---- what a program keeps ------------------------------------------------------------------------------------------------

_meshes = {}
_engine = [None, None]


def _mesh(case, h):
    key = (case["model"], case["shape"], h, case["k"], case["distance"])
    if key not in _meshes:
        while len(_meshes) >= 8:
            del _meshes[next(iter(_meshes))]
        a, b = _SHAPES[case["shape"]]
        _meshes[key] = Mesh(case["model"], case["shape"], a, b, h, case["k"], case["distance"])
    return _meshes[key]


def _network(case):
    """Glorot-uniform weights, small biases, no weight on the alpha channel, softmax at the end."""
    layers = iter(_layers(case["net"], _neighbours(case)))
    rng = np.random.default_rng(17)
    groups = []
    for group in case["net"].split(","):
        groups.append([])
        for _ in group.split("+"):
            slots, c_in, c_out = next(layers)
            limit = math.sqrt(6.0 / (slots * c_in + c_out))
            w = rng.uniform(-limit, limit, (slots, c_in, c_out)).astype(np.float32)
            if len(groups) == 1 and len(groups[0]) == 0:
                w[:, 3, :] = 0.0
            b = rng.uniform(-0.1, 0.1, c_out).astype(np.float32)
            groups[-1].append(W.Layer(np.ascontiguousarray(w.reshape(slots * c_in, c_out)), b, _ACTIVATIONS[case["activation"]]))
    groups[-1][-1].activation = W.SOFTMAX
    return groups


def _engine_of(case):
    """One engine for a network, kept for as long as the program works with it."""
    key = (case["net"], _neighbours(case) if case["net"] else 0, case["activation"])
    if _engine[0] != key:
        _engine[:] = [None, None]
        _engine[:] = [key, Engine(_network(case) if case["net"] else None)]
    return _engine[1]


def _lens(case):
    w, h = case["width"], case["height"]
    if case["projection"] == "rectilinear":
        f = 0.6 * w
        return W.Lens((w, h), W.RECTILINEAR, f, (0.0, 0.0), (-0.05 / w**2, 0.01 / w**4), 2.0 * math.atan(math.hypot(w, h) * 0.5 / f))
    if case["projection"] == "equisolid":
        return W.Lens((w, h), W.EQUISOLID, 0.35 * w, (0.0, 0.0), (0.0, 0.0), math.pi)
    return W.Lens((w, h), W.EQUIDISTANT, 0.3 * w, (0.0, 0.0), (-0.1 / w**2, 0.02 / w**4), math.pi)


def _views(case):
    """(mesh, Hoc) of every frame: a camera that looks down at the field, pitched and rolled as it walks."""
    rng = random.Random(5)
    views = []
    for f in range(case["frames"]):
        h = round(case["h"] * (1 + f % case["heights"]) * (1.0 if case["heights"] == 1 else 1.0 / 3.0), 4)
        pitch, roll = rng.uniform(-70.0, -20.0), rng.uniform(-10.0, 10.0)
        views.append((_mesh(case, h), W.make_Hoc(math.radians(pitch), math.radians(roll), h)))
    return views


# ---- the cases -----------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    engine, lens = _engine_of(case), _lens(case)
    views = _views(case)
    random.Random(seed).shuffle(views)
    state = {"entry": case["entry"], "engine": engine, "lens": lens, "views": views}
    if case["entry"] == "project":
        state["frames"] = [FrameInput(mesh, Hoc, lens) for mesh, Hoc in views]
        return state
    size = case["width"] * case["height"] * _BYTES[case["code"]]
    generator = torch.Generator(device="cuda").manual_seed(seed)
    images = torch.randint(0, 256, (case["frames"], (size + 255) // 256 * 256), dtype=torch.uint8, device="cuda", generator=generator)
    code = W.fourcc(case["code"])
    if case["entry"] == "call":
        state["image"], state["format"] = np.array(images[0, :size].cpu().numpy()), code
        return state
    on_device = case["entry"] != "host"
    if not on_device:
        images = torch.empty(images.shape, dtype=torch.uint8, pin_memory=True).copy_(images)
    torch.cuda.synchronize()
    state["images"] = images
    state["frames"] = [FrameInput(mesh, Hoc, lens, images[f].data_ptr() if on_device else images[f, :size].numpy(), code, None, on_device)
                       for f, (mesh, Hoc) in enumerate(views)]
    if case["entry"] != "stream":
        state["batch"] = engine.prepare_batch(state["frames"])
    return state


class _Device:
    """An array that the engine left in device memory, for torch.as_tensor."""

    def __init__(self, pointer, shape, kind):
        self.__cuda_array_interface__ = {"data": (ctypes.cast(pointer, ctypes.c_void_p).value, False), "shape": shape, "typestr": kind, "version": 3}


def _whole(result):
    """The arrays of a batch as the engine holds them, its frames one after another."""
    raw, points, rows = result.raw, result.total_points, result.total_points + result.n_frames
    parts = [("pixel_coordinates", raw.pixel_coordinates, (points, 2), "<f4"), ("global_indices", raw.global_indices, (points,), "<i4"),
             ("neighbourhood", raw.neighbourhood, (rows, result.n_neighbours), "<i4")]
    if result.n_classes:
        parts.append(("classifications", raw.classifications, (rows, result.n_classes), "<f4"))
    out = {"offsets": result.offsets}
    for name, pointer, shape, kind in parts:
        if result.on_device:
            out[name] = torch.as_tensor(_Device(pointer, shape, kind), device="cuda")
        else:
            out[name] = np.ctypeslib.as_array(pointer, shape=shape)
    return out


def run(state):
    engine, lens = state["engine"], state["lens"]
    if state["entry"] == "call":
        mesh, Hoc = state["views"][0]
        return vars(engine(mesh, Hoc, lens, state["image"], state["format"]))
    if state["entry"] in ("project", "stream"):
        return _whole(engine.run_batch(state["frames"], results_on_device=state["entry"] == "stream"))
    return _whole(engine.run_prepared(state["batch"], results_on_device=state["entry"] == "device"))


def work(case):
    """Every table of a mesh, the sampled texels and the results once; the multiplications and additions of the layers."""
    lens, neighbours, layers = _lens(case), _neighbours(case), _layers(case["net"], _neighbours(case))
    views = _views(case)
    points = 0
    for mesh, Hoc in views:
        ranges = mesh.lookup(Hoc, lens)
        points += int((ranges[:, 1] - ranges[:, 0]).sum())
    rows = points + len(views)
    tables = sum(m.n_nodes * (12 + 4 * neighbours) + 28 * len(m.bsp_ranges) for m in {id(m): m for m, _ in views}.values())
    moved = tables + 12 * points + 4 * neighbours * rows
    if layers:
        image = case["width"] * case["height"] * _BYTES[case["code"]]
        moved += min(image * len(views), 4 * _BYTES[case["code"]] * points) + 4 * layers[-1][2] * rows
        moved += 4 * sum(s * i * o + o for s, i, o in layers)
    return {"bytes": moved, "flops": 2 * rows * _products(case["net"], neighbours)}


def tolerance(case):
    # projections are rounded operation by operation and come out the same; classifications are 32-bit sums over up to thirteen
    # layers (1e-4 of a probability is what a result may be off by)
    return {"rel": 1e-5, "max": 2e-4} if case["net"] else "exact"
