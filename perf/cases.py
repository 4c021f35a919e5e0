"""Workloads of the package: training and mapping of rotation- and flip-invariant self-organising maps.

`listed()` holds one case for each kind of use, `draw(rng)` gives further ones over the same ranges; `prepare` makes
what a program has in hand before the call (images, the map, an engine or a trainer object), `run` is one pass through
the public entry points, `work` the bytes and operations the pass cannot do without, `tolerance` how far another
correct implementation's results may be off.

Keys of a case
    op          "train" or "map"
    via         "device": images (and mapping results) are torch tensors on the GPU, Engine.*_device takes their
                addresses; "host": whole numpy arrays, Engine.train / Engine.map; "objects": pink.Trainer /
                pink.Mapper, called for one image at a time
    type        "uint8", "uint16" or "float32" distances
    hexagonal   hexagonal grid of diameter `side` (odd), else a cartesian grid of `side` x `side2` neurons
    channels, image, neuron, region     channels, image side, neuron side, side of the distance region
    circular    circular instead of square distance region
    rotations, flip, sigma, damping     rotations per image, mirrored copies too, the Gaussian neighbourhood
    n           images of one pass
"""
import math

import numpy as np
import torch

from pink_b200 import capi, engine, pink

TYPES = {"uint8": capi.UINT8, "uint16": capi.UINT16, "float32": capi.FLOAT}


def _case(name, op, via, kind, grid, dims, rotations=360, flip=True, circular=False, sigma=1.1, damping=0.2, n=1):
    hexagonal, side, side2 = grid
    channels, image, neuron, region = dims
    return {"name": name, "op": op, "via": via, "type": kind, "hexagonal": hexagonal, "side": side, "side2": side2,
            "channels": channels, "image": image, "neuron": neuron, "region": region, "circular": circular,
            "rotations": rotations, "flip": flip, "sigma": sigma, "damping": damping, "n": n}


def listed():
    return [
        # The smallest call: the best match of a single image, as an interactive session or a request handler asks it.
        _case("map one image", "map", "objects", "uint8", (False, 10, 10), (1, 64, 44, 31)),
        # A short Python loop over images with a small map, the way the module's training script is written.
        _case("train image by image", "train", "objects", "uint8", (False, 8, 8), (1, 64, 45, 31), n=32),
        # An ordinary small map: part of an epoch over images that are already on the GPU.
        _case("train 10x10 uint8", "train", "device", "uint8", (False, 10, 10), (1, 64, 44, 31), n=512),
        # A survey catalogue with a middling hexagonal map, images in plain host memory.
        _case("train hex 331 uint8", "train", "host", "uint8", (True, 21, 21), (1, 124, 64, 45), n=256),
        # The large hexagonal map with fine rotations: the longest training runs.
        _case("train hex 2791 uint8", "train", "device", "uint8", (True, 61, 61), (1, 128, 90, 64), rotations=720,
              sigma=3.0, damping=0.05, n=512),
        # Two-channel images at 16 bits: the largest neurons and the longest distance vectors.
        _case("train 40x40x2 uint16", "train", "device", "uint16", (False, 40, 40), (2, 150, 106, 75), sigma=2.0,
              damping=0.1, n=64),
        # Training with float distances, the type of the reference's CPU path.
        _case("train 20x20 float32", "train", "device", "float32", (False, 20, 20), (1, 128, 90, 64), n=64),
        # Neurons larger than the images (every rotated image fits whole), a hundred steps from host memory.
        _case("train 183 uint8", "train", "host", "uint8", (False, 10, 10), (1, 130, 183, 91), n=100),
        # Odd sizes throughout: neuron planes that are no multiple of four floats, a circular region, no mirroring.
        _case("train ragged circular", "train", "device", "uint8", (False, 7, 9), (1, 101, 71, 49), rotations=92,
              flip=False, circular=True, n=100),
        # Mapping a catalogue to the large map.
        _case("map hex 2791 uint8", "map", "device", "uint8", (True, 61, 61), (1, 128, 90, 64), rotations=720, n=512),
        # Mapping with float distances, images and results in plain host memory.
        _case("map 20x20 float32", "map", "host", "float32", (False, 20, 20), (1, 128, 90, 64), n=512),
        # Mapping of two-channel images at 16 bits.
        _case("map 40x40x2 uint16", "map", "device", "uint16", (False, 40, 40), (2, 150, 106, 75), n=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["train", "train", "map"])
    via = rng.choice(["device", "device", "host", "objects"])
    kind = rng.choice(["uint8", "uint8", "uint16", "float32"])
    channels = rng.choice([1, 1, 1, 2, 3])
    image = _log_int(rng, 40, 160)
    # the default neuron is the largest square inside every rotated image; whole images and their diagonals occur too
    neuron = max(24, min(190, int(image * rng.choice([0.70710678, rng.uniform(0.5, 1.0), 1.41421356]))))
    if channels > 1:
        neuron = min(neuron, 120)
    region = max(15, int(neuron * rng.choice([0.70710678, rng.uniform(0.45, 1.0)])))
    region = min(region, neuron, int(math.sqrt((16500 if kind == "uint16" else 33000) / channels)))
    hexagonal = rng.random() < 0.4
    if hexagonal:
        side = side2 = 2 * _log_int(rng, 2, 30) + 1
    else:
        side, side2 = _log_int(rng, 4, 48), _log_int(rng, 4, 48)
    rotations = rng.choice([360, 360, 4 * _log_int(rng, 4, 180)])
    flip = rng.random() < 0.75
    circular = rng.random() < 0.15
    if circular:
        region -= region % 2 == 0 and neuron % 2 == 1        # the circle then lies centred in its square
    case = _case("", op, via, kind, (hexagonal, side, side2), (channels, image, neuron, region), rotations, flip, circular,
                 sigma=round(rng.uniform(1.0, 3.0), 2), damping=round(rng.uniform(0.05, 0.2), 3))
    del case["name"]
    # as many images as the pass may cost, over a logarithmic range
    one = work(case)["flops"]
    limit = {"uint8": 1.2e13, "uint16": 2.5e12, "float32": 2.5e12}[kind] / one
    limit = min(limit, 4e10 / (8.0 * _neurons(case) * channels * neuron * neuron), 1e9 / (channels * image * image))
    case["n"] = max(1, min(_log_int(rng, 1, 512), int(limit), 64 if via == "objects" else 512))
    return case


def _neurons(case):
    if case["hexagonal"]:
        r = (case["side"] - 1) // 2
        return 3 * r * (r + 1) + 1
    return case["side"] * case["side2"]


def _blobs(n, channels, side, gen):
    """Images on the GPU: one to three elliptical Gaussians and a little noise, clipped at 0, largest value 1; further
    channels show the same objects shifted by up to three pixels and rescaled."""
    def uniform(*shape, lo=0.0, hi=1.0):
        return torch.rand(*shape, generator=gen, device="cuda") * (hi - lo) + lo

    count = torch.randint(1, 4, (n, 1), generator=gen, device="cuda")
    sigma, ratio = uniform(n, 3, lo=2.0, hi=12.0), uniform(n, 3, lo=0.3, hi=1.0)
    angle, amp = uniform(n, 3, hi=math.pi), uniform(n, 3, lo=0.2, hi=1.0)
    amp = amp * (torch.arange(3, device="cuda")[None, :] < count)
    cx, cy = uniform(n, 3, lo=0.3 * side, hi=0.7 * side), uniform(n, 3, lo=0.3 * side, hi=0.7 * side)
    at = torch.arange(side, device="cuda", dtype=torch.float32)
    cos, sin = torch.cos(angle), torch.sin(angle)
    out = torch.empty(n, channels, side, side, device="cuda")
    for c in range(channels):
        if c:
            cx, cy = cx + uniform(n, 3, lo=-3.0, hi=3.0), cy + uniform(n, 3, lo=-3.0, hi=3.0)
            amp = amp * uniform(n, 3, lo=0.5, hi=1.5)
        img = torch.randn(n, side, side, generator=gen, device="cuda") * 0.01
        for b in range(3):
            def p(t):
                return t[:, b, None, None]
            dx, dy = at[None, None, :] - p(cx), at[None, :, None] - p(cy)
            u, v = dx * p(cos) + dy * p(sin), dy * p(cos) - dx * p(sin)
            img += p(amp) * torch.exp(-0.5 * ((u / p(sigma)) ** 2 + (v / (p(sigma) * p(ratio))) ** 2))
        img = img.clamp_(min=0)
        out[:, c] = img / img.amax((1, 2), keepdim=True)
    return out


def _map_weights(case, gen):
    """The map before the call: uniform random numbers before training; for mapping a map as training leaves it, every
    neuron an average of similar objects."""
    n, c, side = _neurons(case), case["channels"], case["neuron"]
    if case["op"] == "train":
        som = torch.rand(n, c, side, side, generator=gen, device="cuda")
        return som.clamp_(max=1.0 - 2.0 ** -24)
    som = _blobs(n, c, side, gen)
    return (0.7 * som + 0.3 * som.flip(3)).mul_(0.9)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    images = _blobs(case["n"], case["channels"], case["image"], gen)
    weights = _map_weights(case, gen).cpu().numpy()
    kind, layout = TYPES[case["type"]], capi.LAYOUT_HEXAGONAL if case["hexagonal"] else capi.LAYOUT_CARTESIAN
    n_neurons, shape = _neurons(case), capi.CIRCULAR if case["circular"] else capi.QUADRATIC
    state = {"op": case["op"], "via": case["via"], "n": case["n"]}
    if case["via"] == "objects":
        many = case["channels"] > 1
        unit = weights.shape[1:] if many else weights.shape[2:]
        grid = (n_neurons,) if case["hexagonal"] else (case["side"], case["side2"])
        som = pink.SOM(weights.reshape(grid + unit), som_layout="hexagonal-2d" if case["hexagonal"] else "cartesian-2d",
                       neuron_layout="cartesian-3d" if many else "cartesian-2d")
        options = {"number_of_rotations": case["rotations"], "use_flip": case["flip"],
                   "euclidean_distance_dim": case["region"], "euclidean_distance_shape": pink.EuclideanDistanceShape(shape),
                   "euclidean_distance_type": pink.DataType(kind)}
        host = images.cpu().numpy()
        state["images"] = host if many else host[:, 0]
        state["layout"] = "cartesian-3d" if many else "cartesian-2d"
        state["som"] = som
        if case["op"] == "train":
            state["trainer"] = pink.Trainer(som, pink.GaussianFunctor(case["sigma"], case["damping"]), **options)
        else:
            state["mapper"] = pink.Mapper(som, **options)
        return state
    eng = engine.Engine(n_neurons, case["channels"], case["image"], case["neuron"], case["region"], case["rotations"],
                        case["flip"], kind, ed_shape=shape)
    eng.set_som(weights)
    state["engine"] = eng
    state["images"] = images if case["via"] == "device" else images.cpu().numpy()
    if case["op"] == "train":
        eng.set_update_function(layout, case["side"], case["side2"], capi.FUNC_GAUSSIAN, case["sigma"], case["damping"])
        # a program that keeps its images on the GPU also keeps a page-locked buffer for the map
        state["result"] = torch.empty(weights.shape, pin_memory=True).numpy() if case["via"] == "device" else np.empty_like(weights)
    elif case["via"] == "device":
        state["distances"] = torch.empty(case["n"], n_neurons, device="cuda")
        state["transforms"] = torch.empty(case["n"], n_neurons, dtype=torch.int32, device="cuda")
    return state


def run(state):
    images, n = state["images"], state["n"]
    if state["via"] == "objects":
        if state["op"] == "map":
            mapper = state["mapper"]
            pairs = [mapper(pink.Data(image, layout=state["layout"])) for image in images]
            return np.array([d for d, _ in pairs], np.float32), np.array([t for _, t in pairs], np.uint32)
        trainer = state["trainer"]
        for image in images:
            trainer(pink.Data(image, layout=state["layout"]))
        trainer.update_som()
        return np.array(state["som"], copy=False), trainer.get_update_info()
    eng = state["engine"]
    if state["op"] == "map":
        if state["via"] == "host":
            return eng.map(images)
        eng.map_device(images.data_ptr(), n, state["distances"].data_ptr(), state["transforms"].data_ptr())
        return state["distances"], state["transforms"]
    if state["via"] == "host":
        eng.train(images)
    else:
        eng.train_device(images.data_ptr(), n)
    return eng.get_som(state["result"]), eng.update_counts(), eng.bmu_log(n)


def work(case):
    """Bytes: images and map read once, the results written once.  Operations: a multiply and an add for every element
    of every (neuron, transform) pair, and the interpolation of a quarter turn's rotations (the others are permutations)."""
    n, c = case["n"], case["channels"]
    neurons, pixels = _neurons(case), c * case["neuron"] ** 2
    transforms = case["rotations"] * (2 if case["flip"] else 1)
    som = 4.0 * neurons * pixels
    out = som if case["op"] == "train" else 8.0 * n * neurons
    distance = 2.0 * n * neurons * transforms * c * case["region"] ** 2
    return {"bytes": 4.0 * n * c * case["image"] ** 2 + som + out,
            "flops": distance + 8.0 * n * (case["rotations"] // 4) * pixels}


def tolerance(case):
    """Integer distances are exact, and so is all that follows from them.  float32 sums differ in their order; where two
    transforms or neurons are closer than that, either may win."""
    if case["type"] != "float32":
        return "exact"
    return {"rel": 1e-5, "max": 1e-3, "differ": 0.005}
