"""The work a user of this library has it do, as cases for timing and comparison.

Faces go in as host arrays and embeddings come out as host arrays: that is the library's public interface
(include/fastface.h, mirrored by fastface_b200.FastFace), so every pass here is one such call, copies included.
Memory is "pageable" (an array from numpy or malloc, what the command-line driver and the wrappers pass) or "pinned"
(page-locked buffers, what a throughput pipeline passes).  Pixels are 8-bit images or the same images normalised to
float32 as callers of the reference do, (p - 127.5) / 127.5.  `ctx` is the context's step batch (256 is what
fastface_create gives; the command-line driver makes one of exactly its --batch).
"""
import math
import tempfile

import numpy as np
import torch

import fastface_b200 as ff
from fastface_b200 import synth

OPS_PER_FACE = 12.619e9          # 6.3093 GMAC: 53 convolutions + FC
WEIGHT_BYTES = 43.6e6            # int8 weights of the whole network
PIXELS = ff.FACE_NELEMS

_engines = {}                    # (step batch, epilogue order) -> FastFace: a program loads its model once


def listed():
    def faces(name, n, pixels, memory, ctx, order="contract"):
        return {"name": name, "what": "faces", "n": n, "pixels": pixels, "memory": memory, "ctx": ctx, "order": order}

    def match(name, n, m):
        return {"name": name, "what": "match", "n": n, "m": m}

    return [
        faces("one_face", 1, "f32", "pageable", 256),                  # unlock / verify: the latency of fastface_embed
        faces("photo_3_u8", 3, "u8", "pageable", 256),                 # the faces of one photo, straight from the decoder
        faces("cli_batch_8", 8, "f32", "pageable", 8),                 # the command-line driver's default batch
        faces("frame_17", 17, "f32", "pageable", 256),                 # one crowded frame, an odd count
        faces("batch_64", 64, "f32", "pageable", 256),                 # a small server batch
        faces("batch_100_u8", 100, "u8", "pinned", 256),               # a server batch of what has arrived, 8-bit pixels
        faces("strict_160_u8", 160, "u8", "pageable", 256, "strict"),  # the other epilogue order, a ragged batch
        faces("batch_256", 256, "f32", "pinned", 256),                 # one full step of the default context
        faces("folder_1000", 1000, "f32", "pageable", 256),            # indexing a folder: several steps, a ragged last one
        faces("batch_1024_u8", 1024, "u8", "pinned", 1024),            # a throughput context, one full step
        faces("stream_4096", 4096, "f32", "pinned", 1024),             # bulk indexing: many full steps in one call
        match("match_1024x1024", 1024, 1024),                          # all pairs: clustering, duplicate search
    ]


def draw(rng):
    if rng.random() < 0.15:
        n = int(round(math.exp(rng.uniform(0.0, math.log(1024)))))
        m = int(round(math.exp(rng.uniform(math.log(100), math.log(10000)))))
        return {"what": "match", "n": n, "m": m}
    n = min(3500, int(math.exp(rng.uniform(0.0, math.log(3500)))))
    return {"what": "faces", "n": n, "pixels": rng.choice(["f32", "u8"]),
            "memory": rng.choice(["pageable", "pinned"]) if n <= 1200 else "pinned",
            "ctx": 256 if n <= 256 else rng.choice([256, 1024]),
            "order": "strict" if rng.random() < 0.2 else "contract"}


def _engine(ctx, order):
    key = (ctx, order)
    if key not in _engines:
        while len(_engines) >= 3:                    # the oldest goes; a state still using it keeps it open
            _engines.pop(next(iter(_engines)))
        with tempfile.TemporaryDirectory() as root:  # the library has copied the files by the time it returns
            e = ff.FastFace(synth.materialize(root, 0), cwd=root, max_batch=ctx)
        e.set_epilogue_mode(ff.EPILOGUE_STRICT if order == "strict" else ff.EPILOGUE_CONTRACT)
        _engines[key] = e
    return _engines[key]


def _array(shape, dtype, memory):
    if memory == "pinned":
        return torch.empty(shape, dtype=torch.uint8 if dtype == np.uint8 else torch.float32, pin_memory=True).numpy()
    return np.empty(shape, dtype)


def _embeddings(rng, count, people):
    """Embeddings as a recogniser gives them: a person's direction plus what differs between that person's pictures."""
    who = rng.integers(0, len(people), count)
    return people[who] + np.float32(0.6) * rng.standard_normal((count, ff.EMB_DIM), dtype=np.float32)


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["what"] == "match":
        people = rng.standard_normal((200, ff.EMB_DIM), dtype=np.float32)
        return {"case": case, "engine": _engine(256, "contract"), "a": _embeddings(rng, case["n"], people),
                "b": _embeddings(rng, case["m"], people)}
    shape = (case["n"],) + ff.FACE_SHAPE
    pixels = np.frombuffer(rng.bytes(case["n"] * PIXELS), np.uint8).reshape(shape)
    x = _array(shape, np.uint8 if case["pixels"] == "u8" else np.float32, case["memory"])
    if case["pixels"] == "u8":
        x[...] = pixels
    else:
        np.subtract(pixels, np.float32(127.5), out=x, dtype=np.float32)
        np.divide(x, np.float32(127.5), out=x)
    state = {"case": case, "engine": _engine(case["ctx"], case["order"]), "x": x}
    if case["memory"] == "pinned":
        state["out"] = _array((case["n"], ff.EMB_DIM), np.float32, "pinned")
    return state


def run(state):
    case, engine = state["case"], state["engine"]
    if case["what"] == "match":
        return engine.cos_sim_matrix(state["a"], state["b"])
    if case["memory"] == "pinned":                   # the pipeline's own buffers
        (engine.embed_into_u8 if case["pixels"] == "u8" else engine.embed_into)(state["x"], state["out"])
        return state["out"]
    if case["pixels"] == "u8":
        return engine.embed_batch_u8(state["x"])
    if case["n"] == 1:
        return engine.embed(state["x"])
    return engine.embed_batch(state["x"])


def work(case):
    n = case["n"]
    if case["what"] == "match":
        return {"bytes": 4 * (ff.EMB_DIM * (n + case["m"]) + n * case["m"]), "flops": 2 * ff.EMB_DIM * n * case["m"]}
    return {"bytes": n * (PIXELS * (1 if case["pixels"] == "u8" else 4) + 4 * ff.EMB_DIM) + WEIGHT_BYTES, "flops": OPS_PER_FACE * n}


def tolerance(case):
    """The library's contract is the reference's bits: integer accumulators, fp32 roundings in a stated order, float64
    sums in index order.  Every size, option and launch list gives the same embedding for the same face."""
    return "exact"
