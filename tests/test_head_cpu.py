"""First layers in chunks of faces (csrc/host/ff_plan.c, ff_plan_head_end): no chunk may write over what an earlier chunk
has left for the rest of the network.  Checked by running launch lists on tags instead of activations: every unit of
memory remembers which layer wrote it for which face."""
import ctypes as C
import os

import numpy as np
import pytest

import fastface_b200 as ff

QUANT, CONV = 0, 1


class Plan(C.Structure):                     # ff_plan (csrc/host/ff_plan.h)
    _fields_ = [("n_layers", C.c_int), ("layers", C.POINTER(ff.FfcuLayer)), ("n_bufs", C.c_int), ("bytes_per_face", C.c_size_t),
                ("pool", C.c_void_p), ("pool_n", C.c_int), ("pool_cap", C.c_int)]


@pytest.fixture(scope="module")
def lib(built_lib):
    L = ff.load_library()
    L.ff_plan_head_end.restype = C.c_int
    L.ff_plan_head_end.argtypes = [C.POINTER(ff.FfcuLayer), C.c_int, C.c_int, C.c_char_p]
    return L


def layer(src, dst, size, res=-1, bn2=-1, kind=CONV):
    """A layer that writes `size` units a face (as one row of `size` channels)."""
    return ff.FfcuLayer(kind=kind, src_buf=src, dst_buf=dst, res_buf=res, bn2_dst_buf=bn2, Ho=1, Wo=1, Cout=size)


def survives(layers, end, unit, faces, chunk):
    """Layers [1, end) chunk by chunk, then the rest: does every layer read what it reads in one piece?"""
    sizes = [l.Ho * l.Wo * l.Cout // unit for l in layers]
    room = faces * max(sizes)

    def run(head):
        mem = np.full((8, room, 2), -1, np.int64)          # [buffer][unit of memory]: writing layer, face
        size_in = [0] * 8
        seen = [[None] * faces for _ in layers]

        def step(k, f0, f1):
            l = layers[k]
            for f in range(f0, f1):
                seen[k][f] = [mem[b, f * n:(f + 1) * n].copy() for b, n in inputs[k] if b >= 0]
            for b in (l.dst_buf, l.bn2_dst_buf):
                if b >= 0:
                    for f in range(f0, f1):
                        mem[b, f * sizes[k]:(f + 1) * sizes[k]] = (k, f)

        inputs = []                                        # per layer: (buffer, units a face of the tensor it finds there)
        for k, l in enumerate(layers):
            inputs.append([(b, size_in[b]) for b in (l.src_buf, l.res_buf) if b >= 0])
            for b in (l.dst_buf, l.bn2_dst_buf):
                if b >= 0:
                    size_in[b] = sizes[k]
        for f0 in range(0, faces, head):
            for k in range(1, end):
                step(k, f0, min(f0 + head, faces))
        for k in range(end, len(layers)):
            step(k, 0, faces)
        return seen

    whole, parts = run(faces), run(chunk)
    return all(np.array_equal(x, y) for k in range(1, len(layers)) for f in range(faces) for x, y in zip(whole[k][f], parts[k][f]))


def head_end(lib, layers, end, with_next=None):
    a = (ff.FfcuLayer * len(layers))(*layers)
    return lib.ff_plan_head_end(a, len(layers), end, bytes(with_next or [0] * len(layers)))


def test_networks_own_plan(lib, model_root, ffw4):
    """The leading layers with 64 input channels are a head up to the last one of the 56 x 56 stage (layer 9 writes a buffer
    at twice the bytes a face that layer 7 did), and chunks leave the rest as it is."""
    model, plan = C.create_string_buffer(1 << 16), Plan()
    root = os.path.join(model_root, "models")
    assert lib.ff_model_load_ffw4(model, ffw4.encode()) == 0
    assert lib.ff_model_load_opsc(model, os.path.join(root, "op_scales.bin").encode()) == 0
    assert lib.ff_model_load_opsc2(model, os.path.join(root, "op_scales_v2.bin").encode()) == 0
    assert lib.ff_plan_build(C.byref(plan), model) == 0
    layers = [ff.FfcuLayer.from_buffer_copy(plan.layers[k]) for k in range(plan.n_layers)]
    lib.ff_plan_free(C.byref(plan))
    lib.ff_model_free(model)
    end = 2
    while layers[end].kind == CONV and layers[end].Cin_pad == 64:
        end += 1
    pairs = [int(a.kind == CONV and a.Kh == 3 and a.stride == 2 and b.Kh == 1 and b.stride == 2) for a, b in zip(layers, layers[1:])] + [0]
    got = head_end(lib, layers, end, pairs)
    assert got == 9 and end == 10 and layers[8].H == 56 and not pairs[got - 1]
    layers[1].src_buf = -1                                 # the stem of a head reads the input itself
    unit = 32 * 49                                         # divides every activation tensor of the network
    assert survives(layers[:-1], got, unit, 5, 2) and survives(layers[:-1], got, unit, 4, 3)
    assert not survives(layers[:-1], end, unit, 5, 2)


def test_rule_gives_way(lib):
    """A small tensor before a large one in the same buffer: chunk 1 of the small one would lie where chunk 0's large one does."""
    grow = [layer(-1, 0, 1, kind=QUANT), layer(-1, 1, 4), layer(1, 2, 2), layer(2, 3, 4), layer(3, 2, 8), layer(2, 1, 4)]
    assert not survives(grow, 5, 1, 5, 2) and survives(grow, 4, 1, 5, 2)
    assert head_end(lib, grow, 5) == 4
    shrink = [layer(-1, 0, 1, kind=QUANT), layer(-1, 1, 8), layer(1, 2, 4), layer(2, 1, 4), layer(1, 3, 2), layer(3, 1, 2)]
    assert head_end(lib, shrink, 5) == 5 and survives(shrink, 5, 1, 5, 2)
    assert head_end(lib, shrink, 4, [0, 0, 0, 1, 0, 0]) == 3          # layers 3 and 4 are one launch
    assert head_end(lib, shrink, 2) == 2


def test_rule_over_random_plans(lib):
    rng = np.random.default_rng(0)
    longer = cut = 0
    for _ in range(400):
        n = int(rng.integers(4, 9))
        layers = [layer(-1, 0, 1, kind=QUANT), layer(-1, 0, 4)]
        written = {0}
        for k in range(2, n):
            src = int(rng.choice(sorted(written)))
            dst, bn2 = (int(b) for b in rng.permutation(4)[:2])
            bn2 = bn2 if rng.random() < 0.3 else -1
            res = int(rng.choice(sorted(written))) if rng.random() < 0.3 else -1
            if {src, res} & {dst, bn2} - {-1}:
                dst, bn2 = next(b for b in range(6) if b not in (src, res)), -1
            layers.append(layer(src, dst, int(rng.choice([1, 2, 4])), res, bn2))
            written |= {dst, bn2} - {-1}
        got = head_end(lib, layers, n - 1)
        assert 2 <= got <= n - 1
        assert survives(layers, got, 1, 5, 2), [(l.src_buf, l.res_buf, l.dst_buf, l.bn2_dst_buf, l.Cout) for l in layers]
        longer += got > 2
        cut += got < n - 1
    assert longer > 50 and cut > 50
