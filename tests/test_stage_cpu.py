"""Which runs of layers may go through the network face by face with only their last tensors in memory
(csrc/host/ff_plan.c, ff_plan_stage).  Checked by running launch lists on tags: every buffer remembers which layer's result
(or which layer's fused BN) it holds."""
import ctypes as C
import os

import numpy as np
import pytest

import fastface_b200 as ff
from test_head_cpu import CONV, Plan, layer


@pytest.fixture(scope="module")
def lib(built_lib):
    L = ff.load_library()
    L.ff_plan_stage.restype = C.c_int
    L.ff_plan_stage.argtypes = [C.POINTER(ff.FfcuLayer), C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int)]
    return L


def stage(lib, layers, first, count):
    a, frm = (ff.FfcuLayer * len(layers))(*layers), (C.c_int * count)()
    return list(frm) if lib.ff_plan_stage(a, len(layers), first, count, frm) else None


def reads(layers, first=0, count=0, frm=None):
    """What each layer reads, source and residual.  The run [first, first + count) as the stage's kernel works: each of its layers
    is handed the one before's result, residuals come from a buffer or from the one result that is kept, and only the last
    layer writes buffers."""
    mem, seen, kept = {}, [], None
    for k, l in enumerate(layers):
        inside = first <= k < first + count
        src, res = mem.get(l.src_buf), mem.get(l.res_buf)
        if inside and k > first:
            src = (k - 1, layers[k - 1].bn2_dst_buf >= 0)
        if inside and l.res_buf >= 0 and frm[k - first] >= 0:
            res = kept
        if inside and l.res_buf >= 0:
            kept = (k, False)
        seen.append((src, res if l.res_buf >= 0 else None))
        if not inside or k == first + count - 1:
            mem[l.dst_buf] = (k, False)
            if l.bn2_dst_buf >= 0:
                mem[l.bn2_dst_buf] = (k, True)
    return seen


def test_networks_own_plan(lib, model_root, ffw4):
    """The 26 layers of the 14 x 14 stage: each second one adds what the one two before it gave, the first of them the block's
    input; taking the stage without its last layer would lose a tensor."""
    model, plan = C.create_string_buffer(1 << 16), Plan()
    root = os.path.join(model_root, "models")
    assert lib.ff_model_load_ffw4(model, ffw4.encode()) == 0
    assert lib.ff_model_load_opsc(model, os.path.join(root, "op_scales.bin").encode()) == 0
    assert lib.ff_model_load_opsc2(model, os.path.join(root, "op_scales_v2.bin").encode()) == 0
    assert lib.ff_plan_build(C.byref(plan), model) == 0
    layers = [ff.FfcuLayer.from_buffer_copy(plan.layers[k]) for k in range(plan.n_layers)]
    lib.ff_plan_free(C.byref(plan))
    lib.ff_model_free(model)
    run = [k for k, l in enumerate(layers) if l.kind == CONV and l.H == 14 and l.Cin == l.Cout == 256 and l.stride == 1]
    first, count = run[0], len(run)
    assert count == 26 and run == list(range(first, first + 26))
    frm = stage(lib, layers, first, count)
    assert frm == [-1 if i % 2 == 0 or i == 1 else i - 2 for i in range(26)]
    assert reads(layers, first, count, frm) == reads(layers)
    assert stage(lib, layers, first, count - 1) is None


def test_rule_over_random_plans(lib):
    """Where the rule says yes, every layer reads what it reads layer by layer; and it does not say no to everything."""
    rng = np.random.default_rng(1)
    yes = no = 0
    for _ in range(2000):
        count = int(rng.integers(2, 6))
        layers = [layer(-1, 0, 1), layer(0, 1, 1)]
        first, src = 2, int(rng.integers(0, 2))
        for i in range(count):
            dst, bn2 = (int(b) for b in rng.permutation([b for b in range(6) if b != src])[:2])
            bn2 = bn2 if rng.random() < 0.5 else -1
            have = {0, 1} | {l.dst_buf for l in layers} | {l.bn2_dst_buf for l in layers} - {-1}
            res = int(rng.choice([b for b in have if b not in (dst, bn2)])) if rng.random() < 0.5 else -1
            layers.append(layer(src, dst, 1, res, bn2))
            src = bn2 if bn2 >= 0 else dst
        held = [b for b in range(6) if any(b in (l.dst_buf, l.bn2_dst_buf) for l in layers)]
        for _ in range(3):
            a, r = (int(rng.choice(held)) for _ in range(2))
            dst = next(b for b in range(8) if b not in (a, r) and (b > 5 or rng.random() < 0.4))
            layers.append(layer(a, dst, 1, r if rng.random() < 0.5 else -1))
            held = sorted(set(held) | {dst})
        frm = stage(lib, layers, first, count)
        if frm is None:
            no += 1
            continue
        yes += 1
        assert reads(layers, first, count, frm) == reads(layers), [(l.src_buf, l.res_buf, l.dst_buf, l.bn2_dst_buf) for l in layers]
    assert yes > 100 and no > 100
