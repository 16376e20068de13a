"""The device context's own calls (include/ff_cuda.h): submits that nobody waits for."""
import ctypes as C
import os

import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth

pytestmark = pytest.mark.gpu


class Plan(C.Structure):                     # ff_plan (csrc/host/ff_plan.h)
    _fields_ = [("n_layers", C.c_int), ("layers", C.POINTER(ff.FfcuLayer)), ("n_bufs", C.c_int), ("bytes_per_face", C.c_size_t),
                ("pool", C.c_void_p), ("pool_n", C.c_int), ("pool_cap", C.c_int)]


@pytest.fixture
def context(built_lib, model_root, ffw4):
    L = ff.load_library()
    model, plan = C.create_string_buffer(1 << 20), Plan()          # ff_model: far smaller
    root = os.path.join(model_root, "models")
    assert L.ff_model_load_ffw4(model, ffw4.encode()) == 0
    assert L.ff_model_load_opsc(model, os.path.join(root, "op_scales.bin").encode()) == 0
    assert L.ff_model_load_opsc2(model, os.path.join(root, "op_scales_v2.bin").encode()) == 0
    assert L.ff_plan_build(C.byref(plan), model) == 0
    L.ffcu_create.restype = C.c_void_p
    L.ffcu_create.argtypes = [C.c_int, C.c_int, C.c_int, C.c_size_t]
    L.ffcu_add_layer.argtypes = [C.c_void_p, C.POINTER(ff.FfcuLayer)]
    L.ffcu_finalize.argtypes = [C.c_void_p]
    L.ffcu_set_mode.argtypes = [C.c_void_p, C.c_int]
    L.ffcu_submit.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    L.ffcu_wait.argtypes = [C.c_void_p]
    L.ffcu_destroy.restype = None
    L.ffcu_destroy.argtypes = [C.c_void_p]
    c = L.ffcu_create(0, 48, plan.n_bufs, plan.bytes_per_face)
    assert c
    for k in range(plan.n_layers):
        assert L.ffcu_add_layer(c, C.byref(plan.layers[k])) >= 0
    assert L.ffcu_finalize(c) == 0
    L.ffcu_set_mode(c, ff.EPILOGUE_CONTRACT)
    L.ff_plan_free.restype = None
    L.ff_plan_free(C.byref(plan))
    L.ff_model_free.restype = None
    L.ff_model_free(model)
    return L, c


@pytest.mark.parametrize("sizes", [(1,), (5, 3), (48,), (48, 40, 7)], ids=str)
def test_outputs_arrive_without_a_wait(context, model_root, ffw4, sizes):
    """Outputs to ordinary memory pass through the context's own on their way: destroying the context hands over
    what is still there, as it always completed the copies under way."""
    L, c = context
    faces = [synth.faces(n, seed=60 + n) for n in sizes]
    outs = [np.full((n, 512), 9, np.float32) for n in sizes]
    for x, out in zip(faces, outs):
        assert L.ffcu_submit(c, x.ctypes.data, len(x), out.ctypes.data) == 0
    L.ffcu_destroy(c)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=8) as e:
        for x, out in zip(faces, outs):
            assert np.array_equal(out, np.concatenate([e.embed_batch(x[i:i + 8]) for i in range(0, len(x), 8)]))
