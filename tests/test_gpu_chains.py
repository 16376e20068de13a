"""Layer-chain launches (runs of same-shape convolutions in one launch) beyond a single face: same bytes as one
launch per layer, and as the oracle."""
import ctypes as C

import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth
from oracle import ffo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4, 15, 16, 17, 24, 32, 33, 34, 35, 36, 37, 38])
def test_small_batch_layer_chains(built_lib, model_root, ffw4, oracle, monkeypatch, n):
    """One cluster per face, for as many faces as the device holds clusters (of eight CTAs: 15-18, of four: 32-37, by
    its GPC sizes; beyond that one launch per layer): eager, captured and replayed, both epilogue orders.  The comparison is exact: integer accumulators and stated fp32 roundings."""
    faces = synth.faces(n, seed=500 + n)
    sample = sorted({0, n // 2, n - 1})
    got = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("FF_CHAIN", flag)
        with ff.FastFace(ffw4, cwd=model_root, max_batch=40) as e:
            for mode in (ffo.CONTRACT, ffo.STRICT):
                e.set_epilogue_mode(mode)
                for rep in range(3):
                    got[flag, mode, rep] = e.embed_batch(faces)
            launches = e.launches_per_forward
        if n <= 24:        # 24 clusters of four: far below what a B200 holds (15-18 of eight up to 15 faces, 32-37 of four)
            assert (launches < 30) == (flag == "1"), launches
    for mode in (ffo.CONTRACT, ffo.STRICT):
        want = oracle.forward(faces[sample], mode)
        for rep in range(3):
            assert np.array_equal(got["1", mode, rep], got["0", mode, rep]), f"mode {mode} rep {rep}"
            assert np.array_equal(got["1", mode, rep][sample], want), f"mode {mode} rep {rep}"


@pytest.mark.parametrize("n", [8, 20], ids=["clusters-of-eight", "clusters-of-four"])
def test_bounded_waits_run_out_with_several_clusters(built_lib, model_root, ffw4, oracle, n):
    """The timeout path with a cluster per face, without faulting anything: the hook makes the first CTA of every
    cluster of the next chain launch leave out one step of its weights and limits every wait of that launch to two million
    cycles.  All of them must give up, meet at their cluster's barrier and return; the call reports 1000 + the error word, and
    the same context then serves the same faces bit-exactly (eager, captured, replayed)."""
    lib = ff.load_library()
    lib.ffcu_test_arm_chain_timeout.restype = None
    lib.ffcu_test_arm_chain_timeout.argtypes = [C.c_int, C.c_longlong]
    faces = synth.faces(n, seed=77)
    want = oracle.forward(faces, ffo.CONTRACT)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=40) as e:
        lib.ffcu_test_arm_chain_timeout(12, 2_000_000)          # layer 1, fourth tap; a shape's first call runs eagerly
        with pytest.raises(RuntimeError) as ei:
            e.embed_batch(faces)
        assert "rc=1001" in str(ei.value) or "rc=1004" in str(ei.value), str(ei.value)
        for _ in range(4):
            assert np.array_equal(e.embed_batch(faces), want)
        assert e.launches_per_forward < 30
