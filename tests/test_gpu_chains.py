"""Stages of a small call in one launch each (runs of same-shape convolutions, conv_tc_stage.cu): same bytes as one
launch per layer, and as the oracle."""
import ctypes as C
import os
import threading
import time

import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth
from oracle import ffo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4, 15, 16, 17, 24, 32, 33, 34, 35, 36, 37, 38])
def test_small_batch_layer_chains(built_lib, model_root, ffw4, oracle, monkeypatch, n):
    """One cluster per face, for as many faces as the device holds clusters (of eight CTAs: 15-18, of four: 32-37, by
    its GPC sizes; beyond that CTA pairs on 14x14 maps, two faces a cluster on 7x7 ones): eager, captured and replayed, both epilogue orders.  The comparison is exact: integer accumulators and stated fp32 roundings."""
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
    cluster of the next stage launch leave out one step of its weights and limits every wait of that launch to two million
    cycles.  All of them must give up, meet at their cluster's barrier and return; the call reports 1000 + the error word, and
    the same context then serves the same faces bit-exactly (eager, captured, replayed)."""
    lib = ff.load_library()
    lib.ffcu_test_arm_chain_timeout.restype = None
    lib.ffcu_test_arm_chain_timeout.argtypes = [C.c_int, C.c_longlong]
    faces = synth.faces(n, seed=77)
    want = oracle.forward(faces, ffo.CONTRACT)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=40) as e:
        lib.ffcu_test_arm_chain_timeout(12, 2_000_000)          # second layer; a shape's first call runs eagerly
        with pytest.raises(RuntimeError) as ei:
            e.embed_batch(faces)
        assert "rc=1001" in str(ei.value) or "rc=1004" in str(ei.value), str(ei.value)
        for _ in range(4):
            assert np.array_equal(e.embed_batch(faces), want)
        assert e.launches_per_forward < 30


def test_contexts_share_the_device(built_lib, model_root, ffw4):
    """A stage keeps eight SMs per face for 90 us; the kernels queued behind it must not keep the others waiting with them.
    Four threads with a context each get 3.5 times one thread's single-face rate on an idle machine, and got 1.5 times with a
    successor launched at the stage's start."""
    if len(os.sched_getaffinity(0)) < 6:
        pytest.skip("needs a CPU for each of the calling threads")
    face = synth.faces(1, seed=8)[0]
    engines = [ff.FastFace(ffw4, cwd=model_root, max_batch=1) for _ in range(4)]
    want = [e.embed(face) for e in engines for _ in range(4)][0]

    def rate(k):
        counts, start = [0] * k, threading.Barrier(k + 1)

        def work(i):
            start.wait()
            while time.perf_counter() < until:
                got = engines[i].embed(face)
                counts[i] += 1
            assert np.array_equal(got, want)

        ts = [threading.Thread(target=work, args=(i,)) for i in range(k)]
        until = time.perf_counter() + 0.3
        [t.start() for t in ts]
        start.wait()
        [t.join() for t in ts]
        return sum(counts)

    ratios = []
    for _ in range(5):                                     # the best of five: other work on the host only slows it down
        one = rate(1)
        ratios.append(rate(4) / one)
        if ratios[-1] >= 2.2:
            break
    [e.close() for e in engines]
    assert max(ratios) >= 2.2, ratios
