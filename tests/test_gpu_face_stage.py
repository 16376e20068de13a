"""Stages as one launch, the 14x14 one with a CTA pair per face, 28x28, 14x14 and 7x7 with a cluster per face: same bytes as one launch
per layer, and as the oracle."""
import ctypes as C

import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth
from oracle import ffo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [34, 73, 74, 75, 147, 148, 149, 163, 164, 182, 190, 222, 223, 296, 297])
def test_stage_in_one_launch(built_lib, model_root, ffw4, oracle, monkeypatch, n):
    """One and two faces per pair, a round more, and what is left of a round in clusters (74 pairs on a B200): eager, captured and
    replayed, both epilogue orders.  The comparison is exact: integer accumulators and stated fp32 roundings."""
    faces = synth.faces(n, seed=700 + n)
    sample = sorted({0, n // 2, n - 1})
    got, launches = {}, {}
    for flag in ("1", "0"):
        monkeypatch.setenv("FF_FACE", flag)
        with ff.FastFace(ffw4, cwd=model_root, max_batch=297) as e:
            for mode in (ffo.CONTRACT, ffo.STRICT):
                e.set_epilogue_mode(mode)
                for rep in range(3 if flag == "1" else 1):
                    got[flag, mode, rep] = e.embed_batch(faces)
            launches[flag] = e.launches_per_forward
    # 26 layers of the 14x14 stage in one launch or two; in one, up to 66 faces the four 7x7 layers, from 49 to 74 the six 28x28 ones
    assert launches["0"] - launches["1"] - (3 if n <= 66 else 0) - (5 if 49 <= n <= 74 else 0) in (24, 25), launches
    for mode in (ffo.CONTRACT, ffo.STRICT):
        for rep in range(3):
            bad = np.flatnonzero((got["1", mode, rep] != got["0", mode, 0]).any(axis=1))
            assert bad.size == 0, f"mode {mode} rep {rep}: faces {bad[:16].tolist()}"
        assert np.array_equal(got["1", mode, 0][sample], oracle.forward(faces[sample], mode))


@pytest.mark.parametrize("max_batch,n", [(1, 1), (3, 1), (3, 2), (4, 4), (5, 1), (5, 5), (40, 2), (40, 14), (40, 15), (40, 16), (40, 17), (40, 20), (40, 21),
                                         (40, 32), (40, 33), (40, 34), (80, 35), (80, 65), (80, 66), (80, 67), (80, 48), (80, 49), (80, 74), (80, 75)])
def test_stages_in_clusters(built_lib, model_root, ffw4, oracle, monkeypatch, max_batch, n):
    """A cluster per face (7x7 also two faces a cluster), the forms' last faces on a B200 and one more: eager, captured and replayed, both epilogue orders,
    against one launch per layer (exact, as above)."""
    faces = synth.faces(n, seed=900 + n)
    got, launches = {}, {}
    for flag in ("1", "0"):
        monkeypatch.setenv("FF_FACE", flag)
        monkeypatch.setenv("FF_CHAIN", flag)
        with ff.FastFace(ffw4, cwd=model_root, max_batch=max_batch) as e:
            for mode in (ffo.CONTRACT, ffo.STRICT):
                e.set_epilogue_mode(mode)
                for rep in range(3 if flag == "1" else 1):
                    got[flag, mode, rep] = e.embed_batch(faces)
            launches[flag] = e.launches_per_forward
    # one launch for the 6 + 26 + 4 layers of the three stages
    if n <= 32:
        assert launches["0"] - launches["1"] == 5 + 25 + 3, launches
    for mode in (ffo.CONTRACT, ffo.STRICT):
        for rep in range(3):
            assert np.array_equal(got["1", mode, rep], got["0", mode, 0]), (mode, rep)
        assert np.array_equal(got["1", mode, 0][[0, n - 1]], oracle.forward(faces[[0, n - 1]], mode))


@pytest.mark.parametrize("n", [40, 80], ids=["one-face-a-pair", "two-faces-a-pair"])
def test_bounded_waits_run_out(built_lib, model_root, ffw4, oracle, n):
    """The timeout path, without faulting anything: the hook makes the first CTA of every pair leave out one step of its weights
    and limits every wait of that launch to two million cycles.  All must give up, meet at their pair's barrier and return; the
    call reports 1000 + the error word, and the same context then serves the same faces bit-exactly."""
    lib = ff.load_library()
    lib.ffcu_test_arm_chain_timeout.restype = None
    lib.ffcu_test_arm_chain_timeout.argtypes = [C.c_int, C.c_longlong]
    faces = synth.faces(n, seed=78)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=80) as e:
        want = e.embed_batch(faces)
    assert np.array_equal(want[:2], oracle.forward(faces[:2], ffo.CONTRACT))
    with ff.FastFace(ffw4, cwd=model_root, max_batch=80) as e:
        lib.ffcu_test_arm_chain_timeout(25, 2_000_000)          # second layer, or the second face's first
        with pytest.raises(RuntimeError) as ei:
            e.embed_batch(faces)
        assert "rc=1001" in str(ei.value) or "rc=1004" in str(ei.value), str(ei.value)
        for _ in range(4):
            assert np.array_equal(e.embed_batch(faces), want)


@pytest.mark.parametrize("n", [1, 17, 64, 80, 160, 296, 330], ids=["clusters-of-eight", "clusters-of-four", "two-faces-a-cluster", "a-pair-and-two-faces",
                                                                   "pairs-and-clusters", "two-rounds", "three-rounds"])
def test_a_late_loader_changes_nothing(built_lib, model_root, ffw4, oracle, n):
    """One CTA of each cluster loads its first input, and every byte table, several layers' time (a layer takes five to ten thousand
    cycles) after the others have theirs: neighbours' first results must not be overwritten by an input that lands after them, and
    nobody may lose count of the layers.  Exact: integer accumulators and stated fp32 roundings."""
    lib = ff.load_library()
    lib.ffcu_test_hold_stage_loader.restype = None
    lib.ffcu_test_hold_stage_loader.argtypes = [C.c_int, C.c_longlong]
    faces = synth.faces(n, seed=79)
    want = oracle.forward(faces[[0, n - 1]], ffo.CONTRACT)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=330) as e:
        lib.ffcu_test_hold_stage_loader(8, 40_000)              # a shape's first call runs eagerly
        held = e.embed_batch(faces)
        lib.ffcu_test_hold_stage_loader(0, 0)
        assert np.array_equal(held, e.embed_batch(faces))
    assert np.array_equal(held[[0, n - 1]], want)


@pytest.mark.parametrize("at", [0, 1], ids=["first-call", "while-captured"])
@pytest.mark.parametrize("refused", [1, 2, 1000], ids=["one", "two", "all"])
@pytest.mark.parametrize("n", [1, 17, 64, 160])
def test_refused_clusters(built_lib, model_root, ffw4, oracle, n, refused, at):
    """A device that cannot place a cluster: the call goes on with CTA pairs on 14x14 maps, one launch per layer on the others, one CTA per tile
    in the stride-2 convolutions, and does not ask again.  In the first (eager) call or in the one that is captured; exact, as above."""
    lib = ff.load_library()
    lib.ffcu_test_refuse_clusters.restype = None
    lib.ffcu_test_refuse_clusters.argtypes = [C.c_int]
    faces = synth.faces(n, seed=80)
    want = oracle.forward(faces[[0, n - 1]], ffo.CONTRACT)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=160) as e:
        before = e.embed_batch(faces) if at else None
        lib.ffcu_test_refuse_clusters(refused)
        try:
            got = [e.embed_batch(faces) for _ in range(4)]
        finally:
            lib.ffcu_test_refuse_clusters(0)
        launches = e.launches_per_forward
        got.append(e.embed_batch(faces))
    for g in got + ([before] if at else []):
        assert np.array_equal(g, got[0])
    assert np.array_equal(got[0][[0, n - 1]], want)
    if n <= 17 and refused == 1000:
        assert launches == 54 - 4 - 25                             # all 54 but the shortcuts' and the 14x14 stage's


def stage_layers(layers):
    """Map size -> its 3x3 stride-1 C -> C layers, C >= 128: those that a stage's launch takes."""
    out = {}
    for k, l in enumerate(layers):
        if l["kind"] == 1 and l["Kh"] == 3 and l["stride"] == 1 and l["Cin"] == l["Cout"] >= 128:
            out.setdefault(l["H"], []).append(k)
    return out


@pytest.mark.parametrize("n,shared", [(1, {28, 14, 7}), (17, {28, 14, 7}), (40, {14, 7}), (64, {28, 14, 7}), (160, {14})])
def test_layer_timing_follows_the_forward(built_lib, model_root, ffw4, n, shared):
    """bench_layers times the launches that a forward of n faces makes: a stage in one launch gives its layers equal shares, layers with
    a launch each have times of their own (six equal event times in a row do not happen), and no layer is left out."""
    faces = synth.faces(n, seed=81)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=160) as e:
        layers, ms = e.layers(), e.bench_layers(faces, 3)
        stages = stage_layers(layers)
        assert {h: len(k) for h, k in stages.items()} == {28: 6, 14: 26, 7: 4}
        assert {h for h, k in stages.items() if len({ms[i] for i in k}) == 1} == shared
        made = e.layer_launches()
        assert sum(m["layers"] for m in made) == len(layers)
        assert sum(m["single"] + m["pairs"] + m["clusters"] for m in made) == e.launches_per_forward
        assert {h for h, k in stages.items() if made[k[0]]["pairs"] + made[k[0]]["clusters"]} == shared
        assert made[stages[14][0]] == {"layers": 26, "single": 0, "pairs": int(n > 33), "clusters": int(n <= 33 or n == 160)}
        forward = e.bench_resident(faces, 20) / 20
        assert 0.6 * forward < sum(ms) / 3 < 2.0 * forward, (sum(ms) / 3, forward)


def test_layer_timing_with_refused_clusters(built_lib, model_root, ffw4):
    """Refused in the forward before the timing: the layers' own launches are timed, and the count returned is that of the layers.  A wait
    that ran out is an error below zero, not a count."""
    lib = ff.load_library()
    lib.ffcu_test_refuse_clusters.restype = None
    lib.ffcu_test_refuse_clusters.argtypes = [C.c_int]
    faces = synth.faces(64, seed=81)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=64) as e:
        lib.ffcu_test_refuse_clusters(1000)
        try:
            ms = e.bench_layers(faces, 3)
        finally:
            lib.ffcu_test_refuse_clusters(0)
        stages = stage_layers(e.layers())
        assert {h for h, k in stages.items() if len({ms[i] for i in k}) == 1} == {14}
        assert all(ms[i] > 0 for k in stages.values() for i in k)
    lib.ffcu_test_arm_chain_timeout.restype = None
    lib.ffcu_test_arm_chain_timeout.argtypes = [C.c_int, C.c_longlong]
    with ff.FastFace(ffw4, cwd=model_root, max_batch=64) as e:
        lib.ffcu_test_arm_chain_timeout(12, 2_000_000)
        with pytest.raises(RuntimeError) as ei:
            e.bench_layers(faces, 3)
        assert "rc=-1001" in str(ei.value) or "rc=-1004" in str(ei.value), str(ei.value)
