"""Layer-chain launches (runs of same-shape convolutions in one launch) beyond a single face: same bytes as one
launch per layer, and as the oracle."""
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
        if n <= 4:
            assert (launches < 30) == (flag == "1"), launches
    for mode in (ffo.CONTRACT, ffo.STRICT):
        want = oracle.forward(faces[sample], mode)
        for rep in range(3):
            assert np.array_equal(got["1", mode, rep], got["0", mode, rep]), f"mode {mode} rep {rep}"
            assert np.array_equal(got["1", mode, rep][sample], want), f"mode {mode} rep {rep}"
