"""Kernels whose K loop several CTAs share: the FC at the edges of its tiles (128 outputs x up to 256 faces, faces in steps of 16),
and the stride-2 convolutions of small batches."""
import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth
from oracle import ffo

pytestmark = pytest.mark.gpu

SIZES = [3, 4, 15, 16, 17, 47, 49, 112, 113, 240, 241, 256, 257, 272, 273, 289, 511, 512, 513, 529]


@pytest.fixture(scope="module")
def want(built_lib, model_root, ffw4):
    """Two faces at a time: the CUDA-core FC.  Both forms add the same integers, so the comparison is exact."""
    faces = synth.faces(max(SIZES), seed=73)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=2) as e:
        out = {}
        for mode in (ffo.CONTRACT, ffo.STRICT):
            e.set_epilogue_mode(mode)
            out[mode] = e.embed_batch(faces)
    return faces, out


@pytest.mark.parametrize("room", [0, 100], ids=["full-context", "larger-context"])
def test_tiles_of_faces(built_lib, model_root, ffw4, want, room):
    """Whole and ragged tiles, one to three of them, calls in between that leave other faces in the buffers; twice each, so that
    sums and tickets are seen to be left clean."""
    faces, ref = want
    with ff.FastFace(ffw4, cwd=model_root, max_batch=max(SIZES) + room) as e:
        for n in SIZES + SIZES[::-1]:
            mode = (ffo.CONTRACT, ffo.STRICT)[n & 1]
            e.set_epilogue_mode(mode)
            for start in (0, max(SIZES) - n):
                got = e.embed_batch(faces[start:start + n])
                bad = np.flatnonzero((got != ref[mode][start:start + n]).any(axis=1))
                assert bad.size == 0, f"{n} faces from {start}, mode {mode}: {bad[:8].tolist()} differ"


@pytest.mark.parametrize("n", [1, 2, 4, 7, 13, 18, 19, 20])
def test_stride2_pairs_of_ctas(built_lib, model_root, ffw4, oracle, monkeypatch, n):
    """A stride-2 convolution and its shortcut by two CTAs per tile, up to the last batch at which the device holds both (on a B200 18
    faces on 14 x 14 -> 7 x 7 maps) and beyond, against two launches with whole K loops (exact: sums of integers)."""
    faces = synth.faces(n, seed=90 + n)
    got = {}
    for flag in ("1", "0"):
        monkeypatch.setenv("FF_FUSE_SC", flag)
        with ff.FastFace(ffw4, cwd=model_root, max_batch=n) as e:
            for mode in (ffo.CONTRACT, ffo.STRICT):
                e.set_epilogue_mode(mode)
                for rep in range(3 if flag == "1" else 1):
                    got[flag, mode, rep] = e.embed_batch(faces)
    for mode in (ffo.CONTRACT, ffo.STRICT):
        for rep in range(3):
            assert np.array_equal(got["1", mode, rep], got["0", mode, 0]), (mode, rep)
        assert np.array_equal(got["1", mode, 0][[0, n - 1]], oracle.forward(faces[[0, n - 1]], mode))
