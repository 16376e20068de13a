"""Launches whose per-channel constants are kernel parameters (stem from 30 tiles per CTA, 56x56 residual + BN layers from 8):
the faces on both sides of each line, with a ragged last tile wave, give the bytes of batch-8 calls."""
import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth

pytestmark = pytest.mark.gpu
SIZES = (42, 43, 45, 46, 47, 90)


@pytest.mark.parametrize("mode", [ff.EPILOGUE_CONTRACT, ff.EPILOGUE_STRICT], ids=["contract", "strict"])
def test_both_sides_of_the_lines(built_lib, model_root, ffw4, mode):
    faces = synth.faces(max(SIZES), seed=900)
    px = np.random.default_rng(901).integers(0, 256, faces.shape, dtype=np.uint8)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=8) as e:
        e.set_epilogue_mode(mode)
        want = np.concatenate([e.embed_batch(faces[i:i + 8]) for i in range(0, len(faces), 8)])
        want8 = np.concatenate([e.embed_batch_u8(px[i:i + 8]) for i in range(0, len(px), 8)])
    with ff.FastFace(ffw4, cwd=model_root, max_batch=max(SIZES)) as e:
        e.set_epilogue_mode(mode)
        for n in SIZES:
            for _ in range(2):
                assert np.array_equal(e.embed_batch(faces[:n]), want[:n]), n
                assert np.array_equal(e.embed_batch_u8(px[:n]), want8[:n]), n
