"""Launches whose per-channel constants are kernel parameters: both sides of each line, with ragged last tile waves, give
the bytes of batch-8 calls.  On 148 SMs: the stem from 46 faces per launch (30 tiles of 98 a face for every CTA), the 56x56
residual + BN layers from 43 (8 tiles of 28 a face), the 28x28 ones from 43 per call (two tiles per CTA pair).  A call below
128 faces runs the stem, and for fp32 the 56x56 layers too, in two chunks of (n + 1) / 2 and n / 2 faces."""
import numpy as np
import pytest

import fastface_b200 as ff
from fastface_b200 import synth

pytestmark = pytest.mark.gpu
# 8-bit: stem 45 + 45 | 46 + 45 | 46 + 46 faces at 90 | 91 | 92; 56x56 and 28x28 at 42 | 43.  fp32: the same for the stem;
# 56x56 42 + 42 | 43 + 42 | 43 + 43 at 84 | 85 | 86.  128: chunks of 64
SIZES = (42, 43, 45, 47, 84, 85, 86, 90, 91, 92, 128)


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
