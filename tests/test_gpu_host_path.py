"""Input and output paths of a call: pageable and page-locked memory, one stream or the pipeline, first layers in
chunks.  Every face must come out with the bytes a batch-8 call gives it."""
import ctypes as C

import numpy as np
import pytest

import fastface_b200 as ff

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
N = 300


@pytest.fixture(scope="module")
def data(built_lib, model_root, ffw4):
    px = np.random.default_rng(11).integers(0, 256, (N,) + ff.FACE_SHAPE, dtype=np.uint8)
    f32 = ((px.astype(np.float32) - np.float32(127.5)) / np.float32(127.5)).astype(np.float32)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=8) as e:
        want = {m: np.concatenate([(e.set_epilogue_mode(m), e.embed_batch(f32[i:i + 8]))[1] for i in range(0, N, 8)])
                for m in (ff.EPILOGUE_STRICT, ff.EPILOGUE_CONTRACT)}
    return px, f32, want


def pinned(a):
    t = torch.empty(a.shape, dtype=torch.uint8 if a.dtype == np.uint8 else torch.float32, pin_memory=True).numpy()
    t[...] = a
    return t


# around the smallest chunked step (40), two and more full chunks (128 on), a last chunk of one face (129), several steps of
# a context with a ragged last one, a chunked step after unchunked ones
@pytest.mark.parametrize("max_batch,sizes", [(300, (39, 40, 41, 63, 127, 128, 129, 200, 300)), (64, (40, 64, 65, 150, 300)), (16, (1, 16, 17, 100)),
                                             (1, (1, 3))])
@pytest.mark.parametrize("u8", [False, True], ids=["f32", "u8"])
def test_call_sizes_and_memory_kinds(data, model_root, ffw4, max_batch, sizes, u8):
    px, f32, want = data
    src = px if u8 else f32
    with ff.FastFace(ffw4, cwd=model_root, max_batch=max_batch) as e:
        run = e.embed_into_u8 if u8 else e.embed_into
        for mode in (ff.EPILOGUE_CONTRACT, ff.EPILOGUE_STRICT):
            e.set_epilogue_mode(mode)
            for rep in range(3):                       # eager, captured, replayed
                for n in sizes:
                    o = (7 * n + rep) % (N - n + 1)
                    for pin_in in (False, True):
                        for pin_out in (False, True):
                            x = pinned(src[o:o + n]) if pin_in else src[o:o + n]
                            out = pinned(np.full((n, 512), 9, np.float32)) if pin_out else np.full((n, 512), 9, np.float32)
                            run(x, out)
                            assert np.array_equal(out, want[mode][o:o + n]), (mode, rep, n, pin_in, pin_out)


def test_unaligned_and_interleaved_calls(data, model_root, ffw4):
    """Sources and destinations at odd addresses, small and large calls in turn (one stream <-> pipeline)."""
    px, f32, want = data
    want = want[ff.EPILOGUE_CONTRACT]
    rng = np.random.default_rng(12)
    raw = np.empty(N * ff.FACE_NELEMS + 3, np.uint8)
    raw[3:] = px.reshape(-1)
    odd = raw[3:].reshape(px.shape)
    with ff.FastFace(ffw4, cwd=model_root, max_batch=100) as e:
        for _ in range(60):
            n = int(rng.choice([1, 2, 5, 20, 39, 40, 90, 100, 130, 230]))
            o = int(rng.integers(0, N - n + 1))
            out = np.empty(n * 512 + 1, np.float32)[1:].reshape(n, 512)
            if rng.random() < 0.5:
                e.embed_into_u8(odd[o:o + n], out)
            else:
                e.embed_into(f32[o:o + n], out)
            assert np.array_equal(out, want[o:o + n]), (n, o)


@pytest.mark.parametrize("denied", [1, 2, 3], ids=["no-ring", "one-output-slot", "nothing"])
def test_hosts_without_memory_to_lock(data, model_root, ffw4, denied):
    """Page-locked staging is not needed: where the host has none to give, the context is made all the same and
    pageable calls go through the driver's own staging."""
    px, f32, want = data
    want = want[ff.EPILOGUE_CONTRACT]
    lib = ff.load_library()
    lib.ffcu_test_deny_staging.restype = None
    lib.ffcu_test_deny_staging.argtypes = [C.c_int]
    lib.ffcu_test_deny_staging(denied)                 # the ring, then the two output slots
    try:
        e = ff.FastFace(ffw4, cwd=model_root, max_batch=130)
    finally:
        lib.ffcu_test_deny_staging(0)
    with e:
        for rep in range(3):
            for n in (1, 39, 40, 129, 300):
                o = (11 * n + rep) % (N - n + 1)
                for src, run in ((f32, e.embed_into), (px, e.embed_into_u8)):
                    for pin_in in (False, True):
                        out = np.full((n, 512), 9, np.float32)
                        run(pinned(src[o:o + n]) if pin_in else src[o:o + n], out)
                        assert np.array_equal(out, want[o:o + n]), (rep, n)


def test_launch_count_does_not_depend_on_chunks(data, model_root, ffw4):
    """The reported launches are those a face goes through: the same resident, in one piece and in chunks, a last chunk
    of a single face included (129)."""
    px, f32, _ = data
    with ff.FastFace(ffw4, cwd=model_root, max_batch=N) as e:
        for n in (39, 40, 127, 128, 129, 256):
            e.bench_resident(f32[:n], iters=1)
            whole = e.launches_per_forward
            for _ in range(3):
                e.embed_batch_u8(px[:n])
                assert e.launches_per_forward == whole, n
                e.embed_batch(f32[:n])
                assert e.launches_per_forward == whole, n
