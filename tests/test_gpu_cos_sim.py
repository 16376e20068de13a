"""Similarity matrix at the edges of its tiles and slices: the bits of fastface_cos_sim for every pair looked at."""
import ctypes as C
import threading

import numpy as np
import pytest

import fastface_b200 as ff

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(built_lib, model_root, ffw4):
    with ff.FastFace(ffw4, cwd=model_root, max_batch=2) as e:
        yield e


def check(got, a, b, rng, count=400):
    n, m = len(a), len(b)
    assert got.shape == (n, m)
    edge_i = [i for i in (0, 15, 16, 63, 64, n - 65, n - 2, n - 1, 2047, 2048) if 0 <= i < n]
    edge_j = [j for j in (0, 63, 64, 65, m - 66, m - 2, m - 1, 4095, 4096) if 0 <= j < m]
    pairs = [(i, j) for i in edge_i for j in edge_j]
    pairs += [(int(rng.integers(n)), int(rng.integers(m))) for _ in range(count)]
    want = np.array([ff.FastFace.cos_sim(a[i], b[j]) for i, j in pairs], np.float32)
    have = np.array([got[i, j] for i, j in pairs], np.float32)
    same = (have.view(np.uint32) == want.view(np.uint32)) | (np.isnan(have) & np.isnan(want))
    assert same.all(), [pairs[k] for k in np.flatnonzero(~same)[:5]]


# 16- and 64-row blocks (32 | 33 rows, and 64-row blocks only where they fill half the SMs), ragged last tiles, one
# slice and several of 2048 x 4096
@pytest.mark.parametrize("n,m", [(1, 1), (1, 4097), (15, 65), (17, 64), (32, 4736), (33, 4737), (33, 100), (64, 4736), (65, 4800),
                                 (1000, 333), (2049, 130), (70, 8193), (2049, 4097)])
def test_matrix_edges(engine, n, m):
    rng = np.random.default_rng(n * 7919 + m)
    a = rng.standard_normal((n, 512), dtype=np.float32)
    b = rng.standard_normal((m, 512), dtype=np.float32) * np.float32(7.0)
    b[m // 2] = 0
    a[n - 1] *= np.float32(1e-30)
    check(engine.cos_sim_matrix(a, b), a, b, rng)


# each tile (16, 32 and 64 rows and columns a block) at its edges, one row or column more or less than whole tiles included;
# 148 SMs change tile between 128 x 500 and 128 x 1000, between 256 x 1000 and 512 x 1000, and at few rows by columns
@pytest.mark.parametrize("n,m", [(1, 15), (16, 16), (17, 17), (15, 2369), (1, 10001), (16, 9999), (128, 500), (128, 1000), (95, 1023),
                                 (97, 1025), (256, 1000), (512, 1000), (511, 1023), (513, 1025), (1024, 300), (64, 10000)])
def test_matrix_tiles(engine, n, m):
    rng = np.random.default_rng(n * 104729 + m)
    a = rng.standard_normal((n, 512), dtype=np.float32)
    b = rng.standard_normal((m, 512), dtype=np.float32)
    a[n // 2] = 0
    b[0] = np.float32(1e-30) * b[0]
    got = engine.cos_sim_matrix(a, b)
    check(got, a, b, rng)
    # every output: two float64 evaluations of a sum of 512 terms differ by at most 1024 * 2^-53 of the norms' product
    # (Cauchy-Schwarz), far below the half unit of the float32 result (2^-25 for |value| <= 1)
    x, y = a.astype(np.float64), b.astype(np.float64)
    nx, ny = np.sqrt((x * x).sum(1)), np.sqrt((y * y).sum(1))
    want = np.divide(x @ y.T, np.outer(nx, ny), out=np.zeros((n, m)), where=np.outer(nx, ny) != 0)
    assert np.abs(got - want).max() <= 2.0 ** -25 + 1e-12


def test_matrix_special_values(engine):
    rng = np.random.default_rng(3)
    a = rng.standard_normal((20, 512), dtype=np.float32)
    b = rng.standard_normal((70, 512), dtype=np.float32)
    a[1, 5], a[2, 6], a[3, 7] = np.inf, -np.inf, np.nan
    a[4] = np.float32(1e-45)            # denormal: the squared norm is representable in float64
    a[5] = np.float32(3e38)
    a[6] = np.float32(-0.0)
    b[1, 5], b[2] = np.nan, 0
    check(engine.cos_sim_matrix(a, b), a, b, rng, 1400)


def test_matrix_from_several_threads(engine):
    """Calls that overlap on one context (also beside an embedding call) each give their own matrix."""
    rng = np.random.default_rng(4)
    sets = [(rng.standard_normal((40 + 100 * k, 512), dtype=np.float32), rng.standard_normal((300 - 50 * k, 512), dtype=np.float32))
            for k in range(4)]
    want = [engine.cos_sim_matrix(a, b) for a, b in sets]
    face = rng.uniform(-1, 1, ff.FACE_SHAPE).astype(np.float32)
    emb = engine.embed(face)
    bad = []

    def work(k):
        for _ in range(20):
            if not np.array_equal(engine.cos_sim_matrix(*sets[k]).view(np.uint32), want[k].view(np.uint32)):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    for _ in range(20):
        if not np.array_equal(engine.embed(face), emb):
            bad.append("embed")
    [t.join() for t in ts]
    assert not bad


@pytest.mark.parametrize("n,m,over", [(500, 5000, "b"), (2500, 520, "a"), (300, 600, "b"), (2048, 1400, "a"), (2048, 4096, "b")])
def test_matrix_written_over_an_input(engine, n, m, over):
    """A result that takes the place of an input, also where the matrix goes in slices: the inputs are read first."""
    rng = np.random.default_rng(n + m)
    a = rng.standard_normal((n, 512), dtype=np.float32)
    b = rng.standard_normal((m, 512), dtype=np.float32)
    want = engine.cos_sim_matrix(a, b)
    src = a if over == "a" else b
    shared = np.empty(max(n * m, src.size), np.float32)
    shared[:src.size] = src.reshape(-1)
    pa, pb = (shared, b) if over == "a" else (a, shared)
    assert engine.lib.fastface_cos_sim_matrix(engine.h, pa.ctypes.data, n, pb.ctypes.data, m, shared.ctypes.data) == 0
    assert np.array_equal(shared[:n * m].reshape(n, m), want)


def test_matrix_after_an_error_of_the_callers(engine):
    """The CUDA runtime is the process's: an error that other code has left behind on this thread is none of the call's."""
    rng = np.random.default_rng(9)
    a, b = rng.standard_normal((5, 512), dtype=np.float32), rng.standard_normal((9, 512), dtype=np.float32)
    want = engine.cos_sim_matrix(a, b)
    rt = C.CDLL("libcudart.so.12")
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(1 << 60)) == 2         # more than any device has: out of memory
    assert np.array_equal(engine.cos_sim_matrix(a, b), want)
    rt.cudaGetLastError()


# both sides of the lines of a call's path: inputs of a megabyte (512 rows), results of a megabyte, launches of whole waves
# (1024 columns: 512 rows), the launch's largest result, the widest gallery kept at once
@pytest.mark.parametrize("n,m", [(12, 500), (13, 500), (255, 257), (512, 512), (513, 511), (1024, 1024), (1500, 1024), (1, 16385), (160, 16384), (161, 16390)])
def test_matrix_paths(engine, n, m):
    """Pageable and page-locked arrays, in every combination, give the same matrix; two calls, so that buffers are used again."""
    import torch
    rng = np.random.default_rng(n * 31 + m)
    a = rng.standard_normal((n, 512), dtype=np.float32)
    b = rng.standard_normal((m, 512), dtype=np.float32)
    b[m // 3] = 0

    def locked(x):
        t = torch.empty(x.shape, dtype=torch.float32, pin_memory=True).numpy()
        t[...] = x
        return t

    want = engine.cos_sim_matrix(a, b)
    check(want, a, b, rng, 200)
    la, lb = locked(a), locked(b)
    for pa, pb, lo in ((a, b, False), (la, b, False), (a, lb, True), (la, lb, True), (a, b, True)):
        out = locked(np.zeros((n, m), np.float32)) if lo else np.zeros((n, m), np.float32)
        assert engine.lib.fastface_cos_sim_matrix(engine.h, pa.ctypes.data, n, pb.ctypes.data, m, out.ctypes.data) == 0
        assert np.array_equal(out, want)
