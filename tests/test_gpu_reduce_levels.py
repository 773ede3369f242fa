"""sppm_reduce_texture folds several levels per launch: every number of levels its launches take
(three, two, one from memory, the last ones in one block) against the oracle's level-by-level fold,
bit for bit -- each output is the same operations in the same order -- with values that are not
finite, and from two threads on streams of their own at once."""
import threading

import numpy as np
import pytest

from oracle.binding import reduce_texture as oracle_reduce

pytestmark = pytest.mark.gpu


def reduce(t, R, op, stream):
    import glslppm_gb300 as g
    return g.renderer.reduce_texture(t.data_ptr(), R, op, stream.cuda_stream)


@pytest.mark.parametrize("R", [2, 16, 32, 64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("special", [False, True])
def test_levels(R, special):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(R)
    t = (rng.standard_normal((R * R, 4)) * 100).astype(np.float32)
    if special:
        n = max(1, R * R // 50)
        t[rng.integers(0, R * R, n), 0] = np.inf
        t[rng.integers(0, R * R, n), 1] = -np.inf
        t[rng.integers(0, R * R, n), 2] = np.nan
        t[rng.integers(0, R * R, n), 3] = -0.0
    d = torch.from_numpy(t).cuda()
    for op in (0, 1, 2):
        got, want = reduce(d, R, op, torch.cuda.current_stream()), oracle_reduce(t, R, op)
        same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
        assert same.all(), (R, op, got, want)


def test_two_threads():
    torch = pytest.importorskip("torch")
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        stream = torch.cuda.Stream()
        for R in (64, 1024, 256, 2048) * 3:
            t = rng.standard_normal((R * R, 4)).astype(np.float32)
            with torch.cuda.stream(stream):
                d = torch.from_numpy(t).cuda()
                got = reduce(d, R, 2, stream)
            if not np.array_equal(got.view(np.uint32), oracle_reduce(t, R, 2).view(np.uint32)):
                bad.append((seed, R))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
