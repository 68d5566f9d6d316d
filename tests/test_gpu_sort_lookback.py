"""The radix sort's look-back over digit counts: right sums at every kind of
tile whether or not inclusive words are there, and one time limit for all the
waits of a look-back whose predecessors never publish."""
import ctypes as C
import shutil
import subprocess
import time
from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
READY, GROUP, SUPER, TILES, BINS = 1 << 31, 8, 64, 24, 256
TIMEOUT = 2  # kDevTimeout
LIMIT = 2.0  # seconds (kWaitLimitNs)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc is needed to build the test's kernel")
    out = tmp_path_factory.mktemp("lookback") / "liblookback.so"
    cmd = ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-shared",
           "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
           str(Path(__file__).with_name("sort_lookback.cu")), "-o", str(out)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    lib = C.CDLL(str(out))
    lib.lookback.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p]
    return lib


def words_of(counts, tile, inclusive):
    """The words once every tile before `tile` has published its counts, with
    the inclusive words of the super-groups in `inclusive`."""
    tiles = counts.shape[0]
    rows = [-(-tiles // n) for n in (1, GROUP, SUPER, SUPER)]
    t, g, s, i = (np.zeros((r, BINS), np.uint32) for r in rows)
    t[:tile] = READY | counts[:tile]
    for n, w in ((GROUP, g), (SUPER, s)):
        for k in range(tile):
            w[k // n] += (1 << TILES) | counts[k]
    for k in inclusive:
        i[k] = READY | counts[: (k + 1) * SUPER].sum(0, dtype=np.uint32)
    return np.concatenate([t, g, s, i])


def run(lib, words, tiles, tile):
    assert words.shape[0] == lib.lookback_rows(tiles)
    w = torch.from_numpy(words.view(np.int32)).cuda()
    out = torch.full((BINS,), -1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    t0 = time.monotonic()
    assert lib.lookback(w.data_ptr(), tiles, tile, 3, out.data_ptr(), status.data_ptr()) == 0
    return out.cpu().numpy().view(np.uint32), int(status.item()), time.monotonic() - t0, w


@pytest.mark.parametrize("tile", [0, 1, 7, 8, 63, 64, 65, 200, 64 * 4 + 63, 64 * 5, 64 * 9 + 44])
def test_sums(cuda, lib, tile):
    rng = np.random.default_rng(tile)
    tiles = 64 * 10 + 3
    counts = rng.integers(0, 4097, (tiles, BINS)).astype(np.uint32)
    full = tile // SUPER
    for inclusive in ([], range(full), range(max(0, full - 1)), [0] if full else []):
        out, status, _, w = run(lib, words_of(counts, tile, inclusive), tiles, tile)
        assert status == 0
        assert np.array_equal(out, counts[:tile].sum(0, dtype=np.uint32))
        if tile % SUPER == SUPER - 1:  # the last of its super-group publishes the sum
            row = w.cpu().numpy().view(np.uint32)[-(-(-tiles // SUPER)) + full]
            assert np.array_equal(row, READY | (out + 3))


def test_one_limit_for_all_waits(cuda, lib):
    tiles = 64 * 12
    tile = 64 * 11 + 7 * 8 + 7  # waits for super-groups, groups and tiles
    rng = np.random.default_rng(5)
    counts = rng.integers(1, 4097, (tiles, BINS)).astype(np.uint32)
    out, status, seconds, _ = run(lib, np.zeros((lib.lookback_rows(tiles), BINS), np.uint32),
                                  tiles, tile)
    assert status == TIMEOUT and not out.any()
    assert 0.9 * LIMIT < seconds < 1.5 * LIMIT
    # one group of eight tiles is missing: the rest of the sum, in one limit
    words = words_of(counts, tile, range(11))
    words[tiles + 11 * 8 + 2] = 0
    out, status, seconds, _ = run(lib, words, tiles, tile)
    assert status == TIMEOUT
    missing = counts[64 * 11 + 16: 64 * 11 + 24].sum(0, dtype=np.uint32)
    assert np.array_equal(out, counts[:tile].sum(0, dtype=np.uint32) - missing)
    assert 0.9 * LIMIT < seconds < 1.5 * LIMIT
