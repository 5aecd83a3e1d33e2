"""Node records of scene files, checked where no GPU is needed: records that
the library writes are canonical, and each way of not being one is refused
(a slot's kind against the mask, a triangle count of zero, offsets that do not
follow from the counts, unused bits)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "bvh8.cuh"
#include <cstring>
extern "C" int is_canonical(const void *p) { ilg::FileNode8 f; memcpy(&f, p, sizeof f); return ilg::canonical(f); }
extern "C" void round_trip(const void *p, void *out)
{
    ilg::FileNode8 f, g;
    memcpy(&f, p, sizeof f);
    g = ilg::to_file(ilg::from_file(f));
    memcpy(out, &g, sizeof g);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("records")
    (d / "r.cu").write_text(SRC)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "illuminaprt_b200", "csrc"),
                    str(d / "r.cu"), "-o", str(d / "r.so")], check=True)
    return ctypes.CDLL(str(d / "r.so"))


def _record(kinds):
    """kinds: per slot 0 empty, "n" a node, 1..3 a leaf's triangles."""
    rng = np.random.default_rng(len(kinds))
    q = rng.integers(0, 2 ** 32, 20, dtype=np.uint64).astype(np.uint32)
    meta, imask, off = np.zeros(8, np.uint8), 0, 0
    for s, k in enumerate(kinds):
        if k == "n":
            meta[s], imask = 0x80, imask | 1 << s
        elif k:
            meta[s], off = k << 5 | off, off + k
    q[3] = 120 | 121 << 8 | 122 << 16 | imask << 24
    q[6:8] = meta.view(np.uint32)
    return q


@pytest.mark.parametrize("kinds", [[0] * 8, ["n"] * 8, [3] * 8, [1, "n", 2, 0, 3, "n", 0, 1], [0, 0, 2, 2, "n", 1, 3, 0]])
def test_canonical_records(lib, kinds):
    q = _record(kinds)
    assert lib.is_canonical(q.ctypes.data_as(ctypes.c_void_p))
    out = np.zeros_like(q)
    lib.round_trip(q.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p))
    assert np.array_equal(out, q)


def test_other_records_are_refused(lib):
    good = _record([1, "n", 2, 0, 3, "n", 0, 1])
    meta = good[6:8].view(np.uint8)
    n = 0
    for s in range(8):
        for m in range(256):
            if m == meta[s]:
                continue
            q = good.copy()
            q[6:8].view(np.uint8)[s] = m
            # (the last leaf's count may change: nothing behind it depends on it)
            free = s == 7 and m >> 7 == 0 and m >> 5 and m & 31 == meta[7] & 31 or s == 7 and m == 0
            assert bool(lib.is_canonical(q.ctypes.data_as(ctypes.c_void_p))) == bool(free), (s, m)
            n += 1
        q = good.copy()
        q[3] ^= np.uint32(1 << (24 + s))
        assert not lib.is_canonical(q.ctypes.data_as(ctypes.c_void_p))
    assert n == 8 * 255


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(1, 1), (256, 128), (331, 199)])
def test_records_survive_chunk_by_chunk(tmp_path, nx, ny):
    # 2, 65,536 (one chunk of triangle records) and 131,738 triangles
    from illuminaprt_b200 import scenes
    from illuminaprt_b200.ilg import GpuSpace
    pos, idx = scenes.heightfield(nx, ny, 0.2, 4)
    a, b = GpuSpace(), GpuSpace()
    a.initialise(pos, idx, np.arange(idx.shape[0]) % 7)
    a.build()
    a.save(tmp_path / "a.ilg")
    b.load(tmp_path / "a.ilg")
    b.save(tmp_path / "b.ilg")
    assert (tmp_path / "a.ilg").read_bytes() == (tmp_path / "b.ilg").read_bytes()
    o4, d4 = scenes.incoherent_rays(pos, idx, 50000, seed=6)
    for x, y in zip(a.intersects(o4, d4), b.intersects(o4, d4)):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    a.close()
    b.close()
