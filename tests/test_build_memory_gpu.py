"""Device memory that a build leaves allocated. A context built once holds its
mesh and its records alone (their capacity: 96 bytes of nodes and 64 of
triangle records a triangle), not the 180 bytes of scratch a triangle; one
that builds again may keep the scratch, up to 256 MB. 16 MB are allowed for
allocation granularity and for kernels loaded on first use."""
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("nx,ny,kept", [(640, 320, True), (1300, 700, False)])
def test_scratch_is_given_back(nx, ny, kept):
    import torch
    from illuminaprt_b200.ilg import GpuSpace
    warm = GpuSpace()
    warm.initialise(*scenes.heightfield(64, 32, 0.2, 1))
    for _ in range(2):
        warm.build()
    pos, idx = scenes.heightfield(nx, ny, 0.2, 1)
    n = idx.shape[0]

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    sp = GpuSpace()
    sp.initialise(pos, idx)
    before = free()
    sp.build()
    assert before - free() <= 160 * n + 16 * MB
    first = sp.stats()["n_nodes"]
    for _ in range(3):
        sp.build()
    assert before - free() <= (160 + (200 if kept else 0)) * n + 16 * MB
    assert sp.stats()["n_nodes"] == first
    sp.close()
    warm.close()
