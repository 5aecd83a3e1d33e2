"""Training after a cached render, where the device alone knows how many
records there are: steps beyond them do nothing, a frame without records takes
no Adam step, and ragged batches use every record."""
import numpy as np
import pytest

from illuminaprt_b200 import scenes

pytestmark = pytest.mark.gpu


def _frame(steps, batch, encoding="hashgrid", hit=True, epochs=1, frames=1):
    from illuminaprt_b200.ilg import GpuSpace
    f = scenes.sphere_field(3, 3, seed=5, width=160, height=90)
    sp = GpuSpace()
    scenes.load_sphere_field(sp, f)
    sp.mlp_init(seed=3, lr=1e-2, encoding=encoding)
    w0 = sp.mlp_params()
    cam = dict(f["camera"], aspect=160 / 90)
    if not hit:
        cam["target"] = (0.0, 100.0, 0.0)  # the sky
        cam["eye"] = (0.0, 50.0, 0.0)
    for k in range(frames):
        sp.render(cam, 160, 90, 2, max_depth=6, seed=7 + k, sky=f["sky"], cache_depth=1, train_every=4,
                  train_steps=steps, train_batch=batch, train_tail=1, train_epochs=epochs)
    n, w1, stats = sp.last_train_stats()[0], sp.mlp_params(), sp.mlp_grid() if encoding == "hashgrid" else None
    sp.close()
    return n, w0, w1, stats


def test_no_records_no_step():
    n, w0, w1, _ = _frame(4, 256, hit=False)
    assert n == 0 and np.array_equal(w0, w1)


@pytest.mark.parametrize("encoding", ["hashgrid", "freq12"])
@pytest.mark.parametrize("batch", [4096, 5001])
def test_steps_past_the_records_do_nothing(batch, encoding):
    # one batch holds every record, so the records' order (which differs from
    # run to run) matters to the sums' rounding only; a further Adam step would
    # move every weight by about the learning rate, 1e-2
    a = _frame(1, batch, encoding)
    assert 200 < a[0] <= batch and not np.array_equal(a[1], a[2])
    # (more than 64 steps leave the captured frame: both ways are taken)
    for steps in (4, 71):
        b = _frame(steps, batch, encoding)
        assert b[0] == a[0]
        assert np.median(np.abs(b[2] - a[2])) < 1e-3
        if encoding == "hashgrid":
            assert np.mean(b[3] == a[3]) > 0.5  # untouched entries stay


def test_epochs_and_frames_keep_training():
    one, two = _frame(2, 1000), _frame(2, 1000, epochs=2, frames=3)
    assert np.abs(two[2] - two[1]).mean() > 2.0 * np.abs(one[2] - one[1]).mean()
