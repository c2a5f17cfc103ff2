"""Batches out of pinned host memory: rows of samples and labels that are aligned for 16-byte loads or not, and a short last batch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x_size,y_size", [(784, 10), (517, 6), (64, 4), (33, 8), (1, 1), (784, 1001)])
def test_every_batch_of_two_epochs(x_size, y_size):
    from oxidized_neural_orchestra_b200.runtime.gpu_rank import BatchFeeder

    rng, rows, batch = np.random.default_rng(0), 100, 32
    xs, ys = rng.random((rows, x_size), dtype=np.float32), rng.random((rows, y_size), dtype=np.float32)
    f = BatchFeeder(xs.reshape(-1), ys.reshape(-1), x_size, y_size, batch, torch.device("cuda", 0), seed=5)
    seen = []
    for epoch in range(2):
        for step in range(f.steps_per_epoch()):
            slot = step % 2
            f.dev_x[slot].fill_(-7.0)
            f.dev_y[slot].fill_(-7.0)
            torch.cuda.synchronize()
            n = f.stage(slot, epoch, step)
            torch.cuda.current_stream().wait_event(f.ready[slot])
            idx = f._indices(epoch, step).numpy()
            assert n == len(idx) == (4 if step == 3 else batch)
            x, y = f.dev_x[slot].cpu().numpy(), f.dev_y[slot].cpu().numpy()
            assert np.array_equal(x[:n], xs[idx]) and np.array_equal(y[:n], ys[idx])
            assert (x[n:] == -7.0).all() and (y[n:] == -7.0).all()
            f.consumed[slot].record()
            seen.append(idx)
    assert sorted(np.concatenate(seen[:4])) == list(range(rows)) and sorted(np.concatenate(seen[4:])) == list(range(rows))


# more rows of a warp than row numbers it holds at a time, fewer rows than warps, labels about a warp wide, rows about its loads in flight
@pytest.mark.parametrize("x_size,y_size,rows,batch", [(1, 1, 37, 37), (3, 2, 1, 1), (255, 31, 19, 6), (128, 32, 5, 5), (129, 33, 7, 7), (516, 36, 33, 33),
                                                      (508, 160, 65, 64), (2, 1, 4501, 4501), (4, 4, 2500, 2499)])
def test_edges_of_rows_and_warps(x_size, y_size, rows, batch):
    from oxidized_neural_orchestra_b200.runtime.gpu_rank import BatchFeeder

    rng = np.random.default_rng(1)
    xs, ys = rng.random((rows, x_size), dtype=np.float32), rng.random((rows, y_size), dtype=np.float32)
    f = BatchFeeder(xs.reshape(-1), ys.reshape(-1), x_size, y_size, batch, torch.device("cuda", 0), seed=5)
    for step in range(f.steps_per_epoch()):
        n = f.stage(step % 2, 0, step)
        torch.cuda.current_stream().wait_event(f.ready[step % 2])
        idx = f._indices(0, step).numpy()
        assert n == len(idx)
        assert np.array_equal(f.dev_x[step % 2][:n].cpu().numpy(), xs[idx]) and np.array_equal(f.dev_y[step % 2][:n].cpu().numpy(), ys[idx])
        f.consumed[step % 2].record()


def test_an_epoch_that_was_asked_about_before_it_is_fed():
    """Row numbers of an epoch may be looked up ahead of its first batch, and of another epoch between its batches."""
    from oxidized_neural_orchestra_b200.runtime.gpu_rank import BatchFeeder

    rng, rows, batch = np.random.default_rng(2), 50, 16
    xs, ys = rng.random((rows, 5), dtype=np.float32), rng.random((rows, 3), dtype=np.float32)
    f = BatchFeeder(xs.reshape(-1), ys.reshape(-1), 5, 3, batch, torch.device("cuda", 0), seed=5)
    f._indices(0, 0)
    for k, (epoch, step) in enumerate([(0, 0), (0, 1), (1, 0), (1, 3), (0, 2), (2, 1), (2, 2)]):
        f._indices(epoch + k % 3, 0)
        n = f.stage(k % 2, epoch, step)
        torch.cuda.current_stream().wait_event(f.ready[k % 2])
        idx = f._indices(epoch, step).numpy()
        assert n == len(idx)
        assert np.array_equal(f.dev_x[k % 2][:n].cpu().numpy(), xs[idx]) and np.array_equal(f.dev_y[k % 2][:n].cpu().numpy(), ys[idx])
        f.consumed[k % 2].record()


def test_row_numbers_in_ordinary_memory_are_refused():
    """The kernel reads them where they are; a call that names memory it cannot read is an error, and the next one runs."""
    from oxidized_neural_orchestra_b200.ops import _lib
    from oxidized_neural_orchestra_b200.runtime.gpu_rank import BatchFeeder

    xs, ys = np.arange(40, dtype=np.float32), np.arange(20, dtype=np.float32)
    f = BatchFeeder(xs, ys, 4, 2, 5, torch.device("cuda", 0), seed=5)
    job, feed, args = f.feeds[0]
    pageable = np.arange(5, dtype=np.int32)
    job.idx, job.n = pageable.ctypes.data, 5
    assert feed(*args) == -1 and b"pinned" in _lib.load().ono_last_error()
    assert f.stage(0, 0, 0) == 5
    f.copy_stream.synchronize()
    assert np.array_equal(f.dev_x[0].cpu().numpy(), xs.reshape(10, 4)[f._indices(0, 0).numpy()])
