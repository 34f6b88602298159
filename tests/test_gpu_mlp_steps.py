"""Trainings of several epochs and mini-batches, step for step against the
network in 64 bits: a step that reads parameters or deltas of a step before it
shows in the weights."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,rows,batch,epochs", [(38, 600, 64, 3), (5, 300, 100, 4),
                                                    (64, 1000, 256, 4), (1, 33, 8, 6)])
def test_training_against_64_bits(gat, n_in, rows, batch, epochs):
    """Rounding alone leaves a root mean square of 4e-8 in the weights (the
    64-bit steps repeated in 32 bits on the CPU); one step of the training
    taken from the weights of the step before it leaves 4e-5 and more."""
    for seed in range(10):
        case = dict(kind="train", rows=rows, features=n_in, epochs=epochs, batch=batch)
        got = cases.run(cases.prepare(case, seed))
        want = cases.exact(case, seed)
        assert np.sqrt(np.mean((got["params"] - want["params"]) ** 2)) < 1e-6, seed
        assert abs(got["loss"] - want["loss"]) < 1e-5 * max(1.0, want["loss"]), seed
