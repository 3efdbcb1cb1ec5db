"""Track records on their way to and from tensors: every device argument torch takes, and memory of their
own on the host."""

import numpy as np
import pytest
import torch

from cuvslam_b200.frontend import tracks_from_device, tracks_to_device
from cuvslam_b200.types import make_tracks


def _records(n=7):
    rng = np.random.default_rng(n)
    return make_tracks(rng.uniform(0, 100, (n, 2)), rng.normal(size=(n, 2)), 12.0, 0.8)


@pytest.mark.parametrize("device", [None, "cpu", torch.device("cpu")])
@pytest.mark.parametrize("readonly", [False, True])
def test_host_tensors_own_their_memory(device, readonly):
    recs = _records()
    want = recs.view(np.uint8).copy()
    recs.flags.writeable = not readonly
    t = tracks_to_device(recs, device)
    assert t.device.type == "cpu" and t.shape == (7, 80) and t.dtype == torch.uint8
    t[0] = 0  # does not reach the caller's records
    assert np.array_equal(recs.view(np.uint8), want)
    back = tracks_from_device(t)
    back["track"][1] = -1.0  # nor the tensor
    assert np.array_equal(t.numpy()[1:], want.reshape(7, 80)[1:])


def test_no_records():
    assert tracks_to_device(_records()[:0], None).shape == (0, 80)
