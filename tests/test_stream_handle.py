"""The stream a call is queued on: the one it is given, else the current one, with torch's check of the
process (no driver, a fork after CUDA was used) and without relying on a getter that torch does not publish."""

import types

import pytest
import torch

from cuvslam_b200 import frontend


@pytest.fixture
def device(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: types.SimpleNamespace(cuda_stream=0x51))


def test_given_stream():
    assert frontend._stream_handle(types.SimpleNamespace(cuda_stream=0x77)).value == 0x77


def test_current_stream_of_the_current_device(device, monkeypatch):
    monkeypatch.setattr(frontend, "_raw_stream", lambda d: 0x100 + d)
    assert frontend._stream_handle().value == 0x103


def test_without_the_raw_getter(device, monkeypatch):
    monkeypatch.setattr(frontend, "_raw_stream", None)
    assert frontend._stream_handle().value == 0x51


def test_torchs_check_comes_first(monkeypatch):
    def refuse():
        raise RuntimeError("Cannot re-initialize CUDA in forked subprocess")

    monkeypatch.setattr(torch.cuda, "current_device", refuse)
    with pytest.raises(RuntimeError, match="forked"):
        frontend._stream_handle()
