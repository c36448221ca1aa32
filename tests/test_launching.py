"""How a call changes the current device around its launches (ateniaengine_b200/moe.py, `_launching`), with torch's calls
replaced: no device is set where the right one is current, and another one is entered and left through torch.cuda.device, which
creates no context on the device that was current before."""
import pytest
import torch

from ateniaengine_b200 import moe


@pytest.fixture
def cuda(monkeypatch):
    state = {"current": 0, "log": []}

    class Device:
        def __init__(self, index):
            self.index = index

        def __enter__(self):
            self.before, state["current"] = state["current"], self.index
            state["log"].append(("enter", self.index))

        def __exit__(self, *exc):
            state["current"] = self.before
            state["log"].append(("leave", self.index))

    def forbidden(*a):
        raise AssertionError("set_device creates a context")

    monkeypatch.setattr(torch.cuda, "current_device", lambda: state["current"])
    monkeypatch.setattr(torch.cuda, "set_device", forbidden)
    monkeypatch.setattr(torch.cuda, "device", Device)
    monkeypatch.setattr(moe, "_current_stream", lambda i: (i, state["current"]), raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda i: (i, state["current"]), raising=False)
    return state


def test_the_current_device_is_left_alone(cuda):
    with moe._launching(torch.device("cuda", 0)) as stream:
        assert stream == (0, 0)
    assert cuda["log"] == [] and cuda["current"] == 0


def test_another_device_is_entered_and_left(cuda):
    with moe._launching(torch.device("cuda", 1)) as stream:
        assert stream == (1, 1) and cuda["current"] == 1
    assert cuda["log"] == [("enter", 1), ("leave", 1)] and cuda["current"] == 0


def test_it_is_left_when_the_call_raises(cuda):
    with pytest.raises(ValueError), moe._launching(torch.device("cuda", 1)):
        raise ValueError
    assert cuda["current"] == 0 and cuda["log"][-1] == ("leave", 1)
