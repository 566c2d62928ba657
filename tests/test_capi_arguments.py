"""What the Python binding passes on to the library, with a stand-in for the library."""
import numpy as np
import pytest

from deepscalemd_b200 import capi


class Library:
    """Counts calls and reports success; nothing is read through the pointers."""
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append(name) or 0


@pytest.fixture
def context(monkeypatch):
    torch = pytest.importorskip("torch")
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    ctx = capi.Context.__new__(capi.Context)
    ctx.lib, ctx.h, ctx.device = Library(), None, 0
    return ctx


@pytest.mark.parametrize("pos,vel", [(np.zeros((5, 2)), None), (np.zeros(15), None), (np.zeros((5, 3)), np.zeros((5, 2))), (np.zeros((5, 0)), None)])
def test_upload_refuses_rows_of_fewer_than_three(context, pos, vel):
    with pytest.raises(IndexError):
        context.upload(pos, vel=vel)
    assert context.lib.calls == []


@pytest.mark.parametrize("pos", [np.zeros((5, 3)), np.zeros((5, 4), dtype=np.float32), np.asfortranarray(np.ones((5, 3))), [[0, 1, 2]], np.zeros((0, 3))])
def test_upload_takes_rows_of_three_and_more(context, pos):
    context.upload(pos, vel=pos)
    assert context.lib.calls == ["dsmd_upload_rows"]
