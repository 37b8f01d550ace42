"""PathModel's gather and its adjoint make the positions' device current for their launches (a stage may live on another
GPU than the current one): shown with a recorded device guard and library, without a GPU."""
from types import SimpleNamespace

import torch

from feffgpu_b200 import model as M


def test_gather_and_scatter_launch_under_the_tensors_device(monkeypatch):
    events = []

    class Guard:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            events.append(("enter", self.device))

        def __exit__(self, *exc):
            events.append(("exit", self.device))

    class Library:
        def __getattr__(self, name):
            return lambda *args: events.append((name, args)) or 0

    def stream(device):
        return SimpleNamespace(cuda_stream=("stream of", device))

    monkeypatch.setattr(torch.cuda, "device", Guard)
    monkeypatch.setattr(torch.cuda, "current_stream", stream)
    monkeypatch.setattr(M._lib, "load", Library)
    x = torch.zeros(4, 3, dtype=torch.float64)
    batch = SimpleNamespace(n=2, nleg_max=2, nleg=torch.full((2,), 2, dtype=torch.int32))
    m = SimpleNamespace(batch=batch, natoms=4, min_image=SimpleNamespace(cell=None, cell18=None),
                        atoms=torch.zeros(2, 2, dtype=torch.long), entry=torch.zeros(4, dtype=torch.int32),
                        entry_off=torch.zeros(5, dtype=torch.long))
    ctx = SimpleNamespace()
    out = M._Gather.forward(ctx, x, m)
    M._Gather.backward(ctx, torch.zeros_like(out))
    names = [e[0] for e in events]
    assert names == ["enter", "fg_path_gather", "exit", "enter", "fg_path_scatter", "exit"]
    for guard, call in ((events[0], events[1]), (events[3], events[4])):
        assert guard[1] == x.device and call[1][-1] == ("stream of", x.device)
