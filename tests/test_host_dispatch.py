"""CPU tests of what the kernel wrappers decide before a launch: devices they refuse, and which calls take which route.
The library is replaced by a recorder, so nothing is launched."""
import pytest
import torch

from hetu_dit_b200 import _C, kernels


class Recorder:
    """Stands in for the loaded library: records the entry points that are called and reports success."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, args))
            return 0
        return entry


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(_C, "lib", lambda: rec)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 1000 + index)
    return rec


BOX = (16, 32, 1, 0, 0, 1, 0, 0, 8)


def test_host_tensors_never_reach_a_kernel(lib):
    """A wrapper without an is_cuda check of its own still refuses a host tensor: a kernel on a host address would fault."""
    t = torch.zeros(1, 8, 2, 64, dtype=torch.bfloat16)
    calls = (lambda: kernels.copy_pieces([BOX], torch.device("cpu")),
             lambda: kernels.copy_2d(torch.empty(4, 8), torch.zeros(4, 8)),
             lambda: kernels.kv_scatter(torch.zeros(1, 8, 256), t.view(1, 8, 128).float(), t.view(1, 8, 128).float(), 0),
             lambda: kernels.qk_norm_rope([(t, None, 1, False)]))
    for call in calls:
        with pytest.raises(ValueError, match="cuda"):
            call()
    assert lib.calls == []


@pytest.mark.parametrize("device", ["cuda:0", "cuda", 0, -1, None, torch.device("cuda"), torch.device("cuda", 0)])
def test_devices_are_named_as_torch_names_them(lib, device):
    kernels.copy_pieces([BOX], device)
    (name, args), = lib.calls
    assert name == "hdit_copy_pieces" and args[1:] == (1, 1000)
    with pytest.raises(ValueError):
        kernels.copy_pieces([BOX], "cpu")
    assert len(lib.calls) == 1
