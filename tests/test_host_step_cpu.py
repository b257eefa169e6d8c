"""attention.HostDecodeStep without a GPU: the CUDA calls are replaced by recorders, so that what the object keeps alive can
be compared with the raw addresses that its launches were given."""
import contextlib
import gc
import weakref

import pytest


class _Nothing:
    def __init__(self, *args, **kwargs):
        pass

    def __getattr__(self, name):
        return lambda *args, **kwargs: None


@pytest.fixture
def recorded(pkg, monkeypatch):
    """The attention module with its CUDA parts faked: (module, argument structures of the launches, workspaces made)."""
    import torch
    from llm_infer_b200 import attention as A
    launches, made = [], []

    class FakeWorkspace:
        def __init__(self, batch, n_heads, n_kv_heads, head_dim, device=None):
            self.key = (batch, n_heads, n_kv_heads, head_dim, None)  # a CPU tensor's device has no index
            self.nbytes = 4096
            self.buf = torch.zeros(self.nbytes, dtype=torch.uint8)
            self.status = torch.zeros(1, dtype=torch.int32)
            made.append(weakref.ref(self))

    monkeypatch.setattr(A, "DecodeWorkspace", FakeWorkspace)
    monkeypatch.setattr(A, "_require_cuda", lambda *tensors: None)
    monkeypatch.setattr(A, "_call", lambda entry, device, stream, *args, what=None: launches.append((entry, args[0]._obj)))
    monkeypatch.setattr(torch.Tensor, "is_pinned", lambda self: True)
    for name in ("Stream", "CUDAGraph", "current_stream"):
        monkeypatch.setattr(torch.cuda, name, _Nothing)
    for name in ("device", "stream", "graph"):
        monkeypatch.setattr(torch.cuda, name, lambda *args, **kwargs: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *args: None)
    return A, launches, made


@pytest.mark.parametrize("given", ["none", "matching", "other batch"])
def test_the_step_keeps_the_workspace_that_its_graph_was_captured_with(recorded, given):
    import torch
    A, launches, made = recorded
    B, T, H, Hkv, D = 2, 8, 4, 2, 64
    host_in, out_host = torch.zeros(B * (H + 2 * Hkv) * D), torch.zeros(B, H, D)
    k, v = (torch.zeros((B, T, Hkv, D), dtype=torch.float16) for _ in range(2))
    pos = torch.zeros(B, dtype=torch.int32)
    workspace = {"none": lambda: None, "matching": lambda: A.DecodeWorkspace(B, H, Hkv, D),
                 "other batch": lambda: A.DecodeWorkspace(B + 1, H, Hkv, D)}[given]()
    step = A.HostDecodeStep(host_in, k, v, pos, pos, out_host, n_heads=H, theta=1e4, workspace=workspace)
    gc.collect()
    decodes = [a for entry, a in launches if entry == "attn_decode"]
    assert len(decodes) == 2  # warm-up and capture
    alive = {ws().buf.data_ptr(): ws() for ws in made if ws() is not None}
    for a in decodes:
        assert a.workspace in alive, "the launches were given the address of a workspace that is gone"
        assert alive[a.workspace] is step.workspace and a.status == step.workspace.status.data_ptr()
    assert step.workspace.key == (B, H, Hkv, D, None)
    assert (step.workspace is workspace) == (given == "matching")
