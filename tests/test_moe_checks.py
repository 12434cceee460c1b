"""What the expert feed-forward refuses before a kernel gets an address, on the host."""
import pytest
import torch

from neuralfn_b200.ops import _lib
from neuralfn_b200.ops import moe


class _Library:
    """Stands for the kernel library: any entry point takes its arguments and returns 0."""

    def __getattr__(self, name):
        def entry(*args):
            return 0
        setattr(self, name, entry)
        return entry


def _operands(T=6, d=64, h=128, E=4, k=2):
    bf = dict(dtype=torch.bfloat16)
    return dict(x=torch.zeros(T, d, **bf), w1=torch.zeros(E, d, h, **bf), w2=torch.zeros(E, h, d, **bf), w3=torch.zeros(E, d, h, **bf),
                weights=torch.ones(T, k), indices=torch.zeros(T, k, dtype=torch.int64))


@pytest.mark.parametrize("change", [
    dict(indices=torch.zeros(5, 2, dtype=torch.int64)), dict(indices=torch.zeros(2, dtype=torch.int64)), dict(indices=torch.zeros(6, 2)),
    dict(indices=torch.zeros(6, 2, 1, dtype=torch.int64)), dict(weights=torch.ones(5, 2)), dict(weights=torch.ones(6, 3)), dict(weights=torch.ones(5, 1)),
    dict(w3=torch.zeros(4, 64, 64, dtype=torch.bfloat16)), dict(w3=torch.zeros(3, 64, 128, dtype=torch.bfloat16)), dict(w3=torch.zeros(4, 64, 128)),
    dict(w2=torch.zeros(4, 64, 128, dtype=torch.bfloat16)), dict(w1=torch.zeros(4, 128, 128, dtype=torch.bfloat16)),
    dict(x=torch.zeros(6, 128, dtype=torch.bfloat16)), dict(x=torch.zeros(6, 64)), dict(x=torch.zeros(2, 3, 64, dtype=torch.bfloat16)),
    dict(w2=torch.zeros(4, 128, 64, dtype=torch.bfloat16, device="meta")),
], ids=lambda c: next(f"{n} {tuple(t.shape)} {str(t.dtype)[6:]} {t.device}" for n, t in c.items()))
def test_moe_experts_refuses_operands_that_do_not_fit(monkeypatch, change):
    monkeypatch.setattr(_lib, "load", lambda: _Library())
    monkeypatch.setattr(_lib, "stream_ptr", lambda: 0)
    with pytest.raises(RuntimeError, match="moe_experts|expand"):
        moe.moe_experts(**{**_operands(), **change})


def test_moe_experts_refuses_host_tensors(monkeypatch):
    monkeypatch.setattr(_lib, "load", lambda: _Library())
    monkeypatch.setattr(_lib, "stream_ptr", lambda: 0)
    with pytest.raises(RuntimeError, match="CUDA"):
        moe.moe_experts(**_operands())


@pytest.mark.parametrize("weights", [torch.ones(6, 1), torch.ones(1, 2), torch.ones(2), torch.tensor(1.0)])
def test_expert_operands_expands_weights(weights):
    full, indices = moe._expert_operands(**{**_operands(), "weights": weights, "indices": torch.zeros(6, 2, dtype=torch.int32)})
    assert full.shape == (6, 2) and indices.shape == (6, 2)


@pytest.mark.skipif(torch.cuda.is_available(), reason="addresses that must never reach a device")
@pytest.mark.parametrize("name,entry", [("work", "forward"), ("work", "backward"), ("scratch", "backward")])
def test_workspaces_off_32_bytes_are_refused_before_a_launch(name, entry):
    """The epilogues store 32 bytes at a time. Addresses that are never read: the check is the first thing the entry does."""
    import ctypes
    lib = _lib.load()
    where = {n: 1 << 20 for n in ("x", "w1", "w2", "w3", "weights", "indices", "out", "work", "dout", "scratch", "dx", "dw1", "dw2", "dw3", "dweights")}
    where[name] += 16
    args = moe._ExpertsArgs(**where, tokens=6, d=64, ff=128, experts=4, top=2, capacity_rows=640, save=1)
    assert getattr(lib, f"nfn_moe_experts_{entry}")(ctypes.byref(args), None) == -1
    assert b"32-byte aligned" in lib.nfn_last_error()
