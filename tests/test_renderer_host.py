"""Host-side decisions of the renderer module, on the CPU."""
import pytest
import torch

from supernormal_gb300.fields import SingleVarianceNetwork
from supernormal_gb300.renderer import NeuSRenderer


def _renderer():
    r = NeuSRenderer.__new__(NeuSRenderer)   # (the constructor puts an occupancy grid on a GPU)
    r.deviation_network = SingleVarianceNetwork(0.3)
    return r


@pytest.mark.parametrize("seen_by", ["forward hook", "forward pre-hook", "backward hook", "backward pre-hook",
                                     "global forward hook", "global backward hook", "instance forward", "class forward"])
def test_a_watched_variance_network_is_called(seen_by, monkeypatch):
    """Whatever would see a call of the variance network sees it, and a replaced
    forward gives the value."""
    r, calls = _renderer(), []
    net = r.deviation_network
    plain = r._inv_s(torch.device("cpu")).detach()
    note = lambda *a, **k: calls.append(1)
    every = torch.nn.modules.module
    handle = {"forward hook": lambda: net.register_forward_hook(note),
              "forward pre-hook": lambda: net.register_forward_pre_hook(note),
              "backward hook": lambda: net.register_full_backward_hook(note),
              "backward pre-hook": lambda: net.register_full_backward_pre_hook(note),
              "global forward hook": lambda: every.register_module_forward_hook(note),
              "global backward hook": lambda: every.register_module_full_backward_hook(note)}.get(seen_by)
    try:
        handle = handle and handle()
        if seen_by == "instance forward":
            net.forward = lambda x: calls.append(1) or SingleVarianceNetwork.forward(net, x)
        elif seen_by == "class forward":
            own = SingleVarianceNetwork.forward
            monkeypatch.setattr(SingleVarianceNetwork, "forward", lambda m, x: calls.append(1) or own(m, x))
        inv_s = r._inv_s(torch.device("cpu"))
        inv_s.sum().backward()
    finally:
        if handle:
            handle.remove()
    assert calls and torch.equal(inv_s.detach(), plain)
    assert net.variance.grad is not None and float(net.variance.grad) == pytest.approx(10 * float(plain), rel=1e-6)


def test_step_inputs_are_copied_as_values(monkeypatch):
    """Every form of a batch's tensors arrives as its values; the ones that lie in
    memory as the inputs do go through the library's copy (here: its C semantics on
    host memory)."""
    import ctypes as C

    from supernormal_gb300 import trainer

    fused = []

    def copy_many(name, n, buffers, stream):
        assert name == "sn_copy_many"
        for b in list(buffers)[:n]:
            C.memmove(b.dst, b.src, 4 * b.n)
            fused.append(b.n)

    monkeypatch.setattr(trainer, "call", copy_many)
    monkeypatch.setattr(trainer, "stream_handle", lambda: 0)
    g = trainer.GraphStep.__new__(trainer.GraphStep)
    g.inputs = tuple(torch.zeros(4, 3) for _ in range(6))
    x = torch.arange(12.0).reshape(4, 3) + 1
    batch = (x, torch._neg_view(x), x.double(), x.T.contiguous().T, x[:1].expand(4, 3), x.flatten().as_strided((4, 3), (3, 1)))
    g._fill_inputs(batch)
    assert all(torch.equal(a, b.float()) for a, b in zip(g.inputs, batch)) and fused == [12, 12]
