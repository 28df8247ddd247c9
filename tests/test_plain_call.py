"""Which eager calls go round the custom ops' wrapping (ops.plain_call), and that the others still reach the registered op."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.profiler import ProfilerActivity, profile

from tests.scan_cases import make_inputs


class Watch(TorchFunctionMode):
    def __init__(self):
        super().__init__()
        self.seen = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.seen.append(str(func))
        return func(*args, **(kwargs or {}))


def test_what_is_a_plain_call():
    from slotscan_b200.ops import plain_call, plain_grads
    x = torch.zeros(3, requires_grad=True)
    assert plain_call(x, None, torch.nn.Parameter(x.detach()))
    assert not plain_call(x, torch._neg_view(x))
    got = []

    class Probe(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x * 2

        @staticmethod
        def backward(ctx, g):
            got.append(plain_grads(g))
            return g * 2
    torch.autograd.grad(Probe.apply(x), x, torch.ones(2, 3), is_grads_batched=True)
    torch.autograd.grad(Probe.apply(x), x, torch.ones(3))
    assert got == [False, True]
    with Watch():
        assert not plain_call(x)
    with torch.device("cpu"):
        assert plain_call(x)
        with Watch():
            assert not plain_call(x)
    with profile(activities=[ProfilerActivity.CPU]):
        assert not plain_call(x)
    assert plain_call(x)


def _call(mode, x):
    import slotscan_b200 as S
    k, q, v, g, fr = x
    N, G = 24, 8
    if mode == "keyless":
        wa = torch.randn(*g.shape, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
        return [S.slot_scan_v(v, wa, g, 2.0, N, G=G)]
    if mode == "read":
        kb, vb, kinv, valid = S.write_memory(k.detach(), v.detach(), g.detach(), fr.detach(), N, 16.0, G=G, q=q.detach(),
                                             occ_bin=True, out_dtype=torch.float32)
        return [S.read_snapshots(q.unsqueeze(3), g.unsqueeze(3) + 1, kb, vb, kinv, valid, G)]
    return list(S.kv_scan_g(k, v, g, fr, N, 16.0, G=G, hard=mode == "hard", detach_addr=True, q=q, occ_bin=True))


@pytest.mark.gpu
@pytest.mark.parametrize("mode,op", [("hard", "hard_fwd"), ("soft", "dense_fwd"), ("keyless", "keyless_fwd"), ("read", "read_fwd")])
def test_batched_gradients_modes_and_profiles(mode, op):
    """Three upstream gradients in one batched call give the bits of three calls; a function mode and a profile see the op; a
    lazily negated input is read negated."""
    inp = make_inputs("clustered", 2, 40, 2, 64, 64, seed=3)
    x = [inp[n].cuda().requires_grad_() for n in ("k", "q", "v", "gate", "fr")]
    out = _call(mode, x)
    gen = torch.Generator(device="cuda").manual_seed(2)
    ups = [torch.randn(3, *o.shape, device="cuda", generator=gen) for o in out]
    many = torch.autograd.grad(out, x, ups, is_grads_batched=True, allow_unused=True, retain_graph=True)
    for i in range(3):
        one = torch.autograd.grad(out, x, [u[i] for u in ups], allow_unused=True, retain_graph=True)
        for a, b in zip(many, one):
            assert (a is None) == (b is None) and (a is None or torch.equal(a[i], b))
    plain = [t.detach() for t in x]
    with Watch() as w:
        _call(mode, plain)
    assert any(op in s for s in w.seen)
    with profile(activities=[ProfilerActivity.CPU]) as pr:
        _call(mode, plain)
    assert any("slotscan::" + op in e.key for e in pr.key_averages())
    i = 1 if mode == "read" else 2                            # the query of a read, else the values
    want = _call(mode, plain)
    plain[i] = torch._neg_view(-plain[i])
    for a, b in zip(want, _call(mode, plain)):
        assert torch.equal(a, b)
