"""What the autograd nodes hand to the kernels: 16-byte loads need rows on 16-byte boundaries, whatever views a caller passes. The kernel
library is replaced by a recorder, so a wrong address shows here and never reaches a device."""
import pytest
import torch

from torchllmtuner_b200.ops import functional as F


class Recorder:
    """Stands in for the extension: answers with zeros, keeps the operands of the last call of each name and the places of all that were off a boundary."""

    def __init__(self, **answers):
        self.answers, self.seen, self.off = answers, {}, []

    def __getattr__(self, name):
        def call(*args):
            self.seen[name] = [a for a in args if isinstance(a, torch.Tensor)]
            self.off += [(name, i) for i, t in enumerate(self.seen[name]) if t.dtype != torch.int64 and t.data_ptr() % 16]
            return self.answers[name](*args)
        return call


def shifted(*shape, dtype=torch.bfloat16, by=1):
    """A contiguous tensor whose first element is `by` elements past a 16-byte boundary."""
    n = 1
    for s in shape:
        n *= s
    flat = torch.randn(n + 16).to(dtype)
    start = next(i for i in range(16) if flat[i:].data_ptr() % 16 == by * flat.element_size())
    t = flat[start:start + n].view(shape)
    assert t.is_contiguous() and t.data_ptr() % 16
    return t


def zeros(*like):
    return lambda *args: tuple(torch.zeros_like(args[i]) for i in like)


def test_gated_norm_operands(monkeypatch):
    ext = Recorder(gated_norm_fwd=lambda x, gate, w, eps: torch.zeros_like(x), gated_norm_bwd=zeros(1, 2, 3))
    monkeypatch.setattr(F, "_ext", lambda: ext)
    x, gate, w = shifted(5, 64).requires_grad_(), shifted(5, 64).requires_grad_(), torch.randn(64, 2).bfloat16()[:, 0].requires_grad_()
    F._GatedRMSNorm.apply(x, gate, w, 1e-6, None).backward(shifted(5, 64))
    assert set(ext.seen) == {"gated_norm_fwd", "gated_norm_bwd"} and not ext.off
    assert all(t.is_contiguous() for ts in ext.seen.values() for t in ts)
    assert torch.equal(ext.seen["gated_norm_fwd"][0], x)


def test_convolution_operands(monkeypatch):
    ext = Recorder(conv_silu_fwd=lambda x, w, pos: torch.zeros_like(x), conv_silu_bwd=lambda dy, x, w, pos: (torch.zeros_like(x), torch.zeros_like(w)))
    monkeypatch.setattr(F, "_ext", lambda: ext)
    for x in (shifted(5, 16), torch.randn(1, 17).bfloat16()[:, :16], torch.randn(16, 5).bfloat16().t()):      # off the boundary, odd row stride, column-major
        F._ConvSiLU.apply(x.requires_grad_(), torch.randn(16, 4).bfloat16().requires_grad_(), torch.arange(x.shape[0]), None).backward(shifted(*x.shape))
        assert set(ext.seen) == {"conv_silu_fwd", "conv_silu_bwd"} and not ext.off
        assert all(t.stride(1) == 1 and t.stride(0) % 8 == 0 for t in (ext.seen["conv_silu_fwd"][0], *ext.seen["conv_silu_bwd"][:2]))


def test_delta_qkv_operands(monkeypatch):
    ext = Recorder(delta_qkv_fwd=lambda m, Hk, Hv, scale, eps: [torch.zeros(m.shape[0], Hv, 64) for _ in range(3)],
                   delta_qkv_bwd=lambda dq, dk, dv, m, *cfg: torch.zeros_like(m))
    monkeypatch.setattr(F, "_ext", lambda: ext)
    ys = F._DeltaQKV.apply(shifted(5, 4 * 64).requires_grad_(), 1, 2, 0.125, 1e-6, None)
    torch.autograd.backward(ys, [shifted(5, 2, 64, dtype=torch.float32) for _ in ys])
    assert set(ext.seen) == {"delta_qkv_fwd", "delta_qkv_bwd"} and not ext.off


def test_wide_attention_upstream_gradient(monkeypatch):
    from torchllmtuner_b200.ops import AttnMeta
    ext = Recorder(attn_bwd_wide=lambda q, k, v, *rest: (torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)))
    monkeypatch.setattr(F, "_ext", lambda: ext)
    meta = AttnMeta.build([0, 5], device="cpu")
    meta.q_tiles, meta.k_tile_passes = torch.zeros(1, 8, dtype=torch.int32), [torch.zeros(1, 8, dtype=torch.int32)]
    q, k, v = (torch.randn(5, 1, 256).bfloat16().requires_grad_() for _ in range(3))
    kept = (torch.randn(5, 1, 256).bfloat16(), torch.randn(1, 5))
    for do in (shifted(5, 1, 256), torch.randn(5, 1, 260).bfloat16()[..., :256]):        # off the boundary, odd row stride
        o, _ = F._Attention.apply(q, k, v, meta, 0.0625, kept)
        o.backward(do)
        assert not ext.off and ext.seen["attn_bwd_wide"][4].stride() == (256, 256, 1) and torch.equal(ext.seen["attn_bwd_wide"][4], do)


def test_grouped_projection_upstream_gradients(monkeypatch):
    from torchllmtuner_b200.models.moe import experts
    ext = Recorder(grouped_gemm=lambda *a: None, grouped_wgrad=lambda *a: None)
    monkeypatch.setattr(experts, "_ext", lambda: ext)
    x, ws = torch.randn(128, 16).bfloat16().requires_grad_(), [torch.randn(1, 24, 16).bfloat16().requires_grad_() for _ in range(2)]
    ys = experts._GroupedLinear.apply(x, torch.tensor([0, 128], dtype=torch.int32), *ws)
    torch.autograd.backward(ys, [shifted(128, 24), torch.randn(128, 49).bfloat16()[:, :24]])
    assert set(ext.seen) == {"grouped_gemm", "grouped_wgrad"} and not ext.off


def _batched(call, *ins):
    """Gradients of three upstream gradients at once against one after another."""
    ins = [t.detach().requires_grad_() for t in ins]
    ys = call(*ins)
    ys = ys if isinstance(ys, tuple) else (ys,)
    dys = [torch.randn(3, *y.shape).to(y.dtype) for y in ys]
    return torch.autograd.grad(ys, ins, dys, is_grads_batched=True, retain_graph=True), ins, [[d[i] for d in dys] for i in range(3)]


def test_batched_upstream_gradients_take_the_expressions(monkeypatch):
    """`is_grads_batched` hands a backward tensors without memory: no kernel is called with one, and the result is that of the expressions."""
    from torchllmtuner_b200.models.families import _chunk_expressions
    from torchllmtuner_b200.models.qwen3_5 import GatedRMSNorm
    zero = lambda t: lambda *a: torch.zeros_like(t)  # noqa: E731
    x, z, w = torch.randn(5, 64), torch.randn(5, 64), torch.randn(64)
    q, k, v = (torch.randn(70, 2, 64) for _ in range(3))
    beta, decay = torch.rand(70, 2), -torch.rand(70, 2, 1)
    norm = lambda x, z, w: GatedRMSNorm._expressions(x, z, w, 1e-6)  # noqa: E731
    conv = lambda x, w, pos: (x * w[:, 0]).sin()  # noqa: E731
    rule = lambda *a: _chunk_expressions(*a, 64)  # noqa: E731
    split = lambda m: (m[:, :64].sin(), m[:, 64:128].cos(), m[:, 128:])  # noqa: E731
    nodes = {"norm": ((x, z, w), dict(gated_norm_fwd=zero(x)), lambda *a: F._GatedRMSNorm.apply(*a, 1e-6, lambda *b: GatedRMSNorm._expressions(*b)), norm),
             "conv": ((x, torch.randn(64, 4)), dict(conv_silu_fwd=zero(x)), lambda x, w: F._ConvSiLU.apply(x, w, torch.arange(5), conv), lambda x, w: conv(x, w, None)),
             "qkv": ((torch.randn(5, 192),), dict(delta_qkv_fwd=lambda *a: [torch.zeros(5, 64) for _ in range(3)]),
                     lambda m: F._DeltaQKV.apply(m, 1, 1, 1.0, 1e-6, split), split),
             "rule": ((q, k, v, beta, decay), dict(delta_rule_fwd=lambda *a: [torch.zeros_like(v)]), lambda *a: F._DeltaRule.apply(*a, rule), rule)}
    for name, (ins, answers, call, statement) in nodes.items():
        ext = Recorder(**answers)
        monkeypatch.setattr(F, "_ext", lambda: ext)
        got, leaves, dys = _batched(call, *ins)
        for i in range(3):
            for a, b in zip(got, torch.autograd.grad(statement(*leaves), leaves, dys[i])):
                assert torch.allclose(a[i], b, rtol=1e-4, atol=1e-5), name
        assert set(ext.seen) == set(answers)


def test_batched_gradients_of_the_losses_take_the_expressions(monkeypatch):
    ext = Recorder(ce_fwd_bwd=lambda work, *a: (torch.ones(work.shape[0]), None), gemm=lambda a, b, out, *rest: out.fill_(2.0))
    monkeypatch.setattr(F, "_ext", lambda: ext)
    target = torch.zeros(8, dtype=torch.int64)
    for call, ins in ((lambda t: F._CrossEntropySum.apply(t, target), (torch.randn(8, 16).bfloat16(),)),
                      (lambda h, w: F._LinearCrossEntropy.apply(h, w, target, 1), (torch.randn(8, 16).bfloat16(), torch.randn(24, 16).bfloat16()))):
        got, leaves, dys = _batched(call, *ins)
        for i in range(3):
            for a, b, t in zip(got, torch.autograd.grad(call(*leaves), leaves, dys[i], create_graph=True), leaves):
                assert a[i].shape == t.shape and torch.equal(a[i], b)


@pytest.mark.parametrize("owner,name", [(torch._C._functorch, "peek_interpreter_stack"), (torch._C, "_len_torch_dispatch_stack"),
                                        (torch.autograd.forward_ad, "_current_level")])
def test_a_torch_without_the_private_queries_takes_the_expressions(monkeypatch, owner, name):
    assert F._has_rules(torch.ones(1))
    monkeypatch.delattr(owner, name)
    monkeypatch.setattr(F, "_NO_TRANSFORM", F._transform_probes())
    assert not F._has_rules(torch.ones(1))
