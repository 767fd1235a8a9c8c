"""Kernels of the gated delta rule mixers vs plain PyTorch statements in 32 and 64 bits."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from tolerances import ELEMENTWISE, REDUCED, assert_close


def _close(a, b, name, reduced=False):
    assert_close(a, b, name=name, **(REDUCED if reduced else ELEMENTWISE))


@pytest.mark.parametrize("cuts,C,K", [([0, 1], 8, 4), ([0, 3, 4, 21], 16, 4), ([0, 16, 33], 1032, 2), ([0, 15, 31, 100], 2056, 3), ([0, 700], 264, 4)])
def test_causal_conv_silu(cuts, C, K):
    """Documents shorter than the kernel, cuts on and off the 16-row blocks, channel counts that leave threads idle."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(C)
    T = cuts[-1]
    x, dy = (torch.randn(T, C, device="cuda").bfloat16() for _ in range(2))
    w = (0.5 * torch.randn(C, K, device="cuda")).bfloat16()
    pos = torch.cat([torch.arange(b - a, device="cuda") for a, b in zip(cuts[:-1], cuts[1:])])
    a = [t.clone().requires_grad_() for t in (x, w)]
    y = ops.causal_conv_silu(*a, pos)
    g = torch.autograd.grad(y, a, dy)
    b = [t.double().requires_grad_() for t in (x, w)]
    z = []
    for s, e in zip(cuts[:-1], cuts[1:]):
        p = F.pad(b[0][s:e], (0, 0, K - 1, 0))
        z.append(sum(p[j:j + e - s] * b[1][:, j] for j in range(K)))
    want = F.silu(torch.cat(z))
    gw = torch.autograd.grad(want, b, dy.double())
    _close(y, want.float(), "y"); _close(g[0], gw[0].float(), "dx"); _close(g[1], gw[1].float(), "dw", True)


@pytest.mark.parametrize("T,Hk,Hv,d", [(1, 1, 1, 64), (7, 2, 6, 64), (33, 4, 8, 128), (5, 1, 2, 256)])
def test_delta_qkv(T, Hk, Hv, d):
    from torchllmtuner_b200 import ops
    torch.manual_seed(T)
    x = torch.randn(T, (2 * Hk + Hv) * d, device="cuda").bfloat16().requires_grad_()
    got = ops.delta_qkv(x, Hk, Hv, d, d, d ** -0.5, 1e-6)
    xd = x.detach().double().requires_grad_()
    q, k, v = xd[:, :Hk * d].view(T, Hk, d), xd[:, Hk * d:2 * Hk * d].view(T, Hk, d), xd[:, 2 * Hk * d:].view(T, Hv, d)
    q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    want = ((q * d ** -0.5).repeat_interleave(Hv // Hk, 1), k.repeat_interleave(Hv // Hk, 1), v)
    for a, b in zip(got, want):
        assert a.dtype == torch.float32 and torch.allclose(a.double(), b, rtol=1e-5, atol=1e-6)
    dys = [torch.randn_like(t) for t in got]
    (g,) = torch.autograd.grad(got, x, dys)
    (gw,) = torch.autograd.grad(want, xd, [t.double() for t in dys])
    _close(g, gw.float(), "dmixed")


@pytest.mark.parametrize("R,D", [(1, 64), (37, 128), (1000, 128), (65, 256)])
def test_gated_rms_norm(R, D):
    from torchllmtuner_b200 import ops
    torch.manual_seed(R)
    x, gate, dy = (torch.randn(R, D, device="cuda").bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    a = [t.clone().requires_grad_() for t in (x, gate, w)]
    y = ops.gated_rms_norm(*a, 1e-6)
    g = torch.autograd.grad(y, a, dy)
    b = [t.double().requires_grad_() for t in (x, gate, w)]
    want = b[0] * torch.rsqrt(b[0].square().mean(-1, keepdim=True) + 1e-6) * b[2] * F.silu(b[1])
    gw = torch.autograd.grad(want, b, dy.double())
    _close(y, want.float(), "y")
    for n, p, q in zip(("dx", "dgate", "dw"), g, gw):
        _close(p, q.float(), n, n == "dw")


def _shifted(t):
    """The same values in contiguous memory one element past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    v = flat[1:t.numel() + 1].view(t.shape)
    v.copy_(t)
    assert v.is_contiguous() and v.data_ptr() % 16
    return v


def _same_from_shifted(op, ins, dys):
    """`op` on operands and upstream gradients off the 16-byte boundary gives the bits that it gives for aligned ones."""
    def run(ins, dys):
        ins = [t.detach().requires_grad_() for t in ins]
        ys = op(*ins)
        ys = ys if isinstance(ys, tuple) else (ys,)
        return (*ys, *torch.autograd.grad(ys, ins, dys))
    want, got = run(ins, dys), run([_shifted(t) for t in ins], [_shifted(t) for t in dys])
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_gated_rms_norm_off_the_16_byte_boundary():
    from torchllmtuner_b200 import ops
    torch.manual_seed(1)
    x, gate, dy = (torch.randn(37, 128, device="cuda").bfloat16() for _ in range(3))
    w = torch.randn(128, device="cuda").bfloat16()
    _same_from_shifted(lambda *a: ops.gated_rms_norm(*a, 1e-6), (x, gate, w), (dy,))


def test_causal_conv_silu_on_any_positions():
    """Positions that no packed row has (negative, beyond the row's own index, jumping): the node takes what the tensor expressions take."""
    from torchllmtuner_b200.models.kimi_k3 import CausalConvolution
    torch.manual_seed(6)
    x, dy = (torch.randn(50, 16, device="cuda").bfloat16() for _ in range(2))
    conv = CausalConvolution(16, 4, dtype=torch.float32, device="cuda")
    torch.nn.init.normal_(conv.weight)
    conv.weight.data.copy_(conv.weight.data.bfloat16())
    low = CausalConvolution(16, 4, dtype=torch.bfloat16, device="cuda")
    low.load_state_dict(conv.state_dict())
    pos = torch.randint(-2, 5, (50,), device="cuda")
    a, b = x.clone().requires_grad_(), x.float().requires_grad_()
    y, want = low(a, pos), conv(b, pos)
    g, gw = torch.autograd.grad(y, [a, low.weight], dy), torch.autograd.grad(want, [b, conv.weight], dy.float())
    _close(y, want, "y"); _close(g[0], gw[0], "dx"); _close(g[1], gw[1], "dw", True)


@pytest.mark.parametrize("T,C", [(65536, 16), (65537, 16), (1048640, 8)])
def test_causal_conv_silu_on_long_rows(T, C):
    """Rows on both sides of the length from which a block walks more than 16 of them, and more than 65535 blocks of 16 would cover:
    against the convolution of the library in fp32, cut into documents of 1000 rows."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(5)
    x, dy = (torch.randn(T, C, device="cuda").bfloat16() for _ in range(2))
    w, pos = torch.randn(C, 4, device="cuda").bfloat16(), torch.arange(T, device="cuda") % 1000
    a = [t.clone().requires_grad_() for t in (x, w)]
    y = ops.causal_conv_silu(*a, pos)
    g = torch.autograd.grad(y, a, dy)
    b = [t.float().requires_grad_() for t in (x, w)]
    z = sum(torch.where((pos >= j)[:, None], F.pad(b[0], (0, 0, j, 0))[:T], 0.0) * b[1][:, 3 - j] for j in range(4))
    want = F.silu(z)
    gw = torch.autograd.grad(want, b, dy.float())
    _close(y, want, "y"); _close(g[0], gw[0], "dx"); _close(g[1], gw[1], "dw", True)


def test_causal_conv_silu_off_the_16_byte_boundary():
    from torchllmtuner_b200 import ops
    torch.manual_seed(2)
    x, dy = (torch.randn(37, 264, device="cuda").bfloat16() for _ in range(2))
    w, pos = torch.randn(264, 4, device="cuda").bfloat16(), torch.arange(37, device="cuda")
    _same_from_shifted(lambda x, w: ops.causal_conv_silu(x, w, pos), (x, w), (dy,))


def test_delta_qkv_off_the_16_byte_boundary():
    from torchllmtuner_b200 import ops
    torch.manual_seed(3)
    x, dys = torch.randn(37, 8 * 64, device="cuda").bfloat16(), [torch.randn(37, 4, 64, device="cuda") for _ in range(3)]
    _same_from_shifted(lambda x: ops.delta_qkv(x, 2, 4, 64, 64, 0.125, 1e-6), (x,), dys)


@pytest.mark.parametrize("T,H,d", [(1, 1, 64), (63, 2, 128), (64, 3, 64), (65, 2, 128), (300, 2, 64), (700, 1, 128)])
@pytest.mark.parametrize("decay", [0.05, 3.0])
def test_delta_rule_kernels_match_the_scan_in_64_bits(T, H, d, decay):
    """Forward and all five gradients against the token-by-token recurrence in 64 bits, at lengths around the 64-token chunk and
    with weak and strong decay. fp32 sums of a few hundred terms of unit size: 2e-5 of the root mean square."""
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.models.families import delta_rule_scan
    g = torch.Generator(device="cuda").manual_seed(T + d)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = [F.normalize(r(T, H, d), dim=-1), F.normalize(r(T, H, d), dim=-1), r(T, H, d), torch.rand(T, H, generator=g, device="cuda"),
         -decay * F.softplus(r(T, H, 1))]
    do = r(T, H, d)
    a = [t.clone().requires_grad_() for t in x]
    o = ops.delta_rule(*a)
    got = (o, *torch.autograd.grad(o, a, do))
    b = [t.double().requires_grad_() for t in x]
    ow = delta_rule_scan(*b)
    want = (ow, *torch.autograd.grad(ow, b, do.double()))
    for n, p, q in zip(("o", "dq", "dk", "dv", "dbeta", "dlog_decay"), got, want):
        assert p.shape == q.shape
        err = (p.double() - q).abs().max() / q.square().mean().sqrt().clamp_min(1e-6)
        assert err < 2e-5 * max(1.0, float(q.detach().abs().max() / q.detach().square().mean().sqrt().clamp_min(1e-6))), (n, float(err))
    o2 = ops.delta_rule(*a)
    for p, q in zip(got, (o2, *torch.autograd.grad(o2, a, do))):
        assert torch.equal(p, q)                       # no atomics
    with torch.no_grad():
        assert torch.equal(ops.delta_rule(*x), o)      # the form without a backward


@pytest.mark.parametrize("H,d", [(2, 64), (1, 128)])
def test_long_documents_of_few_heads_take_the_expressions(H, d):
    """Both sides of the rule that sends a long document with few heads to the tensor expressions, and the two forms against each other
    beyond it (each within 2e-5 of 64 bits at the lengths above; the states of a thousand chunks decay, so length adds nothing)."""
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.models.families import chunked_delta_rule
    from torchllmtuner_b200.ops.functional import _DeltaRule
    g = torch.Generator(device="cuda").manual_seed(d)
    T = (1 << 22) // d + 1
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = [F.normalize(r(T, H, d), dim=-1), F.normalize(r(T, H, d), dim=-1), r(T, H, d), torch.rand(T, H, generator=g, device="cuda"), -F.softplus(r(T, H, 1))]
    x = [t.requires_grad_() for t in x]
    assert ops.delta_rule(*x) is None and ops.delta_rule(*(t[:-1] for t in x)) is not None
    with torch.no_grad():
        assert ops.delta_rule(*(t[:-1] for t in x)) is None and ops.delta_rule(*(t[:(1 << 21) // d] for t in x)) is not None
    many = [t.detach().repeat_interleave(4, 1).requires_grad_() for t in x]
    assert ops.delta_rule(*many) is not None
    do = r(T, H, d)
    a, b = _DeltaRule.apply(*x, None), chunked_delta_rule(*x)
    for p, q in zip((a, *torch.autograd.grad(a, x, do)), (b, *torch.autograd.grad(b, x, do))):
        assert (p - q).norm() <= 4e-5 * q.norm()


def test_second_derivatives_and_transforms_of_the_delta_rule():
    """What the node cannot do stays with the tensor expressions: a gradient of the gradient, forward-mode derivatives and vmap give
    what 64 bits give (a second derivative sums a few thousand fp32 terms of its own size: 1e-4 of the largest)."""
    from torchllmtuner_b200.models.families import chunked_delta_rule
    g = torch.Generator(device="cuda").manual_seed(5)
    T, H, d = 70, 2, 64
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x = [F.normalize(r(T, H, d), dim=-1), F.normalize(r(T, H, d), dim=-1), r(T, H, d), torch.rand(T, H, generator=g, device="cuda"),
         -F.softplus(r(T, H, 1))]

    def second(a):
        a = [t.clone().requires_grad_() for t in a]
        first = torch.autograd.grad(chunked_delta_rule(*a).square().sum(), a, create_graph=True)
        return (*first, *torch.autograd.grad(sum(t.square().sum() for t in first), a))

    tangent = r(T, H, d)
    forward = lambda a, t: torch.func.jvp(lambda v: chunked_delta_rule(a[0], a[1], v, a[3], a[4]), (a[2],), (t,))  # noqa: E731
    mapped = lambda a: torch.func.vmap(lambda v: chunked_delta_rule(a[0], a[1], v, a[3], a[4]))(torch.stack((a[2], 2 * a[2])))  # noqa: E731
    y = [t.double() for t in x]
    got, want = (*second(x), *forward(x, tangent), mapped(x)), (*second(y), *forward(y, tangent.double()), mapped(y))
    for p, q in zip(got, want):
        assert (p.double() - q).abs().max() <= 1e-4 * q.abs().max()


@pytest.mark.parametrize("cuts", [[0, 200], [0, 1, 70, 134, 200], [0, 64, 129, 193]])
@pytest.mark.parametrize("Hk,Hv,d", [(2, 4, 64), (1, 3, 128)])
def test_mixer_over_packed_documents(cuts, Hk, Hv, d):
    """The whole mixer on several documents in one row (three heads: the decay rows of a later document start off the 16-byte boundary)
    against the same weights in fp32 on the CPU: output and every gradient. The intermediate tensors of the device are bf16: a dozen
    roundings of 2^-9 between input and the farthest gradient, 2e-2 of the norm (0.009 measured with the same modules in bf16 on the CPU;
    A_log and dt_bias are sums of a few hundred signed terms that cancel to a third of their size: three times that, 0.023)."""
    from torchllmtuner_b200.models.qwen3_5 import GatedDeltaNet, Qwen35Config, Qwen35Context
    from torchllmtuner_b200.ops import AttnMeta
    torch.manual_seed(d + Hk)
    T, D = cuts[-1], 128
    cfg = Qwen35Config(hidden_size=D, linear_num_value_heads=Hv, linear_num_key_heads=Hk, linear_key_head_dim=d, linear_value_head_dim=d)
    cpu = GatedDeltaNet(cfg, dtype=torch.float32)
    for n, p in cpu.named_parameters():
        torch.nn.init.normal_(p, mean=1.0 if n == "norm.weight" else 0.0, std=0.1 if n in ("norm.weight", "A_log", "dt_bias") else 0.08)
        p.data.copy_(p.data.bfloat16().float())
    gpu = GatedDeltaNet(cfg, dtype=torch.bfloat16, device="cuda")
    gpu.load_state_dict(cpu.state_dict())
    x, dy = torch.randn(T, D).bfloat16(), torch.randn(T, D).bfloat16()
    pos = torch.cat([torch.arange(b - a) for a, b in zip(cuts[:-1], cuts[1:])])

    def run(module, x, dy, dev):
        x = x.to(dev).requires_grad_()
        ctx = Qwen35Context(None, None, AttnMeta.build(cuts, causal=True, device=dev), positions=pos.to(dev))
        y = module(x, ctx)
        return (y, *torch.autograd.grad(y, [x, *module.parameters()], dy.to(dev)))
    for n, a, b in zip(("y", "x", *(n for n, _ in cpu.named_parameters())), run(gpu, x, dy, "cuda"), run(cpu, x.float(), dy.float(), "cpu")):
        err = (a.detach().float().cpu() - b.detach()).norm() / b.detach().norm()
        assert err < (6e-2 if n in ("A_log", "dt_bias") else 2e-2), (n, float(err))
