"""Memory-bound sm_100a kernels vs the plain PyTorch fp32 statements in ops/reference.py."""
import pytest
import torch

pytestmark = pytest.mark.gpu


from tolerances import ELEMENTWISE, REDUCED, assert_close, f32_leaves


def _close(a, b, kind=None, name="tensor"):
    """`kind` None: one-rounding element-wise result; "reduced": a sum over rows of bf16-rounded terms (weight gradients,
    gradients that pass through bf16 logits)."""
    assert_close(a, b, name=name, **(REDUCED if kind else ELEMENTWISE))


def _grads(fn, inputs, seed=0):
    torch.manual_seed(seed)
    outs = fn(*inputs)
    outs = outs if isinstance(outs, tuple) else (outs,)
    gs = [torch.randn_like(o.float()).bfloat16().to(o.dtype) for o in outs]  # same bf16-rounded upstream grads for both arms
    grads = torch.autograd.grad(outs, [i for i in inputs if i.requires_grad], gs, allow_unused=True)
    return outs, grads


@pytest.mark.parametrize("T,D", [(64, 256), (1000, 4096), (33, 2048), (7, 64), (129, 8192)])
def test_rmsnorm_and_add(T, D):
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(0)
    x = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    r = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16().requires_grad_()
    o1, g1 = _grads(lambda a, b: ops.rms_norm(a, b, 1e-6), [x, w])
    o2, g2 = _grads(lambda a, b: ref.rms_norm(a, b, 1e-6), f32_leaves(x, w))
    _close(o1[0], o2[0], name="y"); _close(g1[0], g2[0], name="dx"); _close(g1[1], g2[1], "reduced", "dw")
    o1, g1 = _grads(lambda a, b, c: ops.add_rms_norm(a, b, c, 1e-6), [x, r, w])
    o2, g2 = _grads(lambda a, b, c: ref.add_rms_norm(a, b, c, 1e-6), f32_leaves(x, r, w))
    names = ("y", "sum", "dx", "dres", "dw")
    for n, a, b in zip(names, o1 + tuple(g1), o2 + tuple(g2)):
        _close(a, b, "reduced" if n == "dw" else None, n)


@pytest.mark.parametrize("T,Hq,Hkv,d", [(128, 4, 2, 64), (300, 32, 8, 128), (17, 2, 1, 256)])
@pytest.mark.parametrize("with_norm", [True, False])
def test_qk_norm_rope(T, Hq, Hkv, d, with_norm):
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(0)
    qkv = torch.randn(T, (Hq + 2 * Hkv) * d, device="cuda").bfloat16().requires_grad_()
    qw = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16().requires_grad_() if with_norm else None
    kw = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16().requires_grad_() if with_norm else None
    cos, sin = ops.rope_tables(torch.arange(T, device="cuda"), d, 1e6)

    def run(fn):
        q = qkv[:, :Hq * d].view(T, Hq, d)
        k = qkv[:, Hq * d:(Hq + Hkv) * d].view(T, Hkv, d)
        return fn(q, k, qw, kw, cos, sin, 1e-6)
    ins = [qkv] + ([qw, kw] if with_norm else [])
    o1, g1 = _grads(lambda *a: run(ops.qk_norm_rope), ins)
    o2, g2 = _grads(lambda *a: run(ref.qk_norm_rope), ins)
    names = ("q", "k", "dqkv", "dqw", "dkw")
    for n, a, b in zip(names, o1 + tuple(g1), o2 + tuple(g2)):
        _close(a, b, "reduced" if n in ("dqw", "dkw") else None, n)


def test_qk_norm_weight_gradient_is_the_same_bits_on_every_call():
    """The per-block partial sums of the norm-weight gradient are combined in a fixed order (no atomic adds), so repeated
    calls on the same inputs agree bit for bit: what the reproducible training mode relies on."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(1)
    T, Hq, Hkv, d = 4096, 8, 2, 128
    qkv = torch.randn(T, (Hq + 2 * Hkv) * d, device="cuda").bfloat16().requires_grad_()
    qw = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16().requires_grad_()
    kw = (1 + 0.1 * torch.randn(d, device="cuda")).bfloat16().requires_grad_()
    cos, sin = ops.rope_tables(torch.arange(T, device="cuda"), d, 1e6)
    gq, gk = torch.randn(T, Hq, d, device="cuda").bfloat16(), torch.randn(T, Hkv, d, device="cuda").bfloat16()
    seen = []
    for _ in range(8):
        q, k = ops.qk_norm_rope(qkv[:, :Hq * d].view(T, Hq, d), qkv[:, Hq * d:(Hq + Hkv) * d].view(T, Hkv, d), qw, kw, cos, sin, 1e-6)
        seen.append(torch.autograd.grad([q, k], [qw, kw, qkv], [gq, gk]))
    for other in seen[1:]:
        for a, b in zip(seen[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("T,F", [(256, 768), (1000, 12288), (3, 64)])
def test_swiglu(T, F):
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(0)
    gu = torch.randn(T, 2 * F, device="cuda").bfloat16().requires_grad_()
    o1, g1 = _grads(lambda a: ops.swiglu(a[:, :F], a[:, F:]), [gu])
    o2, g2 = _grads(lambda a: ref.swiglu(a[:, :F], a[:, F:]), [gu])
    _close(o1[0], o2[0]); _close(g1[0], g2[0])


@pytest.mark.parametrize("T,D,V,chunks", [(256, 128, 1000, 1), (500, 256, 32000, 3), (128, 64, 151936, 1)])
def test_linear_cross_entropy(T, D, V, chunks):
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    from torchllmtuner_b200.ops.cuda_ext import check_status
    torch.manual_seed(0)
    h = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, D, device="cuda")).bfloat16().requires_grad_()
    y = torch.randint(0, V, (T,), device="cuda")
    y[::7] = -100
    l1 = ops.linear_cross_entropy_sum(h, w, y, chunks)
    g1 = torch.autograd.grad(l1 / 100.0, [h, w])
    check_status("ce")
    l2 = ref.linear_cross_entropy_sum(h.float(), w.float(), y, chunks)
    g2 = torch.autograd.grad(l2 / 100.0, [h, w])
    assert abs(l1.item() - l2.item()) / abs(l2.item()) < 5e-3
    _close(g1[0], g2[0], "reduced", "dh"); _close(g1[1], g2[1], "reduced", "dw")
    lg = (h.float() @ w.float().t()).bfloat16().requires_grad_()
    l3 = ops.cross_entropy_sum(lg, y)
    (g3,) = torch.autograd.grad(l3, [lg])
    l4 = ref.cross_entropy_sum(lg.float(), y)
    (g4,) = torch.autograd.grad(l4, [lg])
    assert abs(l3.item() - l4.item()) / abs(l4.item()) < 5e-3
    _close(g3, g4, name="dlogits")


def test_adamw_and_sqnorm():
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(0)
    n = 1_000_003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda").bfloat16()
    m, v = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    p16 = p.bfloat16()
    pr, mr, vr = p.clone(), m.clone(), v.clone()
    coef = torch.tensor([0.5], device="cuda")
    for step in (1, 2, 3):
        ops.adamw_step_(p, g, m, v, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step, p_lowp=p16, clip_coef=coef)
        ref.adamw_step_(pr, g, mr, vr, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step, grad_scale=0.5)
    assert (p - pr).abs().max().item() < 1e-4
    assert torch.equal(p16, p.bfloat16())
    a, b = torch.randn(300_001, device="cuda").bfloat16(), torch.randn(77, device="cuda")
    s1 = ops.sq_norm([a, b])
    s2 = a.float().pow(2).sum() + b.pow(2).sum()
    assert abs(s1.item() - s2.item()) / s2.item() < 1e-4
    assert torch.equal(ops.sq_norm([a, b]), s1)


@pytest.mark.parametrize("rows,V,shards", [(300, 1000, 1), (128, 2007, 3), (64, 18992, 2)])
def test_vocab_parallel_cross_entropy_kernel_on_one_gpu(rows, V, shards):
    """`ce_vocab_parallel` with all R vocabulary shards of a row on this one GPU. Launches on one GPU may not wait on one
    another, so the shards run in two passes over tables that are plain device tensors: the first pass (flags pre-set, no
    gradient) only publishes every shard's (max, sum-exp, target) triple, the second pass finds all R triples present,
    combines them and writes the gradient. Loss and gradient must equal the full-vocabulary fp32 statement."""
    from torchllmtuner_b200.ops.cuda_ext import load
    from torchllmtuner_b200.ops import reference as ref
    ext = load()
    torch.manual_seed(0)
    full = (torch.randn(rows, V, device="cuda") * 2).bfloat16()
    labels = torch.randint(0, V, (rows,), device="cuda")
    labels[::9] = -100
    chunk = -(-V // shards)
    chunk = -(-chunk // 8) * 8
    # one table set per "rank": stats [R][rows] float4, flags [R][rows] uint32
    stats = [torch.zeros(shards * rows * 4, device="cuda") for _ in range(shards)]
    flags = [torch.zeros(shards * rows, dtype=torch.int32, device="cuda") for _ in range(shards)]
    sp, fp = [s.data_ptr() for s in stats], [f.data_ptr() for f in flags]
    # pass 1: publish every shard's triple (flags pre-set so that nothing waits), pass 2: the real run
    for f in flags:
        f.fill_(1)
    work = []
    for r in range(shards):
        lo, hi = r * chunk, min(V, (r + 1) * chunk)
        buf = torch.zeros(rows, chunk, dtype=torch.bfloat16, device="cuda")
        buf[:, : hi - lo] = full[:, lo:hi]
        work.append((lo, hi, buf))
    for grad_pass in (False, True):
        losses = []
        for r, (lo, hi, buf) in enumerate(work):
            losses.append(ext.ce_vocab_parallel(buf[:, : hi - lo], labels, lo, r, sp, fp, rows, 1, 1.0, -100, grad_pass))
    torch.cuda.synchronize()
    from torchllmtuner_b200.ops.cuda_ext import check_status
    check_status("ce_vocab_parallel")
    lf = full.float().requires_grad_()
    want = ref.cross_entropy_sum(lf, labels)
    (g,) = torch.autograd.grad(want, [lf])
    for l in losses:      # every shard reports the same full-vocabulary row losses
        assert abs(l.sum().item() - want.item()) / abs(want.item()) < 2e-3
    got = torch.cat([buf[:, : hi - lo] for lo, hi, buf in work], dim=1)
    _close(got, g, name="dlogits")


@pytest.mark.parametrize("D", [8, 504, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("T", [1, 3, 301])
def test_rmsnorm_at_the_edges_of_the_row_groups(T, D):
    """Widths on both sides of each row-group size (32, 64, 128, 256, 512 threads per row) and row counts that leave groups of a
    block without a row. The weight gradient comes back in bf16 from the summing kernel: the fp32 sum rounded once."""
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    from torchllmtuner_b200.ops.cuda_ext import load
    torch.manual_seed(T + D)
    x, r, dy, ds = (torch.randn(T, D, device="cuda").bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    a = [t.clone().requires_grad_() for t in (x, r, w)]
    b = f32_leaves(*a)
    got = torch.autograd.grad(ops.add_rms_norm(*a, 1e-6), a, [dy, ds])
    want = torch.autograd.grad(ref.add_rms_norm(*b, 1e-6), b, [dy.float(), ds.float()])
    for n, p, q in zip(("dx", "dres", "dw"), got, want):
        _close(p, q, "reduced" if n == "dw" else None, n)
    y, rstd, s = load().rmsnorm_fwd(x, r, w, 1e-6)
    _, dw32 = load().rmsnorm_bwd(dy, s, w, rstd, ds)
    assert torch.equal(dw32.bfloat16(), got[2])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 7, 8, 255, 257, 4097, 303104, 303105, 5000003, 20000008,
                               # 1 to 31 steps of 303104 elements and a few more: every combination of batch sizes
                               *(303104 * k + 4 * k + 3 for k in (1, 2, 3, 5, 7, 10, 15, 16, 23, 31))])
def test_sq_norm_has_the_same_bits_on_any_alignment(n, dtype):
    """The kernel for 16-byte aligned data and the one for any slice add the same terms in the same order: equal bits. Thousands of
    fp32 terms per partial sum stay within 1e-5 of the 64-bit sum."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(n)
    x = torch.randn(n, device="cuda").to(dtype)
    moved = torch.empty(n + 1, device="cuda", dtype=dtype)[1:].copy_(x)
    got, want = ops.sq_norm([x]), x.double().square().sum()
    assert torch.equal(got, ops.sq_norm([moved]))
    assert abs(float(got) - float(want)) <= 1e-5 * float(want)


@pytest.mark.parametrize("rows,V", [(1, 8), (3, 17), (5, 4096), (4, 8192), (4, 8208), (3, 20480), (3, 20520), (2, 76800), (2, 76808), (2, 151936)])
@pytest.mark.parametrize("mask", [None, float("-inf"), torch.finfo(torch.bfloat16).min])
def test_cross_entropy_kernel_at_its_size_limits(rows, V, mask):
    """Both sides of each thread-count and shared-memory-cache limit, rows that end off a vector, labels in the last column, rows
    without a label, and a masked stretch that covers whole threads. Gradients are one bf16 rounding of fp32 values."""
    from torchllmtuner_b200.ops.cuda_ext import load
    torch.manual_seed(V)
    ld = -(-V // 8) * 8
    x = torch.randn(rows, ld, device="cuda").mul_(3).bfloat16()[:, :V]
    y = torch.randint(0, V, (rows,), device="cuda")
    y[0] = V - 1
    if rows > 2:
        y[1] = -100
    if mask is not None and V > 100:
        x[:, : V // 2 // 8 * 8] = mask
        y[2:] = V - 2
    lf = x.double().requires_grad_()
    want = torch.nn.functional.cross_entropy(lf, y, ignore_index=-100, reduction="none")
    (dref,) = torch.autograd.grad(want.sum() * 0.5, lf)
    loss, lse = load().ce_fwd_bwd(x, y, 0.5, None, -100, True)
    assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)
    assert torch.allclose(lse.double(), lf.logsumexp(-1), rtol=1e-5, atol=1e-5)
    _close(x, dref.float(), name="dlogits")


@pytest.mark.parametrize("rows", [2, 600])
@pytest.mark.parametrize("V", [4096, 4104, 8192, 8200, 16384, 16392, 51200, 51208, 76800, 76808])
def test_cross_entropy_kernel_on_both_sides_of_its_rule(rows, V):
    """Thread counts depend on the width, on whether there are more rows than SMs and on whether gradients are written: loss and gradients
    against 64 bits, and the loss alone leaves the logits as they are."""
    from torchllmtuner_b200.ops.cuda_ext import load
    torch.manual_seed(V)
    x, y = torch.randn(rows, V, device="cuda").mul_(3).bfloat16(), torch.randint(0, V, (rows,), device="cuda")
    lf = x.double()
    lse_ref = lf.logsumexp(-1)
    want = lse_ref - lf.gather(1, y[:, None])[:, 0]
    for grad in (False, True):
        buf = x.clone()
        loss, lse = load().ce_fwd_bwd(buf, y, 0.5, None, -100, grad)
        assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5) and torch.allclose(lse.double(), lse_ref, rtol=1e-5, atol=1e-5)
        if grad:
            d = (lf - lse_ref[:, None]).exp_()
            d[torch.arange(rows, device="cuda"), y] -= 1
            _close(buf, d.mul_(0.5).float(), name="dlogits")
        else:
            assert torch.equal(buf, x)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 7, 8, 1000003])
def test_scale_to_bf16(n, dtype):
    from torchllmtuner_b200.ops.cuda_ext import load
    torch.manual_seed(n)
    x, g = torch.randn(n, device="cuda").to(dtype), torch.tensor(0.3, device="cuda")
    assert torch.equal(load().scale_to_bf16(x, g), (x.float() * g).bfloat16())


@pytest.mark.parametrize("T,D", [(5, 256), (5, 264), (9472, 264), (9473, 264), (9473, 512), (3000, 1344)])
def test_rmsnorm_forward_at_the_edges_of_its_rule(T, D):
    """Widths of one vector per lane and one more, row counts on both sides of one wave of eight-row blocks on 148 SMs, and a
    width between two groups."""
    from torchllmtuner_b200 import ops
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(T + D)
    x, r = (torch.randn(T, D, device="cuda").bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    _close(ops.rms_norm(x, w, 1e-6), ref.rms_norm(x.float(), w.float(), 1e-6), name="y")
    y, s = ops.add_rms_norm(x, r, w, 1e-6)
    want, ws = ref.add_rms_norm(x.float(), r.float(), w.float(), 1e-6)
    _close(y, want, name="y"), _close(s, ws, name="sum")


def test_cross_entropy_gradient_of_a_confident_row():
    """Where the label's probability is close to 1, p - 1 is exact in fp32 and the gradient is that times the factor: the gradients of a
    factor of 1 and of 1/3 agree up to the rounding of each to bf16 (8 bits of significand: 2^-8 relative each, 2^-7 together). Rounding p times the factor first would leave an
    error of 2^-26, the size of the gradient itself on the most confident rows."""
    from torchllmtuner_b200.ops.cuda_ext import load
    d = torch.arange(10.0, 17.0, 0.0625)
    logits = torch.zeros(len(d), 64, device="cuda", dtype=torch.bfloat16)
    label = torch.arange(len(d), device="cuda") % 64
    logits[torch.arange(len(d), device="cuda"), label] = d.to("cuda", torch.bfloat16)
    one, third = logits.clone(), logits.clone()
    load().ce_fwd_bwd(one, label, 1.0, None, -100, True)
    load().ce_fwd_bwd(third, label, 1.0 / 3.0, None, -100, True)
    a, b = (t.gather(1, label[:, None]).double() for t in (one, third))
    assert (a < 0).sum() > len(d) // 2                      # confident, and not yet exactly 1
    assert ((b - a / 3).abs() <= 2.0 ** -7 * (a / 3).abs()).all()


def test_qk_norm_rope_outputs_are_differentiated_apart():
    """A backward through the queries frees their graph and leaves that of the keys."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(0)
    q, k = (torch.randn(37, h, 64, device="cuda").bfloat16().requires_grad_() for h in (4, 2))
    ws = [torch.randn(64, device="cuda").bfloat16().requires_grad_() for _ in range(2)]
    ang = torch.rand(37, 32, device="cuda")
    dys = [torch.randn_like(t) for t in (q, k)]
    call = lambda: ops.qk_norm_rope(q, k, *ws, ang.cos(), ang.sin(), 1e-6)  # noqa: E731
    want = torch.autograd.grad(call(), (q, k, *ws), dys)
    yq, yk = call()
    got = (torch.autograd.grad(yq, (q, ws[0]), dys[0]), torch.autograd.grad(yk, (k, ws[1]), dys[1]))
    for a, b in zip((got[0][0], got[1][0], got[0][1], got[1][1]), want):
        assert torch.equal(a, b)


def test_traced_ops_follow_their_inputs():
    """A trace calls the ops again on new inputs, forward and backward: nothing that an op computed while it was recorded is a constant."""
    from torchllmtuner_b200 import ops
    torch.manual_seed(0)
    new = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    w, W, qw, ang = new(128), new(64, 128), new(64), torch.rand(16, 32, device="cuda")
    calls = [(lambda x, y: ops.rms_norm(x + y, w, 1e-6), (16, 128)), (lambda x, y: ops.add_rms_norm(x, y, w, 1e-6), (16, 128)),
             (lambda x, y: ops.swiglu(x, y), (16, 128)), (lambda x, y: ops.linear(x + y, W), (16, 128)), (lambda x, y: ops.linears(x + y, W, W), (16, 128)),
             (lambda x, y: ops.qk_norm_rope(x, y, qw, None, ang.cos(), ang.sin(), 1e-6), (16, 2, 64))]
    for call, shape in calls:
        traced = torch.jit.trace(call, (new(*shape), new(*shape)), check_trace=False)
        ins = [new(*shape).requires_grad_() for _ in range(2)]
        ys = [t if isinstance(t, tuple) else (t,) for t in (traced(*ins), call(*ins))]
        dys = [torch.randn_like(t) for t in ys[0]]
        for a, b in zip((*ys[0], *torch.autograd.grad(ys[0], ins, dys)), (*ys[1], *torch.autograd.grad(ys[1], ins, dys))):
            assert torch.equal(a, b)


def test_row_kernels_refuse_views_off_the_16_byte_boundary():
    """The host answers with an error where a 16-byte access would be misaligned; no kernel is launched."""
    from torchllmtuner_b200.models.moe.experts import plan_segments
    from torchllmtuner_b200.ops.cuda_ext import load
    ext = load()
    flat = torch.randn(8 * 64 + 8, device="cuda").bfloat16()
    off, x, w = flat[1:8 * 64 + 1].view(8, 64), torch.randn(8, 64, device="cuda").bfloat16(), torch.randn(64, device="cuda").bfloat16()
    rstd, y = torch.ones(8, device="cuda"), torch.zeros(8, dtype=torch.int64, device="cuda")
    dest, seg, counts = plan_segments(torch.zeros(8, dtype=torch.int64, device="cuda"), 1)
    rows, ones = torch.zeros(128, 64, device="cuda", dtype=torch.bfloat16), torch.ones(8, device="cuda")
    calls = [lambda: ext.rmsnorm_fwd(off, None, w, 1e-6), lambda: ext.rmsnorm_fwd(x, off, w, 1e-6), lambda: ext.rmsnorm_fwd(x, None, flat[1:65], 1e-6),
             lambda: ext.rmsnorm_bwd(off, x, w, rstd, None), lambda: ext.rmsnorm_bwd(x, off, w, rstd, None), lambda: ext.rmsnorm_bwd(x, x, w, rstd, off),
             lambda: ext.ce_fwd_bwd(off, y, 1.0, None, -100, True), lambda: ext.permute_rows(off, dest, rows, 1, seg, counts),
             lambda: ext.combine_rows(off, y, None, 8, 1), lambda: ext.combine_bwd(off, rows, dest, ones, 1, seg, counts)]
    before = ext.launch_count()
    for call in calls:
        with pytest.raises(RuntimeError, match="-10"):
            call()
    assert ext.launch_count() == before
