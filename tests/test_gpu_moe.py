"""MoE kernels (router top-k, permute, combine, grouped experts) vs the plain PyTorch statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(a, b, tol=3e-2):
    a, b = a.float(), b.float()
    assert (a - b).abs().max().item() <= tol * (b.abs().max().item() + 1e-6), ((a - b).abs().max().item(), b.abs().max().item())


@pytest.mark.parametrize("T,E,k,fn,renorm,use_bias", [(300, 128, 8, "softmax", True, True), (64, 8, 2, "sigmoid", True, False),
                                                      (1000, 256, 6, "softmax", False, False), (17, 64, 4, "sigmoid", False, True),
                                                      # both sides of 128 and 256 experts (4, 8 or 16 per lane), and the most
                                                      (33, 127, 8, "softmax", True, True), (33, 129, 8, "sigmoid", True, True),
                                                      (33, 255, 8, "softmax", True, False), (33, 257, 8, "softmax", True, True),
                                                      (33, 512, 16, "sigmoid", True, True)])
def test_router_topk_matches_reference(T, E, k, fn, renorm, use_bias):
    from torchllmtuner_b200.models.moe.routing import _RouterTopK
    from torchllmtuner_b200.ops import reference as ref
    torch.manual_seed(0)
    logits = torch.randn(T, E, device="cuda", requires_grad=True)
    bias = 0.1 * torch.randn(E, device="cuda") if use_bias else None
    w, idx, counts = _RouterTopK.apply(logits, bias, k, fn, renorm, 1.5)
    l2 = logits.detach().clone().requires_grad_()
    w2, idx2, counts2 = ref.router_topk(l2, bias, k, fn, renorm, 1.5)
    assert torch.equal(idx, idx2) and torch.equal(counts, counts2)
    assert (w - w2).abs().max().item() < 1e-5
    g = torch.randn_like(w)
    (d1,) = torch.autograd.grad(w, [logits], g)
    (d2,) = torch.autograd.grad(w2, [l2], g)
    assert (d1 - d2).abs().max().item() < 1e-5 * max(1.0, d2.abs().max().item())


def test_moe_block_cuda_matches_cpu_reference():
    from torchllmtuner_b200.models.moe import MoE
    torch.manual_seed(0)
    D, E, k, F_ = 256, 8, 2, 128
    cpu = MoE(D, E, k, F_, dtype=torch.float32)
    for p in cpu.parameters():
        torch.nn.init.normal_(p, std=0.05)
    gpu = MoE(D, E, k, F_, dtype=torch.bfloat16, device="cuda")
    gpu.load_state_dict({n: v.to("cuda") for n, v in cpu.state_dict().items()})
    x = torch.randn(500, D)
    xc = x.clone().requires_grad_()
    xg = x.to("cuda", torch.bfloat16).requires_grad_()
    # use the bf16-rounded weights/inputs on both sides
    with torch.no_grad():
        for pc, pg in zip(cpu.parameters(), gpu.parameters()):
            pc.copy_(pg.float().cpu())
    yc = cpu(xg.detach().float().cpu().requires_grad_() if False else xc.detach().bfloat16().float().requires_grad_())
    yg = gpu(xg)
    _close(yg, yc.to("cuda"), 5e-2)
    go = torch.randn_like(yg)
    gg = torch.autograd.grad(yg, [xg] + list(gpu.parameters()), go, allow_unused=True)
    xc2 = xc.detach().bfloat16().float().requires_grad_()
    yc2 = cpu(xc2)
    gc = torch.autograd.grad(yc2, [xc2] + list(cpu.parameters()), go.float().cpu(), allow_unused=True)
    for a, b in zip(gg, gc):
        if a is not None and b is not None:
            _close(a, b.to("cuda"), 6e-2)


@pytest.mark.parametrize("n,E,R", [(1000, 8, 2), (32768, 128, 8), (4097, 64, 4), (5, 16, 2)])
def test_ep_plan_matches_stable_sort(n, E, R):
    """Destination rows of the peer-memory dispatcher: stable position inside each expert's run plus the run's start."""
    from torchllmtuner_b200.ops.cuda_ext import load
    ext = load()
    g = torch.Generator(device="cuda").manual_seed(n + E)
    flat = torch.randint(0, E, (n,), generator=g, device="cuda")
    send_off = torch.randint(0, 1000, (E,), generator=g, device="cuda").to(torch.int32)
    drank, drow = ext.ep_plan(flat, E, R, send_off)
    counts = torch.bincount(flat, minlength=E)
    start = counts.cumsum(0) - counts
    order = torch.argsort(flat, stable=True)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device="cuda")
    pos = rank - start[flat]
    assert torch.equal(drow.long(), send_off.long()[flat] + pos)
    assert torch.equal(drank.long(), flat // (E // R))


@pytest.mark.parametrize("n,E", [(0, 4), (1, 1), (5, 16), (1023, 8), (1024, 512), (1025, 100), (32768, 128), (70001, 3)])
@pytest.mark.parametrize("skew", [False, True])
def test_plan_segments_kernel_matches_tensor_statement(n, E, skew):
    """The planning kernels against the tensor expressions of the CPU path: whole numbers, so equal."""
    from torchllmtuner_b200.models.moe.experts import plan_segments
    from torchllmtuner_b200.ops.cuda_ext import check_status
    g = torch.Generator().manual_seed(n + E)
    flat = torch.randint(0, E, (n,), generator=g)
    if skew:
        flat = torch.where(torch.rand(n, generator=g) < 0.9, torch.full_like(flat, E - 1), flat)
    want = plan_segments(flat, E)
    got = plan_segments(flat.cuda(), E)
    check_status("moe_plan")
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and torch.equal(a.cpu(), b)


def test_traced_plan_follows_its_input():
    from torchllmtuner_b200.models.moe.experts import plan_segments
    torch.manual_seed(0)
    first, second = (torch.randint(0, 8, (100,), device="cuda") for _ in range(2))
    traced = torch.jit.trace(lambda f: plan_segments(f, 8), (first,), check_trace=False)
    for a, b in zip(traced(second), plan_segments(second, 8)):
        assert a.dtype == b.dtype and torch.equal(a, b)


@pytest.fixture
def poisoned():
    """Every buffer that is allocated without a value is full of NaN (torch's deterministic mode does that)."""
    fill = torch.utils.deterministic.fill_uninitialized_memory
    before, warn = torch.are_deterministic_algorithms_enabled(), torch.is_deterministic_algorithms_warn_only_enabled()
    torch.use_deterministic_algorithms(True, warn_only=True)
    torch.utils.deterministic.fill_uninitialized_memory = True
    assert torch.empty(64, device="cuda", dtype=torch.bfloat16).isnan().all()
    yield
    torch.utils.deterministic.fill_uninitialized_memory = fill
    torch.use_deterministic_algorithms(before, warn_only=warn)


@pytest.mark.parametrize("T,E,k,D", [(3, 16, 2, 8), (130, 8, 4, 264), (257, 32, 8, 512), (65, 4, 1, 1032), (512, 4, 1, 64)])
def test_padding_rows_are_written(poisoned, T, E, k, D):
    """The dispatch copy and the combine's backward on buffers full of NaN: every copy arrives, every padding row of a segment is zero
    and rows past the last segment are not touched."""
    from torchllmtuner_b200.models.moe.experts import padded_capacity, plan_segments
    from torchllmtuner_b200.ops.cuda_ext import load
    torch.manual_seed(D)
    x, w = torch.randn(T, D, device="cuda").bfloat16(), torch.rand(T * k, device="cuda")
    flat = torch.randint(0, E - 1, (T * k,), device="cuda")            # the last expert has no copies
    dest, seg, counts = plan_segments(flat, E)
    cap, end = padded_capacity(T * k, E), int(seg[-1])
    padding = torch.ones(cap, dtype=torch.bool, device="cuda")
    padding[dest] = False
    padding[end:] = False
    rows = torch.full((cap, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    load().permute_rows(x, dest, rows, k, seg, counts)
    assert torch.equal(rows[dest], x.repeat_interleave(k, 0)) and (rows[padding] == 0).all() and rows[end:].isnan().all()
    y = torch.randn(cap, D, device="cuda").bfloat16()
    dy, dw = load().combine_bwd(x, y, dest, w, k, seg, counts)
    want = (w[:, None] * x.repeat_interleave(k, 0).float()).bfloat16()
    assert torch.equal(dy[dest], want) and (dy[padding] == 0).all() and dw.isfinite().all()


@pytest.mark.parametrize("T,E,k,D,F_", [(3, 16, 2, 8, 64), (130, 8, 4, 264, 72), (257, 32, 8, 512, 136), (65, 4, 1, 1032, 64)])
def test_routed_experts_write_their_padding_rows(poisoned, T, E, k, D, F_):
    """Buffers are no longer cleared before use: the same call on poisoned memory gives finite results that match the CPU
    statement, for narrow rows, a top-k that is no multiple of the combine's eight loads, and empty experts."""
    from torchllmtuner_b200.models.moe.experts import GroupedExperts, RoutedExperts
    torch.manual_seed(T)
    gpu = RoutedExperts(GroupedExperts(E, D, F_, dtype=torch.bfloat16, device="cuda"))
    cpu = RoutedExperts(GroupedExperts(E, D, F_, dtype=torch.float32))
    for p, q in zip(gpu.parameters(), cpu.parameters()):
        torch.nn.init.normal_(p, std=0.05)
        q.data.copy_(p.detach().float().cpu())
    x = torch.randn(T, D, device="cuda").bfloat16().requires_grad_()
    w = torch.rand(T, k, device="cuda", requires_grad=True)
    idx = torch.randint(0, E, (T, k), device="cuda")
    xc, wc = x.detach().float().cpu().requires_grad_(), w.detach().cpu().requires_grad_()
    go = torch.randn(T, D, device="cuda").bfloat16()
    yg = gpu(x, w, idx)
    gg = torch.autograd.grad(yg, [x, w, *gpu.parameters()], go)
    yc = cpu(xc, wc, idx.cpu())
    gc = torch.autograd.grad(yc, [xc, wc, *cpu.parameters()], go.float().cpu())
    for a, b in zip((yg, *gg), (yc, *gc)):
        assert torch.isfinite(a).all()
        _close(a, b.to("cuda"), 3e-2)
