"""Element-wise / reduction CUDA kernels against PyTorch fp32 references of the same ops."""
import math

import pytest
import torch

from levanter_b200.layers.rotary import DefaultRotaryEmbeddingsConfig, Llama3RotaryEmbeddingsConfig
from levanter_b200.ops import cross_entropy as CE
from levanter_b200.ops import glu, lib, norm, optim_kernels, rope
from levanter_b200.utils.activation import ActivationFunctionEnum

pytestmark = pytest.mark.gpu


def _close(a, b, tol=2e-2):
    a, b = a.float(), b.float()
    err = (a - b).abs().max().item()
    scale = b.abs().max().item() + 1e-6
    assert err / scale < tol, f"rel err {err / scale}"


@pytest.mark.parametrize("rows,dim", [(64, 4096), (1000, 128), (33, 1024), (7, 8192), (300, 64)])
@pytest.mark.parametrize("ln", [False, True])
def test_norm_fwd_bwd(rows, dim, ln):
    torch.manual_seed(0)
    x = torch.randn(rows, dim, device="cuda").bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).requires_grad_()
    b = (0.1 * torch.randn(dim, device="cuda")).requires_grad_() if ln else None
    y, _ = norm.fused_norm(x, w, b, 1e-5, layer_norm=ln)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_()
    wr = w.detach().clone().requires_grad_()
    br = b.detach().clone().requires_grad_() if ln else None
    if ln:
        yr = torch.nn.functional.layer_norm(xr, (dim,), wr, br, 1e-5)
    else:
        yr = xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + 1e-5) * wr
    yr.backward(g.float())
    _close(y, yr)
    _close(x.grad, xr.grad)
    _close(w.grad, wr.grad)
    if ln:
        _close(b.grad, br.grad)


def test_norm_residual_and_gemma_offset():
    torch.manual_seed(1)
    x = torch.randn(96, 512, device="cuda").bfloat16().requires_grad_()
    r = torch.randn(96, 512, device="cuda").bfloat16().requires_grad_()
    w = (0.1 * torch.randn(512, device="cuda")).requires_grad_()
    y, h = norm.fused_norm(x, w, None, 1e-6, w_offset=1.0, residual=r)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    (y * gy).sum().backward(retain_graph=True)
    (h * gh).sum().backward()
    xr, rr, wr = x.detach().float().requires_grad_(), r.detach().float().requires_grad_(), w.detach().clone().requires_grad_()
    hr = xr + rr
    yr = hr * torch.rsqrt(hr.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + wr)
    ((yr * gy.float()).sum() + (hr * gh.float()).sum()).backward()
    _close(y, yr)
    _close(h, hr)
    _close(x.grad, xr.grad)
    _close(r.grad, rr.grad)
    _close(w.grad, wr.grad)


@pytest.mark.parametrize("cfg", [DefaultRotaryEmbeddingsConfig(), Llama3RotaryEmbeddingsConfig()])
def test_rope(cfg):
    torch.manual_seed(2)
    B, S, H, KV, D = 2, 64, 8, 2, 128
    rot = cfg.build(D)
    q = torch.randn(B, S, H, D, device="cuda").bfloat16().requires_grad_()
    k = torch.randn(B, S, KV, D, device="cuda").bfloat16().requires_grad_()
    q2, k2 = rope.apply_rope(q * 1, k * 1, rot, None)
    gq, gk = torch.randn_like(q2), torch.randn_like(k2)
    ((q2 * gq).sum() + (k2 * gk).sum()).backward()
    qr, kr = q.detach().float().requires_grad_(), k.detach().float().requires_grad_()
    pos = torch.arange(S, device="cuda")
    q3, k3 = rot(qr, pos), rot(kr, pos)
    ((q3 * gq.float()).sum() + (k3 * gk.float()).sum()).backward()
    _close(q2, q3)
    _close(k2, k3)
    _close(q.grad, qr.grad)
    _close(k.grad, kr.grad)
    # explicit per-token positions
    pos2 = torch.randint(0, 500, (B, S), device="cuda")
    q4, _ = rope.apply_rope(q.detach() * 1, k.detach() * 1, rot, pos2)
    _close(q4, rot(q.detach().float(), pos2))
    lib.check_status()


@pytest.mark.parametrize("act", [ActivationFunctionEnum.silu, ActivationFunctionEnum.gelu_new, ActivationFunctionEnum.gelu])
def test_glu(act):
    torch.manual_seed(3)
    gu = torch.randn(50, 2 * 264, device="cuda").bfloat16().requires_grad_()
    g, u = gu[:, :264], gu[:, 264:]
    out = glu.gated_activation(g, u, act)
    go = torch.randn_like(out)
    out.backward(go)
    gur = gu.detach().float().requires_grad_()
    outr = act.to_fn()(gur[:, :264]) * gur[:, 264:]
    outr.backward(go.float())
    _close(out, outr)
    _close(gu.grad, gur.grad)


@pytest.mark.parametrize("V,cap,z", [(1000, None, None), (32000, None, 1e-4), (50264, 30.0, None)])
def test_fused_linear_cross_entropy(V, cap, z):
    torch.manual_seed(4)
    T, E = 300, 256
    x = (0.5 * torch.randn(T, E, device="cuda")).bfloat16().requires_grad_()
    w = (0.05 * torch.randn(V, E, device="cuda")).bfloat16().requires_grad_()
    tgt = torch.randint(0, V, (T,), device="cuda")
    loss, lse = CE.fused_linear_cross_entropy(x, w, tgt, soft_cap=cap, z_weight=z, chunk_rows=128)
    gl = torch.rand(T, device="cuda")
    (loss * gl).sum().backward()
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    logits = xr @ wr.t()
    if cap:
        logits = torch.tanh(logits / cap) * cap
    lz = torch.logsumexp(logits, -1)
    lr = lz - logits.gather(-1, tgt[:, None]).squeeze(-1)
    if z:
        lr = lr + z * lz * lz
    (lr * gl).sum().backward()
    _close(loss, lr, 1e-2)
    _close(x.grad, xr.grad, 3e-2)
    _close(w.grad, wr.grad, 3e-2)
    lib.check_status()


def test_adamw_and_sumsq():
    torch.manual_seed(5)
    n = 100_003
    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    m = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    pb = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    sq = optim_kernels.sumsq(g)
    assert abs(sq.item() - (g.double() ** 2).sum().item()) / sq.item() < 1e-5
    coef = torch.ones(1, device="cuda")
    nrm = torch.zeros(1, device="cuda")
    optim_kernels.clip_coef(sq, 1.0, coef, nrm)
    assert abs(nrm.item() - g.norm().item()) / nrm.item() < 1e-5
    p0 = p.clone()
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.95, 1e-8, 0.1
    optim_kernels.adamw(p, m, v, g, pb, lr, b1, b2, eps, wd, 1 - b1, 1 - b2, coef, 1.0, False)
    gs = g * coef
    mr = (1 - b1) * gs
    vr = (1 - b2) * gs * gs
    u = (mr / (1 - b1)) / ((vr / (1 - b2)).sqrt() + eps) + wd * p0
    pr = p0 - lr * u
    _close(p, pr, 1e-5)
    _close(pb, pr, 1e-2)
    _close(m, mr, 1e-5)


@pytest.mark.parametrize("rows,dim", [(1, 4096), (8, 2048), (1024, 512), (1025, 512), (999, 768), (5, 776), (3, 8), (40000, 128), (2, 12288), (700, 2056)])
@pytest.mark.parametrize("ln,residual,wdtype", [(True, False, torch.bfloat16), (False, True, torch.float32), (False, False, torch.bfloat16), (True, True, torch.float32)])
def test_norm_block_shapes(rows, dim, ln, residual, wdtype):
    """Widths around a warp, a block and several vectors per thread; few rows and many; a bias with and without a mean.  Sums in fp32 over bf16
    inputs: the results' bf16 rounding is 2^-9, and a bf16 weight's gradient is rounded once."""
    torch.manual_seed(rows + dim)
    x = torch.randn(rows, dim, device="cuda").bfloat16().requires_grad_()
    r = torch.randn(rows, dim, device="cuda").bfloat16().requires_grad_() if residual else None
    w = (1 + 0.1 * torch.randn(dim, device="cuda")).to(wdtype).requires_grad_()
    b = (0.1 * torch.randn(dim, device="cuda")).to(wdtype).requires_grad_()
    y, h = norm.fused_norm(x, w, b, 1e-5, layer_norm=ln, residual=r)
    gy, gh = torch.randn_like(y), torch.randn_like(y)
    torch.autograd.backward([y] + ([h] if residual else []), [gy] + ([gh] if residual else []))
    x64 = (h if residual else x).detach().double().requires_grad_()
    w64, b64 = (t.detach().double().requires_grad_() for t in (w, b))
    c = x64 - x64.mean(-1, keepdim=True) if ln else x64
    y64 = c * torch.rsqrt(c.pow(2).mean(-1, keepdim=True) + 1e-5) * w64 + b64
    torch.autograd.backward([y64] + ([x64 * 1] if residual else []), [gy.double()] + ([gh.double()] if residual else []))
    for got, want in ((y, y64), (x.grad, x64.grad), (w.grad, w64.grad), (b.grad, b64.grad)):
        assert (got.double() - want).norm() <= 2 ** -8 * want.norm() + 1e-6
    if residual:
        assert torch.equal(r.grad, x.grad)


@pytest.mark.parametrize("rows,cols,dtype", [(1, 8, torch.bfloat16), (31, 264, torch.float32), (33, 768, torch.bfloat16), (999, 2304, torch.float32), (5000, 6144, torch.bfloat16)])
def test_col_sum(rows, cols, dtype):
    """fp32 sums of up to 5000 bf16 numbers (2^-24 sqrt(rows) relative to their norm), then at most one bf16 rounding."""
    from levanter_b200.ops.gemm import col_sum

    x = torch.randn(rows, cols + 8, device="cuda").bfloat16()[:, 8:]
    got = col_sum(x, dtype)
    want = x.double().sum(0)
    assert got.dtype == dtype
    assert (got.double() - want).norm() <= (2 ** -8 if dtype == torch.bfloat16 else 1e-5) * want.norm()


@pytest.mark.parametrize("rows,outputs,cols,dtype", [(1024, 8, 8, torch.float32), (1500, 8, 1024, torch.bfloat16), (5003, 24, 776, torch.float32), (16384, 32, 264, torch.bfloat16)])
def test_few_outputs_dw(rows, outputs, cols, dtype):
    """Exact products of bf16 numbers in fp32 sums (2^-24 sqrt(rows)), then at most one bf16 rounding; fewer rows or more outputs are the GEMM's."""
    from levanter_b200.ops.gemm import few_outputs_dw

    dy, x = (torch.randn(rows, n + 8, device="cuda").bfloat16()[:, 8:] for n in (outputs, cols))
    got = few_outputs_dw(dy, x, dtype)
    want = dy.double().t() @ x.double()
    assert got.dtype == dtype
    assert (got.double() - want).norm() <= (2 ** -8 if dtype == torch.bfloat16 else 1e-5) * want.norm()
    assert few_outputs_dw(dy[:1000], x[:1000], dtype) is None


@pytest.mark.parametrize("rows", [7, 1100])
def test_projections_of_the_same_rows_and_a_norm_that_forks(rows):
    """Sums of input gradients in the products' epilogues, and a block's input beside its norm: what separate functions give, with fewer roundings
    (2^-8 of a gradient's norm)."""
    from levanter_b200.nn import LayerNorm, Linear, fork_norm, linear_many

    torch.manual_seed(0)
    with torch.device("cuda"):
        mods = [Linear(264, n).bfloat16() for n in (264, 8, 520)]
        ln = LayerNorm(264).bfloat16()
    x = torch.randn(rows, 264, device="cuda").bfloat16().requires_grad_()
    gs = [torch.randn(rows, n, device="cuda").bfloat16() for n in (264, 8, 520)]
    params = [m.weight for m in mods] + [ln.weight, ln.bias]

    def grads(joint):
        for p in params + [x]:
            p.grad = None
        h, r = fork_norm(ln, x) if joint else (ln(x), x)
        ys = linear_many(h, *mods) if joint else [m(h) for m in mods]
        torch.autograd.backward([*ys, r * 1], [*gs, gs[0]])
        return [t.detach() for t in ys], [p.grad.float() for p in params + [x]]

    (y1, g1), (y2, g2) = grads(True), grads(False)
    assert all(torch.equal(a, b) for a, b in zip(y1, y2))
    for a, b in zip(g1, g2):
        assert (a - b).norm() <= 2 ** -7 * b.norm()
    h, r = fork_norm(ln, x.detach())
    assert torch.equal(h, ln(x.detach())) and torch.equal(r, x.detach())


def test_norm_backward_from_two_threads():
    """Rows of 64 and of 4096 with a residual's gradient go through the same kernel with 8 and 96 KB of shared memory: neither thread may take the
    other's room away between its request and its launch."""
    import threading

    from levanter_b200.ops import norm as N

    failed = []

    def work(dim, seed):
        try:
            g = torch.Generator(device="cuda").manual_seed(seed)
            x = torch.randn(64, dim, device="cuda", generator=g).bfloat16().requires_grad_()
            w = torch.ones(dim, device="cuda").bfloat16().requires_grad_()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(200):
                    y, h = N.norm_and_input(x, w, None, 1e-6, layer_norm=False)
                    torch.autograd.grad((y.float() + h.float()).sum(), (x, w))
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(dim, i)) for i, dim in enumerate((4096, 64, 4096, 64))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed


@pytest.mark.parametrize("used", [(0,), (1,), (0, 2)])
def test_joint_projections_that_nothing_uses_have_no_gradient(used):
    from levanter_b200.nn import Linear, linear_many

    torch.manual_seed(0)
    mods = [Linear(64, n).cuda().bfloat16() for n in (64, 128, 32)]
    x = torch.randn(48, 64, device="cuda").bfloat16().requires_grad_()
    ys = linear_many(x, *mods)
    sum(ys[i].float().sum() for i in used).backward()
    assert [m.weight.grad is not None for m in mods] == [i in used for i in range(3)]
    want = sum(torch.ones(48, mods[i].out_features, device="cuda", dtype=torch.double) @ mods[i].weight.double() for i in used)
    assert (x.grad.double() - want).norm() / want.norm() < 2 ** -7


@pytest.mark.parametrize("rows,outputs,cols,lanes", [(1024, 16, 1024, True), (1024, 8, 4096, False), (2047, 32, 1024, False), (2048, 32, 1024, True), (2048, 8, 4096, True),
                                                     (16384, 16, 4096, False)])
def test_few_outputs_dw_where_it_is_the_faster_form(rows, outputs, cols, lanes):
    from levanter_b200.ops.gemm import few_outputs_dw

    dy, x = (torch.zeros(rows, n, device="cuda").bfloat16() for n in (outputs, cols))
    assert (few_outputs_dw(dy, x, torch.bfloat16) is not None) == lanes
