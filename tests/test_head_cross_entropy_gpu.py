"""The language-model head's cross-entropy in the epilogues of the CTA-pair GEMM, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plain(x, w, tgt, cap, z, gl):
    x, w = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    logits = x @ w.t()
    if cap:
        logits = torch.tanh(logits / cap) * cap
    lz = torch.logsumexp(logits, -1)
    V = w.shape[0]
    at = logits.gather(1, tgt.clamp(0, V - 1)[:, None])[:, 0]
    loss = lz - torch.where((tgt >= 0) & (tgt < V), at, torch.zeros_like(at)) + (z or 0.0) * lz * lz
    (loss * gl.double()).sum().backward()
    return loss.detach(), x.grad, w.grad


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# vocabularies around 128 (the old path), a tile of 256 and K blocks of 64; multiples of 8 (one part) and others (two, or three up to 1024 tokens); rows around a tile
@pytest.mark.parametrize("T,V,E,cap,z,chunk", [
    (1, 129, 8, None, None, None), (255, 136, 72, None, None, None), (256, 256, 64, 5.0, None, None), (257, 257, 64, None, 1e-3, None),
    (700, 1000, 768, None, None, 256), (300, 4093, 264, 7.0, 1e-3, 256), (513, 50257, 768, None, None, None), (1000, 8191, 128, None, None, 512),
    (1300, 4093, 264, 7.0, 1e-3, 256)])
def test_head_cross_entropy(T, V, E, cap, z, chunk):
    from levanter_b200.ops import cross_entropy as CE

    torch.manual_seed(0)
    x = torch.randn(T, E, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(V, E, device="cuda") * 2.0 / E ** 0.5).bfloat16().requires_grad_()
    tgt = torch.randint(0, V, (T,), device="cuda")
    tgt[0] = -1
    gl = torch.rand(T, device="cuda") + 0.1
    loss, _ = CE.fused_linear_cross_entropy(x, w, tgt, soft_cap=cap, z_weight=z, chunk_rows=chunk)
    (loss * gl).sum().backward()
    ref, dx, dw = _plain(x, w, tgt, cap, z, gl)
    # fp32 sums of up to 768 products and of V exponentials that are good to 2^-21
    assert float((loss.detach().double() - ref).abs().max()) < 2e-5 * max(1.0, float(ref.abs().max()))
    # results in bf16: half a unit in the last place is between 2^-9 and 2^-8 of a number; a gradient in one bf16 part adds as much
    limit = 2.0 ** -8 if V % 8 else 2.0 ** -7
    assert _rel(x.grad, dx) < limit
    assert _rel(w.grad, dw) < limit


@pytest.mark.parametrize("T,limit", [(300, 1e-6), (1024, 4e-6), (1025, 4e-6), (4100, 1.6e-5)])
def test_gradients_in_parts_over_an_fp32_accumulator(T, limit):
    """With an fp32 buffer for dW nothing is rounded to bf16.  Three parts (up to 1024 tokens) hold all of an fp32 number, two 16 bits, whose rounding
    averages out over the tokens; the lowest part is added first.  What shows is the accumulator, which cuts every addend off below its own last bit: at
    most 2^-24 of the sum for each of the T / 16 steps, 3.8e-9 per token, and a few 2^-24 of the probabilities."""
    from levanter_b200.ops import cross_entropy as CE

    torch.manual_seed(1)
    V, E = 1003, 128
    x = torch.randn(T, E, device="cuda").bfloat16()
    w = (torch.randn(V, E, device="cuda") * 0.2).bfloat16().requires_grad_()
    w.main_grad = torch.zeros(V, E, device="cuda")
    tgt = torch.randint(0, V, (T,), device="cuda")
    gl = torch.rand(T, device="cuda")
    loss, _ = CE.fused_linear_cross_entropy(x, w, tgt)
    (loss * gl).sum().backward()
    assert w.grad is None
    assert _rel(w.main_grad, _plain(x, w, tgt, None, None, gl)[2]) < limit


@pytest.mark.parametrize("V", [256, 257, 1003])
def test_infinite_logits(V):
    """+inf and -inf as in torch.logsumexp: a +inf anywhere makes the log-sum-exp +inf, columns of -inf are as if they were not there, NaN shows."""
    from levanter_b200.ops import cross_entropy as CE

    torch.manual_seed(3)
    inf = float("inf")
    base = (torch.randn(V, 64) * 0.2).bfloat16()
    x = torch.ones(4, 64, device="cuda").bfloat16()
    x[1] = -1.0
    for rows, value in (([5], inf), ([V - 1], inf), ([5, V - 1], inf), ([7, 40, V - 2], -inf), (range(V - 1), -inf), ([9], float("nan"))):
        w = base.clone()
        w[list(rows)] = 0.0
        w[list(rows), 0] = value  # one infinite product per logit: x[0] sees `value`, x[1] its opposite
        w = w.cuda()
        tgt = torch.tensor([0, 1, 2, V - 3], device="cuda")
        loss, lse = CE.fused_linear_cross_entropy(x, w, tgt)
        logits = x.double() @ w.double().t()
        want = torch.logsumexp(logits, -1)
        assert torch.allclose(lse.double(), want, rtol=1e-5, equal_nan=True), (lse, want)
        assert torch.allclose(loss.double(), want - logits.gather(1, tgt[:, None])[:, 0], rtol=1e-5, atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("V", [264, 331])
def test_rows_and_accumulators_of_other_layouts(V):
    """Rows that overlap or repeat and a weight of other strides are copied for the tensor maps, and the parameter itself keeps its accumulator; a bf16
    accumulator gets bf16 sums (2^-8), one of another shape is refused."""
    from levanter_b200.ops import cross_entropy as CE

    torch.manual_seed(4)
    T, E = 40, 64
    rows = torch.randn(E + 8 * T, device="cuda").bfloat16()
    tgt = torch.randint(0, V, (T,), device="cuda")
    gl = torch.rand(T, device="cuda") + 0.1
    for x in (rows.as_strided((T, E), (8, 1)), rows[:E].expand(T, E), torch.randn(T * E + 1, device="cuda").bfloat16()[1:].view(T, E)):
        for dtype in (torch.float32, torch.bfloat16):
            w = (torch.randn(E, V, device="cuda") * 0.2).bfloat16().t().requires_grad_()  # columns in a row
            w.main_grad = torch.full((V, E), 0.5, device="cuda", dtype=dtype)
            loss, _ = CE.fused_linear_cross_entropy(x, w, tgt)
            (loss * gl).sum().backward()
            ref, _, dw = _plain(x, w, tgt, None, None, gl)
            assert float((loss.detach().double() - ref).abs().max()) < 2e-5 * max(1.0, float(ref.abs().max()))
            assert w.grad is None
            assert _rel(w.main_grad, dw + 0.5) < (2e-3 if dtype == torch.float32 and V % 8 == 0 else 1e-5 if dtype == torch.float32 else 2 ** -8)
    w.main_grad = torch.zeros(V, E + 8, device="cuda")
    with pytest.raises(ValueError):
        CE.fused_linear_cross_entropy(x, w, tgt)[0].sum().backward()


def test_odd_vocabulary_in_the_loss_takes_what_it_took():
    """Targets out of range, strided operands and second derivatives, which the library products of these vocabularies allowed."""
    from levanter_b200.models.loss import maybe_fused_next_token_loss
    from levanter_b200.ops import lib

    torch.manual_seed(2)
    B, S, V, E = 2, 50, 331, 64
    x = torch.randn(B, S, 2 * E, device="cuda").bfloat16()[..., :E].requires_grad_()
    w = (torch.randn(V, 3 * E, device="cuda") * 0.2).bfloat16()[:, 1:E + 1].requires_grad_()
    ids = torch.randint(0, V, (B, S), device="cuda")
    ids[0, 5], ids[1, 7] = V + 3, -2
    got = maybe_fused_next_token_loss(x, w, ids)
    with lib.reference_ops():
        want = maybe_fused_next_token_loss(x, w, ids)
    assert abs(float(got) - float(want)) < 1e-5 * abs(float(want))
    for block in (None, 64):
        got = maybe_fused_next_token_loss(x, w, ids, block_size=block, reduction=None)
        with lib.reference_ops():
            want = maybe_fused_next_token_loss(x, w, ids, block_size=block, reduction=None)
        assert torch.allclose(got, want, rtol=1e-4, atol=1e-4)
    lib.check_status()

    def twice(loss):
        (g,) = torch.autograd.grad(loss, x, create_graph=True)
        return torch.autograd.grad(g.float().square().sum(), w)[0]

    got = twice(maybe_fused_next_token_loss(x, w, ids))
    with lib.reference_ops():
        want = twice(maybe_fused_next_token_loss(x, w, ids))
    assert _rel(got, want.double()) < 2e-2  # bf16 first derivatives on both sides
