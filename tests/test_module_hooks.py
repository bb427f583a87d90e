"""Hooks on the modules inside a block see what they always saw, although blocks do some modules' work in other ways when nothing looks."""
import pytest
import torch

from levanter_b200.nn import LayerNorm, Linear, RmsNorm, plain

DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


def _model(family, device):
    torch.manual_seed(0)
    kw = dict(seq_len=64, hidden_dim=128, num_layers=1, num_heads=2, gradient_checkpointing=False)
    if family == "gpt2":
        from levanter_b200.models.gpt2 import Gpt2Config

        cfg = Gpt2Config(resid_pdrop=0.0, attn_pdrop=0.0, embed_pdrop=0.0, **kw)
    else:
        from levanter_b200.models.llama import LlamaConfig

        cfg = LlamaConfig(intermediate_dim=256, num_kv_heads=2, **kw)
    return cfg.build(256, device=device, dtype=torch.bfloat16).train()


def _linears(model):
    return {n: m for n, m in model.named_modules() if type(m) is Linear and n != "lm_head"}


def _ids(device):
    return torch.randint(0, 256, (2, 64), generator=torch.Generator().manual_seed(1)).to(device)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("family", ["gpt2", "llama"])
def test_forward_hooks_see_the_module_s_own_result(family, device):
    model = _model(family, device)
    want = model(_ids(device), None)
    seen = {}
    for n, m in model.named_modules():
        if isinstance(m, (RmsNorm, LayerNorm, Linear)) or n.endswith(".attn") or n.endswith(".mlp"):
            m.register_forward_hook(lambda m, args, out, n=n: seen.__setitem__(n, out))
    got = model(_ids(device), None)
    assert set(_linears(model)) - {n for n in seen} <= {n for n in _linears(model) if n.endswith(("o_proj", "down_proj"))}  # added in an epilogue
    for n, out in seen.items():
        assert type(out) is torch.Tensor, n
    if family == "gpt2":  # a part of the block without the stream that it is added to
        block = "transformer.blocks.0."
        assert torch.equal(seen[block + "mlp"], seen[block + "mlp.c_proj"])
        assert torch.equal(seen[block + "attn"], seen[block + "attn.c_proj"])
    assert (got.float() - want.float()).norm() / want.float().norm() < 2 ** -7


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("family", ["gpt2", "llama"])
def test_backward_hooks_run(family, device):
    model, seen = _model(family, device), set()
    for n, m in _linears(model).items():
        if not n.endswith(("o_proj", "down_proj")):
            m.register_full_backward_hook(lambda m, gi, go, n=n: seen.add(n))
    norms = [n for n, m in model.named_modules() if isinstance(m, (RmsNorm, LayerNorm))]
    for n in norms:
        model.get_submodule(n).register_full_backward_hook(lambda m, gi, go, n=n: seen.add(n))
    model(_ids(device), None).float().square().sum().backward()
    assert seen == {n for n in _linears(model) if not n.endswith(("o_proj", "down_proj"))} | set(norms)


def test_plain():
    m = Linear(8, 8)
    assert plain(m, Linear) and not plain(m, RmsNorm)
    for register in (m.register_forward_hook, m.register_forward_pre_hook, m.register_full_backward_hook, m.register_full_backward_pre_hook):
        handle = register(lambda *a: None)
        assert not plain(m, Linear)
        handle.remove()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert not plain(m, Linear)
    handle.remove()
    m.forward = lambda x: x
    assert not plain(m, Linear)


@pytest.mark.gpu
def test_hooks_of_a_serving_step():
    """Joint products only where nothing looks at the projections; what a hook kept is not rotated under its hands."""
    import numpy as np

    from levanter_b200.inference.page_table import PageTable

    model = _model("llama", "cuda").eval()
    table = PageTable.init(4, 2, 16, 2)
    for s in range(2):
        table, _ = table.assign_seq_id_to_seq(s)
    table, info = table.allocate_for_seq(np.repeat(np.arange(2, dtype=np.int32), 5), np.tile(np.arange(5, dtype=np.int32), 2))
    info, pos = info.to("cuda"), torch.arange(5, dtype=torch.int32, device="cuda").repeat(2)
    ids = torch.arange(10, dtype=torch.int32, device="cuda")

    def step():
        with torch.no_grad():
            return model.decode(ids, model.initial_cache(table, dtype=torch.bfloat16), info, pos)[0].float()

    want, seen = step(), {}
    for n, m in _linears(model).items():
        m.register_forward_hook(lambda m, args, out, n=n: seen.__setitem__(n, (out, out.clone())))
    got = step()
    assert {n.rsplit(".", 1)[1] for n in seen} >= {"q_proj", "k_proj", "v_proj", "gate_proj", "up_proj"}
    assert all(torch.equal(kept, then) for kept, then in seen.values())
    assert (got - want).norm() / want.norm() < 2 ** -7
