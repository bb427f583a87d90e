"""When an operation may run without its autograd function."""
import torch

from levanter_b200.ops import lib


def test_plain_call_is_false_wherever_an_autograd_function_has_to_be_seen():
    assert not lib.plain_call()  # gradients are recorded
    with torch.no_grad():
        assert lib.plain_call()
        seen = []
        torch.func.vmap(lambda x: (seen.append(lib.plain_call()), x)[1])(torch.ones(2))
        torch.func.jvp(lambda x: (seen.append(lib.plain_call()), x)[1], (torch.ones(2),), (torch.ones(2),))
        with torch.autograd.forward_ad.dual_level():
            seen.append(lib.plain_call())
        with torch.enable_grad():
            seen.append(lib.plain_call())
        assert seen == [False] * 4
        assert lib.plain_call()
