"""Parameters that are slices of one matrix."""
import copy

import torch
import torch.nn as nn

from levanter_b200.nn import FusedRows


def test_fused_rows_follow_the_parameters():
    a, b = nn.Parameter(torch.randn(3, 4)), nn.Parameter(torch.randn(2, 4))
    values = torch.cat([a, b]).detach().clone()
    rows = FusedRows(pad=3)
    assert rows.get([a, b], build=False) is None  # nothing is moved unless asked to
    with torch.inference_mode():  # a cache may be made there, and the parameters stay parameters
        whole = rows.get([a, b])
    assert torch.equal(whole, torch.cat([values, torch.zeros(3, 4)])) and not a.is_inference()
    assert rows.get([a, b], build=False).data_ptr() == a.data_ptr() and b.data_ptr() == a.data_ptr() + 12 * 4
    with torch.no_grad():
        b.mul_(2.0)
    assert torch.equal(rows.get([a, b], build=False)[3:5], 2.0 * values[3:])
    assert rows.get([b, a], build=False) is None and rows.get([a], build=False) is None and FusedRows().get([a, b], build=False) is None
    assert copy.deepcopy(rows).get([a, b], build=False) is not None
    b.data = b.data.clone()  # an assignment, a conversion or a move takes it out again
    assert rows.get([a, b], build=False) is None
    a.main_grad = torch.zeros(3, 4)
    assert rows.get([a, b]) is None
