"""Host side of the weight-streaming linears: workspaces and the cut of the weight."""

import torch

import voyager_b200 as vb


def test_scratch_belongs_to_one_call():
    calls = [[t for t in vb.packed._scratch(torch.device("cpu"), 1, n, 4096) if isinstance(t, torch.Tensor)]
             for n in (4096, 4096, 128256)]
    spans = [[(t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in call] for call in calls]
    for i, one in enumerate(spans):
        for other in spans[:i]:
            assert all(a[1] <= b[0] or b[1] <= a[0] for a in one for b in other)
