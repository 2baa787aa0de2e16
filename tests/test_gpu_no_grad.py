"""A pass that no gradient can follow keeps nothing for one, and gives the result of a tracked pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [None, "causal", "keypad"])
def test_untracked_forward_equals_the_tracked_one_and_saves_no_projections(mask):
    from pom_b200 import PoM

    torch.manual_seed(0)
    B, N, D, E = 4, 512, 256, 4
    mod = PoM(D, 2, E).cuda().bfloat16()
    x = torch.randn(B, N, D, device="cuda", dtype=torch.bfloat16)
    m = (torch.arange(N, device="cuda")[None] < torch.tensor([[512], [100], [511], [1]], device="cuda")) if mask == "keypad" else mask
    y = mod(x, mask=m)
    assert y.requires_grad
    projection = B * N * D * E * 2  # bytes of the saved projection of one phase
    torch.cuda.synchronize()
    for ctx in (torch.no_grad(), torch.inference_mode()):
        with ctx:
            base = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            z = mod(x, mask=m)
            assert torch.equal(z, y.detach())
            assert torch.cuda.max_memory_allocated() - base < (3.5 if mask == "causal" else 2.5) * projection
    with torch.no_grad():
        with torch.enable_grad():
            w = mod(x, mask=m)
    w.sum().backward()  # tracked: everything a backward pass reads is there
    assert mod.qc_proj.weight.grad is not None and bool(torch.isfinite(mod.qc_proj.weight.grad).all())


def test_state_and_stack_without_gradients():
    from pom_b200.stack import PoMStack

    torch.manual_seed(1)
    stack = PoMStack(128, 2, 2, 2).cuda().bfloat16()
    x = torch.randn(2, 64, 128, device="cuda", dtype=torch.bfloat16)
    y1, s1 = stack.frame_forward(x)
    y2, s2 = stack.frame_forward(x, s1)
    h = stack.mixers[0].state_forward(x, None, None)[1]["h"]  # tracked call
    assert torch.equal(h.detach(), s1[0]["h"]) and s2[0]["n"] == 2 and not y2.requires_grad
