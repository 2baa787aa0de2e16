"""Key-padding masks that empty whole tiles: the backward pass leaves their half of the data gradient's sum and of the
streamed aggregation out, with the result of the phase-by-phase calls, whose data gradient computes everything, and of
the oracle's float32 arithmetic."""
import pytest
import torch

from oracle import pom_oracle as O

pytestmark = pytest.mark.gpu


def _mask(kind, B, N):
    m = torch.zeros(B, N)
    g = torch.Generator().manual_seed(N)
    for b in range(B):
        if kind == "lengths":
            m[b, :int(torch.randint(1, N + 1, (1,), generator=g))] = 1
        elif kind == "tail":       # only the last tokens of a sample count
            m[b, N - 1 - b:] = 1
        elif kind == "holes":      # weights between 0 and 1 in every third run of 64 tokens
            m[b] = torch.rand(N, generator=g) * ((torch.arange(N) // 64) % 3 == 0)
    if kind == "lengths":
        m[0] = 1
    return m


@pytest.mark.parametrize("degree", [2, 3, 4])
@pytest.mark.parametrize("kind", ["lengths", "tail", "holes"])
@pytest.mark.parametrize("B,N,D,E", [(4, 128, 64, 2), (5, 300, 64, 1), (3, 1000, 128, 2), (6, 517, 40, 1), (7, 96, 136, 1)])
def test_skipped_tiles_change_nothing(B, N, D, E, kind, degree, monkeypatch):
    from pom_b200 import PoM
    from pom_b200 import functional as Fn

    torch.manual_seed(degree)
    mod = PoM(D, degree, E).cuda()
    torch.nn.init.normal_(mod.po_coeff, std=0.2)
    mod = mod.bfloat16()
    mask = _mask(kind, B, N).cuda()
    x, dy = (torch.randn(B, N, D, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_()
    wrt = [x, mod.qc_proj.weight, mod.se_bias, mod.po_coeff, mod.ag_proj.weight]
    skipped = torch.autograd.grad(mod(x, mask=mask), wrt, dy)
    monkeypatch.setattr(Fn, "WHOLE_LAYER_CALLS", False)
    whole = torch.autograd.grad(mod(x, mask=mask), wrt, dy)
    assert torch.equal(skipped[0], whole[0])
    for a, b in zip(skipped[1:], whole[1:]):  # split products add their partial sums in any order: one bf16 rounding
        assert (a.double() - b.double()).norm() <= 4e-3 * b.double().norm()
    ps = {k: v.detach().float().cpu().requires_grad_() for k, v in mod.state_dict().items()}
    xf = x.detach().float().cpu().requires_grad_()
    y = O.OraclePoM(ps, degree, E).forward(xf, None, mask.cpu())
    names = ["qc_proj.weight", "se_bias", "po_coeff", "ag_proj.weight"]
    want = torch.autograd.grad(y, [xf] + [ps[n] for n in names], dy.float().cpu())
    for a, b in zip(skipped, want):
        assert (a.double().cpu() - b.double()).norm() <= 2e-2 * b.double().norm()


@pytest.mark.parametrize("kind", ["across samples", "inside a tile"])
def test_weights_of_both_signs_that_cancel_in_a_tile(kind):
    """A tile is left out where every weight is 0, not where the weights add up to 0."""
    from pom_b200 import PoM

    torch.manual_seed(3)
    B, N, D = 2, (64 if kind == "across samples" else 300), 64
    mask = torch.ones(B, N)
    if kind == "across samples":  # 128 rows of the flattened tokens: 64 weights of 1, 64 of -1
        mask[1] = -1
    else:                         # the first tile of a sample
        mask[0, :128:2] = -1
        mask[1, 64:128] = -1
    mod = PoM(D, 2, 2).cuda()
    torch.nn.init.normal_(mod.po_coeff, std=0.2)
    mod = mod.bfloat16()
    x, dy = (torch.randn(B, N, D, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_()
    wrt = [x, mod.qc_proj.weight, mod.se_bias, mod.po_coeff, mod.ag_proj.weight]
    y = mod(x, mask=mask.cuda())
    got = [y, *torch.autograd.grad(y, wrt, dy)]
    ps = {k: v.detach().float().cpu().requires_grad_() for k, v in mod.state_dict().items()}
    xf = x.detach().float().cpu().requires_grad_()
    y = O.OraclePoM(ps, 2, 2).forward(xf, None, mask)
    names = ["qc_proj.weight", "se_bias", "po_coeff", "ag_proj.weight"]
    want = [y, *torch.autograd.grad(y, [xf] + [ps[n] for n in names], dy.float().cpu())]
    for a, b in zip(got, want):
        assert (a.double().cpu() - b.double()).norm() <= 2e-2 * b.double().norm()


def test_a_gradient_that_is_not_finite_reaches_the_empty_tiles():
    """0 times an infinite gradient of the aggregate is NaN, in a tile that the mask empties as in any other."""
    from pom_b200 import PoM

    torch.manual_seed(4)
    B, N, D = 2, 640, 64
    mod = PoM(D, 2, 2).cuda().bfloat16()
    mask = torch.ones(B, N, device="cuda")
    mask[:, 100:] = 0
    x, dy = (torch.randn(B, N, D, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_()
    dy[0, 3] = float("inf")
    dx, dcoeff = torch.autograd.grad(mod(x, mask=mask), [x, mod.po_coeff], dy)
    assert bool(dx[0].isnan().all()) and bool(dx[1].isfinite().all()) and bool(dcoeff.isnan().any())


def test_a_sample_without_any_valid_token():
    from pom_b200 import PoM

    mod = PoM(64, 2, 2).cuda().bfloat16()
    mask = torch.ones(3, 300, device="cuda")
    mask[1] = 0
    x = torch.randn(3, 300, 64, device="cuda").bfloat16().requires_grad_()
    y = mod(x, mask=mask)
    y.float().sum().backward()
    assert not bool(y[1].any()) and not bool(x.grad[1].any()) and bool(x.grad[0].any())
