"""Rotary tables as programs hold them: a table whose first row is not the identity, and tables rounded to bf16 with the
module.  Positions that are neither shared nor consecutive inside a 32-token group are rotated by their own table row,
so the layer is as close to the oracle (float64, the same tables) as the operators, forward and every gradient."""
import pytest
import torch

from oracle import pom_oracle as O

pytestmark = pytest.mark.gpu

PARAMS = ("qc_proj.weight", "se_bias", "po_coeff", "ag_proj.weight")


def _module(kind, two_d, heights, D, K, E):
    """A bf16 module; "centred": float32 tables whose angle is 0 in the middle; "cast": tables cast with the module."""
    from pom_b200 import PoMRoPE

    torch.manual_seed(sum(heights))
    mod = PoMRoPE(D, K, E, rope_2d=two_d, max_h=heights[0], max_w=heights[-1], max_seq_len=heights[0]).cuda()
    torch.nn.init.normal_(mod.po_coeff, std=0.2)
    mod = mod.bfloat16()
    names = ("row_cos", "row_sin", "col_cos", "col_sin") if two_d else ("freqs_cos", "freqs_sin")
    if kind == "centred":
        pairs = D * E // (4 if two_d else 2)
        inv = 10000.0 ** (-torch.arange(pairs, dtype=torch.float64) / pairs)
        for i, n in enumerate(heights):
            ang = torch.outer(torch.arange(n, dtype=torch.float64) - (n - 1) / 2, inv)
            setattr(mod, names[2 * i], ang.cos().float().cuda())
            setattr(mod, names[2 * i + 1], ang.sin().float().cuda())
    return mod, names


def _errors(mod, names, pos, x, dy, two_d, heights):
    K, E = mod.order, mod.order_expand
    key = "positions_hw" if two_d else "positions"
    xg = x.cuda().requires_grad_()
    named = dict(mod.named_parameters())
    y = mod(xg, **{key: pos.cuda()})
    got = [y.detach(), *torch.autograd.grad(y, [xg] + [named[n] for n in PARAMS], dy.cuda())]
    ps = {n: p.detach().double().cpu().requires_grad_() for n, p in named.items()}
    ref = O.OraclePoM(ps, K, E, 1, O.RopeConfig(two_d, heights[0], heights[0], heights[-1]))
    ref.tables = tuple(getattr(mod, n).double().cpu() for n in names)
    xr = x.double().requires_grad_()
    want = ref.forward(xr, None, None, **{key: pos})
    want = [want, *torch.autograd.grad(want, [xr] + [ps[n] for n in PARAMS], dy.double())]
    return [float((a.double().cpu() - b.detach()).norm() / b.detach().norm()) for a, b in zip(got, want)]


@pytest.mark.parametrize("kind", ["centred", "cast"])
@pytest.mark.parametrize("two_d,heights", [(True, (24, 24)), (True, (9, 40)), (True, (5, 62)), (False, (400,)), (False, (30,))],
                         ids=["24x24", "9x40", "5x62", "1d", "1d_below_32"])
@pytest.mark.parametrize("degree", [2, 4])
def test_every_token_is_rotated_by_its_own_table_row(kind, two_d, heights, degree, monkeypatch):
    from pom_b200 import ops

    D, E, B = 128, 2, 2
    mod, names = _module(kind, two_d, heights, D, degree, E)
    g = torch.Generator().manual_seed(heights[0])
    if two_d:
        N = heights[0] * heights[1]
        pos = torch.stack([torch.arange(N) // heights[1], torch.arange(N) % heights[1]], 1)
    else:
        N = 203
        span = min(62, heights[0])
        start = torch.randint(0, heights[0] - span + 1, ((N + 31) // 32,), generator=g).repeat_interleave(32)[:N]
        pos = start + torch.randint(0, span, (N,), generator=g)
    x, dy = (torch.randn(B, N, D, generator=g).bfloat16() for _ in range(2))
    assert ops.rope_pos_info(pos.cuda())[-1][2] == (3 if heights[-1] < 32 else 2)
    fused = _errors(mod, names, pos, x, dy, two_d, heights)
    monkeypatch.setattr(ops.RopeSpec, "fusable", lambda *_, **__: False)
    operators = _errors(mod, names, pos, x, dy, two_d, heights)
    for a, b in zip(fused, operators):
        assert a <= 1.02 * b, (fused, operators)  # the same roundings; sums in another order
