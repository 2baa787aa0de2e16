"""Rotary positions that are neither shared nor consecutive inside aligned 32-token groups: grids whose rows do not end
on 32 tokens, and positions in any order within 61 of one another, stay in the tensor-core epilogues; wider ones, and
token-causal layers, take the operators.  Layer against the oracle, forward and every gradient."""
import pytest
import torch

from tests.helpers import assert_status_clean
from tests.test_gpu_rope_fused import _case, _check_layer, _Spy

pytestmark = pytest.mark.gpu


# grid heights and widths: one token, rows shorter than a group, an offset of -30 and of 31 (width 62), the first
# width whose row ends span too much (63), and rows longer than two groups
@pytest.mark.parametrize("mask", [None, "causal"])
@pytest.mark.parametrize("gh,gw,fused", [(1, 1, True), (7, 5, True), (24, 24, True), (9, 33, True), (5, 47, True),
                                         (4, 62, True), (4, 63, False), (3, 80, False)])
def test_grids_of_any_width(gh, gw, fused, mask, monkeypatch):
    N = gh * gw
    cfg, params, x, gy, kw = _case(2, N, 128, 2, 2, seed=40 + gw, two_d=True, side=max(gh, gw), bias_scale=0.1)
    kw["positions_hw"] = torch.stack([torch.arange(N) // gw, torch.arange(N) % gw], 1)
    if mask:
        kw["mask"] = mask
    spy = _Spy(monkeypatch)
    _check_layer(cfg, params, x, gy, kw, f"{gh} x {gw} {mask}")
    assert (spy.calls == 0) == (fused and (mask is None or N == 1))


@pytest.mark.parametrize("degree", [1, 3, 4])
def test_every_degree_and_a_shuffled_order(degree, monkeypatch):
    """1-D positions in any order inside a window of 62 per group, ragged length, table end included."""
    N = 203
    cfg, params, x, gy, kw = _case(3, N, 64, degree, 2, seed=60 + degree, two_d=False, max_len=400, bias_scale=0.1)
    g = torch.Generator().manual_seed(degree)
    start = torch.randint(0, 400 - 61, ((N + 31) // 32,), generator=g).repeat_interleave(32)[:N]
    pos = start + torch.randint(0, 62, (N,), generator=g)
    pos[5], pos[6] = start[5], start[5] + 61  # both ends of the window
    pos[-1] = 399 if start[-1] > 337 else pos[-1]
    spy = _Spy(monkeypatch)
    _check_layer(cfg, params, x, gy, dict(kw, positions=pos), f"shuffled, degree {degree}")
    assert spy.calls == 0


def test_both_gemm_kernels_and_tile_widths(monkeypatch):
    from pom_b200 import _abi

    cfg, params, x, gy, kw = _case(2, 24 * 24, 320, 2, 2, seed=71, two_d=True, side=24, bias_scale=0.1)
    try:
        for mode in (11, 21, 31, 12, 22, 32, 132):
            assert _abi.lib().pom_set_gemm_mode(mode) == 0
            _check_layer(cfg, params, x, gy, kw, f"mode {mode}")
    finally:
        _abi.lib().pom_set_gemm_mode(0)
    assert_status_clean()


def test_position_scan_tells_the_kinds_apart():
    from pom_b200 import ops

    cases = {0: torch.full((70,), 9), 1: torch.arange(70) + 5, 2: torch.arange(70) % 62, -1: torch.arange(70) * 2}
    for want, pos in cases.items():
        assert ops.rope_pos_info(pos.cuda())[0] == (int(pos.min()), int(pos.max()), want)
    both = torch.stack([cases[2], cases[-1]], 1).cuda()
    assert [s for _, _, s in ops.rope_pos_info(both)] == [2, -1]
