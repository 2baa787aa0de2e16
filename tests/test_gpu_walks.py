"""The operator kernels' token walks: whole chunks, token lanes and short spans give one result, at the sizes where
the cut changes and at ragged ends; row sums and masks of every dtype they read."""
import pytest
import torch

from oracle import pom_oracle as O

pytestmark = pytest.mark.gpu

# (B, N, P): one token, one chunk and its edges, channels narrower than a warp, one and several lanes, no cut at all
SHAPES = [(1, 1, 8), (2, 63, 16), (1, 65, 40), (3, 130, 256), (2, 200, 264), (1, 1000, 2304), (9, 700, 2304)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_selection_and_per_token_features_at_every_cut(shape, dtype):
    from pom_b200 import ops

    B, N, P = shape
    g = torch.Generator().manual_seed(B * N + P)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    tol = 1e-5 if dtype == torch.float32 else 8e-3  # fp32 sums; one bf16 rounding of each result (2^-8 at most)
    z, dsh, ht = rnd(B, N, P), rnd(B, N, P), rnd(B, N, P)
    bias, h, coeff = torch.randn(P, generator=g).cuda(), torch.randn(B, P, generator=g).cuda(), rnd(P, 3).float()
    s = O.hardsigmoid(z.double() + bias.double())
    inside = ((z.double() + bias.double()).abs() < 3).double() / 6
    close = lambda got, want: ((got.double() - want).norm() / want.norm()).item() <= tol
    for H, wide in ((h, h.double()[:, None]), (ht, ht.double())):
        assert close(ops.select_fwd(z, bias, H), s * wide)
        dz = torch.empty_like(z)
        dH, dbias = ops.select_bwd(dsh, z, bias, H, dz)
        want = dsh.double() * wide * inside
        assert close(dz, want) and ((dbias.double() - want.sum((0, 1))).norm() / want.norm()).item() <= tol
        grad = dsh.double() * s
        assert close(dH, grad) if H is ht else ((dH.double() - grad.sum(1)).norm() / grad.norm()).item() <= tol
    f = O.poly_features(z.double(), coeff.double())
    assert close(ops.poly_agg_fwd(z, coeff, per_token=True), f)
    dx, leaf = torch.empty_like(z), z.double().requires_grad_()
    c64 = coeff.double().requires_grad_()
    wx, wc = torch.autograd.grad(O.poly_features(leaf, c64), [leaf, c64], dsh.double())
    dc, _ = ops.poly_agg_bwd(z, coeff, dx_out=dx, dout=dsh, per_token=True)
    assert close(dx, wx) and ((dc.double() - wc).norm() / wc.norm()).item() <= max(tol, 1e-4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,P", [(1, 8), (63, 16), (65, 40), (300, 256), (1000, 1152), (77, 2304)])
def test_a_samples_gradients_have_the_same_bits_in_every_batch(N, P, dtype):
    """Launch shapes follow the batch; the order of a sample's sums, and every result, does not."""
    from pom_b200 import ops

    g = torch.Generator().manual_seed(N + P)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    z, dsh = rnd(64, N, P), rnd(64, N, P)
    bias, h = torch.randn(P, generator=g).cuda(), torch.randn(64, P, generator=g).cuda()
    s32, coeff = torch.rand(64, N, P // 8, generator=g).cuda(), torch.randn(P, 4, generator=g).cuda()
    rope = None
    if P % 16 == 0:
        ang = torch.rand(N, P // 2, generator=g).cuda()
        rope = ops.RopeSpec(1, ang.cos(), ang.sin(), torch.arange(N, device="cuda"))
    want = None
    for B in (64, 16, 4, 1):
        got = []
        for r in (None, rope):
            dz = torch.empty_like(z[:B])
            got += [ops.select_bwd(dsh[:B], z[:B], bias, h[:B], dz, rope=r)[0][0], dz[0]]
            got.append(ops.select_fwd(z[:B], bias, h[:B], rope=r)[0])
            for c in (coeff[:, :2].contiguous(), coeff):
                got += [ops.poly_agg_fwd(z[:B], c, rope=r)[0], ops.poly_agg_fwd(z[:B], c, per_token=True, rope=r)[0],
                        ops.poly_agg_fwd(z[:B], c, causal=True, rope=r)[0][0]]
                for kw in (dict(dH=h[:B]), dict(dout=dsh[:B], causal=True), dict(dout=dsh[:B], per_token=True)):
                    dx = torch.empty_like(z[:B])
                    ops.poly_agg_bwd(z[:B], c, dx_out=dx, rope=r, **kw)
                    got.append(dx[0])
        got.append(ops.select_heads_bwd(dsh[:B], s32[:B], h[:B], torch.zeros_like(s32[:B]))[0])
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want)), B


@pytest.mark.parametrize("chunks", [64, 1023, 1024, 4100])
def test_a_samples_partial_sums_have_the_same_bits_in_every_batch(chunks):
    from pom_b200 import ops

    x = torch.randn(40, chunks, 264, device="cuda")
    want = ops.reduce_partials(x)
    for B in (1, 7, 33):
        assert torch.equal(ops.reduce_partials(x[:B]), want[:B])
    many = torch.ones(2100, 1024, 8, device="cuda")  # more groups than a launch's grid takes
    assert bool((ops.reduce_partials(many) == 1024).all())


@pytest.mark.parametrize("B", [1, 3, 16, 64])
def test_a_samples_input_gradient_has_the_same_bits_in_every_batch(B):
    from pom_b200 import PoM

    torch.manual_seed(0)
    mod = PoM(256, 2, 2).cuda()
    x, dy = torch.randn(64, 300, 256, device="cuda"), torch.randn(64, 300, 256, device="cuda")

    def dx(n):
        q = x[:n].clone().requires_grad_()
        return torch.autograd.grad(mod(q), q, dy[:n])[0][0]

    assert torch.equal(dx(B), dx(64))


@pytest.mark.parametrize("n", [1, 31, 1000, 4096, 4097, 70001])
@pytest.mark.parametrize("rows", [1, 7, 40])
def test_row_sums_of_one_column(rows, n):
    from pom_b200 import ops

    x = torch.rand(rows, n, 1, device="cuda")
    got = ops.reduce_partials(x, scale=0.5, denom=torch.arange(rows, device="cuda", dtype=torch.float32))
    want = 0.5 * x.double().sum((1, 2)) / torch.arange(rows, device="cuda")
    want[0] = 0  # a denominator of zero gives zero
    assert torch.allclose(got.view(-1).double(), want, rtol=1e-5)


@pytest.mark.parametrize("chunks", [1, 8, 64, 65, 127, 500, 1024, 1500])
def test_partial_sums_at_every_lane_count(chunks):
    from pom_b200 import ops

    x = torch.randn(2, chunks, 72, device="cuda")
    want = x.double().sum(1)
    assert ((ops.reduce_partials(x).double() - want).norm() / want.norm()).item() <= 1e-5


@pytest.mark.parametrize("n", [1, 7, 8, 250, 264])
@pytest.mark.parametrize("src", [torch.bool, torch.uint8, torch.bfloat16, torch.float32])
def test_mask_rows_keep_values_and_sum_them(src, n):
    from pom_b200 import functional as Fn

    g = torch.Generator().manual_seed(n)
    mask = (torch.randint(0, 4, (2, 19, n), generator=g)).to(src).cuda()
    for dst in (torch.bfloat16, torch.float32):
        op, sums = Fn._mask_and_sums(mask, mask.device, dst)
        assert op.dtype == dst and torch.equal(op.float(), mask.float()) and op.stride(1) % 8 == 0
        assert torch.equal(sums, mask.float().sum(-1).view(-1))
    other, sums = Fn._mask_and_sums(mask.to(torch.int64), mask.device, torch.bfloat16)
    assert torch.equal(other.float(), mask.to(torch.int64).float()) and torch.equal(sums, mask.to(torch.int64).sum(-1).view(-1).float())
