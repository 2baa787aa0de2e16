"""float32 GEMM on the tensor cores (three bf16 planes) against float64: every operand order, edges of tiles, K splits,
and the values that the planes cannot carry."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu


def _gemm64(a, b, a_mn, b_mn):
    a64, b64 = a.double(), b.double()
    return (a64.t() if a_mn else a64) @ (b64 if b_mn else b64.t())


def _operands(M, N, K, a_mn, b_mn, seed, pad=0):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn((K, M + pad) if a_mn else (M, K + pad), generator=g).cuda()
    b = torch.randn((K, N + pad) if b_mn else (N, K + pad), generator=g).cuda()
    return (a[:, :M] if a_mn else a[:, :K]), (b[:, :N] if b_mn else b[:, :K])


def _planes(a, b, use=True, **kw):
    from unittest import mock

    from pom_b200 import ops

    with mock.patch.object(ops, "f32_planes_pay", lambda *_: use):
        return ops.gemm(a, b, **kw)


# A float32 chain of K fused multiply-adds is off by about sqrt(K) / 4 units of 2^-24 of sum |a||b| / sqrt(K): 4e-7 at
# K = 1000 for these inputs.  The planes add K / 64 block sums; 2.5e-7 holds for every K here.
BOUND = 2.5e-7
SHAPES = [(1, 1, 1), (3, 5, 7), (128, 128, 64), (129, 127, 65), (256, 256, 128), (257, 300, 63), (500, 1152, 200),
          (512, 256, 1000), (255, 513, 4100), (2048, 2312, 96)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_every_operand_order_matches_float64(shape):
    M, N, K = shape
    for i, (a_mn, b_mn) in enumerate(itertools.product((False, True), repeat=2)):
        for pad in (0, 3):
            a, b = _operands(M, N, K, a_mn, b_mn, 10 * i + pad, pad)
            want = _gemm64(a, b, a_mn, b_mn)
            got = _planes(a, b, a_mn=a_mn, b_mn=b_mn)
            assert ((got.double() - want).norm() / want.norm()).item() <= BOUND, (a_mn, b_mn, pad)
            acc = torch.randn(M, N, device="cuda")
            both = _planes(a, b, a_mn=a_mn, b_mn=b_mn, out=acc.clone(), accumulate=True, alpha=0.5)
            want = acc.double() + 0.5 * want
            assert ((both.double() - want).norm() / want.norm()).item() <= BOUND


@pytest.mark.parametrize("scale", [1e-12, 1.0, 1e9])
def test_sums_of_one_sign_and_far_scales_keep_float32_accuracy(scale):
    """Sums of positive terms are where a truncating accumulator drifts; rows of very different magnitude are where a
    common scale would lose bits."""
    M, N, K = 384, 320, 6000
    g = torch.Generator().manual_seed(3)
    a = torch.rand(M, K, generator=g).cuda() * scale
    a *= torch.logspace(-6, 6, M).cuda()[:, None]
    b = torch.rand(N, K, generator=g).cuda()
    want = _gemm64(a, b, False, False)
    err = ((_planes(a, b).double() - want).abs() / want).max().item()
    assert err <= 1e-6  # a chain of 6000 float32 FMAs is 5e-6 off on these inputs


@pytest.mark.parametrize("a_scale,b_scale", [(1e-34, 1), (1e-38, 1), (1e-41, 1e3), (1, 1e-38), (1e-20, 1e-15), (1e-19, 1e-19),
                                             (1e-22, 1e-22), (1e-30, 1e20), (1e12, 1e12), (1e25, 1e-25), (1e31, 1e-20)])
def test_small_and_large_magnitudes_are_no_further_off_than_a_chain(a_scale, b_scale):
    """Operands near either end of float32's range, subnormal ones among them, and products near it: the error, as a
    share of the sum of magnitudes, is at most that of the FMA chain (or, where results are subnormal, one of their
    steps)."""
    g = torch.Generator().manual_seed(4)
    a, b = (torch.randn(256, 512, generator=g).cuda() * s for s in (a_scale, b_scale))
    a[:, ::7] *= 1e-3
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    err = [((_planes(a, b, use=u).double() - want).abs() - 2.0 ** -149).clamp(min=0).div(mag).max().item()
           for u in (True, False)]
    assert err[0] <= max(err[1], BOUND), err


@pytest.mark.parametrize("alpha", [3.0, -2.0 ** -60, 2.0 ** -90, 0.0])
def test_products_times_any_alpha(alpha):
    """The factor of the planes is part of the epilogue's alpha, down to where that would be subnormal."""
    a, b = _operands(300, 290, 260, False, False, 5)
    got, want = _planes(a, b, alpha=alpha), alpha * _gemm64(a, b, False, False)
    if 0 < alpha < 2.0 ** -78:  # the FMA kernel, times a power of two
        assert torch.equal(got, alpha * _planes(a, b, use=False))
    else:
        assert (got.double() - want).norm().item() <= BOUND * want.norm().item()
    acc = _planes(a, b, alpha=alpha, out=torch.ones_like(got), accumulate=True)
    assert (acc.double() - 1 - want).norm().item() <= BOUND * (1 + want).norm().item()


def test_values_outside_the_range_of_the_planes_move_the_product_to_the_fma_kernel():
    a, b = _operands(300, 290, 260, False, False, 5)
    b = b.sign() * (1 + b.abs())
    for x, y, carried in ((1e-30, 1e-20, False), (1e24, 1e22, False), (1e-44, 1.0, True)):
        p, q = a.clone(), b.clone()
        p[17], q[5, 9] = x, y
        assert torch.equal(_planes(p, q), _planes(p, q, use=False)) != carried, (x, y)


@pytest.mark.parametrize("shape", [(1, 1, 1), (63, 65, 17), (200, 1000, 40), (129, 257, 100), (2049, 2500, 33)],
                         ids=lambda s: "x".join(map(str, s)))
def test_fma_kernel_is_one_chain_over_k(shape):
    """Every output is the chain of fused multiply-adds over k from zero, whatever the tile, the storage order and the
    alignment: bit for bit the chain formed here in float64 and rounded after every step (exact: a product of two
    float32 values has 48 bits, its sum with a float32 value is rounded once by a float64 addition only when it needs
    more than 53, so the inputs are kept to 12 bits)."""
    M, N, K = shape
    for i, (a_mn, b_mn) in enumerate(itertools.product((False, True), repeat=2)):
        for pad in (0, 3):
            a, b = (t.half().float() for t in _operands(M, N, K, a_mn, b_mn, 20 * i + pad))
            if pad:  # rows that do not start on 16 bytes
                a = torch.nn.functional.pad(a, (1, 2))[:, 1:-2]
                b = torch.nn.functional.pad(b, (1, 2))[:, 1:-2]
            a64, b64 = (a.double().t() if a_mn else a.double()), (b.double().t() if b_mn else b.double())
            want = torch.zeros(M, N, device="cuda")
            for k in range(K):
                want = (want.double() + a64[:, k, None] * b64[None, :, k]).float()
            assert torch.equal(_planes(a, b, use=False, a_mn=a_mn, b_mn=b_mn), want), (a_mn, b_mn, pad)


@pytest.mark.parametrize("shape", [(300, 290, 260), (255, 513, 4100)], ids=["one pass", "split sums"])
def test_infinities_nan_and_huge_values_take_the_fma_kernel(shape):
    from pom_b200 import _abi

    M, N, K = shape
    assert bool(_abi.lib().pom_gemm_f32_planes_scratch(M, N, K, _abi.OUT_F32_ACCUM)) == (K > 4000)  # K is split
    a, b = _operands(M, N, K, False, False, 5)
    for value in (float("inf"), float("-inf"), float("nan"), 1e30, -2e38):
        x = a.clone()
        x[17, 31] = value
        got = _planes(x, b)
        want = _planes(x, b, use=False)
        assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))
        before = torch.randn(M, N, device="cuda")
        acc = _planes(x, b, out=before.clone(), accumulate=True)
        assert torch.equal(torch.nan_to_num(acc, nan=7.0), torch.nan_to_num(before + want, nan=7.0))


def test_shared_planes_and_repeated_runs_give_the_same_bits():
    from pom_b200 import ops

    a, b = _operands(640, 1152, 700, False, False, 6)
    w = torch.randn(1152, 640, device="cuda")
    pl = ops.F32Planes()
    first, second = _planes(a, b, a_planes=pl), _planes(a, w, a_mn=True, a_planes=pl)
    assert torch.equal(first, _planes(a, b)) and torch.equal(second, _planes(a, w, a_mn=True))


@pytest.mark.parametrize("rows,cols", [(512, 1152), (1000, 72)], ids=["wide", "narrow"])
@pytest.mark.parametrize("value", [None, float("inf")])
def test_planes_of_a_projection_serve_a_later_product(rows, cols, value):
    """pom_gemm_f32_planes with an operand that pom_project_f32 has split, through the C ABI: the words that say which
    kernel computes the product are found whichever split wrote them."""
    import ctypes as C

    from pom_b200 import _abi, ops

    x, w = _operands(rows, 96, cols, False, False, 11)
    if value is not None:
        x[rows - 1, 0] = value
    dy = torch.randn(rows, 40, device="cuda")
    L, status, st = _abi.lib(), _abi.ptr(_abi.status_word(x.device)), _abi.stream_ptr()
    # what words that no call writes hold: "not finite", or "all zeros"
    for junk in (255 << 16, 255):
        bufs = []
        for t in (x, w, dy):
            bufs.append(torch.zeros(int(L.pom_f32_planes_bytes(*t.shape)), dtype=torch.uint8, device="cuda"))
            bufs[-1][:4096].view(torch.int32).fill_(junk)
        norms, out = torch.empty(rows + 96, device="cuda"), torch.empty(rows, 96, device="cuda")
        g = _abi.GemmArgs()
        g.A, g.Bm, g.C, g.M, g.N, g.K = x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, 96, cols
        g.lda, g.ldb, g.ldc, g.batches, g.out_mode, g.split_k, g.alpha = cols, cols, 96, 1, _abi.OUT_F32, 1, 1.0
        _abi.check(L.pom_project_f32(C.byref(g), bufs[0].data_ptr(), bufs[1].data_ptr(), norms.data_ptr(), 96, None,
                                     status, st), "pom_project_f32")
        got = torch.zeros(cols, 40, device="cuda")  # xT . dy, x read in the other major
        g.A, g.Bm, g.C, g.M, g.N, g.K = x.data_ptr(), dy.data_ptr(), got.data_ptr(), cols, 40, rows
        g.lda, g.ldb, g.ldc, g.a_mn_major, g.b_mn_major = cols, 40, 40, 1, 1
        _abi.check(L.pom_gemm_f32_planes(C.byref(g), bufs[0].data_ptr(), 1, bufs[2].data_ptr(), 0, None, status, st),
                   "pom_gemm_f32_planes")
        fresh = _planes(x, dy, a_mn=True, b_mn=True)
        assert torch.equal(got.nan_to_num(nan=7.0), fresh.nan_to_num(nan=7.0)), junk


@pytest.mark.parametrize("shape", [(1, 8, 128), (130, 258, 129), (500, 1000, 256), (1021, 2304, 1152)],
                         ids=lambda s: "x".join(map(str, s)))
def test_projection_takes_the_chain_beside_the_kinks(shape, monkeypatch):
    """Every comparison that a derivative makes (activation at 0, 6, -10; gate at +-3) falls as the FMA chain's does, and
    the elements closest to a kink carry the chain's bits; wide weights reach all five kinks."""
    from pom_b200 import ops

    monkeypatch.setattr(ops, "F32_PROJECT_MIN_WEIGHTS", 0)
    M, N, K = shape
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, K, generator=g).cuda()
    w = (torch.randn(N, K, generator=g) * 6 / K ** 0.5).cuda()
    P = N // 2
    bias = torch.randn(N - P, generator=g).cuda()
    got, chain = ops.project_f32(x, w, P, bias), _planes(x, w, use=False, fma=True)
    want = _gemm64(x, w, False, False)
    assert ((got.double() - want).norm() / want.norm()).item() <= BOUND
    eps = 2.0 ** -24 * K ** 0.5 * x.norm(dim=1)[:, None] * w.norm(dim=1)[None]  # an eighth of the kernel's own bound
    for v, c, cut, e in ((got[:, :P], chain[:, :P], (0.0, 6.0, -10.0), eps[:, :P]),
                         (got[:, P:] + bias, chain[:, P:] + bias, (3.0, -3.0), eps[:, P:])):
        for k in cut:
            assert torch.equal(v > k, c > k) and torch.equal(v < k, c < k)
            near = (c - k).abs() <= 4 * e
            assert torch.equal(v[near], c[near])
    assert M * N < 100000 or bool((chain[:, :P].abs() <= 4 * eps[:, :P]).any())  # the test meets such elements


def test_projection_of_values_that_are_not_finite(monkeypatch):
    from pom_b200 import ops

    monkeypatch.setattr(ops, "F32_PROJECT_MIN_WEIGHTS", 0)
    x, w = _operands(70, 90, 200, False, False, 8)
    for value in (float("inf"), float("nan"), 3e38):
        y = x.clone()
        y[3, 5] = value
        a, b = ops.project_f32(y, w, 90), _planes(y, w, use=False, fma=True)
        assert torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))


def _us(fn, runs=5):
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    times = []
    for _ in range(runs):
        ev[0].record()
        fn()
        ev[1].record()
        torch.cuda.synchronize()
        times.append(ev[0].elapsed_time(ev[1]) * 1e3)
    return min(times[1:])


def test_projection_of_zero_rows_runs_no_chains():
    """Padded tokens and zero weight rows sit on the kink at 0 with all their elements: exactly 0 without a chain, the
    other rows as they were, and the time of a product without them (a chain per element took a hundred times it)."""
    from pom_b200 import ops

    M, N, K = 2048, 1000, 1152
    x, w = _operands(M, N, K, False, False, 9)
    dense = ops.project_f32(x, w, N)
    xz, wz = x.clone(), w.clone()
    xz[M // 2:] = 0
    wz[100:200] = 0
    got = ops.project_f32(xz, wz, N)
    keep = torch.ones(N, dtype=torch.bool, device="cuda")
    keep[100:200] = False
    assert torch.equal(got[:M // 2, keep], dense[:M // 2, keep])
    assert not bool(got[M // 2:].any()) and not bool(got[:, 100:200].any())
    assert _us(lambda: ops.project_f32(xz, wz, N)) <= 3 * _us(lambda: ops.project_f32(x, w, N))


@pytest.mark.parametrize("scale", [2.0 ** -75, 2.0 ** -100])
def test_projection_beside_a_kink_where_squares_underflow(scale, monkeypatch):
    """Rows whose 2-norm underflows in float32 still take the chain's side of the kink at 0."""
    from pom_b200 import ops

    monkeypatch.setattr(ops, "F32_PROJECT_MIN_WEIGHTS", 0)
    x, w = _operands(256, 512, 300, False, False, 10)
    got, chain = ops.project_f32(x * scale, w, 512), _planes(x * scale, w, use=False, fma=True)
    assert torch.equal(got > 0, chain > 0)
    eps = 2.0 ** -24 * 300 ** 0.5 * (x.norm(dim=1)[:, None].double() * scale * w.norm(dim=1)[None].double())
    near = chain.abs().double() <= 4 * eps
    assert bool(near.any()) and torch.equal(got[near], chain[near])


class _Budget:
    """Stands in for a GPU that has ``cap`` bytes: torch.empty raises beyond it, as the caching allocator would."""

    def __init__(self, monkeypatch, cap):
        self.refused = 0
        empty = torch.empty

        def limited(*size, dtype=torch.float32, device=None, **kw):
            t = empty(*size, dtype=dtype, device=device, **kw)
            if t.is_cuda and torch.cuda.memory_allocated() > cap:
                self.refused += 1
                del t
                raise torch.OutOfMemoryError("no room")
            return t

        monkeypatch.setattr(torch, "empty", limited)


@pytest.mark.parametrize("cross", [False, True], ids=["self", "cross"])
def test_a_step_that_fits_without_planes_fits_with_them(cross, monkeypatch):
    """Planes are there when memory is: a training step runs in the memory that the FMA kernel alone needs, and the
    result is the same but for the order of additions."""
    from unittest import mock

    from pom_b200 import PoM, ops

    torch.manual_seed(2)
    mod = PoM(384, 2, 2).cuda()
    x, xc, dy = (torch.randn(4, 500, 384, device="cuda") for _ in range(3))
    ins = [x.requires_grad_()] + ([xc.requires_grad_()] if cross else [])
    wrt = ins + [mod.qc_proj.weight, mod.se_bias, mod.po_coeff, mod.ag_proj.weight]

    def step():
        return torch.autograd.grad(mod(*ins), wrt, dy)

    with mock.patch.object(ops, "f32_planes_pay", lambda *_: False):
        step()  # caches of the layer
        base = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        want = step()
        needs = torch.cuda.max_memory_allocated() - base
    with monkeypatch.context() as m:
        budget = _Budget(m, torch.cuda.memory_allocated() + needs)
        got = step()
    assert budget.refused > 0
    for a, b in zip(got, want):
        assert ((a - b).norm() / b.norm()).item() <= 1e-5  # float32 sums in another order


def test_planes_give_way_to_an_output_that_does_not_fit(monkeypatch):
    from pom_b200 import ops

    a, b = _operands(512, 300, 256, False, False, 12)
    pl, spare = ops.F32Planes(), ops.F32Planes()
    want = _planes(a, b, a_planes=pl)
    spare.take(a)
    with monkeypatch.context() as m:
        _Budget(m, torch.cuda.memory_allocated() + 4096)  # the output takes more, and less than the planes
        got = ops.gemm(a, b, a_planes=pl, spare=(spare,))
    assert pl.buf is None and spare.buf is None
    assert ((got - want).norm() / want.norm()).item() <= 1e-6
    with pytest.raises(torch.OutOfMemoryError), monkeypatch.context() as m:
        _Budget(m, torch.cuda.memory_allocated())
        ops.gemm(a, b)
