"""The float32 projections against sums in 64 bits, at the edges of their tiles and of the ranges that pick a kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (M, N, K): one and the most tokens of a kernel, token counts between its templates, columns and rows that end inside a tile,
# a K that leaves warps and blocks of the split without rows
SHAPES = [(1, 4096, 4096), (2, 132, 4), (3, 260, 72), (8, 12288, 4096), (9, 128, 1000), (16, 4, 4096), (17, 1024, 36), (31, 36, 11008), (64, 516, 260),
          (5, 70, 33), (65, 70, 33), (33, 4100, 100),
          # the tensor-core kernel: token counts at and beside its blocks, ends inside a tile, a stage and a split
          (65, 4, 4), (80, 260, 72), (192, 128, 64), (193, 516, 2048), (352, 4096, 512), (400, 36, 11008), (1000, 384, 96)]


def worst(got, x, w):
    """Largest error in units of what a sum of K float products in any order may be off: the norm of the products."""
    ref = x.astype(np.float64) @ w.astype(np.float64)
    size = np.sqrt((x.astype(np.float64) ** 2) @ (w.astype(np.float64) ** 2)) + 1e-300
    return (np.abs(got - ref) / size).max()


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("nk", [False, True])
@pytest.mark.parametrize("pad", [0, 4, 3])
def test_gemm_f32_against_64_bits(ob, cuda, M, N, K, nk, pad):
    torch = cuda
    rng = np.random.default_rng(M * N + K)
    x, w = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    dw = torch.from_numpy(np.ascontiguousarray(w.T if nk else w)).cuda()
    y = torch.full((M, N + pad), 7.0, device="cuda")
    import ctypes as C
    ob._check(ob.lib().onellm_gemm_ld(C.c_int(ob.F32), ob._p(torch.from_numpy(x).cuda()), ob._p(dw), ob._p(y), C.c_long(N + pad), C.c_int(M),
                                      C.c_int(N), C.c_int(K), C.c_int(ob.W_NK if nk else ob.W_KN), ob._stream(None)))
    got = y.cpu().numpy()
    # random rounding: sqrt(K) sums, each off by at most 2^-24 of a partial sum, which is at most the norm of the products or so
    assert worst(got[:, :N].astype(np.float64), x, w) < 4 * np.sqrt(K) * 2.0 ** -24 + 2.0 ** -22
    assert (got[:, N:] == 7.0).all()


@pytest.mark.parametrize("M", [3, 40, 70, 200])
def test_gemm_f32_keeps_infinities_and_nan(ob, cuda, M):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, 256, generator=g, device="cuda"), torch.randn(256, 384, generator=g, device="cuda")
    x[1, 5], x[2, 9], w[7, 11], w[200, 300] = float("inf"), float("nan"), float("-inf"), 3e38
    x[0, 200] = 100.0
    y = torch.empty(M, 384, device="cuda")
    ob.gemm(ob.F32, x, w, y, M, 384, 256)
    ref = (x.double() @ w.double()).float()
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(y), same(ref))


def both_ways(ob, torch, x, w, nk):
    """The product by the kernel that takes the call, and by the chain of multiply-adds of the tiled kernel, which takes unaligned rows."""
    (M, K), N = x.shape, w.shape[1]
    shifted = torch.empty(M * K + 1, device="cuda")[1:].view(M, K)
    shifted.copy_(x)
    dw, out = w.T.contiguous() if nk else w, []
    for a in (x, shifted):
        y = torch.empty(M, N, device="cuda")
        ob.gemm(ob.F32, a, dw, y, M, N, K, ob.W_NK if nk else ob.W_KN)
        out.append(y)
    return out


def off(y, x, w):
    ref = x.double() @ w.double()
    return float((y.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("K", [4, 16, 64, 252, 256, 260, 1024, 4096])
@pytest.mark.parametrize("kind", ["normal", "positive", "constant", "ends"])
@pytest.mark.parametrize("nk", [False, True])
def test_more_than_64_tokens_are_no_less_exact_than_a_chain(ob, cuda, K, kind, nk):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(K)
    make = {"normal": lambda *s: torch.randn(*s, generator=g, device="cuda"), "positive": lambda *s: torch.rand(*s, generator=g, device="cuda"),
            "constant": lambda *s: torch.full(s, 1.0078124, device="cuda"), "ends": lambda *s: torch.full(s, 1 + 2.0 ** -7 - 2.0 ** -23, device="cuda")}[kind]
    x, w = make(130, K), make(K, 260)
    fast, chain = (off(y, x, w) for y in both_ways(ob, torch, x, w, nk))
    # equal operands are the chain's good or bad luck: one step of the result's last place is let pass
    assert fast <= (1.02 * chain if kind in ("normal", "positive") else max(chain, 2.0 ** -23))


@pytest.mark.parametrize("K", [256, 1100])
@pytest.mark.parametrize("sx,sw", [(1e-35, 1), (1e-39, 1), (1, 1e-38), (1e30, 1e-36), (1e-20, 1e-19), (1e-30, 1e-10), (3e37, 1e-3)])
@pytest.mark.parametrize("nk", [False, True])
def test_operands_at_the_ends_of_the_range(ob, cuda, K, sx, sw, nk):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(K)
    rnd = lambda s, *n: (torch.randn(*n, generator=g, device="cuda", dtype=torch.double) * s).float()
    x, w = rnd(sx, 70, K), rnd(sw, K, 132)
    fast, chain = (off(y, x, w) for y in both_ways(ob, torch, x, w, nk))
    assert fast <= 1.02 * chain


@pytest.mark.parametrize("M,N,K", [(200, 384, 256), (300, 132, 4096)])
def test_few_small_operands_among_others(ob, cuda, M, N, K):
    # too small for three bf16 values, and of no weight in any result but one; a row of zeros and one whose results are tiny
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(K, N, generator=g, device="cuda")
    x[3, ::7], x[M - 1, 5], w[2, ::3], x[9], x[M - 2] = 1.1e-36, -3e-40, 1.3e-37, 0.0, 1e-36 * x[0]
    fast, chain = both_ways(ob, torch, x, w, False)
    assert off(fast, x, w) <= 1.02 * off(chain, x, w)
    assert off(fast[M - 2:M - 1], x[M - 2:M - 1], w) <= 1.02 * off(chain[M - 2:M - 1], x[M - 2:M - 1], w) and not fast[9].any()


@pytest.mark.parametrize("M,N,K", [(130, 200, 512), (70, 132, 8192)])
def test_values_that_are_not_finite_beside_a_residual_in_place(ob, cuda, M, N, K):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w, r = (torch.randn(*s, generator=g, device="cuda") for s in ((M, K), (K, N), (M, N)))
    x[4], x[60, K - 1], w[100, 7] = float("nan"), float("inf"), float("-inf")
    y = r.clone()
    ob.project(ob.F32, x, w, None, y, M, N, K, resid=y, scale=0.5)
    ref = r.double() + 0.5 * (x.double() @ w.double())
    finite = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(y), finite) and torch.equal(torch.isnan(y), torch.isnan(ref))
    assert float((y.double() - ref)[finite].norm() / ref[finite].norm()) < 2e-6


@pytest.mark.parametrize("M", [1, 6, 30, 100])
def test_projection_f32_gate_and_residual(ob, cuda, M):
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    K, N = 200, 140
    x, w, w2, r = rnd(M, K), rnd(K, N), rnd(K, N), rnd(M, N + 4)
    y = r.clone()
    ob.project(ob.F32, x, w, None, y, M, N, K, ldy=N + 4, resid=y, scale=0.3)
    ref = r[:, :N].double() + 0.3 * (x.double() @ w.double())
    assert (y[:, :N] - ref).abs().max() < 1e-4 and torch.equal(y[:, N:], r[:, N:])
    y = torch.zeros(M, N, device="cuda")
    ob.project(ob.F32, x, w, w2, y, M, N, K, act=ob.GATE_RELU)
    ref = (x.double() @ w.double()).clamp(min=0) * (x.double() @ w2.double())
    assert (y - ref).abs().max() < 2e-3 * 0.1 * ref.abs().max()
