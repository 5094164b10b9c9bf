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
