"""The end of a context projection: gates of any size, float outputs on top of a residual, at the edges of tiles and forms."""
import numpy as np
import pytest

from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


# one tile, the last tile of rows and of columns cut, one wave and several, blocks alone and in pairs, K split
@pytest.mark.parametrize("M,N,K", [(65, 8, 128), (129, 264, 192), (300, 5640, 512), (1030, 4096, 512), (2060, 2056, 1024)])
@pytest.mark.parametrize("form", ["float", "element", "gated"])
def test_outputs_at_the_edges(cuda, ob, M, N, K, form):
    g = cuda.Generator(device="cuda").manual_seed(M + N)
    rnd = lambda *s: cuda.randn(s, generator=g, device="cuda")
    x, W, W2 = rnd(M, K).bfloat16(), (rnd(K, N) * 0.05).bfloat16(), (rnd(K, N) * 0.05).bfloat16()
    ld, f32 = N + 24, form != "element"
    y = rnd(M, ld) if f32 else rnd(M, ld).bfloat16()
    old = y.double().clone()
    ob.project(ob.BF16, x, W, W2 if form == "gated" else None, y, M, N, K, act=ob.GATE_SILU, resid=y if f32 else None, scale=0.5 if f32 else 1.0, ldy=ld,
               f32=f32)
    ref = x.double() @ W.double()
    if form == "gated":
        ref = cuda.nn.functional.silu(ref) * (x.double() @ W2.double())
    if f32:  # on top of a residual
        ref = old[:, :N] + 0.5 * ref
    assert cuda.equal(y[:, N:].double(), old[:, N:])
    # float: the order of sums of K products and the fast exponential; elements: one rounding to bfloat16
    assert rel_err(y[:, :N].double().cpu().numpy(), ref.cpu().numpy()) < (1e-5 if f32 else 4e-3)
    assert ob.lib().onellm_gemm_timeout_flag() == 0


@pytest.mark.parametrize("act,name", [("GATE_SILU", "silu"), ("GATE_CLAMPED", "clamped"), ("GATE_RELU", "relu")])
@pytest.mark.parametrize("M", [100, 1000])
def test_gates_of_any_size(cuda, ob, act, name, M):
    # column n: g = a[n], u = b[n], products of one K row; sizes from far below one to where the exponential and the product leave float
    N, K, limit = 4096, 64, 7.0
    rng = np.random.default_rng(0)
    a = rng.choice([-1, 1], N) * 10.0 ** rng.uniform(-30, 3, N)
    a[:64] = np.linspace(-95, -60, 64)
    a[64:72] = [-3e38, -1e30, 1e30, 3e38, 0.0, -104, np.nan if name == "silu" else 1.0, np.inf]  # the others' bounds win over NaN
    b = rng.choice([-1, 1], N) * 10.0 ** rng.uniform(-3, 3, N)
    x, W, W2 = cuda.zeros(M, K, device="cuda"), cuda.zeros(K, N, device="cuda"), cuda.zeros(K, N, device="cuda")
    x[:, 0], W[0], W2[0] = 1.0, cuda.from_numpy(a).cuda().float(), cuda.from_numpy(b).cuda().float()
    x, W, W2, y = x.bfloat16(), W.bfloat16(), W2.bfloat16(), cuda.zeros(M, N, device="cuda")
    ob.project(ob.BF16, x, W, W2, y, M, N, K, act=getattr(ob, act), limit=limit, f32=True)
    g, u = W[0].double(), W2[0].double()
    if name == "clamped":
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        ref = g * cuda.sigmoid(1.702 * g) * (u + 1)
    else:
        ref = (cuda.nn.functional.silu(g) if name == "silu" else cuda.relu(g)) * u
    got, ref = y.double().cpu().numpy(), ref.cpu().numpy()
    for row in (0, M // 2, M - 1):
        assert np.array_equal(np.isnan(got[row]), np.isnan(ref))
        at = np.isfinite(ref) & (np.abs(ref) < 3e38) & (np.abs(ref) > 1e-33)
        # the fast exponential: 2 ulp and 1.2e-7 of its argument
        assert np.all(np.abs(got[row][at] / ref[at] - 1) < 4e-7 + 2.4e-7 * np.minimum(np.abs(g.cpu().numpy()[at]) * 1.702, 110))
        assert np.all(np.abs(got[row][~np.isnan(ref) & (np.abs(ref) <= 1e-33)]) < 1e-32)
