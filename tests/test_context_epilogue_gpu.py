"""The end of a context projection: gates of any size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
