"""Context-phase projections with few tiles: the K split over a cluster, against products in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# tokens at the edges of one and two row tiles, K that leaves ranks uneven slices and a last slice cut short, columns that end inside a tile
SHAPES = [(65, 256, 4096), (128, 8, 4096), (129, 264, 1032), (238, 4096, 4096), (256, 1000, 11008), (257, 520, 512), (300, 4096, 136), (1000, 32, 4096),
          # many tiles: blocks in pairs on 256 rows, the last of which only one of them has, and several tiles per pair
          (1290, 8712, 224), (1500, 8008, 1056)]


def err(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


def operands(torch, M, N, K, dtype, seed=0, n=1):
    g = torch.Generator(device="cuda").manual_seed(M + N + K + seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    return rnd(M, K).to(dtype), [(rnd(K, N) / K ** 0.5).to(dtype) for _ in range(n)], rnd


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain_and_gated(ob, cuda, M, N, K):
    torch = cuda
    x, (w, w2), _ = operands(torch, M, N, K, torch.half, n=2)
    y = torch.empty(M, N, device="cuda", dtype=torch.half)
    ref = x.double() @ w.double()
    ob.gemm(ob.F16, x, w, y, M, N, K)
    assert err(y, ref) < 3e-4  # half a unit in the last place of fp16, root mean square
    if K % 32 == 0:
        ob.gemm(ob.F16, x, w.T.contiguous(), y.zero_(), M, N, K, ob.W_NK)
        assert err(y, ref) < 3e-4
    if K % 16 == 0:
        ob.gemm_swiglu(ob.F16, x, w, w2, y.zero_(), M, N, K)
        assert err(y, torch.nn.functional.silu(ref) * (x.double() @ w2.double())) < 4e-4
    assert ob.lib().onellm_gemm_timeout_flag() <= 0


@pytest.mark.parametrize("M,N,K", [s for s in SHAPES if s[1] % 8 == 0 and s[2] % 16 == 0])
def test_row_statistics_residual_and_bias(ob, cuda, M, N, K):
    torch = cuda
    x, (w,), rnd = operands(torch, M, N, K, torch.half)
    ss = x.float().square().view(M, 1, K).sum(-1).contiguous()
    r, bias = rnd(M, N).half(), rnd(N).half()
    y, parts = r.clone(), ob.gemm_rows_parts(N)
    out = torch.full((M, parts), -1.0, device="cuda")
    ob.gemm_rows(ob.F16, x, w, None, y, M, N, K, ss, 1, 1e-5, y, bias, out)
    ref = r.double() + bias.double() + (x.double() @ w.double()) * torch.rsqrt(ss.double() / K + 1e-5)
    assert err(y, ref) < 4e-4
    pad = torch.zeros(M, parts * 256, device="cuda", dtype=torch.double)
    pad[:, :N] = y.double()
    assert err(out, pad.view(M, parts, 256).square().sum(-1)) < 1e-6
    again = r.clone()
    ob.gemm_rows(ob.F16, x, w, None, again, M, N, K, ss, 1, 1e-5, again, bias, out)
    assert torch.equal(y, again)


@pytest.mark.parametrize("M,N,K", [s for s in SHAPES if s[2] % 16 == 0])
def test_bfloat16_into_a_float_stream(ob, cuda, M, N, K):
    torch = cuda
    x, (w,), rnd = operands(torch, M, N, K, torch.bfloat16)
    y = rnd(M, N + 8)
    ref = y[:, :N].double() + 0.3 * (x.double() @ w.double())
    side = y[:, N:].clone()
    ob.project(ob.BF16, x, w, None, y, M, N, K, ldy=N + 8, f32=True, resid=y, scale=0.3)
    assert err(y[:, :N], ref) < 2e-6 and torch.equal(y[:, N:], side)  # float sums of exact products


# every kernel a gated projection can take: few tokens, K split, blocks alone and in pairs
@pytest.mark.parametrize("M,N,K", [(64, 256, 512), (65, 256, 512), (100, 1024, 1024), (128, 5632, 2048), (300, 200, 176)] + [s for s in SHAPES if s[2] % 16 == 0])
@pytest.mark.parametrize("resid", [False, True])
def test_gated_bfloat16_into_floats(ob, cuda, M, N, K, resid):
    torch = cuda
    x, (w, w2), rnd = operands(torch, M, N, K, torch.bfloat16, n=2)
    y = rnd(M, N + 8)
    side, start = y[:, N:].clone(), y[:, :N].double()
    ref = (x.double() @ w.double()).clamp(min=0) * (x.double() @ w2.double())
    if resid:
        ob.project(ob.BF16, x, w, w2, y, M, N, K, ldy=N + 8, act=ob.GATE_RELU, f32=True, resid=y, scale=0.3)
        ref = start + 0.3 * ref
    else:
        ob.project(ob.BF16, x, w, w2, y, M, N, K, ldy=N + 8, act=ob.GATE_RELU, f32=True)
    assert err(y[:, :N], ref) < 4e-6 and torch.equal(y[:, N:], side)  # two float sums of exact products, multiplied


def test_first_call_of_a_shape_inside_a_capture(ob, cuda):
    torch = cuda
    x, (w,), _ = operands(torch, 200, 776, 1000, torch.half)
    y = torch.zeros(200, 776, device="cuda", dtype=torch.half)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ob.gemm(ob.F16, x, w, y, 200, 776, 1000)
    g.replay()
    torch.cuda.synchronize()
    assert err(y, x.double() @ w.double()) < 3e-4


# decode projections: every K split from one to eight, the last of them with fewer rows or none, columns that end inside a block
@pytest.mark.parametrize("M", [1, 9, 17, 32])
@pytest.mark.parametrize("N,K", [(4096, 16384), (4096, 4096), (2080, 4096), (4096, 928), (5632, 2048), (12304, 512), (32000, 256), (136, 48), (8, 4096)])
def test_decode_projection_plans(ob, cuda, M, N, K):
    torch = cuda
    x, (w, w2), _ = operands(torch, M, N, K, torch.half, n=2)
    y, ref = torch.empty(M, N, device="cuda", dtype=torch.half), x.double() @ w.double()
    ob.gemm(ob.F16, x, w, y, M, N, K)
    assert err(y, ref) < 3e-4
    ob.gemm_swiglu(ob.F16, x, w, w2, y.zero_(), M, N, K)
    assert err(y, torch.nn.functional.silu(ref) * (x.double() @ w2.double())) < 4e-4
    k_split, ring, blocks = ob.gemm_plan_query(M, N, K)
    assert 1 <= k_split <= 8 and ring >= 3 and blocks == k_split * -(-N // 128)
