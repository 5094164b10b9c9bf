"""Decode projections of up to 16 tokens: the partial sums that the blocks of a cluster send one another."""
import numpy as np
import pytest

from tests.conftest import rel_err

pytestmark = pytest.mark.gpu


# shares of a tile that end inside a token's row, ranks with few elements, columns behind the last one, two weights, several rings of stages
@pytest.mark.parametrize("ks", [1, 2, 3, 5, 7, 8])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(8, 512), (136, 1040), (640, 4096)])
def test_every_split(cuda, ob, M, N, K, ks):
    g = cuda.Generator(device="cuda").manual_seed(M * N + ks)
    rnd = lambda *s: cuda.randn(s, generator=g, device="cuda")
    x, W, W2 = rnd(M, K).bfloat16(), (rnd(K, N) * 0.05).bfloat16(), (rnd(K, N) * 0.05).bfloat16()
    one, two = x.double() @ W.double(), x.double() @ W2.double()
    y = cuda.zeros(M, N, device="cuda")
    for dual in (0, 1):
        ob.gemm_plan_override(N, K, dual, ks, 4)
        try:
            ob.project(ob.BF16, x, W, W2 if dual else None, y, M, N, K, act=ob.GATE_RELU, f32=True)
            again = y.clone()
            ob.project(ob.BF16, x, W, W2 if dual else None, y, M, N, K, act=ob.GATE_RELU, f32=True)
        finally:
            ob.gemm_plan_override(N, K, dual, 0)
        assert cuda.equal(y, again)
        # a range adds up in K / (16 ks) steps of the tensor cores, each of which cuts off at most 2^-23 of the sum; then ks float sums
        bound = (1 + dual) * (K / (16 * ks) + ks) * 2.0 ** -23
        assert rel_err(y.double().cpu().numpy(), (cuda.relu(one) * two if dual else one).cpu().numpy()) < bound


@pytest.mark.parametrize("ks", [1, 3, 8])
@pytest.mark.parametrize("M", [3, 16])
def test_row_norms_of_the_split_rows(cuda, ob, M, ks):
    N, K = 264, 2048
    g = cuda.Generator(device="cuda").manual_seed(M + ks)
    x, W = cuda.randn(M, K, generator=g, device="cuda").half() * 3, (cuda.randn(K, N, generator=g, device="cuda") * 0.02).half()
    y = cuda.zeros(M, N, device="cuda", dtype=cuda.float16)
    ob.gemm_plan_override(N, K, 0, ks, 5)
    try:
        ob.gemm_fused(ob.F16, x, W, None, y, M, N, K, rms_eps=1e-5)
    finally:
        ob.gemm_plan_override(N, K, 0, 0)
    xd = x.double()
    ref = (xd * cuda.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)) @ W.double()
    assert rel_err(y.double().cpu().numpy(), ref.cpu().numpy()) < 1e-3  # one rounding to half: 2^-11
