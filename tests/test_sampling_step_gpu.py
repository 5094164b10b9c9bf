"""Top-K of rows at the edges of a block's registers, and the sampling that follows it in the same launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(kind, V, rng):
    if kind == "equal":
        return np.full((3, V), 1.5)
    if kind == "runs":  # ties across the groups of columns that a thread holds
        return rng.integers(0, 3, (3, V)).astype(np.float64)
    x = rng.standard_normal((3, V))
    x[1, ::2] = -np.inf
    x[2, : V // 2] = np.nan
    return x


@pytest.mark.parametrize("dt", ["f16", "f32"])
@pytest.mark.parametrize("kind", ["equal", "runs", "wide"])
@pytest.mark.parametrize("V,K", [(64, 64), (255, 1), (4097, 16), (8200, 7), (32761, 64), (32767, 17), (32768, 16)])
def test_topk_at_the_edges(ob, cuda, orc, dt, kind, V, K):
    torch = cuda
    x = _rows(kind, V, np.random.default_rng(V)).astype(np.float16).astype(np.float32)
    val = torch.zeros(3, K, device="cuda")
    idx = torch.zeros(3, K, device="cuda", dtype=torch.int32)
    ob.topk(ob.F16 if dt == "f16" else ob.F32, torch.from_numpy(x).cuda().to(torch.float16 if dt == "f16" else torch.float32), 3, V, K, val, idx)
    rv, ri = orc.topk(x, K)
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(val.cpu().numpy(), rv, equal_nan=True)


@pytest.mark.parametrize("literal", [False, True])
@pytest.mark.parametrize("vocab", [1000, 32768, 33001])  # the last one is too long for one launch
@pytest.mark.parametrize("K", [1, 5, 33, 64])
def test_a_step_samples_what_the_two_launches_sample(ob, cuda, vocab, K, literal):
    torch = cuda
    B, T = 5, 0.7
    m = ob.Llama(num_layers=1, hidden=128, head_num=2, kv_head_num=2, head_size=64, inter_size=256, vocab_size=vocab, max_seq_len=32, max_batch=B)
    m.init_random(K, 0.1)
    m.set_sampling(top_k=K, temperature=T, literal_walk=literal)
    rng = np.random.default_rng(vocab)
    first = m.prefill(rng.integers(0, vocab, (B, 4)).astype(np.int32))
    out = np.zeros(B, np.int32)
    for at in range(5):
        if at:
            m.decode_step(None, out)
        got = out if at else np.asarray(first)
        u, step, _ = m.last_draws()
        logits = torch.from_numpy(m.logits(B)).cuda()  # 16-bit logits are exact in float
        val, idx = torch.zeros(B, K, device="cuda"), torch.zeros(B, K, device="cuda", dtype=torch.int32)
        ids, u2 = torch.zeros(B, device="cuda", dtype=torch.int32), torch.zeros(B, device="cuda")
        ob.topk(ob.F32, logits, B, vocab, K, val, idx)
        ob.topk_sample(idx, val, B, K, T, step, vocab, 2, ids, u_out=u2, literal_walk=literal)
        assert np.array_equal(u[:B], u2.cpu().numpy())
        assert np.array_equal(got, ids.cpu().numpy())
    m.close()
