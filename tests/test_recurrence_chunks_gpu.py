"""Context passes of the gated recurrences in chunks of 128 tokens on the tensor cores, against the token by token sums in 64 bits."""
import numpy as np
import pytest

from oracle import finuvik_ref as fr
from tests.conftest import rel_err
from tests.device import Dev, host, rounded
from tests.test_finuvik_kernels_gpu import ref_recurrence, run_recurrence
from tests.test_fuposun_kernels_gpu import ref_gla, run_gla

pytestmark = pytest.mark.gpu
TOL = 1.2e-2
# The state is float and its sums are taken as closely as float adds them: 1e-7 for the gates of a trained model, up to 4.4e-7 where hundreds
# of gates are the same one close to 1, 3e-7 where all terms have one sign.  The outputs are rounded to bfloat16.
STATE = 1e-6


def positions(ob, d, counts, hist):
    return ob.TokenPositions(d.i32(np.concatenate([[0], np.cumsum(counts)])).data_ptr(), d.i32(hist).data_ptr(), len(counts), None, None)


# sequences that end at, in front of and behind the edges of a chunk; the second portion starts from the state of the first
COUNTS = [([384, 640, 129], [1, 500, 512]), ([300], [1031]), ([255, 257, 640, 128], [511, 1, 513, 127])]


@pytest.mark.parametrize("H,dk,dv", [(2, 64, 128), (3, 128, 128), (1, 192, 256), (2, 256, 384)])
@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("gates", ["learned", "slow", "fast"])
def test_tied(cuda, ob, H, dk, dv, counts, gates):
    # slow: nearly every gate is the same one close to 1; fast: chunks forget channels far below 2^-80, others hardly anything
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(dk + dv)
    zb = fr.round_bf16({"learned": rng.uniform(-1, 6, H * dk), "slow": np.full(H * dk, 9.0), "fast": rng.uniform(-12, 8, H * dk)}[gates])
    lower = fr.round_bf16(rng.uniform(0, 0.95, H * dk) * (rng.uniform(size=H * dk) > 0.3)) if gates == "learned" else np.zeros(H * dk)
    w = fr.round_bf16(1 + 0.3 * rng.standard_normal(dv))
    B = len(counts[0])
    state = d.zeros(B, H, dk, dv, f32=True) + float("nan")  # what a freed sequence left behind: a new one must not see it
    ref_state, hist = [np.zeros((H, dk, dv)) for _ in range(B)], [0] * B
    for portion in counts:
        z_std = 0.0 if gates == "slow" else 1.0
        q, z, v = (rounded(rng.standard_normal((sum(portion), H, m)) * s, "bf16") for m, s in ((dk, 1.0), (dk, z_std), (dv, 1.0)))
        got = run_recurrence(ob, d, H, dk, dv, q, z, v, zb, lower, w, state, positions(ob, d, portion, hist), B, scale_out=0.6)
        assert ob.lib().onellm_gemm_timeout_flag() == 0
        at = 0
        for b, n in enumerate(portion):
            s = slice(at, at + n)
            assert rel_err(got[s], 0.6 * ref_recurrence(q[s], z[s], v[s], zb, lower, w, ref_state[b])) < TOL, (portion, b)
            at += n
            hist[b] += n
    for b in range(B):
        assert rel_err(host(state[b]), ref_state[b]) < STATE


@pytest.mark.parametrize("H,dk,dv,rank", [(2, 64, 128, 5), (1, 128, 128, 16), (2, 256, 512, 16), (1, 192, 1024, 64)])
@pytest.mark.parametrize("tau,gated", [(16.0, True), (0.3, False)])
def test_keyed(cuda, ob, H, dk, dv, rank, tau, gated):
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(dk + dv)
    A, zb = (fr.round_bf16(x) for x in (rng.standard_normal((H * dk, rank)) / np.sqrt(rank), rng.uniform(-1, 6, H * dk)))
    w, qs = fr.round_bf16(1 + 0.3 * rng.standard_normal(dv)), dk ** -0.5
    for counts in COUNTS[:2]:
        B = len(counts[0])
        state = d.zeros(B, H, dk, dv, f32=True) + float("nan")
        ref_state, hist = [np.zeros((H, dk, dv)) for _ in range(B)], [0] * B
        for portion in counts:
            T = sum(portion)
            x = tuple(rounded(rng.standard_normal(s), "bf16") for s in ((T, H, dk), (T, H, dk), (T, H, dv), (T, rank), (T, H, dv)))
            got = run_gla(ob, d, H, dk, dv, x, A, zb, w, state, positions(ob, d, portion, hist), tau, qs, scale_out=0.6, gated=gated)
            at = 0
            for b, n in enumerate(portion):
                ref = 0.6 * ref_gla([y[at:at + n] for y in x], A, zb, w, ref_state[b], tau, qs, gated=gated)
                assert rel_err(got[at:at + n], ref) < TOL, (portion, b)
                at += n
                hist[b] += n
        for b in range(B):
            assert rel_err(host(state[b]), ref_state[b]) < STATE


@pytest.mark.parametrize("what", ["value", "query", "gate", "key"])
def test_what_is_not_finite_reaches_its_own_and_later_tokens_only(cuda, ob, what):
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(1)
    H, dk, dv, n, rank, t = 1, 64, 128, 300, 4, 200
    x = [rounded(rng.standard_normal(s), "bf16") for s in ((n, H, dk), (n, H, dk), (n, H, dv), (n, rank), (n, H, dv))]
    A, zb, w = rng.standard_normal((dk, rank)).astype(np.float32), np.ones(dk), np.ones(dv)
    run = lambda state: run_gla(ob, d, H, dk, dv, x, A, zb, w, state, positions(ob, d, [n], [0]), 16.0, 1.0, gated=False)
    states = [d.zeros(1, H, dk, dv, f32=True) for _ in range(2)]
    clean = run(states[0])
    x[{"value": 2, "query": 0, "gate": 3, "key": 1}[what]][(t,) + (0,) * (1 if what == "gate" else 2)] = np.inf if what == "value" else np.nan
    got = run(states[1])
    assert rel_err(got[:t], clean[:t]) < TOL and np.all(np.isnan(got[t]).any(-1))
    if what == "query":
        assert rel_err(got[t + 1:], clean[t + 1:]) < TOL and rel_err(host(states[1]), host(states[0])) < STATE
    else:
        assert np.isnan(got[t + 1:]).any(-1).all() and not np.isfinite(host(states[1])).all()


@pytest.mark.parametrize("left", [0x00, 0x01, 0xff])
@pytest.mark.parametrize("dv,col", [(128, 0), (128, 100), (256, 5), (256, 130), (384, 130), (384, 200)])
@pytest.mark.parametrize("keyed", [False, True])
def test_a_value_that_is_not_finite_is_its_column_alone(cuda, ob, left, dv, col, keyed):
    # in either half of a head's columns (which two blocks look through) and in its second tile, whatever the work space holds
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(dv + col)
    H, dk, n, rank, t = 2, 64, 400, 4, 200
    x = [rounded(rng.standard_normal(s), "bf16") for s in ((n, H, dk), (n, H, dk), (n, H, dv), (n, rank), (n, H, dv))]
    A, zb, w = rng.standard_normal((H * dk, rank)), np.ones(H * dk), np.ones(dv)

    def run(state):
        tp = positions(ob, d, [n], [0])
        if keyed:
            return run_gla(ob, d, H, dk, dv, x, A, zb, w, state, tp, 16.0, 1.0, gated=False, left=left)
        return run_recurrence(ob, d, H, dk, dv, x[0], x[1], x[2], zb, np.zeros(H * dk), w, state, tp, 1, left=left)

    states = [d.zeros(1, H, dk, dv, f32=True) for _ in range(2)]
    clean = run(states[0])
    x[2][t, 0, col] = np.inf
    got = run(states[1])
    assert np.array_equal(got[:t], clean[:t]) and np.array_equal(got[:, 1], clean[:, 1])
    assert np.isnan(got[t:, 0]).any(-1).all()
    was, now = (host(s)[0] for s in states)
    others = np.arange(dv) != col
    assert np.array_equal(now[1], was[1]) and np.array_equal(now[0][:, others], was[0][:, others])
    assert not np.isfinite(now[0][:, col]).any()


@pytest.mark.parametrize("keyed", [False, True])
@pytest.mark.parametrize("size", [2.0 ** 20, 2.0 ** 50])
def test_large_values_beside_channels_that_nearly_forget(cuda, ob, keyed, size):
    # half a chunk keeps 2^-79 of some channels: a key over that share, times such a value, is beyond float, the state is not
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(3)
    H, dk, dv, n = 2, 64, 128, 300
    x = [rounded(rng.standard_normal(s), "bf16") for s in ((n, H, dk), (n, H, dk), (n, H, dv), (n, 4), (n, H, dv))]
    x[2][:, 1, 64:] *= size  # of one head and one half of its columns
    w, zb = np.ones(dv), np.full(H * dk, 4.0)
    keep = 2.0 ** (-79 / 64)  # of a channel and token
    zb[::16] = np.log(keep / (1 - keep))
    state, ref_state = d.zeros(1, H, dk, dv, f32=True), np.zeros((H, dk, dv))
    tp = positions(ob, d, [n], [0])
    if keyed:
        A = np.zeros((H * dk, 4))
        got = run_gla(ob, d, H, dk, dv, x, A, zb, w, state, tp, 1.0, 1.0, gated=False)
        ref = ref_gla(x, A, zb, w, ref_state, 1.0, 1.0, gated=False)
    else:
        x[1][:] = 0.0
        got = run_recurrence(ob, d, H, dk, dv, x[0], x[1], x[2], zb, np.zeros(H * dk), w, state, tp, 1)
        ref = ref_recurrence(x[0], x[1], x[2], zb, np.zeros(H * dk), w, ref_state)
    for h in range(H):
        assert rel_err(got[:, h], ref[:, h]) < TOL
        for half in (slice(0, 64), slice(64, 128)):
            assert rel_err(host(state)[0, h][:, half], ref_state[h][:, half]) < STATE


@pytest.mark.parametrize("dk,fast", [(64, 1), (64, 64), (128, 17), (128, 40), (192, 25), (192, 192), (256, 1), (256, 33), (256, 256)])
@pytest.mark.parametrize("keyed", [False, True])
def test_channels_that_forget(cuda, ob, dk, fast, keyed):
    # so many channels of one head below 2^-80 in half a chunk, none of the other: one of a pair, more than a group takes, all
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(dk + fast)
    H, dv, counts = 2, 128, [300, 1, 600]
    n = sum(counts)
    x = [rounded(rng.standard_normal(s), "bf16") for s in ((n, H, dk), (n, H, dk), (n, H, dv), (n, 4), (n, H, dv))]
    w, zb, A = np.ones(dv), np.full((H, dk), 4.0), fr.round_bf16(rng.standard_normal((H * dk, 4)) * 0.2)
    zb[1, rng.permutation(dk)[:fast]] = -2.0
    state, ref_state = d.zeros(3, H, dk, dv, f32=True), [np.zeros((H, dk, dv)) for _ in counts]
    tp = positions(ob, d, counts, [0, 0, 0])
    if keyed:
        got = run_gla(ob, d, H, dk, dv, x, A, zb.ravel(), w, state, tp, 1.0, 1.0, gated=False)
    else:
        got = run_recurrence(ob, d, H, dk, dv, x[0], x[1], x[2], zb.ravel(), np.zeros(H * dk), w, state, tp, 3)
    at = 0
    for b, m in enumerate(counts):
        y = [a[at:at + m] for a in x]
        if keyed:
            ref = ref_gla(y, A, zb.ravel(), w, ref_state[b], 1.0, 1.0, gated=False)
        else:
            ref = ref_recurrence(y[0], y[1], y[2], zb.ravel(), np.zeros(H * dk), w, ref_state[b])
        assert rel_err(got[at:at + m], ref) < TOL
        assert rel_err(host(state[b]), ref_state[b]) < STATE
        at += m


@pytest.mark.parametrize("keyed,H,dk,dv,B", [(False, 8, 256, 128, 40), (True, 2, 64, 256, 70), (False, 3, 64, 128, 33), (True, 1, 128, 512, 1)])
def test_many_chunks(cuda, ob, keyed, H, dk, dv, B):
    # Clusters of the output kernel take several (chunk, head) pairs; a warp looks through the sequences more than once; the first case goes
    # through its heads in two passes.
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(B)
    counts = rng.integers(300, 725, B) if B > 1 else np.array([8000])
    T, ends = int(counts.sum()), np.cumsum(counts)
    x = [rounded(rng.standard_normal(s).astype(np.float32), "bf16") for s in ((T, H, dk), (T, H, dk), (T, H, dv), (T, 4), (T, H, dv))]
    w, zb = fr.round_bf16(1 + 0.3 * rng.standard_normal(dv)), fr.round_bf16(rng.uniform(-1, 6, H * dk))
    A, lower = fr.round_bf16(rng.standard_normal((H * dk, 4)) * 0.3), np.zeros(H * dk)
    state = d.zeros(B, H, dk, dv, f32=True)
    tp = positions(ob, d, counts, [0] * B)
    if keyed:
        got = run_gla(ob, d, H, dk, dv, x, A, zb, w, state, tp, 16.0, 1.0)
    else:
        got = run_recurrence(ob, d, H, dk, dv, x[0], x[1], x[2], zb, lower, w, state, tp, B)
    for b in sorted({0, 1, 31, 32, 33, B // 2, B - 1} & set(range(B))):
        s = slice(int(ends[b] - counts[b]), int(ends[b]))
        for h in {0, H // 2, H - 1}:
            ch, ref_state = slice(h * dk, (h + 1) * dk), np.zeros((1, dk, dv))
            y = [a[s, h:h + 1] for a in x[:3]]
            if keyed:
                ref = ref_gla(y + [x[3][s], x[4][s, h:h + 1]], A[ch], zb[ch], w, ref_state, 16.0, 1.0)
            else:
                ref = ref_recurrence(*y, zb[ch], lower[ch], w, ref_state)
            assert rel_err(got[s, h:h + 1], ref) < TOL, (b, h)
            assert rel_err(host(state[b, h:h + 1]), ref_state) < STATE, (b, h)


@pytest.mark.parametrize("keyed", [False, True])
def test_state_from_operands_of_one_sign(cuda, ob, keyed):
    # where every term adds up, so do the errors that the tensor cores make when they cut sums off
    d = Dev(cuda, ob, "bf16")
    rng = np.random.default_rng(11)
    H, dk, dv, n = 2, 128, 128, 1500
    x = [rounded(np.abs(rng.standard_normal(s)) if i in (1, 2) and (keyed or i == 2) else rng.standard_normal(s), "bf16")
         for i, s in enumerate(((n, H, dk), (n, H, dk), (n, H, dv), (n, 4), (n, H, dv)))]
    A, zb, w = fr.round_bf16(rng.standard_normal((H * dk, 4)) * 0.3), fr.round_bf16(rng.uniform(2, 7, H * dk)), np.ones(dv)
    state, ref_state = d.zeros(1, H, dk, dv, f32=True), np.zeros((H, dk, dv))
    tp = positions(ob, d, [n], [0])
    if keyed:
        run_gla(ob, d, H, dk, dv, x, A, zb, w, state, tp, 4.0, 1.0)
        ref_gla(x, A, zb, w, ref_state, 4.0, 1.0)
    else:
        run_recurrence(ob, d, H, dk, dv, x[0], x[1], x[2], zb, np.zeros(H * dk), w, state, tp, 1)
        ref_recurrence(x[0], x[1], x[2], zb, np.zeros(H * dk), w, ref_state)
    assert rel_err(host(state)[0], ref_state) < STATE
