"""Input ids of decode steps that nobody waits for: each step has to read its own, however many are on their way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CFG = dict(num_layers=2, hidden=256, head_num=4, kv_head_num=4, head_size=64, inter_size=512, vocab_size=1000, max_seq_len=256, max_batch=8)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("batch,steps", [(1, 1), (8, 63), (3, 64), (5, 200)])
def test_steps_read_their_own_ids(ob, cuda, graphs, batch, steps):
    import torch
    m = ob.Llama(**CFG)
    m.init_random(3, 0.05)
    m.set_graphs(graphs)
    rng = np.random.default_rng(steps)
    prompt = rng.integers(0, CFG["vocab_size"], (batch, 5)).astype(np.int32)
    ids = rng.integers(0, CFG["vocab_size"], (steps, batch)).astype(np.int32)
    out = np.zeros(batch, np.int32)
    m.prefill(prompt)
    for t in range(steps):
        m.decode_step(ids[t], out)  # waits
    want = m.logits(batch)
    pinned = torch.from_numpy(ids).pin_memory()
    for how in ("pageable", "pinned"):
        m.prefill(prompt)
        got = np.zeros(batch, np.int32)
        for t in range(steps):
            last = got.ctypes.data if t == steps - 1 else 0
            if how == "pinned":
                m.decode_step_raw(pinned[t].data_ptr(), last)
            else:
                again = ids[t].copy()
                m.decode_step_raw(again.ctypes.data, last)
                again[:] = -1  # the caller's memory is free again
        # the same kernels in the same order: the same bits
        assert np.array_equal(got, out)
        assert np.array_equal(m.logits(batch), want)
    m.close()


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("behind", [0, 3])
def test_a_step_after_one_that_failed_reads_its_own_ids(ob, cuda, graphs, behind):
    # a step fails behind its layers where fewer logits than candidates are asked for; the next one is at the same position
    m = ob.Llama(**dict(CFG, vocab_size=40))
    m.init_random(3, 0.05)
    m.set_graphs(graphs)
    rng = np.random.default_rng(behind)
    prompt = rng.integers(0, 40, (2, 5)).astype(np.int32)
    ids = rng.integers(0, 40, (behind + 3, 2)).astype(np.int32)
    out = np.zeros(2, np.int32)

    def steps(fail):
        m.set_sampling(1)
        m.prefill(prompt)
        rows = []
        for t in range(len(ids)):
            if fail and t == behind:
                m.set_sampling(64)
                for _ in range(2):
                    with pytest.raises(ob.OnellmError):
                        m.decode_step((ids[t] + 1) % 40, out)
                m.set_sampling(1)
            m.decode_step(ids[t], out)
            rows.append(m.logits(2))
        return np.array(rows)

    want = steps(False)
    assert np.array_equal(steps(True), want)
    m.close()
