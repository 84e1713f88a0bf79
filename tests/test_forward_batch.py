"""The step's index arrays (``ForwardBatch.build``, ``attention.build_work``) against a token-by-token construction."""
import pytest
import torch

from gemm_b200.models.transformer import ForwardBatch
from gemm_b200.ops import attention


def _plain(q_lens, ctx, bt, page, all_logits):
    pos, slots, cu = [], [], [0]
    for s, n in enumerate(q_lens):
        for p in range(ctx[s], ctx[s] + n):
            pos.append(p)
            slots.append(int(bt[s, p // page]) * page + p % page)
        cu.append(cu[-1] + n)
    rows = list(range(cu[-1])) if all_logits else [cu[s + 1] - 1 for s, n in enumerate(q_lens) if n > 0]
    return pos, slots, cu, rows


def _plain_work(q_lens, hq, hkv, splits):
    tpt = 128 // (hq // hkv)
    return [[s, h, ti * tpt, sp] for s, n in enumerate(q_lens) for ti in reversed(range((n + tpt - 1) // tpt)) for sp in range(splits) for h in range(hkv)]


@pytest.mark.parametrize("q_lens,ctx", [([1], [0]), ([1, 1, 1], [0, 127, 128]), ([5, 0, 300, 1], [120, 7, 3, 255]), ([0, 0], [1, 2]), ([129, 16, 17], [0, 0, 0])])
@pytest.mark.parametrize("page,all_logits,hq,hkv,splits", [(128, False, 8, 2, 1), (16, True, 32, 4, 3), (128, False, 16, 16, 2)])
def test_build(q_lens, ctx, page, all_logits, hq, hkv, splits):
    pages = max(-(-(q + c) // page) for q, c in zip(q_lens, ctx)) + 2
    bt = torch.randperm(len(q_lens) * pages).view(len(q_lens), pages).to(torch.int32)
    ids = list(range(sum(q_lens)))
    fb = ForwardBatch.build(q_lens, ctx, ids, bt, page, hq, hkv, "cpu", num_splits=splits, all_logits=all_logits, seq_slots=[3 + i for i in range(len(q_lens))])
    pos, slots, cu, rows = _plain(q_lens, ctx, bt, page, all_logits)
    for name, want in (("positions", pos), ("slots", slots), ("cu_q", cu), ("kv_len", [a + b for a, b in zip(q_lens, ctx)]), ("ids", ids),
                       ("seq_slots", [3 + i for i in range(len(q_lens))]), ("logit_rows", rows)):
        got = getattr(fb, name)
        assert got.tolist() == want and got.dtype == (torch.int64 if name == "logit_rows" else torch.int32), name
    assert fb.work.tolist() == _plain_work(q_lens, hq, hkv, splits)
    assert fb.block_table.tolist() == bt.tolist() and fb.n_tokens == sum(q_lens) and fb.is_decode == all(q == 1 for q in q_lens)
    # the kernels read the work list 16 bytes at a time
    assert all(getattr(fb, n).storage_offset() % 4 == 0 for n in ("work", "cu_q", "kv_len", "slots"))


def test_build_refuses_tokens_past_the_block_table():
    with pytest.raises(IndexError):
        ForwardBatch.build([10], [250], list(range(10)), torch.zeros(1, 2, dtype=torch.int32), 128, 8, 2, "cpu")


def test_staged_layout():
    bt = torch.zeros(3, 4, dtype=torch.int32)
    fb = ForwardBatch.build([20, 16, 1], [0, 0, 0], list(range(37)), bt, 16, 8, 2, "cpu", stage=True)
    assert fb.stage_slots.tolist() == list(range(20)) + list(range(32, 48)) + [48]
    assert fb.stage_bt.tolist() == [[0, 1], [2, 0], [3, 0]]
    with pytest.raises(NotImplementedError):
        ForwardBatch.build([2, 1], [0, 5], [0, 1, 2], bt, 16, 8, 2, "cpu", stage=True)
    fb = ForwardBatch.build([1, 1, 1], [3, 4, 5], [0, 1, 2], bt, 16, 8, 2, "cpu", stage=True)
    assert fb.stage_slots.tolist() == [0, 1, 2] and fb.stage_bt is None


def test_build_takes_whole_numbers_only():
    bt = torch.zeros(2, 4, dtype=torch.int32)
    for q_lens, ctx in (([2.5, 1], [0, 0]), ([2, 1], [0.5, 0]), ([2.0, 1.0], [0, 0])):
        with pytest.raises(TypeError):
            ForwardBatch.build(q_lens, ctx, [1, 2, 3], bt, 16, 8, 2, "cpu")
    with pytest.raises(TypeError):
        attention.build_work([2.5], 8, 2)
    want = ForwardBatch.build([2, 1], [3, 0], [1, 2, 3], bt, 16, 8, 2, "cpu")
    got = ForwardBatch.build(torch.tensor([2, 1]), torch.tensor([3, 0]), [1, 2, 3], bt, 16, 8, 2, "cpu")
    assert got.positions.tolist() == want.positions.tolist() and got.work.tolist() == want.work.tolist()


def _wide_table():
    bt = torch.arange(12, dtype=torch.int64).view(2, 6)
    bt[:, 4:] = 2 ** 40 + 7                               # entries past the sequences' pages: whatever the memory held
    return bt


def test_build_takes_tables_with_anything_in_unused_entries():
    fb = ForwardBatch.build([20, 1], [10, 63], list(range(21)), _wide_table(), 16, 8, 2, "meta")
    assert fb.block_table.shape == (2, 6) and fb.block_table.dtype == torch.int32


@pytest.mark.gpu
def test_build_on_the_device():
    """One copy of all arrays to the GPU: the values of the CPU's batch, a table of 64-bit entries among them."""
    args = ([20, 1], [10, 63], list(range(21)), _wide_table(), 16, 8, 2)
    cpu, gpu = ForwardBatch.build(*args, "cpu", num_splits=2), ForwardBatch.build(*args, "cuda", num_splits=2)
    for name in ("ids", "positions", "slots", "cu_q", "kv_len", "work", "seq_slots", "block_table", "logit_rows"):
        a, b = getattr(cpu, name), getattr(gpu, name)
        assert b.is_cuda and b.dtype == a.dtype and torch.equal(b.cpu(), a), name
        assert b.data_ptr() % 16 == 0, name
