"""Rows whose cluster lets its CTAs go before the row's end, because further rows wait for a place (csrc/row_fast.cuh): at the
number of clusters that run at a time and just above it (32 of eight CTAs, 148 of two, 296 of one), rows cut by top-k and rows whose
mask leaves few ids, mixed with rows that another path finishes, and in the persistent grid that takes what the streaming path
leaves over.  Tokens against the CPU oracle."""
import numpy as np
import pytest
import torch

import __graft_entry__ as entry

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    entry.build()
    return entry.load_package()


def u64(a):
    return torch.from_numpy(np.asarray(a, np.uint64).view(np.int64)).cuda()


@pytest.mark.parametrize("rows,vocab,top_k", [(37, 33001, 40), (38, 33001, 40), (80, 40000, 7), (149, 20000, 20), (297, 9000, 20),
                                              (300, 40000, 40), (32, 33001, 40), (33, 33001, 40), (34, 33001, 40), (148, 20000, 20),
                                              (296, 9000, 20), (300, 900, 0)])
def test_top_k_rows_that_wait_for_a_place(pkg, oracle, rows, vocab, top_k):
    x = oracle.gen_logits(5 + vocab, rows, vocab)
    x[::3, 100:400] = x[::3].max(axis=1, keepdims=True)          # more ties at the top than the streaming path keeps
    x[1, : vocab // 2] = x[1].max()                              # more than the list of the fast path holds: the general search
    seeds, steps = np.arange(rows) * 31 + 5, np.arange(rows) * 3 + 1
    want, _ = oracle.sample_rows(x, 0.8, 0.9, seeds, steps, top_k=top_k, threads=8)
    for _ in range(3):
        tok, st = pkg.sample_logits(torch.from_numpy(x).cuda(), 0.8, 0.9, u64(seeds), u64(steps), top_k=top_k)
        torch.cuda.synchronize()
        assert (st.cpu().numpy() >= 0).all() and (tok.cpu().numpy() == want).all()


@pytest.mark.parametrize("rows,vocab,allowed", [(33, 33001, 900), (40, 129280, 1024), (149, 20000, 300), (297, 9000, 50)])
def test_masked_rows_that_wait_for_a_place(pkg, oracle, rows, vocab, allowed):
    """No top-k, but few ids in the mask; every fifth row has all ids in it and takes another path."""
    x = oracle.gen_logits(6 + vocab, rows, vocab)
    rng = np.random.default_rng(rows)
    open_ = np.zeros((rows, (vocab + 31) // 32 * 32), bool)
    for r in range(rows):
        open_[r, rng.choice(vocab, allowed, replace=False)] = True
        if r % 5 == 4:
            open_[r, :vocab] = True
    mask = np.packbits(open_, axis=1, bitorder="little").view(np.uint32)
    seeds, steps = np.arange(rows) * 13 + 1, np.arange(rows) * 7 + 2
    want, _ = oracle.sample_rows(x, 0.8, 0.9, seeds, steps, mask=mask, threads=8)
    words = torch.from_numpy(mask.view(np.int32)).cuda()
    for _ in range(3):
        tok, st = pkg.sample_logits(torch.from_numpy(x).cuda(), 0.8, 0.9, u64(seeds), u64(steps), mask=words)
        torch.cuda.synchronize()
        assert (st.cpu().numpy() >= 0).all() and (tok.cpu().numpy() == want).all()
