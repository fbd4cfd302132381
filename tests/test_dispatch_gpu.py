"""The sizes at which a sampling or verification call changes its path (csrc/sampler.cu, csrc/verify.cu): the last batch of the
cluster kernel and the first of the grid-wide passes, rows at odd addresses, vocabularies around the cluster sizes.  Tokens
and records against the CPU oracle."""
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


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def u64(a):
    return cu(np.asarray(a, np.uint64).view(np.int64))


@pytest.mark.parametrize("rows,vocab,lead", [(12, 129280, 0), (13, 129280, 0), (48, 50001, 1), (49, 50001, 1), (49, 16385, 2),
                                             (50, 16383, 3), (5, 32769, 0), (5, 131072, 0), (3, 1025, 1)])
@pytest.mark.parametrize("t,top,top_k", [(0.7, 0.95, 0), (1.0, 1.0, 0), (0.8, 0.9, 40), (0.0, 1.0, 0)])
def test_sampling(pkg, oracle, rows, vocab, lead, t, top, top_k):
    x = oracle.gen_logits(7 + vocab, rows, vocab)
    x[1] = oracle.gen_normal(8, vocab, (1, vocab), 1.28)[0]      # a flat row: a nucleus of thousands
    x[2, : vocab // 2] = x[2].max()                               # half of the row tied at the top
    buf = torch.zeros(rows, vocab + 5, device="cuda")
    view = buf[:, lead: lead + vocab]
    view.copy_(torch.from_numpy(x))
    seeds, steps = np.arange(rows) * 31 + 5, np.arange(rows) * 3 + 1
    want, _ = oracle.sample_rows(x, t, top, seeds, steps, top_k=top_k, slot=1, purpose=0, threads=8)
    tok, st = pkg.sample_logits(view, t, top, u64(seeds), u64(steps), slot=1, top_k=top_k)
    torch.cuda.synchronize()
    assert (st.cpu().numpy() >= 0).all() and (tok.cpu().numpy() == want).all()


@pytest.mark.parametrize("seqs,drafts,vocab", [(8, 2, 50001), (9, 2, 50001), (41, 0, 16384), (4, 5, 129280), (1, 1, 1025)])
@pytest.mark.parametrize("t,top,sigma", [(0.7, 0.95, 0.6), (1.0, 1.0, 1.0)])
def test_verification(pkg, oracle, seqs, drafts, vocab, t, top, sigma):
    target = oracle.gen_logits(11 + vocab, seqs * (drafts + 1), vocab)
    target[0] = oracle.gen_normal(9, vocab, (1, vocab), 1.28)[0]  # flat: the residual spreads over the whole row
    draft = oracle.gen_perturbed(12, target.reshape(seqs, drafts + 1, vocab)[:, :drafts].reshape(-1, vocab), sigma)
    seeds, steps = np.arange(seqs, dtype=np.uint64) + 3, np.arange(seqs, dtype=np.uint64) * 5 + 2
    ids = np.zeros((seqs, drafts), np.int32)
    for k in range(drafts):
        ids[:, k], _ = oracle.sample_rows(draft[k::drafts], t, top, seeds, steps, slot=k, purpose=1, threads=8)
    want, _ = oracle.verify_rows(target, draft, ids.reshape(-1), drafts, t, top, seeds, steps, threads=8)
    res, st = pkg.verify_logits(cu(target), cu(draft) if drafts else None, cu(ids.reshape(-1)) if drafts else None, drafts, t,
                                top, u64(seeds), u64(steps))
    torch.cuda.synchronize()
    got = pkg.results_to_numpy(res)
    assert (st.cpu().numpy() == 0).all()
    assert all((got[f] == want[f]).all() for f in ("tokens", "emitted", "accepted_drafts", "rejected")), (got, want)
