"""The sizes at which a sampling or verification call changes its path (csrc/sampler.cu, csrc/verify.cu): the last batch of the
cluster kernel and the first of the grid-wide passes, rows at odd addresses, vocabularies around the cluster sizes.  Tokens
and records against the CPU oracle; likewise the operators on probability rows (csrc/prob.cu).  Which side a size takes is
seen in the kernels that its call launches."""
import numpy as np
import pytest
import torch

import __graft_entry__ as entry
from captured import kernels_of

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
                                             (50, 16383, 3), (5, 32769, 0), (5, 131072, 0), (3, 1025, 1),
                                             (32, 50001, 1), (33, 50001, 1), (256, 16385, 2), (257, 16385, 2),
                                             (257, 16384, 0), (257, 32768, 0)])
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


@pytest.mark.parametrize("rows,vocab,lead", [(49, 1000, 0), (300, 4000, 1), (64, 1024, 0)])
def test_uncertified_rows_of_the_streaming_path_are_redone(pkg, oracle, rows, vocab, lead):
    """Four ids share most of the mass and top-p lies 1e-9 from the sum of the first two, closer than the chunks' sums can tell: the row is
    redone in the reference's order and certified."""
    x = np.repeat((-9.0 - np.arange(vocab) / 1024).astype(np.float32)[None], rows, 0)
    for r in range(rows):
        x[r, (np.arange(4) * 31 + r) % vocab] = 0.0
    p = np.sort(oracle.probabilities(x[0], 1.0, 1.0))[::-1]
    assert abs(p[0] - p[3]) < 1e-15 and 0.2 < p[0] < 0.25
    seeds, steps = np.arange(rows) * 31 + 5, np.arange(rows) * 3 + 1
    buf = torch.zeros(rows, vocab + 5, device="cuda")
    view = buf[:, lead: lead + vocab]
    view.copy_(torch.from_numpy(x))
    for top in (2 * p[0] * (1 - 1e-9), 2 * p[0] * (1 + 1e-9)):
        want, _ = oracle.sample_rows(x, 1.0, top, seeds, steps, threads=8)
        tok, st = pkg.sample_logits(view, 1.0, top, u64(seeds), u64(steps))
        torch.cuda.synchronize()
        assert (st.cpu().numpy() == 0).all() and (tok.cpu().numpy() == want).all()


@pytest.mark.parametrize("seqs,drafts,vocab", [(6, 2, 50001), (3, 5, 33001), (7, 2, 33001), (8, 2, 50001), (9, 2, 50001), (41, 0, 16384), (4, 5, 129280), (1, 1, 1025),
                                               (160, 0, 16384), (161, 0, 16384), (32, 4, 24000), (54, 1, 32768)])
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


@pytest.mark.parametrize("rows,vocab,top_k,kernels", [(32, 50001, 0, 2), (33, 50001, 0, 5), (127, 50001, 0, 5), (128, 50001, 0, 7),
                                                       (256, 32768, 0, 2), (257, 32768, 0, 7), (202, 50001, 40, 1), (203, 50001, 40, 3),
                                                       (59, 50001, 5, 1), (60, 50001, 5, 3),
                                                       (256, 32768, 40, 1), (257, 32768, 40, 3),
                                                       (48, 1024, 0, 2), (49, 1024, 0, 4), (49, 129, 0, 4), (256, 128, 0, 2), (256, 1025, 0, 2)])
def test_launches_of_a_sampling(pkg, rows, vocab, top_k, kernels):
    """Top-p: the cluster kernel and the replay; or the batch path's front (one launch or three), masses and resolve before them.
    Top-k, and top-p with few ids (and the replay): the cluster kernel, or the streaming path's two before it."""
    x = torch.randn(rows, vocab, device="cuda")
    z = torch.zeros(rows, dtype=torch.int64, device="cuda")
    scratch = torch.empty(pkg.sample_scratch_bytes(rows, vocab), dtype=torch.uint8, device="cuda")
    call = dict(top_k=top_k, scratch=scratch, tokens=torch.empty(rows, dtype=torch.int32, device="cuda"),
                status=torch.empty(rows, dtype=torch.int32, device="cuda"))
    pkg.sample_logits(x, 0.7, 0.95, z, z, **call)
    assert kernels_of(lambda: pkg.sample_logits(x, 0.7, 0.95, z, z, **call)) == kernels


@pytest.mark.parametrize("seqs,drafts,vocab,kernels", [(6, 2, 33001, 3), (32, 0, 33001, 3), (3, 5, 33001, 6), (8, 2, 33001, 6), (9, 2, 33001, 6),
                                                       (32, 2, 32768, 3), (160, 0, 16384, 3), (161, 0, 16384, 8)])
def test_launches_of_a_verification(pkg, seqs, drafts, vocab, kernels):
    """Statistics by one launch of the cluster kernel, or by three of the batch path in front of it; verification; replay."""
    rows = seqs * (drafts + 1)
    target, draft = torch.randn(rows, vocab, device="cuda"), torch.randn(max(1, seqs * drafts), vocab, device="cuda")
    ids = torch.zeros(max(1, seqs * drafts), dtype=torch.int32, device="cuda")
    z = torch.zeros(seqs, dtype=torch.int64, device="cuda")
    scratch = torch.empty(pkg.verify_scratch_bytes(seqs, drafts, vocab), dtype=torch.uint8, device="cuda")
    out, st = pkg.verify_logits(target, draft if drafts else None, ids if drafts else None, drafts, 0.7, 0.95, z, z, scratch=scratch)
    assert kernels_of(lambda: pkg.verify_logits(target, draft if drafts else None, ids if drafts else None, drafts, 0.7, 0.95, z, z,
                                                scratch=scratch, results=out, status=st)) == kernels


@pytest.mark.parametrize("rows,vocab", [(34, 700), (3, 16384), (3, 16385), (3, 32769), (3, 131072), (2, 1)])
@pytest.mark.parametrize("t,top", [(0.7, 0.95), (1.0, 1.0)])
def test_probability_rows(pkg, oracle, rows, vocab, t, top):
    x = oracle.gen_logits(17 + vocab, rows, vocab)
    x[1] = oracle.gen_normal(18, vocab, (1, vocab), 1.28)[0]
    if rows > 2:
        x[2, : (vocab + 1) // 2] = x[2].max()                     # thousands tied at the cut: the order is sorted as a whole
    got, st = pkg.probabilities(cu(x), t, top)
    got = got.cpu().numpy()
    assert (st.cpu().numpy() == 0).all()
    for r in range(rows):
        want = oracle.probabilities(x[r], t, top)
        assert np.array_equal(got[r] > 0, want > 0), (r, int((got[r] > 0).sum()), int((want > 0).sum()))
        assert (np.abs(got[r] - want) <= 8 * 2.0 ** -52 * want).all()


@pytest.mark.parametrize("vocab", [129280, 16385, 700])
def test_verified_rows_and_their_faults(pkg, oracle, vocab):
    """Every transaction has its own fault; the status and, without one, the record are the reference's."""
    cases, drafts = 9, 3
    target = oracle.gen_logits(27, cases * (drafts + 1), vocab)
    draft = oracle.gen_perturbed(27, target.reshape(cases, drafts + 1, vocab)[:, :drafts].reshape(-1, vocab), 0.2)
    p = np.stack([oracle.probabilities(r, 0.7, 0.95) for r in target]).reshape(cases, drafts + 1, vocab)
    q = np.stack([oracle.probabilities(r, 0.7, 0.95) for r in draft]).reshape(cases, drafts, vocab)
    seeds, steps = np.arange(cases) + 5, np.arange(cases) + 70
    ids = np.array([[oracle.sample(q[s, k], int(seeds[s]), int(steps[s]), k, 1) for k in range(drafts)] for s in range(cases)],
                   np.int32)
    p[1, drafts] *= 1.001                       # the last target row counts although it may not be reached
    p[2, 0, 3] = np.nan
    q[3, 0, 5] = -1e-3
    ids[4, 0] = vocab
    q[5, 0, ids[5, 0]] = 0.0                     # not normalised either: that comes first
    p[6, 1] *= 1.0 + 1.00005e-8 / p[6, 1].sum()  # too close to the limit for the parallel sums
    q[7, drafts - 1, 0] = np.inf                 # counts only if that position is reached
    p[8, 0, :] = 0.0                            # rejected or accepted, from a row with one entry
    p[8, 0, 1] = 1.0
    res, st = pkg.verify_probabilities(cu(ids.reshape(-1)), cu(q.reshape(-1, vocab)), cu(p.reshape(-1, vocab)), drafts,
                                       u64(seeds), u64(steps))
    got, st = pkg.results_to_numpy(res), st.cpu().numpy()
    for s in range(cases):
        try:
            want = oracle.verify(ids[s], q[s], p[s], False, int(seeds[s]), int(steps[s]))
        except ValueError:
            assert st[s] < 0 and got["emitted"][s] == -1, s
            continue
        assert st[s] == 0 and got["emitted"][s] == want.emitted and got["rejected"][s] == want.rejected, s
        assert got["accepted_drafts"][s] == want.accepted_drafts
        assert list(got["tokens"][s][:want.emitted]) == list(want.tokens[:want.emitted]), s
    assert st[1] == -10 and st[4] < 0 and (st[[2, 3]] < 0).all()
