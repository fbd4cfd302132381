"""The batch path's front in one launch (csrc/flat.cu, flat_front_kernel): the smallest and largest batches that take it, slices that end
anywhere, rows at odd addresses, flat, peaked, tied and unusable rows, with and without the head's records; tokens against the CPU
oracle.  And the first batches of the passes behind its lines."""
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


def ordered(v):
    b = np.where(v == 0, np.float32(0), v).astype(np.float32).view(np.uint32)
    return b ^ np.where(b >> 31, np.uint32(0xffffffff), np.uint32(0x80000000)).astype(np.uint32)


def records(x):
    """What the head leaves of each row (include/ds41_b200.h): first maximum, minimum, whether a logit is not finite."""
    out = np.zeros((x.shape[0], 2), np.uint64)
    for r, row in enumerate(x):
        usable = row[np.isfinite(row)]
        top = int(np.flatnonzero(row == usable.max())[0])
        out[r, 0] = (np.uint64(ordered(usable.max()[None])[0]) << np.uint64(32)) | np.uint64(0xffffffff - top)
        out[r, 1] = np.uint64(~ordered(usable.min()[None])[0]) | np.uint64(0 if np.isfinite(row).all() else 1) << np.uint64(32)
    return torch.from_numpy(out.view(np.uint8).reshape(-1, 16)).cuda()


@pytest.mark.parametrize("rows,vocab,lead", [(33, 32769, 0), (34, 33003, 1), (33, 131072, 0), (33, 129280, 2), (100, 33001, 3), (101, 33001, 0),
                                             (130, 40000, 0), (131, 40000, 0),
                                             (127, 40000, 0), (128, 40000, 0)])
@pytest.mark.parametrize("known", [False, True])
def test_front(pkg, oracle, rows, vocab, lead, known):
    x = oracle.gen_logits(3 + vocab, rows, vocab)
    x[1] = oracle.gen_normal(8, vocab, (1, vocab), 1.28)[0]       # flat: a nucleus of thousands
    x[2, : vocab // 2] = x[2].max()                               # half of the row tied at the top: a bin's count overflows
    x[3, ::7] = x[3, 5]                                           # plateaus
    x[4] = 1.5                                                    # no range at all
    x[5, vocab - 1] = x[5].max() + 3                              # the maximum is the last id
    x[6, 11] = np.nan
    buf = torch.zeros(rows, vocab + 5, device="cuda")
    view = buf[:, lead: lead + vocab]
    view.copy_(torch.from_numpy(x))
    seeds, steps = np.arange(rows) * 31 + 5, np.arange(rows) * 3 + 1
    ok = [r for r in range(rows) if r != 6]
    want, _ = oracle.sample_rows(x[ok], 0.7, 0.95, seeds[ok], steps[ok], threads=8)
    scratch = torch.full((pkg.sample_scratch_bytes(rows, vocab),), 0x5a, dtype=torch.uint8, device="cuda")   # nothing relies on zeros
    for _ in range(2):
        tok, st = pkg.sample_logits(view, 0.7, 0.95, u64(seeds), u64(steps), scratch=scratch, row_extremes=records(x) if known else None)
        torch.cuda.synchronize()
        tok, st = tok.cpu().numpy(), st.cpu().numpy()
        assert (tok[ok] == want).all() and (st[ok] == 0).all() and tok[6] == -1 and st[6] == -1
