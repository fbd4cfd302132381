"""The kernels of the FP8 head (csrc/head_fp8.cu).  Up to 64 rows (head_fp8_decode_kernel): batch sizes around its tiles of 16, 32
and 64 rows and around the halves that a tile is split into, vocabularies whose last tile is cut and that take a CTA several
tiles, stages of one, two and four K blocks; with the row records, against the product in 64 bits."""
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


def unorder(o):
    o = np.asarray(o, np.uint32)
    return np.where(o >> 31, o ^ np.uint32(0x80000000), ~o).view(np.float32)


@pytest.mark.parametrize("N,K", [(129, 128), (1000, 512), (20011, 384), (40000, 256), (300, 16384)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 63, 64, 65])
def test_product_and_records(pkg, M, N, K):
    check_product_and_records(pkg, M, N, K)


@pytest.mark.parametrize("N,K", [(100, 128), (257, 512), (20011, 384), (40000, 256), (300, 16384)])
@pytest.mark.parametrize("M", [127, 128, 129, 256, 257, 350, 385, 700])
def test_larger_batches(pkg, M, N, K):
    """Around one CTA's 128 rows and a pair's 256 (head_fp8_kernel, head_fp8_pair_kernel): a second half with one row and with all, several
    batch tiles, rows behind the whole pair tiles in a launch of their own (257 and 350), vocabularies shorter than a tile, fewer K blocks
    than stages."""
    check_product_and_records(pkg, M, N, K)


def check_product_and_records(pkg, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    blocks, kb = (N + 127) // 128, K // 128
    w = (100 * torch.randn(N, K, device="cuda", generator=g)).clamp(-448, 448).to(torch.float8_e4m3fn)
    scale = 1e-4 * (0.5 + torch.rand(blocks, kb, device="cuda", generator=g))
    a, a_scale = pkg.quantize_activations(x)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((M, N + 3), 7.0, device="cuda")          # rows of odd length: the stores have no alignment to rely on
    records = torch.empty(M, 16, dtype=torch.uint8, device="cuda")
    got = pkg.head_fp8(a, a_scale, w.view(torch.uint8), scale, out[:, :N], flag, row_extremes=records)
    plain = pkg.head_fp8(a, a_scale, w.view(torch.uint8), scale, error_flag=flag)
    assert flag.item() == 0 and torch.equal(got, plain) and (out[:, N:] == 7.0).all()
    wide = w.double() * scale.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    left = a.view(torch.float8_e4m3fn).double() * a_scale.double().repeat_interleave(128, 1)
    want = left @ wide.T
    # a K block's 128 products are added in about fp32, the blocks one by one: (128 + K / 128 + 2) units of the sum of magnitudes
    bound = (130 + kb) * 2.0 ** -23 * (left.abs() @ wide.abs().T)
    assert ((got.double() - want).abs() <= bound).all()
    # and, since the errors of the additions hardly line up, within the tolerance that the head is documented with
    assert (got.double() - want).abs().max() <= 2e-5 * want.abs().max() + 1e-6
    rec, logits = records.cpu().numpy().view(np.uint64), got.cpu().numpy()
    key = rec[:, 0]
    assert (unorder(key >> np.uint64(32)) == logits.max(axis=1)).all()
    assert ((np.uint64(0xffffffff) - (key & np.uint64(0xffffffff))).astype(np.int64) == logits.argmax(axis=1)).all()
    assert (unorder(~(rec[:, 1] & np.uint64(0xffffffff)).astype(np.uint32)) == logits.min(axis=1)).all()
    assert ((rec[:, 1] >> np.uint64(32)) == 0).all()


@pytest.mark.parametrize("M", [5, 40])
def test_records_of_rows_that_are_not_finite(pkg, M):
    """An activation row whose scale is infinite: its logits are NaN or infinite, the other rows stay as they are."""
    N, K = 3000, 512
    g = torch.Generator(device="cuda").manual_seed(M)
    a, a_scale = pkg.quantize_activations(torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16))
    w = (100 * torch.randn(N, K, device="cuda", generator=g)).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
    scale = torch.full(((N + 127) // 128, K // 128), 1e-4, device="cuda")
    want = pkg.head_fp8(a, a_scale, w, scale)
    a_scale[M - 2, 1] = float("inf")
    records = torch.empty(M, 16, dtype=torch.uint8, device="cuda")
    got = pkg.head_fp8(a, a_scale, w, scale, row_extremes=records)
    others = [r for r in range(M) if r != M - 2]
    assert torch.equal(got[others], want[others]) and not torch.isfinite(got[M - 2]).any()
    flags = (records.cpu().numpy().view(np.uint64)[:, 1] >> np.uint64(32)).astype(int)
    assert flags[M - 2] == 1 and flags.sum() == 1
