"""The streaming heads over several rounds of their persistent grids (rows enough for a second and third group per warp, a last
group that is not full), and the compact head where the activations leave no room for a ring (csrc/head_f32.cu,
csrc/head_bf16.cu, csrc/draft_head.cu)."""
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


def operands(M, N, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    return (torch.randn(M, K, device="cuda", generator=g),
            (0.05 * torch.randn(N, K, device="cuda", generator=g)).to(dtype))


def bits(w):
    return w.view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("M,N,K", [(1, 20011, 128), (2, 20011, 384), (6, 28417, 128), (7, 20011, 256)])
def test_f32(pkg, M, N, K):
    x, w = operands(M, N, K, torch.float32)
    got = pkg.head_f32(x, w).double()
    bound = (K / 32 + 6) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)
    assert ((got - x.double() @ w.double().T).abs() <= bound).all()


@pytest.mark.parametrize("M,N,K", [(4, 28417, 256), (5, 28417, 512), (7, 20011, 256), (8, 300, 7168)])
def test_compact(pkg, oracle, M, N, K):
    x, w = operands(M, N, K, torch.bfloat16)
    assert np.array_equal(pkg.head_compact(x, w).cpu().numpy(), oracle.head_compact(x.cpu().numpy(), bits(w)))


@pytest.mark.parametrize("M,N,K", [(3, 70001, 256), (4, 70001, 256)])
def test_bf16(pkg, M, N, K):
    x, w = operands(M, N, K, torch.bfloat16)
    whole, parts = pkg.head_bf16(x, w), [pkg.head_bf16(x, w[i:i + 9001].contiguous()) for i in range(0, N, 9001)]
    assert torch.equal(whole, torch.cat(parts, 1))     # (a single round each, which the oracle is compared with elsewhere)
