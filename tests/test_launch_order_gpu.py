"""Every call reads what the work in front of it on the stream has written, weights included.  The kernels are launched before the
one in front has finished, and the quantiser, the final norm and the Markov bias let their successor start before they have
written anything: here they write the weights of the head that follows, behind a long wait so that both calls are queued."""
import pytest
import torch

import __graft_entry__ as entry

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    entry.build()
    return entry.load_package()


def rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, device="cuda", generator=g) * scale


def check(write, head, weights):
    """`head()` right behind `write()`, against the same call once the weights are at rest."""
    weights.zero_()
    torch.cuda.synchronize()
    for _ in range(3):
        torch.cuda._sleep(400_000)
        write()
        got = head()
        torch.cuda.synchronize()
        want = head()
        torch.cuda.synchronize()
        assert bool(torch.isfinite(want).all()) and bool((want != 0).any())
        assert torch.equal(got, want)
        weights.zero_()
        torch.cuda.synchronize()


@pytest.mark.parametrize("N,K", [(128, 4096), (256, 1024), (2048, 4096), (18944, 4096), (4000, 512)])
@pytest.mark.parametrize("M,records", [(1, False), (5, True), (64, True), (130, False)])
def test_fp8_weights_of_the_quantiser(pkg, N, K, M, records):
    a, a_scale = pkg.quantize_activations(rand((M, K), 1).to(torch.bfloat16))
    source = rand((N, K), 2).to(torch.bfloat16)
    w = torch.zeros((N, K), dtype=torch.uint8, device="cuda")
    spare = torch.empty((N, K // 128), device="cuda")
    ws = torch.full(((N + 127) // 128, K // 128), 0.01, device="cuda")
    ext = torch.empty((M, 16), dtype=torch.uint8, device="cuda") if records else None
    check(lambda: pkg.quantize_activations(source, w, spare), lambda: pkg.head_fp8(a, a_scale, w, ws, row_extremes=ext), w)


def as_bf16(w):
    return w.view(torch.bfloat16)


# inputs far below the quantiser's least scale: its codes stay small, so that two of them are a finite BF16
@pytest.mark.parametrize("N,K", [(16, 256), (100, 512), (2050, 5120), (9000, 1024)])
@pytest.mark.parametrize("M", [1, 2, 4, 6])
def test_bf16_weights_of_the_quantiser(pkg, N, K, M):
    source = rand((N, 2 * K), 3, 1e-6).to(torch.bfloat16)
    w = torch.zeros((N, 2 * K), dtype=torch.uint8, device="cuda")
    spare = torch.empty((N, 2 * K // 128), device="cuda")
    x = rand((M, K), 4)
    write = lambda: pkg.quantize_activations(source, w, spare)
    check(write, lambda: pkg.head_bf16(x, as_bf16(w)), w)
    check(write, lambda: pkg.head_compact(x, as_bf16(w)), w)


@pytest.mark.parametrize("vocab", [1, 33, 5000, 129280])
def test_markov_weights_of_the_quantiser(pkg, vocab):
    source = rand((vocab, 512), 5, 1e-6).to(torch.bfloat16)
    w = torch.zeros((vocab, 512), dtype=torch.uint8, device="cuda")
    spare = torch.empty((vocab, 4), device="cuda")
    u, e = rand((vocab,), 6), rand((256,), 7).to(torch.bfloat16)
    check(lambda: pkg.quantize_activations(source, w, spare), lambda: pkg.markov_logits(u, as_bf16(w), e), w)


@pytest.mark.parametrize("K", [128, 5120])
@pytest.mark.parametrize("M", [1, 3, 7])
def test_f32_weights_of_the_final_norm(pkg, M, K):
    h, pre, g = rand((8, 4, K), 8).to(torch.bfloat16), rand((8, 4), 9), rand((K,), 10).to(torch.bfloat16)
    w, x = torch.zeros((8, K), device="cuda"), rand((M, K), 11)
    check(lambda: pkg.final_norm(h, pre, g, out=w), lambda: pkg.head_f32(x, w), w)
