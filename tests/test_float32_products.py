"""float32 products on the tensor cores, as three bfloat16 parts, over what float32 holds: operands and results down to the smallest numbers,
exact sums, mantissas that lose most when cut off, sums of one sign. The other side is the chain of multiply-adds that serves addresses of
no 16 bytes, or float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
UNIT = 2.0 ** -24
ROWS = [1, 3, 8, 12, 40, 200]          # the forms for a few rows, the tiles of 64 and of 128


def product(a, w):
    from llmplayer_b200.kernels import ops
    out = torch.full((a.shape[0], w.shape[0]), 7.0, device=DEV)
    ops.gemm_plain(a, w, out)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    return out


def by_multiply_adds(a, w):
    shifted = torch.empty(a.numel() + 1, device=DEV)[1:].view(a.shape)
    shifted.copy_(a)
    return product(shifted, w)


def draw(kind, g, *shape):
    normal = torch.randn(*shape, generator=g, device=DEV)
    if kind == "one sign":
        return torch.rand(*shape, generator=g, device=DEV) + 1
    if kind == "worst mantissas":       # parts of ones only: 1.ffff in all three
        mantissa = torch.full(shape, 0x3f80ffff, dtype=torch.int32, device=DEV).view(torch.float32)
        return mantissa * torch.exp2(torch.randint(0, 2, shape, generator=g, device=DEV).float())
    return normal * torch.exp(2 * torch.randn(*shape, generator=g, device=DEV)) if kind == "many sizes" else normal


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("K", [32, 36, 64, 260, 1024, 2048])
@pytest.mark.parametrize("kind", ["normal", "one sign", "worst mantissas", "many sizes"])
def test_no_further_from_64_bits_than_multiply_adds(kind, K, M):
    g = torch.Generator(device=DEV).manual_seed(K + M)
    a, w = draw(kind, g, M, K), draw(kind, g, 300, K)
    want = a.double() @ w.double().T
    size = a.double().abs() @ w.double().abs().T
    off = [((out.double() - want) / size).square().mean().sqrt() / UNIT for out in (product(a, w), by_multiply_adds(a, w))]
    assert float(off[0]) <= float(off[1])


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("K", [32, 64, 260, 2048])
def test_exact_sums_stay_exact(K, M):
    """Whole numbers whose sums float32 holds (2^11 terms of up to 60 x 60), and rows of one 1 that pick any values out."""
    g = torch.Generator(device=DEV).manual_seed(K + M)
    a = torch.randint(-60, 61, (M, K), generator=g, device=DEV).float()
    w = torch.randint(-60, 61, (70, K), generator=g, device=DEV).float()
    assert torch.equal(product(a, w).double(), a.double() @ w.double().T)
    values = draw("many sizes", g, M, K)
    picked = torch.randint(0, K, (70,), generator=g, device=DEV)
    one = torch.zeros(70, K, device=DEV)
    one[torch.arange(70, device=DEV), picked] = 1.0
    assert torch.equal(product(values, one), values[:, picked])
    weights = draw("many sizes", g, 70, K)
    one, picked = torch.zeros(M, K, device=DEV), torch.randint(0, K, (M,), generator=g, device=DEV)
    one[torch.arange(M, device=DEV), picked] = 1.0
    assert torch.equal(product(one, weights), weights[:, picked].T)


@pytest.mark.parametrize("M", ROWS)
def test_a_product_that_stands_alone(M):
    """What is left out is at most 2^-8 2^-15 + 2^-17 2^-7 of the product (tokens rounded, weights cut off), 3 units; the token's third part is cut off
    at 2^-25 and has half a unit added to it; the sum is cut off at a last bit, 2 units: 6 and what the small sums lose, below 1/4."""
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = torch.zeros(M, 64, device=DEV), torch.zeros(3000, 64, device=DEV)
    a[:, 5], w[:, 5] = draw("one sign", g, M), draw("one sign", g, 3000)
    a[0, 5], w[0, 5] = draw("worst mantissas", g, 1)[0], draw("worst mantissas", g, 1)[0]
    want = a.double() @ w.double().T
    assert float(((product(a, w).double() - want) / want).abs().max()) <= 6.25 * UNIT


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("of_a,of_w", [(-60, -60), (-118, 60), (60, -118), (-126, 90), (90, -126), (-133, 0), (0, -133), (-141, 100), (60, 30), (110, -20),
                                       (-20, 110)])
def test_the_ends_of_the_range(of_a, of_w, M):
    """Operands of 2^of_a and 2^of_w: small results, operands whose third part bfloat16 has no room for, numbers below the normal ones, sums
    and operands that the scaled parts have no room for. Bound: 11 units of the sum of magnitudes (6.25 of a product that stands alone, 4.75 for
    the two cuts and the additions of eight sums behind it) and half a last bit of the smallest numbers."""
    g = torch.Generator(device=DEV).manual_seed(M + of_a)
    a, w = torch.randn(M, 256, generator=g, device=DEV), torch.randn(90, 256, generator=g, device=DEV)
    a, w = a * 2.0 ** (of_a // 2) * 2.0 ** (of_a - of_a // 2), w * 2.0 ** (of_w // 2) * 2.0 ** (of_w - of_w // 2)
    assert bool((a != 0).any()) and bool((w != 0).any())
    want = a.double() @ w.double().T
    bound = 11 * UNIT * (a.double().abs() @ w.double().abs().T) + 2.0 ** -150
    assert bool(((product(a, w).double() - want).abs() <= bound).all())


@pytest.mark.parametrize("mode", ["store", "accumulate", "swiglu"])
@pytest.mark.parametrize("N,K,M", [(7, 32, 1), (7, 64, 1), (40, 8192, 2), (40, 8192, 5), (2391, 100, 1), (2391, 512, 3), (5000, 2048, 4), (2391, 2048, 8), (2391, 4096, 8)])
def test_a_few_rows_in_every_form(N, K, M, mode):
    """A tile of features per SM or fewer, several for each of two groups of warps, the short ring beside many tokens, tokens that fit no
    shared memory; chains of odd numbers of blocks, ragged last tiles: the bits of the same rows in a tile of 64."""
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(N + K + M)
    code = {"store": ops.STORE, "accumulate": ops.ACCUMULATE, "swiglu": ops.SWIGLU}[mode]
    a = torch.randn(17, K, generator=g, device=DEV)
    w = torch.randn(N * (2 if mode == "swiglu" else 1), K, generator=g, device=DEV)
    first = torch.randn(17, N, generator=g, device=DEV)
    whole, out = first.clone(), torch.cat([first[:M], torch.full((1, N), 7.0, device=DEV)])
    ops.gemm_plain(a, w, whole, code)
    ops.gemm_plain(a[:M].contiguous(), w, out[:M], code)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    assert torch.equal(out[:M], whole[:M]) and bool((out[M] == 7.0).all())
