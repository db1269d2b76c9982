"""The residual sum of a parallel block with the next block's layer norm in the same kernel, at the edges of what one block of threads holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(x, want):
    return float((x.double() - want).norm() / want.norm())


@pytest.mark.parametrize("d", [4, 30, 2044, 2048, 2052, 8192, 8196])
@pytest.mark.parametrize("depth", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
def test_gated_sum_norm(d, depth, shift):
    """Widths and column offsets that the one kernel takes, and those that go through two. Float32 sums of d values: 3e-6; a 16-bit
    norm is rounded once: 2^-8."""
    from llmplayer_b200.kernels import ops
    T = 3
    g = torch.Generator(device=DEV).manual_seed(d + 2 * depth + shift)
    r = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
    x, a, b, wide, ba, gain = r(T, d) + 3.0, r(T, d), r(T, d), r(T, 2 * d + 4), r(d), r(d)
    logits_a, logits_b = wide[:, shift:shift + d], wide[:, d + 2 * shift:2 * d + 2 * shift]
    streams, mix = r(4, T, d), r(3)
    y = x.double() + a.double() * torch.sigmoid(logits_a.double() + ba.double()) + b.double() * torch.sigmoid(logits_b.double())
    want = mix[0].double() * streams[0].double() + mix[1].double() * x.double() + mix[2].double() * y if depth else y
    c = want - want.mean(-1, keepdim=True)
    norm = c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-5) * gain.double()
    for dtype, limit in ((torch.float32, 3e-6), (torch.bfloat16, 2.0 ** -8)):
        got, out, kept = x.clone(), torch.full((T, d), float("nan"), dtype=dtype, device=DEV), streams.clone()
        extra = dict(streams=kept, mix=mix, count=3, keep_input=True) if depth else {}
        ops.gated_sum(got, a, (logits_a, ba), b, (logits_b, None), norm_after=(gain, 1e-5, out), **extra)
        assert rel(got, want) < 3e-6
        assert rel(out, norm) < limit
        if depth:
            assert torch.equal(kept[1], x) and torch.equal(kept[3], streams[3]) and rel(kept[2], y) < 3e-6
