"""Queries, keys and values prepared four features per lane: against the kernel that takes any size (reached by moving the projection
off its 16-byte boundaries) with every combination of what a layer's heads may need."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hd,H,G,T", [(64, 3, 1, 1), (64, 5, 2, 77), (128, 4, 2, 130), (128, 1, 1, 3), (64, 2, 0, 9)])
@pytest.mark.parametrize("rd,interleaved", [(0, False), (64, False), (64, True), (32, False), (8, True), (40, False)])
@pytest.mark.parametrize("extras", ["", "bias unit", "bias gain vnorm keep", "unit first"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_against_the_general_kernel(hd, H, G, T, rd, interleaved, extras, dtype):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(hd + T + rd)
    width = (H + 2 * G) * hd
    bias = torch.randn(width, generator=g, device=DEV) if "bias" in extras else None
    gain = torch.randn(2, hd, generator=g, device=DEV) if "gain" in extras else None
    first = torch.randn(T, G * hd, generator=g, device=DEV) if "first" in extras and G else None
    share = torch.tensor([0.3], device=DEV)
    values = torch.randn(T, width, generator=g, device=DEV)
    rotation = ops.Rotation(torch.rand(rd // 2, generator=g, device=DEV), rd, interleaved) if rd else ops.NO_ROTATION
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, seq = i32([5 + t // 2 for t in range(T)]), i32([t % 2 for t in range(T)])
    pages_n = (5 + T // 2) // 64 + 1
    table = i32([[2 * i + b for i in range(pages_n)] for b in range(2)])
    angles = torch.empty(T, rd // 2, 2, device=DEV) if rd and T > 50 else None
    if angles is not None:
        ops.rope_angles(pos, rotation, angles)
    got = []
    for shift in (0, 1):
        wide = torch.zeros(T, width + 4, device=DEV)
        wide[:, shift:shift + width] = values
        q = torch.full((T, H * hd), 7.0, device=DEV, dtype=dtype)
        pages = torch.full((2 * pages_n, 2, max(G, 1), 64, hd), 7.0, device=DEV, dtype=dtype)
        kept = torch.full((T, G * hd), 7.0, device=DEV) if "keep" in extras and G else None
        ops.qkv_prepare(wide[:, shift:shift + width], bias, rotation, pos, seq, table, q, pages, num_heads=H, num_kv_heads=max(G, 1),
                        key_dim=hd, value_dim=hd, unit_norm_eps=1e-5 if "unit" in extras else None, q_gain=None if gain is None else gain[0],
                        k_gain=None if gain is None or not G else gain[1], gain_eps=1e-6, write_kv=G > 0,
                        value_norm_eps=1e-5 if "vnorm" in extras and G else None, angles=angles, keep_values=kept,
                        blend=(first, share) if first is not None else None)
        got.append([t.float() for t in (q, pages, kept) if t is not None])
    for a, b in zip(*got):
        # the sums of squares are taken in another order: a unit in the last place of float32, or a bfloat16 that rounds the other way
        lim = 1e-6 if dtype == torch.float32 else 2.0 ** -7
        assert float(((a - b).abs() - lim * b.abs()).max()) <= 1e-6
