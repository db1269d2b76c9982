"""Cache rows and absorbed queries of latent attention in one launch, against the two kernels that do it one after the other: at the edges of
a tile of 16 tokens, with queries of their own, both pairings of the rotation, and sizes that the one launch leaves to the two."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1, 16, 17, 35])
@pytest.mark.parametrize("H,dn,dr,rot,rank", [(3, 16, 8, 8, 64), (16, 128, 64, 64, 512), (2, 48, 12, 4, 128), (2, 32, 0, 0, 64), (2, 24, 16, 8, 40)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("own_queries", [False, True])
def test_queries(T, H, dn, dr, rot, rank, interleaved, own_queries):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T + rank)
    r = lambda *shape: torch.randn(*shape, generator=g, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    first = T // 2                                        # two sequences, the second one starts inside a page
    pos, seq = i32(list(range(first)) + [60 + i for i in range(T - first)]), i32([0] * first + [1] * (T - first))
    table = i32([[3, 1], [0, 2]])
    rotation = ops.Rotation(torch.rand(rot // 2, generator=g, device=DEV), rot, interleaved, 1.25) if rot else ops.Rotation()
    gain, uk = r(rank), r(H * dn, rank).to(torch.bfloat16)
    proj, q = r(T, H * (dn + dr) + rank + dr + 4), r(T, H * (dn + dr) + 4)[:, :H * (dn + dr)] if own_queries else None
    kw = dict(num_heads=H, nope_dim=dn, rope_dim=dr, kv_rank=rank, q_from=q)
    pages = [torch.zeros(4, 64, rank + dr, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    got, want = [torch.full((T, H, rank + dr), float("nan"), device=DEV) for _ in range(2)]
    buffer = lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device=DEV)  # noqa: E731
    ops.latent_queries(proj, 0, H * (dn + dr), gain, 1e-5, rotation, pos, seq, table, pages[0], uk, got, buffer, **kw)
    mid = torch.empty(T, H, dn + dr, device=DEV)
    ops.latent_prepare(proj, 0, H * (dn + dr), gain, 1e-5, rotation, pos, seq, table, mid, pages[1], **kw)
    ops.latent_absorb(mid, uk, want, nope_dim=dn, rope_dim=dr)
    assert torch.equal(got, want)
    assert torch.equal(pages[0], pages[1])


def test_a_rotary_width_that_the_separate_kernel_refuses_stays_refused():
    from llmplayer_b200.errors import KernelError
    from llmplayer_b200.kernels import ops
    T, H, dn, dr, rank = 2, 2, 16, 264, 64
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    buffer = lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device=DEV)  # noqa: E731
    with pytest.raises(KernelError, match="rotary width"):
        ops.latent_queries(torch.randn(T, H * (dn + dr) + rank + dr, device=DEV), 0, H * (dn + dr), torch.ones(rank, device=DEV), 1e-5,
                           ops.Rotation(torch.rand(dr // 2, device=DEV), dr), i32([0, 1]), i32([0, 0]), i32([[0]]),
                           torch.zeros(1, 64, rank + dr, device=DEV, dtype=torch.bfloat16),
                           torch.randn(H * dn, rank, device=DEV).to(torch.bfloat16), torch.empty(T, H, rank + dr, device=DEV), buffer,
                           num_heads=H, nope_dim=dn, rope_dim=dr, kv_rank=rank)
