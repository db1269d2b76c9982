"""Latent attention over a bfloat16 cache on the tensor cores: queries, weights and latents in three bfloat16 parts. Each kernel
against float64, at the edges of its blocks of 64 keys and tiles of 16 rows, with windows, shares and several new tokens."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(got, ref):
    return float((got.double() - ref).abs().max() / ref.abs().max())


@pytest.mark.parametrize("rank,dr,H", [(64, 0, 3), (128, 16, 16), (256, 32, 8), (512, 64, 16), (512, 64, 40)])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("shares", [1, 3, 7])
def test_attend(rank, dr, H, window, shares):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(rank + H)
    before, new = [0, 63, 64, 200, 129], [5, 1, 1, 1, 3]
    lengths = [a + b for a, b in zip(before, new)]
    width, Dk = 5, rank + dr
    pages = torch.randn(len(before) * width, 64, Dk, generator=g, device=DEV).to(torch.bfloat16)
    order = torch.randperm(len(before) * width, generator=torch.Generator().manual_seed(1)).reshape(len(before), width)
    for i, n in enumerate(lengths):                       # what lies behind a sequence's last row is no number
        page = order[i, (n - 1) // 64]
        pages[page, (n - 1) % 64 + 1:] = float("nan")
    table = order.clone().to(torch.int32)
    for i, b in enumerate(before):                        # pages that no row reaches any more are gone
        if window is not None:
            table[i, :max(0, b - window + 1) // 64] = -1
    T = sum(new)
    q = torch.randn(T, H, Dk, generator=g, device=DEV)
    part = torch.full((T, H, shares, rank + 2), float("nan"), device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    starts = [sum(new[:i]) for i in range(len(new) + 1)]
    scale = Dk ** -0.5
    ops.latent_attend(q, pages, table.to(DEV), i32(starts), i32(lengths), part, max_new=max(new), kv_rank=rank, scale=scale, window=window)
    assert bool(torch.isfinite(part[..., :rank]).all())
    for i, n in enumerate(new):
        rows = torch.cat([pages[order[i, p // 64], p % 64][None] for p in range(lengths[i])]).double()
        for k in range(n):
            t, pos = starts[i] + k, before[i] + k
            lo = max(0, pos - window + 1) if window else 0
            s = q[t].double() @ rows[lo:pos + 1].T * scale
            w = torch.softmax(s, -1)
            p = part[t].double()
            m = p[:, :, rank].max(-1, keepdim=True).values
            f = torch.exp(p[:, :, rank] - m)
            got = (p[:, :, :rank] * f[..., None]).sum(1) / (p[:, :, rank + 1] * f).sum(-1, keepdim=True)
            # float32 sums of 24-bit products
            assert rel(got, w @ rows[lo:pos + 1, :rank]) < 3e-6, (i, k)


@pytest.mark.parametrize("T,H,dn,dr,rank", [(1, 3, 16, 8, 64), (16, 2, 48, 0, 128), (33, 16, 128, 64, 512)])
def test_absorb(T, H, dn, dr, rank):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    q = torch.randn(T, H, dn + dr, generator=g, device=DEV)
    uk = torch.randn(H * dn, rank, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((T, H, rank + dr), float("nan"), device=DEV)
    ops.latent_absorb(q, uk, out, nope_dim=dn, rope_dim=dr)
    ref = torch.einsum("thd,hdr->thr", q[..., :dn].double(), uk.double().reshape(H, dn, rank))
    assert rel(out[..., :rank], ref) < 2e-6 and torch.equal(out[..., rank:], q[..., dn:])


@pytest.mark.parametrize("T,H,dv,rank,shares", [(1, 3, 8, 64, 1), (17, 2, 40, 192, 5), (33, 16, 128, 512, 4), (80, 4, 64, 256, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_expand(T, H, dv, rank, shares, dtype):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    part = torch.randn(T, H, shares, rank + 2, generator=g, device=DEV)
    part[..., rank + 1] = 0.5 + part[..., rank + 1].abs()
    if shares > 1:                                        # an empty share
        part[:, :, 1] = 0.0
        part[:, :, 1, rank] = -float("inf")
    uv = torch.randn(H * dv, rank, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(T, H, generator=g, device=DEV)
    out = torch.empty(T, H * dv, device=DEV, dtype=dtype)
    junk = torch.ones(1000, device=DEV)
    ops.latent_expand(part, uv, gate, out, value_dim=dv, clear=junk)
    p = part.double()
    f = torch.exp(p[..., rank] - p[..., rank].max(-1, keepdim=True).values)
    latent = (p[..., :rank] * f[..., None]).sum(2) / (p[..., rank + 1] * f).sum(-1, keepdim=True)
    ref = torch.einsum("thr,hvr->thv", latent, uv.double().reshape(H, dv, rank)) * torch.sigmoid(gate.double())[..., None]
    assert rel(out.reshape(T, H, dv), ref) < (3e-6 if dtype == torch.float32 else 5e-3) and float(junk.abs().sum()) == 0.0


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("dn,dr,rot,rank,dv", [(24, 16, 8, 40, 16), (128, 64, 64, 512, 128), (64, 32, 32, 256, 64)])
def test_prompt_layouts_four_and_eight_at_a_time(dn, dr, rot, rank, dv, interleaved):
    """The kernels that read and write several values at a time against the ones that take any size: a column to the right
    moves the same projection off their alignment."""
    from llmplayer_b200.kernels import ops
    H, lengths = 3, [70, 1, 64]
    g = torch.Generator(device=DEV).manual_seed(dn)
    T, hd = sum(lengths), next(s for s in (64, 128, 192, 256) if dn + dr <= s)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, seq = i32([p for n in lengths for p in range(n)]), i32([i for i, n in enumerate(lengths) for _ in range(n)])
    table = i32([[3, 1], [0, 0], [2, 0]])
    wide = torch.randn(T, H * (dn + dr) + rank + dr + 4, generator=g, device=DEV)
    rotation = ops.Rotation(torch.rand(rot // 2, generator=g, device=DEV), rot, interleaved, 1.25)
    gain = torch.randn(rank, generator=g, device=DEV)
    got = []
    for shift in (0, 1):
        proj = torch.cat([wide[:, wide.shape[1] - shift:], wide[:, :wide.shape[1] - shift]], dim=1).contiguous()
        pages = torch.zeros(4, 64, rank + dr, device=DEV, dtype=torch.bfloat16)
        latent, shared = torch.zeros(T, rank, device=DEV, dtype=torch.bfloat16), torch.zeros(T, dr, device=DEV, dtype=torch.bfloat16)
        half = torch.full((T, H * hd), 7.0, device=DEV, dtype=torch.bfloat16)
        q = torch.zeros(T, H, dn + dr, device=DEV)
        kw = dict(num_heads=H, nope_dim=dn, rope_dim=dr, kv_rank=rank, latent_out=latent, shared_out=shared, q_half=half)
        ops.latent_prepare(proj, shift, shift + H * (dn + dr), gain, 1e-5, rotation, pos, seq, table, q, pages, **kw)
        first = half.clone()
        ops.latent_prepare(proj, shift, shift + H * (dn + dr), gain, 1e-5, rotation, pos, seq, table, None, pages, **kw)
        assert torch.equal(first, half)
        got.append((q, half, shared, latent.float(), pages.float()))
    for a, b in zip(got[0][:3], got[1][:3]):
        assert torch.equal(a, b)
    for a, b in zip(got[0][3:], got[1][3:]):              # the norm's sum is taken in another order: a last bit may round the other way
        assert float((a - b).abs().max()) <= 2.0 ** -7 * float(b.abs().max())
    kv = torch.randn(T, H * (dn + dv), generator=g, device=DEV).to(torch.bfloat16)
    pages = torch.full((5, 2, H, 64, hd), float("nan"), device=DEV, dtype=torch.bfloat16)
    table = i32([[4, 2], [0, 0], [3, 0]])
    ops.latent_heads_to_pages(kv, got[0][2].to(torch.bfloat16), pos, seq, table, i32(lengths), pages, num_heads=H, nope_dim=dn, rope_dim=dr,
                              value_dim=dv)
    assert bool(torch.isnan(pages[1]).all())              # nobody's page
    for i, n in enumerate(lengths):
        t0 = sum(lengths[:i])
        k = torch.cat([pages[int(p), 0] for p in table[i, :-(-n // 64)]], dim=1).transpose(0, 1)
        v = torch.cat([pages[int(p), 1] for p in table[i, :-(-n // 64)]], dim=1).transpose(0, 1)
        rows = kv[t0:t0 + n]
        assert torch.equal(k[:n, :, :dn], rows[:, :H * dn].reshape(n, H, dn)) and torch.equal(v[:n, :, :dv], rows[:, H * dn:].reshape(n, H, dv))
        assert torch.equal(k[:n, :, dn:dn + dr], got[0][2][t0:t0 + n, None].to(torch.bfloat16).expand(n, H, dr))
        assert not k[:, :, dn + dr:].any() and not v[:, :, dv:].any() and not k[n:].any() and not v[n:].any()
    heads = torch.randn(T, H * hd, generator=g, device=DEV).to(torch.bfloat16)
    gate = torch.randn(T, H, generator=g, device=DEV)
    out = torch.empty(T, H * dv, device=DEV, dtype=torch.bfloat16)
    ops.latent_gate_heads(heads, gate, out, num_heads=H, head_dim=hd, value_dim=dv)
    ref = heads.reshape(T, H, hd)[..., :dv].double() * torch.sigmoid(gate.double())[..., None]
    assert rel(out.reshape(T, H, dv), ref) < 5e-3


@pytest.mark.parametrize("lengths", [[400, 200], [70, 1, 64], [1, 1]])
@pytest.mark.parametrize("H", [3, 16])
def test_prepared_rows_and_queries(lengths, H):
    """What is written to the cache and as queries against float64, in steps where the heads have CTAs of their own and in steps where
    a CTA takes a whole token: normed latents and the rotated shared part at every token's page and place, nothing anywhere else."""
    from llmplayer_b200.kernels import ops
    dn, dr, rank, P = 64, 32, 256, 64
    g = torch.Generator(device=DEV).manual_seed(len(lengths) + H)
    T = sum(lengths)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    positions = [5 + p for n in lengths for p in range(n)]
    seq = [i for i, n in enumerate(lengths) for _ in range(n)]
    width = -(-(max(lengths) + 5) // P)
    table = torch.randperm(len(lengths) * width + 1, generator=torch.Generator().manual_seed(2))[1:].reshape(len(lengths), width)
    proj = torch.randn(T, H * (dn + dr) + rank + dr, generator=g, device=DEV)
    freq, gain = torch.rand(dr // 2, generator=g, device=DEV), torch.randn(rank, generator=g, device=DEV)
    pages = torch.full((len(lengths) * width + 1, P, rank + dr), 7.0, device=DEV, dtype=torch.bfloat16)
    q = torch.zeros(T, H, dn + dr, device=DEV)
    ops.latent_prepare(proj, 0, H * (dn + dr), gain, 1e-5, ops.Rotation(freq, dr, False), i32(positions), i32(seq), table.to(torch.int32).to(DEV),
                       q, pages, num_heads=H, nope_dim=dn, rope_dim=dr, kv_rank=rank)
    angle = (torch.tensor(positions, device=DEV, dtype=torch.float32)[:, None] * freq).double()        # as float32 forms them

    def rotated(x):
        a, b = x[..., :dr // 2].double(), x[..., dr // 2:].double()
        shape = (T,) + (1,) * (x.dim() - 2) + (dr // 2,)
        c, s = torch.cos(angle).reshape(shape), torch.sin(angle).reshape(shape)
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    heads, kv = proj[:, :H * (dn + dr)].reshape(T, H, dn + dr), proj[:, H * (dn + dr):].double()
    assert torch.equal(q[..., :dn], heads[..., :dn]) and rel(q[..., dn:], rotated(heads[..., dn:])) < 1e-6
    latent = kv[:, :rank] / torch.sqrt((kv[:, :rank] ** 2).mean(-1, keepdim=True) + 1e-5) * gain.double()
    want = torch.cat([latent, rotated(proj[:, H * (dn + dr) + rank:])], -1)
    page = table[torch.tensor(seq), torch.tensor(positions) // P].to(DEV)
    place = torch.tensor(positions, device=DEV) % P
    got = pages[page, place].double()
    # one rounding to bfloat16 of a float32 value: 2^-8 of its power of two at most, and a bit for the value itself
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())
    touched = torch.zeros(pages.shape[:2], dtype=torch.bool, device=DEV)
    touched[page, place] = True
    assert bool((pages[~touched] == 7.0).all())
