"""The attention kernels alone (plain, tensor-core prefill, tensor-core decode) against a
float64 softmax attention, on caches whose pages are scattered and partly stale."""
import math

import pytest
import torch

from helpers import check_error

pytestmark = pytest.mark.gpu

PAGE = 64
# Largest |kernel - float64 attention| allowed in bfloat16, on outputs of order one: at most four times the worst
# that each kernel achieved on a B200 (decode and fused decode 4.3e-3, prompt kernels 1.0e-2, plain kernel 7.8e-3).
BOUND = {"decode": 1.5e-2, "fused": 1.5e-2, "prefill": 2e-2, "plain": 2e-2}


def build_cache(lengths, G, hd, dtype, seed, extra_pages=5):
    """Dense K/V per sequence plus their scattered paged form. Unused rows hold large junk."""
    g = torch.Generator().manual_seed(seed)
    need = [-(-n // PAGE) for n in lengths]
    num_pages = sum(need) + extra_pages
    order = torch.randperm(num_pages, generator=g).tolist()
    pages = (torch.randn(num_pages, 2, G, PAGE, hd, generator=g) * 30.0).to(dtype)      # junk everywhere
    width = max(need)
    table = torch.full((len(lengths), width), -1, dtype=torch.int32)
    dense = []
    for b, n in enumerate(lengths):
        k = torch.randn(n, G, hd, generator=g).to(dtype)
        v = torch.randn(n, G, hd, generator=g).to(dtype)
        dense.append((k, v))
        for blk in range(need[b]):
            page = order.pop()
            table[b, blk] = page
            rows = slice(blk * PAGE, min(n, (blk + 1) * PAGE))
            cnt = rows.stop - rows.start
            pages[page, 0, :, :cnt] = k[rows].transpose(0, 1)
            pages[page, 1, :, :cnt] = v[rows].transpose(0, 1)
    return dense, pages, table


def reference(q, k, v, positions, scale, window):
    """q [Tq, H, hd]; k, v [Tk, G, hd] (positions 0..Tk-1); float64 softmax attention."""
    q, k, v = q.double(), k.double(), v.double()
    H, G = q.shape[1], k.shape[1]
    out = torch.zeros_like(q)
    t = torch.arange(k.shape[0])
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T) * scale
        ok = t[None, :] <= positions[:, None]
        if window:
            ok &= t[None, :] > positions[:, None] - window
        s = s.masked_fill(~ok, float("-inf"))
        out[:, h] = torch.softmax(s, dim=-1) @ v[:, g]
    return out


def run_case(kind, lengths, new, H, G, hd, window, dtype, seed=0, crafted=False, shares=None):
    """``new[b]`` tokens of sequence b are the step's queries (the last ``new[b]`` positions).
    ``shares``: into how many shares a decode kernel cuts the page tables (None: its own choice);
    ``kind="fused"`` runs the decode kernel that starts from the projection (no rotation, no cache write)."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    dense, pages, table = build_cache(lengths, G, hd, dtype, seed)
    g = torch.Generator().manual_seed(seed + 1)
    T = sum(new)
    q = torch.randn(T, H, hd, generator=g).to(dtype)
    positions, seq_ids, q_start = [], [], [0]
    for b, (n, m) in enumerate(zip(lengths, new)):
        positions += list(range(n - m, n))
        seq_ids += [b] * m
        q_start.append(q_start[-1] + m)
    positions = torch.tensor(positions)
    if crafted:
        # one far key must win: scale a query and a key at the far end of each sequence's context
        for b, (n, m) in enumerate(zip(lengths, new)):
            far = 1 if not window else max(0, n - window)      # just inside the window's edge
            k, v = dense[b]
            row = q_start[b] + m - 1
            q[row] = 0
            q[row, :, 0] = 16.0
            k[far] = 0
            k[far, :, 0] = 16.0
            blk, off = divmod(far, PAGE)
            pages[table[b, blk], 0, :, off] = k[far]
    ref = torch.cat([reference(q[q_start[b]:q_start[b + 1]], dense[b][0], dense[b][1],
                               positions[q_start[b]:q_start[b + 1]], 1.0 / math.sqrt(hd), window)
                     for b in range(len(lengths))])
    qd = q.reshape(T, H * hd).to(dev)
    out = torch.full_like(qd, 7.0)
    pages_d, table_d = pages.to(dev), table.to(dev)
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd, scale=1.0 / math.sqrt(hd), window=window)
    kv_len = torch.tensor(lengths, dtype=torch.int32, device=dev)
    if kind == "plain":
        ops.attention_plain(qd, out, pages_d, table_d, torch.tensor(seq_ids, dtype=torch.int32, device=dev),
                            positions.to(torch.int32).to(dev), **kw)
    elif kind == "prefill":
        ops.attention_prefill(qd, out, pages_d, table_d, torch.tensor(q_start, dtype=torch.int32, device=dev), kv_len,
                              max(new), **kw)
    else:
        assert all(m == 1 for m in new)
        scratch = {}

        def buf(name, shape, dt):
            scratch[name] = torch.full(shape, float("nan"), dtype=dt, device=dev)
            return scratch[name]
        split = {}
        if shares:
            per = -(-table.shape[1] // shares)
            split = dict(pages_per_split=per, num_splits=-(-table.shape[1] // per))
        if kind == "fused":
            # the queries as the float32 projection would deliver them; this layer keeps no keys of its own, so
            # the kernel attends over the pages as they are
            counters = torch.zeros(ops.decode_groups(len(lengths), H, G), dtype=torch.int32, device=dev)
            ops.attention_decode_fused(qd.float(), ops.NO_ROTATION, out, pages_d, table_d, kv_len, buf, counters,
                                       write_kv=False, **kw, **split)
            assert int(counters.abs().sum()) == 0
        else:
            ops.attention_decode(qd, out, pages_d, table_d, kv_len, buf, **kw, **split)
    torch.cuda.synchronize()
    got = out.reshape(T, H, hd).double().cpu()
    assert torch.isfinite(got).all()
    err = float((got - ref).abs().max())
    from helpers import record_error
    record_error(f"attention kernel ({kind}), {str(dtype).split('.')[-1]}", f"H{H} G{G} hd{hd} window {window}", err,
                 2e-5 if dtype == torch.float32 else BOUND.get(kind, 2e-2))
    if crafted:
        for b in range(len(lengths)):
            row = q_start[b + 1] - 1
            far = 1 if not window else max(0, lengths[b] - window)
            want = dense[b][1][far].double()            # the far key dominates: output = its value
            H_G = H // G
            for h in range(H):
                assert (got[row, h] - want[h // H_G]).abs().max() < 0.05, (b, h)
    return err


GEOMETRIES = [(4, 2, 16), (3, 1, 32), (6, 3, 48), (32, 8, 64), (8, 2, 128), (2, 2, 256), (20, 1, 64), (4, 4, 96),
              (6, 2, 192)]


@pytest.mark.parametrize("H,G,hd", GEOMETRIES)
@pytest.mark.parametrize("window", [None, 70])
def test_plain_attention(H, G, hd, window):
    for dtype, tol in ((torch.float32, 2e-5), (torch.bfloat16, 2e-2)):
        err = run_case("plain", [1, 64, 65, 300], [1, 64, 3, 150], H, G, hd, window, dtype)
        assert err < tol, err


@pytest.mark.parametrize("H,G,hd", GEOMETRIES)
@pytest.mark.parametrize("window", [None, 70])
def test_tensor_core_prefill(H, G, hd, window):
    """Heads of 64 with long runs of new tokens take the tcgen05 kernel, everything else mma.sync."""
    err = run_case("prefill", [1, 64, 65, 300, 129], [1, 64, 3, 150, 129], H, G, hd, window, torch.bfloat16)
    assert err < BOUND["prefill"], err


@pytest.mark.parametrize("H,G,hd", [(32, 8, 64), (20, 1, 64), (3, 3, 64), (8, 2, 128), (24, 8, 128), (5, 5, 128)])
@pytest.mark.parametrize("window", [None, 70, 200])
@pytest.mark.parametrize("tcgen05", [True, False])
def test_both_prefill_kernels_at_head_sizes_64_and_128(H, G, hd, window, tcgen05, monkeypatch):
    from llmplayer_b200.kernels import ops
    monkeypatch.setattr(ops, "tcgen05_attention", tcgen05)
    lengths, new = [700, 128, 129, 391, 65], [700, 128, 100, 130, 65]        # whole prompts and continued ones
    err = run_case("prefill", lengths, new, H, G, hd, window, torch.bfloat16, seed=7)
    assert err < BOUND["prefill"], err
    run_case("prefill", [900, 333], [200, 70], H, G, hd, window, torch.bfloat16, seed=3, crafted=True)


@pytest.mark.parametrize("hd", [64, 128])
def test_prefill_whose_maximum_keeps_growing(hd):
    """The tcgen05 prompt kernel keeps a reference maximum per row that moves only when the row's true maximum
    has outgrown it by a factor of 256; here every later page holds a key that beats all earlier ones by far more
    (and by less, in alternation), so the output in tensor memory is brought down again and again."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    H, G, n = 4, 2, 640
    dense, pages, table = build_cache([n], G, hd, torch.bfloat16, seed=5)
    k, v = dense[0]
    g = torch.Generator().manual_seed(6)
    q = torch.randn(n, H, hd, generator=g).to(torch.bfloat16)
    q[:, :, 0] = 4.0
    for page in range(n // PAGE):                      # one key per page whose score grows page by page
        at = page * PAGE + 17
        k[at] = 0
        k[at, :, 0] = (1.5 if page % 2 else 6.0) * (page + 1)
        pages[table[0, page], 0, :, 17] = k[at]
    ref = reference(q, k, v, torch.arange(n), 1.0 / math.sqrt(hd), None)
    qd = q.reshape(n, H * hd).to(dev)
    out = torch.zeros_like(qd)
    ops.attention_prefill(qd, out, pages.to(dev), table.to(dev), torch.tensor([0, n], dtype=torch.int32, device=dev),
                          torch.tensor([n], dtype=torch.int32, device=dev), n, num_heads=H, num_kv_heads=G, head_dim=hd,
                          scale=1.0 / math.sqrt(hd), window=None)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    err = float((out.reshape(n, H, hd).double().cpu() - ref).abs().max())
    assert err < BOUND["prefill"], err


@pytest.mark.parametrize("H,G,hd", GEOMETRIES)
@pytest.mark.parametrize("window", [None, 70])
def test_tensor_core_decode(H, G, hd, window):
    lengths = [1, 64, 65, 700, 129, 17]
    err = run_case("decode", lengths, [1] * len(lengths), H, G, hd, window, torch.bfloat16)
    assert err < BOUND["decode"], err


@pytest.mark.parametrize("kind", ["decode", "fused"])
@pytest.mark.parametrize("shares", [2, 3, 5])
@pytest.mark.parametrize("window", [None, 70, 200])
def test_decode_in_several_shares_against_float64(kind, shares, window):
    """The pages of a sequence cut into shares: with a window some shares lie wholly before it, one share may
    hold nothing but the newest page, short sequences leave most shares empty. Compared with the float64
    attention (not with another entry point of the same kernel), random and with one far key made to win."""
    lengths = [1, 64, 65, 700, 129, 17, 641]
    err = run_case(kind, lengths, [1] * len(lengths), 8, 2, 64, window, torch.bfloat16, seed=11, shares=shares)
    assert err < BOUND[kind], err
    err = run_case(kind, lengths, [1] * len(lengths), 6, 3, 48, window, torch.bfloat16, seed=12, shares=shares)
    assert err < BOUND[kind], err
    run_case(kind, [900, 333, 70], [1, 1, 1], 8, 2, 64, window, torch.bfloat16, seed=3, crafted=True, shares=shares)


@pytest.mark.parametrize("kind", ["decode", "fused"])
@pytest.mark.parametrize("window", [None, 300, 1000])
def test_shares_fitted_to_each_sequence(kind, window):
    """Left to themselves the decode kernels cut every sequence into as many shares as its own length (within the
    window) gives pages for: here four, two, one and one shares in one grid, some CTAs with nothing to do."""
    lengths = [2000, 70, 1100, 513]
    err = run_case(kind, lengths, [1] * 4, 8, 2, 64, window, torch.bfloat16, seed=31)
    assert err < BOUND[kind], err
    run_case(kind, lengths, [1] * 4, 4, 2, 128, window, torch.bfloat16, seed=32, crafted=True)


def test_a_sequence_of_length_zero_reads_and_writes_nothing():
    """A row whose length is zero is an empty sequence: its output is zero, and neither its neighbours'
    results nor any page changes (the fused kernel stores no key for it)."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    H, G, hd = 8, 2, 64
    lengths = [130, 0, 65]
    _, pages, table = build_cache([130, 1, 65], G, hd, torch.bfloat16, seed=21)
    g = torch.Generator().manual_seed(22)
    qkv = torch.randn(3, (H + 2 * G) * hd, generator=g).to(dev)
    table_d = table.to(dev)
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd, scale=hd ** -0.5, window=None)

    def scratch(name, shape, dt):
        return torch.full(shape, float("nan"), dtype=dt, device=dev)

    def run(lens, shares):
        p = pages.to(dev).clone()
        out = torch.full((3, H * hd), 5.0, dtype=torch.bfloat16, device=dev)
        counters = torch.zeros(ops.decode_groups(3, H, G), dtype=torch.int32, device=dev)
        per = -(-table.shape[1] // shares)
        ops.attention_decode_fused(qkv, ops.NO_ROTATION, out, p, table_d,
                                   torch.tensor(lens, dtype=torch.int32, device=dev), scratch, counters,
                                   write_kv=True, pages_per_split=per, num_splits=-(-table.shape[1] // per), **kw)
        torch.cuda.synchronize()
        return out, p

    for shares in (1, 3):
        with_empty, pages_empty = run(lengths, shares)
        with_one, pages_one = run([130, 1, 65], shares)
        assert torch.isfinite(with_empty.float()).all()
        assert float(with_empty[1].float().abs().max()) == 0.0
        assert torch.equal(with_empty[0], with_one[0]) and torch.equal(with_empty[2], with_one[2])
        # only the page of the middle sequence may differ between the two runs, and with a length of zero
        # it is exactly what it was
        middle = int(table[1, 0])
        assert torch.equal(pages_empty[middle], pages.to(dev)[middle])
        others = [i for i in range(pages.shape[0]) if i != middle]
        assert torch.equal(pages_empty[others], pages_one[others])
    q = torch.randn(3, H * hd, generator=g).to(torch.bfloat16).to(dev)
    out = torch.full_like(q, 5.0)
    ops.attention_decode(q, out, pages.to(dev), table_d, torch.tensor(lengths, dtype=torch.int32, device=dev), scratch,
                         pages_per_split=1, num_splits=table.shape[1], **kw)
    torch.cuda.synchronize()
    assert float(out[1].float().abs().max()) == 0.0 and torch.isfinite(out.float()).all()


def test_shared_memory_grants_do_not_cross_between_head_sizes():
    """Each kernel instantiation remembers its own grant of dynamic shared memory: a decode step at a head
    size of 96 (which needs a large grant) must not make the kernel for heads of 64 skip asking for its own."""
    for hd in (96, 64, 112, 128, 64):
        for kind in ("decode", "fused"):
            err = run_case(kind, [700, 65], [1, 1], 4, 2, hd, None, torch.bfloat16, seed=hd, shares=2)
            assert err < BOUND[kind], (hd, kind, err)


@pytest.mark.parametrize("kind", ["plain", "prefill", "decode"])
@pytest.mark.parametrize("window", [None, 200])
def test_a_far_key_among_hundreds_is_found(kind, window):
    lengths = [900, 333]
    new = [1, 1] if kind == "decode" else [5, 1]
    run_case(kind, lengths, new, 8, 2, 64, window, torch.bfloat16, seed=3, crafted=True)


@pytest.mark.parametrize("H,G,hd,rd,pairing", [(32, 8, 64, 64, "split_half"), (6, 3, 48, 32, "interleaved"),
                                               (20, 1, 64, 64, "split_half"), (4, 2, 128, 0, "split_half")])
@pytest.mark.parametrize("window", [None, 70])
@pytest.mark.parametrize("splits", [1, 3])
def test_fused_decode_equals_rotation_then_attention(H, G, hd, rd, pairing, window, splits):
    """The fused decode kernel (rotation, cache write, attention, merge) against the separate kernels."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    lengths = [1, 64, 65, 700, 129, 17]
    B = len(lengths)
    _, pages, table = build_cache(lengths, G, hd, torch.bfloat16, seed=hd + H)
    g = torch.Generator().manual_seed(5)
    qkv = torch.randn(B, (H + 2 * G) * hd, generator=g).to(dev)
    inv = (torch.rand(max(rd // 2, 1), generator=g) * 0.5).to(dev) if rd else None
    table_d = table.to(dev)
    kv_len = torch.tensor(lengths, dtype=torch.int32, device=dev)
    positions = kv_len - 1
    seq_ids = torch.arange(B, dtype=torch.int32, device=dev)
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd)
    per = -(-table.shape[1] // splits)
    n_splits = -(-table.shape[1] // per)

    def scratch(name, shape, dt):
        return torch.full(shape, float("nan"), dtype=dt, device=dev)

    pages_a = pages.to(dev).clone()
    q = torch.empty(B, H * hd, dtype=torch.bfloat16, device=dev)
    rotation = ops.Rotation(inv, rd, pairing == "interleaved") if rd else ops.NO_ROTATION
    ops.rope_cache_write(qkv, rotation, positions, seq_ids, table_d, q, pages_a, **kw)
    want = torch.zeros_like(q)
    ops.attention_decode(q, want, pages_a, table_d, kv_len, scratch, scale=hd ** -0.5, window=window,
                         pages_per_split=per, num_splits=n_splits, **kw)

    pages_b = pages.to(dev).clone()
    got = torch.full_like(q, 3.0)
    counters = torch.zeros(ops.decode_groups(B, H, G), dtype=torch.int32, device=dev)
    for _ in range(2):                       # twice: the share counters must be back at zero
        ops.attention_decode_fused(qkv, rotation, got, pages_b, table_d, kv_len, scratch, counters, write_kv=True,
                                   scale=hd ** -0.5, window=window, pages_per_split=per, num_splits=n_splits, **kw)
    assert int(counters.abs().sum()) == 0
    torch.cuda.synchronize()
    assert torch.equal(pages_a, pages_b)                      # the same keys and values were stored
    assert float((got.float() - want.float()).abs().max()) <= 2e-2


@pytest.mark.parametrize("H,G,hd", [(8, 2, 64), (4, 1, 128)])
def test_fused_decode_over_more_than_32_pages_in_one_share(H, G, hd):
    """One share per sequence holding 33 to 47 pages: the kernel that brings its pages by TMA keeps 32 entries
    of the page table in the first warp's lanes and has to fetch the next 32 on the way. Against the separate
    rotation and decode kernels (16-byte copies), on pages that are scattered over the cache."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    lengths = [2500, 2049, 3000, 70, 2113]
    B = len(lengths)
    _, pages, table = build_cache(lengths, G, hd, torch.bfloat16, seed=hd)
    g = torch.Generator().manual_seed(8)
    qkv = torch.randn(B, (H + 2 * G) * hd, generator=g).to(dev)
    rd = hd
    inv = (torch.rand(rd // 2, generator=g) * 0.01).to(dev)
    table_d = table.to(dev)
    kv_len = torch.tensor(lengths, dtype=torch.int32, device=dev)
    positions = kv_len - 1
    seq_ids = torch.arange(B, dtype=torch.int32, device=dev)
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd)
    per = table.shape[1]

    def scratch(name, shape, dt):
        return torch.full(shape, float("nan"), dtype=dt, device=dev)

    rotation = ops.Rotation(inv, rd, False)
    pages_a = pages.to(dev).clone()
    q = torch.empty(B, H * hd, dtype=torch.bfloat16, device=dev)
    ops.rope_cache_write(qkv, rotation, positions, seq_ids, table_d, q, pages_a, **kw)
    want = torch.zeros_like(q)
    ops.attention_decode(q, want, pages_a, table_d, kv_len, scratch, scale=hd ** -0.5, window=None,
                         pages_per_split=per, num_splits=1, **kw)
    pages_b = pages.to(dev).clone()
    got = torch.full_like(q, 3.0)
    counters = torch.zeros(ops.decode_groups(B, H, G), dtype=torch.int32, device=dev)
    ops.attention_decode_fused(qkv, rotation, got, pages_b, table_d, kv_len, scratch, counters, write_kv=True,
                               scale=hd ** -0.5, window=None, pages_per_split=per, num_splits=1, **kw)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    assert torch.equal(pages_a, pages_b)
    assert float((got.float() - want.float()).abs().max()) <= 2e-2


@pytest.mark.parametrize("H,G,hd", [(4, 2, 64), (9, 1, 48), (3, 3, 128), (2, 1, 256), (2, 2, 20)])
@pytest.mark.parametrize("form", ["all", "window", "kept", "chunk", "distance", "gate"])
def test_float32_attention_in_blocks(form, H, G, hd):
    """Tiles of queries over blocks of keys, and blocks of keys side by side: against float64, and the same bits from both
    however the sequences are cut into calls. Lengths at the edges of blocks (128), tiles (32, 64) and pages."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    g = torch.Generator().manual_seed(hd + H)
    lengths, P = [300, 129, 1, 64], 64
    width = -(-max(lengths) // P)
    table = torch.randperm(len(lengths) * width, generator=g).reshape(len(lengths), width).to(torch.int32)
    pages = torch.randn(len(lengths) * width, 2, G, P, hd, generator=g)
    T = sum(lengths)
    q = torch.randn(T, H * hd, generator=g) * 2
    seq = torch.tensor([i for i, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32)
    pos = torch.tensor([p for n in lengths for p in range(n)], dtype=torch.int32)
    window = 70 if form in ("window", "kept") else None
    keep = 5 if form == "kept" else 0
    chunk = 100 if form == "chunk" else 0
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd, scale=hd ** -0.5, window=window, keep_first=keep, chunk=chunk,
              softcap=20.0 if form == "kept" else None)
    sinks = torch.randn(H, generator=g) if form != "all" else None
    distance = (torch.rand(H, generator=g), 0.05 * torch.rand(H, generator=g)) if form in ("distance", "gate") else None
    gate = torch.randn(T, H + 3, generator=g) if form == "gate" else None
    ref = torch.empty(T, H, hd, dtype=torch.float64)
    for t in range(T):
        p, i = int(pos[t]), int(seq[t])
        keys = [j for j in range(p + 1) if (window is None or j > p - window or j < keep) and (not chunk or j // chunk == p // chunk)]
        for h in range(H):
            kv = torch.stack([pages[table[i, j // P], :, h * G // H, j % P] for j in keys]).double()     # [keys, 2, hd]
            s = kv[:, 0] @ q[t].reshape(H, hd)[h].double() * hd ** -0.5
            if kw["softcap"]:
                s = 20.0 * torch.tanh(s / 20.0)
            if distance is not None:
                s = s - distance[0][h].double() * torch.log1p(distance[1][h].double() * torch.arange(p, -1, -1, dtype=torch.float64))
            w = torch.softmax(s if sinks is None else torch.cat([s, sinks[h:h + 1].double()]), 0)[:len(keys)]
            ref[t, h] = w @ kv[:, 1] * (1.0 if gate is None else torch.sigmoid(gate[t, 2 + h].double()))
    if window is not None:          # pages that no query of the last call below reaches are gone
        gone = table.clone()
        gone[0, 1 if keep else 0:2] = -1
    d = lambda t: t.to(dev)  # noqa: E731
    whole = torch.empty(T, H * hd, device=dev)
    scratch = lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device=dev)  # noqa: E731
    sk = {"sinks": None if sinks is None else d(sinks), "distance": None if distance is None else tuple(map(d, distance))}
    gated = lambda rows: None if gate is None else d(gate[rows])[:, 2:2 + H]  # noqa: E731
    ops.attention_plain(d(q), whole, d(pages), d(table), d(seq), d(pos), **kw, **sk, gate=gated(slice(None)))
    # scores carry hd products, exponentials and sums of up to 300 weights: a few hundred units of 2^-24 times scores of up to 20
    assert float((whole.double().cpu().reshape(T, H, hd) - ref).abs().max()) < 2e-5 * float(ref.abs().max())
    for rows in ([299, 300, 428, 429, 493], [0, 63, 64, 127, 128], list(range(250, 300))):
        at = torch.tensor(rows)
        late = window is not None and min(rows) >= 250 and max(rows) < 300
        for use in (None, scratch):
            out = torch.empty(len(rows), H * hd, device=dev)
            ops.attention_plain(d(q[at]), out, d(pages), d(gone if late else table), d(seq[at]), d(pos[at]), **kw, **sk, scratch=use,
                                gate=gated(at), longest=int(pos[at].max()) + 1)
            assert torch.equal(out, whole[at.to(dev)]), (rows, use is None)


SHAPED = [dict(exact_weights=True), dict(exact_weights=True, softcap=15.0, sinks=True), dict(exact_weights=True, window=100, keep_first=5),
          dict(exact_weights=True, window=150, keep_first=70, sinks=True, gate=True), dict(exact_weights=True, chunk=96, gate=True),
          dict(exact_weights=True, chunk=200, softcap=20.0)]


@pytest.mark.parametrize("hd,vd,H,G", [(64, 64, 4, 2), (128, 128, 4, 1), (192, 128, 3, 3), (192, 72, 2, 1)])
@pytest.mark.parametrize("shape", [{}, dict(window=130)] + SHAPED, ids=lambda s: "-".join(s) or "plain")
def test_tcgen05_prompt_attention_with_everything_that_shapes_it(hd, vd, H, G, shape):
    """Long runs of new tokens against float64: sequences that start at their first token and ones that continue, at the edges of
    tiles of 128 rows and pages; pages that no query reaches are gone."""
    from llmplayer_b200.kernels import ops
    dev, P = "cuda:0", 64
    g = torch.Generator(device=dev).manual_seed(hd + len(shape))
    before, new = [0, 0, 300, 129, 64], [257, 128, 65, 200, 1]
    lengths = [a + b for a, b in zip(before, new)]
    width = -(-max(lengths) // P)
    order = torch.randperm(len(new) * width, generator=torch.Generator().manual_seed(3)).reshape(len(new), width)
    pages = torch.randn(len(new) * width, 2, G, P, hd, generator=g, device=dev).to(torch.bfloat16)
    pages[:, 1, :, :, vd:] = 0
    T = sum(new)
    q = (1.5 * torch.randn(T, H * hd, generator=g, device=dev)).to(torch.bfloat16)
    shape = dict(shape)
    window, keep, chunk, cap = shape.get("window"), shape.get("keep_first", 0), shape.get("chunk", 0), shape.get("softcap")
    table = order.clone().to(torch.int32)
    for i, b in enumerate(before):
        first = max(b - window + 1 if window else 0, b // chunk * chunk if chunk else 0)
        table[i, -(-keep // P):max(0, first) // P] = -1
    if shape.pop("sinks", False):
        shape["sinks"] = 2 * torch.randn(H, generator=g, device=dev)
    if shape.pop("gate", False):
        shape["gate"] = torch.randn(T, H + 3, generator=g, device=dev)[:, 2:2 + H]
    out = torch.full((T, H * hd), 7.0, device=dev, dtype=torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    starts = [sum(new[:i]) for i in range(len(new) + 1)]
    scale = hd ** -0.5
    kw = dict({"window": None}, **shape)
    ops.attention_prefill(q, out, pages, table.to(dev), i32(starts), i32(lengths), max(new), num_heads=H, num_kv_heads=G, head_dim=hd,
                          scale=scale, value_dim=vd, **kw)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    worst, top = 0.0, 0.0
    for i, n in enumerate(new):
        kv = torch.cat([pages[int(p)] for p in order[i, :-(-lengths[i] // P)]], dim=2)[:, :, :lengths[i]].double()      # [2, G, len, hd]
        pos = before[i] + torch.arange(n, device=dev)[:, None]
        key = torch.arange(lengths[i], device=dev)[None, :]
        seen = key <= pos
        if window:
            seen &= (key > pos - window) | (key < keep)
        if chunk:
            seen &= key // chunk == pos // chunk
        for h in range(H):
            s = q[starts[i]:starts[i] + n].reshape(n, H, hd)[:, h].double() @ kv[0, h * G // H].T * scale
            s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(~seen, float("-inf"))
            if "sinks" in shape:
                s = torch.cat([s, shape["sinks"][h].double().expand(n, 1)], dim=1)
            ref = torch.softmax(s, -1)[:, :lengths[i]] @ kv[1, h * G // H]
            if "gate" in shape:
                ref = ref * torch.sigmoid(shape["gate"][starts[i]:starts[i] + n, h].double())[:, None]
            got = out[starts[i]:starts[i] + n].reshape(n, H, hd)[:, h, :vd].double()
            worst, top = max(worst, float((got - ref[:, :vd]).abs().max())), max(top, float(ref.abs().max()))
    # the result's own rounding to bfloat16 is 2^-9 of a value; weights rounded to bfloat16 add as much again and more in short rows
    check_error("attention kernel (tcgen05, " + ("float32 weights)" if "exact_weights" in shape else "bfloat16 weights)"), f"{H}/{G} x {hd}",
                worst / top, 4e-3 if "exact_weights" in shape else 2e-2)


@pytest.mark.parametrize("vd", [128, 72])
def test_a_rows_largest_weight_is_not_rounded_at_192(vd):
    """Rows whose largest score stands in a later page, less than 2^8 above the first page's in weight: that weight is one and enters
    the product exactly, so the only rounding left is the result's own. A value between 2^k and 2^(k + 1)
    has 2^7 steps, so the error is uniform within 2^(k - 8); relative to mantissas spread evenly in the logarithm that is
    2^-8 sqrt(3 / (8 ln 2) / 3) = 1.66e-3 in the root mean square, and sqrt(2) times as much if the weight were rounded as well. The
    bound lies between the two."""
    from llmplayer_b200.kernels import ops
    dev, P, B, n, H, hd = "cuda:0", 64, 4, 256, 3, 192
    pages = torch.zeros(B * (n // P), 2, 1, P, hd, device=dev, dtype=torch.bfloat16)
    table = torch.arange(B * (n // P), device=dev, dtype=torch.int32).reshape(B, n // P)
    at = 100                                              # the key that stands out, in the second page
    pages[at // P::n // P, 0, :, at % P, 0] = 1.0
    pages[at // P::n // P, 1, :, at % P, :vd] = 1.0
    q = torch.zeros(B * n, H, hd, device=dev)
    q[..., 0] = torch.linspace(1.0, 5.5, B * n * H, device=dev).reshape(B * n, H)       # in log2: 1.4 to 7.9
    q = q.reshape(B * n, H * hd).to(torch.bfloat16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)  # noqa: E731
    out = torch.empty(B * n, H * hd, device=dev, dtype=torch.bfloat16)
    ops.attention_prefill(q, out, pages, table, i32([n * i for i in range(B + 1)]), i32([n] * B), n, num_heads=H, num_kv_heads=1,
                          head_dim=hd, scale=1.0, window=None, value_dim=vd)
    ops.check_kernel_status()
    e = torch.exp(q.reshape(B, n, H, hd)[..., 0].double())
    ref = e / (e + torch.arange(n, device=dev)[None, :, None])                          # the other t keys have score zero
    got = out.reshape(B, n, H, hd)[..., :vd].double()
    error = ((got - ref[..., None]) / ref[..., None])[:, 128:]
    check_error("attention kernel (tcgen05, a largest weight that is one)", f"{hd} x {vd}", float(error.square().mean().sqrt()), 1.95e-3)


@pytest.mark.parametrize("form", ["no number", "minus infinity"])
@pytest.mark.parametrize("H,G,hd", [(4, 2, 64), (3, 3, 20)])
def test_float32_scores_that_are_no_number_reach_the_result(H, G, hd, form):
    """A block of 128 keys all of whose scores are no number makes the rows that see it no number, also where it holds a single key;
    scores of minus infinity weigh nothing. Tiles of queries, and blocks side by side."""
    from llmplayer_b200.kernels import ops
    dev, P, lengths = "cuda:0", 64, [300, 129, 257]
    g = torch.Generator().manual_seed(hd)
    pages = torch.randn(15, 2, G, P, hd, generator=g).abs()
    table = torch.arange(15, dtype=torch.int32).reshape(3, 5)
    T = sum(lengths)
    q = torch.randn(T, H * hd, generator=g).abs()
    seq = torch.tensor([i for i, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32)
    pos = torch.tensor([p for n in lengths for p in range(n)], dtype=torch.int32)
    bad = [(0, range(0, 128)), (1, range(128, 129)), (2, range(128, 256))]            # (sequence, keys)
    for i, keys in bad:
        for key in keys:
            pages[int(table[i, key // P]), 0, :, key % P] = float("nan") if form == "no number" else -float("inf")
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd, scale=hd ** -0.5, window=None)
    d = lambda t: t.to(dev)  # noqa: E731
    whole = torch.empty(T, H * hd, device=dev)
    ops.attention_plain(d(q), whole, d(pages), d(table), d(seq), d(pos), **kw)
    parts = torch.empty(T, H * hd, device=dev)
    scratch = lambda name, shape, dtype: torch.full(shape, 3.0, dtype=dtype, device=dev)  # noqa: E731
    ops.attention_plain(d(q), parts, d(pages), d(table), d(seq), d(pos), **kw, scratch=scratch, longest=max(lengths))
    for out in (whole, parts):
        none = torch.isnan(out).reshape(T, -1).cpu()
        for t in range(T):
            first, count = next((keys[0], len(keys)) for i, keys in bad if i == int(seq[t]))
            # a row of nothing but minus infinities has no weights either
            want = int(pos[t]) >= first if form == "no number" else first == 0 and int(pos[t]) < count
            assert bool((none[t] == want).all()), (form, t, int(seq[t]), int(pos[t]))
