"""Blocks of keys side by side: room for every position of the page table, whatever the step's lengths were when it was made."""
import types

import pytest
import torch


def _step(table, positions, max_kv_len, buffer):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=table.device)  # noqa: E731
    return types.SimpleNamespace(all_single=True, max_new=1, max_kv_len=max_kv_len, seq_ids=i32(list(range(len(positions)))),
                                 positions=i32(positions), buffer=buffer)


@pytest.mark.parametrize("pages_each,max_kv_len", [(4, 100), (8, 129), (1, 1)])
def test_room_follows_the_table_and_not_the_lengths_of_the_moment(pages_each, max_kv_len, monkeypatch):
    """A captured step is replayed at later positions of the same table: its blocks must reach them."""
    from llmplayer_b200.kernels import ops
    launched, taken = [], []

    class Library:                                        # records the launch instead of making it
        def __getattr__(self, name):
            return lambda *args: launched.append(args) or 0

    monkeypatch.setattr(ops, "library", lambda name: Library())
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_want", lambda *args, **kw: None)
    H, G, hd, P, B = 4, 2, 64, 64, 2
    table = torch.zeros(B, pages_each, dtype=torch.int32)

    def buffer(name, shape, dtype):
        taken.append(torch.empty(shape, dtype=dtype, device="meta").numel())
        return torch.empty(1, dtype=dtype)

    q, out = torch.zeros(B, H * hd), torch.zeros(B, H * hd)
    ops.attention(_step(table, [max_kv_len - 1] * B, max_kv_len, buffer), q, out, torch.zeros(3, 2, G, P, hd), table, num_heads=H,
                  num_kv_heads=G, head_dim=hd, scale=0.1, window=None, fast=False)
    blocks = launched[0][-2]
    assert blocks * ops.PLAIN_KEY_BLOCK >= pages_each * P
    assert taken == [B * H * blocks * (hd + 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("position", [0, 127, 128, 300, 511])
def test_a_step_moved_on_gives_the_same_bits(position):
    """The lengths a step was made with do not matter to its result."""
    from llmplayer_b200.kernels import ops
    H, G, hd, P, B, each = 4, 2, 64, 64, 3, 8
    g = torch.Generator(device="cuda:0").manual_seed(position)
    pages = torch.randn(B * each, 2, G, P, hd, generator=g, device="cuda:0")
    q = torch.randn(B, H * hd, generator=g, device="cuda:0")
    table = torch.arange(B * each, dtype=torch.int32, device="cuda:0").reshape(B, each)
    buffer = lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device="cuda:0")  # noqa: E731
    kw = dict(num_heads=H, num_kv_heads=G, head_dim=hd, scale=0.1, window=None)
    ctx = _step(table, [position, position // 2, 0], 1, buffer)
    out, want = torch.empty_like(q), torch.empty_like(q)
    ops.attention(ctx, q, out, pages, table, fast=False, **kw)
    ops.attention_plain(q, want, pages, table, ctx.seq_ids, ctx.positions, **kw)
    assert torch.equal(out, want)
