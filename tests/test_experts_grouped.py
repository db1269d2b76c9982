"""Experts run for the tokens that chose them only: the lists, the gathered rows and the two products together."""
import pytest
import torch

CASES = [  # tokens, experts, chosen, hidden size, shared hidden size, width, spread
    (256, 8, 2, 128, 0, 256, "even"), (257, 4, 1, 256, 128, 264, "even"), (300, 3, 2, 128, 384, 520, "one"),
    (1025, 16, 4, 128, 0, 64, "even"), (513, 8, 3, 384, 256, 1024, "rare"), (5, 2, 1, 128, 128, 8, "none"), (2048, 32, 6, 128, 0, 128, "even"),
]


def test_rows_cover_every_spread_of_the_choices():
    from llmplayer_b200.kernels import ops
    for T, E, top, _, shared, _, _ in CASES:
        worst = 0
        # k experts with one token each and the rest of the choices in as few experts as can hold them
        for k in range(E + 1):
            left, tiles = T * min(top, E) - k, k
            for _ in range(E - k):
                n = min(T, max(0, left))
                tiles, left = tiles + -(-n // 128), left - n
            worst = max(worst, tiles)
        assert ops.expert_rows(T, E, top, shared > 0) >= 128 * (worst + (-(-T // 128) if shared else 0))


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,top,ff,shared,d,spread", CASES)
@pytest.mark.parametrize("overwrite", [False, True])
def test_experts_against_float64(T, E, top, ff, shared, d, spread, overwrite):
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(T + E)
    x = torch.randn(T, d, generator=g, device=dev).to(torch.bfloat16)
    total = E * ff + shared
    gate, up = ((torch.randn(total, d, generator=g, device=dev) / d ** 0.5).to(torch.bfloat16) for _ in range(2))
    down = (torch.randn(d, total, generator=g, device=dev) / ff ** 0.5).to(torch.bfloat16)
    score = torch.rand(T, E, generator=g, device=dev)
    if spread == "one":                      # everybody's first choice is the last expert, the first one is nobody's
        score[:, -1] += 2.0
        score[:, 0] -= 2.0
    elif spread == "rare":                   # an expert with a single token, in the last row
        score[:, 2] -= 2.0
        score[-1, 2] += 4.0
    weights = torch.zeros(T, E + 2, device=dev)          # two further columns that belong to nobody here
    weights[:, E:] = 7.0
    if spread != "none":
        at = score.topk(top, dim=1).indices
        weights.scatter_(1, at, 0.1 + torch.rand(T, top, generator=g, device=dev))
    out0 = torch.randn(T, d, generator=g, device=dev)
    out = out0.clone()
    scratch = lambda name, shape, dtype: torch.full(shape, -1, dtype=dtype, device=dev)  # noqa: E731
    ops.experts(x, weights, ops.interleave_gate_up(gate, up), down, out, scratch, num_experts=E, top=top, expert_size=ff, shared_size=shared,
                overwrite=overwrite)
    torch.cuda.synchronize()
    ops.check_kernel_status()
    z = x.double() @ gate.double().T
    h = z * torch.sigmoid(z) * (x.double() @ up.double().T)
    h[:, :E * ff] *= weights[:, :E].double().repeat_interleave(ff, dim=1)
    ref = h @ down.double().T + (0 if overwrite else out0.double())
    # the hidden values are rounded to bfloat16 once (half of 2^-8), activation and sums are float32
    bound = (2.0 ** -9 + 1e-4) * (h.abs() @ down.double().abs().T) + 1e-6 * (1 + ref.abs())
    assert bool(((out.double() - ref).abs() <= bound).all())


@pytest.mark.gpu
def test_more_choices_than_announced_are_reported():
    from llmplayer_b200.errors import LLMPlayerError
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    T, E, d = 300, 8, 64
    x = torch.randn(T, d, device=dev).to(torch.bfloat16)
    w = torch.randn(E * 128, d, device=dev).to(torch.bfloat16)
    scratch = lambda name, shape, dtype: torch.zeros(shape, dtype=dtype, device=dev)  # noqa: E731
    ops.experts(x, torch.ones(T, E, device=dev), ops.interleave_gate_up(w, w), w.T.contiguous(), torch.zeros(T, d, device=dev), scratch,
                num_experts=E, top=1, expert_size=128)
    with pytest.raises(LLMPlayerError):
        ops.check_kernel_status()
    ops.check_kernel_status()                # said once


@pytest.mark.gpu
@pytest.mark.parametrize("scoring,shared,identity", [("sigmoid_groups", 128, 0), ("softmax_groups", 0, 4)])
@pytest.mark.parametrize("overwrite", [False, True])
def test_mixture_of_many_tokens(scoring, shared, identity, overwrite):
    """The part takes the grouped products from a number of tokens on; both ways against float64."""
    from llmplayer_b200.engine.step import StepContext, Workspace
    from llmplayer_b200.kernels import ops
    from llmplayer_b200.parts import FEED_FORWARDS
    from llmplayer_b200.parts.base import Runtime
    from llmplayer_b200.parts.specs import ExpertRoutingSpec, MixtureSpec
    d, ff, E, top = 1024, 512, 8, 2
    routing = ExpertRoutingSpec(E, top, 4, 2, "router", scoring=scoring, identity_experts=identity, correction="c" if identity else None)
    part = FEED_FORWARDS.build(MixtureSpec(d, ff, routing, "", shared_size=shared, shared_prefix="s." if shared else None))
    g = torch.Generator().manual_seed(shared + 5)
    w = {n: (torch.randn(*s.shape, generator=g) * s.shape[-1] ** -0.5 * (0.1 if n == "c" else 1.0)).to(torch.bfloat16)
         for n, s in part.tensor_specs().items()}
    part.load(w, Runtime(torch.device("cuda:0")))
    w = {n: t.double().cuda() for n, t in w.items()}
    for T in (130, 520):
        assert part.grouped and ops.experts_grouped_pays(T, d, E, top, ff) == (T == 520)
        x = torch.randn(T, d, generator=g).to(torch.bfloat16).cuda()
        out0 = torch.randn(T, d, generator=g).cuda()
        out = out0.clone()
        part.forward(StepContext(Workspace("cuda:0"), [], [0] * T, [], []), x, out, overwrite=overwrite)
        h = x.double()
        z = h @ w["router"].T
        n, per = E + identity, (E + identity) // 4
        scores = torch.sigmoid(z) if scoring == "sigmoid_groups" else torch.softmax(z, -1)
        choice = scores + (w["c"] if identity else 0.0)
        groups = choice.reshape(T, 4, per)
        best = (groups.topk(2, -1).values.sum(-1) if not identity else groups.max(-1).values).topk(2, -1).indices
        opened = torch.zeros(T, 4, dtype=torch.bool, device="cuda").scatter_(1, best, True).repeat_interleave(per, 1)
        at = choice.masked_fill(~opened, -1e9).topk(top, -1).indices
        weights = torch.zeros(T, n, dtype=torch.float64, device="cuda").scatter_(1, at, scores.gather(1, at))
        if not identity:
            weights = weights / weights.sum(-1, keepdim=True)
        run = lambda p: (torch.nn.functional.silu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T  # noqa: E731
        ref = sum(weights[:, e, None] * run(f"e{e}.") for e in range(E)) + (run("s.") if shared else 0)
        ref = ref + weights[:, E:].sum(-1, keepdim=True) * h + (0 if overwrite else out0.double())
        # hidden values rounded to bfloat16 (twice where the weight is applied behind the rounding): 2^-8 of the sum's parts, which
        # the float64 run shows to stay within 2e-2 of the largest output; a token whose choice is closer than float32 may differ
        off = ((out.double() - ref).abs().max(-1).values > 2e-2 * float(ref.abs().max()))
        assert int(off.sum()) <= 1, int(off.sum())


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,top,ff,shared,d", [(1025, 16, 4, 128, 128, 1032), (2048, 8, 3, 256, 0, 264)])
@pytest.mark.parametrize("overwrite", [False, True])
def test_the_same_inputs_give_the_same_bits(T, E, top, ff, shared, d, overwrite, monkeypatch):
    """However the tiles finish, and in however many slices of columns the results are held."""
    from llmplayer_b200.kernels import ops
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(T)
    x = torch.randn(T, d, generator=g, device=dev).to(torch.bfloat16)
    total = E * ff + shared
    gate, up = ((torch.randn(total, d, generator=g, device=dev) / d ** 0.5).to(torch.bfloat16) for _ in range(2))
    w_up, w_down = ops.interleave_gate_up(gate, up), torch.randn(d, total, generator=g, device=dev).to(torch.bfloat16)
    weights = torch.zeros(T, E, device=dev)
    weights.scatter_(1, torch.rand(T, E, generator=g, device=dev).topk(top, dim=1).indices, 0.1 + torch.rand(T, top, generator=g, device=dev))
    out0 = torch.randn(T, d, generator=g, device=dev)
    scratch = lambda name, shape, dtype: torch.full(shape, -1, dtype=dtype, device=dev)  # noqa: E731
    first = None
    for room in (ops.EXPERTS_RESULT_BYTES,) * 6 + (1, 4 * ops.expert_rows(T, E, top, False) * 512):      # slices of 256, of 512
        monkeypatch.setattr(ops, "EXPERTS_RESULT_BYTES", room)
        out = out0.clone()
        ops.experts(x, weights, w_up, w_down, out, scratch, num_experts=E, top=top, expert_size=ff, shared_size=shared, overwrite=overwrite)
        first = out if first is None else first
        assert torch.equal(out, first), room
    ops.check_kernel_status()


@pytest.mark.gpu
@pytest.mark.parametrize("T,d", [(520, 1024), (1300, 2048)])
def test_a_routed_layer_gives_the_same_bits(T, d):
    from llmplayer_b200.engine.step import StepContext, Workspace
    from llmplayer_b200.kernels import ops
    from llmplayer_b200.parts import FEED_FORWARDS
    from llmplayer_b200.parts.base import Runtime
    from llmplayer_b200.parts.specs import ExpertRoutingSpec, MixtureSpec
    part = FEED_FORWARDS.build(MixtureSpec(d, 512, ExpertRoutingSpec(8, 2, 4, 2, "router"), "", shared_size=128, shared_prefix="s."))
    g = torch.Generator().manual_seed(T)
    part.load({n: (torch.randn(*s.shape, generator=g) * s.shape[-1] ** -0.5).to(torch.bfloat16) for n, s in part.tensor_specs().items()},
              Runtime(torch.device("cuda:0")))
    x = torch.randn(T, d, generator=g).to(torch.bfloat16).cuda()
    out0 = torch.randn(T, d, generator=g).cuda()
    ctx = StepContext(Workspace("cuda:0"), [], [0] * T, [], [])
    assert ops.experts_grouped_pays(T, d, 8, 2, 512) and part.buffer_to_clear(ctx, T) is None
    outs = []
    for _ in range(8):
        outs.append(out0.clone())
        part.forward(ctx, x, outs[-1])
        assert torch.equal(outs[-1], outs[0])


@pytest.mark.parametrize("T,E,top,ff,shared,d", [(2048, 32, 4, 512, 8192, 2048), (4096, 64, 8, 256, 0, 7168), (600, 8, 2, 2048, 128, 1024)])
def test_scratch_follows_each_experts_own_size(T, E, top, ff, shared, d, monkeypatch):
    """Hidden values of a routed row at the routed size and of a token at the shared one, the gathered rows and their results in one
    place, results never beyond their room."""
    from llmplayer_b200.kernels import ops
    launched = []

    class Library:                                        # records the launch instead of making it
        def __getattr__(self, name):
            return lambda *args: launched.append(args) or 0

    monkeypatch.setattr(ops, "library", lambda name: Library())
    monkeypatch.setattr(ops, "kernel_status", lambda: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_want", lambda *args, **kw: None)
    taken = {}

    def scratch(name, shape, dtype):
        taken[name] = torch.empty(shape, dtype=dtype, device="meta").numel() * dtype.itemsize
        return torch.empty(1, dtype=dtype)

    empty = lambda *shape, dtype=torch.bfloat16: torch.empty(shape, dtype=dtype, device="meta")  # noqa: E731
    total = E * ff + shared
    ops.experts(empty(T, d), empty(T, E, dtype=torch.float32), empty(2 * total, d), empty(d, total), empty(T, d, dtype=torch.float32), scratch,
                num_experts=E, top=top, expert_size=ff, shared_size=shared)
    rows = ops.expert_rows(T, E, top, False)
    assert len(launched) == 1
    assert taken["expert_hidden"] == 2 * (rows * ff + T * shared)
    assert taken["expert_rows"] == max(2 * rows * d, min(4 * rows * d, 4 * rows * max(256, (256 << 20) // (4 * rows) // 256 * 256)))
    assert sum(n for name, n in taken.items() if name not in ("expert_hidden", "expert_rows")) <= 8 * rows + 8 * T * E + 4 * E
