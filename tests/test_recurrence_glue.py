"""What stands around the recurrences of prompts, at the edges of its tiles, and the chunked recurrence with three, two and one
record in flight, each against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(got, ref):
    return float((got.double() - ref).abs().max() / ref.abs().max())


@pytest.mark.parametrize("T,C,R", [(1, 24, 5), (33, 256, 16), (1185, 1024, 16), (2047, 600, 37), (4800, 8, 3)])
@pytest.mark.parametrize("tanh", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_decays(T, C, R, tanh, dtype):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    wide = torch.randn(T, R + 3, generator=g, device=DEV)
    up = (torch.randn(C, R, generator=g, device=DEV) / R ** 0.5).to(dtype)
    bias = torch.randn(C, generator=g, device=DEV)
    out = torch.full((T, C), 7.0, device=DEV)
    ops.gla_decay(wide[:, 2:2 + R], up, bias, out, 16.0, double_exp=tanh)
    low = wide[:, 2:2 + R].double()
    z = (torch.tanh(low) if tanh else low) @ up.double().T + bias.double()
    ref = torch.exp(-torch.exp(z)) if tanh else torch.sigmoid(z) ** (1 / 16.0)
    assert rel(out, ref) < 2e-6


@pytest.mark.parametrize("T,H,dk,ra,dv,rg", [(17, 1, 16, 16, 8, 16), (64, 2, 40, 48, 129, 32), (129, 8, 128, 128, 128, 128), (200, 3, 96, 256, 64, 16)])
def test_low_rank_gates(T, H, dk, ra, dv, rg):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T)
    for shift in (0, 1):                                  # columns that start on 16 bytes, and columns that do not
        proj = torch.randn(T, shift + ra + rg + H + (-(shift + ra + rg + H)) % 4, generator=g, device=DEV)
        a_up = (torch.randn(H * dk, ra, generator=g, device=DEV) / ra ** 0.5).to(torch.bfloat16)
        g_up = (torch.randn(H * dv, rg, generator=g, device=DEV) / rg ** 0.5).to(torch.bfloat16)
        dt, a_log = torch.randn(H * dk, generator=g, device=DEV), 0.3 * torch.randn(H, generator=g, device=DEV)
        decay, strength = torch.full((T, H * dk), 7.0, device=DEV), torch.full((T, H), 7.0, device=DEV)
        gate = torch.full((T, H * dv), 7.0, device=DEV)
        ops.low_rank_gates(proj, shift, a_up, dt, a_log, decay, shift + ra + rg, strength, key_dim=dk, g_off=shift + ra, g_up=g_up, gate=gate)
        p = proj.double()
        z = p[:, shift:shift + ra] @ a_up.double().T + dt.double()
        ref = torch.exp(-torch.exp(a_log.double()).repeat_interleave(dk) * torch.nn.functional.softplus(z))
        assert rel(decay, ref) < 3e-6
        assert rel(gate, p[:, shift + ra:shift + ra + rg] @ g_up.double().T) < 2e-6
        assert rel(strength, torch.sigmoid(p[:, shift + ra + rg:shift + ra + rg + H])) < 1e-6


@pytest.mark.parametrize("T,H,dv", [(1, 1, 4), (37, 3, 100), (65, 2, 128), (20, 5, 132), (9, 2, 256), (11, 3, 300), (7, 2, 512), (5, 2, 516), (6, 2, 30)])
@pytest.mark.parametrize("sigmoid,per_head", [(False, False), (True, True)])
def test_finish(T, H, dv, sigmoid, per_head):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(dv)
    raw, wide = torch.randn(T, H * dv, generator=g, device=DEV), torch.randn(T, H * dv + 4, generator=g, device=DEV)
    gain = torch.randn(H * dv if per_head else dv, generator=g, device=DEV)
    x = raw.double().reshape(T, H, dv)
    ref = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    ref = (ref * (gain.double().reshape(H, dv) if per_head else gain.double())).reshape(T, H * dv)
    for shift in (0, 3):
        gate = wide[:, shift:shift + H * dv]
        z = gate.double()
        want = ref * torch.sigmoid(z) * (1.0 if sigmoid else z)
        for dtype, lim in ((torch.float32, 1e-6), (torch.bfloat16, 5e-3)):
            out = torch.empty(T, H * dv, device=DEV, dtype=dtype)
            ops.gla_finish(raw, gain, 1e-5, gate, out, num_heads=H, value_dim=dv, gate_sigmoid=sigmoid,
                           gain_per_head=per_head)
            assert rel(out, want) < lim


@pytest.mark.parametrize("dk,dv", [(64, 48), (128, 40), (160, 16), (192, 16), (256, 24)])
@pytest.mark.parametrize("delta", [False, True])
def test_chunked_recurrence(dk, dv, delta):
    """Records of every size, so that three, two and one of them fit; sequences of several chunks, one, and a part of one."""
    from llmplayer_b200.kernels import ops
    H, lengths = 2, [300, 32, 5, 97]
    g = torch.Generator(device=DEV).manual_seed(dk + dv)
    T = sum(lengths)
    k = torch.randn(T, H, dk, generator=g, device=DEV)
    k = k / k.norm(dim=-1, keepdim=True)
    q, v = torch.randn(T, H, dk, generator=g, device=DEV), torch.randn(T, H, dv, generator=g, device=DEV)
    decay = 1.0 - 0.1 * torch.rand(T, H, dk, generator=g, device=DEV) ** 2
    beta = torch.rand(T, H, generator=g, device=DEV)
    proj = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1).contiguous()
    start = torch.randn(len(lengths) + 1, H, dv, dk, generator=g, device=DEV)
    state = start.clone()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    out = torch.empty(T, H * dv, device=DEV)
    scratch = lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device=DEV)  # noqa: E731
    at = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    ops.gla_scan(proj, 0, H * dk, 2 * H * dk, decay.reshape(T, -1).contiguous(), state, i32([3, 0, 4, 1]), i32(at), out, num_heads=H, key_dim=dk,
                 value_dim=dv, q_scale=0.5, max_new=max(lengths), scratch=scratch, delta_strength=beta if delta else None, tensor_cores=True)
    for i, (n, slot) in enumerate(zip(lengths, (3, 0, 4, 1))):
        S = start[slot].double()
        for t in range(at[i], at[i] + n):
            S = S * decay[t].double()[:, None, :]
            u = v[t].double()
            if delta:
                u = beta[t].double()[:, None] * (u - (S @ k[t].double()[:, :, None])[:, :, 0])
            S = S + u[:, :, None] * k[t].double()[:, None, :]
            o = (S @ q[t].double()[:, :, None])[:, :, 0] * 0.5
            assert float((out[t].double().reshape(H, dv) - o).abs().max()) < 2e-5 * float(o.abs().max() + 1), (i, t)
        assert rel(state[slot], S) < 1e-5
    assert torch.equal(state[2], start[2])


@pytest.mark.parametrize("dk", [20, 64, 100, 128, 160])
@pytest.mark.parametrize("form", ["channel", "head", "fixed"])
def test_chunked_recurrence_reads(dk, form):
    """Rows read four channels at a time and rows whose slices start at an odd column: the same arithmetic, bit for bit."""
    from llmplayer_b200.kernels import ops
    H, dv, lengths = 2, 24, [70, 33, 3]
    g = torch.Generator(device=DEV).manual_seed(dk)
    T = sum(lengths)
    wide = torch.randn(T, H * (2 * dk + dv), generator=g, device=DEV) * dk ** -0.5
    odd = torch.cat([torch.full((T, 1), float("nan"), device=DEV), wide], dim=1).contiguous()
    shape = {"channel": (T, H * dk), "head": (T, H), "fixed": (H,)}[form]
    decay = 1.0 - 0.1 * torch.rand(*shape, generator=g, device=DEV)
    gain, beta = torch.rand(T, H, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    start = torch.randn(len(lengths), H, dv, dk, generator=g, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    at = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    scratch = lambda name, shape, dtype: torch.full(shape, float("nan"), dtype=dtype, device=DEV)  # noqa: E731
    results = []
    for proj, off in ((wide, 0), (odd, 1)):
        state, out = start.clone(), torch.empty(T, H * dv, device=DEV)
        ops.gla_scan(proj, off, off + H * dk, off + 2 * H * dk, decay, state, i32([2, 0, 1]), i32(at), out, num_heads=H, key_dim=dk,
                     value_dim=dv, q_scale=0.5, max_new=max(lengths), scratch=scratch, delta_strength=beta, key_gain=gain,
                     decay_per_head=form == "head", decay_fixed=form == "fixed", tensor_cores=True)
        results.append((out, state))
    assert torch.isfinite(results[0][0]).all()
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
