"""Which form the product of many tokens takes, that its callers clear an output exactly where it adds partial sums, and the
narrow products themselves."""
import pytest
import torch


def test_few_tiles_share_k_out_and_callers_know(monkeypatch):
    from llmplayer_b200.kernels import ops
    from llmplayer_b200.parts.linear import Linear
    monkeypatch.setattr(ops, "_num_sms", 148)
    launched = []

    class Library:                                        # records the launch instead of making it
        def __getattr__(self, name):
            return lambda *args: launched.append((name, args)) or 0

    monkeypatch.setattr(ops, "library", lambda name: Library())
    monkeypatch.setattr(ops, "kernel_status", lambda: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(ops, "_want", lambda *args, **kw: None)
    monkeypatch.setattr(ops, "_out_matrix", lambda t, what: (t.data_ptr(), t.shape[1]))
    forms = set()
    for T in (1, 65, 511, 512, 600, 1024, 2048, 5000):
        for N in (8, 40, 128, 300, 1024, 2056):
            for K in (64, 1024, 2048, 4096):
                a, w, out = torch.empty(T, K, dtype=torch.bfloat16), torch.empty(N, K, dtype=torch.bfloat16), torch.ones(T, N)
                linear = Linear.__new__(Linear)
                linear.weight, linear.out_features, linear.in_features = w, N, K
                linear._fast = lambda: True
                ops.gemm(a, w, out, ops.STORE)
                name, args = launched.pop()
                persistent = name == "lp_gemm_persistent"
                tiles = -(-N // 128) * -(-T // 256)
                assert not (persistent and tiles * 4 <= 148), (T, N, K)
                # an output that nobody cleared: cleared here if partial sums (more than one split) are added into it
                assert bool((out == 0).all()) == (not persistent and args[12] > 1), (T, N, K)
                ops.gemm(a, w, out, ops.STORE, cleared=True)
                name, args = launched.pop()
                adds = name != "lp_gemm_persistent" and args[12] > 1
                assert linear.needs_zero(T) == adds, (T, N, K)
                assert not adds or T < 512 or K > ops.ORDERED_MAX_K, (T, N, K)
                forms.add((persistent, adds))
                ops.gemm(a, w, out, ops.ACCUMULATE)
                assert not (launched.pop()[0] == "lp_gemm_persistent" and tiles * 4 <= 148), (T, N, K)
    assert forms == {(True, False), (False, True), (False, False)}


@pytest.mark.gpu
@pytest.mark.parametrize("N", [8, 40, 128, 264])
@pytest.mark.parametrize("T,K", [(600, 2048), (2049, 1032), (512, 520)])
@pytest.mark.parametrize("mode", ["store", "accumulate"])
def test_narrow_products_of_many_tokens(N, T, K, mode):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device="cuda:0").manual_seed(N + T)
    a = torch.randn(T, K, generator=g, device="cuda:0").to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device="cuda:0") / K ** 0.5).to(torch.bfloat16)
    out0 = torch.randn(T, N, generator=g, device="cuda:0")
    ref = a.double() @ w.double().T
    # float32 sums of K exact products: K units of 2^-24 of the sum of magnitudes
    bound = 2.0 ** -24 * K * float((a.double().abs() @ w.double().abs().T).max())
    out = out0.clone()
    if mode == "accumulate":
        ops.gemm(a, w, out, ops.ACCUMULATE)
        assert float((out.double() - ref - out0.double()).abs().max()) <= bound
        return
    ops.gemm(a, w, out)
    assert float((out.double() - ref).abs().max()) <= bound
    if ops.gemm_adds_parts(T, N, K):                      # the kernel in front has cleared the output
        cleared = torch.zeros_like(out)
        ops.gemm(a, w, cleared, cleared=True)
        assert float((cleared.double() - ref).abs().max()) <= bound
    half = out0.to(torch.bfloat16)
    ops.gemm(a, w, half)
    assert float((half.double() - ref).abs().max()) <= bound + 2.0 ** -8 * float(ref.abs().max())
    ops.check_kernel_status()
