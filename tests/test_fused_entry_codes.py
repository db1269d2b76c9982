"""What an entry of fused work returns: "not served" sends the call to the separate kernels, a failed launch (a positive
code) or a refusal raises and runs nothing else, above all no second sum into the stream. On the CPU, with a library that only answers."""
import os
import re

import pytest
import torch

from llmplayer_b200.errors import KernelError
from llmplayer_b200.kernels import build, ops


class Answers:
    """A library whose fused entries return ``code`` and whose other entries succeed; keeps the names called."""

    def __init__(self, code):
        self.code, self.called = code, []

    def __getattr__(self, name):
        def entry(*args):
            self.called.append(name)
            return self.code if name in ("lp_gated_sum_norm", "lp_latent_queries") else 0
        return entry

    def lp_last_error(self):
        return b"said by the library"


@pytest.fixture
def answers(monkeypatch):
    def install(code):
        lib = Answers(code)
        monkeypatch.setattr(ops, "library", lambda name: lib)
        monkeypatch.setattr(ops, "_want", lambda t, *a, **k: t)
        monkeypatch.setattr(ops, "_stream", lambda: 0)
        return lib
    return install


def sum_and_norm():
    x = torch.zeros(2, 8)
    ops.gated_sum(x, x.clone(), norm_after=(torch.ones(8), 1e-5, torch.empty(2, 8)))


def queries():
    i32 = torch.zeros(2, dtype=torch.int32)
    buffer = lambda name, shape, dtype: torch.empty(shape, dtype=dtype)  # noqa: E731
    ops.latent_queries(torch.zeros(2, 32), 0, 24, torch.ones(4), 1e-5, ops.Rotation(), i32, i32, i32.view(2, 1), torch.zeros(1, 32, 8),
                       torch.zeros(8, 4), torch.zeros(2, 2, 8), buffer, num_heads=2, nope_dim=4, rope_dim=4, kv_rank=4)


@pytest.mark.parametrize("call,separate", [(sum_and_norm, ["lp_gated_sum", "lp_layernorm"]), (queries, ["lp_latent_prepare", "lp_latent_absorb"])])
def test_codes(answers, call, separate):
    served = answers(0)
    call()
    assert len(served.called) == 1
    lib = answers(ops.NOT_SERVED)
    call()
    assert lib.called[1:] == separate
    for code in (1, 719, -1):             # cudaErrorInvalidValue, cudaErrorLaunchFailure, a refusal
        lib = answers(code)
        with pytest.raises(KernelError, match="said by the library"):
            call()
        assert len(lib.called) == 1


def test_not_served_is_no_cuda_error_and_no_refusal():
    with open(os.path.join(build.CSRC, "common.cuh")) as fh:
        code = int(re.search(r"#define LP_NOT_SERVED \((-?\d+)\)", fh.read()).group(1))
    assert code == ops.NOT_SERVED and code < -1
