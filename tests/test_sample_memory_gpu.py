"""Device memory of the gradient and score calls: what a large call needs beyond
64 MiB is given back when it returns, a small call's stays, and a readback's
buffer is left alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("call", ["gradient", "score"])
def test_large_calls_give_back(call):
    from oracle import mlp as omlp
    from sdl_gb300 import Chain, build
    build.build()
    ch = Chain(0)
    ch.mlp_set_params(omlp.init_params(5), 0.0)

    def run(n):
        x = np.full((n, omlp.N_IN), 0.25, dtype=np.float32)
        if call == "score":
            return ch.mlp_score(x)
        return ch.mlp_gradient(x, np.ones(n, dtype=np.float32), np.ones(n, dtype=np.float32))[0]

    small = run(1000)
    before = free_bytes()
    large = run(4_000_000)  # 208 or 224 MB
    assert free_bytes() >= before - 8 * MIB
    assert np.all(np.isfinite(large))
    assert np.allclose(run(1000), small, rtol=1e-5, atol=0)
    run(500_000)  # 26 or 28 MB and a quarter: kept
    kept = free_bytes()
    assert kept < before - 16 * MIB
    run(500_000)
    assert free_bytes() == kept
