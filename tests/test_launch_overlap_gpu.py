"""Kernels that start under the end of the one before them read and write memory in stream order."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(rows, sync):
    """Operators that feed one another; the GEMMs overwrite the buffer that the kernel just before them read."""
    from kareus_b200.kernels import cuda as KC
    g = torch.Generator(device="cuda").manual_seed(rows)
    draw = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, up, down, ln = draw(rows, 512), draw(1024, 512) / 16, draw(512, 512) / 16, draw(512)
    wide = torch.empty(rows, 1024, device="cuda", dtype=torch.bfloat16)
    qkv = torch.empty(rows, 1, 4, 128, device="cuda", dtype=torch.bfloat16)
    dw = torch.zeros(1024, 512, device="cuda")
    wait = torch.cuda.synchronize if sync else (lambda: None)

    def body():
        y = x
        for _ in range(4):
            n, rstd = KC.rmsnorm_fwd(y, ln, 1e-5)
            wait()
            KC.gemm(n, up, out=wide)
            wait()
            h = KC.swiglu_fwd(wide)
            wait()
            KC.gemm(h, down, out=qkv.view(rows, 512))
            wait()
            o, _ = KC.attention_fwd(qkv[:, :, :2].unsqueeze(2), qkv[:, :, 2:3], qkv[:, :, 3:], 1 / math.sqrt(128))
            wait()
            KC.gemm(n, up, out=wide)
            wait()
            KC.gemm(wide, n, trans_a=True, trans_b=False, accumulate=dw)
            wait()
            y = KC.add(qkv.view(rows, 512), y)
            wait()
        return [y, o, dw]

    return body, dw


# weight gradients over more than 960 rows may be split into parts that add in any order
@pytest.mark.parametrize("rows", [1, 130, 900])
def test_chains_give_the_results_of_waiting_after_each_kernel(rows):
    from kareus_b200.kernels import cuda as KC, replay
    body, dw = _chain(rows, sync=True)
    want = [t.clone() for t in body()]
    body, dw = _chain(rows, sync=False)
    with replay.Recording() as r:
        outs = body()
    for _ in range(20):
        dw.zero_()
        for a, b in zip(body(), want):
            assert torch.equal(a, b)
        dw.zero_()
        r.result.replay()
        for a, b in zip(outs, want):
            assert torch.equal(a, b)
    assert r.result.is_graph
    torch.cuda.synchronize()
    KC.check_status()
    r.result.free()
