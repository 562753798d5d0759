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


def test_second_kernels_read_what_the_first_ones_wrote():
    """Calls of two and three launches (K parts and their sum, ordered weight gradients, row statistics and the loss), each on buffers
    that the call before it has read or written."""
    from kareus_b200.kernels import cuda as KC, replay
    import kareus_b200.kernels as K
    g = torch.Generator(device="cuda").manual_seed(7)
    draw = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, up, down, head = draw(4096, 3072), draw(5120, 3072) / 55, draw(3072, 5120) / 72, draw(3000, 3072) / 55
    tgt = torch.randint(0, 3000, (4096,), device="cuda", generator=g)
    weight = torch.rand(4096, device="cuda", generator=g)
    wide, back = torch.empty(4096, 5120, device="cuda", dtype=torch.bfloat16), torch.empty(4096, 3072, device="cuda", dtype=torch.bfloat16)
    dw = torch.zeros(5120, 3072, device="cuda")

    def body(wait=lambda: None):
        y, outs = x, []
        for _ in range(3):
            KC.gemm(y, up, out=wide)
            wait()
            KC.gemm(wide, down, out=back)
            wait()
            K.gemm(wide, back, trans_a=True, trans_b=False, accumulate=dw)
            wait()
            _, m, se, tl, loss = K.linear_cross_entropy_stats(back, head, tgt, 0, store=False, weight=weight)
            wait()
            logits, *_, again = K.linear_cross_entropy_stats(back, head, tgt, 0, weight=weight)
            wait()
            outs += [m, se, tl, loss, again, logits]
            y = KC.add(back, y)
            wait()
        return outs + [dw, y]

    try:
        KC.lib().kb_gemm_parts_force(3, 128)
        assert KC.lib().kb_gemm_scratch_floats(4096, 5120, 3072, 0, 0) > 0
        assert KC.lib().kb_gemm_accum_scratch_floats(5120, 3072, 4096, 0) > 0
        want = [t.clone() for t in body(torch.cuda.synchronize)]
        with replay.Recording() as r:
            recorded = body()
        for _ in range(10):
            dw.zero_()
            for a, b in zip(body(), want, strict=True):
                assert torch.equal(a, b)
            dw.zero_()
            r.result.replay()
            for a, b in zip(recorded, want, strict=True):
                assert torch.equal(a, b)
    finally:
        KC.lib().kb_gemm_parts_force(0, 0)
    assert r.result.is_graph
    torch.cuda.synchronize()
    KC.check_status()
    r.result.free()
