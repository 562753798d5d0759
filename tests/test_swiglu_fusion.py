"""fc1, SwiGLU and fc2 of a layer as one fusion chain: the activation in the epilogues of the GEMMs beside it gives what the three
operators give, in a chain that is whole, and only there."""
import pytest
import torch

import kareus_b200.kernels as K
from kareus_b200.config import ParallelConfig, get_model_config
from kareus_b200.engine.block import BlockEngine
from kareus_b200.engine.context import OpContext
from kareus_b200.engine.graph import GraphOperator
from kareus_b200.kernels import ref
from kareus_b200.models.llama import GPTModel, TransformerLayer
from kareus_b200.ops.basic import SwiGLUOp
from kareus_b200.ops.extras import BiasOp
from kareus_b200.parallel.collectives import CommFactory


@pytest.fixture
def stand_in(monkeypatch):
    """Fused calls on the CPU, stated in PyTorch; returns how often each was taken."""
    taken = {"forward": 0, "saving": 0, "backward": 0}

    def install(forward=True, backward=True):
        def fwd(x, w, store=True):
            if not forward:
                return None
            taken["forward"] += 1
            taken["saving"] += store
            y = ref.gemm(x, w, False, True, None, None)
            return (y if store else None), ref.swiglu_fwd(y)

        def bwd(dy, w, x):
            if not backward:
                return None
            taken["backward"] += 1
            return ref.swiglu_bwd(ref.gemm(dy, w, False, False, None, None), x)
        monkeypatch.setattr(K, "linear_swiglu", fwd)
        monkeypatch.setattr(K, "linear_swiglu_dgrad", bwd)
        return taken
    return install


def _grads(model, batch):
    model(*batch).backward()
    return [p.main_grad.clone() for p in model.parameters()]


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("backward", [False, True])
def test_whole_chains_fuse(stand_in, recompute, backward):
    cfg = get_model_config("tiny")
    g = torch.Generator().manual_seed(0)
    tokens, labels = (torch.randint(0, cfg.vocab_size, (4, 32), generator=g) for _ in range(2))
    batch = tokens, labels, torch.ones(4, 32)
    par = ParallelConfig(num_nanobatches=2, recompute=recompute)
    want = _grads(GPTModel(cfg, par, dtype="fp64"), batch)
    taken = stand_in(backward=backward)
    got = _grads(GPTModel(cfg, par, dtype="fp64"), batch)
    calls = 2 * cfg.num_layers
    assert taken == {"forward": calls * (2 if recompute else 1), "saving": calls, "backward": calls if backward else 0}
    for a, b in zip(got, want, strict=True):
        torch.testing.assert_close(a, b, rtol=1e-12, atol=1e-15)
    with torch.no_grad():
        n = taken["saving"]
        GPTModel(cfg, par, dtype="fp64")(*batch)
        assert taken["saving"] == n                       # nothing is kept for a backward pass that does not come


class _Doubled(SwiGLUOp):
    """Another activation in the place of the layer's own."""

    def forward(self, ctx, x):
        (y,) = super().forward(ctx, x)
        return (2 * y,)

    def backward(self, ctx, dy):
        return super().backward(ctx, 2 * dy)


class _Square(GraphOperator):
    group = "activation"
    name = "square"

    def forward(self, ctx, x):
        ctx.save_for_backward(x)
        return (x[..., :x.shape[-1] // 2] * x[..., x.shape[-1] // 2:],)

    def backward(self, ctx, dy):
        a, b = ctx.saved_tensors[0].chunk(2, -1)
        return (torch.cat([dy * b, dy * a], -1),)


@pytest.mark.parametrize("form", ["bias", "subclass", "replaced"])
def test_anything_else_in_the_chain_gets_the_product(stand_in, form):
    cfg = get_model_config("tiny")

    def run():
        layer = TransformerLayer(cfg, ParallelConfig(), CommFactory(), 0, torch.float64, "cpu", seed=3)
        ops = layer.operators()
        i = ops.index(layer.fc1)
        if form == "bias":
            b = BiasOp(2 * cfg.ffn_hidden_size, dtype=torch.float64)
            b.bias.data.normal_(generator=torch.Generator().manual_seed(4))
            ops.insert(i + 1, b)
        else:
            ops[i + 1] = _Doubled() if form == "subclass" else _Square()
        engine = BlockEngine([ops], 1, recompute=False)
        x = torch.randn(16, 2, cfg.hidden_size, dtype=torch.float64, generator=torch.Generator().manual_seed(5)).requires_grad_()
        (y,) = engine([x], ref.rope_table(16, cfg.hd, cfg.rope_theta, device="cpu"))
        y.square().sum().backward()
        return [y.detach(), x.grad, layer.fc1.weight.main_grad, layer.fc2.weight.main_grad]

    want = run()
    taken = stand_in()
    for a, b in zip(run(), want, strict=True):
        torch.testing.assert_close(a, b, rtol=1e-12, atol=1e-15)
    assert taken["forward"] == taken["backward"] == 0


def test_an_operator_alone_returns_its_product(stand_in):
    cfg = get_model_config("tiny")
    stand_in()
    layer = TransformerLayer(cfg, ParallelConfig(), CommFactory(), 0, torch.float64, "cpu", seed=3)
    x = torch.randn(8, cfg.hidden_size, dtype=torch.float64)
    (y,) = layer.fc1.forward(OpContext(), x)
    torch.testing.assert_close(y, x @ layer.fc1.weight.t())
    (h,) = layer.act.forward(OpContext(), y)
    torch.testing.assert_close(h, ref.swiglu_fwd(y))
    narrow = layer.act.forward(OpContext(), h)[0]          # a [gate | up] input of any width is one
    torch.testing.assert_close(narrow, ref.swiglu_fwd(h))


# ----------------------------------------------------------------------------- the rule and its callers
def _library():
    import ctypes
    from kareus_b200.kernels import build
    if not build.LIB.exists():
        pytest.skip("native library not built")
    return ctypes.CDLL(str(build.LIB))


def test_passes_with_and_without_a_product_take_the_same_kernels(monkeypatch):
    """A recomputing step runs a layer once without keeping fc1's product and once with it: the second activation has to be the first."""
    from kareus_b200.kernels import cuda as KC
    real = _library()

    class Lib:
        kb_gemm_swiglu_pays = staticmethod(real.kb_gemm_swiglu_pays)
        kb_gemm_swiglu = staticmethod(lambda *a: 0)
    monkeypatch.setattr(KC, "lib", lambda: Lib)
    monkeypatch.setattr(KC, "_stream", lambda: 0)
    monkeypatch.setattr(KC, "status_word", lambda dev: torch.zeros(1, dtype=torch.int32))
    answers = set()
    for h, f in [(512, 1024), (2048, 3072), (3072, 4096), (3072, 8192)]:
        w = torch.empty(2 * f, h, dtype=torch.bfloat16)
        for tokens in list(range(64, 1024, 32)) + [1728, 2016, 2560, 4096]:
            x = torch.empty(tokens, h, dtype=torch.bfloat16)
            with_, without = (KC.linear_swiglu(x, w, store) is None for store in (True, False))
            assert with_ == without, (tokens, h, f)
            answers.add(with_)
    assert answers == {True, False}


@pytest.mark.parametrize("backward,tokens,h,f,fused", [
    # us of two kernels / one: 13 / 17, 18 / 22, 28 / 23, 21 / 18, 101 / 73, 866 / 590
    (0, 157, 2048, 1536, 0), (0, 316, 3072, 2048, 0), (0, 427, 3072, 4096, 1), (0, 1237, 2048, 1536, 1), (0, 3798, 2048, 3072, 1),
    (0, 16646, 2048, 6144, 1),
    # 13 / 14, 13 / 14, 36 / 38, 52 / 58; a short last wave that the product alone has in K parts 128 / 135, 114 / 120
    (1, 148, 2048, 3072, 0), (1, 357, 2048, 1536, 0), (1, 4074, 2048, 1536, 0), (1, 16806, 512, 1024, 0), (1, 904, 4096, 14336, 0),
    (1, 900, 4096, 14336, 0),
    # 127 / 114, 516 / 390, 216 / 173
    (1, 7784, 2048, 3072, 1), (1, 16646, 2048, 6144, 1), (1, 6703, 2048, 6144, 1)])
def test_epilogue_is_taken_where_it_is_faster_than_the_route_beside_it(backward, tokens, h, f, fused):
    assert _library().kb_gemm_swiglu_pays(tokens, f, h, backward) == fused


# ----------------------------------------------------------------------------- the kernels
@pytest.fixture
def force():
    from kareus_b200.kernels import cuda as KC
    yield lambda how: KC.lib().kb_gemm_swiglu_force(how)       # 1 everywhere, 2 forward only, 3 nowhere
    KC.lib().kb_gemm_swiglu_force(0)


def _steps(recompute, replay, seq=192, steps=3):
    """Losses of some steps and the gradients of the last, on weights that no step changes."""
    from kareus_b200.config import TrainConfig
    from kareus_b200.kernels import cuda as KC
    from kareus_b200.train.trainer import Trainer, synthetic_batch
    cfg = get_model_config("tiny128")
    tc = TrainConfig(micro_batch_size=2, global_batch_size=2, seq_len=seq, warmup_steps=0, lr=0.0, min_lr=0.0, seed=1)
    tr = Trainer(cfg, ParallelConfig(num_nanobatches=2, recompute=recompute), tc, device="cuda")
    tr.model.decoder.engine.replay = replay
    batch = synthetic_batch(cfg, tc, tr.num_microbatches, seed=2)
    losses = [tr.train_step(batch) for _ in range(steps)]
    torch.cuda.synchronize()
    KC.check_status()
    if recompute and replay:
        assert tr.model.decoder.engine.replayed_regions > 0
    return losses, tr.optimizer.grad_flat.double()


@pytest.mark.gpu
@pytest.mark.parametrize("recompute,replay", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("how", [1, 2])
def test_a_step_with_the_fusion_is_the_step_without(force, monkeypatch, how, recompute, replay):
    force(3)
    want_loss, want = _steps(recompute, replay)
    taken = []
    real = K.linear_swiglu_dgrad
    monkeypatch.setattr(K, "linear_swiglu_dgrad", lambda *a: (lambda r: (taken.append(r is not None), r)[1])(real(*a)))
    force(how)
    loss, grads = _steps(recompute, replay)
    # every backward pass of fc2 had fc1's product at hand, and used it or left it to the SwiGLU operator
    assert taken and all(t == (how == 1) for t in taken)
    # a different order of sums moves roundings to bf16 (2^-9) of two layers: well under a percent of a gradient's norm
    assert all(abs(a - b) < 5e-3 for a, b in zip(loss, want_loss, strict=True))
    assert (grads - want).norm() < 1e-2 * want.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("how", [0, 1])
@pytest.mark.parametrize("tokens,h,f", [(130, 512, 1024), (200, 3072, 8192), (400, 3072, 4096), (600, 2048, 3072), (2016, 512, 1024)])
def test_recomputed_activation_is_the_one_of_the_forward_pass(force, how, tokens, h, f):
    force(how)
    layer = TransformerLayer(get_model_config("tiny128").replace(hidden_size=h, ffn_hidden_size=f), ParallelConfig(), CommFactory(), 0,
                             torch.bfloat16, "cuda", seed=3)
    x = torch.randn(tokens, h, device="cuda").bfloat16()
    outs = []
    for saving in (False, True):
        ctxs = [OpContext() for _ in range(3)]
        y = x
        for c, op in zip(ctxs, (layer.fc1, layer.act, layer.fc2)):
            c.requires_grad, c.chained = saving, True
            (y,) = op.forward(c, y)
            outs.append(y)
    torch.cuda.synchronize()
    assert torch.equal(outs[1], outs[4]) and torch.equal(outs[2], outs[5])
