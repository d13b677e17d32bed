"""The native one-call passes of the single-GPU models against the op-by-op Python methods."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_native_passes_match_the_op_by_op_path():
    """The one-call native passes launch what the Python methods launch: the same bits, also when a
    split weight gradient needs its workspace and when a weight is a strided view (op-by-op path)."""
    from megray_b200.models import MoEConfig, MoELayer, TPMLPConfig, TPMLPStack

    for cfg in (TPMLPConfig(d_model=256, ffn=384, layers=2, tokens=128, lr=1e-2),
                TPMLPConfig(d_model=768, ffn=256, layers=1, tokens=8192, lr=1e-2)):
        x = torch.randn(cfg.tokens, cfg.d_model, device="cuda").to(torch.bfloat16)
        a, b = TPMLPStack(cfg), TPMLPStack(cfg)
        assert a._native_args() is not None
        b._native_args = lambda: None
        ya, yb = a.forward(x).clone(), b.forward(x).clone()
        dy = torch.randn_like(ya)
        assert torch.equal(ya, yb) and torch.equal(a.backward(dy), b.backward(dy))
        for la, lb in zip(a.layers, b.layers):
            assert torch.equal(la.g_gu, lb.g_gu) and torch.equal(la.g_down, lb.g_down)
        wide = torch.zeros(cfg.d_model, cfg.ffn + 64, device="cuda", dtype=torch.bfloat16)
        wide[:, :cfg.ffn] = a.layers[0].w_down
        a.layers[0].w_down = wide[:, :cfg.ffn]
        assert a._native_args() is None and torch.equal(a.forward(x), ya)
    cfg = MoEConfig(experts=4, hidden=256, ffn=128, tokens=200)
    x = torch.randn(cfg.tokens, cfg.hidden, device="cuda").to(torch.bfloat16)
    logits = torch.randn(cfg.tokens, cfg.experts, device="cuda")
    a, b = MoELayer(cfg), MoELayer(cfg)
    b._native_args = lambda: None
    ya, yb = a.forward(x, logits).clone(), b.forward(x, logits).clone()
    dy = torch.randn_like(ya)
    assert torch.equal(ya, yb)
    (dxa, dla), (dxb, dlb) = a.backward(dy), b.backward(dy)
    assert torch.equal(dxa, dxb) and torch.equal(dla, dlb)
    # (the order of an expert's rows, and with it of the sums over them, differs from pass to pass)
    for ga, gb in ((a.g_gu, b.g_gu), (a.g_down, b.g_down)):
        assert float((ga.double() - gb.double()).norm()) < 2.0 ** -8 * float(gb.double().norm())


def models(tokens=256):
    """(model, inputs of forward, gradient of its result, owner of the gradient tensors) of each kind"""
    from megray_b200.models import MoEConfig, MoELayer, TPMLPConfig, TPMLPStack

    torch.manual_seed(2)
    rnd = lambda c, dtype=torch.bfloat16: torch.randn(tokens, c, device="cuda").to(dtype)  # noqa: E731
    mlp = TPMLPStack(TPMLPConfig(d_model=256, ffn=384, layers=1, tokens=tokens))
    yield mlp, (rnd(256),), rnd(256), mlp.layers[0]
    moe = MoELayer(MoEConfig(experts=4, hidden=256, ffn=128, tokens=tokens))
    yield moe, (rnd(256), rnd(4, torch.float32)), rnd(256), moe


def test_forward_looks_at_nothing_that_only_backward_uses():
    """A model whose gradients (and, here, backward buffers) were dropped for inference."""
    for model, inputs, _, holder in models():
        want = model.forward(*inputs).clone()
        holder.g_gu = holder.g_down = None
        for name in ("dgu", "dn", "dres", "dx", "dw", "dlogits", "dy_perm", "dx_perm"):
            if hasattr(model, name):
                setattr(model, name, None)
        assert model._native_forward_args() is not None
        model.forward(*inputs).zero_()
        assert torch.equal(model.forward(*inputs), want)


def test_backward_into_gradients_that_are_no_plain_matrices():
    """Strided gradients: op by op, and nothing beside them is written."""
    for model, inputs, dy, holder in models():
        model.forward(*inputs)
        first = lambda r: (r[0] if isinstance(r, tuple) else r).clone()  # noqa: E731
        dx = first(model.backward(dy))
        want = holder.g_gu, holder.g_down
        wide = [torch.full((g.shape[0], g.shape[1] + 64), 7.0, device="cuda", dtype=torch.bfloat16) for g in want]
        holder.g_gu, holder.g_down = (t[:, :g.shape[1]] for t, g in zip(wide, want))
        assert model._native_backward_args() is None and model._native_forward_args() is not None
        assert torch.equal(first(model.backward(dy)), dx)
        for got, g, t in zip((holder.g_gu, holder.g_down), want, wide):
            assert torch.equal(got, g) and bool((t[:, g.shape[1]:] == 7.0).all())


def test_saved_activations_that_are_no_plain_matrices():
    """Strided buffers in a model: op by op, the same result, and nothing beside them is written."""
    for model, inputs, dy, holder in models():
        want = model.forward(*inputs).clone()
        model.backward(dy)
        grad = holder.g_down.clone()
        saved = {"h": model.h[0] if isinstance(model.h, list) else model.h, "dgu": model.dgu}
        wide = {}
        for name, t in saved.items():
            wide[name] = torch.full((t.shape[0], t.shape[1] + 64), 7.0, device="cuda", dtype=torch.bfloat16)
            view = wide[name][:, :t.shape[1]]
            setattr(model, name, [view] if name == "h" and isinstance(model.h, list) else view)
        assert model._native_forward_args() is None and model._native_backward_args() is None
        assert torch.equal(model.forward(*inputs), want)
        model.backward(dy)
        assert float((holder.g_down.double() - grad.double()).norm()) <= 2.0 ** -8 * float(grad.double().norm())
        for name, t in saved.items():
            assert bool((wide[name][:, t.shape[1]:] == 7.0).all()) and not bool((wide[name][:, :t.shape[1]] == 7.0).all())


def test_buffers_are_asked_for_their_size():
    """A saved activation of another size is nothing the native passes write to."""
    for model, inputs, _, _ in models():
        h = model.h[0] if isinstance(model.h, list) else model.h
        for other in (h[:-1], h[1:], h.float(), torch.cat([h, h])):
            setattr(model, "h", [other] if isinstance(model.h, list) else other)
            assert model._native_forward_args() is None


def test_steps_of_its_own_are_run():
    """A weight-gradient product, routing or exchange that a program puts in place of the library's."""
    from megray_b200.models import TPMLPStack
    from megray_b200.parallel.expert_parallel import ExpertParallelOps

    seen = []

    class OwnProduct(TPMLPStack):
        def _wgrad(self, a_t, b_t, out):
            seen.append("wgrad")
            super()._wgrad(a_t, b_t, out)

    class OwnRouting(ExpertParallelOps):
        def route(self, logits):
            seen.append("route")
            super().route(-logits)

    (mlp, inputs, dy, _), (moe, (x, logits), _, _) = models()
    own = OwnProduct(mlp.cfg)
    assert own._native_forward_args() is not None  # it has no weight gradient
    own.forward(*inputs)
    own.backward(dy)
    assert seen == ["wgrad"] * 2
    moe.ep = OwnRouting(None, moe.cfg.tokens, moe.cfg.hidden, moe.cfg.experts, moe.cfg.capacity_factor)
    moe.forward(x, logits)
    assert seen[2:] == ["route"] and torch.equal(moe.ep.idx.long(), (-logits).topk(2, dim=1).indices)
    moe.ep = ExpertParallelOps(None, moe.cfg.tokens, moe.cfg.hidden, moe.cfg.experts, moe.cfg.capacity_factor)
    assert moe._native_forward_args() is not None
    combine = moe.ep.combine
    moe.ep.combine = lambda *a, **kw: (seen.append("combine"), combine(*a, **kw))
    moe.forward(x, logits)
    assert seen[3:] == ["combine"]
