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
