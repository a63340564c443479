"""Decoder steps of more than 8 rows through layers of which only some take the norms and residual adds into their products."""
import dataclasses

import pytest
import torch

from return_b200.config.model_config import Qwen3Config

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
H = 256
WIDE = 40 * 1024                                              # gate and up rows of such a layer hold more weights than ``rows_limit`` admits


def _model(widths, seed=0):
    from return_b200.models import qwen3
    from return_b200.models.decoder import DecoderModel
    from return_b200.parts.base import BuildEnv
    cfg = Qwen3Config.from_dict(dict(vocab_size=320, hidden_size=H, intermediate_size=512, num_hidden_layers=len(widths), num_attention_heads=4,
                                     num_key_value_heads=2, head_dim=64, rope_theta=1e4, rms_norm_eps=1e-5, tie_word_embeddings=True,
                                     max_position_embeddings=512))
    spec = qwen3.decoder_spec(cfg, 512)
    layers = tuple(dataclasses.replace(b, feed_forward=dataclasses.replace(b.feed_forward, intermediate_size=w)) for b, w in zip(spec.layers, widths))
    model = DecoderModel(dataclasses.replace(spec, layers=layers), BuildEnv(torch.bfloat16, DEV))
    model.bind(_weights(model, seed))
    return model


def _weights(model, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return {n: torch.empty(p.shape, device=DEV).normal_(1.0 if len(p.shape) == 1 else 0.0, 0.1 if len(p.shape) == 1 else 0.03, generator=g).bfloat16()
            for n, p in model.params().items()}


def _step(model, T, monkeypatch=None):
    """Logits of a prompt's T tokens, and which fused products ran with a next norm."""
    from return_b200.engine.batch import StepBatch, StepEntry, build_host_batch
    from return_b200.engine.config import EngineConfig
    from return_b200.engine.runner import ModelRunner
    from return_b200.ext import ops
    runner = ModelRunner(model, EngineConfig(max_token=1024, max_reside=2, page_size=16, dtype="bfloat16", max_model_len=512, use_cuda_graph=False), 512)
    runner.add_request(0)
    entry = runner.reserve(0, [(7 * i) % 320 for i in range(T)], range(T))
    batch = StepBatch(build_host_batch([entry], runner.manager, 320, 512, runner.tilings), DEV, runner.staging)
    left = []
    if monkeypatch is not None:
        fused = ops.gemm_rows_fused

        def seen(x, w, out, gated=False, scale=None, residual=None, **kw):
            if residual is not None and w.shape[1] != H:      # a feed-forward's last product
                left.append(residual[1] is not None)
            return fused(x, w, out, gated, scale, residual, **kw)

        monkeypatch.setattr(ops, "gemm_rows_fused", seen)
    with torch.no_grad():
        logits = model.forward(batch, runner.storage)
    ops.check_status(DEV)
    return logits, left, "block.prenormed" in batch.scratch


# the layers' widths, and for each fused layer's last product whether the layer behind it reads what it leaves
@pytest.mark.parametrize("widths,left", [((512, 512, 512), [True, True]), ((512, WIDE, 512), []), ((WIDE, 512, 512), [True]), ((512, 768, WIDE, 512), [True])])
@pytest.mark.parametrize("T", [9, 100])
def test_what_a_layer_leaves_is_read(monkeypatch, widths, left, T):
    from return_b200.ext import ops
    model = _model(widths)
    got, what, over = _step(model, T, monkeypatch)
    assert what == left and not over
    monkeypatch.undo()
    monkeypatch.setattr(ops, "rows_limit", lambda *a: 0)       # part by part, the library's products
    monkeypatch.setattr(ops, "_rows_form", lambda *a: None)
    want, _, _ = _step(_model(widths), T)
    assert torch.isfinite(got).all() and (got - want).norm() <= 2e-2 * want.norm()


@pytest.mark.parametrize("T", [3, 9, 100])
def test_weights_bound_again_are_used(T):
    model = _model((512, 512))
    old, _, _ = _step(model, T)
    model.bind(_weights(model, 7))
    got, _, _ = _step(model, T)
    want, _, _ = _step(_model((512, 512), 7), T)
    assert torch.equal(got, want) and not torch.equal(got, old)
