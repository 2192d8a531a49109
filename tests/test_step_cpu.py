"""H3Runtime.step on models that change how the tokens become a latent again: what they define is what runs."""
import pytest
import torch

from rapid_h3_b200 import model, step


def _runtime(m):
    """A runtime without blocks: embedding and output projection only, which run on the CPU."""
    rt = step.H3Runtime.__new__(step.H3Runtime)
    rt.model, rt.cfg, rt.linears, rt.blocks = m, m.cfg, {}, []
    return rt


def _inputs(cfg):
    return step.make_inputs(cfg, (2, 3, 4), 5, 2, 8, seed=3)


class OwnUntokens(model.H3Transformer):
    def untokens(self, x, latent_shape):
        v, a = super().untokens(x, latent_shape)
        return 2 * v, 3 * a


class NoFinalNorm(model.H3Transformer):
    def __init__(self, cfg):
        super().__init__(cfg)
        del self.final_norm

    def untokens(self, x, latent_shape):
        n = latent_shape[1] * latent_shape[2] * latent_shape[3]
        return self.unembed(x[:n]).t().reshape(latent_shape), self.audio_unembed(x[n:])


def _patched(cfg):
    m = model.H3Transformer(cfg)
    m.untokens = lambda x, latent_shape: model.H3Transformer.untokens(m, -x, latent_shape)
    return m


@pytest.mark.parametrize("make", [model.H3Transformer, OwnUntokens, NoFinalNorm, _patched])
def test_the_models_own_untokens_runs(make):
    cfg = model.H3Config.tiny(n_blocks=1)
    m = model.init_weights(make(cfg), seed=1)
    latent, audio, t_emb, rope, ctx = _inputs(cfg)
    vid, aud = _runtime(m).step(latent, audio, t_emb, rope, ctx)
    for i in range(2):
        v, a = m.untokens(m.tokens(latent[i], audio[i]), latent.shape[1:])
        assert torch.equal(vid[i], v) and torch.equal(aud[i], a)


def test_a_norm_somebody_watches_is_called(monkeypatch):
    """Hooks of the module or on all modules, and a replaced forward or __call__, keep the module's own call."""
    norm = model.RMSNorm(8, 1e-6)
    plain = step._plain_final_norm
    assert plain(norm) and not plain(torch.nn.LayerNorm(8))

    class Sub(model.RMSNorm):
        pass

    assert not plain(Sub(8, 1e-6))
    hooks = torch.nn.modules.module
    for register in (norm.register_forward_hook, norm.register_forward_pre_hook, hooks.register_module_forward_hook,
                     hooks.register_module_forward_pre_hook, hooks.register_module_full_backward_hook):
        handle = register(lambda *a: None)
        assert not plain(norm)
        handle.remove()
        assert plain(norm)
    forward, call = model.RMSNorm.forward, torch.nn.Module.__call__
    for owner, name, was in ((model.RMSNorm, "forward", forward), (torch.nn.Module, "__call__", call)):
        with monkeypatch.context() as patch:
            patch.setattr(owner, name, lambda self, x: was(self, x))
            assert not plain(norm)
    assert plain(norm)
