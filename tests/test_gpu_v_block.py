"""A prompt's block as one library call (cd_complexity_block) against the general route of the same block: the same launches
on the same inputs, so logits, cache and mu agree to the bit.  Rows below and above 64 (one launch for both up-projections or
two), head sizes 64 and 128 (rotation after or inside the projection), with and without Q/K norm and cache; whatever is not
plain takes the general route."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(hidden, inner, heads, kv, experts, qk_norm=True, layers=2):
    from complexity_deep_b200.models import ComplexityConfig, ComplexityModel
    torch.manual_seed(hidden + heads)
    cfg = ComplexityConfig(vocab_size=1000, hidden_size=hidden, intermediate_size=inner, num_hidden_layers=layers,
                           num_attention_heads=heads, num_key_value_heads=kv, num_experts=experts, use_qk_norm=qk_norm)
    model = ComplexityModel(cfg)
    with torch.no_grad():
        for layer in model.layers:
            layer.mu_guidance.mu_proj.weight.normal_(0, 0.05)
    return model.to("cuda", torch.bfloat16).eval()


def _both(model, ids, monkeypatch, **kw):
    from complexity_deep_b200.core.layer import TransformerBlock
    ran = []
    native = TransformerBlock._forward_native

    def counted(self, *a):
        out = native(self, *a)
        ran.append(out is not None)
        return out
    with torch.no_grad():
        monkeypatch.setattr(TransformerBlock, "_forward_native", counted)
        got = model(ids, **kw)
        monkeypatch.setattr(TransformerBlock, "_forward_native", lambda self, *a: None)
        want = model(ids, **kw)
        monkeypatch.setattr(TransformerBlock, "_forward_native", native)
    return got, want, ran


@pytest.mark.parametrize("hidden,inner,heads,kv,experts,qk_norm", [(256, 704, 4, 2, 4, True), (512, 1408, 4, 4, 4, True),
                                                                   (256, 768, 4, 1, 8, False), (1024, 2816, 8, 4, 2, True)])
@pytest.mark.parametrize("B,S", [(1, 2), (1, 37), (2, 32), (1, 65), (3, 171), (2, 513)])
def test_same_bits(hidden, inner, heads, kv, experts, qk_norm, B, S, monkeypatch):
    model = _model(hidden, inner, heads, kv, experts, qk_norm)
    ids = torch.randint(0, 1000, (B, S), device="cuda")
    for cached in (False, True):
        got, want, ran = _both(model, ids, monkeypatch, use_cache=cached)
        assert ran == [True] * 2
        assert torch.equal(got.logits, want.logits)
        if cached:
            for a, b in zip(got.past_key_values, want.past_key_values):
                assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_general_route_for_all_else(monkeypatch):
    model = _model(256, 704, 4, 2, 4)
    ids = torch.randint(0, 1000, (1, 33), device="cuda")
    seen = []
    handle = model.layers[0].mu_guidance.register_forward_hook(lambda m, a, out: seen.append(out))
    got, want, ran = _both(model, ids, monkeypatch)
    assert ran == [False, True] and len(seen) == 2 and torch.equal(got.logits, want.logits)
    handle.remove()
    model.split_residual_stream = False
    got, want, ran = _both(model, ids, monkeypatch)
    assert ran == [False, False] and torch.equal(got.logits, want.logits)
    model.split_residual_stream = True
    # a weight that was replaced by one of another shape is refused as before
    model.layers[1].self_attn.o_proj.weight = torch.nn.Parameter(torch.zeros(256, 128, dtype=torch.bfloat16, device="cuda"))
    with torch.no_grad(), pytest.raises(RuntimeError):
        model(ids)


@pytest.mark.parametrize("cached", [False, True])
@pytest.mark.parametrize("hidden,inner,heads,kv,experts,T", [(1024, 2816, 8, 4, 2, 3000), (512, 2048, 8, 8, 1, 4001)])
def test_no_more_memory_than_launch_by_launch(hidden, inner, heads, kv, experts, T, cached, monkeypatch):
    """What a block holds at its fullest: intermediate results that do not live at the same time share their memory."""
    from complexity_deep_b200.core.layer import TransformerBlock
    model = _model(hidden, inner, heads, kv, experts)
    ids = torch.randint(0, 1000, (1, T), device="cuda")
    native, peaks = TransformerBlock._forward_native, []
    for run in (native, lambda self, *a: None):
        monkeypatch.setattr(TransformerBlock, "_forward_native", run)
        with torch.no_grad():
            model(ids, use_cache=cached)                   # weights are packed, tables made
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            base = torch.cuda.memory_allocated()
            out = model(ids, use_cache=cached)
            peaks.append(torch.cuda.max_memory_allocated() - base)
            del out
    assert peaks[0] <= peaks[1] + 16 * 512                 # an allocation is rounded up to 512 bytes
