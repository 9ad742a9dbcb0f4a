"""A norm whose work the products before and behind it do, against 64 bits and against the norm as a kernel of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D", [64, 1024, 3072, 8192])
@pytest.mark.parametrize("M", [1, 2, 3, 8])
@pytest.mark.parametrize("swiglu", [False, True])
def test_products_around_a_norm(D, M, swiglu):
    from oracle_engine_b200.csrc import ops, ops_tc
    g = torch.Generator().manual_seed(D + M)
    K, N, eps = 200, 136, 1e-5
    rand = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(DEV)                    # noqa: E731
    a, w1, w2 = rand(M, K).bfloat16(), rand(D, K, scale=0.1).bfloat16(), rand(N, D, scale=D ** -0.5).bfloat16()
    x, weight = rand(M, D, scale=3.0), 1 + rand(D, scale=0.1)
    x[-1] *= 1e-3                                                          # a row whose norm sees the epsilon

    def second(h):
        y = torch.empty(M, N // 2 if swiglu else N, dtype=torch.bfloat16, device=DEV)
        ops_tc.gemm(y, h, w2, swiglu=swiglu)
        return y.double()
    left = ops_tc.ScaledRows(torch.empty(M, D, dtype=torch.bfloat16, device=DEV), torch.empty(M, D // 16, device=DEV), eps)
    mine, plain = x.clone(), x.clone()
    ops_tc.gemm(mine, a, w1, accumulate=True, leave=(weight, left))
    ops_tc.gemm(plain, a, w1, accumulate=True)
    assert torch.equal(mine, plain)                                        # the stream's bits
    h = torch.empty(M, D, dtype=torch.bfloat16, device=DEV)
    ops.rmsnorm(h, plain, weight, eps)
    z = plain.double() / torch.sqrt((plain.double() ** 2).mean(1, keepdim=True) + eps) * weight.double() @ w2.double().T
    want = torch.nn.functional.silu(z[:, 0::2]) * z[:, 1::2] if swiglu else z
    err = lambda y: ((y - want).norm(dim=1) / want.norm(dim=1)).max().item()                      # noqa: E731
    fused, apart = err(second(left)), err(second(h))
    # both round the normed value and the result to bfloat16 once (2^-9 relative each, twice that through gate times up)
    assert fused < 8e-3 and fused < 1.5 * apart + 1e-4, (fused, apart)


def test_forms_that_are_refused():
    from oracle_engine_b200.csrc import ops, ops_tc
    weight = torch.ones(64, device=DEV)
    assert not ops_tc.scaled_rows_supported(5, 64, weight) and not ops_tc.scaled_rows_supported(1, 72, torch.ones(72))
    left = ops_tc.ScaledRows(torch.empty(2, 64, dtype=torch.bfloat16, device=DEV), torch.empty(2, 4, device=DEV), 1e-5)
    a, w = torch.zeros(2, 8, dtype=torch.bfloat16, device=DEV), torch.zeros(64, 8, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(ops.KernelError):                                   # the sums go into a stream
        ops_tc.gemm(torch.empty(2, 64, device=DEV), a, w, leave=(weight, left))


@pytest.mark.parametrize("batch", [1, 4, 5])
def test_a_decoder_uses_it(batch, monkeypatch):
    from oracle_engine_b200.config.base import get_architecture
    from oracle_engine_b200.engine.batch import SequenceStep
    from oracle_engine_b200.engine.engine import Engine
    from oracle_engine_b200.engine.runtime import Runtime
    cfg = get_architecture("LlamaForCausalLM").config_cls.from_dict(dict(
        architectures=["LlamaForCausalLM"], vocab_size=256, hidden_size=256, num_hidden_layers=3, num_attention_heads=4, num_key_value_heads=2,
        head_dim=64, intermediate_size=512, rms_norm_eps=1e-5, max_position_embeddings=512, tie_word_embeddings=True))
    used, leave = [], Runtime.leave_normed

    def run(form):
        monkeypatch.setattr(Runtime, "leave_normed", form)
        eng = Engine.from_config(cfg, seed=3, std=0.1, dtype="bfloat16", max_tokens=64 * 2 * batch)
        slots = [eng.alloc() for _ in range(batch)]
        return torch.stack([eng.step([SequenceStep(s, [(31 * b + 7 * i) % 256], [0]) for b, s in enumerate(slots)]).clone() for i in range(8)])

    def counted(self, out):
        got = leave(self, out)
        used.append(got is not None)
        return got
    mine = run(counted)
    assert sum(used[:6]) == (5 if batch <= 4 else 0)                       # two norms a layer but the first and the last
    other = run(lambda self, out: None)
    assert torch.isfinite(mine).all() and ((mine - other).norm() / other.norm()).item() < 2e-2


@pytest.mark.parametrize("tokens", [4, 5, 300])
def test_passes_of_more_rows_do_not_look_for_it(tokens, monkeypatch):
    """What a pass launched kernel by kernel would pay for on the host in every layer."""
    from oracle_engine_b200.config.base import get_architecture
    from oracle_engine_b200.engine.batch import SequenceStep
    from oracle_engine_b200.engine.engine import Engine
    from oracle_engine_b200.engine.runtime import Runtime
    from oracle_engine_b200.parts import block
    cfg = get_architecture("LlamaForCausalLM").config_cls.from_dict(dict(
        architectures=["LlamaForCausalLM"], vocab_size=256, hidden_size=256, num_hidden_layers=3, num_attention_heads=4, num_key_value_heads=2,
        head_dim=64, intermediate_size=512, rms_norm_eps=1e-5, max_position_embeddings=512, tie_word_embeddings=True))
    eng, calls = Engine.from_config(cfg, seed=3, std=0.1, dtype="bfloat16", max_tokens=1024, use_graphs=False), []
    for owner, name in ((block, "leaves_to"), (Runtime, "leave_normed")):
        monkeypatch.setattr(owner, name, lambda *a, f=getattr(owner, name): (calls.append(1), f(*a))[1])
    out = eng.step([SequenceStep(eng.alloc(), [t % 256 for t in range(tokens)], [tokens - 1])])
    assert torch.isfinite(out).all() and bool(calls) == (tokens <= 4)
