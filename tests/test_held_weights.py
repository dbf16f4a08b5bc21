"""A weight-streaming product begins to read its matrix while the kernel before it ends only if a model holds the matrix: any
other may be that kernel's output."""
import pytest
import torch

from flexengine_b200 import ops
from flexengine_b200.bench.hybrid import bebulorn_config, fuvuvik_config, ribozen_config
from flexengine_b200.weights import random_model

QWEN = dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", num_hidden_layers=2, hidden_size=64, num_attention_heads=4,
            num_key_value_heads=2, head_dim=16, intermediate_size=128, vocab_size=96, rope_theta=10000.0, rms_norm_eps=1e-6,
            max_position_embeddings=128, tie_word_embeddings=True, use_sliding_window=False, hidden_act="silu")


def _begins_early(monkeypatch, call):
    """What the entry points of the products are told about their matrix (the argument before the stream)."""
    seen = []
    for name, value in (("_need_cuda", lambda *t: None), ("_bf16", lambda: None), ("_ptr", lambda t: None), ("_stream", lambda: "stream"),
                        ("status_word", lambda device: None), ("_run", lambda lib, name, *args: seen.append((name, args[-2], args[-1])))):
        monkeypatch.setattr(ops, name, value)
    call()
    assert seen and all(name.startswith("fe_skinny") and stream == "stream" for name, _, stream in seen)
    return [early for _, early, _ in seen]


CALLS = {
    "linear": lambda x, w: ops.linear(x, w),
    "float result": lambda x, w: ops.linear(x, w, None, out_float32=True),
    "ends a branch": lambda x, w: ops.linear(x, w, follow=(torch.zeros(2, 64), torch.ones(64), 1e-6)),
    "gated": lambda x, w: ops.linear_gated(x, w, 32, "gelu_tanh"),
    "swiglu": lambda x, w: ops.linear_swiglu(x, w, 32),
    "activated": lambda x, w: ops.linear_activated(x, w, "relu2"),
    "qkv": lambda x, w: ops.qkv_projection(x, w, None, torch.zeros(2, dtype=torch.int32), torch.ones(8), 16, None,
                                           torch.empty(1, 1, 16, 16, dtype=torch.bfloat16), torch.empty(1, 1, 16, 16, dtype=torch.bfloat16), 2, 1, 16, 16),
}


@pytest.mark.parametrize("kind", CALLS)
def test_only_held_matrices_are_read_early(kind, monkeypatch):
    x, w = torch.zeros(2, 64, dtype=torch.bfloat16), torch.zeros(64, 64, dtype=torch.bfloat16)
    assert _begins_early(monkeypatch, lambda: CALLS[kind](x, w)) == [0]
    w.held = True
    assert _begins_early(monkeypatch, lambda: CALLS[kind](x, w)) == [1]
    assert _begins_early(monkeypatch, lambda: CALLS[kind](x, w * 1)) == [0], "what is made of it is another matrix"


@pytest.mark.parametrize("config", [QWEN, fuvuvik_config(64, 4, 96, 4), bebulorn_config(64, 6, 96, 4), ribozen_config(256, 3, 96, 8)],
                         ids=["qwen2", "fuvuvik", "bebulorn", "ribozen"])
def test_a_bound_model_holds_its_matrices(config):
    _typed, _plan, model = random_model(config, seed=1, dtype="bfloat16", device="cpu")
    count = 0

    def look(part):
        nonlocal count
        for name, value in vars(part).items():
            for v in value if isinstance(value, (list, tuple)) else [value]:
                if isinstance(v, torch.Tensor):
                    assert v.held, (type(part).__name__, name)
                    count += v.dim() == 2
                elif hasattr(v, "parameter_shapes"):
                    look(v)
    for part in [p for _, p in model._outer_parts()] + [p for b in model.blocks for p in b.parts().values()]:
        look(part)
    assert count >= 8


@pytest.mark.gpu
@pytest.mark.parametrize("K", [64, 256, 1024])
@pytest.mark.parametrize("rows", [1, 8])
def test_products_of_a_matrix_the_kernel_before_made(K, rows):
    """The matrix comes from this package's own activation kernel, which lets its successor begin early, and is another each time."""
    gen = torch.Generator("cuda:0").manual_seed(K)
    N = 4096
    x = torch.randn((rows, K), generator=gen, device="cuda:0").to(torch.bfloat16)
    made = torch.randn((24, N, 2 * K), generator=gen, device="cuda:0").to(torch.bfloat16)
    got, want = [], []
    for m in made:
        got.append(ops.linear(x, ops.swiglu(m, K)))
        got.append(ops.linear_gated(x, ops.swiglu(m, K), N // 2, "silu"))
    for m in made:
        w = ops.swiglu(m, K)
        torch.cuda.synchronize()
        want.append(ops.linear(x, w))
        want.append(ops.linear_gated(x, w, N // 2, "silu"))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_a_vocabulary_keeps_the_chain_of_multiply_adds_whatever_its_size(monkeypatch):
    """A step wants few rows of logits, which the product in three parts would not serve faster; what a model calls its head is by
    the model's word and not by the rows, so that a row's logits do not depend on the batch."""
    class Core:
        fe_gemm_split_room = staticmethod(lambda M, N, K: 0)
    seen = []
    for name, value in (("_need_cuda", lambda *t: None), ("_core", lambda: Core), ("_ptr", lambda t: None), ("_stream", lambda: None),
                        ("status_word", lambda device: None), ("_run", lambda lib, name, *args: seen.append(name))):
        monkeypatch.setattr(ops, name, value)
    w = torch.empty(8192, 1024)
    for rows in (1, 300):
        ops.linear(torch.empty(rows, 1024), w)
    w.vocabulary = True
    for rows in (1, 300):
        ops.linear(torch.empty(rows, 1024), w)
    assert seen == ["fe_gemm_split"] * 2 + ["fe_gemm_fp32"] * 2


@pytest.mark.parametrize("tied", [True, False])
def test_a_bound_model_says_which_matrix_is_its_vocabulary(tied):
    _typed, _plan, model = random_model(dict(QWEN, tie_word_embeddings=tied), seed=1, dtype="float32", device="cpu")
    assert model.head.weight.vocabulary
    assert not any(getattr(t, "vocabulary", False) for block in model.blocks for part in block.parts().values() for t in vars(part).values())
