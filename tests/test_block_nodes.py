"""Which decoder blocks may run as two autograd nodes (engine/blocks.py): blocks with other modules in place of their own may not.
The kernels are not asked for here, so these run without a GPU."""
import pytest
import torch
from torch import nn

from opaque_b200.engine import blocks, fused
from opaque_b200.models import GPT2Config, GPT2LMHeadModel, LlamaConfig, LlamaForCausalLM
from opaque_b200.models.gpt2 import GPT2Block


@pytest.fixture(autouse=True)
def _as_on_a_gpu(monkeypatch):
    monkeypatch.setattr(blocks, "available", lambda: True)
    monkeypatch.setattr(fused, "_own_gemm_ok", lambda *a: True)


def _layer():
    model = LlamaForCausalLM(LlamaConfig.tiny())
    model.add_lora(8, 16.0)
    layer = model.model.layers[0]
    return layer, lambda: layer._two_nodes(torch.zeros(1, 8, 128, dtype=torch.bfloat16), model.rope_cos, model.rope_sin, None)


class _Other(nn.Module):
    def forward(self, x, *args):
        return x


def test_llama_blocks_with_other_modules():
    layer, two_nodes = _layer()
    assert two_nodes()
    for part in ("self_attn", "mlp"):
        own = getattr(layer, part)
        for other in (torch.compile(own), _Other()):
            setattr(layer, part, other)
            assert not two_nodes()
        setattr(layer, part, own)
    att, own = layer.self_attn, layer.self_attn.q_proj
    for other in (nn.Linear(128, 128), torch.compile(own)):
        att.q_proj = other
        assert not two_nodes()
    att.q_proj = own
    assert two_nodes()


def test_llama_attention_patched_as_a_class(monkeypatch):
    """The patched forward may need none of the projections."""
    layer, two_nodes = _layer()
    monkeypatch.setattr(type(layer.self_attn), "forward", lambda self, x, *a: x)
    del layer.self_attn.k_proj
    assert not two_nodes()


def test_gpt2_blocks_that_override_a_part():
    class Block(GPT2Block):
        def _attention(self, y):
            return y
    block = GPT2LMHeadModel(GPT2Config.tiny()).requires_grad_(False).h[0]
    x = torch.zeros(1, 8, 128, dtype=torch.bfloat16)
    assert block._two_nodes(x)
    block.__class__ = Block
    assert not block._two_nodes(x)


def _as_plain_tensor(module, name):
    t = getattr(module, name).detach()
    delattr(module, name)
    setattr(module, name, t)


@pytest.mark.parametrize("path,name", [("self_attn.q_proj", "weight"), ("self_attn.o_proj", "lora_B"), ("self_attn.k_proj", "lora_A"), ("mlp.down_proj", "weight")])
def test_llama_blocks_with_plain_tensors_for_parameters(path, name):
    layer, two_nodes = _layer()
    _as_plain_tensor(layer.get_submodule(path), name)
    assert not two_nodes()


@pytest.mark.parametrize("path,name", [("attn_c_attn", "bias"), ("mlp_c_proj", "weight"), ("ln_2", "weight")])
def test_gpt2_blocks_with_plain_tensors_for_parameters(path, name):
    block = GPT2LMHeadModel(GPT2Config.tiny()).requires_grad_(False).h[0]
    _as_plain_tensor(getattr(block, path), name)
    assert not block._two_nodes(torch.zeros(1, 8, 128, dtype=torch.bfloat16))


def test_exceptions_of_the_compiled_sequences_keep_their_type():
    """What torch's own call raises in Python: an IndexError here, as torch.OutOfMemoryError where an allocation fails."""
    import importlib.util

    from opaque_b200.utils import build
    spec = importlib.util.spec_from_file_location("opaque_b200.ops._blocks", build.build_block_steps())
    steps = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(steps)
    with pytest.raises(IndexError):
        steps.gpt2_in(torch.zeros(()), None, torch.zeros(1), torch.zeros(1), torch.zeros(1, 1), torch.zeros(1), 1e-5)


@pytest.mark.parametrize("examples,rows,width,in_kernel", [(1, 8192, 768, False), (2, 8192, 768, False), (3, 8193, 768, True), (3, 8193, 1024, False),
                                                           (4, 8192, 1024, True), (1, 8192, 256, True), (5, 5000, 768, True), (32, 4096, 768, False),
                                                           (3, 8192, 768, False)])
def test_norm_sums_of_few_long_examples_are_apart(monkeypatch, examples, rows, width, in_kernel):
    """The kernel that adds a norm's sums has at most 16 blocks per example; the last two: few rows, and rows that are no multiple."""
    class Capture:
        batch_size, sums_wait = examples, staticmethod(fused.Capture.sums_wait)

        def pe_view(self, p):
            return torch.zeros(examples, width)
    monkeypatch.setattr(fused, "_ACTIVE", Capture())
    sums = blocks._norm_sums(True, nn.LayerNorm(width), rows)
    assert (sums[0] is not None) == in_kernel == (sums[1] is not None)
    assert blocks._norm_sums(False, nn.LayerNorm(width), rows) == (None, None)
