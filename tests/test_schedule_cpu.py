"""The launch schedule of the models without a GPU: the native library is replaced by a recorder, so that the order of the
calls, and what each is handed, can be looked at."""
import array

import pytest
import torch

from llm_kittens_b200.models.config import ModelConfig
from llm_kittens_b200.models.transformer import Transformer
from llm_kittens_b200.ops import _native, attention, elementwise, gemm


class _Lib:
    """Every entry point exists and returns 0."""

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture
def calls(monkeypatch):
    """List of (entry point, arguments) of the native calls made so far."""
    out = []
    monkeypatch.setattr(_native, "lib", lambda: _Lib())
    monkeypatch.setattr(_native, "call", lambda name, *a: out.append((name, a)))
    monkeypatch.setattr(_native, "require_cuda_tensor", lambda *a, **k: None)
    monkeypatch.setattr(_native, "status_word", lambda: None)
    monkeypatch.setattr(_native, "scratch_buffer", lambda pool, nbytes, min_bytes, name: torch.empty(16, dtype=torch.uint8))
    monkeypatch.setattr(gemm, "tile_rows", lambda: 256)
    monkeypatch.setattr(attention, "_sms", lambda: 148)
    return out


def _model(head_size, recompute=0):
    cfg = ModelConfig(family="gpt2", max_seq_len=512, vocab_size=250, padded_vocab_size=256, num_layers=2, num_heads=2,
                      num_kv_heads=2, channels=2 * head_size, hidden_dim=8 * head_size)
    return Transformer(cfg, device="cpu", recompute=recompute)


@pytest.mark.parametrize("head_size,T,forks", [(64, 64, 0), (64, 192, 0), (64, 128, 0), (128, 64, 0), (128, 192, 0), (128, 128, 2),
                                               (128, 320, 2)])
def test_the_side_stream_is_used_only_for_work(calls, monkeypatch, head_size, T, forks):
    """The backward pass forks to the side stream only where something is launched there: the pre-pass of the attention
    backward, once per layer, when the tcgen05 kernels run and the pre-pass is not in the epilogue of a GEMM (heads of 64)."""
    model = _model(head_size)
    work = []

    def fork(fn):
        before = len(calls)
        fn()
        work.append([name for name, _ in calls[before:]])

    monkeypatch.setattr(model, "_fork", fork)
    tokens = torch.zeros(1, T, dtype=torch.int32)
    model.forward(tokens, tokens)
    model.backward()
    assert work == [["llmk_attention_bwd_prep"]] * forks


def test_a_replaced_tensor_is_used_by_every_layer_of_the_next_forward(calls):
    """Per-layer views are made once; replacing one stacked tensor, in whatever way, makes them again."""
    model = _model(64)
    tokens = torch.zeros(1, 64, dtype=torch.int32)
    model.forward(tokens)

    def pointers(entry, position):
        calls.clear()
        model.forward(tokens)
        return [a[position].data_ptr() for name, a in calls if name == entry]

    for put in (lambda t: model.p.__setitem__("qkvw", t), lambda t: model.p.update(qkvw=t), lambda t: setattr(model, "p", {**model.p, "qkvw": t})):
        mine = torch.randn_like(model.p["qkvw"])
        put(mine)
        seen = pointers("llmk_gemm", 3)
        assert all(mine[layer].data_ptr() in seen for layer in range(2))
        assert model.p["qkvw"] is mine
    mine = torch.empty_like(model.acts["lse"])
    model.acts["lse"] = mine
    assert pointers("llmk_attention_fwd", 1) == [mine[0].data_ptr(), mine[1].data_ptr()]
    acts = model.acts
    model.acts = acts                       # handing the same table back keeps it (and what identifies it)
    assert model.acts is acts


@pytest.mark.parametrize("index,address,native", [(0, 4096, True), (1, 4096, False), (0, 4098, False)])
def test_zeroing_a_tensor_of_another_device_is_left_to_pytorch(calls, monkeypatch, index, address, native):
    """Kernels are launched on the current device's stream: a tensor of another device would be written there without order
    to the work of its own device."""
    class Tensor:
        device = torch.device("cuda", index)
        zeroed = False

        def data_ptr(self):
            return address

        def numel(self):
            return 8

        def element_size(self):
            return 2

        def zero_(self):
            self.zeroed = True
            return self

    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0)
    t = Tensor()
    assert elementwise.zero_(t) is t
    assert (t.zeroed, [name for name, _ in calls]) == ((False, ["llmk_zero"]) if native else (True, []))


@pytest.mark.parametrize("B,T,NH,HS,tc", [(1, 64, 12, 64, False), (64, 192, 12, 64, False), (1, 128, 1, 128, True), (1, 320, 12, 64, False),
                                          (2, 320, 32, 64, True), (7, 448, 6, 64, True), (7, 448, 12, 64, True), (2, 576, 6, 64, True),
                                          (2, 576, 12, 64, True), (1, 320, 32, 128, True), (2, 320, 32, 128, True),
                                          (7, 448, 16, 128, True), (2, 576, 32, 128, True), (1, 320, 35, 64, False), (1, 320, 36, 64, True),
                                          (2, 128, 37, 64, False), (3, 128, 25, 64, True), (1, 256, 37, 64, False), (2, 256, 19, 64, True),
                                          (1, 384, 1, 64, True)])
def test_forward_attention_kernel_by_size(calls, monkeypatch, B, T, NH, HS, tc):
    """Which kernel a forward takes on a GPU of 148 SMs, and that asking for one gets it where it takes the length."""
    monkeypatch.setattr(attention, "IMPL", "tc")
    qkv = torch.empty(B, T, 3 * NH * HS, dtype=torch.bfloat16)
    for impl in (None, "tc", "warp"):
        attention.attention_fwd(qkv, B, T, NH, NH, HS, impl=impl)
    name = lambda on: "llmk_attention_fwd_tc" if on else "llmk_attention_fwd"
    assert [c[0] for c in calls] == [name(tc), name(T % 128 == 0 or T > 256), name(False)]


@pytest.mark.parametrize("llama,short,entry", [(0, 0, "llmk_layernorm_fwd"), (1, 0, "llmk_rmsnorm_fwd"), (0, 1, "llmk_forward_layers")])
def test_what_the_native_forward_refuses_is_named(monkeypatch, llama, short, entry):
    """The entry point that refuses a shape is named, as when the blocks run one by one (an odd width, which the norm refuses
    before it launches anything); an argument block of another length is not read."""
    words = [1, 1, 64, 13, 1, 1, 13, 52, llama] + [0] * (7 + 2 * 29 - short)
    block = array.array("q", words)
    monkeypatch.setattr(_native, "_invoke", lambda name, args: getattr(_native.lib(), name)(*[_native._conv(a) for a in args], None))
    with pytest.raises(_native.NativeError, match=f"^{entry} failed: unsupported or misaligned shape"):
        _native.call("llmk_forward_layers", *block.buffer_info(), 1e-5)
