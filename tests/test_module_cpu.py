"""Host side of the module and of its launches: what needs no GPU."""
from types import SimpleNamespace

import pytest
import torch

from cobalt_b200 import CobaltSparseLinear, FusedProjections
from cobalt_b200._lib import CobaltError
from cobalt_b200.decoder import CobaltDecoder
from cobalt_b200.linear import called_plainly


def small_module(scale2=None, K=16, N=256):
    keep, q = torch.ones(K, N, dtype=torch.bool), torch.zeros(K, N, dtype=torch.uint8)
    sz = torch.ones(K, N // 128).half()
    return CobaltSparseLinear(q, sz, sz, keep, scale2, None, {"nbits": 4})


def test_column_scale_is_kept_where_vector_loads_can_read_it():
    """A slice of a larger buffer starts anywhere and a column of a matrix is strided; the kernels read 16 bytes at a time."""
    buf = torch.rand(256 + 8).half() + 0.5
    for scale2 in (buf[1:257], buf[3:259].view(1, 256), torch.stack([buf[:256]] * 2, 1)[:, 0]):
        m = small_module(scale2)
        assert m.scale2.data_ptr() % 16 == 0 and m.scale2.is_contiguous()
        assert torch.equal(m.scale2, scale2.reshape(-1))
        state = m.state_dict()
        assert CobaltSparseLinear.from_state_dict(dict(state, scale2=scale2), device="cpu").scale2.data_ptr() % 16 == 0


def test_status_words_of_fused_launches_and_decoders():
    """A code that a kernel left in the scratch of a fused launch, or for a prompt's attention, is reported."""
    fused = [FusedProjections([small_module()]) for _ in range(5)]
    assert [f.device_status() for f in fused] == [0] * 5
    for f in fused:
        f._scratch = torch.zeros(1024, dtype=torch.uint8)
    word = torch.zeros(1, dtype=torch.int32)
    dec = SimpleNamespace(lin={0: small_module()}, prompt_status=word, att_fused=None, qkv=fused[:1], gate_up=fused[1:2], o_f=fused[2:3],
                          down=fused[3:4], head=small_module(), head_f=fused[4], reducer=None)
    assert CobaltDecoder.device_status(dec) == 0
    for f in fused:
        at = (-f._scratch.data_ptr()) % 256                 # the kernels' status word: the first aligned byte
        f._scratch[at] = 3
        assert f.device_status() == 3 and CobaltDecoder.device_status(dec) == 3
        f._scratch[at] = 0
    CobaltDecoder._check_prompt_attention(dec)
    word.fill_(5)
    assert CobaltDecoder.device_status(dec) == 5
    with pytest.raises(CobaltError, match="prompt"):
        CobaltDecoder._check_prompt_attention(dec)
    assert int(word) == 0


def test_modules_whose_call_runs_more_than_their_kernel():
    """Hooks, replaced and overridden forwards: a fused launch must not stand in for the call."""
    class Sub(CobaltSparseLinear):
        def forward(self, x):
            return super().forward(x)

    plain = small_module()
    assert called_plainly(plain)
    sub = small_module()
    sub.__class__ = Sub
    replaced = small_module()
    replaced.forward = lambda x: x
    compiled = small_module()
    compiled._compiled_call_impl = lambda x: x
    assert not any(called_plainly(m) for m in (sub, replaced, compiled))
    noop = lambda *a: None
    for register in (plain.register_forward_hook, plain.register_forward_pre_hook, plain.register_full_backward_hook,
                     plain.register_full_backward_pre_hook, torch.nn.modules.module.register_module_forward_hook,
                     torch.nn.modules.module.register_module_forward_pre_hook):
        handle = register(noop)
        assert not called_plainly(plain)
        handle.remove()
        assert called_plainly(plain)


def test_how_many_prompts_run_together():
    """As many as fit the rows that the caller allows; one by one where it says so, and where a module's call runs more than its kernel."""
    dec = SimpleNamespace(world=1, prompt_kernel=True, fused_prompt_attention=False, B=8, prompt_rows=8192, lin={0: small_module()}, head=None)
    at_once = lambda T: CobaltDecoder._prompts_at_once(dec, T)
    assert [at_once(T) for T in (16, 17, 1000, 1024, 1025, 4096, 4097, 20000)] == [1, 8, 8, 8, 7, 2, 1, 1]
    dec.prompt_rows = 400
    assert [at_once(T) for T in (100, 133, 201)] == [4, 3, 1]
    dec.prompt_rows = 0
    assert at_once(100) == 1
    dec.prompt_rows = 8192
    dec.head = small_module()
    dec.head.register_forward_hook(lambda *a: None)
    assert at_once(100) == 1
