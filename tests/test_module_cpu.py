"""Host side of the module and of its launches: what needs no GPU."""
import torch

from cobalt_b200 import CobaltSparseLinear


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
