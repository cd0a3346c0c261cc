"""Embedding lookup in one launch against the tensor-library form, ids outside the table included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of one vector, of part of a warp's 512 bytes, of exactly that and of one vector more; 4 and 2 byte types
@pytest.mark.parametrize("D,dtype", [(8, torch.bfloat16), (40, torch.float32), (256, torch.bfloat16), (264, torch.bfloat16),
                                     (4096, torch.float16), (12, torch.bfloat16)])
@pytest.mark.parametrize("shape", [(1,), (3, 1), (7, 33)])
@pytest.mark.parametrize("kind", [torch.int64, torch.int32, torch.float32])
def test_lookup_equals_the_masked_form(D, dtype, shape, kind):
    from ghost_flow_b200.nn import Embedding

    e = Embedding(11, D, device="cuda", dtype=dtype)
    ids = torch.randint(-3, 14, shape, device="cuda").to(kind)
    with torch.no_grad():
        got = e(ids)
    want = e(ids)                                    # with a gradient to record: the tensor-library form
    assert want.requires_grad and not got.requires_grad
    assert got.shape == (*shape, D) and torch.equal(got, want.detach())
    if len(shape) == 2:
        with torch.no_grad():
            assert torch.equal(e(ids.t()), want.detach().transpose(0, 1))


def test_traced_and_transformed_calls_keep_the_tensor_library_form():
    from torch.autograd import forward_ad

    from ghost_flow_b200.nn import Embedding

    e = Embedding(6, 8, device="cuda").requires_grad_(False)
    ids, other = torch.tensor([[1, 7, 2]], device="cuda"), torch.tensor([[5, 0, -1]], device="cuda")
    want = e(other)
    assert torch.equal(torch.vmap(e)(other), want)
    with torch.no_grad():
        assert torch.equal(torch.jit.trace(e, ids)(other), want)
    with forward_ad.dual_level():
        w = forward_ad.make_dual(e.weight.detach(), torch.ones_like(e.weight))
        tangent = forward_ad.unpack_dual(torch.func.functional_call(e, {"weight": w}, (other,))).tangent
    assert torch.equal(tangent, torch.ones_like(want) * (want.abs().sum(-1, keepdim=True) > 0))
    e.weight = torch.nn.Parameter(torch.ones(8, 8, device="cuda"), requires_grad=False)    # more rows than ids that count
    assert e(ids)[0, 1].count_nonzero().item() == 0


def test_a_table_off_the_current_device_keeps_the_tensor_library_form(monkeypatch):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.nn import Embedding
    from ghost_flow_b200.ops import _lib

    e = Embedding(6, 8, device="cuda").requires_grad_(False)
    ids = torch.tensor([[1, 7, 2]], device="cuda")
    want = e(ids)
    other = torch.cuda.current_device() + 1
    monkeypatch.setattr(torch.cuda, "current_device", lambda: other)
    n0 = _lib.launch_count()
    assert ops.embedding_rows(ids, e.weight) is None and torch.equal(e(ids), want) and _lib.launch_count() == n0
