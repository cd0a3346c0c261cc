"""Cross-entropy over the row lengths at which the launch changes, against
fp64: loss and gradient, ignored rows, in place, -inf and all-masked logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# row lengths around a vector, a round of 256 threads, and those at which one CTA less fits an SM (six rows of 34.5 KB, two of
# 108 KB, one above); ragged last vectors; the longest row of all
@pytest.mark.parametrize("V", [5, 8, 1000, 2047, 2056, 17664, 17672, 30522, 50257, 55295, 55304, 102400])
@pytest.mark.parametrize("T", [1, 150, 901])
def test_loss_and_gradient_match_fp64(V, T):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(V + T)
    buf = torch.zeros(T, (V + 63) // 64 * 64, device="cuda", dtype=torch.bfloat16)
    buf[:, :V] = (torch.randn(T, V, generator=g, device="cuda") * 3).bfloat16()
    tg = torch.randint(0, V, (T,), generator=g, device="cuda")
    tg[0] = V - 1
    if T > 2:
        buf[1, : V // 2] = float("-inf")           # a mask over half the classes
        tg[1] = V - 1
        tg[2] = -100
    logits = buf[:, :V]
    logits.requires_grad_(True)
    lg = logits.detach().double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(lg, tg, ignore_index=-100)
    want.backward()
    loss = ops.cross_entropy(logits, tg, ignore_index=-100)
    (dl,) = torch.autograd.grad(loss, logits)
    # fp32 sums of up to 102400 positive terms over T rows; the gradient is one bf16 rounding away (2^-9)
    assert abs(loss.item() - want.item()) < 1e-5 * abs(want.item())
    assert dl.shape == logits.shape and ((dl.double() - lg.grad).norm() / lg.grad.norm()).item() < 4e-3
    assert torch.allclose(dl.double(), lg.grad, rtol=2 ** -7, atol=1e-9)
    if T > 2:
        assert not dl[2].any() and not dl[1, : V // 2].any()
    with torch.no_grad():                          # loss only, no gradient buffer
        assert torch.allclose(ops.cross_entropy(logits.detach(), tg, ignore_index=-100), loss.detach())


@pytest.mark.parametrize("V", [1000, 32000])
def test_rows_without_finite_logits_give_nan(V):
    from ghost_flow_b200 import ops

    x = torch.randn(3, V, device="cuda").bfloat16()
    x[0] = float("-inf")
    x[1, 5] = float("nan")
    x[2, 7] = float("inf")
    for r in range(3):
        assert torch.isnan(ops.cross_entropy(x[r:r + 1], torch.tensor([3], device="cuda")))


def test_in_place_gradient_overwrites_the_logits():
    from ghost_flow_b200.ops import raw

    x = torch.randn(300, 32000, device="cuda").bfloat16()
    tg = torch.randint(0, 32000, (300,), device="cuda")
    p = torch.softmax(x.double(), -1)
    p[torch.arange(300), tg] -= 1
    raw.xent_fwd_bwd(x, tg)
    assert ((x.double() - p / 300).norm() / p.norm() * 300).item() < 4e-3


def test_a_launch_without_a_status_word_is_refused():
    from ghost_flow_b200.ops import _lib

    x, tg, rows = torch.zeros(2, 64, device="cuda").bfloat16(), torch.zeros(2, dtype=torch.int64, device="cuda"), torch.zeros(2, device="cuda")
    args = (x.data_ptr(), tg.data_ptr(), rows.data_ptr(), None, 2, 64, 64, 0.5, -100)
    assert _lib.cuda_lib().gf_xent_fused(*args, None, _lib.stream_ptr()) == -1
    assert _lib.cuda_lib().gf_xent_fused(*args, _lib.status_word().data_ptr(), _lib.stream_ptr()) == 0
