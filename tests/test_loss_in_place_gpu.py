"""fbw_loss and fbw_loss_cached read float32 CUDA log_probs as they are; against the op on a negated, transposed
copy, for the layouts a caller's tensor can have, and with a graph that is kept for a second backward pass."""
import pytest
import torch

from i6_native_ops_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["contiguous", "transposed", "offset", "strided", "negated"])
@pytest.mark.parametrize("cached", [False, True])
def test_same_as_the_op_on_a_copy(cuda, layout, cached):
    import i6_native_ops_b200.fbw as m

    batch = wl.make_batch("ctc_tiny")
    fsa, lens = wl.to_torch(batch, cuda)
    am = wl.make_scores(batch, cuda)  # (T, B, F) negative log scores
    T, B, F = am.shape
    lp = am.neg().transpose(0, 1)
    if layout == "contiguous":
        x = lp.contiguous()
    elif layout == "transposed":
        x = lp
    elif layout == "offset":  # not aligned to 16 bytes
        x = torch.empty(B * T * F + 1, device=cuda)[1:].view(B, T, F).copy_(lp)
    elif layout == "negated":  # a view whose sign is a bit of the tensor: the memory holds the negated values
        x = torch._neg_view(lp.neg().contiguous())
    else:
        x = torch.empty(B, T, F, 2, device=cuda)[..., 0].copy_(lp)
    x = x.detach().requires_grad_(True)
    cache = m.PlanCache()

    def loss_of(t):
        return m.fbw_loss_cached(t, fsa, lens, cache) if cached else m.fbw_loss(t, fsa, lens)

    y = x.detach().clone().requires_grad_(True)
    want = m.FastBaumWelchLoss.apply(y.neg().transpose(0, 1).contiguous(), fsa, lens)
    (want_grad,) = torch.autograd.grad(want.sum(), y)
    loss = loss_of(x)
    assert torch.equal(loss, want)
    (first,) = torch.autograd.grad(loss.sum(), x, retain_graph=True)
    # exp of the same values by two implementations, each within 2 ulp of values at most 1
    assert float((first - want_grad).abs().max()) <= 4 * 2.0 ** -23
    first.zero_()  # the caller's to change; the kept graph gives the gradient again
    (second,) = torch.autograd.grad(loss.sum(), x)
    assert float((second - want_grad).abs().max()) <= 4 * 2.0 ** -23
    assert second.shape == x.shape
