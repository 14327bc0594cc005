"""The bias of a compressed linear, whatever way it is held (a stand-in tensor takes the place of the GPU)."""
import pytest

torch = pytest.importorskip("torch")


class Stand:
    shape = (3, 2)

    def linear(self, x, bias=None):
        y = x.float().sum(-1, keepdim=True).expand(*x.shape[:-1], 3).to(torch.bfloat16)
        return y if bias is None else y + bias


def module(bias):
    from georefine_b200.serving import BctxLinear

    return BctxLinear(Stand(), None if bias is None else torch.nn.Parameter(bias, requires_grad=False))


BIAS, X = torch.tensor([1.0, 2.0, 3.0]), torch.ones(1, 2, dtype=torch.bfloat16)


def test_a_bias_of_any_kind_is_added():
    assert module(None)(X).tolist() == [[2.0, 2.0, 2.0]]
    for dtype in (torch.bfloat16, torch.float32):
        assert module(BIAS.to(dtype))(X).tolist() == [[3.0, 4.0, 5.0]]
    plain = module(BIAS)
    del plain.bias
    plain.bias = BIAS * 2
    assert plain(X).tolist() == [[4.0, 6.0, 8.0]]
    swapped = module(BIAS)
    assert torch.func.functional_call(swapped, {"bias": BIAS * 3}, (X,)).tolist() == [[5.0, 8.0, 11.0]]
    assert swapped.forward_calls == 1


def test_a_parametrized_bias_is_added():
    from torch.nn.utils import parametrize

    class Negated(torch.nn.Module):
        def forward(self, b):
            return -b

    layer = module(BIAS)
    parametrize.register_parametrization(layer, "bias", Negated())
    assert layer(X).tolist() == [[1.0, 0.0, -1.0]] and layer.forward_calls == 1
