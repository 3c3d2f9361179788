"""norm_act calls a module whose call is more than its class's forward by itself, with one argument."""
import pytest
import torch

from exact_b200 import layers
from exact_b200.layers import QBatchNorm1d, QReLUDropout, norm_act


class FakeBatchNorm:
    """Stands for the kernels behind QBatchNorm1d, which have no CPU form."""

    @staticmethod
    def apply(input, *args):
        return input + 1


class FakeActivation:
    @staticmethod
    def act_quantized_relu_dropout(input, p, train):
        return input * 2


def replaced_on_instance(module, calls, monkeypatch):
    own = module.forward
    module.forward = lambda *args: (calls.append(args), own(*args))[1]


def replaced_on_class(module, calls, monkeypatch):
    own = type(module).forward
    monkeypatch.setattr(type(module), "forward", lambda self, *args: (calls.append(args), own(self, *args))[1])


def hooked(module, calls, monkeypatch):
    module.register_forward_hook(lambda m, args, out: calls.append(args))


def compiled(module, calls, monkeypatch):
    own = module._call_impl
    module._compiled_call_impl = lambda *args: (calls.append(args), own(*args))[1]


def traced(module, calls, monkeypatch):
    own, watched = torch.nn.Module.__call__, module
    monkeypatch.setattr(torch.nn.Module, "__call__",
                        lambda self, *args: (calls.append(args) if self is watched else None, own(self, *args))[1])


@pytest.mark.parametrize("change", [replaced_on_instance, replaced_on_class, hooked, compiled, traced])
@pytest.mark.parametrize("which", ["norm", "act"])
def test_module_that_is_watched_is_called_by_itself(change, which, monkeypatch):
    monkeypatch.setattr(QBatchNorm1d, "takes_activation", lambda self, input: True)
    monkeypatch.setattr(layers, "qbatch_norm", FakeBatchNorm)
    monkeypatch.setattr(layers, "ext_quantization", FakeActivation)
    norm, act, calls = QBatchNorm1d(4).train(), QReLUDropout(0.5).train(), []
    change(norm if which == "norm" else act, calls, monkeypatch)
    x = torch.ones(3, 4)
    assert torch.equal(norm_act(norm, act, x), (x + 1) * 2)
    assert len(calls) == 1 and len(calls[0]) == 1


def test_forward_of_the_batch_norm_takes_the_input_alone():
    with pytest.raises(TypeError):
        QBatchNorm1d(4).eval()(torch.ones(3, 4), 0.5)
