"""Host side of the sharded linear layer: what it hands to the native extension (a stand-in here; no GPU)."""
import pytest
import torch

from odc_b200.parallel import OdcLinear
from odc_b200.parallel import linear as L


class _Extension:
    def __init__(self):
        self.kept = []

    def sharded_linear(self, x, bias, residual, matrix, bias_sink, keep_weight):
        self.kept.append(keep_weight)
        return x


class _OnGpu:
    is_cuda = True


def test_keep_weight_is_read_at_every_call(monkeypatch):
    ext = _Extension()
    monkeypatch.setattr(L.ops, "_ext", lambda: ext)
    layer = OdcLinear.__new__(OdcLinear)
    torch.nn.Module.__init__(layer)
    layer.bias, layer.keep_weight = None, False
    layer.weight = type("Weight", (), {"_matrix": object()})()
    layer(_OnGpu())
    layer.keep_weight = True
    layer(_OnGpu())
    assert ext.kept == [False, True]


def _layer(cls=OdcLinear):
    layer = cls.__new__(cls)
    torch.nn.Module.__init__(layer)
    layer.bias, layer.keep_weight = None, False
    layer.weight = type("Weight", (), {"_matrix": object(), "world": 1})()
    return layer


class _Wrapped(torch.nn.Module):
    def __init__(self, inner):
        super().__init__()
        self.inner = inner

    def forward(self, x, **kw):
        return self.inner(x, **kw)


class _OwnForward(OdcLinear):
    def forward(self, x, *args, **kw):
        return super().forward(x, *args, **kw)


def test_replaced_layers_are_called_and_not_passed_by(monkeypatch):
    """The MLP takes both matrices at once only from layers that are what they were built as."""
    layer = _layer()
    assert L.plain_matrix(layer, _OnGpu()) is layer.weight._matrix
    assert L.plain_matrix(_Wrapped(layer), _OnGpu()) is None
    assert L.plain_matrix(_layer(_OwnForward), _OnGpu()) is None
    patched = _layer()
    patched.forward = lambda *args, **kw: None
    assert L.plain_matrix(patched, _OnGpu()) is None
    monkeypatch.setattr(OdcLinear, "forward", lambda self, x, **kw: x)
    assert L.plain_matrix(layer, _OnGpu()) is None


@pytest.mark.parametrize("everywhere", [False, True])
@pytest.mark.parametrize("register", ["register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook",
                                      "register_full_backward_pre_hook"])
def test_watched_layers_are_called(register, everywhere):
    layer = _layer()
    where, name = (torch.nn.modules.module, register.replace("register", "register_module")) if everywhere else (layer, register)
    handle = getattr(where, name)(lambda *args: None)
    assert L.plain_matrix(layer, _OnGpu()) is None
    handle.remove()
    assert L.plain_matrix(layer, _OnGpu()) is layer.weight._matrix


def _no_op(*args):
    return None


@pytest.mark.parametrize("part", ["attn_norm", "attn", "mlp_norm", "mlp"])
def test_a_layer_is_one_function_only_as_it_was_built(part):
    """Hooks, wrappers, other classes, another forward and hooks on all modules make the layer call its parts."""
    from odc_b200.models import DecoderLayer, get_config
    make = lambda: DecoderLayer(get_config("tiny"))
    layer = make()
    assert layer._as_built()
    for register in ("register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook", "register_full_backward_pre_hook"):
        handle = getattr(getattr(layer, part), register)(_no_op)
        assert not layer._as_built(), register
        handle.remove()
        assert layer._as_built()
    handle = torch.nn.modules.module.register_module_forward_hook(_no_op)
    assert not layer._as_built()
    handle.remove()
    setattr(getattr(layer, part), "forward", _no_op)
    assert not layer._as_built()
    layer = make()
    setattr(layer, part, torch.nn.Identity())
    assert not layer._as_built()
    layer = make()
    mod = getattr(layer, part)
    mod.__class__ = type("Sub", (type(mod),), {})
    assert not layer._as_built()
    layer = make()
    layer.attn.cfg.rope_scaling = {"rope_type": "linear", "factor": 2.0}
    assert not layer._as_built()
