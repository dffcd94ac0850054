"""Host side of the sharded linear layer: what it hands to the native extension (a stand-in here; no GPU)."""
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
