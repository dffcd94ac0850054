"""NVTX ranges that cost nothing on CPU (reference: odc/fsdp/fsdp2.py:54-61)."""
from __future__ import annotations

import torch
from torch.profiler import record_function

from .. import config


_cuda = False


def _enabled() -> bool:
    global _cuda
    if not _cuda:
        _cuda = torch.cuda.is_available()   # asked until it is true, then remembered
    return _cuda and config.nvtx_enabled()


class nvtx_range:
    """``with nvtx_range(name):`` opens an NVTX range when NVTX is on and a GPU is there."""

    __slots__ = ("name", "on")

    def __init__(self, name: str):
        self.name = name

    def __enter__(self):
        self.on = _enabled()
        if self.on:
            torch.cuda.nvtx.range_push(self.name)

    def __exit__(self, *exc):
        if self.on:
            torch.cuda.nvtx.range_pop()


class nvtx_record_function(record_function):
    """``record_function`` that also opens an NVTX range, so FSDP phases show up in Nsight."""

    def __enter__(self):
        self._nvtx = _enabled()
        if self._nvtx:
            torch.cuda.nvtx.range_push(self.name)
        return super().__enter__()

    def __exit__(self, exc_type, exc_value, traceback):
        super().__exit__(exc_type, exc_value, traceback)
        if self._nvtx:
            torch.cuda.nvtx.range_pop()
