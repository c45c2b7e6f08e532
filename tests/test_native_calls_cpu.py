"""The calls of the CPython extension, as far as they go without a GPU: what
reaches the library, seen through stand-ins for it."""
import copy
import ctypes as C
import pickle

import numpy as np
import pytest

import fbgemm_b200 as F
from fbgemm_b200 import _capi
from fbgemm_b200 import embedding as E


class FakeTensor:
    """Enough of a CUDA tensor for a call that a stand-in receives."""

    def __init__(self, device=0):
        self._device = device

    def get_device(self):
        return self._device

    def data_ptr(self):
        return 1 << 20

    def element_size(self):
        return 8


class Recorder:
    """Stands in for the extension."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 1 if name == "spmdm" else 0
        return call


@pytest.fixture
def recorder(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(_capi, "_native", r)
    monkeypatch.setitem(E._handles, 0, 1 << 16)
    monkeypatch.setattr(E, "_current_stream", lambda device: 0)
    return r


def kernel():
    return F.GenerateEmbeddingSpMDM(64, False, False, index_dtype=np.int64, offset_dtype=np.int64)


@pytest.mark.parametrize("how", [copy.copy, copy.deepcopy, lambda k: pickle.loads(pickle.dumps(k))])
def test_a_copied_kernel_calls_with_its_own_configuration(recorder, how):
    k = kernel()
    c = how(k)
    assert bytes(c.cfg) == bytes(k.cfg)
    del k
    c.cfg.normalize_by_lengths = 1   # the copy's, as the call has to see it
    t = FakeTensor()
    c.launch(1, 1, 1, t, t, t, None, t)
    assert c(1, 1, 1, t, t, t, None, t)
    for name, args in recorder.calls:
        assert args[1] == C.addressof(c.cfg), name
        assert _capi.SpmdmConfig.from_address(args[1]).normalize_by_lengths == 1
