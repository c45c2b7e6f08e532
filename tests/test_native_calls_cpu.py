"""The calls of the CPython extension, as far as they go without a GPU: what
reaches the library, seen through stand-ins for it."""
import copy
import ctypes as C
import gc
import importlib.machinery
import importlib.util
import os
import pickle
import subprocess
import sys
import sysconfig

import numpy as np
import pytest
import torch

import fbgemm_b200 as F
from fbgemm_b200 import _capi
from fbgemm_b200 import build, tbe
from fbgemm_b200 import embedding as E

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


class FakeLibrary:
    """Hands out table sets and counts how often each is given back."""

    def __init__(self):
        self.destroyed = {}

    def fbgemm_b200_table_set_create(self, ctx, calls, columns, n, out):
        out._obj.value = 1000 + len(self.destroyed)
        self.destroyed[out._obj.value] = 0
        return 0

    def fbgemm_b200_table_set_destroy(self, handle):
        self.destroyed[handle] += 1


@pytest.mark.parametrize("how", [copy.copy, copy.deepcopy, lambda op: pickle.loads(pickle.dumps(op))])
def test_copies_of_an_operator_give_back_one_table_set_each(monkeypatch, how):
    library = FakeLibrary()
    monkeypatch.setattr(_capi, "lib", lambda: library)
    monkeypatch.setattr(E, "get_context", lambda device: type("Ctx", (), {"handle": None}))
    k = object.__new__(F.SpmdmKernel)
    k.cfg = _capi.SpmdmConfig()
    op = object.__new__(tbe.IntNBitTableBatchedEmbeddingBags)
    op.T, op.kernels, op.rows, op.D_offsets, op.device = 1, [k], [3], np.array([0, 4]), torch.device("cpu")
    op.tables = [torch.zeros(48, dtype=torch.uint8)]
    op._plans, op._set = {}, None
    op._table_set()
    other = how(op)
    other._table_set()
    assert other._table_set().handle is not None and len(library.destroyed) == 2
    del op
    gc.collect()
    assert sorted(library.destroyed.values()) == [0, 1]
    del other
    gc.collect()
    assert list(library.destroyed.values()) == [1, 1]


# ---- the extension's file ----------------------------------------------------------

def test_another_interpreter_builds_its_own_extension(monkeypatch):
    assert os.path.basename(build.NATIVE_PATH) == "_native_calls" + sysconfig.get_config_var("EXT_SUFFIX")
    stamp = build._fingerprint()
    monkeypatch.setattr(build, "NATIVE_PATH", build.NATIVE_PATH.replace("cpython-3", "cpython-9"))
    assert build._fingerprint() != stamp
    assert build.needs_build()


def test_an_extension_that_could_not_be_built_is_named(monkeypatch):
    def no_compiler():
        raise RuntimeError("no Python.h here")

    _capi.lib()
    monkeypatch.setattr(build, "needs_build", lambda: True)
    monkeypatch.setattr(build, "build", no_compiler)
    for name in ("_lib", "_native", "_build_error"):
        monkeypatch.setattr(_capi, name, None)
    monkeypatch.setitem(sys.modules, "fbgemm_b200._native_calls", None)
    monkeypatch.delattr(F, "_native_calls", raising=False)
    _capi.lib()
    with pytest.raises(_capi.Fbgemmb200Error, match="_native_calls.*no Python.h here"):
        _capi.native()


# ---- the extension itself, over stand-ins for the library's functions ------------

@pytest.fixture(scope="module")
def stubbed(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("native") / "_native_calls.so")
    subprocess.run(["gcc", "-O1", "-Wall", "-shared", "-fPIC", "-I", build.INCLUDE, "-I", sysconfig.get_paths()["include"],
                    os.path.join(build.CSRC, build.NATIVE_SOURCE), os.path.join(ROOT, "tests", "cpp", "native_calls_stub.c"),
                    "-o", path], check=True)
    loader = importlib.machinery.ExtensionFileLoader("_native_calls", path)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_native_calls", loader))
    loader.exec_module(module)
    return module


class Array(FakeTensor):
    def is_contiguous(self):
        return True


#: name -> arguments: "h" a handle, "t" a tensor, numbers as they are
CALLS = {
    "spmdm_launch": ["h", "h", 1, 1, 1, "t", "t", "t", "t", "t", "t", 0, "h"],
    "spmdm": ["h", "h", 1, 1, 1, "t", "t", "t", "t", "t", "t", "h"],
    "table_set_forward": ["h", 1, "t", 1, "t", "t", "t", 0, "h"],
    "quantize": [0, "t", 1, 4, "t", "h"],
    "pruned_lookup": [1, "h", 1, 1, "t", "t", 8, 1, "t", 8, "t", "t", 0, "h"],
    "sequence_lookup": [1, "h", "t", "t", 1, 1, 4, "t", "t", 8, 1, "t", 0, 16, 1, 4, 7, 0, "h"],
}


def arguments(name):
    return [1 << 16 if a == "h" else Array() if a == "t" else a for a in CALLS[name]]


def test_every_call_of_the_extension_is_listed(stubbed):
    assert set(CALLS) == {n for n in dir(stubbed) if not n.startswith("_")}


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("first", [0, 1, 4])   # the calls that choose between two entry points choose by it
def test_calls_give_up_the_interpreters_lock(stubbed, name, first):
    """A launch waits while the stream's queue is full, and lengths mode may lock or allocate: other Python threads, on
    which that may depend, run on meanwhile."""
    args = arguments(name)
    if isinstance(CALLS[name][0], int):
        args[0] = first
    assert getattr(stubbed, name)(*args) == 0, "the lock was held"


@pytest.mark.parametrize("name", CALLS)
def test_numbers_are_no_tensors(stubbed, name):
    """Handles and streams are numbers; where an array is due a number is refused, not taken for its address."""
    for i, kind in enumerate(CALLS[name]):
        args = arguments(name)
        if kind == "t":
            for wrong in (0, 1 << 20, True, 1.5):
                args[i] = wrong
                with pytest.raises((TypeError, AttributeError)):
                    getattr(stubbed, name)(*args)
            args[i] = None
            getattr(stubbed, name)(*args)
        elif kind == "h":
            args[i] = Array()
            with pytest.raises(TypeError):
                getattr(stubbed, name)(*args)


def test_strided_tensors_and_pageable_arrays_are_refused(stubbed):
    class Strided(FakeTensor):
        def is_contiguous(self):
            return False

    for wrong, error in ((Strided(), AssertionError), (np.zeros(4), TypeError), (np.zeros((4, 4))[:, 1], AssertionError)):
        args = arguments("spmdm_launch")
        args[6] = wrong
        with pytest.raises(error):
            stubbed.spmdm_launch(*args)
