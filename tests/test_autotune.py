"""What the launch-shape tuner times: the plain FP64 classes above order 32 shape the launch
behind the fixed-point kernels, so their matrices must lie outside fixed point (diagonals
beyond 2^800); every other class keeps its own. CPU: the timed call is replaced."""
import importlib.util
import os

import numpy as np

from conftest import ROOT


def load():
    path = os.path.join(ROOT, "kblas-gpu_gb300", "autotune.py")
    spec = importlib.util.spec_from_file_location("kblas_autotune_test", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


class FakeHandle:
    ptr = None

    def __init__(self, stream=None):
        pass

    def allocate_workspace(self):
        return 1

    def close(self):
        pass


class FakeLib:
    def __getattr__(self, name):
        return lambda *a: 1


class FakeKb:
    Handle = FakeHandle
    lib = staticmethod(FakeLib)
    check = staticmethod(lambda *a: None)


class FakeTorch:
    class cuda:
        @staticmethod
        def current_stream():
            return type("S", (), {"cuda_stream": 0})

        @staticmethod
        def synchronize():
            pass


def test_plain_classes_time_the_fp64_launch(monkeypatch):
    at = load()
    real = at.ClassBatch

    class Batch(real):
        def __init__(self, torch, lo, hi, seed=0):
            self.lo, self.hi, self.max_n, self.batch = lo, hi, hi, 4
            self.A0 = self.A0_form = np.full(4, 2.0 * hi)
            self.A, self.B, self.B0 = Copy(4), Copy(4), np.zeros(4)

    class Copy(np.ndarray):
        def __new__(cls, n):
            return np.zeros(n).view(cls)

        def copy_(self, other):
            self[...] = other

    seen = []

    def timed(torch, kb, h, cb, mixed, reps):
        cb.restore()
        seen.append((mixed, cb.hi, float(cb.A.max())))
        return 1.0

    monkeypatch.setattr(at, "ClassBatch", Batch)
    monkeypatch.setattr(at, "time_call", timed)
    monkeypatch.setattr(at, "set_table", lambda *a: None)
    at.tune(FakeTorch, FakeKb, reps=1, log=lambda *a: None)
    assert {hi for mixed, hi, _ in seen if not mixed} == set(at.CLASS_TOP)
    for mixed, hi, top in seen:
        if not mixed and hi > 32:
            assert 2.0 ** 800 <= top < np.inf
        else:
            assert top == 2.0 * hi
