"""Which GPU a launch goes to: the current one of the calling thread, whatever other threads have selected."""
import ctypes
import threading

import torch

from ghost_flow_b200.ops import _lib


def _in_turn(steps):
    """Runs ``steps`` = [(thread number, function)] one after the other, each on its own thread; their results in order."""
    out, turn = [None] * len(steps), threading.Condition()
    at = [0]

    def work(who):
        for i, (t, fn) in enumerate(steps):
            if t != who:
                continue
            with turn:
                assert turn.wait_for(lambda: at[0] == i, 20)
                out[i] = fn()
                at[0] += 1
                turn.notify_all()

    ts = [threading.Thread(target=work, args=(w,)) for w in {t for t, _ in steps}]
    for t in ts:
        t.start()
    for t in ts:
        t.join(30)
    return out


def test_library_keeps_the_device_of_each_thread():
    lib = ctypes.CDLL(str(_lib.lib_path()))
    lib.gf_set_device.argtypes, lib.gf_set_device.restype = [ctypes.c_int], None
    lib.gf_selected_device.argtypes, lib.gf_selected_device.restype = [], ctypes.c_int
    get = lib.gf_selected_device
    got = _in_turn([(0, lambda: lib.gf_set_device(0)), (1, lambda: lib.gf_set_device(1)), (0, get), (1, get), (2, get)])
    # a thread that selected none follows the last selection
    assert got[2:] == [0, 1, 1]
    lib.gf_set_device(0)


def test_each_thread_binds_its_current_device(monkeypatch):
    bound, current = [], threading.local()

    class Lib:
        def gf_set_device(self, d):
            bound.append((threading.current_thread().name, d))

    monkeypatch.setattr(_lib, "cuda_lib", Lib)
    monkeypatch.setattr(_lib, "_RAW_STREAM", lambda d: d)
    monkeypatch.setattr(_lib, "_BOUND", threading.local(), raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current.d)

    def at(d):
        def go():
            current.d = d
            n = len(bound)
            assert _lib.stream_ptr() == d
            return [x for _, x in bound[n:]]
        return go

    # thread 1 binds its own device although thread 0 bound another in between; nobody binds twice
    assert _in_turn([(0, at(0)), (1, at(1)), (0, at(0)), (1, at(1)), (1, at(0))]) == [[0], [1], [], [], [0]]
