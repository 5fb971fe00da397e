"""calc_volume and monte_carlo_volume from several threads: one hidden handle per device and precision
serves every caller, and holds one staging buffer and one result. No GPU: a library double whose calls
go through shared state as the handle's do."""
import ctypes as C
import importlib
import threading
import time

import pytest
import torch

from helpers import cc

cache = importlib.import_module("cutcell_b200.cache")


class _Library:
    """cc_calc_volume and cc_monte_carlo_volume through one word per handle: the body's constant goes in, and
    comes out once the "device" is done with it."""

    def __init__(self):
        self.word = None

    def _through(self, tape):
        self.word = C.cast(tape.params, C.POINTER(C.c_double))[0]
        time.sleep(0.002)
        return self.word

    def cc_calc_volume(self, handle, grid, tape, out, stream):
        out._obj.value = self._through(tape._obj)
        return 0

    def cc_monte_carlo_volume(self, handle, tape, lo, hi, n, seed, inside, volume, stream):
        volume._obj.value = self._through(tape._obj)
        return 0


class _Handle:
    made = []

    def __init__(self, *args):
        self.lib, self.h = _Library(), None
        time.sleep(0.002)  # creating one takes a while
        _Handle.made.append(args)


@pytest.mark.parametrize("mixed_calls", [False, True])
def test_threads_get_their_own_result(monkeypatch, mixed_calls):
    monkeypatch.setattr(cache, "_vol_handles", {})
    monkeypatch.setattr(cache, "_Handle", _Handle)
    monkeypatch.setattr(cache, "_stream", lambda device: None)
    monkeypatch.setattr(_Handle, "made", [])
    g = cc.CartesianGrid((0.0, 0.0, 0.0), (2, 2, 2), (0.5,) * 3)
    wrong, start = [], threading.Barrier(6)

    def work(t):
        start.wait()
        for i in range(8):
            want = 100.0 * t + i
            if mixed_calls and t % 2:
                got, _ = cc.monte_carlo_volume(cc.Const(want), (0.0,) * 3, (1.0,) * 3, 10, device=torch.device("cuda", 0))
            else:
                got = cc.calc_volume(cc.Const(want), g, device=torch.device("cuda", 0))
            if got != want:
                wrong.append((t, i, got))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
    assert len(_Handle.made) == 1


def test_a_failed_call_leaves_the_handle_usable(monkeypatch):
    monkeypatch.setattr(cache, "_vol_handles", {})
    monkeypatch.setattr(cache, "_Handle", _Handle)
    monkeypatch.setattr(cache, "_stream", lambda device: None)
    g = cc.CartesianGrid((0.0, 0.0, 0.0), (2, 2, 2), (0.5,) * 3)
    dev = torch.device("cuda", 0)
    with pytest.raises(ValueError):
        cc.calc_volume(cc.Circle((0.0, 0.0), 1.0), g, device=dev)
    assert cc.calc_volume(cc.Const(3.0), g, device=dev) == 3.0
