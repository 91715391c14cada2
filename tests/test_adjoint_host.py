"""The six-unknown settle's host loop with the device's calls faked: the sums a round hands to zeb_settle6 are
still allocated when the call is made (given back earlier, another thread on the stream could be handed their
memory and write it first)."""
import ctypes
import weakref

import pytest

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("gradient,width", [("reference", 43), ("adjoint", 61)])
def test_the_sums_outlive_the_call_that_reads_them(monkeypatch, gradient, width):
    from zebsdsolve_b200 import adjoint

    n, made, calls = 40, [], []

    class Plan:
        def __init__(self):
            self.n = n

        def run(self, mode, x, q):
            sums = torch.zeros(n, width)
            made.append(weakref.ref(sums))
            return sums

    def call(name, sums, w, count, trust, first, state, x, q, parts, stream):
        assert name == "zeb_settle6" and (w, count) == (width, n)
        calls.append((made[-1]() is not None, first))
        ctypes.memset(parts, 0, 8 * 3 * ((n + 31) // 32))  # nothing gained: the loop ends

    monkeypatch.setattr(adjoint.N, "call", call)
    monkeypatch.setattr(adjoint, "stream_ptr", lambda: None)
    q, shift, ncc, rounds = adjoint.refine6(Plan(), torch.randn(n, 4), 0.05, gradient=gradient)
    assert calls == [(True, 1), (True, 0)] and rounds == 0
    assert q.shape == (n, 4) and shift.shape == (n, 3) and ncc.shape == (n,)
