"""The stream note of the Python handles against a stand-in for the library's set_stream (no GPU)."""
import threading
from types import SimpleNamespace

import pytest

import fftm_b200 as F


def _stream(raw):
    return SimpleNamespace(cuda_stream=raw)


def _object(monkeypatch, setter):
    """An ffts whose library is a stand-in: only set_stream is there."""
    monkeypatch.setattr(F._lib, "load", lambda: SimpleNamespace(fftb_ffts_set_stream=setter))
    f = F.ffts()
    f._h = SimpleNamespace(value=None)
    return f


def test_set_only_when_the_stream_changes(monkeypatch):
    calls = []
    f = _object(monkeypatch, lambda h, s: calls.append(s) or 0)
    for s in (0, 0, 7, 7, 9, 7, 0):
        f._bind(_stream(s))
    assert calls == [7, 9, 7, 0]


def test_a_refused_set_is_tried_again(monkeypatch):
    status, calls = [-5, 0], []
    f = _object(monkeypatch, lambda h, s: calls.append(s) or status.pop(0))
    monkeypatch.setattr(F._lib, "status_string", lambda st: "refused")
    monkeypatch.setattr(F._lib, "last_error_message", lambda: "")
    with pytest.raises(F.FftbError):
        f._bind(_stream(7))
    f._bind(_stream(7))
    f._bind(_stream(7))
    assert calls == [7, 7]


def test_the_note_follows_the_handle_across_threads(monkeypatch):
    """Thread B has set the handle to stream 2 and has not returned yet when thread A binds stream 1.
    Whichever comes last, the next call on either stream must find the handle on its own."""
    handle = {"stream": 0}
    b_has_set, a_is_done = threading.Event(), threading.Event()

    def setter(h, s):
        handle["stream"] = s
        if s == 2:
            b_has_set.set()
            a_is_done.wait(0.3)  # A gets in here where nothing holds it back
        return 0

    f = _object(monkeypatch, setter)
    b = threading.Thread(target=lambda: f._bind(_stream(2)))

    def a_body():
        b_has_set.wait(5)
        f._bind(_stream(1))
        a_is_done.set()

    a = threading.Thread(target=a_body)
    a.start()
    b.start()
    a.join()
    b.join()
    monkeypatch.setattr(F._lib, "load",
                        lambda: SimpleNamespace(fftb_ffts_set_stream=lambda h, s: handle.update(stream=s) or 0))
    last = handle["stream"]
    for s in (3 - last, last, last):
        f._bind(_stream(s))
        assert handle["stream"] == s
