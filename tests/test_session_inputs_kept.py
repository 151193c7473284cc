"""A session's frames are read in place after submit returns, so the wrapper
holds every submitted frame's arrays until wait has returned (the library's
calls are replaced here: only the lifetime is looked at)."""
from __future__ import annotations

import gc
import weakref

import numpy as np
import pytest

from yetanotherslam_gb300 import _lib as L
from yetanotherslam_gb300 import rgbdfusion as rf


def _session(monkeypatch, submit_code=0):
    class Fake:
        def __getattr__(self, name):
            return lambda *a: submit_code if name == "yas_session_submit" else 0

    fake = Fake()
    monkeypatch.setattr(L, "load", lambda: fake)
    monkeypatch.setattr(rf, "session_config", lambda *a: L.SessionConfig())
    return rf.Session(8, 6, (1, 1, 0, 0))


def _frame():
    return np.zeros((6, 8, 3), np.uint8), np.zeros((6, 8), np.uint16)


def _submit(s, refs):
    rgb, depth = _frame()
    refs += [weakref.ref(rgb), weakref.ref(depth)]
    s.submit(rgb, depth)


def test_arrays_of_every_submitted_frame_live_until_wait(monkeypatch):
    s, refs = _session(monkeypatch), []
    for _ in range(3):
        _submit(s, refs)
    gc.collect()
    assert all(r() is not None for r in refs)
    s.wait()
    gc.collect()
    assert all(r() is None for r in refs)


def test_copies_made_for_the_call_live_until_wait(monkeypatch):
    s, made = _session(monkeypatch), []
    copy = np.ascontiguousarray

    def noted(a, *args, **kw):
        out = copy(a, *args, **kw)
        made.append(weakref.ref(out))
        return out

    monkeypatch.setattr(np, "ascontiguousarray", noted)
    for _ in range(2):
        s.submit(np.zeros((6, 16, 3), np.uint8)[:, ::2], np.zeros((6, 16), np.uint16)[:, ::2])
    gc.collect()
    assert len(made) == 4 and all(r() is not None for r in made)
    s.wait()
    gc.collect()
    assert all(r() is None for r in made)


def test_a_refused_frame_is_held_too(monkeypatch):
    s, refs = _session(monkeypatch, submit_code=3), []
    with pytest.raises(Exception):
        _submit(s, refs)
    assert len(s._keep) == 1
    s.wait()
    gc.collect()
    assert all(r() is None for r in refs)
