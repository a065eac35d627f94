"""Split-K workspaces handed out to several threads at once: no buffer whose address was returned is dropped."""

import contextlib
import threading
import time

import torch

from flydsl_b200.kernels.gemm import preshuffle_gemm as pg


def test_first_calls_of_several_threads_share_one_buffer(monkeypatch):
    made, zeros = [], torch.zeros

    def slow_zeros(*a, **kw):
        made.append(1)
        time.sleep(0.02)
        return zeros(*a, **kw)

    monkeypatch.setattr(pg, "_workspaces", {})
    monkeypatch.setattr(pg, "_retired", [])
    monkeypatch.setattr(pg, "_on_stream", lambda device, stream: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch, "zeros", slow_zeros)
    for nbytes in (1 << 16, 1 << 18):  # the second size replaces the buffer
        got = []
        threads = [threading.Thread(target=lambda n=nbytes: got.append(pg._workspace(torch.device("cpu"), 5, n))) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        kept = {w.data_ptr() for w in list(pg._workspaces.values()) + pg._retired}
        assert len(got) == 4 and {p for p, _ in got} <= kept
    assert len(made) == 2
