"""The error words that calls reuse: an error is raised once, by the call it
belongs to, and the next call on the stream -- or on another stream or thread --
starts clear; backend().synchronize() keeps a stream's context while there is
no error and names the right invocation after many error-free ones."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _select(bad):
    import torch

    from awkward_gb300 import jagged

    off = torch.tensor([0, 3, 5], dtype=torch.int64, device="cuda")
    x = torch.arange(5, dtype=torch.float32, device="cuda")
    ioff = torch.tensor([0, 1, 2], dtype=torch.int64, device="cuda")
    idx = torch.tensor([2, 7 if bad else -1], dtype=torch.int64, device="cuda")
    return jagged.index_select(off, x, ioff, idx)[1].tolist()


def _alternate():
    for _ in range(3):
        with pytest.raises(ValueError, match="index out of range"):
            _select(True)
        assert _select(False) == [2.0, 4.0]


def test_selection_errors_do_not_stay():
    import torch

    _alternate()
    with torch.cuda.stream(torch.cuda.Stream()):
        _alternate()
    failed = []

    def work():
        try:
            _alternate()
        except BaseException as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def test_backend_context_survives_error_free_synchronisations():
    import torch

    import awkward_gb300

    be = awkward_gb300.backend()
    be.synchronize()
    off = torch.tensor([0, 3, 5], dtype=torch.int64, device="cuda")
    x = torch.arange(5, dtype=torch.float64, device="cuda")
    out = torch.empty(2, dtype=torch.float64, device="cuda")
    total = be["awkward_reduce_sum", np.float64, np.float64, np.int64]
    expand = be.by_name("awkward_ListArray64_getitem_jagged_expand_64")
    i8 = torch.empty(4, dtype=torch.int64, device="cuda")
    for _ in range(3):
        for _ in range(2):
            total(out, x, off, 2)
            be.synchronize()
        total(out, x, off, 2)
        expand(i8, i8.clone(), torch.zeros(3, dtype=torch.int64, device="cuda"), i8.clone(), off[:-1],
               off[1:], 2, 2)
        with pytest.raises(ValueError, match=r"cannot fit jagged slice.*getitem_jagged_expand"):
            be.synchronize()
    total(out, x, off, 2)
    be.synchronize()
    assert out.tolist() == [3.0, 7.0]


def _failing_call(be):
    import torch

    i8 = torch.empty(4, dtype=torch.int64, device="cuda")
    off = torch.tensor([0, 3, 5], dtype=torch.int64, device="cuda")
    return be.by_name("awkward_ListArray64_getitem_jagged_expand_64"), (
        i8, i8.clone(), torch.zeros(3, dtype=torch.int64, device="cuda"), i8.clone(), off[:-1],
        off[1:], 2, 2)


def test_a_late_error_of_another_thread_has_its_own_name():
    """A call whose launch is under way when another thread synchronises the same
    stream: its error is raised once, in its name, by whoever reads it."""
    import torch

    import awkward_gb300

    be = awkward_gb300.backend()
    be.synchronize()
    kernel, args = _failing_call(be)
    torch.cuda.synchronize()
    launching, synchronised = threading.Event(), threading.Event()
    real = kernel._f

    def slow(*cargs):
        launching.set()
        synchronised.wait(1.0)
        return real(*cargs)

    kernel._f = slow
    raised = []
    try:
        other = threading.Thread(target=kernel, args=args)
        other.start()
        assert launching.wait(30)
        for _ in range(2):
            try:
                be.synchronize()
            except ValueError as e:
                raised.append(str(e))
            synchronised.set()
            other.join()
    finally:
        kernel._f = real
    assert len(raised) == 1 and "getitem_jagged_expand" in raised[0]
    be.synchronize()


def test_threads_share_a_stream():
    import torch

    import awkward_gb300

    be = awkward_gb300.backend()
    be.synchronize()
    off = torch.tensor([0, 3, 5], dtype=torch.int64, device="cuda")
    x = torch.arange(5, dtype=torch.float64, device="cuda")
    total = be["awkward_reduce_sum", np.float64, np.float64, np.int64]
    kernel, args = _failing_call(be)
    torch.cuda.synchronize()
    errors, others = [], []

    def work(call, n):
        for _ in range(n):
            try:
                call()
                be.synchronize()
            except ValueError as e:
                errors.append(str(e))
            except BaseException as e:  # noqa: BLE001
                others.append(repr(e))

    outs = [torch.empty(2, dtype=torch.float64, device="cuda") for _ in range(3)]
    threads = [threading.Thread(target=work, args=(lambda o=o: total(o, x, off, 2), 300)) for o in outs]
    threads.append(threading.Thread(target=work, args=(lambda: kernel(*args), 100)))
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    be.synchronize()
    assert not others
    assert 0 < len(errors) <= 100 and all("getitem_jagged_expand" in e for e in errors)
    assert all(o.tolist() == [3.0, 7.0] for o in outs)


@pytest.mark.parametrize("failing", ["awkward_gb300_jagged_index_select", "read_words"])
def test_a_call_that_fails_midway_leaves_no_error_behind(monkeypatch, failing):
    """The kernel has raised its error, and the call ends before it has read it: by a
    return code, or by the read itself (as during a capture)."""
    from awkward_gb300 import _abi

    assert _select(False) == [2.0, 4.0]
    real_cfunc, real_read = _abi.ext_cfunc, _abi.read_words

    def cfunc(name):
        f = real_cfunc(name)
        return (lambda *args: f(*args) or 2) if name == failing else f

    def read(*args):
        raise RuntimeError("read_words: cudaError 900")

    with monkeypatch.context() as m:
        m.setattr(_abi, "ext_cfunc", cfunc)
        if failing == "read_words":
            m.setattr(_abi, "read_words", read)
        with pytest.raises(RuntimeError, match="cudaError"):
            _select(True)
    assert _select(False) == [2.0, 4.0]
    _alternate()
