"""Two host threads on one operator.  Each one's single operations run on its own
current stream of torch; the library lets one thread in at a time from
pdg_run_on to pdg_run_done.  On CPU with a fake library that has that rule, and
on the GPU with results."""
import ctypes
import sys
import threading
import types

import numpy as np
import pytest

WAIT = 10.0        # seconds after which a hand-over between the threads has failed


class _FakeLib:
    """pdg_run_on .. pdg_run_done as in pdg.h; what ran, on which stream."""

    def __init__(self):
        self.mutex, self.stream, self.ran = threading.Lock(), "own", []
        self.waiting = {}              # thread -> it has called pdg_run_on

    def pdg_run_on(self, h, stream):
        self.waiting.setdefault(threading.get_ident(), threading.Event()).set()
        if not self.mutex.acquire(timeout=WAIT):
            return 5
        self.stream = stream
        return 0

    def pdg_run_done(self, h):
        self.stream = "own"
        self.mutex.release()
        return 0


def test_each_thread_runs_on_its_own_stream(monkeypatch):
    import pdg
    lib, local = _FakeLib(), threading.local()
    monkeypatch.setattr(pdg, "load", lambda *a: lib)
    cuda = types.SimpleNamespace(
        is_initialized=lambda: True,
        current_stream=lambda device=None: types.SimpleNamespace(cuda_stream=local.stream))
    monkeypatch.setitem(sys.modules, "torch", types.SimpleNamespace(cuda=cuda))
    go = types.SimpleNamespace(_h=ctypes.c_void_p(1), _explicit_stream=False, _lib_stream=None,
                               _running=None, cfg=types.SimpleNamespace(device=0))
    inside, b_seen, errors = threading.Event(), threading.Event(), []

    class Op:
        def __init__(self):
            self.go = go

        @pdg._on_current_stream
        def apply(self, name):
            lib.ran.append((name, lib.stream))
            if name == "A":
                inside.set()
                b_seen.wait(WAIT)      # until B has tried to come in
            return self.nested(name)

        @pdg._on_current_stream
        def nested(self, name):        # within the same thread: no second pdg_run_on
            lib.ran.append((name, lib.stream))
            return name

    def thread(name, stream):
        try:
            local.stream = stream
            if name == "B":
                inside.wait(WAIT)
                lib.waiting[threading.get_ident()] = b_seen
            assert Op().apply(name) == name
        except Exception as e:
            errors.append(e)
        finally:
            if name == "B":
                b_seen.set()

    ts = [threading.Thread(target=thread, args=a) for a in (("A", 1), ("B", 2))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    assert lib.ran == [("A", 1), ("A", 1), ("B", 2), ("B", 2)]
    assert go._running is None


def test_stream_bound_by_a_c_call(monkeypatch):
    """pdg_run_on refuses while a stream is bound; a binding that did not bind it
    itself orders against that stream with events, as every other call does."""
    import pdg
    log = []

    class Stream:
        def __init__(self, name):
            self.name, self.cuda_stream = name, 7

        def wait_stream(self, other):
            log.append(f"{self.name} waits {other.name}")

    def get_stream(h, out):
        out._obj.value = 0x1000
        return pdg.PDG_OK

    lib = types.SimpleNamespace(pdg_run_on=lambda h, s: pdg.PDG_ESTATE, pdg_get_stream=get_stream)
    monkeypatch.setattr(pdg, "load", lambda *a: lib)
    cuda = types.SimpleNamespace(is_initialized=lambda: True,
                                 ExternalStream=lambda ptr, device=None: Stream("bound"),
                                 current_stream=lambda device=None: Stream("torch"))
    monkeypatch.setitem(sys.modules, "torch",
                        types.SimpleNamespace(cuda=cuda, device=lambda *a: a))
    go = types.SimpleNamespace(_h=ctypes.c_void_p(1), _explicit_stream=False, _lib_stream=None,
                               _running=None, cfg=types.SimpleNamespace(device=0))

    class Op:
        def __init__(self):
            self.go = go

        @pdg._on_current_stream
        def apply(self):
            log.append("call")
            return 7

    assert Op().apply() == 7
    assert log == ["bound waits torch", "call", "torch waits bound"]


@pytest.mark.gpu
def test_threads_on_one_operator():
    """Applies of two threads behind writes on their own streams, beside a third
    one's solves: the results are those of one thread."""
    import pdg
    import torch
    rng = np.random.default_rng(1)
    go = pdg.GridOperator(3, 2, (12, 11, 10), alpha=3.0)
    go.set_permeability(np.exp(rng.standard_normal(go.ncell)))
    go.set_source(fc=np.ones(go.ncell))
    op = pdg.OnTheFlyOperator(go)
    xs = [torch.tensor(rng.uniform(-1, 1, go.ndof), device="cuda") for _ in range(2)]
    refs = [torch.zeros_like(x) for x in xs]
    for x, r in zip(xs, refs):
        op.apply(x, r)
    u = torch.zeros_like(xs[0])
    ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go)
    slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-8)
    slp.apply()
    uref = u.clone()
    torch.cuda.synchronize()
    errors = []

    def applies(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for n in range(100):
                    if n % 20 == 0:
                        torch.cuda._sleep(2_000_000)
                    x = xs[i] * 1.0
                    y = torch.zeros_like(x)
                    op.apply(x, y)
                    d = (y - refs[i]).abs().max()
                    if float(d) != 0.0:
                        raise AssertionError(f"thread {i}, apply {n}: {float(d)}")
        except BaseException as e:
            errors.append(e)

    def solves():
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for n in range(10):
                    u.zero_()
                    slp.apply()
                    if not torch.equal(u, uref):
                        raise AssertionError(f"solve {n}")
        except BaseException as e:
            errors.append(e)

    ts = [threading.Thread(target=applies, args=(i,)) for i in range(2)]
    ts.append(threading.Thread(target=solves))
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    go.close()


@pytest.mark.gpu
def test_threads_on_their_own_operators():
    """Contexts are independent: 2D solves (one cooperative launch each) of two
    threads, the first of their kind in both."""
    import pdg
    import torch
    out, errors = [[], []], []
    start = threading.Barrier(2)

    def solves(i):
        try:
            go = pdg.GridOperator(2, 2, (24, 20 + i), alpha=3.0)
            rng = np.random.default_rng(i)
            go.set_permeability(np.exp(rng.standard_normal(go.ncell)))
            go.set_source(fc=np.ones(go.ncell))
            u = torch.zeros(go.ndof, dtype=torch.float64, device="cuda")
            ls = pdg.ISTLBackend_SEQ_MatrixFree_Base(go)
            slp = pdg.StationaryLinearProblemSolver(go, ls, u, 1e-8)
            start.wait()
            for _ in range(5):
                u.zero_()
                slp.apply()
                out[i].append(u.cpu().numpy())
            go.close()
        except BaseException as e:
            errors.append(e)

    ts = [threading.Thread(target=solves, args=(i,)) for i in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for o in out:
        assert all(np.array_equal(v, o[0]) for v in o) and np.abs(o[0]).max() > 0
