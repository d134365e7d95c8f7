"""CPU tests of the host path around the kernels: what a call may still read after it has returned,
which descriptors an optimizer step uses, and what the C-ABI call layer refuses. The GPU is replaced by
a queue of deferred operations where the order of host and device work matters."""
import contextlib
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


class _Queue:
    """A stream that runs nothing until someone waits for it: the slowest GPU there can be."""

    def __init__(self):
        self.ops = []

    def push(self, op):
        self.ops.append(op)
        return len(self.ops)

    def drain(self, upto=None):
        upto = len(self.ops) if upto is None else upto
        for i in range(upto):
            if self.ops[i] is not None:
                op, self.ops[i] = self.ops[i], None
                op()


def _graphed_model(monkeypatch, queue):
    """StackedMAG with everything but step_graphed itself replaced; replay() notes the static inputs that
    the step would have trained on."""
    from nl_hecate_b200.stacked_mag import StackedMAG

    class Event:
        def __init__(self, *a, **k):
            self.at = 0

        def record(self, *a):
            self.at = queue.push(lambda: None)

        def synchronize(self):
            queue.drain(self.at)

    class Graph:
        def replay(self):
            queue.push(lambda: m.trained_on.append((int(m._static_tok.t[0]), int(m._static_tgt.t[0]))))

    class Stream:
        def wait_stream(self, s):
            pass

    class Static:
        def __init__(self, t):
            self.t = t

        def copy_(self, src, non_blocking=False):
            queue.push(lambda: self.t.copy_(src))

    nothing = lambda *a, **k: None
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", nothing)
    monkeypatch.setattr(torch.cuda, "empty_cache", nothing)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(torch.cuda, "graph", lambda g: contextlib.nullcontext())
    m = StackedMAG.__new__(StackedMAG)
    m.step = m.sync_gradients = m._device_update = m._host_schedule = nothing
    m.forward_backward = lambda *a: torch.zeros(())
    m.opt = type("Opt", (), {"upload": nothing})()
    m.trained_on = []
    # the first call captures; the static inputs that it clones become deferred buffers
    inputs = torch.zeros(1), torch.zeros(1)
    clone = torch.Tensor.clone
    with monkeypatch.context() as mp:
        mp.setattr(torch.Tensor, "clone", lambda t: Static(clone(t)))
        m.step_graphed(*inputs)
    queue.drain()
    m.trained_on.clear()
    return m


@pytest.mark.parametrize("buffers", [1, 2])
def test_graphed_step_has_read_its_inputs_when_it_returns(monkeypatch, buffers):
    """A loader refills one pinned buffer, or two in turn, as soon as a call returned: every step must
    train on what the buffers held when it was called."""
    queue = _Queue()
    m = _graphed_model(monkeypatch, queue)
    host = [(torch.zeros(1), torch.zeros(1)) for _ in range(buffers)]
    for step in range(6):
        tok, tgt = host[step % buffers]
        tok.fill_(step), tgt.fill_(100 + step)
        m.step_graphed(tok, tgt)
    queue.drain()
    assert m.trained_on == [(s, 100 + s) for s in range(6)]


@pytest.mark.parametrize("form", ["plain", "double", "transposed", "per head"])
def test_carried_memory_takes_every_form_that_copy_takes(monkeypatch, form):
    """The row-gather kernel writes n x d*d contiguous fp32 values: a carry of another type, stride or
    shape is copied by torch as before (and refused by it where the shapes do not match)."""
    from nl_hecate_b200 import stacked_mag as sm
    n, s, d = 3, 5, 4
    ms = torch.randn(n, s + 1, d * d)
    kernel = []
    monkeypatch.setattr(sm.D, "titans_forward_dd", lambda *a, **k: (ms, None, torch.zeros(n, s, d)))
    monkeypatch.setattr(sm.D, "call", lambda name, **k: kernel.append((name, k)))
    ctx = type("Ctx", (), {"save_for_backward": lambda self, *t: None})()
    carry = {"plain": torch.zeros(n, d * d), "double": torch.zeros(n, d * d, dtype=torch.float64),
             "transposed": torch.zeros(d * d, n).t(), "per head": torch.zeros(1, n, d * d)}[form]
    x = torch.zeros(n, s, d)
    version = carry._version
    sm._TitansMemory._forward(ctx, x, x, x, x, x, x, ms[:, 0], ms[:, 0], 0, carry)
    if form == "plain":
        assert [c[0] for c in kernel] == ["nlh_copy_rows"] and carry._version > version
    else:
        assert not kernel and torch.equal(carry.reshape(n, d * d).float(), ms[:, -1])
    with pytest.raises(RuntimeError):
        sm._TitansMemory._forward(ctx, x, x, x, x, x, x, ms[:, 0], ms[:, 0], 0, torch.zeros(n - 1, d * d))


def _rows(opt):
    return opt._desc_rows[opt._row]


def test_prepare_reads_clamp_and_no_decay_at_every_step():
    """Both are public attributes: a change between two steps counts from the next step on, in every row of
    the descriptor ring; an index that names no tensor names none."""
    from nl_hecate_b200.optimizer import RING, FlatAdamW
    opt = FlatAdamW([8, 8, 8], device="cpu", weight_decay=0.1, clamp={1: (-1.0, 1.0)}, no_decay=[0, -1, 7])
    for i in range(2 * RING + 1):
        if i == RING - 1:
            opt.clamp[2] = (-2.0, 3.0)
            del opt.clamp[1]
            opt.no_decay = {2}
        opt.prepare([1, 1, 1])
        r = _rows(opt)
        changed = i >= RING - 1
        assert list(r["has_clamp"]) == ([0, 0, 1] if changed else [0, 1, 0])
        assert list(r["clamp_lo"]) == ([0, 0, -2] if changed else [0, -1, 0])
        assert list(r["clamp_hi"]) == ([0, 0, 3] if changed else [0, 1, 0])
        assert [x > 0 for x in r["weight_decay"]] == ([True, True, False] if changed else [False, True, True])


def test_prepare_takes_one_step_count_and_flag_per_tensor():
    """Anything that can be indexed by tensor, more entries than tensors among it; too few are refused."""
    from nl_hecate_b200.optimizer import FlatAdamW
    opt = FlatAdamW([8, 8, 8], device="cpu")
    want = [1.0 / (1.0 - 0.9 ** t) for t in (1, 2, 3)]
    for steps in ([1, 2, 3], (0, 2, 3), [1, 2, 3, 9], {0: 1, 1: 2, 2: 3}, torch.tensor([1, 2, 3]), [1.5, 2.5, 3.0]):
        opt.prepare(steps, [1, 0, 2, 0])
        assert _rows(opt)["bc1_inv"].tolist() == pytest.approx(want, rel=1e-7)
        assert list(_rows(opt)["active"]) == [1, 0, 1]
    for steps, active in (([1], None), ([], None), ([1, 2], None), ([1, 2, 3], [True]), ([1, 2, 3], True)):
        with pytest.raises((IndexError, TypeError)):
            opt.prepare(steps, active)
    opt.beta1 = 1.0
    with pytest.raises(ZeroDivisionError):
        opt.prepare([1, 2, 3])


def _optimizer_on_a_fake_device(monkeypatch):
    """FlatAdamW whose launches note the descriptors on the device; `captured` collects what a stream capture
    would record (uploads and launches), to be replayed."""
    from nl_hecate_b200 import optimizer as om
    opt = om.FlatAdamW([8, 8], device="cpu")
    opt.seen = []
    captured = []
    state = {"capturing": False}
    nt, item = len(opt.sizes), om._DESC

    def launch(name, **k):
        if name == "nlh_adamw_multi_tensor":
            op = lambda: opt.seen.append(opt._desc_dev.t.numpy().view(item)["active"].tolist())
            captured.append(op) if state["capturing"] else op()

    class Dev:
        def __init__(self, t):
            self.t = t

        def copy_(self, src, non_blocking=False):
            op = lambda: self.t.copy_(src)
            captured.append(op) if state["capturing"] else op()

    class Event:
        def record(self, *a):
            assert not state["capturing"]

        def synchronize(self):
            pass

    monkeypatch.setattr(om, "call", launch)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    opt._desc_dev = Dev(torch.zeros(nt * item.itemsize, dtype=torch.uint8))
    opt._uploaded = [Event() for _ in range(om.RING)]

    @contextlib.contextmanager
    def capture():
        state["capturing"] = True
        yield
        state["capturing"] = False

    def replay():
        for op in captured:
            op()
    return opt, capture, replay


FLAGS = [[1, 0], [0, 1], [1, 1], [0, 0], [1, 0], [0, 1], [0, 0]]


@pytest.mark.parametrize("warmed_up", [False, True])
def test_a_captured_launch_uploads_the_descriptors_of_each_replay(monkeypatch, warmed_up):
    """prepare() and replay() in turn: the graph that captured launch() holds the upload, whether or not a
    prepare() was pending when it was captured."""
    opt, capture, replay = _optimizer_on_a_fake_device(monkeypatch)
    if warmed_up:
        opt.step(1e-3, [1, 1], [1, 1])
    else:
        opt.prepare([1, 1], [1, 1])
    with capture():
        opt.launch(1e-3)
    opt.seen.clear()
    for f in FLAGS:
        opt.prepare([1, 1], f)
        replay()
    assert opt.seen == FLAGS


def test_an_upload_before_the_capture_stays_out_of_the_graph(monkeypatch):
    """prepare(), upload() and replay() in turn, as StackedMAG does: the rows of the ring are used in turn and
    the graph copies none of them; eager steps before and after use their own."""
    opt, capture, replay = _optimizer_on_a_fake_device(monkeypatch)
    opt.step(1e-3, [1, 1], [1, 1])
    opt.prepare([1, 1], [0, 0])
    opt.upload()
    with capture():
        opt.launch(1e-3)
    opt.seen.clear()
    rows = set()
    for f in FLAGS:
        opt.prepare([1, 1], f)
        opt.upload()
        rows.add(opt._row)
        replay()
    assert opt.seen == FLAGS and len(rows) > 1
    opt.step(1e-3, [1, 1], [0, 1])
    opt.launch(1e-3)                       # the same descriptors again
    assert opt.seen[-2:] == [[0, 1], [0, 1]]


def test_call_refuses_wrong_arguments_with_a_type_error(monkeypatch):
    """Names are checked before anything else, an empty call's too; a value that its C type cannot hold
    raises TypeError, a pointer of an unknown kind ctypes.ArgumentError."""
    import ctypes
    from nl_hecate_b200 import dispatch as D
    bound = []
    monkeypatch.setattr(D, "bind_stream", lambda: bound.append(1))
    for kw in ({}, {"option": 3}, {"option": 3, "valu": 1}, {"option": 3, "value": 1, "more": 0}):
        with pytest.raises(TypeError, match="missing"):
            D.call("nlh_set_option", **kw)
    assert not bound
    with pytest.raises(TypeError):
        D.call("nlh_set_option", option=3.0, value=1)
    with pytest.raises(ctypes.ArgumentError):
        D.call("nlh_simple_rng_fill", state=1.5, scale=1.0, out_host=None, n=0)
    assert D.call("nlh_set_option", option=torch.tensor(3), value=True) == 0


def test_copy_rows_refuses_overlapping_rows():
    """Rows closer than their length are refused whatever their alignment, before anything is launched."""
    from nl_hecate_b200 import ffi
    for stride, row_len in ((4, 8), (0, 4), (2, 3), (-4, 4)):
        assert ffi.lib().nlh_copy_rows(64, stride, 64, 2, row_len) == ffi.lib().nlh_copy_rows(64, 4, 64, -1, 4)
