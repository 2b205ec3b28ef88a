"""Which buffer a block call takes (no GPU needed): streams apart, continuing calls with the call they continue, captures
with their graph.  Streams, captures and the allocator are stand-ins."""

import pytest

torch = pytest.importorskip("torch")

from skyrl_tx_rocm_b200 import ops  # noqa: E402

CUDA0 = torch.device("cuda", 0)


class Machine:
    def __init__(self):
        self.stream, self.captures = 0, {}


@pytest.fixture
def machine(monkeypatch):
    m = Machine()
    empty = torch.empty
    monkeypatch.setattr(ops, "_stream_of", lambda idx: m.stream)
    monkeypatch.setattr(ops, "_capture_id", lambda stream: m.captures.get(stream, 0))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: m.stream in m.captures)
    monkeypatch.setattr(ops.torch, "empty", lambda n, dtype, device: empty(n, dtype=dtype))
    ops._drop_workspaces(0)
    ops._thread.capture = None
    yield m
    ops._drop_workspaces(0)
    ops._thread.capture = None
    ops._replayed_workspaces.clear()


def take(machine, stream, nbytes=1000, fresh=True):
    machine.stream = stream
    return ops._workspace_buffer(CUDA0, nbytes, fresh)


def test_streams_have_buffers_of_their_own_and_keep_them(machine):
    a, b = take(machine, 0), take(machine, 7)
    assert a is not b and take(machine, 0) is a and take(machine, 7) is b
    assert take(machine, 0, 5000) is not a and take(machine, 7) is b


def test_a_call_that_continues_another_takes_its_buffer_on_any_stream(machine):
    side = take(machine, 7)
    main = take(machine, 0)
    assert take(machine, 7, fresh=False) is main and take(machine, 0, fresh=False) is main
    assert take(machine, 7) is side            # what is fresh there does not share it
    assert take(machine, 0, fresh=False) is side and take(machine, 0) is main


def test_a_capture_owns_its_buffers(machine):
    eager = take(machine, 7)
    machine.captures[7] = 41
    first = take(machine, 7)
    assert first is not eager and take(machine, 7, fresh=False) is first and take(machine, 7) is first
    machine.captures[9] = 41                   # a stream forked into the same capture
    assert take(machine, 9, fresh=False) is first and take(machine, 9) is not first
    machine.captures = {7: 42}
    assert take(machine, 7) is not first
    machine.captures = {}
    assert take(machine, 7) is eager and ops._thread.capture is None


def test_an_eager_buffer_that_a_capture_continues_on_is_kept(machine):
    eager = take(machine, 0)
    machine.captures[7] = 43
    assert take(machine, 7, fresh=False) is eager
    machine.captures = {}
    take(machine, 0, 10000)
    assert any(kept is eager for kept in ops._replayed_workspaces)


def test_registered_buffers_come_first_and_are_never_outgrown(machine):
    buf = torch.zeros(4096, dtype=torch.uint8)
    ops._registered_workspaces[0] = buf
    assert take(machine, 0) is buf and take(machine, 7, fresh=False) is buf
    with pytest.raises(ops.SkyrlKernelError, match="registered"):
        take(machine, 0, 1 << 20)


def test_the_number_of_kept_buffers_is_bounded(machine):
    for s in range(3 * ops.MAX_STREAM_WORKSPACES):
        take(machine, s)
    assert len(ops._stream_workspaces) == ops.MAX_STREAM_WORKSPACES
